// 4- and 5-level Cayley kernels. FP32: the tensor-core kernels (1 x 128) for
// dense field-free matrices, the CUDA-core ones (1 x 256; for 4 levels 1 x
// 192, which fits 12 warps on an SM) for the block-diagonal ones of media
// with a diagonal Hamiltonian, which skip most of that product; the autotuner
// times both (65,536 points, us a step, dense / diagonal: 4 levels 6.3 and
// 7.7 / 5.9 and 5.1, 5 levels 12.5 and 14.1 / 12.1 and 9.6, 6 levels 21.5 and
// 31.7 / 21.0 and 15.8).
#include "inst.cuh"
MBG_REG_TC_P(ALGO_CAYLEY, 4)
MBG_REG_CAY_P(float, 4, 1, 192)
MBG_REG_CAY(double, 4, 1, 128)
MBG_REG_TC_P(ALGO_CAYLEY, 5)
MBG_REG_CAY(float, 5, 1, 256)
MBG_REG_CAY(double, 5, 1, 128)
