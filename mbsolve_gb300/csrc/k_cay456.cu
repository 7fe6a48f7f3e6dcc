// 4- and 5-level Cayley kernels. FP32 at 1 x 128: the tensor-core kernels for
// dense field-free matrices, the CUDA-core ones (k_cay_diag.cu), which skip
// most of that product, where every medium's is block-diagonal; at 1 x 256 (4
// levels: 1 x 192, which fits 12 warps on an SM) the CUDA-core ones for both.
// The autotuner times all that fit the media. 65,536 points, us a step,
// tensor cores 1 x 128 / CUDA cores 1 x 128 / CUDA cores at the wider shape:
//   dense     4 levels 6.26 / 6.54 / 6.67, 5: 12.8 / 14.3 / 13.9, 6: 21.9 / 33.5 / 31.5
//   diagonal  4 levels 6.25 / 4.97 / 5.10, 5: 12.8 / 9.97 / 9.62, 6: 21.8 / 18.2 / 15.8
#include "inst.cuh"
MBG_REG_TC_P(ALGO_CAYLEY, 4, MEDIUM_OTHER)
MBG_REG_CAY_P(float, 4, 1, 192, MEDIUM_ANY)
MBG_REG_CAY(double, 4, 1, 128)
MBG_REG_TC_P(ALGO_CAYLEY, 5, MEDIUM_OTHER)
MBG_REG_CAY(float, 5, 1, 256)
MBG_REG_CAY(double, 5, 1, 128)
