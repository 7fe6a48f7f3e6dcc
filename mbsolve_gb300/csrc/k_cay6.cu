// 6-level Cayley kernels (see k_cay456.cu).
#include "inst.cuh"
MBG_REG_TC_P(ALGO_CAYLEY, 6, MEDIUM_OTHER)
MBG_REG_CAY(float, 6, 1, 256)
MBG_REG_CAY(double, 6, 1, 128)
