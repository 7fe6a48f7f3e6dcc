// FP32 Cayley kernels of 4 to 6 levels at 1 x 128 for media with diagonal
// Hamiltonians (see k_cay456.cu).
#include "inst.cuh"
MBG_REG_CAY_P(float, 4, 1, 128, MEDIUM_DIAG)
MBG_REG_CAY_P(float, 5, 1, 128, MEDIUM_DIAG)
MBG_REG_CAY_P(float, 6, 1, 128, MEDIUM_DIAG)
