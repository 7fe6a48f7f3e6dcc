// 6-level coherence-vector kernels (V = 35).
#include "inst.cuh"
MBG_REG_TC_P(ALGO_CVR, 6, MEDIUM_ANY)
MBG_REG_CVR(float, 6, 1, 256)
MBG_REG_CVR(double, 6, 1, 128)
