// 4- and 5-level coherence-vector kernels (V = 15, 24).
#include "inst.cuh"
MBG_REG_TC_P(ALGO_CVR, 4, MEDIUM_ANY)
MBG_REG_CVR(float, 4, 1, 256)
MBG_REG_CVR(double, 4, 1, 128)
MBG_REG_TC_P(ALGO_CVR, 5, MEDIUM_ANY)
MBG_REG_CVR(float, 5, 1, 256)
MBG_REG_CVR(double, 5, 1, 128)
