// Channelwise kernels of the paths that read an irrep of degree 2, float64.
#include "cw_kernels.cuh"

CW_DEFINE_GROUP_F64(kGroupL2F64, CW_GROUP_L2)
