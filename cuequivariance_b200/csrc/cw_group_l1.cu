// Channelwise kernels of the paths that read an irrep of degree 1.
#include "cw_kernels.cuh"

CW_DEFINE_GROUP(kGroupL1, CW_GROUP_L1)
