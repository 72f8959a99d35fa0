// Channelwise kernels of the paths that read an irrep of degree 3.
#include "cw_kernels.cuh"

CW_DEFINE_GROUP(kGroupL3, CW_GROUP_L3)
