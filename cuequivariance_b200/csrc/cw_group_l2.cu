// Channelwise kernels of the paths that read an irrep of degree 2.
#include "cw_kernels.cuh"

CW_DEFINE_GROUP(kGroupL2, CW_GROUP_L2)
