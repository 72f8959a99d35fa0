// Channelwise kernels of the paths that read an irrep of degree 0.
#include "cw_kernels.cuh"

CW_DEFINE_GROUP(kGroupL0, CW_GROUP_L0)
