// FP32 blocked 2-D step (compiled with FMA contraction).
#include "tb2d_impl.cuh"

XFB_INSTANTIATE_TB2D(float)
