// FP32 two-pass step (compiled with FMA contraction).
#include "twopass_impl.cuh"

XFB_INSTANTIATE_TWOPASS(float)
