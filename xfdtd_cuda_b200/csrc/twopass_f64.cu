// FP64 two-pass step (compiled with --fmad=false: every operation individually
// rounded, in the reference's order).
#include "twopass_impl.cuh"

XFB_INSTANTIATE_TWOPASS(double)
