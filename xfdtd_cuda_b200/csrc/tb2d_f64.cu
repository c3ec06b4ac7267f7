// FP64 blocked 2-D step (compiled with --fmad=false: every operation individually rounded).
#include "tb2d_impl.cuh"

XFB_INSTANTIATE_TB2D(double)
