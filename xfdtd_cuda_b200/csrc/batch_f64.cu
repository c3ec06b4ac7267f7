// FP64 batches of 3-D scenes (compiled with --fmad=false: every operation individually rounded).
#include "engine.cuh"

XFB_INSTANTIATE_BATCH(double)
