// FP32 batches of 3-D scenes (compiled with FMA contraction).
#include "engine.cuh"

XFB_INSTANTIATE_BATCH(float)
