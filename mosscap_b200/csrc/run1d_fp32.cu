// Small 1D problems' main loop, FP32 compute form.
#define MC_REAL float
#define MC_LAUNCH_NAME launch_run1d_fp32
#include "run1d_impl.cuh"
