// Small 1D problems' main loop, FP64 (compiled with -fmad=false: bit-exact).
#define MC_REAL double
#define MC_LAUNCH_NAME launch_run1d_fp64
#include "run1d_impl.cuh"
