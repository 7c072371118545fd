// FP32 instantiation of the column kernel: gas optics and two-stream
// transfer in FP32 (FMA contraction allowed); setcoef interpolation weights,
// Planck integrals, cloud optics and the flux sums / flux divergence stay
// FP64 inside the kernel.
#include <algorithm>
#include <cstdio>

#include <type_traits>

// FP32 gas optics at 4 CTAs per SM (128 registers, no spills), 16,384 x 127: 2.74 ms, against 3.91, 3.12,
// 2.74 and 4.59 ms at 2, 3, 5 and 6; FP64 runs best at 3 (4.40 ms, against 5.41 at 2 and 4.65 at 4).
#define LW_GAS_MINB 4

#include "lw_launch.h"
#include "lw_rt.cuh"
#include "lw_rt_grid.cuh"

#define REAL float
#define LW_SCRATCH_FN scratch_per_column_fp32
#define LW_LAUNCH_FN launch_column_fp32
#define LW_PREPARE_FN prepare_column_fp32
#define LW_NLAUNCH_FN launches_column_fp32
#define LW_DBG_FN rrtmg_lw_gpu_debug_read_fp32
#include "lw_column_launch.inc"
