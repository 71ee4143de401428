// pt_share.h — how the persistent kernels (pt_persist.cu, pt_fp64.cu) share a
// launch's paths among their warps.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define PT_HD __host__ __device__ inline
#else
#define PT_HD inline
#endif

// Path slots a warp uses of the `cap` it has arrays for, in a launch of `share`
// paths a warp: as many as that, in multiples of `step` and at least `least`
// (no more than cap), but never more than cap.
PT_HD int warp_slots(uint64_t share, int least, int step, int cap) {
    if (share >= (uint64_t)cap) return cap;
    const int n = ((int)share + step - 1) / step * step;
    return n < least ? least : n < cap ? n : cap;
}
