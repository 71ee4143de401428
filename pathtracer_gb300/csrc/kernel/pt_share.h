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

// Samples a warp claims at once in a launch of `share` samples a warp: a
// quarter of the share in multiples of 32, so that the last claims leave
// something for every warp, 32 at least and `cap` at most.  (Without the cap up
// to a share of 2048: 512x512 spheres 16 spp, a share of 1379, 0.893 ms for
// 0.863; 23 spp 1.258 for 1.183; Cornell box 23 spp 4.71 for 4.64.)
PT_HD int warp_chunk(uint64_t share, int cap) {
    if (share >= 4 * (uint64_t)cap) return cap;
    const int n = (int)share / 128 * 32;
    return n < 32 ? 32 : n;
}
