// pt_ring.cuh — the job ring and the flags word of a path, shared by the
// staged kernels (pt_wavefront.cu) and the persistent one (pt_persist.cu).
#pragma once

#include "pt_march.cuh"
#include "pt_path.cuh"

namespace {

// The flags word of s8: bit 30 the shadow-ray flag (kShadowFlag), bits
// 28-29 the extension dielectrics' path bits (PathState::medium), the bounce
// count below.
constexpr uint32_t kMediumShift = 28;
constexpr uint32_t kBounceMask = (1u << kMediumShift) - 1u;
PT_DI uint32_t bounce_word(const PathState& ps) {
    return ((uint32_t)ps.medium << kMediumShift) | ((uint32_t)ps.bounce & kBounceMask);
}

// The ring entry of the pass that holds global sample s: the last pass in
// [lo, hi) with first <= s (passes are appended in increasing order of first).
PT_DI uint32_t find_job(const WfJob* __restrict__ jobs, uint32_t cap, uint32_t lo, uint32_t hi, uint64_t s) {
    // invariant: jobs[lo % cap].first <= s < jobs[hi % cap].first (or hi is the end)
    while (hi - lo > 1) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (jobs[mid % cap].first <= s) {
            lo = mid;
        } else {
            hi = mid;
        }
    }
    return lo % cap;
}

// Samples of every pass added so far: the end of the last pass.
PT_DI uint64_t jobs_total(const WfArgs& A, uint32_t hi) {
    if (hi == 0) return 0;
    const WfJob& L = A.jobs[(hi - 1) % A.job_cap];
    return L.first + (uint64_t)L.count;
}

// Adds 1 to jobs[job].finished for every lane with pred, one atomic per
// distinct job in the warp.  Called by all 32 lanes.
PT_DI void count_finished(WfJob* __restrict__ jobs, uint32_t job, bool pred) {
    const unsigned active = __ballot_sync(0xffffffffu, pred);
    if (!active) return;
    const unsigned same = __match_any_sync(0xffffffffu, pred ? job : 0xffffffffu);
    if (pred && (__ffs(same & active) - 1) == (int)(threadIdx.x & 31))
        atomicAdd(&jobs[job].finished, (uint32_t)__popc(same & active));
}

}  // namespace
