// pt_wavefront.cu — the wavefront renderer: path state in HBM, compacted
// ray queues, a persistent SDF-march kernel with per-lane ray refill.
//
// The plain megakernel keeps one pixel per thread, so lanes wait for the
// slowest neighbour's SDF march and for pixels with more work (measured:
// 5.3 of 32 lanes active per warp instruction).  Here every path sample of a
// dispatch is an independent work item in a pool of P slots; each iteration
// runs three stage kernels over compacted queues:
//   march  persistent: each lane holds one ray and does one SDF evaluation
//          per step (sign probe, march step, normal probes), several steps
//          between refills from the queue, so all lanes execute the same SDF
//          code -> finished rays to this iteration's SHADE queues;
//   shade  shadow-ray results, then primary hits: emitter / miss / BRDF
//          sample / light sample / Russian roulette (the shared pt_path.cuh
//          functions); finished samples write their XYZ and free their slot;
//          the ray a path continues with is intersected at once (analytic
//          primitives, SDF boxes) and goes to the next iteration's MARCH or
//          SHADE queue;
//   gen    start new samples in free slots, intersect their camera rays the
//          same way.
// A one-thread bookkeeping kernel advances the counters.  Queues are filled
// with warp-aggregated atomics (ballot + popc + one atomicAdd per warp).
// After the last sample, `resolve` sums each pixel's samples in sample order
// and applies Rendering/Accumulate — the same float operations, in the same
// order, as the megakernel and the shader, so results are bit-identical.
// The larger pt_mathf functions are called out of line here (smaller stage
// kernels); the SDF plug-ins use inlined math regardless.
//
// pt_wavefront_checked.cu compiles this file a second time with
// PT_DEBUG_CHECKS (every queue, pool-slot, ring and sample index checked
// before use; pt_check in pt_march.cuh) and its launch functions renamed by
// PTK_WF; the engine picks either set (ptk_wavefront_kernels).
#define PTM_OUTLINE
#define PT_UNROLL_MENGER
#include <cuda_runtime.h>

#ifndef PTK_WF
#define PTK_WF(name) name
#endif

#include "pt_march.cuh"
#include "pt_path.cuh"
#include "pt_ring.cuh"
#include "pt_wavefront.h"

namespace {

// A shadow-ray result's state: the bounce's next ray (s0, s1), the NEE
// term and the next throughput made with the shadow ray (s3, s5: see
// shade_shadow_made), the SDF set its march started with (s2.w, in s3's
// sector), the radiance, wavelengths and RNG/pass words and,
// traced, the event word.  The light sample's geometry and the BRDF those
// two came from are not stored, so they are neither read here.
template <bool TRACE>
PT_DI void load_for_shadow(const PoolView& v, uint32_t slot, PathState& ps, float4& contrib, uint32_t& sign_set,
                           uint32_t& flags, uint32_t& sample, uint32_t& job) {
    const float4 a = v.s0[slot], b = v.s1[slot];
    ps.org = f3(a.x, a.y, a.z);
    ps.mis = a.w;
    ps.dir = f3(b.x, b.y, b.z);
    ps.brdfPdf = b.w;
    ps.shDir = f3(0.0f, 0.0f, 0.0f);
    ps.cosL = 0.0f;
    ps.nrm = f3(0.0f, 0.0f, 0.0f);
    ps.lightPdf = 0.0f;
    ps.brdf = f4s(0.0f);
    sign_set = __float_as_uint(v.s2[slot].w);
    contrib = v.s3[slot];
    ps.rr = v.s5[slot];
    ps.radiance = v.s6[slot];
    ps.l = v.s7[slot];
    const uint4 m = v.s8[slot];
    ps.seed = m.x;
    flags = m.y;
    ps.bounce = (int)(m.y & kBounceMask);
    ps.medium = (int)((m.y >> kMediumShift) & 3u);
    sample = m.z;
    ps.shObj = word_shobj(m.w);
    job = word_job(m.w);
    if (TRACE) {
        const float4 e = v.s9[slot];
        ps.shLightID = e.x;
        ps.ev = __float_as_uint(e.y);
    } else {
        ps.shLightID = -1.0f;
        ps.ev = 0u;
    }
}

// A new sample's state.  Its first step is a primary ray (march, then
// shade_primary), which reads neither the shadow-ray fields (s2, s3), the
// BRDF (s4) nor the light pick (s9.x) and writes what a shadow ray reads
// before it reads it; at bounce 0 the throughput, the radiance and the event word
// are start_sample's constants (1, 0, 0), which load_for_primary sets
// instead of reading s5, s6 and s9.  So only s0, s1, s7 and s8 are stored.
PT_DI void store_new_sample(const PoolView& v, uint32_t slot, const PathState& ps, uint32_t sample, uint32_t job) {
    v.s0[slot] = make_float4(ps.org.x, ps.org.y, ps.org.z, ps.mis);
    v.s1[slot] = make_float4(ps.dir.x, ps.dir.y, ps.dir.z, ps.brdfPdf);
    v.s7[slot] = ps.l;
    v.s8[slot] = make_uint4(ps.seed, bounce_word(ps), sample, job_word(job, ps.shObj));
}

// Sample id s of a dispatch: k = s / (W*H), pixel = s % (W*H).  The colour
// buffer is [k][pixel], so `resolve` reads it coalesced; traces use the
// megakernel's path index pixel * spf + k.
PT_DI size_t trace_index(const pt_push& pc, uint32_t s) {
    const uint32_t npix = (uint32_t)pc.resolution[0] * (uint32_t)pc.resolution[1];
    return (size_t)(s % npix) * (size_t)pc.samplesPerFrame + (size_t)(s / npix);
}

// Intersection for a ray a stage has just produced (the reference's
// Intersection up to SphereTracing, SC:862-923 and SC:779-790): analytic
// primitives, then the SDF bounding boxes.  Writes the hit record and, for a
// ray that needs sphere tracing, the march start state (the march kernel
// picks it up like a ray it suspended).  Returns true for such a ray.
// `shadow`: a shadow ray towards light object shObj, marched only when an
// SDF hit can change what it reports.  sign_k: the SDF's sign at the origin
// as queue_sign gave it for the set sign_set (0: not known); a ray with that
// set starts past its sign probe.  *set_out: the ray's set (0: no march).
PT_DI bool route_ray(const WfArgs& A, const PoolView& v, const KScene& S, uint32_t slot, float3 org, float3 dir,
                     bool shadow, int shObj, uint32_t sign_k, uint32_t sign_set, uint32_t* set_out) {
    Hit h;
    h.hitdist = PT_MAXDIST;
    h.normal = f3(0.0f, 0.0f, 0.0f);
    h.materialID = 0.0f;
    h.lightID = -1.0f;
    int objectID = -1;
    intersect_analytic(S, S.objects, org, dir, h, objectID, shadow);
    bool march = false;
    uint32_t set1 = 0;
    if (S.meta.n[5] > 0 && !(shadow && !shadow_needs_march(objectID, shObj))) {
        const float3 invdir = f3(1.0f / dir.x, 1.0f / dir.y, 1.0f / dir.z);
        float2 tmm = make_float2(PT_MAXDIST, PT_MAXDIST);
        march = search_sdf(S, org, invdir, tmm, set1);
        if (march) {
            // not suspended, or past the sign probe like a suspended march
            const uint32_t word = (sign_k != 0u && sign_set == set1) ? march_word((float)((int)sign_k - 2), 0, 0) : 0u;
            v.m0[slot] = make_float4(fmaxf(tmm.x, 1e-3f), 0.0f, kOmegaMax, 0.0f);
            v.m1[slot] = make_float4(tmm.x, tmm.y, __uint_as_float(word), __uint_as_float(set1));
        }
    }
    if (set_out) *set_out = march ? set1 : 0u;
    v.h0[slot] = make_float4(h.hitdist, h.materialID, h.lightID, __int_as_float(objectID));
    v.h1[slot] = make_float4(h.normal.x, h.normal.y, h.normal.z, 0.0f);
    return march;
}

// Appends a routed ray to the next iteration's queues: march, or shading of
// a primary hit or of a shadow-ray result.  Called by all 32 lanes.
PT_DI void push_routed(const WfArgs& A, WfCounters& C, uint32_t nxt, uint32_t slot, bool valid, bool march,
                       bool shadow_ray, uint32_t job) {
    const uint32_t group = (A.groups > 1 && valid && march) ? A.jobs[job].group : 0u;
    q_push(A, A.q_march[nxt], &C.n_march[nxt], march_entry(slot, group), valid && march);
    q_push(A, A.q_shade[nxt], &C.n_shade[nxt], slot, valid && !march && !shadow_ray);
    q_push(A, A.q_shadow[nxt], &C.n_shadow[nxt], slot, valid && !march && shadow_ray);
}

__global__ void PT_GEN_BOUNDS wf_gen(const __grid_constant__ WfArgs A) {
    WfCounters& C = *A.counters;
    const uint32_t job_lo = C.job_lo, job_hi = C.job_hi;
    const uint64_t remaining = jobs_total(A, job_hi) - C.next_sample;
    const uint32_t n = (uint32_t)min((uint64_t)C.n_free, remaining);
    const uint32_t nfree = C.n_free;
    const uint64_t first = C.next_sample;
    const uint32_t nxt = C.cur ^ 1u;
    const PoolView v = view(A);
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
        const uint32_t i = base + threadIdx.x;
        bool valid = i < n;
        uint32_t slot = 0, job = 0;
        bool march = false;
        if (valid) valid = pt_check(A, nfree - n + i, A.pool_size, PT_CHECK_FREE_INDEX);
        if (valid) {
            slot = A.q_free[nfree - n + i];
            valid = pt_check(A, slot, A.pool_size, PT_CHECK_QUEUE_SLOT);
        }
        if (valid) {
            const uint64_t s = first + i;
            job = find_job(A.jobs, A.job_cap, job_lo, job_hi, s);
            const WfJob& J = A.jobs[job];
            const uint32_t local = J.local_base + (uint32_t)(s - J.first);
            const pt_push& pc = J.pc;
            const int W = pc.resolution[0], H = pc.resolution[1];
            const uint32_t npix = (uint32_t)W * (uint32_t)H;
            const uint32_t k = local / npix, pix = local % npix;
            const int x = (int)(pix % (uint32_t)W), y = (int)(pix / (uint32_t)W);
            const uint32_t xx = (uint32_t)x, yy = (uint32_t)H - (uint32_t)y;
            const float uvx = (2.0f * (float)xx - (float)W) / (float)H;
            const float uvy = (2.0f * (float)yy - (float)H) / (float)H;
            const CamInfo cam = J.cam;
            PathState ps;
            start_sample(ps, *J.scene, pc, cam, xx, yy, uvx, uvy, (int)k);
            ps.brdfPdf = 0.0f;
            ps.shLightID = -1.0f;
            ps.shObj = 0;
            ps.ev = 0;
            store_new_sample(v, slot, ps, local, job);
            march = route_ray(A, v, *J.scene, slot, ps.org, ps.dir, false, 0, 0u, 0u, nullptr);
        }
        push_routed(A, C, nxt, slot, valid, march, false, job);
    }
}

__global__ void wf_job_add(const __grid_constant__ WfArgs A, const WfJob job, uint32_t index, uint32_t lo) {
    WfJob& J = A.jobs[index % A.job_cap];
    J = job;
    J.finished = 0;
    J.cam = make_camera(job.pc);
    WfCounters& C = *A.counters;
    C.job_hi = index + 1;
    C.job_lo = lo;
}

// A primary hit reads neither the shadow-ray fields (s2, s3) nor the BRDF
// (s4): it writes them.
template <bool TRACE>
PT_DI void load_for_primary(const PoolView& v, uint32_t slot, PathState& ps, uint32_t& flags, uint32_t& sample,
                            uint32_t& job) {
    const float4 a = v.s0[slot], b = v.s1[slot];
    ps.org = f3(a.x, a.y, a.z);
    ps.mis = a.w;
    ps.dir = f3(b.x, b.y, b.z);
    ps.brdfPdf = b.w;
    ps.shDir = f3(0.0f, 0.0f, 0.0f);
    ps.cosL = 0.0f;
    ps.nrm = f3(0.0f, 0.0f, 0.0f);
    ps.lightPdf = 0.0f;
    ps.brdf = f4s(0.0f);
    ps.l = v.s7[slot];
    const uint4 m = v.s8[slot];
    ps.seed = m.x;
    flags = m.y;
    ps.bounce = (int)(m.y & kBounceMask);
    ps.medium = (int)((m.y >> kMediumShift) & 3u);
    sample = m.z;
    ps.shObj = word_shobj(m.w);
    job = word_job(m.w);
    // A first hit (bounce 0) has start_sample's throughput 1, radiance 0 and
    // no events yet (store_new_sample stores none of them).  s9 holds the
    // light pick and the event word, which only a traced dispatch keeps.
    if (ps.bounce == 0) {
        ps.rr = f4s(1.0f);
        ps.radiance = f4s(0.0f);
        ps.ev = 0u;
    } else {
        ps.rr = v.s5[slot];
        ps.radiance = v.s6[slot];
        ps.ev = TRACE ? __float_as_uint(v.s9[slot].y) : 0u;
    }
    ps.shLightID = -1.0f;
}

// After a shadow-ray result only the throughput, the radiance, the RNG and
// bounce word and (traced) the event word change.  The wavelengths (s7)
// never change but are stored with s8 so the pair's sector is written
// whole (a partial sector write makes the L2 read the rest from DRAM).
PT_DI void store_after_shadow(const PoolView& v, uint32_t slot, const PathState& ps, uint32_t sample, uint32_t job,
                              bool trace) {
    v.s5[slot] = ps.rr;
    v.s6[slot] = ps.radiance;
    v.s7[slot] = ps.l;
    v.s8[slot] = make_uint4(ps.seed, bounce_word(ps), sample, job_word(job, ps.shObj));
    if (trace) v.s9[slot] = make_float4(ps.shLightID, __uint_as_float(ps.ev), 0.0f, 0.0f);
}

// The end of a shaded step: trace records, the sample's colour when the
// path ended, the queues.
template <bool TRACE>
PT_DI void finish_shade(const WfArgs& A, const WfJob& J, const PathState& ps, StepResult r, uint32_t sample,
                        bool& freed) {
    const pt_push& pc = J.pc;
    // trace and colour indices
    const bool in_pass = pt_check(A, sample - J.local_base, J.count, PT_CHECK_SAMPLE);
    if (TRACE && r != STEP_SHADOW && A.trace.events && in_pass) {
        const size_t p = trace_index(pc, sample);
        const int b = ps.bounce - 1;
        if (b < A.trace.cap) A.trace.events[p * (size_t)A.trace.cap + b] = ps.ev;
    }
    if (r == STEP_TERMINATED && !in_pass) {
        freed = true;
    } else if (r == STEP_TERMINATED) {
        const float3 col = sample_color(ps, *J.scene, J.cie);
        J.colors[sample] = make_float4(col.x, col.y, col.z, 0.0f);
        if (TRACE) {
            const size_t p = trace_index(pc, sample);
            if (A.trace.nevents) A.trace.nevents[p] = (uint32_t)ps.bounce;
            if (A.trace.colors) {
                A.trace.colors[3 * p] = col.x;
                A.trace.colors[3 * p + 1] = col.y;
                A.trace.colors[3 * p + 2] = col.z;
            }
        }
        freed = true;
    }
}

// Shading in two passes over two queues, so each warp runs one kind of step
// and moves only the state that kind reads and writes: shadow-ray results
// (the light sample's contribution, then the bounce's end), then primary
// hits (emission or BRDF and light sampling).
template <bool TRACE>
__global__ void PT_SHADE_BOUNDS wf_shade(const __grid_constant__ WfArgs A) {
    WfCounters& C = *A.counters;
    const uint32_t cur = C.cur, nxt = cur ^ 1u;
    const PoolView v = view(A);
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t ns = C.n_shadow[cur];
    for (uint32_t base = blockIdx.x * blockDim.x; base < ns; base += stride) {
        const uint32_t i = base + threadIdx.x;
        bool valid = i < ns;
        uint32_t slot = 0, job = 0;
        bool again = false, freed = false, march = false;
        uint32_t entry = 0;
        if (valid) {
            entry = A.q_shadow[cur][i];
            slot = entry & kQueueSlotMask;
            valid = pt_check(A, slot, A.pool_size, PT_CHECK_QUEUE_SLOT) &&
                    pt_check(A, slot_job(v, slot), A.job_cap, PT_CHECK_JOB);
        }
        if (valid) {
            PathState ps;
            float4 contrib;
            uint32_t flags, sample, sign_set;
            load_for_shadow<TRACE>(v, slot, ps, contrib, sign_set, flags, sample, job);
            const WfJob& J = A.jobs[job];
            const int objectID = (entry & kQueueSdfHit) ? -2 : __float_as_int(v.h0[slot].w);
            const float4 rr_next = ps.rr;
            const StepResult r = shade_shadow_made<TRACE>(ps, objectID, contrib, rr_next, J.pc.pathLength);
            finish_shade<TRACE>(A, J, ps, r, sample, freed);
            if (!freed) {
                store_after_shadow(v, slot, ps, sample, job, TRACE);
                again = true;
                // the bounce's next primary ray, set up with the primary hit;
                // it leaves the shadow ray's origin
                march = route_ray(A, v, *J.scene, slot, ps.org, ps.dir, false, 0, queue_sign(entry), sign_set,
                                  nullptr);
            }
        }
        push_routed(A, C, nxt, slot, again, march, false, job);
        q_push(A, A.q_free, &C.n_free, slot, freed);
        count_finished(A.jobs, job, freed);
    }
    const uint32_t np = C.n_shade[cur];
    for (uint32_t base = blockIdx.x * blockDim.x; base < np; base += stride) {
        const uint32_t i = base + threadIdx.x;
        bool valid = i < np;
        uint32_t slot = 0, job = 0;
        bool again = false, freed = false, march = false, shadow_next = false;
        if (valid) {
            slot = A.q_shade[cur][i];
            valid = pt_check(A, slot, A.pool_size, PT_CHECK_QUEUE_SLOT) &&
                    pt_check(A, slot_job(v, slot), A.job_cap, PT_CHECK_JOB);
        }
        if (valid) {
            PathState ps;
            uint32_t flags, sample;
            load_for_primary<TRACE>(v, slot, ps, flags, sample, job);
            const WfJob& J = A.jobs[job];
            const float4 h0 = v.h0[slot], h1 = v.h1[slot];
            Hit h;
            h.hitdist = h0.x;
            h.materialID = h0.y;
            h.lightID = h0.z;
            h.normal = f3(h1.x, h1.y, h1.z);
            const int objectID = __float_as_int(h0.w);
            const StepResult r = shade_primary<TRACE>(ps, *J.scene, h, objectID, J.pc.pathLength);
            finish_shade<TRACE>(A, J, ps, r, sample, freed);
            if (!freed) {
                // the path state.  For a light sample's shadow ray: its
                // direction and first SDF set (s2) and, made now with the
                // shadow step's own operations (shade_shadow_made), the NEE
                // term (s3) and the bounce's next throughput (s5), so the
                // shadow step reads neither the light sample's geometry nor
                // the BRDF (s4 is kept only when traced, beside s9).  A next
                // bounce's primary ray reads none of s2-s4.
                shadow_next = (r == STEP_SHADOW);
                v.s0[slot] = make_float4(ps.org.x, ps.org.y, ps.org.z, ps.mis);
                v.s1[slot] = make_float4(ps.dir.x, ps.dir.y, ps.dir.z, ps.brdfPdf);
                if (shadow_next) {
                    v.s3[slot] = shadow_contribution(ps, *J.scene);
                    if (TRACE) v.s4[slot] = ps.brdf;
                }
                v.s5[slot] = shadow_next ? bounce_throughput(ps) : ps.rr;
                v.s6[slot] = ps.radiance;
                v.s7[slot] = ps.l;  // unchanged: written with s8 so their sector is written whole
                v.s8[slot] =
                    make_uint4(ps.seed, (shadow_next ? kShadowFlag : 0u) | bounce_word(ps), sample, job_word(job, ps.shObj));
                // traced: the light picked and the event word
                if (TRACE) v.s9[slot] = make_float4(ps.shLightID, __uint_as_float(ps.ev), 0.0f, 0.0f);
                // the light sample's shadow ray, or the next bounce
                uint32_t set1 = 0;
                march = route_ray(A, v, *J.scene, slot, ps.org, shadow_next ? ps.shDir : ps.dir, shadow_next,
                                  word_shobj(job_word(job, ps.shObj)), 0u, 0u, &set1);
                if (shadow_next)
                    v.s2[slot] = make_float4(ps.shDir.x, ps.shDir.y, ps.shDir.z, __uint_as_float(set1));
                again = true;
            }
        }
        push_routed(A, C, nxt, slot, again, march, shadow_next, job);
        q_push(A, A.q_free, &C.n_free, slot, freed);
        count_finished(A.jobs, job, freed);
    }
}

// The MARCH queue by group (groups > 1): the entries of each group counted,
// then every entry into its group's range of q_sorted, a tile of the queue per
// block and trip (one atomic per tile and group).  12 B of traffic an entry.
// Without it a march warp's lanes run the snippets of whatever scenes its rays
// come from, one after another: four generated SDF jobs 512x512x32 took 350 ms
// in one batch and 138 ms one by one.
constexpr int kSortItems = 8;  // entries per thread and tile
template <bool SCATTER>
__global__ void __launch_bounds__(kStageThreads) wf_group(const __grid_constant__ WfArgs A) {
    WfCounters& C = *A.counters;
    const uint32_t n = C.n_march[C.cur];
    const uint32_t* __restrict__ q = A.q_march[C.cur];
    __shared__ uint32_t count[kMarchGroups], base[kMarchGroups];
    const uint32_t tile = kStageThreads * kSortItems;
    for (uint32_t t0 = blockIdx.x * tile; t0 < n; t0 += gridDim.x * tile) {
        if (threadIdx.x < kMarchGroups) count[threadIdx.x] = 0;
        __syncthreads();
        uint32_t entry[kSortItems], rank[kSortItems];
#pragma unroll
        for (int k = 0; k < kSortItems; k++) {
            const uint32_t i = t0 + k * kStageThreads + threadIdx.x;
            const bool in = i < n;
            entry[k] = in ? q[i] : 0u;
            // one shared atomic per group in the warp
            const unsigned same = __match_any_sync(0xffffffffu, in ? (entry[k] >> 28) : 16u);
            const int leader = __ffs(same) - 1;
            uint32_t at = 0;
            if (in && (int)(threadIdx.x & 31) == leader) at = atomicAdd(&count[entry[k] >> 28], (uint32_t)__popc(same));
            at = __shfl_sync(0xffffffffu, at, leader);
            rank[k] = at + (uint32_t)__popc(same & ((1u << (threadIdx.x & 31)) - 1u));
        }
        __syncthreads();
        if (threadIdx.x < kMarchGroups && count[threadIdx.x]) {
            if (SCATTER) {
                uint32_t first = 0;
                for (int g = 0; g < (int)threadIdx.x; g++) first += C.group_count[g];
                base[threadIdx.x] = first + atomicAdd(&C.group_next[threadIdx.x], count[threadIdx.x]);
            } else {
                atomicAdd(&C.group_count[threadIdx.x], count[threadIdx.x]);
            }
        }
        __syncthreads();
        if (SCATTER) {
#pragma unroll
            for (int k = 0; k < kSortItems; k++) {
                if (t0 + k * kStageThreads + threadIdx.x >= n) continue;
                const uint32_t at = base[entry[k] >> 28] + rank[k];
                if (pt_check(A, at, A.pool_size, PT_CHECK_QUEUE_APPEND)) A.q_sorted[at] = entry[k];
            }
            __syncthreads();
        }
    }
}

__global__ void wf_book(const __grid_constant__ WfArgs A) {
    WfCounters& C = *A.counters;
    const uint32_t pool = A.pool_size;
    const uint64_t total = jobs_total(A, C.job_hi);
    const uint32_t n = (uint32_t)min((uint64_t)C.n_free, total - C.next_sample);
    C.total = total;
    C.next_sample += n;
    C.n_free -= n;
    C.n_march[C.cur] = 0;
    C.n_shade[C.cur] = 0;
    C.n_shadow[C.cur] = 0;
    C.cur ^= 1u;
    C.march_cursor = 0;
    if (A.groups > 1)
        for (int g = 0; g < kMarchGroups; g++) C.group_count[g] = C.group_next[g] = 0;
    C.iterations += 1;
    C.live = pool - C.n_free;
    // the next iteration's queues and the free list fit the pool
    const uint32_t c = C.cur;
    (void)(pt_check(A, C.n_march[c], pool + 1u, PT_CHECK_QUEUE_COUNT) &&
           pt_check(A, C.n_shade[c], pool + 1u, PT_CHECK_QUEUE_COUNT) &&
           pt_check(A, C.n_shadow[c], pool + 1u, PT_CHECK_QUEUE_COUNT) &&
           pt_check(A, C.n_free, pool + 1u, PT_CHECK_QUEUE_COUNT));
}

__global__ void wf_init(WfCounters* __restrict__ Cp, uint32_t* __restrict__ q_free, uint32_t pool) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < pool) q_free[i] = i;
    if (i == 0) {
        WfCounters& C = *Cp;
        C.n_march[0] = C.n_march[1] = 0;
        C.n_shade[0] = C.n_shade[1] = 0;
        C.n_shadow[0] = C.n_shadow[1] = 0;
        C.cur = 0;
        C.march_cursor = 0;
        C.n_free = pool;
        C.next_sample = 0;
        C.total = 0;
        C.iterations = 0;
        C.live = 0;
        C.job_lo = C.job_hi = 0;
        C.pk_begin = C.pk_end = 0;
        C.check_site = 0;
        C.check_index = 0;
        for (int g = 0; g < kMarchGroups; g++) C.group_count[g] = C.group_next[g] = 0;
    }
}

// Rendering + Accumulate over one pass's ordered sample colours, one thread per pixel.
__global__ void __launch_bounds__(kStageThreads) wf_resolve(const pt_push pc, float4* __restrict__ accum,
                                                           const float4* __restrict__ colors) {
    const uint32_t npix = (uint32_t)pc.resolution[0] * (uint32_t)pc.resolution[1];
    const uint32_t pix = blockIdx.x * blockDim.x + threadIdx.x;
    if (pix >= npix) return;
    float3 sum = f3(0.0f, 0.0f, 0.0f);
    for (int k = 0; k < pc.samplesPerFrame; k++) {
        const float4 c = colors[(size_t)k * npix + pix];
        sum = sum + f3(c.x, c.y, c.z);
    }
    accum[pix] = accumulate(pc, sum, accum[pix]);
}

}  // namespace

cudaError_t PTK_WF(ptk_wavefront_launch_init)(const WfArgs* a, cudaStream_t stream) {
    wf_init<<<(a->pool_size + 255) / 256, 256, 0, stream>>>(a->counters, a->q_free, a->pool_size);
    return cudaGetLastError();
}

cudaError_t PTK_WF(ptk_wavefront_launch_job_add)(const WfArgs* a, const WfJob* job, uint32_t index, uint32_t lo,
                                         cudaStream_t stream) {
    wf_job_add<<<1, 1, 0, stream>>>(*a, *job, index, lo);
    return cudaGetLastError();
}

// Blocks of a stage kernel resident on the device at once (SMs x the
// kernel's occupancy), cached per kernel: a grid beyond it would leave its
// last blocks for a second wave.
static int resident_blocks(const void* kernel, int* cache) {
    if (*cache) return *cache;
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kStageThreads, 0) != cudaSuccess ||
        per_sm <= 0)
        return 1 << 30;  // unknown: no cap
    *cache = sms * per_sm;
    return *cache;
}

const void* PTK_WF(ptk_wavefront_march)(uint32_t kinds) {
    kinds &= ~(1u << PT_SDF_NONE);
    if ((kinds & ~kKindsEven) == 0) return reinterpret_cast<const void*>(wf_march_even);
    if ((kinds & ~kKindsBulb) == 0) return reinterpret_cast<const void*>(wf_march_bulb);
    return reinterpret_cast<const void*>(wf_march);
}

cudaError_t PTK_WF(ptk_wavefront_launch_iteration)(const WfArgs* a, bool trace, int grid, cudaStream_t stream,
                                           cudaEvent_t* stage_events, const void* march_kernel) {
    // stage_events (optional): 6 events recorded before isect, march, shade,
    // gen, bookkeeping and after it, for per-stage device times.
    // (Intersection is done by shade and gen for the rays they produce: the
    // isect interval stays empty.)
    if (stage_events) cudaEventRecord(stage_events[0], stream);
    if (a->groups > 1) {
        wf_group<false><<<grid, kStageThreads, 0, stream>>>(*a);
        wf_group<true><<<grid, kStageThreads, 0, stream>>>(*a);
    }
    if (stage_events) cudaEventRecord(stage_events[1], stream);
    if (march_kernel) {
        void* argv[] = {const_cast<WfArgs*>(a)};
        const cudaError_t e = cudaLaunchKernel(march_kernel, dim3(grid), dim3(kStageThreads), argv, 0, stream);
        if (e != cudaSuccess) return e;
    } else {
        wf_march<<<grid, kStageThreads, 0, stream>>>(*a);
    }
    if (stage_events) cudaEventRecord(stage_events[2], stream);
    static int shade_cap[2] = {0, 0}, gen_cap = 0;
    if (trace) {
        const int g = min(grid, resident_blocks(reinterpret_cast<const void*>(wf_shade<true>), &shade_cap[1]));
        wf_shade<true><<<g, kStageThreads, 0, stream>>>(*a);
    } else {
        const int g = min(grid, resident_blocks(reinterpret_cast<const void*>(wf_shade<false>), &shade_cap[0]));
        wf_shade<false><<<g, kStageThreads, 0, stream>>>(*a);
    }
    if (stage_events) cudaEventRecord(stage_events[3], stream);
    wf_gen<<<min(grid, resident_blocks(reinterpret_cast<const void*>(wf_gen), &gen_cap)), kStageThreads, 0,
             stream>>>(*a);
    if (stage_events) cudaEventRecord(stage_events[4], stream);
    wf_book<<<1, 1, 0, stream>>>(*a);
    if (stage_events) cudaEventRecord(stage_events[5], stream);
    return cudaGetLastError();
}

cudaError_t PTK_WF(ptk_wavefront_launch_resolve)(const WfArgs* a, uint32_t job, const pt_push* pc, float4* accum,
                                         const float4* colors, cudaStream_t stream) {
    (void)a;
    (void)job;
    const uint32_t npix = (uint32_t)pc->resolution[0] * (uint32_t)pc->resolution[1];
    wf_resolve<<<(npix + kStageThreads - 1) / kStageThreads, kStageThreads, 0, stream>>>(*pc, accum, colors);
    return cudaGetLastError();
}

// pt_persist.cu
cudaError_t PTK_WF(ptk_persist_launch)(const WfArgs* a, int variant, int sms, uint64_t budget,
                                       const KScene* one_scene, cudaStream_t stream);
int PTK_WF(ptk_persist_blocks_per_sm)(int variant);

extern const WfKernelSet PTK_WF(ptk_wavefront_kernel_set);
const WfKernelSet PTK_WF(ptk_wavefront_kernel_set) = {
    PTK_WF(ptk_wavefront_launch_init),        PTK_WF(ptk_wavefront_launch_job_add),
    PTK_WF(ptk_wavefront_launch_iteration),   PTK_WF(ptk_wavefront_march),
    PTK_WF(ptk_persist_launch),               PTK_WF(ptk_persist_blocks_per_sm),
    PTK_WF(ptk_wavefront_launch_resolve),
#if !defined(PT_DEBUG_CHECKS)
    ptk_wavefront_finish,
#else
    nullptr,
#endif
};
