// pt_march.cuh — the wavefront engine's SDF march kernel (wf_march) and the
// helpers every stage kernel shares.  Included by pt_wavefront.cu and, for
// scenes whose SDF text is compiled at run time, by the NVRTC program of
// pt_jit.cu (with PT_JIT_USER_SDF, in namespace ptjit), so both builds run
// the same source.
#pragma once

#include "pt_geometry.cuh"
#include "pt_wavefront.h"

#if defined(PT_JIT_USER_SDF)
namespace ptjit {
#else
namespace {
#endif

constexpr uint32_t kShadowFlag = 1u << 30;
constexpr int kStageThreads = 256;
// Launch bounds of the stage kernels: resident blocks of kStageThreads per SM
// asked of the compiler (registers capped at 65536 / (256 x blocks)); the
// host caps each kernel's grid at what is resident.  Measured on GB300: the
// march kernel at 4 blocks (64 registers) and shade and gen, which also
// intersect the rays they produce, at 3 (85 registers, no spills) are 1-12 %
// faster end to end than the neighbouring choices.  PT_WF_<STAGE>_BLOCKS
// overrides a count; 0 leaves only the block size.
#ifndef PT_WF_SHADE_BLOCKS
#define PT_WF_SHADE_BLOCKS 3
#endif
#ifndef PT_WF_MARCH_BLOCKS
#define PT_WF_MARCH_BLOCKS 4
#endif
#ifndef PT_WF_GEN_BLOCKS
#define PT_WF_GEN_BLOCKS 3
#endif
#if PT_WF_SHADE_BLOCKS > 0
#define PT_SHADE_BOUNDS __launch_bounds__(kStageThreads, PT_WF_SHADE_BLOCKS)
#else
#define PT_SHADE_BOUNDS __launch_bounds__(kStageThreads)
#endif
#if PT_WF_MARCH_BLOCKS > 0
#define PT_MARCH_BOUNDS __launch_bounds__(kStageThreads, PT_WF_MARCH_BLOCKS)
#else
#define PT_MARCH_BOUNDS __launch_bounds__(kStageThreads)
#endif
#if PT_WF_GEN_BLOCKS > 0
#define PT_GEN_BOUNDS __launch_bounds__(kStageThreads, PT_WF_GEN_BLOCKS)
#else
#define PT_GEN_BOUNDS __launch_bounds__(kStageThreads)
#endif
// wf_march: after a large queue is drained, a warp with fewer rays than
// WfArgs::drain_lanes suspends those that have marched kDrainMinSteps steps
// in this launch, for the next iteration.
constexpr int kDrainMinSteps = 8;

// SphereTracing's over-relaxation start (SC:781).
constexpr float kOmegaMax = 1.70f;

// Index checks of the checked build (PT_DEBUG_CHECKS, the kernels of
// pt_wavefront_checked.cu and checked run-time compiled march kernels):
// true when i < n; otherwise the first failure since the last reset is
// recorded in the counters (site, index) for the host, and the caller skips
// the access.  The default build checks nothing: the function is constant
// true and its arguments are dead code.
#if defined(PT_DEBUG_CHECKS)
PT_DI bool pt_check(const WfArgs& A, uint32_t i, uint32_t n, uint32_t site) {
    if (i < n) return true;
    if (atomicCAS(&A.counters->check_site, 0u, site) == 0u) A.counters->check_index = i;
    return false;
}
#else
PT_DI constexpr bool pt_check(const WfArgs&, uint32_t, uint32_t, uint32_t) { return true; }
#endif

// Warp-aggregated append of `value` to queue[count++] for lanes with pred.
// Must be called by all 32 lanes of the warp.  Every queue holds up to
// pool_size entries.
PT_DI void q_push(const WfArgs& A, uint32_t* __restrict__ queue, uint32_t* count, uint32_t value, bool pred) {
    const unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (mask == 0) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(count, (uint32_t)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    const uint32_t at = base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
    if (pred && pt_check(A, at, A.pool_size, PT_CHECK_QUEUE_APPEND)) queue[at] = value;
}

// One 16-byte field of the pool's pairs (WfPool): element slot of a field
// is the first or second half of the slot's 32-byte pair.
template <typename T> struct PairField {
    T* p;
    PT_DI T& operator[](uint32_t slot) const { return p[2u * slot]; }
};
template <typename T> PT_DI PairField<T> first_of(float4* pair) { return PairField<T>{reinterpret_cast<T*>(pair)}; }
template <typename T> PT_DI PairField<T> second_of(float4* pair) {
    return PairField<T>{reinterpret_cast<T*>(pair) + 1};
}

struct PoolView {
    PairField<float4> s0, s1, s2, s3, s4, s5, s6, s7;  // see WfPool
    PairField<uint4> s8;
    PairField<float4> s9, h0, h1, m0, m1;
};

// An entry of the shadow queues: the slot and what
// the march kernel found for the shadow ray, so that a marched shadow ray
// writes nothing else: bit 31 an SDF hit, bits 29-30 the SDF's sign at the
// ray's origin + 2 (0: not marched).
constexpr uint32_t kQueueSlotMask = kMaxPoolSlots - 1u;
// An entry of the MARCH queues: the slot and, above it, the ray's march group.
PT_DI uint32_t march_entry(uint32_t slot, uint32_t group) { return slot | (group << 28); }
static_assert(kMarchGroups <= 16, "march groups must fit the four bits above a slot");
constexpr uint32_t kQueueSdfHit = 1u << 31;
PT_DI uint32_t shadow_entry(uint32_t slot, bool hit, float k) {
    return slot | (hit ? kQueueSdfHit : 0u) | ((k > 0.0f ? 3u : (k < 0.0f ? 1u : 2u)) << 29);
}
PT_DI uint32_t queue_sign(uint32_t entry) { return (entry >> 29) & 3u; }

// The word in m1.z of a suspended march: bit 31 set, the SDF sign k
// (-1, 0, 1) + 1 in bits 26-27, points in bits 10-25 and the loop
// iterations in bits 0-9.  A ray fresh from intersection has 0 there.
PT_DI uint32_t march_word(float k, int points, int iter) {
    const uint32_t kc = (k > 0.0f) ? 2u : ((k < 0.0f) ? 0u : 1u);
    return 0x80000000u | (kc << 26) | ((uint32_t)min(points, 0xffff) << 10) | (uint32_t)iter;
}

PT_DI PoolView view(const WfArgs& A) {
    const WfPool& p = A.pool;
    return PoolView{first_of<float4>(p.s01), second_of<float4>(p.s01), first_of<float4>(p.s23),
                    second_of<float4>(p.s23), first_of<float4>(p.s49), first_of<float4>(p.s56),
                    second_of<float4>(p.s56), first_of<float4>(p.s78), second_of<uint4>(p.s78),
                    second_of<float4>(p.s49), first_of<float4>(p.h01), second_of<float4>(p.h01),
                    first_of<float4>(p.m01), second_of<float4>(p.m01)};
}

// s8.w packs the path's pass (its job-ring entry, 20 bits) with the
// object index of its sampled light (12 bits, signed): a ray's pass is read
// with its RNG word and flags in one load.
constexpr uint32_t kJobShift = 12;
static_assert(PT_MAX_SCENE_OBJECTS < 2048, "object indices must fit the 12-bit signed field of s8.w");
static_assert(kMaxJobRing <= (1u << (32 - kJobShift)), "job-ring entries must fit the 20-bit field of s8.w");
PT_DI uint32_t job_word(uint32_t job, int shObj) { return (job << kJobShift) | ((uint32_t)shObj & 0xFFFu); }
PT_DI uint32_t word_job(uint32_t w) { return w >> kJobShift; }
PT_DI int word_shobj(uint32_t w) { return (int)(w << 20) >> 20; }
PT_DI uint32_t slot_job(const PoolView& v, uint32_t slot) { return word_job(v.s8[slot].w); }

// SphereTracing (SC:779-860) with one SDF evaluation per loop iteration per
// lane.  A converged ray takes its six normal probes on its own lane
// (MP_NORMAL0..5), or leaves the lane for the warp's normal stage
// (march_rays<true>).
enum MarchPhase { MP_EMPTY = 0, MP_SIGN = 1, MP_STEP = 2, MP_NORMAL0 = 3, MP_NORMAL5 = 8, MP_CONVERGED = 9 };

// The normal stage: converged rays whose normal (CalculateNumericalSDFNormals,
// SC:721-730) and material are still to be taken, per warp.  Sixteen rays'
// 96 probes are evaluated together, three trips with every lane busy, so
// near-surface probes (the longest loops of an escape-time fractal) run
// beside each other and a ray's own lane goes on to its next ray.
constexpr int kNormalBatch = 16;
constexpr int kNormalCap = kNormalBatch - 1 + 32;  // fewer than a batch kept, and a round's 32
struct NormalStage {
    float4 at[kNormalCap];   // p.xyz, t
    uint4 of[kNormalCap];    // set1, slot, scene pointer
    int sel[kNormalCap];     // hit_sel (scene_sdf_material_hit)
    float probe[6 * kNormalBatch];
};

// The SDFs a lane's evaluation walks (scene_sdf_sel): its set and, of those
// that it may walk with others (group: walk_of), the ones in a set of the
// warp.  Called by all 32 lanes.
PT_DI uint32_t warp_walk(bool on, uint32_t set1, uint32_t group) {
#if defined(PT_ONE_SDF)
    return 1u;
#else
    return (__reduce_or_sync(0xffffffffu, on ? set1 : 0u) & group) | set1;
#endif
}

// Warp-staged queue appends: lanes with pred add `value` to a per-warp
// buffer of 64 in shared memory (count warp-uniform); every 32 entries go to
// the queue with one atomic and one coalesced store.  Called by all 32 lanes.
PT_DI void stage_push(const WfArgs& A, uint32_t* buf, uint32_t& count, bool pred, uint32_t value, uint32_t* queue,
                      uint32_t* qcount, int lane) {
    const unsigned m = __ballot_sync(0xffffffffu, pred);
    if (!m) return;
    if (pred) buf[count + (uint32_t)__popc(m & ((1u << lane) - 1u))] = value;
    count += (uint32_t)__popc(m);  // < 64: it was < 32 before
    if (count < 32) return;
    __syncwarp();
    uint32_t b = 0;
    if (lane == 0) b = atomicAdd(qcount, 32u);
    b = __shfl_sync(0xffffffffu, b, 0);
    if (pt_check(A, b + (uint32_t)lane, A.pool_size, PT_CHECK_QUEUE_APPEND)) queue[b + (uint32_t)lane] = buf[lane];
    const uint32_t rest = count - 32;
    const uint32_t moved = ((uint32_t)lane < rest) ? buf[32 + lane] : 0u;
    __syncwarp();
    if ((uint32_t)lane < rest) buf[lane] = moved;
    __syncwarp();
    count = rest;
}

// Appends what stage_push still holds.  Called by all 32 lanes.
PT_DI void stage_flush(const WfArgs& A, uint32_t* buf, uint32_t count, uint32_t* queue, uint32_t* qcount, int lane) {
    __syncwarp();
    if (!count) return;
    uint32_t b = 0;
    if (lane == 0) b = atomicAdd(qcount, count);
    b = __shfl_sync(0xffffffffu, b, 0);
    if ((uint32_t)lane < count && pt_check(A, b + (uint32_t)lane, A.pool_size, PT_CHECK_QUEUE_APPEND))
        queue[b + (uint32_t)lane] = buf[lane];
}

// Probe j of a hit at p: p +- h.xyy, h.yxy, h.yyx.
template <typename P> PT_DI float3 probe_point(const P& p, int j) {
    const float e = 1e-4f;
    const float ex = (j == 0) ? e : 0.0f, ey = (j == 2) ? e : 0.0f, ez = (j == 4) ? e : 0.0f;
    const float mx = (j == 1) ? e : 0.0f, my = (j == 3) ? e : 0.0f, mz = (j == 5) ? e : 0.0f;
    return (j & 1) ? f3(p.x - mx, p.y - my, p.z - mz) : f3(p.x + ex, p.y + ey, p.z + ez);
}

// The normal stage's evaluation: in run-time compiled kernels by calls of the
// plug-ins' cold copy, since a second inlined copy of a long snippet cost
// registers and instruction cache (12-iteration mandelbulb 131.3 against
// 130.0 ms); inlined it is as fast or faster for the shipped plug-ins.
template <uint32_t KINDS> PT_DI float probe_sdf(const KScene& S, float3 q, uint32_t set1, uint32_t walk) {
    int sel;
#if defined(PT_JIT_USER_SDF)
    return scene_sdf_sel<KINDS, true>(S, q, set1, walk, sel);
#else
    return scene_sdf_sel<KINDS>(S, q, set1, walk, sel);
#endif
}

// Normals and materials of records [from, from + n), n <= kNormalBatch, into
// their hit records; returns the record's slot to lane i < n (for the shade
// queue).  Called by all 32 lanes.
template <uint32_t KINDS>
PT_DI uint32_t take_normals(const PoolView& v, NormalStage& ns, int from, int n, int lane) {
    __syncwarp();
#pragma unroll 1
    for (int base = 0; base < 6 * n; base += 32) {
        const int i = base + lane, r = i / 6, j = i - 6 * r;  // probe j of record r
        const bool on = i < 6 * n;
        float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        uint4 b = make_uint4(0u, 0u, 0u, 0u);
        if (on) {
            a = ns.at[from + r];
            b = ns.of[from + r];
        }
        const KScene& S = *reinterpret_cast<const KScene*>((uint64_t)b.z | ((uint64_t)b.w << 32));
        const uint32_t walk = warp_walk(on, b.x, on ? walk_of(S, b.x) : 0u);
        if (on) {
            const float3 q = probe_point(a, j);
            ns.probe[i] = probe_sdf<KINDS>(S, q, b.x, walk);
        }
    }
    __syncwarp();
    uint32_t slot = 0;
    if (lane < n) {
        const float* d = ns.probe + 6 * lane;
        const float4 a = ns.at[from + lane];
        const uint4 b = ns.of[from + lane];
        const KScene& S = *reinterpret_cast<const KScene*>((uint64_t)b.z | ((uint64_t)b.w << 32));
        slot = b.y;
        const float3 nrm = normalize3(f3(d[0] - d[1], d[2] - d[3], d[4] - d[5]));
        const float mat = scene_sdf_material_hit(S, f3(a.x, a.y, a.z), b.x, ns.sel[from + lane]);
        v.h0[slot] = make_float4(a.w - 1e-3f, mat, -1.0f, __int_as_float(-2));
        v.h1[slot] = make_float4(nrm.x, nrm.y, nrm.z, 0.0f);
    }
    __syncwarp();  // the records may be overwritten from here on
    return slot;
}

// The march loop over the SDF plug-ins KINDS (bit k: kind k).  STAGED: normals
// in the warp's normal stage; otherwise on each ray's lane, where the probes
// fill the rest of the round: better where every evaluation costs about the
// same.  Measured on GB300 with the scene's kinds: menger + terrain 1080p 16
// spp on the lane 93.9 ms, staged 103.5; against probing at the end of every
// round, up to five rays a pass: 12-iteration mandelbulb 1024x1024x64 staged
// 130.0 ms, 132.4 so; shipped mandelbulb 777x431x16 11.4 ms, 11.7 so.
template <bool STAGED, uint32_t KINDS>
PT_DI void march_rays(const WfArgs& A) {
    WfCounters& C = *A.counters;
    const uint32_t cur = C.cur;
    const uint32_t n = C.n_march[cur];
    const uint32_t* __restrict__ qin = A.groups > 1 ? A.q_sorted : A.q_march[cur];
    const PoolView v = view(A);
    const PoolView& M = v;
    const int lane = threadIdx.x & 31;
    const int budget = A.march_budget;
    const int refill_min = A.refill_min;
    const int inner = A.march_inner;
    int steps = 0;
    // Draining only pays while the queue holds more rays than the grid has lanes.
    const bool many = n >= 2u * gridDim.x * blockDim.x;
    // Queue entries per claim: up to 32 while the queue is long, 1 near its end.
    const uint32_t nwarps = gridDim.x * (blockDim.x >> 5);
    const uint32_t chunk = max(1u, min(32u, n / (4u * nwarps)));
    uint32_t cbase = 0, cleft = 0;  // warp-uniform: unused entries of the warp's claim
    // Finished rays are staged per warp and kind and appended to the shade
    // queues 32 at a time.
    __shared__ uint32_t staged[kStageThreads / 32][2][64];
    uint32_t nstaged[2] = {0u, 0u};  // warp-uniform: primary hits, shadow results
    __shared__ NormalStage normals[STAGED ? kStageThreads / 32 : 1];
    int nnormals = 0;  // warp-uniform: records in the warp's normal stage
    const int wib = (int)(threadIdx.x >> 5);

    uint32_t entry = 0;  // the ray's queue entry: slot and group
    const KScene* Sp = nullptr;
    int phase = MP_EMPTY;
    bool exhausted = false;
    float3 org = f3(0.0f, 0.0f, 0.0f), dir = f3(0.0f, 0.0f, 1.0f), p = org;
    float t = 0.0f, insT = 0.0f, omega = 0.0f, prevR = 0.0f, hitdist = 0.0f, k = 0.0f, nplus = 0.0f;
    float3 nv = f3(0.0f, 0.0f, 0.0f);  // nplus, nv: normals on the ray's lane only
    float2 tmm = make_float2(0.0f, 0.0f);
    uint32_t set1 = 0, group = 0;
    int points = 0, iter = 0;
    bool xmarch = false;  // the ray's scene sets march limits (PT_EXT_MARCH; read from it where used)
    int hit_sel = -2;  // >= -1 once the lane's march converged (scene_sdf_material_hit)
    bool shadow_ray = false;
    const float omegaMax = kOmegaMax, omegaSpeed = 0.20f;

    for (;;) {
        // Refill lanes that have no ray (warp-aggregated fetch), once at
        // least refill_min of them are idle or the warp has none left.
        // Queue entries come from a chunk the warp claimed with one atomic
        // (cbase, cleft: warp-uniform); a refill that needs more than the
        // chunk holds claims the next chunk.
        const bool need = (phase == MP_EMPTY) && !exhausted;
        const unsigned mneed = __ballot_sync(0xffffffffu, need);
        if (mneed && (__popc(mneed) >= refill_min || __ballot_sync(0xffffffffu, phase != MP_EMPTY) == 0)) {
            const uint32_t want = (uint32_t)__popc(mneed);
            const uint32_t from_old = min(want, cleft);  // entries left in the current chunk
            const uint32_t old_base = cbase;
            uint32_t nb = 0;
            if (want > from_old) {
                const uint32_t ncount = max(chunk, want - from_old);
                if (lane == 0) nb = atomicAdd(&C.march_cursor, ncount);
                nb = __shfl_sync(0xffffffffu, nb, 0);
                cbase = nb + (want - from_old);
                cleft = ncount - (want - from_old);
            } else {
                cbase += want;
                cleft -= want;
            }
            if (need) {
                const uint32_t rank = (uint32_t)__popc(mneed & ((1u << lane) - 1u));
                const uint32_t idx = (rank < from_old) ? old_base + rank : nb + (rank - from_old);
                const uint32_t e = idx < n ? qin[idx] : 0u, slot = e & kQueueSlotMask;
                if (idx < n && pt_check(A, slot, A.pool_size, PT_CHECK_QUEUE_SLOT) &&
                    pt_check(A, slot_job(v, slot), A.job_cap, PT_CHECK_JOB)) {
                    entry = e;
                    const uint4 w8 = v.s8[slot];
                    Sp = A.jobs[word_job(w8.w)].scene;
                    const float4 o = v.s0[slot];
                    const uint32_t flags = w8.y;
                    shadow_ray = (flags & kShadowFlag) != 0;
                    const float4 d = shadow_ray ? v.s2[slot] : v.s1[slot];
                    org = f3(o.x, o.y, o.z);
                    dir = f3(d.x, d.y, d.z);
                    hitdist = v.h0[slot].x;
                    steps = 0;
                    hit_sel = -2;
                    // A ray from isect (flag bit clear: start with the sign
                    // probe) or one suspended by an earlier launch.
                    const float4 a0 = M.m0[slot], a1 = M.m1[slot];
                    const uint32_t saved = __float_as_uint(a1.z);
                    t = a0.x;
                    insT = a0.y;
                    omega = a0.z;
                    prevR = a0.w;
                    tmm = make_float2(a1.x, a1.y);
                    k = (float)(int)((saved >> 26) & 3u) - 1.0f;
                    set1 = __float_as_uint(a1.w);
                    group = walk_of(*Sp, set1);
                    iter = (int)(saved & 1023u);
                    points = (int)((saved >> 10) & 0xffffu);
                    xmarch = (Sp->ext.flags & PT_EXT_MARCH) != 0;
                    p = fma3s(dir, t, org);
                    phase = (saved & 0x80000000u) ? MP_STEP : MP_SIGN;
                } else if (idx >= n) {
                    exhausted = true;
                }
            }
        }
        const unsigned live = __ballot_sync(0xffffffffu, phase != MP_EMPTY);
        if (live == 0) break;
        // Once the queue is drained, a warp with few rays left would run on
        // with most lanes idle: its marching rays save their state and
        // continue in full warps next iteration instead.
        const bool drain = many && __ballot_sync(0xffffffffu, exhausted) != 0 && __popc(live) < A.drain_lanes;

        // A.march_inner SDF evaluations per lane before the warp refills,
        // shades finished hits and appends to the queues again: the warp
        // pays for those once per several evaluations, and a lane whose ray
        // finishes or is suspended on the way idles until then.
        bool finished = false, hit = false, suspend = false;
#pragma unroll 1
        for (int sub = 0; sub < inner; sub++) {
            // One SDF evaluation.
            const bool evalLane = (phase >= MP_SIGN && phase <= MP_NORMAL5) && !finished && !suspend;
            if (sub > 0 && __ballot_sync(0xffffffffu, evalLane) == 0) break;
            float3 q = p;
            if (phase == MP_SIGN) q = org;
            if (!STAGED && phase >= MP_NORMAL0 && phase <= MP_NORMAL5) q = probe_point(p, phase - MP_NORMAL0);
            float val = 0.0f;
            int esel = -1;
            const uint32_t walk = warp_walk(evalLane, set1, group);
            if (evalLane) val = scene_sdf_sel<KINDS>(*Sp, q, set1, walk, esel);
            if (!evalLane) continue;
            if (phase == MP_SIGN) {
                k = sign_glsl(val);
                phase = MP_STEP;
            } else if (STAGED || phase == MP_STEP) {
                const float radius = val;
                bool exitLoop = false;
                if (xmarch && t > Sp->ext.march_max_distance) {
                    finished = true;  // past the distance cap: no SDF hit
                } else if (insT > (fabsf(prevR) + fabsf(radius))) {
                    t -= insT;
                    omega = 1.0f;
                    insT = prevR * omega * k;
                    t += insT;
                    p = fma3s(dir, t, org);
                } else if (fabsf(radius) < (xmarch ? Sp->ext.march_epsilon : 1e-4f)) {
                    exitLoop = true;
                    hit_sel = esel;
                } else {
                    if (t > tmm.y) {
                        points += 1;
                    } else {
                        points = 0;
                    }
                    bool researched = false;
                    if (points >= 2) {
                        t = tmm.y + 1e-3f;
                        tmm = make_float2(PT_MAXDIST, PT_MAXDIST);
                        const float3 invdir = f3(1.0f / dir.x, 1.0f / dir.y, 1.0f / dir.z);
                        if (search_sdf(*Sp, fma3s(dir, t, org), invdir, tmm, set1)) {
                            group = walk_of(*Sp, set1);
                            tmm.x += t;
                            tmm.y += t;
                            t = fmaxf(tmm.x, t);
                            p = fma3s(dir, t, org);
                            researched = true;
                        } else {
                            finished = true;  // left every SDF box: no SDF hit
                        }
                    }
                    if (!finished && !researched) {
                        insT = radius * omega * k;
                        t += insT;
                        p = fma3s(dir, t, org);
                        const float omegaSpeedFactor = fminf(radius / prevR, 0.99f);
                        omega += omegaSpeed * (fminf(1.0f / (1.0f - omegaSpeedFactor), omegaMax) - omega);
                        prevR = radius;
                    }
                }
                if (!finished && !exitLoop) {
                    iter++;
                    if (iter >= (xmarch ? Sp->ext.march_max_steps : 512)) exitLoop = true;
                }
                if (exitLoop) {
                    if (shadow_ray) {  // reports only whether an SDF was hit
                        hit = t < hitdist;
                        finished = true;
                    } else if (t < hitdist) {
                        p = fma3s(dir, t, org);
                        phase = STAGED ? MP_CONVERGED : MP_NORMAL0;
                    } else {
                        finished = true;
                    }
                } else if (!finished && (++steps >= budget || (drain && steps >= kDrainMinSteps))) {
                    // out of budget for this launch: save the state, continue next iteration
                    const uint32_t slot = entry & kQueueSlotMask;
                    M.m0[slot] = make_float4(t, insT, omega, prevR);
                    M.m1[slot] = make_float4(tmm.x, tmm.y, __uint_as_float(march_word(k, points, iter)),
                                             __uint_as_float(set1));
                    suspend = true;
                }
            } else if (!STAGED) {
                const int j = phase - MP_NORMAL0;
                if ((j & 1) == 0) {
                    nplus = val;
                } else {
                    const float dv = nplus - val;
                    if (j == 1) nv.x = dv;
                    else if (j == 3) nv.y = dv;
                    else nv.z = dv;
                }
                phase++;
                if (phase > MP_NORMAL5) {
                    hit = true;
                    finished = true;
                }
            }
        }

        if constexpr (STAGED) {
            // Converged rays give their lanes up; a full batch of them takes
            // its normals.
            const unsigned conv = __ballot_sync(0xffffffffu, phase == MP_CONVERGED);
            if (conv) {
                NormalStage& ns = normals[wib];
                if (phase == MP_CONVERGED) {
                    const int at = nnormals + __popc(conv & ((1u << lane) - 1u));
                    const uint64_t sp = reinterpret_cast<uint64_t>(Sp);
                    ns.at[at] = make_float4(p.x, p.y, p.z, t);
                    ns.of[at] = make_uint4(set1, entry & kQueueSlotMask, (uint32_t)sp, (uint32_t)(sp >> 32));
                    ns.sel[at] = hit_sel;
                    phase = MP_EMPTY;
                }
                nnormals += __popc(conv);
                while (nnormals >= kNormalBatch) {
                    nnormals -= kNormalBatch;
                    const uint32_t ready = take_normals<KINDS>(v, ns, nnormals, kNormalBatch, lane);
                    stage_push(A, staged[wib][0], nstaged[0], lane < kNormalBatch, ready, A.q_shade[cur], &C.n_shade[cur],
                               lane);
                }
            }
        } else if (finished && hit && !shadow_ray) {
            const uint32_t slot = entry & kQueueSlotMask;
            const float3 nrm = normalize3(nv);
            const float mat = scene_sdf_material_hit(*Sp, p, set1, hit_sel);
            v.h0[slot] = make_float4(t - 1e-3f, mat, -1.0f, __int_as_float(-2));
            v.h1[slot] = make_float4(nrm.x, nrm.y, nrm.z, 0.0f);
        }
        stage_push(A, staged[wib][0], nstaged[0], finished && !shadow_ray, entry & kQueueSlotMask,
                   A.q_shade[cur], &C.n_shade[cur],
                   lane);
        stage_push(A, staged[wib][1], nstaged[1], finished && shadow_ray, shadow_entry(entry & kQueueSlotMask, hit, k), A.q_shadow[cur], &C.n_shadow[cur],
                   lane);
        q_push(A, A.q_march[cur ^ 1u], &C.n_march[cur ^ 1u], entry, suspend);
        if (finished || suspend) phase = MP_EMPTY;
    }
    // The staged remainders.
    if (STAGED && nnormals) {
        const uint32_t ready = take_normals<KINDS>(v, normals[wib], 0, nnormals, lane);
        stage_push(A, staged[wib][0], nstaged[0], lane < nnormals, ready, A.q_shade[cur], &C.n_shade[cur], lane);
    }
    stage_flush(A, staged[wib][0], nstaged[0], A.q_shade[cur], &C.n_shade[cur], lane);
    stage_flush(A, staged[wib][1], nstaged[1], A.q_shadow[cur], &C.n_shadow[cur], lane);
}

// The run-time compiled kernel holds its scenes' kinds (PT_SDF_KINDS); the
// built-in ones are compiled for every kind, for the mandelbulb alone and
// for the kinds without it, whose evaluations cost the same everywhere: the
// host picks the smallest that covers a dispatch.  Code of kinds that a
// scene does not have cost menger + terrain 10 % and the shipped mandelbulb
// 2 % (instruction cache, registers).
#if defined(PT_NO_MARCH_KERNELS)
// (a translation unit that takes only the helpers)
#elif defined(PT_JIT_USER_SDF)
__global__ void PT_MARCH_BOUNDS wf_march(const __grid_constant__ WfArgs A) { march_rays<true, PT_SDF_KINDS>(A); }
#else
constexpr uint32_t kKindsBulb = 1u << PT_SDF_MANDELBULB;
constexpr uint32_t kKindsEven = (1u << PT_SDF_BLOB) | (1u << PT_SDF_MENGER) | (1u << PT_SDF_TERRAIN);
__global__ void PT_MARCH_BOUNDS wf_march(const __grid_constant__ WfArgs A) { march_rays<true, 0xFFFFFFFFu>(A); }
__global__ void PT_MARCH_BOUNDS wf_march_bulb(const __grid_constant__ WfArgs A) { march_rays<true, kKindsBulb>(A); }
__global__ void PT_MARCH_BOUNDS wf_march_even(const __grid_constant__ WfArgs A) { march_rays<false, kKindsEven>(A); }
#endif

}  // namespace
