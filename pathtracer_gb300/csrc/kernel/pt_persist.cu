// pt_persist.cu — the persistent path kernel, every warp a wavefront of its own
// in shared memory: batches and dispatches of scenes without SDFs, dispatches of
// few samples of built-in SDFs, and the last paths of the staged engine
// (pt_wavefront.cu).
//
// pt_persist_checked.cu compiles this file a second time with
// PT_DEBUG_CHECKS (see pt_wavefront_checked.cu), without the takeover of last
// paths, which no caller with checks on runs.
#define PTM_OUTLINE
#define PT_COMPACT
#define PT_NO_MARCH_KERNELS
#include <cuda_runtime.h>

#ifndef PTK_WF
#define PTK_WF(name) name
#endif

#include "pt_march.cuh"
#include "pt_ring.cuh"
#include "pt_share.h"
#include "pt_wavefront.h"

namespace {

// Persistent mode: every warp runs a wavefront of its own.  It keeps
// kPersistSlots paths in shared memory and, per class of the step a path
// needs next, a list of them; each trip takes up to 32 paths of the longest
// list, does that step for all of them together and intersects the rays they
// go on with (one intersect_all for primary and shadow rays alike).  A path
// that ends writes its colour to its pass's colour buffer, which `resolve`
// sums in sample order, so results equal the megakernel's bit for bit, and
// its slot takes the next sample of the launch, across pixels and passes.
// A marched ray is marched to its end within a trip, so many samples of SDFs
// belong to the staged kernels; of few, the longest path decides the time.
//
// Why: with a path per lane every trip ran every step (emission, diffuse,
// mirror and glass surfaces, shadow results, new samples: 60 KB of code) for
// the few lanes that needed each, 16 of 32 lanes a trip, and waited for
// instruction fetch more than for anything else (5 to 7 of 13 cycles an
// issue).  Steps of one class run their code once for full warps.
constexpr int kPersistSlots = 80;
constexpr int kPersistChunk = 256;  // samples a warp claims at once, at most
constexpr int kPersistWarps = kPersistThreads / 32;
// A path's state, 7 x 16 B a slot (an odd count, so that slots spread over
// the banks):
//   0 org.xyz, mis          1 dir.xyz, seed     2 wavelengths   3 radiance
//   4 throughput (shadow ray in flight: the next bounce's)
//   5 hitdist, normal.xyz   (shadow ray: its NEE term)
//   6 materialID, lightID   (shadow ray: light object, object hit), pass
//     sample, flags (medium, bounce)
constexpr int kPersistQuads = 7;
// The classes of steps, and what a path on the PC_END list still needs.
enum PathClass { PC_SHADOW = 0, PC_DIFFUSE, PC_SPECULAR, PC_END, PC_COUNT };
static_assert(kPersistSlots <= 256, "a list entry holds its slot in 8 bits");
enum PathEnd { PE_HIT = 0, PE_COLOUR = 1, PE_START = 2 };  // shade an emitter or miss; write the colour; start
struct PersistShared {
    float4 state[kPersistWarps][kPersistSlots * kPersistQuads];
    uint32_t job[kPersistWarps][kPersistSlots];               // job-ring entry
    uint16_t list[kPersistWarps][PC_COUNT][kPersistSlots];    // slot | PathEnd << 8
    float spheres[6 * PT_MAX_SCENE_SPHERES];                  // the launch's spheres (single-pass launches)
};

__global__ void wf_persist_setup(const __grid_constant__ WfArgs A, uint64_t budget) {
    WfCounters& C = *A.counters;
    const uint64_t total = jobs_total(A, C.job_hi);
    const uint64_t begin = C.pk_end;  // warps of the last launch may have claimed past it
    const uint64_t end = (total - begin > budget) ? begin + budget : total;
    C.next_sample = begin;
    C.pk_begin = begin;
    C.pk_end = end;
    C.total = total;
    C.iterations += 1;
}

// The class of the step after a ray's intersection.
PT_DI int path_class(const KScene& S, const Hit& h, bool shadow) {
    if (shadow) return PC_SHADOW;
    if (!(h.hitdist < PT_MAXDIST) || light_mix(S, h.lightID).y > 0.0f) return PC_END;
    const pt_material_ext* xm = ext_material(S, h.materialID);
    return (xm && xm->type >= PT_BSDF_MIRROR) ? PC_SPECULAR : PC_DIFFUSE;
}

// POOL: takes queue entry e of the staged engine over into slot state q and
// ps.  A marching ray (`march`) is intersected again from its origin, whatever
// it had marched (the result is the same): returns PC_COUNT, with r telling
// its kind.  A hit or a shadow result (`result`) is ready to shade: returns
// its class.  -1: an index check failed.
PT_DI int load_staged(const WfArgs& A, const PoolView& v, uint32_t e, bool march, bool result, PathState& ps,
                      float4& contrib, float4* q, uint32_t& local, uint32_t& job, StepResult& r) {
    const uint32_t slot = e & kQueueSlotMask;
    if (!pt_check(A, slot, A.pool_size, PT_CHECK_QUEUE_SLOT)) return -1;
    const uint4 w = v.s8[slot];
    job = word_job(w.w);
    if (!pt_check(A, job, A.job_cap, PT_CHECK_JOB)) return -1;
    const KScene& S = *A.jobs[job].scene;
    const float4 a = v.s0[slot], b = v.s1[slot];
    const bool shadow = result || (march && (w.y & kShadowFlag) != 0);
    ps.org = f3(a.x, a.y, a.z);
    ps.mis = a.w;
    ps.dir = f3(b.x, b.y, b.z);
    ps.l = v.s7[slot];
    ps.seed = w.x;
    ps.bounce = (int)(w.y & kBounceMask);
    ps.medium = (int)((w.y >> kMediumShift) & 3u);
    ps.shObj = word_shobj(w.w);
    local = w.z;
    if (!shadow && ps.bounce == 0) {  // not stored for a first ray (store_new_sample)
        ps.rr = f4s(1.0f);
        ps.radiance = f4s(0.0f);
    } else {
        ps.rr = v.s5[slot];
        ps.radiance = v.s6[slot];
    }
    if (shadow) contrib = v.s3[slot];
    q[2] = ps.l;
    r = shadow ? STEP_SHADOW : STEP_CONTINUE;
    if (march) {
        if (shadow) {
            const float4 d = v.s2[slot];
            ps.shDir = f3(d.x, d.y, d.z);
        }
        return PC_COUNT;
    }
    const float4 h0 = v.h0[slot], h1 = v.h1[slot];
    const float4 ids = result ? make_float4(__int_as_float(ps.shObj),
                                            (e & kQueueSdfHit) ? __int_as_float(-2) : h0.w, 0.0f, 0.0f)
                              : h0;
    Hit h;
    h.hitdist = h0.x;
    h.normal = f3(h1.x, h1.y, h1.z);
    h.materialID = h0.y;
    h.lightID = h0.z;
    q[0] = a;
    q[1] = make_float4(b.x, b.y, b.z, __uint_as_float(w.x));
    q[3] = ps.radiance;
    q[4] = ps.rr;
    q[5] = result ? contrib : make_float4(h0.x, h1.x, h1.y, h1.z);
    q[6] = make_float4(result ? ids.x : h0.y, result ? ids.y : h0.z, __uint_as_float(local),
                       __uint_as_float(bounce_word(ps)));
    return path_class(S, h, result);
}

// The persistent path loop.  ONE: every sample of the launch belongs to one
// pass, whose scene S1 is the launch's parameter (the constant bank, as
// for the megakernel); otherwise each lane reads its pass's scene through
// the pass's pointer.
// POOL: the paths are those a staged engine has in flight (its queues of the
// coming iteration) instead of new samples; see wf_finish.
template <int FEAT, bool ONE, bool POOL>
PT_DI void persist_paths(const WfArgs& A, const KScene* S1) {
    extern __shared__ __align__(16) unsigned char persist_smem[];
    PersistShared& sh = *reinterpret_cast<PersistShared*>(persist_smem);
    WfCounters& C = *A.counters;
    const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5);
    const unsigned lt = (1u << lane) - 1u;
    // lanes can read different spheres at once
    if constexpr (ONE) {
        for (int i = threadIdx.x; i < 6 * S1->meta.n[0]; i += kPersistThreads) sh.spheres[i] = S1->objects[i];
        __syncthreads();
    }
    float4* const st = sh.state[warp];
    uint32_t* const jobs = sh.job[warp];
    const uint32_t cur = C.cur, nm = C.n_march[cur], np = C.n_shade[cur], ns = C.n_shadow[cur];  // POOL
    const PoolView pool = view(A);
    const uint64_t end = POOL ? (uint64_t)nm + np + ns : C.pk_end;
    const uint32_t job_lo = C.job_lo, job_hi = C.job_hi;
    // A small launch gives every warp its share at once: no more slots than
    // that, and chunks that leave something for the others.
    const uint64_t share = (end - (POOL ? 0 : C.pk_begin)) / ((uint64_t)gridDim.x * kPersistWarps);
    // A staged engine's last paths are spread over every warp: their time is
    // the longest path's, and a warp steps as long as its longest march.
    const int slots = POOL ? warp_slots(share + 1, 1, 1, kPersistSlots) : warp_slots(share, 32, 32, kPersistSlots);
    const uint32_t chunk = POOL ? min(32u, (uint32_t)share + 1) : (uint32_t)warp_chunk(share, kPersistChunk);
    int count[PC_COUNT] = {0, 0, 0, 0};  // warp-uniform: the lists' lengths
    for (int i = lane; i < slots; i += 32) sh.list[warp][PC_END][i] = (uint16_t)(i | (PE_START << 8));
    count[PC_END] = slots;
    __syncwarp();
    uint64_t cbase = 0;   // warp-uniform: unassigned samples of the warp's chunk
    uint32_t cleft = 0;
    uint32_t cjob = 0;      // warp-uniform: pass of the chunk's first sample,
    uint64_t cjob_end = 0;  // and the end of its sample range
    bool exhausted = false;  // warp-uniform: no sample left below `end`
    for (;;) {
        // The longest list; paths that end wait for persist_refill of them
        // while there is other work, so that new samples start together.
        int cls = PC_END, most = (count[PC_END] >= A.persist_refill) ? count[PC_END] : 0;
#pragma unroll
        for (int c = 0; c < PC_END; c++)
            if (count[c] > most) {
                most = count[c];
                cls = c;
            }
        if (most == 0) {
            cls = PC_END;
            most = count[PC_END];
        }
        if (most == 0) break;
        const int n = min(most, 32);
#pragma unroll
        for (int c = 0; c < PC_COUNT; c++)
            if (c == cls) count[c] -= n;
        const int from = most - n;
        bool live = lane < n;
        uint32_t slot = 0;
        int ends = PE_HIT;
        if (live) {
            const uint32_t e = sh.list[warp][cls][from + lane];
            slot = e & 0xffu;
            ends = (int)(e >> 8);
            live = pt_check(A, slot, (uint32_t)slots, PT_CHECK_WARP_SLOT);
        }
        __syncwarp();
        float4* const q = st + slot * kPersistQuads;
        uint32_t job = 0, local = 0;
        PathState ps;
        StepResult r = STEP_TERMINATED;
        bool coloured = false;
        float4 contrib = f4s(0.0f);
        int next = -1, next_end = PE_HIT;
        bool restored = false;  // POOL: taken over from the staged engine this trip
        if (live && ends != PE_START) {
            const float4 q0 = q[0], q1 = q[1], q5 = q[5], q6 = q[6];
            job = jobs[slot];
            const WfJob& J = A.jobs[job];
            const KScene& S = ONE ? *S1 : *J.scene;
            ps.org = f3(q0.x, q0.y, q0.z);
            ps.mis = q0.w;
            ps.dir = f3(q1.x, q1.y, q1.z);
            ps.seed = __float_as_uint(q1.w);
            ps.l = q[2];
            ps.radiance = q[3];
            ps.rr = q[4];
            local = __float_as_uint(q6.z);
            const uint32_t flags = __float_as_uint(q6.w);
            ps.bounce = (int)(flags & kBounceMask);
            ps.medium = (int)((flags >> kMediumShift) & 3u);
            ps.brdfPdf = ps.lightPdf = ps.cosL = ps.shLightID = 0.0f;
            ps.brdf = f4s(0.0f);
            ps.nrm = ps.shDir = f3(0.0f, 0.0f, 0.0f);
            ps.shObj = 0;
            ps.ev = 0u;
            if (cls == PC_SHADOW) {
                ps.shObj = __float_as_int(q6.x);
                const float4 next = ps.rr;
                r = shade_shadow_made<false>(ps, __float_as_int(q6.y), q5, next, J.pc.pathLength);
            } else if (ends == PE_HIT) {
                Hit h;
                h.hitdist = q5.x;
                h.normal = f3(q5.y, q5.z, q5.w);
                h.materialID = q6.x;
                h.lightID = q6.y;
                r = shade_primary<false>(ps, S, h, 0, J.pc.pathLength);
            }
        }
        if (cls == PC_END) {
            if (live && ends != PE_START) {
                const WfJob& J = A.jobs[job];
                const float3 col = sample_color(ps, ONE ? *S1 : *J.scene, J.cie);
                if (pt_check(A, local - J.local_base, J.count, PT_CHECK_SAMPLE))
                    J.colors[local] = make_float4(col.x, col.y, col.z, 0.0f);
                coloured = true;
            }
            count_finished(A.jobs, job, coloured);
            // New samples for these slots, from the warp's chunk.
            bool started = false;
            unsigned need = __ballot_sync(0xffffffffu, live);
            while (need && !exhausted) {
                if (cleft == 0) {
                    unsigned long long b = 0;
                    if (lane == 0)
                        b = POOL ? (unsigned long long)atomicAdd(&C.march_cursor, chunk)
                                 : atomicAdd(reinterpret_cast<unsigned long long*>(&C.next_sample), chunk);
                    b = __shfl_sync(0xffffffffu, b, 0);
                    if (b >= end) {
                        exhausted = true;
                        break;
                    }
                    cbase = b;
                    cleft = (end - b < chunk) ? (uint32_t)(end - b) : chunk;
                    if constexpr (POOL) continue;
                    // The pass of the chunk's first sample, looked up once for the warp.
                    uint32_t cj = 0;
                    if (lane == 0) cj = find_job(A.jobs, A.job_cap, job_lo, job_hi, b);
                    cjob = __shfl_sync(0xffffffffu, cj, 0);
                    const WfJob& CJ = A.jobs[cjob];
                    cjob_end = CJ.first + (uint64_t)CJ.count;
                }
                const uint32_t take = min((uint32_t)__popc(need), cleft);
                const uint32_t rank = (uint32_t)__popc(need & lt);
                if (((need >> lane) & 1u) && rank < take) {
                    const uint64_t s = cbase + rank;
                    started = true;
                    if constexpr (POOL) {
                        const uint32_t i = (uint32_t)s;
                        const uint32_t e = i < nm        ? A.q_march[cur][i]
                                           : i < nm + np ? A.q_shade[cur][i - nm]
                                                         : A.q_shadow[cur][i - nm - np];
                        next = load_staged(A, pool, e, i < nm, i >= nm + np, ps, contrib, q, local, job, r);
                        restored = next >= 0;
                    } else {
                        job = (s < cjob_end) ? cjob : find_job(A.jobs, A.job_cap, job_lo, job_hi, s);
                        local = A.jobs[job].local_base + (uint32_t)(s - A.jobs[job].first);
                    }
                }
                cbase += take;
                cleft -= take;
                need = __ballot_sync(0xffffffffu, live && !started);
            }
            live = started;
            if constexpr (POOL) {
                live = restored;
                if (live) jobs[slot] = job;
            } else if (live) {
                const WfJob& J = A.jobs[job];
                const pt_push& pc = J.pc;
                const int W = pc.resolution[0], H = pc.resolution[1];
                const uint32_t npix = (uint32_t)W * (uint32_t)H;
                const uint32_t k = local / npix, pix = local % npix;
                const uint32_t xx = pix % (uint32_t)W, yy = (uint32_t)H - pix / (uint32_t)W;
                const float uvx = (2.0f * (float)xx - (float)W) / (float)H;
                const float uvy = (2.0f * (float)yy - (float)H) / (float)H;
                const CamInfo cam = J.cam;
                start_sample(ps, ONE ? *S1 : *J.scene, pc, cam, xx, yy, uvx, uvy, (int)k);
                jobs[slot] = job;
                q[2] = ps.l;
                r = STEP_CONTINUE;
            }
        }
        // The ray each path goes on with, and the class of its next step.
        if (POOL && live && restored && next < PC_COUNT) {
            // a staged hit or shadow result: its state is in place
        } else if (live) {
            q[3] = ps.radiance;
            const uint32_t flags = bounce_word(ps);
            if (r == STEP_TERMINATED) {
                next = PC_END;
                next_end = PE_COLOUR;
                q[6] = make_float4(0.0f, 0.0f, __uint_as_float(local), __uint_as_float(flags));
            } else {
                const KScene& S = ONE ? *S1 : *A.jobs[job].scene;
                const bool shadow = r == STEP_SHADOW;
                q[0] = make_float4(ps.org.x, ps.org.y, ps.org.z, ps.mis);
                q[1] = make_float4(ps.dir.x, ps.dir.y, ps.dir.z, __uint_as_float(ps.seed));
                // a shadow ray's NEE term and the next throughput, made now (shade_shadow_made)
                q[4] = (shadow && !(POOL && restored)) ? bounce_throughput(ps) : ps.rr;
                if (shadow) q[5] = (POOL && restored) ? contrib : shadow_contribution(ps, S);
                Hit h;
                h.hitdist = PT_MAXDIST;
                h.normal = f3(0.0f, 0.0f, 0.0f);
                h.materialID = 0.0f;
                h.lightID = -1.0f;
                int objectID = -1;
                OriginSignT<float> sign{0.0f, 0u};
                intersect_all<FEAT>(S, ONE ? sh.spheres : S.objects, ps.org, shadow ? ps.shDir : ps.dir, h, objectID,
                                    shadow, ps.shObj, sign);
                next = path_class(S, h, shadow);
                if (!shadow) q[5] = make_float4(h.hitdist, h.normal.x, h.normal.y, h.normal.z);
                q[6] = make_float4(shadow ? __int_as_float(ps.shObj) : h.materialID,
                                   shadow ? __int_as_float(objectID) : h.lightID, __uint_as_float(local),
                                   __uint_as_float(flags));
            }
        }
#pragma unroll
        for (int c = 0; c < PC_COUNT; c++) {
            const unsigned m = __ballot_sync(0xffffffffu, next == c);
            const uint32_t at = (uint32_t)(count[c] + __popc(m & lt));
            if (next == c && pt_check(A, at, kPersistSlots, PT_CHECK_WARP_LIST))
                sh.list[warp][c][at] = (uint16_t)(slot | (uint32_t)(next_end << 8));
            count[c] += __popc(m);
        }
        __syncwarp();
    }
}

// Blocks that fit on an SM: five of the smaller variants, four of those with
// lenses and cyclides, which spill 148 bytes at five.  ms at five and four,
// 1920x1080x8: feature mix without SDFs 9.69, 8.51, its lenses alone 4.82, 4.63,
// twelve cyclides 10.5, 9.8; 800x600x1 0.43, 0.38, 0.24, 0.21, 0.68, 0.61.
template <int FEAT>
constexpr int kPersistBlocks = (FEAT & PT_FEAT_LENS) || (FEAT & PT_FEAT_SDF) ? 4 : 5;

template <int FEAT>
__global__ void __launch_bounds__(kPersistThreads, kPersistBlocks<FEAT>) wf_persist(const __grid_constant__ WfArgs A) {
    persist_paths<FEAT, false, false>(A, nullptr);
}

template <int FEAT>
__global__ void __launch_bounds__(kPersistThreads, kPersistBlocks<FEAT>)
    wf_persist_one(const __grid_constant__ WfArgs A, const __grid_constant__ KScene S1) {
    persist_paths<FEAT, true, false>(A, &S1);
}

#if !defined(PT_DEBUG_CHECKS)
// The last paths of a staged engine, run to their ends here.  Staged, every
// ray of a path waits for the slowest march of each iteration (64 steps, 25 us
// of launches): with few paths left an iteration costs the same 60 to 100 us
// however few, about 5 ms from the last new sample to the last colour on the
// shipped scenes.  Here a path's steps follow one another.
__global__ void __launch_bounds__(kPersistThreads, 4) wf_finish(const __grid_constant__ WfArgs A) {
    persist_paths<PT_FEAT_ALL, false, true>(A, nullptr);
}

// The pool is empty again: no queue holds a slot, the free list holds all.
__global__ void wf_finish_done(const __grid_constant__ WfArgs A) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < A.pool_size) A.q_free[i] = i;
    if (i == 0) {
        WfCounters& C = *A.counters;
        C.n_march[C.cur] = C.n_shade[C.cur] = C.n_shadow[C.cur] = 0;
        C.n_free = A.pool_size;
        C.live = 0;
        C.march_cursor = 0;
        C.iterations += 1;
    }
}
#endif

// Blocks of a persistent kernel that fit on one SM at once, cached.
template <int FEAT, bool ONE>
int persist_blocks() {
    static int cache = 0;
    if (cache) return cache;
    int n = 0;
    const void* k = ONE ? reinterpret_cast<const void*>(wf_persist_one<FEAT>)
                        : reinterpret_cast<const void*>(wf_persist<FEAT>);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PersistShared)) != cudaSuccess)
        return 1;  // the launch reports it
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, kPersistThreads, sizeof(PersistShared)) != cudaSuccess ||
        n < 1)
        n = 1;
    cache = n;
    return n;
}

template <int FEAT>
void launch_persist(const WfArgs* a, int sms, const KScene* one_scene, cudaStream_t stream) {
    if (one_scene) {
        const int blocks = persist_blocks<FEAT, true>();
        wf_persist_one<FEAT><<<sms * blocks, kPersistThreads, sizeof(PersistShared), stream>>>(*a, *one_scene);
    } else {
        const int blocks = persist_blocks<FEAT, false>();
        wf_persist<FEAT><<<sms * blocks, kPersistThreads, sizeof(PersistShared), stream>>>(*a);
    }
}

}  // namespace

cudaError_t PTK_WF(ptk_persist_launch)(const WfArgs* a, int variant, int sms, uint64_t budget,
                                       const KScene* one_scene, cudaStream_t stream) {
    wf_persist_setup<<<1, 1, 0, stream>>>(*a, budget);
    switch (variant) {
        case 0: launch_persist<0>(a, sms, one_scene, stream); break;
        case PT_FEAT_BOX: launch_persist<PT_FEAT_BOX>(a, sms, one_scene, stream); break;
        case PT_FEAT_ANALYTIC: launch_persist<PT_FEAT_ANALYTIC>(a, sms, one_scene, stream); break;
        default: launch_persist<PT_FEAT_ALL>(a, sms, one_scene, stream); break;
    }
    return cudaGetLastError();
}

int PTK_WF(ptk_persist_blocks_per_sm)(int variant) {
    switch (variant & 15) {
        case 0: return persist_blocks<0, false>();
        case PT_FEAT_BOX: return persist_blocks<PT_FEAT_BOX, false>();
        case PT_FEAT_ANALYTIC: return persist_blocks<PT_FEAT_ANALYTIC, false>();
        default: return persist_blocks<PT_FEAT_ALL, false>();
    }
}

#if !defined(PT_DEBUG_CHECKS)
cudaError_t ptk_wavefront_finish(const WfArgs* a, int sms, cudaStream_t stream) {
    static int blocks = 0;
    if (!blocks) {
        const cudaError_t e = cudaFuncSetAttribute(reinterpret_cast<const void*>(wf_finish),
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PersistShared));
        if (e != cudaSuccess) return e;
        int n = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, wf_finish, kPersistThreads, sizeof(PersistShared)) !=
                cudaSuccess ||
            n < 1)
            n = 1;
        blocks = n;
    }
    wf_finish<<<sms * blocks, kPersistThreads, sizeof(PersistShared), stream>>>(*a);
    wf_finish_done<<<(a->pool_size + 255) / 256, 256, 0, stream>>>(*a);
    return cudaGetLastError();
}
#endif
