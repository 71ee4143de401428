// pt_fp64.cu — the FP64 reference renderer.  The path arithmetic is the same
// templates as the FP32 kernels (pt_path.cuh, pt_geometry.cuh) with R =
// double: every intermediate value carries 53 bits, transcendentals are
// CUDA's double-precision functions, the RNG draws the same 32-bit stream
// (converted exactly, so a draw never rounds up to 1.0), and the scene's
// values are the same floats widened.  Images it renders are the references
// the FP32 method's error is measured against.
//
// Two kernels, the same bits: fp64_paths sorts a warp's paths by the step they
// need (every scene of built-in SDFs), and the plain megakernel's per-pixel
// loop instantiated in double (pt_megakernel_body.cuh) renders traces, passes
// without bounces and dispatches without scratch; the run-time compiled
// module instantiates the latter for scene GLSL.
#include <cuda_runtime.h>

#include "pt_megakernel_body.cuh"
#include "pt_share.h"

namespace {

// GB300 runs double precision at 2 lanes a cycle and SM, so a kernel of it is
// bound by the FP64 instructions its warps issue, full or not.  A path per
// lane ran every kind of step for the few lanes that needed it.  Here, as in
// pt_persist.cu, a warp keeps kFp64Slots paths in shared memory and a list per
// class of their next step, takes up to 32 of the longest list at a time and
// intersects the rays they go on with together.  A sample's colour goes to
// scratch; fp64_sum adds a pixel's in sample order, as the megakernel does.
// The megakernel also left SMs empty: 128x128 pixels are 128 blocks of 152
// SMs, 64x64 32.  ms of a call by itself, an image's first samples, megakernel
// and this: full Cornell box 128x128x4 5.08, 2.83, 64x64x1 1.23, 1.19,
// 512x512x16 221, 109; menger + terrain 128x128x4 86.6, 27.6; shipped mandelbulb
// 128x128x4 68.5, 36.8, 256x256x16 606, 196.  (Another
// frame's samples of the first, perf/cases.py's: 4.17, 2.26.)
constexpr int kFp64Slots = 64;
constexpr int kFp64Threads = 128, kFp64Warps = kFp64Threads / 32;
constexpr int kFp64Refill = 16;     // ended paths gathered before new samples start together
constexpr uint32_t kFp64Chunk = 32;  // samples a warp claims at once after its first
// A path's state, 15 x 16 B a slot (an odd count, so that slots spread over the banks):
//   0, 1 org.xyz, mis    2, 3 dir.xyz, seed and sample    4, 5 wavelengths    6, 7 radiance
//   8, 9 throughput (shadow ray in flight: the next bounce's)
//   10, 11 hitdist, normal.xyz (shadow ray: its NEE term)
//   12 materialID, lightID (shadow ray: light object, object hit)    13 medium, bounce
constexpr int kFp64Quads = 15;
enum Fp64Class { DC_SHADOW = 0, DC_DIFFUSE, DC_SPECULAR, DC_END, DC_COUNT };
enum Fp64End { DE_HIT = 0, DE_COLOUR = 1, DE_START = 2 };  // shade an emitter or miss; write the colour; start
struct Fp64Shared {
    double2 state[kFp64Warps][kFp64Slots * kFp64Quads];
    uint16_t list[kFp64Warps][DC_COUNT][kFp64Slots];  // slot | Fp64End << 8
    CamInfoT<double> cam;
    float spheres[6 * PT_MAX_SCENE_SPHERES];
};
// Samples of a launch at most (whole pixels), which bounds the scratch (48 MB);
// the last paths of a launch cost a few percent of so many.
constexpr uint64_t kFp64Span = 1ull << 21;
// Samples from which two blocks share an SM.  ms with one, two: Cornell box
// 128x128x4 2.74, 3.29; 128x128x8 4.68, 4.76; 256x256x4 8.14, 7.98; 128x128x64
// 22.2, 20.6; menger + terrain 128x128x4 31.6, 40.2.
constexpr uint32_t kFp64Wide = 1u << 18;
// The samples of one launch: all of pixels [first, first + count), sample
// index k * count + pixel.  Every warp begins with `slots` of them.
struct Fp64Span {
    uint32_t first, count, total;
    int slots;
    double* colors;     // 3 per sample
    uint32_t* cursor;   // samples claimed past the warps' first ones
};

template <int FEAT>
__global__ void __launch_bounds__(kFp64Threads) fp64_paths(const __grid_constant__ KParams P, const Fp64Span span) {
    extern __shared__ __align__(16) unsigned char fp64_smem[];
    Fp64Shared& sh = *reinterpret_cast<Fp64Shared*>(fp64_smem);
    const KScene& S = P.s;
    const pt_push& pc = P.pc;
    const int lane = (int)(threadIdx.x & 31), warp = (int)(threadIdx.x >> 5);
    const unsigned lt = (1u << lane) - 1u;
    if (threadIdx.x == 0) sh.cam = make_camera<double>(pc);
    for (int i = threadIdx.x; i < 6 * S.meta.n[0]; i += kFp64Threads) sh.spheres[i] = S.objects[i];
    __syncthreads();
    const int W = pc.resolution[0], H = pc.resolution[1], depth = pc.pathLength;
    double2* const st = sh.state[warp];
    const int slots = span.slots;
    // the warps of a block are a grid apart, so that few samples spread over the SMs
    const uint32_t warps = gridDim.x * kFp64Warps, me = (uint32_t)warp * gridDim.x + blockIdx.x;
    uint64_t cbase = (uint64_t)me * (uint32_t)slots;  // warp-uniform: unassigned samples of the warp's claim
    uint32_t cleft = cbase < span.total ? min((uint32_t)slots, (uint32_t)(span.total - cbase)) : 0u;
    const uint64_t rest = (uint64_t)warps * (uint32_t)slots;
    bool exhausted = cleft == 0;
    int count[DC_COUNT] = {0, 0, 0, 0};  // warp-uniform: the lists' lengths
    for (int i = lane; i < slots; i += 32) sh.list[warp][DC_END][i] = (uint16_t)(i | (DE_START << 8));
    count[DC_END] = slots;
    __syncwarp();
    for (;;) {
        int cls = DC_END, most = (count[DC_END] >= kFp64Refill) ? count[DC_END] : 0;
#pragma unroll
        for (int c = 0; c < DC_END; c++)
            if (count[c] > most) {
                most = count[c];
                cls = c;
            }
        if (most == 0) most = count[DC_END];
        if (most == 0) break;
        const int n = min(most, 32), from = most - n;
#pragma unroll
        for (int c = 0; c < DC_COUNT; c++)
            if (c == cls) count[c] -= n;
        bool live = lane < n;
        uint32_t slot = 0;
        int ends = DE_HIT;
        if (live) {
            const uint32_t e = sh.list[warp][cls][from + lane];
            slot = e & 0xffu;
            ends = (int)(e >> 8);
        }
        __syncwarp();
        double2* const q = st + slot * kFp64Quads;
        uint32_t local = 0;
        PathStateT<double> ps;
        StepResult r = STEP_TERMINATED;
        int next = -1, next_end = DE_HIT;
        if (live && ends != DE_START) {
            const double2 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q10 = q[10], q11 = q[11], q12 = q[12];
            const double2 a = q[4], b = q[5], c = q[6], d = q[7], e = q[8], f = q[9];
            ps.org = v3<double>(q0.x, q0.y, q1.x);
            ps.mis = q1.y;
            ps.dir = v3<double>(q2.x, q2.y, q3.x);
            ps.seed = (uint32_t)__double2hiint(q3.y);
            local = (uint32_t)__double2loint(q3.y);
            ps.l = v4<double>(a.x, a.y, b.x, b.y);
            ps.radiance = v4<double>(c.x, c.y, d.x, d.y);
            ps.rr = v4<double>(e.x, e.y, f.x, f.y);
            const double m = q[13].x;
            ps.medium = __double2hiint(m);
            ps.bounce = __double2loint(m);
            ps.brdfPdf = ps.lightPdf = ps.cosL = ps.shLightID = 0.0;
            ps.brdf = v4s<double>(0.0);
            ps.nrm = ps.shDir = v3<double>(0.0, 0.0, 0.0);
            ps.shObj = 0;
            ps.ev = 0u;
            if (cls == DC_SHADOW) {
                ps.shObj = __double2loint(q12.x);
                const V4<double> after = ps.rr;
                r = shade_shadow_made<false>(ps, __double2loint(q12.y), v4<double>(q10.x, q10.y, q11.x, q11.y), after,
                                             depth);
            } else if (ends == DE_HIT) {
                HitT<double> h;
                h.hitdist = q10.x;
                h.normal = v3<double>(q10.y, q11.x, q11.y);
                h.materialID = q12.x;
                h.lightID = q12.y;
                r = shade_primary<false, FEAT>(ps, S, h, 0, depth);
            }
        }
        if (cls == DC_END) {
            if (live && ends != DE_START) {
                const V3<double> col = sample_color(ps, S, P.cie);
                double* const out = span.colors + 3 * (size_t)local;
                out[0] = col.x;
                out[1] = col.y;
                out[2] = col.z;
            }
            bool started = false;
            unsigned need = __ballot_sync(0xffffffffu, live);
            while (need && !exhausted) {
                if (cleft == 0) {
                    uint32_t b = 0;
                    if (lane == 0) b = atomicAdd(span.cursor, kFp64Chunk);
                    cbase = rest + __shfl_sync(0xffffffffu, b, 0);
                    if (cbase >= span.total) {
                        exhausted = true;
                        break;
                    }
                    cleft = (uint32_t)min((uint64_t)kFp64Chunk, span.total - cbase);
                }
                const uint32_t take = min((uint32_t)__popc(need), cleft);
                const uint32_t rank = (uint32_t)__popc(need & lt);
                if (((need >> lane) & 1u) && rank < take) {
                    local = (uint32_t)(cbase + rank);
                    started = true;
                }
                cbase += take;
                cleft -= take;
                need = __ballot_sync(0xffffffffu, live && !started);
            }
            live = started;
            if (live) {
                const uint32_t k = local / span.count, pix = span.first + local % span.count;
                const uint32_t xx = pix % (uint32_t)W, yy = (uint32_t)H - pix / (uint32_t)W;
                const double uvx = (2.0 * (double)xx - (double)W) / (double)H;
                const double uvy = (2.0 * (double)yy - (double)H) / (double)H;
                start_sample(ps, S, pc, sh.cam, xx, yy, uvx, uvy, (int)k);
                q[4] = double2{ps.l.x, ps.l.y};
                q[5] = double2{ps.l.z, ps.l.w};
                r = STEP_CONTINUE;
            }
        }
        // The ray each path goes on with, and the class of its next step.
        if (live) {
            q[6] = double2{ps.radiance.x, ps.radiance.y};
            q[7] = double2{ps.radiance.z, ps.radiance.w};
            q[3] = double2{ps.dir.z, __hiloint2double((int)ps.seed, (int)local)};
            if (r == STEP_TERMINATED) {
                next = DC_END;
                next_end = DE_COLOUR;
            } else {
                const bool shadow = r == STEP_SHADOW;
                q[0] = double2{ps.org.x, ps.org.y};
                q[1] = double2{ps.org.z, ps.mis};
                q[2] = double2{ps.dir.x, ps.dir.y};
                q[13].x = __hiloint2double(ps.medium, ps.bounce);
                const V4<double> rr = shadow ? bounce_throughput(ps) : ps.rr;
                q[8] = double2{rr.x, rr.y};
                q[9] = double2{rr.z, rr.w};
                if (shadow) {
                    const V4<double> c = shadow_contribution(ps, S);
                    q[10] = double2{c.x, c.y};
                    q[11] = double2{c.z, c.w};
                }
                HitT<double> h;
                h.hitdist = (double)PT_MAXDIST;
                h.normal = v3<double>(0.0, 0.0, 0.0);
                h.materialID = 0.0;
                h.lightID = -1.0;
                int objectID = -1;
                OriginSignT<double> sign{0.0, 0u};
                intersect_all<FEAT>(S, sh.spheres, ps.org, shadow ? ps.shDir : ps.dir, h, objectID, shadow, ps.shObj,
                                    sign);
                if (shadow) {
                    next = DC_SHADOW;
                    q[12] = double2{__hiloint2double(0, ps.shObj), __hiloint2double(0, objectID)};
                } else {
                    q[10] = double2{h.hitdist, h.normal.x};
                    q[11] = double2{h.normal.y, h.normal.z};
                    q[12] = double2{h.materialID, h.lightID};
                    const pt_material_ext* xm = ext_material(S, h.materialID);
                    next = (!(h.hitdist < (double)PT_MAXDIST) || light_mix(S, h.lightID).y > 0.0) ? DC_END
                           : (xm && xm->type >= PT_BSDF_MIRROR)                                  ? DC_SPECULAR
                                                                                                 : DC_DIFFUSE;
                }
            }
        }
#pragma unroll
        for (int c = 0; c < DC_COUNT; c++) {
            const unsigned m = __ballot_sync(0xffffffffu, next == c);
            if (next == c) sh.list[warp][c][count[c] + __popc(m & lt)] = (uint16_t)(slot | (uint32_t)(next_end << 8));
            count[c] += __popc(m);
        }
        __syncwarp();
    }
}

// Adds the span's pixels to their sums, samples in order (the megakernel's
// per-pixel sum and Rendering's exposure, SC:1513-1517).
__global__ void fp64_sum(const pt_push pc, const Fp64Span span, double* __restrict__ sums) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= span.count) return;
    double3 sum = double3{0.0, 0.0, 0.0};
    for (int k = 0; k < pc.samplesPerFrame; k++) {
        const double* c = span.colors + 3 * ((size_t)k * span.count + p);
        sum = sum + double3{c[0], c[1], c[2]};
    }
    const double exposure = (double)pc.apertureSize * (double)pc.apertureSize * (double)pc.ISO;
    double* s4 = sums + 4 * ((size_t)span.first + p);
    s4[0] += sum.x * exposure;
    s4[1] += sum.y * exposure;
    s4[2] += sum.z * exposure;
    s4[3] += (double)pc.samplesPerFrame;
}

template <int FEAT>
cudaError_t launch_paths(const KParams* params, int sms, uint64_t pixels, unsigned char* scratch, cudaStream_t stream) {
    const uint32_t spf = (uint32_t)params->pc.samplesPerFrame;
    const uint64_t per = kFp64Span / spf;  // pixels of a launch; at least one (ptk_fp64_scratch)
    int dev = 0, per_sm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(fp64_paths<FEAT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(Fp64Shared));
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fp64_paths<FEAT>, kFp64Threads, sizeof(Fp64Shared));
    if (e != cudaSuccess) return e;
    per_sm = per_sm < 1 ? 1 : per_sm > 2 ? 2 : per_sm;
    for (uint64_t first = 0; first < pixels; first += per) {
        Fp64Span span;
        span.first = (uint32_t)first;
        span.count = (uint32_t)(pixels - first < per ? pixels - first : per);
        span.total = span.count * spf;
        span.cursor = reinterpret_cast<uint32_t*>(scratch);
        span.colors = reinterpret_cast<double*>(scratch + 256);
        // One block an SM until a launch is large enough for the second to
        // have full lists too; the samples shared by all warps, eight or more each.
        const int blocks = sms * (span.total < kFp64Wide ? 1 : per_sm);
        const uint32_t warps = (uint32_t)(blocks * kFp64Warps), share = (span.total + warps - 1) / warps;
        span.slots = warp_slots(share, 8, 1, kFp64Slots);
        e = cudaMemsetAsync(span.cursor, 0, sizeof(uint32_t), stream);
        if (e != cudaSuccess) return e;
        fp64_paths<FEAT><<<blocks, kFp64Threads, sizeof(Fp64Shared), stream>>>(*params, span);
        fp64_sum<<<(span.count + 127) / 128, 128, 0, stream>>>(params->pc, span, params->sums);
    }
    return cudaGetLastError();
}

}  // namespace

size_t ptk_fp64_scratch(const pt_push* pc) {
    if (pc->samplesPerFrame < 1 || (uint64_t)pc->samplesPerFrame > kFp64Span || pc->pathLength < 1) return 0;
    const uint64_t total =
        (uint64_t)pc->resolution[0] * (uint64_t)pc->resolution[1] * (uint64_t)pc->samplesPerFrame;
    return 256 + 24 * (size_t)(total < kFp64Span ? total : kFp64Span);
}

uint64_t ptk_fp64_kernels(const pt_push* pc, const void* scratch) {
    if (!scratch) return 1;
    const uint64_t per = kFp64Span / (uint64_t)pc->samplesPerFrame;
    return 2 * (((uint64_t)pc->resolution[0] * (uint64_t)pc->resolution[1] + per - 1) / per);
}

cudaError_t ptk_launch_fp64(const KParams* params, bool trace, void* scratch, int sms, cudaStream_t stream) {
    const int W = params->pc.resolution[0], H = params->pc.resolution[1];
    const uint64_t pixels = (uint64_t)W * (uint64_t)H;
    if (scratch && !trace && pixels < (1ull << 32)) {
        unsigned char* s = static_cast<unsigned char*>(scratch);
        return params->s.meta.n[5] > 0 ? launch_paths<PT_FEAT_ALL>(params, sms, pixels, s, stream)
                                       : launch_paths<PT_FEAT_ANALYTIC>(params, sms, pixels, s, stream);
    }
    const dim3 block(PT_MK_BLOCK_X, PT_MK_BLOCK_Y);
    const dim3 grid((W + PT_MK_BLOCK_X - 1) / PT_MK_BLOCK_X, (H + PT_MK_BLOCK_Y - 1) / PT_MK_BLOCK_Y);
    if (trace) {
        megakernel<true, PT_FEAT_ALL, double><<<grid, block, 0, stream>>>(*params);
    } else {
        megakernel<false, PT_FEAT_ALL, double><<<grid, block, 0, stream>>>(*params);
    }
    return cudaGetLastError();
}
