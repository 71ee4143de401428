// pt_export.cuh — SaveRender's per-pixel chain (src/pathtracer.cpp:3491-3518):
// Bradford E->D65 (:971-978), XYZ->linear sRGB (:980-987), max(0), the
// tonemap (Reinhard :989-997, ACES fit :999-1021, DEUCES :1023-1033), sRGB
// companding (:1061-1071) and byte truncation.  Shared by the host export
// (libpt_host) and the device kernel (libpt_cuda), with pt_mathf's exp and
// pow on both, so the two give the same bytes.
#pragma once

#include <stdint.h>

#include "../../include/pt_mathf.h"

#if defined(__CUDACC__)
#define PTX_FN static __device__ __forceinline__
#else
#define PTX_FN static inline
#endif

// glm: vec3 * mat3 (column-major) = dot with each column.
PTX_FN void ptx_row_times(float& x, float& y, float& z, const float* m) {
    const float a = x * m[0] + y * m[1] + z * m[2];
    const float b = x * m[3] + y * m[4] + z * m[5];
    const float c = x * m[6] + y * m[7] + z * m[8];
    x = a;
    y = b;
    z = c;
}

// exp(t) by ptm_expf's operations, for t in [-80, 0], where the scaling by 2^k
// is one multiplication.
PTX_FN float ptx_exp_mid(float t) {
    const float kb = t * PTM_LOG2E + PTM_RINT_MAGIC;
    const float k = kb - PTM_RINT_MAGIC;
    float r = PTM_FMA(-k, PTM_LN2_1, t);
    r = PTM_FMA(-k, PTM_LN2_2, r);
    const float p =
        PTM_FMA(PTM_FMA(PTM_FMA(PTM_FMA(PTM_FMA(PTM_E5, r, PTM_E4), r, PTM_E3), r, PTM_E2), r, PTM_E1), r, PTM_E0);
    const float em1 = PTM_FMA(r * r, p, r);
    return (1.0f + em1) * ptm_from_bits((ptm_bits(kb) - PTM_RINT_MAGIC_BITS + 127u) << 23);
}

// x^(1/2.4) by ptm_powf's operations, for x in [0.003, 1] (or NaN): what
// follows from the range is left out, its checks for other arguments first.
PTX_FN float ptx_pow24(float x) {
    const float y = 1.0f / 2.4f;
    const uint32_t u = ptm_bits(x);
    int e = (int)(u >> 23) - 127;
    float m = ptm_from_bits((u & 0x007fffffu) | 0x3f800000u);
    if (m > 1.414213538f) {
        m *= 0.5f;
        e += 1;
    }
    const float l1p = ptm_log1p_reduced(m - 1.0f);
    const float ef = ptm_from_bits(PTM_RINT_MAGIC_BITS + (uint32_t)e) - PTM_RINT_MAGIC;
    const float L = PTM_FMA(ef, PTM_LN2_1, PTM_FMA(ef, PTM_LN2_2, l1p));
    const float p = y * L;
    const float perr = PTM_FMA(y, L, -p);
    const float ep = ptx_exp_mid(p);
    return (x == x) ? PTM_FMA(ep, perr, ep) : x;
}

PTX_FN float ptx_tonemap(float x, int tonemap) {
    if (tonemap == 1) x = x / (1.0f + x);
    if (tonemap == 2) {
        const float a = 2.51f, b = 0.03f, c = 2.43f, d = 0.59f, e = 0.14f;
        x = x * (a * x + b) / (x * (c * x + d) + e);
    }
    if (tonemap == 3) {
        // exp(-0.25 / x) for x >= +0 or NaN: below e^-80 the byte is 0 whatever
        // the value; -0 (max(-0, 0) keeps it) gives e^+inf
        const float t = -0.25f / x;
        x = (t < -80.0f) ? 0.0f : ((t <= 0.0f) ? ptx_exp_mid(t) : ((t > 0.0f) ? PTM_INF : t));
    }
    return x;
}

PTX_FN float ptx_srgb(float x) {
    x = (x < 0.0f) ? 0.0f : ((1.0f < x) ? 1.0f : x);
    if (x <= 0.0031308f) return 12.92f * x;
    return 1.055f * ptx_pow24(x) - 0.055f;
}

// The integer part of x * 255, exactly, for x in [0, 1] (NaN: 0).  On the GPU
// one fused operation: x * 255 + 2^23 rounded down holds it in the low
// mantissa bits.  The double product it stands for is two conversions and a
// multiplication at GB300's FP64 rate (8 of the 2560x1440 export kernel's 82
// us).
PTX_FN uint8_t ptx_byte(float x) {
#if defined(__CUDA_ARCH__)
    return (x == x) ? (uint8_t)__float_as_uint(__fmaf_rd(x, 255.0f, 8388608.0f)) : (uint8_t)0;
#else
    return (uint8_t)(int)((double)x * 255.0);
#endif
}

// One pixel: XYZ in, three bytes out.
PTX_FN void ptx_pixel(float x, float y, float z, int tonemap, uint8_t* out) {
    // IlluminantEToD65 and XYZToRGB, column-major as glm holds them.
    const float kEToD65[9] = {0.9531874f, -0.0265906f, 0.0238731f, -0.0382467f, 1.0288406f,
                              0.0094060f, 0.0026068f,  -0.0030332f, 1.0892565f};
    const float kXYZToRGB[9] = {3.2404542f, -1.5371385f, -0.4985314f, -0.9692660f, 1.8760108f,
                                0.0415560f, 0.0556434f,  -0.2040259f, 1.0572252f};
    ptx_row_times(x, y, z, kEToD65);
    ptx_row_times(x, y, z, kXYZToRGB);
    x = (x < 0.0f) ? 0.0f : x;  // glm::max(rgb, 0)
    y = (y < 0.0f) ? 0.0f : y;
    z = (z < 0.0f) ? 0.0f : z;
    out[0] = ptx_byte(ptx_srgb(ptx_tonemap(x, tonemap)));
    out[1] = ptx_byte(ptx_srgb(ptx_tonemap(y, tonemap)));
    out[2] = ptx_byte(ptx_srgb(ptx_tonemap(z, tonemap)));
}
