"""Exact shortcuts of the float path: forms that replace slower ones must give
the same bits, checked here on the CPU against the plain forms."""
import os
import re
import subprocess

import pytest

from conftest import ROOT

MATHF_C = r"""
#include "pt_mathf.h"
/* the functions with rintf and float-to-int conversions in place of the magic addition */
static float scale2(float y, int k) {
    if (k > 127) { y *= ptm_from_bits(0x7f000000u); k -= 127; if (k > 127) k = 127; }
    else if (k < -126) { y *= ptm_from_bits(0x00800000u); k += 126; if (k < -126) k = -126; }
    return y * ptm_from_bits((uint32_t)(k + 127) << 23);
}
static float epoly(float r) {
    const float p = PTM_FMA(PTM_FMA(PTM_FMA(PTM_FMA(PTM_FMA(PTM_E5, r, PTM_E4), r, PTM_E3), r, PTM_E2), r, PTM_E1), r, PTM_E0);
    return 1.0f + PTM_FMA(r * r, p, r);
}
static float exp_plain(float x) {
    if (x != x) return x;
    if (x > 88.72283936f) return PTM_INF;
    if (x < -103.9720840f) return 0.0f;
    const float k = rintf(x * PTM_LOG2E);
    float r = PTM_FMA(-k, PTM_LN2_1, x);
    r = PTM_FMA(-k, PTM_LN2_2, r);
    return scale2(epoly(r), (int)k);
}
static float exp2_plain(float x) {
    if (x != x) return x;
    if (x > 128.0f) return PTM_INF;
    if (x < -150.0f) return 0.0f;
    const float k = rintf(x), f = x - k;
    return scale2(epoly(PTM_FMA(f, PTM_LN2_1, f * PTM_LN2_2)), (int)k);
}
static float log_plain(float x) {
    if (x != x) return x;
    if (x < 0.0f) return PTM_NAN;
    if (x == 0.0f) return -PTM_INF;
    if (x == PTM_INF) return x;
    int e;
    const float m = ptm_frexp_sqrt2(x, &e), ef = (float)e;
    return PTM_FMA(ef, PTM_LN2_1, PTM_FMA(ef, PTM_LN2_2, ptm_log1p_reduced(m - 1.0f)));
}
static void sincos_plain(float x, float* s, float* c) {
    if (!(x - x == 0.0f)) { *s = *c = PTM_NAN; return; }
    const float k = rintf(x * PTM_2_OVER_PI);
    float r = PTM_FMA(-k, PTM_PIO2_1, x);
    r = PTM_FMA(-k, PTM_PIO2_2, r);
    r = PTM_FMA(-k, PTM_PIO2_3, r);
    const int q = (int)(k - 4.0f * floorf(k * 0.25f));
    const float z = r * r;
    const float sr = PTM_FMA(r * z, PTM_FMA(PTM_FMA(PTM_FMA(PTM_S3, z, PTM_S2), z, PTM_S1), z, PTM_S0), r);
    const float cr = PTM_FMA(z * z, PTM_FMA(PTM_FMA(PTM_FMA(PTM_C3, z, PTM_C2), z, PTM_C1), z, PTM_C0), PTM_FMA(-0.5f, z, 1.0f));
    *s = q == 0 ? sr : q == 1 ? cr : q == 2 ? -sr : -cr;
    *c = q == 0 ? cr : q == 1 ? -sr : q == 2 ? -cr : sr;
}
long forms_differ(uint32_t first, uint32_t step) {
    long bad = 0;
    uint64_t u;
    for (u = first; u < (1ull << 32); u += step) {
        const float x = ptm_from_bits((uint32_t)u);
        float s, c;
        sincos_plain(x, &s, &c);
        const ptm_sc v = ptm_sincos_inline(x);
        bad += ptm_bits(v.s) != ptm_bits(s) || ptm_bits(v.c) != ptm_bits(c);
        bad += ptm_bits(ptm_expf(x)) != ptm_bits(exp_plain(x));
        bad += ptm_bits(ptm_exp2f(x)) != ptm_bits(exp2_plain(x));
        bad += ptm_bits(ptm_logf(x)) != ptm_bits(log_plain(x));
    }
    return bad;
}
/* c * hi + c * lo against c / divisor for every significand, both signs, in two binades */
long quotients_differ(float divisor, float hi, float lo) {
    long bad = 0;
    uint32_t m;
    int e, sign;
    for (m = 0; m < (1u << 23); m++)
        for (e = 103; e <= 127; e += 24)
            for (sign = 0; sign < 2; sign++) {
                const float c = ptm_from_bits(((uint32_t)sign << 31) | ((uint32_t)e << 23) | m);
                bad += ptm_bits(PTM_FMA(c, hi, c * lo)) != ptm_bits(c / divisor);
            }
    return bad;
}
"""


@pytest.fixture(scope="module")
def forms(tmp_path_factory):
    import ctypes

    d = tmp_path_factory.mktemp("forms")
    src, out = d / "forms.c", d / "forms.so"
    src.write_text(MATHF_C)
    subprocess.run([os.environ.get("CC", "gcc"), "-O2", "-std=c11", "-ffp-contract=off", "-fPIC", "-shared",
                    "-I" + os.path.join(ROOT, "include"), "-o", str(out), str(src), "-lm"], check=True)
    lib = ctypes.CDLL(str(out))
    lib.forms_differ.restype = lib.quotients_differ.restype = ctypes.c_long
    lib.forms_differ.argtypes = [ctypes.c_uint32, ctypes.c_uint32]
    lib.quotients_differ.argtypes = [ctypes.c_float] * 3
    return lib


@pytest.mark.parametrize("first", [0, 1, 1234])
def test_mathf_without_conversions_is_the_plain_form(forms, first):
    """Every 4099th float (NaNs, infinities, subnormals and both zeros among them)."""
    assert forms.forms_differ(first, 4099) == 0


def test_menger_level_division_is_the_quotient(forms):
    """c / 3^N by its two-part reciprocal, with the constants of sdf_menger."""
    with open(os.path.join(ROOT, "pathtracer_gb300", "csrc", "kernel", "pt_geometry.cuh")) as f:
        text = f.read()
    hi, lo = ([float(x.strip().rstrip("f")) for x in re.search(name + r"\[5\] = \{([^}]*)\}", text).group(1).split(",")]
              for name in ("kInvHi", "kInvLo"))
    for n in range(5):
        assert forms.quotients_differ(3.0 ** (n + 1), hi[n], lo[n]) == 0
    assert forms.quotients_differ(9.0, hi[1], 0.0) != 0  # the low part is needed


CULL_C = r"""
#include <math.h>
#include <stdint.h>
#define EPS 1.52587890625e-05
/* the exact test's outcome with nothing hit yet (sphere_hit), in the kernel's order of operations */
static int hits(const float* o, const float* d, const float* s) {
    const float x = o[0] - s[0], y = o[1] - s[1], z = o[2] - s[2];
    const float b = 2.0f * (d[0] * x + d[1] * y + d[2] * z);
    const float c = (x * x + y * y + z * z) - s[3] * s[3];
    const float disc = b * b - 4.0f * c;
    if (disc < 0.0f) return 0;
    const float q = sqrtf(disc), t1 = (-b - q) * 0.5f, t2 = (-b + q) * 0.5f, t = t1 > 0.0f ? t1 : t2;
    if (t < 1e-4f) return 0;
    return t < 1e5f;
}
/* whether the first pass leaves the sphere out (intersect_spheres, pt_derive_cull) */
static int culled(const float* o, const float* d, const float* s, float pmax) {
    const double pp = (double)s[0] * s[0] + (double)s[1] * s[1] + (double)s[2] * s[2], rr = (double)s[3] * s[3];
    const float k = nextafterf((float)(pp - rr - EPS * (pp + rr)), -HUGE_VALF);
    const float oo = fmaf(o[0], o[0], fmaf(o[1], o[1], o[2] * o[2])), od = fmaf(o[0], d[0], fmaf(o[1], d[1], o[2] * d[2]));
    const float ook = oo * (float)(1.0 - EPS);
    const float leaving = 3.814697265625e-06f * (0.5f + 0.5f * oo + pmax);
    const float hb = fmaf(-d[0], s[0], fmaf(-d[1], s[1], fmaf(-d[2], s[2], od)));
    const float c = fmaf(-2.0f * o[0], s[0], fmaf(-2.0f * o[1], s[1], fmaf(-2.0f * o[2], s[2], ook + k)));
    return fmaf(hb, hb, -c) < 0.0f || (hb > leaving && c > 0.0f);
}
/* per ray: bit 0 the exact test hits, bit 1 the sphere is left out */
void outcome(const float* rays, const float* spheres, long n, uint8_t* out) {
    long i;
    for (i = 0; i < n; i++) {
        const float* s = spheres + 4 * i;
        const float pmax = nextafterf((float)sqrt((double)s[0] * s[0] + (double)s[1] * s[1] + (double)s[2] * s[2]), HUGE_VALF);
        out[i] = (uint8_t)(hits(rays + 6 * i, rays + 6 * i + 3, s) | (culled(rays + 6 * i, rays + 6 * i + 3, s, pmax) << 1));
    }
}
"""


@pytest.mark.parametrize("scale", [1e-3, 1.0, 300.0, 1e4, 1e9, 1e19])
@pytest.mark.parametrize("kind", ["any", "grazing", "surface", "inside"])
def test_culled_spheres_are_never_hit(tmp_path, scale, kind):
    """The sphere loop's first pass over rays of every kind, at scene sizes from
    a millimetre to where squares overflow: what it leaves out, the exact test
    refuses; rays aimed past a sphere are mostly left out."""
    import ctypes

    import numpy as np

    src, lib = tmp_path / "cull.c", tmp_path / "cull.so"
    src.write_text(CULL_C)
    subprocess.run([os.environ.get("CC", "gcc"), "-O2", "-std=c11", "-ffp-contract=off", "-fPIC", "-shared", "-o",
                    str(lib), str(src), "-lm"], check=True)
    rng = np.random.default_rng(11)
    n = 400000
    c = rng.normal(size=(n, 3)) * scale
    r = np.exp(rng.uniform(np.log(1e-3), np.log(2.0), n)) * scale
    u = rng.normal(size=(n, 3))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    w = np.cross(u, rng.normal(size=(n, 3)))
    w /= np.linalg.norm(w, axis=1, keepdims=True)
    if kind == "grazing":  # passing within 1e-7 .. 1e-2 radii of the surface
        off = np.exp(rng.uniform(np.log(1e-7), np.log(1e-2), n)) * rng.choice([-1, 1], n)
        o = c + w * (r * (1 + off))[:, None] - u * (rng.uniform(0.5, 20, n) * r)[:, None]
        d = u
    elif kind == "surface":  # leaving or entering from a point on the sphere, to rounding
        o = c + u * r[:, None]
        d = rng.normal(size=(n, 3))
    elif kind == "inside":
        o = c + u * (r * rng.uniform(0, 1, n))[:, None]
        d = rng.normal(size=(n, 3))
    else:
        o = rng.normal(size=(n, 3)) * scale * 3
        d = rng.normal(size=(n, 3))
    d = d / np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.ascontiguousarray(np.concatenate([o, d], axis=1), np.float32)
    spheres = np.ascontiguousarray(np.concatenate([c, r[:, None]], axis=1), np.float32)
    out = np.zeros(n, np.uint8)
    fn = ctypes.CDLL(str(lib)).outcome
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_long, ctypes.c_void_p]
    fn(rays.ctypes.data, spheres.ctypes.data, n, out.ctypes.data)
    assert not (out == 3).any()
    if kind == "any" and scale <= 300.0:
        assert (out == 2).mean() > 0.5  # the pass does leave spheres out


BYTE_C = r"""
#include <fenv.h>
#include <math.h>
#include <stdint.h>
#include <string.h>
static float fb(uint32_t u) { float f; memcpy(&f, &u, 4); return f; }
static uint32_t bits(float f) { uint32_t u; memcpy(&u, &f, 4); return u; }
/* x * 255 + 2^23 rounded down against the truncated double product, at every step-th float of [0, 1] and at the 64
   floats on either side of each k / 255 */
long bytes_differ(uint32_t step) {
    long bad = 0;
    uint32_t u;
    int k, i;
    const uint32_t one = bits(1.0f);
    fesetround(FE_DOWNWARD);
    for (u = 0; u <= one; u += step) {
        volatile float x = fb(u), y = fmaf(x, 255.0f, 8388608.0f);
        bad += (uint8_t)bits(y) != (uint8_t)(int)((double)x * 255.0);
    }
    for (k = 0; k <= 255; k++) {
        const uint32_t c = bits((float)(k / 255.0));
        for (i = -64; i <= 64; i++) {
            if ((int64_t)c + i < 0 || c + i > one) continue;
            volatile float x = fb(c + i), y = fmaf(x, 255.0f, 8388608.0f);
            bad += (uint8_t)bits(y) != (uint8_t)(int)((double)x * 255.0);
        }
    }
    fesetround(FE_TONEAREST);
    return bad;
}
"""


def test_export_byte_is_the_truncated_product(tmp_path):
    import ctypes

    src, lib = tmp_path / "b.c", tmp_path / "b.so"
    src.write_text(BYTE_C)
    subprocess.run([os.environ.get("CC", "gcc"), "-O1", "-std=c11", "-ffp-contract=off", "-frounding-math", "-fPIC",
                    "-shared", "-o", str(lib), str(src), "-lm"], check=True)
    fn = ctypes.CDLL(str(lib)).bytes_differ
    fn.restype, fn.argtypes = ctypes.c_long, [ctypes.c_uint32]
    assert fn(257) == 0


EXPORT_CPP = r"""
#include "pt_export.cuh"
static float srgb(float x) {
    x = (x < 0.0f) ? 0.0f : ((1.0f < x) ? 1.0f : x);
    if (x <= 0.0031308f) return 12.92f * x;
    return 1.055f * ptm_powf(x, 1.0f / 2.4f) - 0.055f;
}
/* companded values (all floats) and tonemap 3's bytes (floats not below zero, as the chain's max leaves them) */
extern "C" long export_differs(uint32_t first, uint32_t step) {
    long bad = 0;
    for (uint64_t u = first; u < (1ull << 32); u += step) {
        const float x = ptm_from_bits((uint32_t)u), a = srgb(x), b = ptx_srgb(x);
        bad += ptm_bits(a) != ptm_bits(b) && !(a != a && b != b);
        if (!(x < 0.0f)) bad += ptx_byte(srgb(ptm_expf(-0.25f / x))) != ptx_byte(ptx_srgb(ptx_tonemap(x, 3)));
    }
    return bad;
}
"""


@pytest.mark.parametrize("first,step", [(0, 4099), (0x80000000, 0x7fffffff), (0x3b4d2e00, 1 << 30)])
def test_export_forms_are_the_plain_chain(tmp_path, first, step):
    """ptx_srgb and the exponential tonemap without their range checks: strided
    over all floats, -0 and the companding border among them."""
    import ctypes

    src, lib = tmp_path / "e.cpp", tmp_path / "e.so"
    src.write_text(EXPORT_CPP)
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared",
                    "-I" + os.path.join(ROOT, "pathtracer_gb300", "csrc"), "-o", str(lib), str(src)], check=True)
    fn = ctypes.CDLL(str(lib)).export_differs
    fn.restype, fn.argtypes = ctypes.c_long, [ctypes.c_uint32, ctypes.c_uint32]
    assert fn(first, step) == 0


INVERSE_C = r"""
#include "pt_mathf.h"
/* the forms with a branch per case: two polynomials, two divisions, a check per special argument of pow */
static float acos_plain(float x) {
    if (x != x) return x;
    const float ax = fabsf(x);
    if (ax > 1.0f) return PTM_NAN;
    if (ax <= 0.5f) return PTM_PIO2_1 - (ptm_asin_poly(x, x * x) - PTM_PIO2_2);
    const float z = (1.0f - ax) * 0.5f, as2 = 2.0f * ptm_asin_poly(sqrtf(z), z);
    return x > 0.0f ? as2 : PTM_PI_1 - (as2 - PTM_PI_2);
}
static float asin_plain(float x) {
    if (x != x) return x;
    const float ax = fabsf(x), z = (1.0f - ax) * 0.5f;
    if (ax > 1.0f) return PTM_NAN;
    const float r = ax <= 0.5f ? ptm_asin_poly(ax, ax * ax) : PTM_PIO2_1 - (2.0f * ptm_asin_poly(sqrtf(z), z) - PTM_PIO2_2);
    return (ptm_bits(x) >> 31) ? -r : r;
}
static float atan_plain(float x) {
    if (x != x) return x;
    const float a = fabsf(x);
    const float r = a > 1.0f ? PTM_PIO2_1 - (ptm_atan_poly(1.0f / a) - PTM_PIO2_2) : ptm_atan_poly(a);
    return (ptm_bits(x) >> 31) ? -r : r;
}
static float pow_plain(float x, float y) {  /* y finite, not 0 and not an integer of magnitude <= 32 */
    if (x == 1.0f) return 1.0f;
    if (x != x) return PTM_NAN;
    const float ax = fabsf(x), ay = fabsf(y);
    const int odd = floorf(ay) == ay && ay < 16777216.0f && (int)(ay - 2.0f * floorf(ay * 0.5f)) == 1;
    const int neg = x < 0.0f && odd;
    if (x < 0.0f && floorf(ay) != ay) return PTM_NAN;
    float r;
    if (ax == 0.0f || ax == PTM_INF) r = ((ax == 0.0f) == (y > 0.0f)) ? 0.0f : PTM_INF;
    else r = ptm_pow_exp_log(ax, y);
    return neg ? -r : r;
}
static int ne(float a, float b) { return ptm_bits(a) != ptm_bits(b) && !(a != a && b != b); }
long inverse_differ(uint32_t first, uint32_t step) {
    static const float ys[] = {1.0f / 2.4f, 8.23f, -2.5f, 0.3333333f, 33.0f, 100.5f, -41.0f, 1e7f};
    long bad = 0;
    uint64_t u;
    unsigned k;
    for (u = first; u < (1ull << 32); u += step) {
        const float x = ptm_from_bits((uint32_t)u), y = ptm_from_bits((uint32_t)u * 2654435761u + 977u);
        bad += ne(ptm_acosf(x), acos_plain(x)) + ne(ptm_asinf(x), asin_plain(x)) + ne(ptm_atanf(x), atan_plain(x));
        for (k = 0; k < sizeof ys / sizeof ys[0]; k++) bad += ne(ptm_powf(x, ys[k]), pow_plain(x, ys[k]));
        if (x == x && y == y && fabsf(x) < 1e38f && fabsf(y) < 1e38f && x != 0.0f) {  /* the general case of atan2 */
            const float ax = fabsf(y), ay = fabsf(x), t = ay > ax ? ax / ay : ay / ax, p = ptm_atan_poly(t);
            float r = ay > ax ? PTM_PIO2_1 - (p - PTM_PIO2_2) : p;
            if (ptm_bits(y) >> 31) r = PTM_PI_1 - (r - PTM_PI_2);
            bad += ne(ptm_atan2f(x, y), (ptm_bits(x) >> 31) ? -r : r);
        }
    }
    return bad;
}
"""


@pytest.mark.parametrize("first", [0, 7])
def test_inverse_functions_and_pow_are_the_plain_forms(tmp_path, first):
    import ctypes

    src, lib = tmp_path / "i.c", tmp_path / "i.so"
    src.write_text(INVERSE_C)
    subprocess.run([os.environ.get("CC", "gcc"), "-O2", "-std=c11", "-ffp-contract=off", "-fPIC", "-shared",
                    "-I" + os.path.join(ROOT, "include"), "-o", str(lib), str(src), "-lm"], check=True)
    fn = ctypes.CDLL(str(lib)).inverse_differ
    fn.restype, fn.argtypes = ctypes.c_long, [ctypes.c_uint32, ctypes.c_uint32]
    assert fn(first, 4099) == 0
