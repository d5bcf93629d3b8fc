// pt_device.cuh -- device-side data views and arithmetic for the offset-field
// synthesis kernels (sm_103a).
//
// Arithmetic contract.  All kernels are compiled with -fmad=false, so no
// multiply-add is fused unless written as fmaf(); the places that use fmaf()
// and the operation order of every sum are fixed, which makes the results
// reproducible on any IEEE FP32 machine.  Bilinear sampling uses exact FP32
// weights or the texture unit's arithmetic (PT_FILTER_TEXTURE: the texture
// unit itself in the tiled kernels, an exact emulation elsewhere),
// sin/cos/atan2/log/acos come from the polynomial routines below, and double
// precision is used exactly where the reference's C++ promotes to double.
#pragma once

#include <cstdint>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "painttween.h"
#include "pt_types.h"

namespace ptk {

// Programmatic dependent launch: the next kernel of the stream may take its
// place on the GPU while this one's last blocks run (launch_dependents), and
// waits before its first access to global memory until this one has ended and
// its writes are visible (wait).  What the kernels that begin with this write
// for one another (offset records, residual, canvas, change tracking, tile
// lists) they read with plain loads only: a read-only load (__ldg) needs data
// that nothing writes while the kernel lives, and these are written while the
// next kernel is already there.  All else is written before the first of a
// chain of them starts (pt_ctx::chained), so read-only loads serve for it.
__device__ __forceinline__ void pdl_start() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

constexpr float kAlphaThreshold = 0.99f;  // types.h:39
constexpr float kEpsilon = 0.000001f;     // types.h:38
constexpr float kBigResidual = (float)10e30;

// ---------------------------------------------------------------------------
// polynomial elementary functions
// ---------------------------------------------------------------------------

// k = rint(t*2/pi); r = t - k*pi/2 (two-term Cody-Waite, fused);
// Taylor series of sin to r^9 and cos to r^10 on |r| <= pi/4.
__device__ __forceinline__ void sincos_poly(float t, float* s, float* c) {
    const float two_over_pi = 0x1.45f306p-1f;
    const float pio2_hi = 0x1.921fb6p+0f;
    const float pio2_lo = -0x1.777a5cp-25f;
    float k = rintf(t * two_over_pi);
    float r = fmaf(-k, pio2_hi, t);
    r = fmaf(-k, pio2_lo, r);
    float r2 = r * r;
    float ps = fmaf(r2, (float)(1.0 / 362880.0), (float)(-1.0 / 5040.0));
    ps = fmaf(r2, ps, (float)(1.0 / 120.0));
    ps = fmaf(r2, ps, (float)(-1.0 / 6.0));
    ps = ps * r2;
    float sr = fmaf(r, ps, r);
    float pc = fmaf(r2, (float)(-1.0 / 3628800.0), (float)(1.0 / 40320.0));
    pc = fmaf(r2, pc, (float)(-1.0 / 720.0));
    pc = fmaf(r2, pc, (float)(1.0 / 24.0));
    pc = fmaf(r2, pc, -0.5f);
    float cr = fmaf(r2, pc, 1.0f);
    int q = ((int)k) & 3;  // cvt.rzi saturates, NaN -> 0
    if (q == 0) { *s = sr; *c = cr; }
    else if (q == 1) { *s = cr; *c = -sr; }
    else if (q == 2) { *s = -sr; *c = -cr; }
    else { *s = -cr; *c = sr; }
}

// atan on [0,1]: atan(u) = pi/4 + atan((u-1)/(u+1)) above tan(pi/8);
// Taylor series to v^19.
__device__ __forceinline__ float atan01_poly(float u) {
    float off = 0.0f;
    float v = u;
    if (u > 0x1.a8279ap-2f) {
        v = (u - 1.0f) / (u + 1.0f);
        off = 0x1.921fb6p-1f;
    }
    float v2 = v * v;
    float p = (float)(-1.0 / 19.0);
    p = fmaf(v2, p, (float)(1.0 / 17.0));
    p = fmaf(v2, p, (float)(-1.0 / 15.0));
    p = fmaf(v2, p, (float)(1.0 / 13.0));
    p = fmaf(v2, p, (float)(-1.0 / 11.0));
    p = fmaf(v2, p, (float)(1.0 / 9.0));
    p = fmaf(v2, p, (float)(-1.0 / 7.0));
    p = fmaf(v2, p, (float)(1.0 / 5.0));
    p = fmaf(v2, p, (float)(-1.0 / 3.0));
    p = p * v2;
    return off + fmaf(v, p, v);
}

__device__ __forceinline__ float atan2_poly(float y, float x) {
    const float pi = 0x1.921fb6p+1f;
    const float pio2 = 0x1.921fb6p+0f;
    float ax = fabsf(x), ay = fabsf(y);
    if (ax == 0.0f && ay == 0.0f) {
        float r = signbit(x) ? pi : 0.0f;
        return signbit(y) ? -r : r;
    }
    float mx = fmaxf(ax, ay), mn = fminf(ax, ay);
    float a = atan01_poly(mn / mx);
    if (ay > ax) a = pio2 - a;
    if (signbit(x)) a = pi - a;
    return signbit(y) ? -a : a;
}

// log(x) = e ln2 + 2 atanh((m-1)/(m+1)), m in [sqrt(1/2), sqrt(2)).
// double log, exp and pow for the Lab conversion (the oracle restates the
// same steps): log by frexp to m in [sqrt(1/2), sqrt(2)) and the atanh
// series to s^23, exp by k = rint(y/ln2) with a two-part ln2 and the Taylor
// series to r^22, pow(x, y) = exp(y log x) for x > 0
static __device__ __noinline__ double log_d(double x) {
    int e;
    double m = frexp(x, &e);
    if (m < 0.70710678118654752440) {
        m = m * 2.0;
        e -= 1;
    }
    const double s = (m - 1.0) / (m + 1.0);
    const double s2 = s * s;
    double p = 1.0 / 23.0;
    for (int k = 21; k >= 3; k -= 2) p = fma(s2, p, 1.0 / (double)k);
    p = p * s2;
    const double lm = 2.0 * fma(s, p, s);
    const double fe = (double)e;
    return fma(fe, 6.93147180369123816490e-01, fma(fe, 1.90821492927058770002e-10, lm));
}
static __device__ __noinline__ double exp_d(double y) {
    const double k = rint(y * 1.44269504088896338700);
    double r = fma(-k, 6.93147180369123816490e-01, y);
    r = fma(-k, 1.90821492927058770002e-10, r);
    double p = 1.0;
    for (int n = 22; n >= 1; n--) p = fma(r / (double)n, p, 1.0);
    return ldexp(p, (int)k);
}
__device__ __forceinline__ double pow_d(double x, double y) {
    if (!(x > 0.0)) return (x == 0.0) ? 0.0 : __longlong_as_double(0x7ff8000000000000LL);
    return exp_d(y * log_d(x));
}
// RGBtoLAB with Clinear and f_Lab (texSynth_util.h:175-192,220-246)
__device__ __forceinline__ float lab_clinear(float c) {
    const float a = 0.055f;
    if ((double)c > 0.04045) return (float)pow_d((double)(c + a) / (1.0 + (double)a), 2.4);
    return (float)((double)c / 12.92);
}
__device__ __forceinline__ float lab_f(float t) {
    const float lim = (float)pow_d((double)(float)(6.0 / 29.0), 3.0);
    if (t > lim) return (float)pow_d((double)t, (double)(float)(1.0 / 3.0));
    const float sq = (float)pow_d((double)(float)(29.0 / 6.0), 2.0);
    return (float)((1.0 / 3.0) * (double)sq * (double)t + (4.0 / 29.0));
}
static __device__ __noinline__ float4 rgb_to_lab(float4 c) {
    const float refX = 95.047f, refY = 100.0f, refZ = 108.883f;
    const float rl = 100.0f * lab_clinear(c.x), gl = 100.0f * lab_clinear(c.y), bl = 100.0f * lab_clinear(c.z);
    const float X = (float)(0.4124 * (double)rl + 0.3576 * (double)gl + 0.1805 * (double)bl);
    const float Y = (float)(0.2126 * (double)rl + 0.7152 * (double)gl + 0.0722 * (double)bl);
    const float Z = (float)(0.0193 * (double)rl + 0.1192 * (double)gl + 0.9505 * (double)bl);
    const float fy = lab_f(Y / refY);
    return make_float4((116.f * fy - 16.0f) / 100.f, (500.f * (lab_f(X / refX) - fy) + 100.0f) / 200.f,
                       (200.f * (fy - lab_f(Z / refZ)) + 100.0f) / 200.f, c.w);
}

__device__ __forceinline__ float log_poly(float x) {
    if (!(x > 0.0f)) return (x == 0.0f) ? -INFINITY : NAN;
    if (isinf(x)) return x;
    int e;
    float m = frexpf(x, &e);
    if (m < 0x1.6a09e6p-1f) { m = m * 2.0f; e -= 1; }
    float s = (m - 1.0f) / (m + 1.0f);
    float s2 = s * s;
    float p = (float)(1.0 / 11.0);
    p = fmaf(s2, p, (float)(1.0 / 9.0));
    p = fmaf(s2, p, (float)(1.0 / 7.0));
    p = fmaf(s2, p, (float)(1.0 / 5.0));
    p = fmaf(s2, p, (float)(1.0 / 3.0));
    p = p * s2;
    float lm = 2.0f * fmaf(s, p, s);
    float fe = (float)e;
    return fmaf(fe, 0x1.62e430p-1f, fmaf(fe, -0x1.05c610p-29f, lm));
}

// asin on [0, 1/2], Taylor series with 12 terms.
__device__ __forceinline__ float asin_small_poly(float x) {
    const double c[12] = {
        1.0 / 6.0, 3.0 / 40.0, 15.0 / 336.0, 105.0 / 3456.0, 945.0 / 42240.0,
        10395.0 / 599040.0, 135135.0 / 9676800.0, 2027025.0 / 175472640.0,
        34459425.0 / 3530096640.0, 654729075.0 / 78033715200.0,
        13749310575.0 / 1880240947200.0, 316234143225.0 / 49049763430400.0};
    float z = x * x;
    float p = (float)c[11];
#pragma unroll
    for (int i = 10; i >= 0; --i) p = fmaf(z, p, (float)c[i]);
    p = p * z;
    return fmaf(x, p, x);
}

__device__ __forceinline__ float acos_poly(float x) {
    const float pi = 0x1.921fb6p+1f;
    const float pio2 = 0x1.921fb6p+0f;
    if (!(fabsf(x) <= 1.0f)) return NAN;
    if (fabsf(x) <= 0.5f) return pio2 - asin_small_poly(x);
    float t = sqrtf((1.0f - fabsf(x)) * 0.5f);
    float a = 2.0f * asin_small_poly(t);
    return (x > 0.0f) ? a : pi - a;
}

__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }
__device__ __forceinline__ float4 f4(float x, float y, float z, float w) { return make_float4(x, y, z, w); }

// ---------------------------------------------------------------------------
// data views
// ---------------------------------------------------------------------------

__device__ __forceinline__ Patch load_patch(const PatchPlanes& p, size_t k) {
    float4 a = p.A[k];
    float4 b = p.B[k];
    Patch r;
    r.x = a.x; r.y = a.y; r.theta = a.z; r.layer = __float_as_int(a.w);
    r.hyst = b.x; r.su = b.y; r.sv = b.z; r.lumy = b.w;
    r.luma = p.C[k];
    return r;
}
__device__ __forceinline__ void store_patch(const PatchPlanes& p, size_t k, const Patch& v) {
    p.A[k] = f4(v.x, v.y, v.theta, __int_as_float(v.layer));
    p.B[k] = f4(v.hyst, v.su, v.sv, v.lumy);
    p.C[k] = v.luma;
}
__device__ __forceinline__ Patch make_patch(float x, float y, float th, float h, int layer, float su, float sv) {
    Patch p;
    p.x = x; p.y = y; p.theta = th; p.hyst = h; p.layer = layer;
    p.su = su; p.sv = sv; p.lumy = 0.f; p.luma = 0.f;
    return p;
}

// --- fetches ----------------------------------------------------------------

template <class T>
__device__ __forceinline__ T zero_of();
template <> __device__ __forceinline__ float zero_of<float>() { return 0.0f; }
template <> __device__ __forceinline__ float2 zero_of<float2>() { return make_float2(0.f, 0.f); }
template <> __device__ __forceinline__ float4 zero_of<float4>() { return make_float4(0.f, 0.f, 0.f, 0.f); }

// A texel as the texture unit reads it for linear filtering: subnormal
// values read as zero of the same sign.  Every read of a linearly filtered
// input goes through the filter in the reference, so with PT_FILTER_TEXTURE
// texel reads at integer coordinates flush the same way.
__device__ __forceinline__ float tex_ftz(float t) {
    return fabsf(t) < 1.17549435e-38f ? __int_as_float(__float_as_int(t) & (int)0x80000000) : t;
}
__device__ __forceinline__ float ftz_of(float t) { return tex_ftz(t); }
__device__ __forceinline__ float2 ftz_of(float2 t) { return make_float2(tex_ftz(t.x), tex_ftz(t.y)); }
__device__ __forceinline__ float4 ftz_of(float4 t) {
    return make_float4(tex_ftz(t.x), tex_ftz(t.y), tex_ftz(t.z), tex_ftz(t.w));
}
template <class T>
__device__ __forceinline__ T lin_texel_of(T t, int hw) { return hw ? ftz_of(t) : t; }

// layered image array texel at integer (x, y); the layered inputs (colour,
// distance transform, velocities) are linearly filtered in the reference
template <class T>
__device__ __forceinline__ T lay_texel(const Arr<T>& a, const Params& P, int x, int y) {
    x = clampi(x, 0, P.W - 1);
    y = clampi(y, 0, P.H - 1);
    if (x >= a.w || y >= a.h) return zero_of<T>();
    return lin_texel_of(__ldg(a.p + (size_t)y * a.w + x), P.hwFilter);
}
// level-size array texel at integer (x, y), clamp addressing (point-filtered
// inputs: orientation, ids, random level)
template <class T>
__device__ __forceinline__ T lvl_texel(const Arr<T>& a, int x, int y) {
    x = clampi(x, 0, a.w - 1);
    y = clampi(y, 0, a.h - 1);
    return __ldg(a.p + (size_t)y * a.w + x);
}
// the same for a linearly filtered level-size input (scale, frame-to-key ribbons)
template <class T>
__device__ __forceinline__ T lvl_texel_lin(const Arr<T>& a, int x, int y, int hw) {
    return lin_texel_of(lvl_texel(a, x, y), hw);
}

// point-filtered index at unnormalised u (+0.5), clamp to [0, n-1]
__device__ __forceinline__ int point_index(float u, int n) {
    float f = floorf(u + 0.5f);
    f = fminf(fmaxf(f, -1.0f), (float)n);
    return clampi((int)f, 0, n - 1);
}

struct Bl {
    int x0, x1, y0, y1;
    float w00, w10, w01, w11;   // PT_FILTER_EXACT: FP32 weights
    int hw;                     // PT_FILTER_TEXTURE
    int q00, q10, q01, q11;     // the texture unit's weights, in 1/256
    int r00, r10, r01, r11;     // their unrounded products are nonzero
};
// bilinear footprint at unnormalised (u, v), clamp to (n x m).  The texture
// coordinate is u + 0.5 (as the reference's fetch macros form it) and the
// lower texel floor(u + 0.5 - 0.5).  hw: the texture unit's weights, the
// fractions quantised to 1/256 with ties up (A, B), q11 = (A*B + 128) / 256
// and the other three by difference, as measured on GB300.
__device__ __forceinline__ Bl bl_setup(float u, float v, int n, int m, int hw = 0) {
    Bl b;
    float xs = u + 0.5f, ys = v + 0.5f;
    float xb = xs - 0.5f, yb = ys - 0.5f;
    float fx = floorf(xb), fy = floorf(yb);
    float a = xb - fx, c = yb - fy;
    fx = fminf(fmaxf(fx, -1.0f), (float)n);
    fy = fminf(fmaxf(fy, -1.0f), (float)m);
    int ix = (int)fx, iy = (int)fy;
    b.x0 = clampi(ix, 0, n - 1); b.x1 = clampi(ix + 1, 0, n - 1);
    b.y0 = clampi(iy, 0, m - 1); b.y1 = clampi(iy + 1, 0, m - 1);
    float oa = 1.0f - a, oc = 1.0f - c;
    b.w00 = oa * oc; b.w10 = a * oc; b.w01 = oa * c; b.w11 = a * c;
    b.hw = hw;
    if (hw) {
        // a coordinate of NaN or +-inf reads the edge texel (NaN the low
        // edge, as measured): the clamps above give its index, the fraction
        // is 0.  floor(256 a + 1/2) without rounding: 256 a is exact, and so
        // is its fractional part.
        if (a != a) a = 0.0f;
        if (c != c) c = 0.0f;
        const float sa = a * 256.0f, sc = c * 256.0f;
        const float fa = floorf(sa), fc = floorf(sc);
        const int A = (int)fa + (sa - fa >= 0.5f ? 1 : 0), B = (int)fc + (sc - fc >= 0.5f ? 1 : 0);
        b.q11 = (A * B + 128) >> 8;
        b.q10 = A - b.q11; b.q01 = B - b.q11; b.q00 = 256 - A - B + b.q11;
        b.r00 = (256 - A) * (256 - B) != 0; b.r10 = A * (256 - B) != 0;
        b.r01 = (256 - A) * B != 0; b.r11 = A * B != 0;
    }
    return b;
}

// One channel of the texture unit's bilinear sum: the texels of nonzero
// weight are aligned to the largest exponent among them and truncated
// toward zero to 28 bits below it, summed exactly with the 1/256 weights,
// and the sum is rounded to float with ties away from zero; with no nonzero
// texel the result is a zero, negative only if every texel of nonzero
// unrounded weight is negative-signed.  Subnormal texels read as zero.
// (Out of line: the kernels that take this path only off their hot loop keep
// it off their register budget.)
static __device__ __noinline__ float hw_sum_q(int q00, int q10, int q01, int q11, int rmask, float t00, float t10, float t01,
                                       float t11) {
    const float t[4] = {tex_ftz(t00), tex_ftz(t10), tex_ftz(t01), tex_ftz(t11)};
    const int q[4] = {q00, q10, q01, q11};
    const int r[4] = {rmask & 1, (rmask >> 1) & 1, (rmask >> 2) & 1, (rmask >> 3) & 1};
    int E = -1000;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const unsigned u = __float_as_uint(t[k]);
        const int e = (int)((u >> 23) & 0xffu) - 126;  // frexp exponent of a normal value
        if (q[k] > 0 && (u & 0x7fffffffu) != 0u) E = max(E, e);
    }
    if (E == -1000) {
        bool neg = true;
#pragma unroll
        for (int k = 0; k < 4; k++) neg = neg && (!r[k] || (__float_as_uint(t[k]) >> 31));
        return neg ? -0.0f : 0.0f;
    }
    long long S = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const unsigned u = __float_as_uint(t[k]);
        if (q[k] <= 0 || (u & 0x7fffffffu) == 0u) continue;
        const int e = (int)((u >> 23) & 0xffu) - 126;
        const long long M = (long long)((u & 0x7fffffu) | 0x800000u);  // t = M * 2^(e - 24)
        const int sh = 4 + e - E;                                      // t * 2^(28 - E) = M * 2^sh, sh <= 4
        long long m = sh >= 0 ? (M << sh) : (sh > -25 ? (M >> -sh) : 0);
        S += (long long)q[k] * ((u >> 31) ? -m : m);
    }
    // value S * 2^(E - 36), |S| < 2^39
    if (S == 0) return 0.0f;
    const bool neg = S < 0;
    unsigned long long mag = (unsigned long long)(neg ? -S : S);
    const int msb = 63 - __clzll((long long)mag);
    int e2 = E - 36;
    if (msb > 23) {
        const int drop = msb - 23;
        const unsigned long long rem = mag & ((1ull << drop) - 1ull);
        mag >>= drop;
        if (rem >= (1ull << (drop - 1))) mag += 1ull;  // half away from zero
        e2 += drop;
    }
    const float f = ldexpf((float)mag, e2);
    return neg ? -f : f;
}

__device__ __forceinline__ float hw_sum(const Bl& b, float t00, float t10, float t01, float t11) {
    return hw_sum_q(b.q00, b.q10, b.q01, b.q11, b.r00 | (b.r10 << 1) | (b.r01 << 2) | (b.r11 << 3), t00, t10, t01,
                    t11);
}

__device__ __forceinline__ float bl1(const Bl& b, float t00, float t10, float t01, float t11) {
    if (b.hw) return hw_sum(b, t00, t10, t01, t11);
    float r = t00 * b.w00;
    r = fmaf(t10, b.w10, r);
    r = fmaf(t01, b.w01, r);
    r = fmaf(t11, b.w11, r);
    return r;
}
__device__ __forceinline__ float4 bl4(const Bl& b, float4 a, float4 c, float4 d, float4 e) {
    return f4(bl1(b, a.x, c.x, d.x, e.x), bl1(b, a.y, c.y, d.y, e.y),
              bl1(b, a.z, c.z, d.z, e.z), bl1(b, a.w, c.w, d.w, e.w));
}
// bl4 with two channels per packed f32x2 multiply-add (each component
// rounds exactly as bl1)
__device__ __forceinline__ float4 bl4p(const Bl& b, float4 a, float4 c, float4 d, float4 e) {
    const float2 w00 = make_float2(b.w00, b.w00), w10 = make_float2(b.w10, b.w10);
    const float2 w01 = make_float2(b.w01, b.w01), w11 = make_float2(b.w11, b.w11);
    float2 l = __fmul2_rn(make_float2(a.x, a.y), w00);
    float2 h = __fmul2_rn(make_float2(a.z, a.w), w00);
    l = __ffma2_rn(make_float2(c.x, c.y), w10, l);
    h = __ffma2_rn(make_float2(c.z, c.w), w10, h);
    l = __ffma2_rn(make_float2(d.x, d.y), w01, l);
    h = __ffma2_rn(make_float2(d.z, d.w), w01, h);
    l = __ffma2_rn(make_float2(e.x, e.y), w11, l);
    h = __ffma2_rn(make_float2(e.z, e.w), w11, h);
    return f4(l.x, l.y, h.x, h.y);
}

__device__ __forceinline__ int ex_layer(const ExView& e, int layer) { return clampi(layer, 0, e.ns - 1); }

// An exemplar colour at unnormalised (u, v) through the texture unit
// (PT_FILTER_TEXTURE, the level's textures bound).  The level sits in the
// corner of a larger array with its edge texels repeated once beyond, so the
// coordinate is clamped to [0, w-1] x [0, h-1] first (NaN to 0): that fetches
// the texels, with the weights, that clamp addressing on a w x h array would.
__device__ __forceinline__ float4 ex_tex(cudaTextureObject_t t, const ExView& e, float u, float v, int layer) {
    u = fminf(fmaxf(u, 0.0f), (float)(e.w - 1));
    v = fminf(fmaxf(v, 0.0f), (float)(e.h - 1));
    return tex2DLayered<float4>(t, u + 0.5f, v + 0.5f, ex_layer(e, layer));
}

// exemplar base and output at unnormalised (u, v), one footprint.  These
// three take the texture unit where the level's textures are bound: its
// emulation in integer arithmetic costs some hundred instructions a channel
// (a propagate pass with temporal terms of both neighbours over 240x180
// pixels took 4.8 ms by it).
__device__ __forceinline__ void ex_sample2(const ExView& e, float u, float v, int layer, float4* base, float4* out) {
    if (e.hw && e.tbase) {
        *base = ex_tex(e.tbase, e, u, v, layer);
        *out = ex_tex(e.tout, e, u, v, layer);
        return;
    }
    Bl b = bl_setup(u, v, e.w, e.h, e.hw);
    const size_t L = (size_t)ex_layer(e, layer) * e.w * e.h;
    const size_t r0 = L + (size_t)b.y0 * e.w, r1 = L + (size_t)b.y1 * e.w;
    float4 b00 = __ldg(e.base + r0 + b.x0), b10 = __ldg(e.base + r0 + b.x1);
    float4 b01 = __ldg(e.base + r1 + b.x0), b11 = __ldg(e.base + r1 + b.x1);
    float4 o00 = __ldg(e.out + r0 + b.x0), o10 = __ldg(e.out + r0 + b.x1);
    float4 o01 = __ldg(e.out + r1 + b.x0), o11 = __ldg(e.out + r1 + b.x1);
    *base = bl4(b, b00, b10, b01, b11);
    *out = bl4(b, o00, o10, o01, o11);
}
__device__ __forceinline__ float4 ex_sample_out(const ExView& e, float u, float v, int layer) {
    if (e.hw && e.tout) return ex_tex(e.tout, e, u, v, layer);
    Bl b = bl_setup(u, v, e.w, e.h, e.hw);
    const size_t L = (size_t)ex_layer(e, layer) * e.w * e.h;
    const size_t r0 = L + (size_t)b.y0 * e.w, r1 = L + (size_t)b.y1 * e.w;
    return bl4(b, __ldg(e.out + r0 + b.x0), __ldg(e.out + r0 + b.x1), __ldg(e.out + r1 + b.x0),
               __ldg(e.out + r1 + b.x1));
}
// offsetsToOutput, texSynth_kernel.cu:263-274, of record k
__device__ __forceinline__ float4 canvas_of(const Params& P, size_t k) {
    const float4 a = P.off.A[k];
    const float lumy = P.off.B[k].w, luma = P.off.C[k];
    const float4 c = ex_sample_out(P.ex, a.x, a.y, __float_as_int(a.w));
    return f4(c.x + lumy, c.y + lumy, c.z + lumy, c.w + luma);
}
__device__ __forceinline__ float ex_sample_out_alpha(const ExView& e, float u, float v, int layer) {
    if (e.hw && e.tout) return ex_tex(e.tout, e, u, v, layer).w;
    Bl b = bl_setup(u, v, e.w, e.h, e.hw);
    const float* L = (const float*)(e.out + (size_t)ex_layer(e, layer) * e.w * e.h);
    const float* r0 = L + (size_t)b.y0 * e.w * 4;
    const float* r1 = L + (size_t)b.y1 * e.w * 4;
    return bl1(b, __ldg(r0 + 4 * b.x0 + 3), __ldg(r0 + 4 * b.x1 + 3),
               __ldg(r1 + 4 * b.x0 + 3), __ldg(r1 + 4 * b.x1 + 3));
}
// What the exemplar level's texels can do (k_interleave_texels): whether any
// output alpha is below 0.995, so that a filtered one may be below
// kAlphaThreshold, and whether any distance transform texel is above `cull`.
__device__ __forceinline__ bool exemplar_transparent(const ExView& e) { return __ldg(e.flags) != 0; }
__device__ __forceinline__ bool exemplar_culls(const ExView& e, float cull) {
    return __int_as_float(__ldg(e.flags + 1)) > cull;
}
// the mask of keyframe layer `key` at pixel (x, y): the key's output alpha
// (PYRAMID_FETCH_LAYER(gExemplarOutput, x, y, keyIndex)); -1 without a key
__device__ __forceinline__ float keymask_alpha(const ExView& e, int x, int y, int key) {
    return key < 0 ? -1.0f : ex_sample_out_alpha(e, (float)x, (float)y, key);
}
__device__ __forceinline__ float ex_sample_dt(const ExView& e, float u, float v, int layer) {
    Bl b = bl_setup(u, v, e.w, e.h, e.hw);
    const float* D = e.dt + (size_t)ex_layer(e, layer) * e.w * e.h;
    return bl1(b, __ldg(D + (size_t)b.y0 * e.w + b.x0), __ldg(D + (size_t)b.y0 * e.w + b.x1),
               __ldg(D + (size_t)b.y1 * e.w + b.x0), __ldg(D + (size_t)b.y1 * e.w + b.x1));
}
__device__ __forceinline__ float ex_texel_dt(const ExView& e, int x, int y, int layer) {
    x = clampi(x, 0, e.w - 1); y = clampi(y, 0, e.h - 1);
    return lin_texel_of(__ldg(e.dt + (size_t)ex_layer(e, layer) * e.w * e.h + (size_t)y * e.w + x), e.hw);
}
__device__ __forceinline__ float ex_point_orient(const ExView& e, float u, float v, int layer) {
    int x = point_index(u, e.w), y = point_index(v, e.h);
    return __ldg(e.orient + (size_t)ex_layer(e, layer) * e.w * e.h + (size_t)y * e.w + x);
}
__device__ __forceinline__ int ex_point_id(const ExView& e, float u, float v, int layer) {
    int x = point_index(u, e.w), y = point_index(v, e.h);
    return __ldg(e.ids + (size_t)ex_layer(e, layer) * e.w * e.h + (size_t)y * e.w + x);
}

// layered image array bilinear at unnormalised (u, v): clamp at level-0 size,
// zero outside the level rectangle
template <class T>
__device__ __forceinline__ T lay_bilinear(const Arr<T>& a, const Params& P, float u, float v);
template <>
__device__ __forceinline__ float2 lay_bilinear<float2>(const Arr<float2>& a, const Params& P, float u, float v) {
    Bl b = bl_setup(u, v, P.W, P.H, P.hwFilter);
    float2 t00 = lay_texel(a, P, b.x0, b.y0), t10 = lay_texel(a, P, b.x1, b.y0);
    float2 t01 = lay_texel(a, P, b.x0, b.y1), t11 = lay_texel(a, P, b.x1, b.y1);
    return make_float2(bl1(b, t00.x, t10.x, t01.x, t11.x), bl1(b, t00.y, t10.y, t01.y, t11.y));
}
template <>
__device__ __forceinline__ float4 lay_bilinear<float4>(const Arr<float4>& a, const Params& P, float u, float v) {
    Bl b = bl_setup(u, v, P.W, P.H, P.hwFilter);
    return bl4(b, lay_texel(a, P, b.x0, b.y0), lay_texel(a, P, b.x1, b.y0),
               lay_texel(a, P, b.x0, b.y1), lay_texel(a, P, b.x1, b.y1));
}

__device__ __forceinline__ bool in_rect(const Params& P, int x, int y, int border = 0) {
    return x >= border && y >= border && x < P.lw - border && y < P.lh - border;
}

}  // namespace ptk
