// H0 and H1 of a real argument x as functions of u = x^2, from a table.
//
//   f(u) = H0(sqrt u),   g(u) = H1(sqrt u) / sqrt u,
//
// the two functions every kernel value of the assembly and of the Green sum is made of
// (with u = ks^2 |v|^2: h0 = f, ks h1 / |v| = ks^2 g, |v| h1 = ks |v|^2 g), so that a
// quadrature point needs neither the distance nor its reciprocal, and no logarithm, sine
// or square root.  With h_m = H_m(x) / x^m, dh_m/du = -h_(m+1) / 2: the Taylor
// coefficients about u_c are f_m = (-1/2)^m h_m / m! and g_m = -2 (m + 1) f_(m+1).
//
// What bounds the kernels that call this is the FP64 pipe: a warp's FP64 instruction
// (an add, a multiply, a comparison or a conversion to or from FP32 as much as an FMA)
// holds its SM sub-partition for 64 cycles, an FP32 or integer one for 1 to 4.  So the
// interval, the position in it and the conversions are integer arithmetic on the bits of
// u, the intervals are so short (a relative half width of 2^-8 in u below 16, at most
// 2^-7.5 in x above) that the terms from the fourth power on are below 2^-33 of the
// value and FP32 serves for them, and 17 FP64 instructions are left for the four real
// functions (measured before: 68 for the Taylor band, about 110 beyond x = 8, each with
// the square root, the reciprocal and the branch on top).
//
// The table covers 2^-110 <= u < 2^18 (x from 3e-17 to 512) in 79,616 intervals of 176
// bytes (14.0 MB, resident in L2; the points of a warp lie close together, so its
// working set is a few KB of L1).  It is made once per device on its first use, in
// double-double arithmetic (ascending series up to x = 25, Hankel's expansion beyond),
// so that its entries are rounded once.  Outside of it callers take hankel01_real.
#pragma once
#include "hbem_device.cuh"

namespace hbem {

struct alignas(16) HkEntry {
    double c[2][4][2];   // f, g: coefficients 0..3 times the half width's powers (re, im)
    float s[2][3][2];    // coefficients 4..6
};

constexpr int kHkEMin = -110, kHkEMax = 18;         // binary exponents of u covered
constexpr int kHkLow = (4 - kHkEMin) * 128;         // intervals below u = 16: 128 per octave
constexpr int kHkEntries = kHkLow + 512 * ((1 << ((kHkEMax - 4) / 2)) - 1);
constexpr unsigned kHkHiMin = (unsigned)(1023 + kHkEMin) << 20;
constexpr unsigned kHkHiSpan = (unsigned)(kHkEMax - kHkEMin) << 20;

// bits of the interval's index within an octave, by the binary exponent of u: 7 below
// u = 16, then one more every two octaves (x doubles): equal steps in x
__host__ __device__ __forceinline__ int hk_bits(int e) { return e < 4 ? 7 : 8 + ((e - 4) >> 1); }

// first interval of octave e
__host__ __device__ __forceinline__ int hk_base(int e) {
    if (e < 4) return (e - kHkEMin) << 7;
    const int p = (e - 4) >> 1;
    return kHkLow + 512 * ((1 << p) - 1) + (((e - 4) & 1) << (8 + p));
}

#ifdef __CUDACC__
// FP32 -> FP64 without the conversion instruction (FP64 pipe): rebias the exponent.  Zero
// and subnormals become values below 2^-125, of no consequence in the sums used here.
__device__ __forceinline__ double hk_widen(float x) {
    const int b = __float_as_int(x);
    return __hiloint2double(((b >> 3) & 0x8fffffff) + 0x38000000, b << 29);
}

// whether u is inside the table
__device__ __forceinline__ bool hk_inside(double u) {
    return (unsigned)__double2hiint(u) - kHkHiMin < kHkHiSpan;
}

// f and g at u inside the table
__device__ __forceinline__ void hk_eval(const HkEntry* __restrict__ tab, double u, cplx& f, cplx& g) {
    const int hi = __double2hiint(u), lo = __double2loint(u);
    const int e = (hi >> 20) - 1023;
    const int b = hk_bits(e);
    const HkEntry* E = tab + hk_base(e) + ((hi & 0xfffff) >> (20 - b));
    // the bits below the index, left-aligned: the position in the interval as a fraction
    const unsigned wh = __funnelshift_l((unsigned)lo, (unsigned)hi, 12 + b), wl = (unsigned)lo << (12 + b);
    const float tf = (float)(int)(wh ^ 0x80000000u) * 4.656612873077393e-10f;   // 2^-31
    const double y = __hiloint2double(0x3ff00000 | (int)(wh >> 12), (int)__funnelshift_r(wl, wh, 12));
    const double t = fma(2., y, -3.);                                           // exact, in [-1, 1)
    const float4* S = reinterpret_cast<const float4*>(&E->s[0][0][0]);
    const float4 s0 = __ldg(S), s1 = __ldg(S + 1), s2 = __ldg(S + 2);
    const double2* c = reinterpret_cast<const double2*>(&E->c[0][0][0]);
    const double2 f0 = __ldg(c), f1 = __ldg(c + 1), f2 = __ldg(c + 2), f3 = __ldg(c + 3);
    const double2 g0 = __ldg(c + 4), g1 = __ldg(c + 5), g2 = __ldg(c + 6), g3 = __ldg(c + 7);
    const double tfr = hk_widen(tf * fmaf(tf, fmaf(tf, s1.x, s0.z), s0.x));
    const double tfi = hk_widen(tf * fmaf(tf, fmaf(tf, s1.y, s0.w), s0.y));
    const double tgr = hk_widen(tf * fmaf(tf, fmaf(tf, s2.z, s2.x), s1.z));
    const double tgi = hk_widen(tf * fmaf(tf, fmaf(tf, s2.w, s2.y), s1.w));
    f.re = fma(fma(fma(f3.x + tfr, t, f2.x), t, f1.x), t, f0.x);
    f.im = fma(fma(fma(f3.y + tfi, t, f2.y), t, f1.y), t, f0.y);
    g.re = fma(fma(fma(g3.x + tgr, t, g2.x), t, g1.x), t, g0.x);
    g.im = fma(fma(fma(g3.y + tgi, t, g2.y), t, g1.y), t, g0.y);
}

// outside the table: u <= 0 counts as the coincidence of the two points (H0 = 1 and no
// contribution of H1, as hankel01_real has it)
static __device__ __noinline__ void hk_slow(double u, cplx& f, cplx& g) {
    if (!(u > 0.)) {
        f = u == u ? mk(1.) : mk(u, u);
        g = u == u ? mk(0.) : mk(u, u);
        return;
    }
    const double x = sqrt(u);
    cplx h1;
    hankel01_real(x, f, h1);
    const double ix = 1.0 / x;
    g = ix * h1;
}

__device__ __forceinline__ void hk_pair(const HkEntry* __restrict__ tab, double u, cplx& f, cplx& g) {
    if (hk_inside(u)) hk_eval(tab, u, f, g);
    else hk_slow(u, f, g);
}

// the table on the current device (made on its first use; null with *err set on failure)
const HkEntry* hankel_table(cudaError_t* err);
#endif

}  // namespace hbem
