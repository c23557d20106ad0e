// The compensated compound-Poisson term w (e^{i k kappa} - 1 - i k kappa) summed over cells in FP32, two cells per
// packed instruction (the inner loop of the 1-D sweep and of the batched solver).
//
// With x = k kappa / 2 (float-float) and r = x - q pi, |r| <= pi/2 + slack, both parts are even / odd functions of r
// alone, so there is no quadrant to select and no small-argument branch:
//     1 - cos(k kappa) = 2 sin^2 x            = 2 r^2 H(r^2),                 H(u) = (sin r / r)^2
//     k kappa - sin(k kappa) = 2 (x - sin x cos x) = 4/3 (r^3 G(r^2) + 1.5 pi q),  G(u) = 1.5 (r - sin r cos r) / r^3
// H and G: degree-6 polynomials in u, least-maximum fits on |r| <= pi/2 with their coefficients rounded to FP32 one
// after the other (relative error 2.3e-9 and 6e-10, mean 1e-10; 1.5e-8 and 4e-9 up to |r| = 1.95).  The factor 1.5 makes G(0) = 1, exact in FP32.  Per term, against 64 bits over
// phases 1e-4 .. 1e7: 1 - cos 5e-8 .. 7e-8 rms (quadrant form with Taylor polynomials: 5e-8 .. 8e-8), k kappa - sin
// 2.4e-8 .. 1e-7 (3e-8 .. 5e-5: sin(ph) - ph cancels below ph = 1).
//
// Bound by the FP32 pipe: 31 packed operations per two terms, against 39 and about 15 of the ALU per term with the
// five-step reduction, the quadrant's selects and the branch.  Sums: Kahan over groups of 8 cells (4 per lane).
#pragma once
#include "common.cuh"

namespace sgl {

constexpr int kCfGroup = 8;                    // cells per Kahan step: lists are padded to it with zeros

__device__ __forceinline__ unsigned long long f32x2_mul(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long f32x2_add(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long f32x2_fma3(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ unsigned long long f32x2_dup(float v) { return f32x2_pack(v, v); }

// Kahan sums of w r^2 H and w (r^3 G + 1.5 pi q), per lane of the pair: value s + c
struct CfSums {
    unsigned long long s0, c0, s1, c1;
    __device__ __forceinline__ void clear() { s0 = c0 = s1 = c1 = 0ull; }
    // the sums' (real, imaginary) parts of sum w (e^{i ph} - 1 - i ph)
    __device__ __forceinline__ double2 value() const {
        const float2 a = f32x2_unpack(s0), b = f32x2_unpack(c0), d = f32x2_unpack(s1), e = f32x2_unpack(c1);
        const double re = ((double)a.x + (double)b.x) + ((double)a.y + (double)b.y);
        const double im = ((double)d.x + (double)e.x) + ((double)d.y + (double)e.y);
        return make_double2(-2.0 * re, -(4.0 / 3.0) * im);
    }
};

// half the wave number, as packed constants
struct CfWave {
    unsigned long long kh, nkh, nkl;
    __device__ __forceinline__ explicit CfWave(double k) {
        const ff h = ff_from_double(0.5 * k);
        kh = f32x2_dup(h.hi);
        nkh = f32x2_dup(-h.hi);
        nkl = f32x2_dup(-h.lo);
    }
};

// Above q = 2^19 (phases of 3.3e6) the rounding of x / pi in FP32 leaves |r| beyond pi/2 + 0.17, up to pi at q = 2^24,
// where the polynomials no longer hold: such tiles reduce r once more (cf_pair<true>, 5 more operations).
constexpr float kCfBigHalfPhase = 1.64e6f;     // pi 2^19

// r^2 H(r^2) and r^3 G(r^2) + 1.5 pi q of two cells (kappa head ah, tail al)
template <bool BIG>
__device__ __forceinline__ void cf_pair(const CfWave& k, unsigned long long ah, unsigned long long al,
                                        unsigned long long& h, unsigned long long& v) {
    const unsigned long long p = f32x2_mul(k.kh, ah);
    unsigned long long nt = f32x2_fma3(k.nkh, ah, p);                  // minus the product's rounding error, then
    nt = f32x2_fma3(k.nkl, ah, nt);                                    // minus the float-float tail
    nt = f32x2_fma3(k.nkh, al, nt);
    const float2 m = f32x2_unpack(f32x2_mul(p, f32x2_dup(0.318309886183790672f)));
    unsigned long long q = f32x2_pack(rintf(m.x), rintf(m.y));
    // x - q pi, pi in three float parts; each FMA rounds once (the first two cancel exactly or nearly so)
    unsigned long long r = f32x2_fma3(q, f32x2_dup(-3.1415927410125732f), p);
    r = f32x2_fma3(q, f32x2_dup(8.742277657347586e-08f), r);
    nt = f32x2_fma3(q, f32x2_dup(-3.4302490e-15f), nt);
    r = f32x2_fma3(nt, f32x2_dup(-1.f), r);
    if (BIG) {
        const float2 m2 = f32x2_unpack(f32x2_mul(r, f32x2_dup(0.318309886183790672f)));
        const unsigned long long q2 = f32x2_pack(rintf(m2.x), rintf(m2.y));
        r = f32x2_fma3(q2, f32x2_dup(-3.1415927410125732f), r);
        r = f32x2_fma3(q2, f32x2_dup(8.742277657347586e-08f), r);
        q = f32x2_add(q, q2);
    }
    const unsigned long long u = f32x2_mul(r, r);
    h = f32x2_fma3(u, f32x2_dup(7.6129993e-08f), f32x2_dup(-4.19144681e-06f));
    h = f32x2_fma3(u, h, f32x2_dup(0.000140896969f));
    h = f32x2_fma3(u, h, f32x2_dup(-0.00317437248f));
    h = f32x2_fma3(u, h, f32x2_dup(0.0444443226f));
    h = f32x2_fma3(u, h, f32x2_dup(-0.333333313f));
    h = f32x2_fma3(u, h, f32x2_dup(1.f));
    h = f32x2_mul(u, h);
    unsigned long long g = f32x2_fma3(u, f32x2_dup(1.60065277e-08f), f32x2_dup(-9.75810735e-07f));
    g = f32x2_fma3(u, g, f32x2_dup(3.84614905e-05f));
    g = f32x2_fma3(u, g, f32x2_dup(-0.00105819001f));
    g = f32x2_fma3(u, g, f32x2_dup(0.0190476216f));
    g = f32x2_fma3(u, g, f32x2_dup(-0.200000003f));
    g = f32x2_fma3(u, g, f32x2_dup(1.f));
    v = f32x2_mul(q, f32x2_dup(-1.1924880638503e-08f));                // 1.5 pi = 4.712389 - 1.19e-8
    v = f32x2_fma3(f32x2_mul(r, u), g, v);
    v = f32x2_fma3(q, f32x2_dup(4.7123889923095703f), v);
}

// adds cells [0, n8) of a tile (n8 a multiple of kCfGroup; heads, tails and weights as 16-byte aligned arrays)
template <bool BIG>
__device__ __forceinline__ void cf_tile(const CfWave& k, const float* ah, const float* al, const float* w, int n8, CfSums& S) {
    const ulonglong2* h2 = reinterpret_cast<const ulonglong2*>(ah);
    const ulonglong2* l2 = reinterpret_cast<const ulonglong2*>(al);
    const ulonglong2* w2 = reinterpret_cast<const ulonglong2*>(w);
    const unsigned long long m1 = f32x2_dup(-1.f);
#pragma unroll 1
    for (int e = 0; e < n8 / 4; e += 2) {
        unsigned long long y0 = S.c0, y1 = S.c1;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const ulonglong2 hh = h2[e + j], ll = l2[e + j], ww = w2[e + j];
            unsigned long long h, v;
            cf_pair<BIG>(k, hh.x, ll.x, h, v);
            y0 = f32x2_fma3(ww.x, h, y0);
            y1 = f32x2_fma3(ww.x, v, y1);
            cf_pair<BIG>(k, hh.y, ll.y, h, v);
            y0 = f32x2_fma3(ww.y, h, y0);
            y1 = f32x2_fma3(ww.y, v, y1);
        }
        const unsigned long long t0 = f32x2_add(S.s0, y0), t1 = f32x2_add(S.s1, y1);
        S.c0 = f32x2_add(f32x2_fma3(t0, m1, S.s0), y0);                // y - (t - s)
        S.c1 = f32x2_add(f32x2_fma3(t1, m1, S.s1), y1);
        S.s0 = t0;
        S.s1 = t1;
    }
}

}  // namespace sgl
