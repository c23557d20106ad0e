// Per-cosmology background and linear-theory tables on the GPU: the default chain's Cosmology of the
// reference (sgl.py:65-640 as pipeline.make_cosmology builds it, pipeline.py:39-79): CPL dark energy
// with curvature and radiation Omega_r = Om / (1 + z_eq); E(z); the radial comoving distance chi(z) and
// the transverse D_M(z); the linear growth D(z) from the growth ODE (sgl.py:310-347); the EH98 transfer
// function with baryons (sgl.py:391-445); sigma(M) through the smooth-k filter with the top-hat sigma_8
// anchor (sgl.py:452-553) on the reference's k and M grids with its not-a-knot spline in ln M; the
// Sheth-Tormen dn/dln M (sgl.py:556-568) and the Ludlow+16 concentration (sgl.py:570-606).
//
// The arithmetic is the reference's (FP64); where it calls an adaptive integrator this file uses fixed
// high-order rules instead: composite 8-point Gauss-Legendre panels of width <= 0.02 for chi (the
// reference: quad), classical RK4 with 2^15 steps in ln a for the growth ODE (the reference: DOP853 at
// rtol 2e-10), and the not-a-knot cubic spline through its tridiagonal system solved by elimination (the
// reference: scipy's CubicSpline / solve_banded).
//
// Three launches, each over (part of the work, cosmology), because one CTA per cosmology left most of the
// chip idle and its one-thread ODE set the time (a call with 24 cosmologies: 712 ms; in this form 3.2 ms):
//   k_cos_parts  growth: the ODE is linear, so the RK4 steps of a chunk compose to a 2 x 2 matrix, one thread
//                per chunk; the transfer function on the k grid; the distance panels, one warp per interval;
//   k_cos_sums   the 500 sums of sigma(M), one warp each, and the growth at the output points (one thread
//                scans the chunks' matrices, then one thread per output steps on from its chunk's start);
//   k_cos_out    per cosmology the spline, the distances' running sums and the tables.
// Bound by the FP64 pipe (2 FMA per clock and SM): see each kernel for its count.
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"

namespace sgl {
namespace {

constexpr double kCkms = 299792.458;          // km/s
constexpr double kRhoc0Unit = 2.77536627e11;  // Msun / Mpc^3 / h^2
constexpr double kTcmb = 2.7255;
constexpr double kDc = 1.686;
constexpr int kNk = 4000;                      // sigma(R) k grid: logspace(-5, 3, 4000)
constexpr int kNm = 500;                       // sigma(M) spline nodes: logspace(4, 17, 500)
constexpr int kOdeSteps = 1 << 15;
constexpr int kThreads = 256;
constexpr int kPartThreads = 64;               // k_cos_parts: small CTAs, so that one cosmology fills many SMs
constexpr int kChunkSteps = 32;                // RK4 steps composed by one thread
constexpr int kChunks = kOdeSteps / kChunkSteps;
constexpr int kGrowthCtas = kChunks / kPartThreads;
constexpr int kKgridCtas = (kNk + kPartThreads - 1) / kPartThreads;
constexpr int kNodeCtas = (kNm + kThreads / 32 - 1) / (kThreads / 32);
// scratch of one cosmology (doubles): k^2 P(k) times the trapezoid weight, k^6, the sigma_8 sum per CTA,
// the sums of sigma(M), the chunks' matrices, the growth at the output points and at z = 0
constexpr int kOffP = 0, kOffK6 = kNk, kOffS8 = 2 * kNk, kOffS2 = kOffS8 + kKgridCtas,
              kOffMat = (kOffS2 + kNm + 1) / 2 * 2 /* read in pairs */,
              kOffGrow = kOffMat + 4 * kChunks;

struct Cos {
    double h, Om, Ob, s8, ns, zeq, Ok, w0, wa;
    double Or, OL, H0, rhom;
};

__device__ __forceinline__ Cos make_cos(const double* p) {
    Cos c;
    c.h = p[0]; c.Om = p[1]; c.Ob = p[2]; c.s8 = p[3]; c.ns = p[4]; c.zeq = p[5]; c.Ok = p[6]; c.w0 = p[7]; c.wa = p[8];
    c.Or = c.Om / (1.0 + c.zeq);
    c.OL = 1.0 - c.Om - c.Ok - c.Or;
    c.H0 = 100.0 * c.h;
    c.rhom = c.Om * kRhoc0Unit * c.h * c.h;
    return c;
}

// E(z), the reference's branches (sgl.py:183-195)
__device__ double cos_E(const Cos& c, double z) {
    if (c.w0 == -1.0 && c.wa == 0.0 && c.Ok == 0.0)
        return sqrt(c.Om * (1 + z) * (1 + z) * (1 + z) + c.Or * (1 + z) * (1 + z) * (1 + z) * (1 + z) + c.OL);
    const double zp1 = 1.0 + z;
    double de;
    if (c.wa == 0.0) de = c.w0 == -1.0 ? c.OL : c.OL * pow(zp1, 3 * (1 + c.w0));
    else de = c.OL * pow(zp1, 3 * (1 + c.w0 + c.wa)) * exp(-3 * c.wa * (1 - 1 / zp1));
    return sqrt(c.Om * zp1 * zp1 * zp1 + c.Or * zp1 * zp1 * zp1 * zp1 + c.Ok * zp1 * zp1 + de);
}

// transverse comoving distance of a radial interval (sgl.py:219-238)
__device__ double cos_fK(const Cos& c, double chi) {
    if (c.Ok == 0.0) return chi;
    const double u = chi * c.H0 / kCkms;
    const double t = c.Ok * u * u;
    if (fabs(t) < 1e-5) return chi * (1 + t / 6 + t * t / 120 + t * t * t / 5040);
    const double x = sqrt(fabs(c.Ok)) * u;
    return chi * (c.Ok > 0 ? sinh(x) / x : sin(x) / x);
}

// the growth ODE in x = ln a (sgl.py:320-336): y0' = y1, y1' = -p y1 + q y0
struct GrowthCoef { double p, q; };

__device__ __forceinline__ GrowthCoef growth_coef(const Cos& c, double x) {
    const double a = exp(x), ia = exp(-x), ia2 = ia * ia;
    const double matter = c.Om * (ia2 * ia);
    const double rad = c.Or * (ia2 * ia2);
    const double curvature = c.Ok * ia2;
    double de = c.OL;
    if (c.w0 != -1.0 || c.wa != 0.0) de *= exp(-3 * (1 + c.w0 + c.wa) * x + 3 * c.wa * (a - 1));
    const double wz = c.w0 + c.wa * (1 - a);
    const double inv = 1.0 / (matter + rad + curvature + de);
    const double dh = -0.5 * (3 * matter + 4 * rad + 2 * curvature + 3 * (1 + wz) * de) * inv;
    return GrowthCoef{2 + dh, 1.5 * (matter * inv)};
}

// one classical RK4 step of length hs with the coefficients at its start, middle and end
__device__ __forceinline__ void rk4(GrowthCoef s, GrowthCoef m, GrowthCoef e, double hs, double& y0, double& y1) {
    const double a0 = y1, a1 = s.q * y0 - s.p * y1;
    const double u0 = y0 + 0.5 * hs * a0, u1 = y1 + 0.5 * hs * a1;
    const double b0 = u1, b1 = m.q * u0 - m.p * u1;
    const double v0 = y0 + 0.5 * hs * b0, v1 = y1 + 0.5 * hs * b1;
    const double c0 = v1, c1 = m.q * v0 - m.p * v1;
    const double w0 = y0 + hs * c0, w1 = y1 + hs * c1;
    const double e0 = w1, e1 = e.q * w0 - e.p * w1;
    y0 += hs / 6 * (a0 + 2 * b0 + 2 * c0 + e0);
    y1 += hs / 6 * (a1 + 2 * b1 + 2 * c1 + e1);
}

// the fixed step grid: x_0 = ln 1e-6, x_s = x_0 + s h, x_{2^15} = 0
__device__ __forceinline__ double growth_x(int s) {
    const double x0 = log(1e-6);
    return s == kOdeSteps ? 0.0 : x0 + s * (-x0 / kOdeSteps);
}

// EH98 CDM + baryon transfer function (sgl.py:391-445; Eisenstein & Hu 1998, ApJ 496, 605)
struct Eh98 {
    double Om, Ob, Oc, keq, ksilk, ac, bc, s, ab, bb, bnode;
};

__device__ Eh98 make_eh98(const Cos& c) {
    Eh98 e;
    const double h = c.h, Om = c.Om, Ob = c.Ob, Oc = Om - Ob;
    const double wm = Om * h * h, wb = Ob * h * h;
    e.Om = Om; e.Ob = Ob; e.Oc = Oc;
    e.keq = (c.H0 / kCkms) * sqrt(2.0 * Om) * sqrt(1.0 + c.zeq);
    e.ksilk = 0.0016 * pow(wb, 0.52) * pow(wm, 0.73) * (1 + pow(10.4 * wm, -0.95));
    const double a1 = pow(46.9 * wm, 0.67) * (1 + pow(32.1 * wm, -0.532));
    const double a2 = pow(12.0 * wm, 0.424) * (1 + pow(45.0 * wm, -0.582));
    const double b1 = 0.944 / (1 + pow(458 * wm, -0.708));
    const double b2 = pow(0.395 * wm, -0.026);
    e.ac = pow(a1, -Ob / Om) * pow(a2, -pow(Ob / Om, 3));
    e.bc = 1.0 / (1 + b1 * (pow(Oc / Om, b2) - 1));
    e.s = 44.5 * log(9.83 / wm) / sqrt(1 + 10 * pow(wb, 0.75));
    const double b3 = 0.313 * pow(wm, -0.419) * (1 + 0.607 * pow(wm, 0.674));
    const double b4 = 0.238 * pow(wm, 0.223);
    const double zd = 1291 * pow(wm, 0.251) / (1 + 0.659 * pow(wm, 0.828)) * (1 + b3 * pow(wb, b4));
    const double Rd = 31.5 * wb * pow(kTcmb / 2.7, -4) / (zd / 1000.0);
    const double y = (1 + c.zeq) / (1 + zd);
    const double g2 = y * (-6 * sqrt(1 + y) + (2.0 + 3.0 * y) * log((sqrt(1 + y) + 1) / (sqrt(1 + y) - 1)));
    e.ab = 2.07 * e.keq * e.s * pow(1 + Rd, -0.75) * g2;
    e.bb = 0.5 + Ob / Om + (3.0 - 2.0 * Ob / Om) * sqrt(1 + (17.2 * wm) * (17.2 * wm));
    e.bnode = 8.41 * pow(wm, 0.435);
    return e;
}

__device__ __forceinline__ double eh_To1(const Eh98& e, double k, double a_c, double b_c) {
    const double qq = k / (13.41 * e.keq);
    const double C1 = 14.2 / a_c + 386.0 / (1 + 69.9 * pow(qq, 1.08));
    const double num = log(M_E + 1.8 * b_c * qq);
    return num / (num + C1 * qq * qq);
}

__device__ double eh_T(const Eh98& e, double k) {
    const double ks = k * e.s;
    const double fk = 1.0 / (1 + pow(ks / 5.4, 4));
    const double TC = fk * eh_To1(e, k, 1.0, e.bc) + (1 - fk) * eh_To1(e, k, e.ac, e.bc);
    const double s3 = e.s / cbrt(1 + pow(e.bnode / ks, 3));
    const double x = k * s3;
    const double jo = x < 1e-8 ? 1.0 - x * x / 6.0 : sin(x) / x;
    const double TB = (eh_To1(e, k, 1.0, 1.0) / (1 + (ks / 5.2) * (ks / 5.2)) +
                       e.ab / (1 + pow(e.bb / ks, 3)) * exp(-pow(k / e.ksilk, 1.4))) * jo;
    return e.Ob / e.Om * TB + e.Oc / e.Om * TC;
}

struct CosArgs {
    const double* params;                 // [cosmology][9]
    int nz; const double* z;              // distance / growth redshifts (ascending)
    const double* x_out;                  // growth output points ln a, ascending, with their slots
    const int* x_slot; int nx;
    int nm; const double* M;              // output masses
    int nzm; const double* zm;            // mass-function redshifts
    double A_st;                          // Sheth-Tormen normalisation
    double* E; double* chi; double* DM; double* D;       // [cosmology][nz]
    double* Dm;                           // [cosmology][nzm] growth at the mass-function redshifts
    double* sigM; double* dlnsig;         // [cosmology][nm] sigma(M, 0), d ln sigma / d ln M
    double* dndlnM; double* conc;         // [cosmology][nzm][nm]
    double* work;                         // [cosmology][work_stride] scratch
    long long work_stride;                // kOffGrow + nx + 1
};

// Part 1 of a cosmology (blockIdx.y), by blockIdx.x: growth chunks, k grid, distance intervals.  FP64 operations:
// 2^15 steps x about 280 (two coefficient points, two columns), 4000 x about 1500 (EH98's powers), 72 E(z) per
// 0.18 of redshift.
__global__ void __launch_bounds__(kPartThreads) k_cos_parts(CosArgs a) {
    const int ci = blockIdx.y, t = threadIdx.x;
    const Cos c = make_cos(a.params + 9LL * ci);
    double* work = a.work + (long long)ci * a.work_stride;
    int part = blockIdx.x;
    if (part < kGrowthCtas) {
        const int chunk = part * kPartThreads + t, s0 = chunk * kChunkSteps;
        double m00 = 1.0, m10 = 0.0, m01 = 0.0, m11 = 1.0;            // the columns of the chunk's matrix
        double x = growth_x(s0);
        GrowthCoef cs = growth_coef(c, x);
        for (int s = s0; s < s0 + kChunkSteps; ++s) {
            const double xn = growth_x(s + 1), hs = xn - x;
            const GrowthCoef cm = growth_coef(c, x + 0.5 * hs), ce = growth_coef(c, xn);
            rk4(cs, cm, ce, hs, m00, m10);
            rk4(cs, cm, ce, hs, m01, m11);
            x = xn;
            cs = ce;
        }
        double* m = work + kOffMat + 4LL * chunk;
        m[0] = m00; m[1] = m01; m[2] = m10; m[3] = m11;
        return;
    }
    part -= kGrowthCtas;
    if (part < kKgridCtas) {
        // k^2 P_shape with its trapezoid weight, and the sigma_8 anchor through the real-space top hat
        const int i = part * kPartThreads + t;
        const Eh98 e = make_eh98(c);
        double s8 = 0.0;
        if (i < kNk) {
            auto kgrid = [](int j) { return j == kNk - 1 ? 1000.0 : pow(10.0, -5.0 + j * (8.0 / (kNk - 1))); };
            const double k = kgrid(i);
            const double wgt = 0.5 * (kgrid(min(i + 1, kNk - 1)) - kgrid(max(i - 1, 0)));
            const double T = eh_T(e, k);
            const double P = k * k * pow(k, c.ns) * T * T * wgt;
            const double x = k * (8.0 / c.h);
            const double W = 3 * (sin(x) - x * cos(x)) / (x * x * x);
            const double k2 = k * k;
            work[kOffP + i] = P;
            work[kOffK6 + i] = k2 * k2 * k2;
            s8 = P * W * W;
        }
        __shared__ double red[kPartThreads / 32];
        s8 = warp_sum(s8);
        if ((t & 31) == 0) red[t >> 5] = s8;
        __syncthreads();
        if (t == 0) work[kOffS8 + part] = red[0] + red[1];
        return;
    }
    part -= kKgridCtas;
    // 8-point Gauss-Legendre panels of width <= 0.02 between consecutive redshifts, lanes over the panels
    const int j = part * (kPartThreads / 32) + (t >> 5), lane = t & 31;
    if (j >= a.nz) return;
    const double za = j == 0 ? 0.0 : a.z[j - 1], zb = a.z[j];
    const int np = max(1, (int)ceil((zb - za) / 0.02));
    const double xg[4] = {0.1834346424956498, 0.5255324099163290, 0.7966664774136267, 0.9602898564975363};
    const double wg[4] = {0.3626837833783620, 0.3137066458778873, 0.2223810344533745, 0.1012285362903763};
    const double hw = 0.5 * (zb - za) / np;
    double acc = 0.0;
    for (int q = lane; q < 4 * np; q += 32) {
        const double mid = za + (2 * (q >> 2) + 1) * hw, d = hw * xg[q & 3];
        acc += wg[q & 3] * (1.0 / cos_E(c, mid - d) + 1.0 / cos_E(c, mid + d));
    }
    acc = warp_sum(acc);
    if (lane == 0) {
        a.chi[(long long)ci * a.nz + j] = acc * hw * kCkms / c.H0;          // this interval; summed in k_cos_out
        a.E[(long long)ci * a.nz + j] = cos_E(c, zb);
    }
}

// 1 / d for 1 <= d < 1e300: PTX's approximate reciprocal (the operand's upper 32 bits, a 20-bit mantissa: relative error
// below 2^-19) and two Newton steps (2^-38, then FP64's own rounding)
__device__ __forceinline__ double recip(double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    r = fma(r, fma(-d, r, 1.0), r);
    return fma(r, fma(-d, r, 1.0), r);
}

// Part 2: CTAs 0 .. kNodeCtas - 1: the sum over k of sigma^2(M) on the spline nodes (smooth-k filter), one warp per
// node; 2e6 terms of 8 FP64 operations per cosmology (with pow and divisions, twice per term, these sums alone took
// 100 ms on one SM).  The last CTA: the growth at the output points.
__global__ void __launch_bounds__(kThreads) k_cos_sums(CosArgs a) {
    const int ci = blockIdx.y, t = threadIdx.x;
    const Cos c = make_cos(a.params + 9LL * ci);
    double* work = a.work + (long long)ci * a.work_stride;
    if (blockIdx.x == kNodeCtas) {
        __shared__ double s_y[2 * (kChunks + 1)];
        for (int i = t; i < kChunks; i += kThreads) {                  // bring the matrices near
            const double* m = work + kOffMat + 4LL * i;
            asm volatile("prefetch.global.L1 [%0];" ::"l"(m));
        }
        if (t == 0) {
            const double x0 = log(1e-6);
            double y0 = exp(x0) + (c.Or != 0.0 ? (2.0 / 3.0) * c.Or / c.Om : 0.0), y1 = exp(x0);
            for (int i = 0; i < kChunks; ++i) {
                s_y[2 * i] = y0;
                s_y[2 * i + 1] = y1;
                const double2* m = reinterpret_cast<const double2*>(work + kOffMat + 4LL * i);
                const double2 r0 = m[0], r1 = m[1];
                const double n0 = r0.x * y0 + r0.y * y1;
                y1 = r1.x * y0 + r1.y * y1;
                y0 = n0;
            }
            s_y[2 * kChunks] = y0;
            s_y[2 * kChunks + 1] = y1;
            work[kOffGrow + a.nx] = y0;
        }
        __syncthreads();
        for (int j = t; j < a.nx; j += kThreads) {
            // the step whose end is the first one not below the output: whole steps up to it, then a partial step
            const double xo = a.x_out[j];
            int lo = 0, hi = kOdeSteps - 1;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (xo <= growth_x(mid + 1)) hi = mid; else lo = mid + 1;
            }
            if ((lo + 1) % kChunkSteps == 0 && xo == growth_x(lo + 1)) {      // a chunk's end (z = 0: D = 1 exactly)
                work[kOffGrow + j] = s_y[2 * ((lo + 1) / kChunkSteps)];
                continue;
            }
            const int chunk = lo / kChunkSteps;
            double y0 = s_y[2 * chunk], y1 = s_y[2 * chunk + 1];
            double x = growth_x(chunk * kChunkSteps);
            for (int s = chunk * kChunkSteps; s <= lo; ++s) {
                const double xn = s == lo ? xo : growth_x(s + 1), hs = xn - x;
                if (hs > 0) rk4(growth_coef(c, x), growth_coef(c, x + 0.5 * hs), growth_coef(c, xn), hs, y0, y1);
                x = xn;
            }
            work[kOffGrow + j] = y0;
        }
        return;
    }
    const int m = blockIdx.x * (kThreads / 32) + (t >> 5), lane = t & 31;
    if (m >= kNm) return;
    const double Mn = pow(10.0, 4.0 + m * (13.0 / (kNm - 1)));
    const double R = 0.43 * cbrt(3 * Mn / (4 * M_PI * c.rhom));
    const double R2 = R * R, R6 = R2 * R2 * R2;
    double acc = 0.0;
    if (R6 < 1e280) {
#pragma unroll 5
        for (int i = lane; i < kNk; i += 32) {
            const double W = recip(fma(R6, work[kOffK6 + i], 1.0));
            acc = fma(work[kOffP + i], W * W, acc);
        }
    } else {                                            // a vanishing matter density: the filter may overflow
        for (int i = lane; i < kNk; i += 32) {
            const double W = 1.0 / fma(R6, work[kOffK6 + i], 1.0);
            acc = fma(work[kOffP + i], W * W, acc);
        }
    }
    acc = warp_sum(acc);
    if (lane == 0) work[kOffS2 + m] = acc;
}

// Part 3, one CTA per cosmology: serial only in the spline's elimination (500 rows, in shared memory) and the
// distances' running sum.
__global__ void __launch_bounds__(kThreads) k_cos_out(CosArgs a) {
    __shared__ double lnM[kNm], lns[kNm], sl[kNm], dg[kNm], up[kNm], rhs[kNm], lo_[kNm];
    const int ci = blockIdx.x, t = threadIdx.x;
    const Cos c = make_cos(a.params + 9LL * ci);
    const double* work = a.work + (long long)ci * a.work_stride;
    double s8 = 0.0;
    for (int i = 0; i < kKgridCtas; ++i) s8 += work[kOffS8 + i];
    const double anorm = c.s8 / sqrt(s8 / (2 * M_PI * M_PI));
    for (int m = t; m < kNm; m += kThreads) {
        lnM[m] = log(m == kNm - 1 ? 1e17 : pow(10.0, 4.0 + m * (13.0 / (kNm - 1))));
        lns[m] = log(anorm * sqrt(work[kOffS2 + m] / (2 * M_PI * M_PI)));
    }
    __syncthreads();
    // ---- the not-a-knot spline's slopes: tridiagonal system, forward elimination and back substitution
    constexpr int n = kNm;
    for (int i = 1 + t; i < n - 1; i += kThreads) {
        const double dx0 = lnM[i] - lnM[i - 1], dx1 = lnM[i + 1] - lnM[i];
        const double m0 = (lns[i] - lns[i - 1]) / dx0, m1 = (lns[i + 1] - lns[i]) / dx1;
        lo_[i] = dx1;
        dg[i] = 2 * (dx0 + dx1);
        up[i] = dx0;
        rhs[i] = 3 * (dx1 * m0 + dx0 * m1);
    }
    if (t == 0) {
        const double dx0 = lnM[1] - lnM[0], dx1 = lnM[2] - lnM[1], d = lnM[2] - lnM[0];
        const double m0 = (lns[1] - lns[0]) / dx0, m1 = (lns[2] - lns[1]) / dx1;
        dg[0] = dx1;
        up[0] = d;
        rhs[0] = ((dx0 + 2 * d) * dx1 * m0 + dx0 * dx0 * m1) / d;
    }
    if (t == 32) {
        const double dx0 = lnM[n - 2] - lnM[n - 3], dx1 = lnM[n - 1] - lnM[n - 2], d = lnM[n - 1] - lnM[n - 3];
        const double m0 = (lns[n - 2] - lns[n - 3]) / dx0, m1 = (lns[n - 1] - lns[n - 2]) / dx1;
        dg[n - 1] = dx0;
        lo_[n - 1] = d;
        rhs[n - 1] = (dx1 * dx1 * m0 + (2 * d + dx1) * dx0 * m1) / d;
    }
    __syncthreads();
    if (t == 0) {
        for (int i = 1; i < n; ++i) {
            const double f = lo_[i] / dg[i - 1];
            dg[i] -= f * up[i - 1];
            rhs[i] -= f * rhs[i - 1];
        }
        sl[n - 1] = rhs[n - 1] / dg[n - 1];
        for (int i = n - 2; i >= 0; --i) sl[i] = (rhs[i] - up[i] * sl[i + 1]) / dg[i];
    }
    if (t == 32) {
        double run = 0.0;
        for (int j = 0; j < a.nz; ++j) {
            run += a.chi[(long long)ci * a.nz + j];
            a.chi[(long long)ci * a.nz + j] = run;
        }
    }
    for (int j = t; j < a.nx; j += kThreads) {
        const int slot = a.x_slot[j];
        const double Dv = work[kOffGrow + j] / work[kOffGrow + a.nx];
        if (slot < a.nz) a.D[(long long)ci * a.nz + slot] = Dv;
        else a.Dm[(long long)ci * a.nzm + (slot - a.nz)] = Dv;
    }
    __syncthreads();
    for (int j = t; j < a.nz; j += kThreads) a.DM[(long long)ci * a.nz + j] = cos_fK(c, a.chi[(long long)ci * a.nz + j]);
    // ---- sigma(M), the mass function and the concentration at the output masses
    for (int e2 = t; e2 < a.nm; e2 += kThreads) {
        const double x = log(a.M[e2]);
        int lo = 0, hi = kNm - 2;                       // the spline interval holding x (clamped)
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (lnM[mid] <= x) lo = mid; else hi = mid - 1;
        }
        const double dx = lnM[lo + 1] - lnM[lo];
        const double slope = (lns[lo + 1] - lns[lo]) / dx;
        const double tt = (sl[lo] + sl[lo + 1] - 2 * slope) / dx;
        const double c0 = tt / dx, c1 = (slope - sl[lo]) / dx - tt, c2 = sl[lo], c3 = lns[lo];
        const double u = x - lnM[lo];
        const double lnsig = ((c0 * u + c1) * u + c2) * u + c3;
        const double dls = (3 * c0 * u + 2 * c1) * u + c2;
        const double sig0 = exp(lnsig);
        a.sigM[(long long)ci * a.nm + e2] = sig0;
        a.dlnsig[(long long)ci * a.nm + e2] = dls;
        for (int q = 0; q < a.nzm; ++q) {
            const double zq = a.zm[q];
            const double sig = sig0 * a.Dm[(long long)ci * a.nzm + q];
            const double nu = (kDc / sig) * (kDc / sig);
            const double qn = 0.8 * nu;
            const double mult = a.A_st * (1 + pow(qn, -0.3)) * sqrt(qn / (2 * M_PI)) * exp(-qn / 2);
            a.dndlnM[((long long)ci * a.nzm + q) * a.nm + e2] = (c.rhom / a.M[e2]) * mult * (-2 * dls);
            const double zc = zq > 7.0 ? 7.0 : zq;
            const double ap = 1.0 + zc;
            const double poly = 4.135 - 0.564 * ap - 0.210 * ap * ap + 0.0557 * ap * ap * ap - 0.00348 * ap * ap * ap * ap;
            const double qc = kDc / (sig0 * poly);
            const double cc0 = 3.395 * pow(ap, -0.215), beta = 0.307 * pow(ap, 0.540);
            const double g1 = 0.628 * pow(ap, -0.047), g2 = 0.317 * pow(ap, -0.893);
            a.conc[((long long)ci * a.nzm + q) * a.nm + e2] = cc0 * pow(qc, -g1) * pow(1.0 + pow(qc, 1.0 / beta), -beta * (g2 - g1));
        }
    }
}

}  // namespace

long long cosmo_work_doubles(int nx) { return (kOffGrow + nx + 1LL + 1) & ~1LL; }     // even: read in pairs

void launch_cosmo_tables(int n, const double* params, int nz, const double* z, const double* x_out, const int* x_slot,
                         int nx, int nm, const double* M, int nzm, const double* zm, double A_st, double* E,
                         double* chi, double* DM, double* D, double* Dm, double* sigM, double* dlnsig,
                         double* dndlnM, double* conc, double* work, cudaStream_t st) {
    CosArgs a{params, nz, z, x_out, x_slot, nx, nm, M, nzm, zm, A_st, E, chi, DM, D, Dm, sigM, dlnsig, dndlnM, conc,
              work, cosmo_work_doubles(nx)};
    const int dist_ctas = ceil_div(nz, kPartThreads / 32);
    for (int c0 = 0; c0 < n; c0 += 65535) {                       // cosmologies are the grid's second dimension
        const int nc = std::min(65535, n - c0);
        k_cos_parts<<<dim3(kGrowthCtas + kKgridCtas + dist_ctas, nc), kPartThreads, 0, st>>>(a);
        k_cos_sums<<<dim3(kNodeCtas + 1, nc), kThreads, 0, st>>>(a);
        k_cos_out<<<nc, kThreads, 0, st>>>(a);
        SGL_COUNT(3);
        a.params += 9LL * nc;
        a.E += (long long)nc * nz; a.chi += (long long)nc * nz; a.DM += (long long)nc * nz; a.D += (long long)nc * nz;
        a.Dm += (long long)nc * nzm;
        a.sigM += (long long)nc * nm; a.dlnsig += (long long)nc * nm;
        a.dndlnM += (long long)nc * nzm * nm; a.conc += (long long)nc * nzm * nm;
        a.work += nc * a.work_stride;
    }
}

}  // namespace sgl
