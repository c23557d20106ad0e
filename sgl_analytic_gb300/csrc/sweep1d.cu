// One-dimensional compensated compound-Poisson CF sweep over a large cell list:
//   Lambda(k_n) = sum_c w_c (e^{i k_n kap_c} - 1 - i k_n kap_c)
// (the kappa part of Psi_1, reference _sep_lam_kernel's A1 term, sgl_full.py:2596-2617), for cell
// lists of any size (16.8M cells x 16384 k in the synthetic plane x mass x impact-parameter sweep).
//
// CTA (k tile of 256 rows, cell chunk): each thread owns one k; the chunk's cells stream through
// shared memory in tiles of 512 (coalesced loads, broadcast reads).  FP64 path: FP64 sincos of the
// half angle; mixed path: the packed FP32 terms of cfterm.cuh, Kahan-compensated within the chunk, FP64
// across chunks (fixed order: deterministic).  1.04 M cells x 5003 k: 11.57 -> 4.93 ms per call (4.5e11 -> 1.06e12
// terms/s) with the packed terms.
//
// Also: FMA-throughput probes used as the measured FP64 / FP32 peaks of the CF-sweep roofline.
#include <algorithm>

#include "cfterm.cuh"
#include "kernels.cuh"

namespace sgl {

constexpr int kSwRows = 256;
constexpr int kSwTile = 512;

template <int MODE>
__global__ void __launch_bounds__(kSwRows)
k_sweep1d(const double* __restrict__ kk, int nk, const double* __restrict__ kap, const double* __restrict__ w,
          const float* __restrict__ kh, const float* __restrict__ kl, const float* __restrict__ wf,
          long long nc, long long per_chunk, double2* __restrict__ part) {
    __shared__ double s_k[MODE == SGL_FP64 ? kSwTile : 1];
    __shared__ double s_w[MODE == SGL_FP64 ? kSwTile : 1];
    __shared__ __align__(16) float s_f[3][MODE == SGL_FP64 ? 4 : kSwTile];     // kappa head, kappa tail, w
    const int n = blockIdx.x * kSwRows + threadIdx.x;
    const double k = n < nk ? kk[n] : 0.0;
    const CfWave kf(k);
    __shared__ unsigned s_khm;                                  // the CTA's largest half wave number (float bits)
    if (threadIdx.x == 0) s_khm = 0u;
    __syncthreads();
    if (MODE != SGL_FP64) atomicMax(&s_khm, __float_as_uint(0.5f * fabsf((float)k)));
    __syncthreads();
    const float khm = __uint_as_float(s_khm);
    const long long c0 = (long long)blockIdx.y * per_chunk;
    const long long c1 = c0 + per_chunk < nc ? c0 + per_chunk : nc;
    double ar = 0.0, ai = 0.0;
    CfSums S;
    S.clear();
    for (long long base = c0; base < c1; base += kSwTile) {
        const int cnt = (int)((c1 - base) < kSwTile ? (c1 - base) : kSwTile);
        __syncthreads();
        bool big = false;
        const int cnt8 = (cnt + kCfGroup - 1) / kCfGroup * kCfGroup;
        for (int e = threadIdx.x; e < (MODE == SGL_FP64 ? cnt : cnt8); e += kSwRows) {
            if (MODE == SGL_FP64) { s_k[e] = kap[base + e]; s_w[e] = w[base + e]; }
            else {
                const bool in = e < cnt;
                s_f[0][e] = in ? kh[base + e] : 0.f;
                s_f[1][e] = in ? kl[base + e] : 0.f;
                s_f[2][e] = in ? wf[base + e] : 0.f;
                big |= fabsf(s_f[0][e]) * khm > kCfBigHalfPhase;
            }
        }
        big = __syncthreads_or(big);
        if (MODE == SGL_FP64) {
            for (int e = 0; e < cnt; ++e) {
                const double ph = k * s_k[e];
                double s, c;
                sincos(0.5 * ph, &s, &c);
                const double cm1 = -2.0 * s * s;
                double smp;
                if (fabs(ph) < 1e-2) {
                    const double p2 = ph * ph;
                    smp = -ph * p2 / 6.0 * (1.0 - p2 / 20.0 * (1.0 - p2 / 42.0));
                } else {
                    smp = 2.0 * s * c - ph;
                }
                ar = fma(s_w[e], cm1, ar);
                ai = fma(s_w[e], smp, ai);
            }
        } else {
            if (big) cf_tile<true>(kf, s_f[0], s_f[1], s_f[2], cnt8, S);
            else cf_tile<false>(kf, s_f[0], s_f[1], s_f[2], cnt8, S);
        }
    }
    if (n < nk) {
        if (MODE == SGL_FP64) part[(long long)blockIdx.y * nk + n] = make_double2(ar, ai);
        else part[(long long)blockIdx.y * nk + n] = S.value();
    }
}

__global__ void k_sweep1d_reduce(const double2* __restrict__ part, int nchunks, int nk, double* __restrict__ re,
                                 double* __restrict__ im) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= nk) return;
    double r = 0.0, i = 0.0;
    for (int c = 0; c < nchunks; ++c) { const double2 v = part[(long long)c * nk + n]; r += v.x; i += v.y; }
    re[n] = r;
    im[n] = i;
}

int sweep1d_chunks(int precision, int nk, long long nc) {
    // At least 4 CTAs per SM over (k tiles x chunks), down to chunks of one tile of cells: few cells at few k need every
    // CTA (FP64, 16384 cells x 100 k: 32 chunks of a tile 3.1 ms, 8 of four 12.2).  Mixed: up to 32 CTAs per SM, about 8
    // waves of 4 resident CTAs, so that the last, partly filled wave costs little, of no less than 4 tiles.
    const long long ktiles = ceil_div(nk, kSwRows);
    auto chunks = [&](long long per_sm, long long tiles) {
        return std::min((per_sm * kNumSMs + ktiles - 1) / ktiles, (nc + tiles * kSwTile - 1) / (tiles * kSwTile));
    };
    long long nch = chunks(4, 1);
    if (precision != SGL_FP64) nch = std::max(nch, chunks(32, 4));
    return (int)std::max(1LL, nch);
}

void launch_sweep1d(int precision, const double* kk, int nk, const double* kap, const double* w, const float* kh,
                    const float* kl, const float* wf, long long nc, int nchunks, double2* part, double* re,
                    double* im, cudaStream_t st) {
    const long long per = (nc + nchunks - 1) / nchunks;
    dim3 grid(ceil_div(nk, kSwRows), nchunks);
    if (precision == SGL_FP64) { k_sweep1d<SGL_FP64><<<grid, kSwRows, 0, st>>>(kk, nk, kap, w, kh, kl, wf, nc, per, part); SGL_COUNT(1); }
    else { k_sweep1d<SGL_MIXED><<<grid, kSwRows, 0, st>>>(kk, nk, kap, w, kh, kl, wf, nc, per, part); SGL_COUNT(1); }
    { k_sweep1d_reduce<<<ceil_div(nk, 256), 256, 0, st>>>(part, nchunks, nk, re, im); SGL_COUNT(1); }
}

// ------------------------------------------------------------------ FMA throughput probes
// 8 independent FMA chains per thread, iters iterations; the result is stored so nothing is elided.
template <typename T>
__global__ void __launch_bounds__(256) k_fma_probe(T* out, int iters, T seed) {
    T a[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) a[j] = seed + (T)(threadIdx.x + j);
    const T m = (T)0.999999, c = (T)1e-7;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = fma(a[j], m, c);
    }
    T s = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) s += a[j];
    out[blockIdx.x * blockDim.x + threadIdx.x] = s;
}

void launch_fma_probe(int fp64, void* out, int blocks, int iters, cudaStream_t st) {
    if (fp64) { k_fma_probe<double><<<blocks, 256, 0, st>>>((double*)out, iters, 1.0); SGL_COUNT(1); }
    else { k_fma_probe<float><<<blocks, 256, 0, st>>>((float*)out, iters, 1.f); SGL_COUNT(1); }
}

}  // namespace sgl
