// Positive (vp) Cox closure: ln R(k, q) = ln E_U exp( sum_s z_s(U_s; k, q) ),
//   z_s(u_j) = sum_{g in shell s} D_g(u_j) Y_g,   Y_g = sum_{c in g} w_c F_c,
//   F_c(k, q) = e_c J_c + J_c - 1,  e = expm1(i k kap_c), J = J0(q gam_c)
// (reference: FusedVP.lnR_blocked pos_closure_fused.py:119-140 = _fused_groups :51-105 +
//  _chain_recursion pos_closure.py:184-240).
//
// D_g(u) = lam_g(u) - 1 is, per group, c + a (u - anchor) + b on an interval of states that reaches
// an end of the state grid (rate_intervals pos_closure_fused.py:18-48), and E_w[D_g] = 0 exactly
// (the rates keep the mean, pos_closure.py:15).  The host sorts each shell's groups into RUNS of
// one kind and one interval bound (linear; "left" = states lo..47; "right" = states 0..hi) and
// stores per-cell weights (w a, w b).  Then
//   z_s(u_j) = u_j A_lin + sum_{left runs, lo <= j} [(u_j - u_lo) A_r + B_r]
//            + sum_{right runs, j <= hi} [(u_j - u_hi) A_r + B_r] + const,
//   A_r = sum_{c in r} (w a)_c F_c,  B_r = sum_{c in r} (w b)_c F_c.
// The constant (c = -1 offsets, linear intercepts) is not formed: z_s has zero stationary mean, so
// z_s = z_partial - E_w[z_partial] exactly, and that projection also removes the common-mode part
// of the rounding error (what keeps the mixed path within 1e-8 of FP64).
//
// Phase 1 (k_vp_z; on a grid of points in mixed precision k_vp_z_mixed, below): one CTA per (shell, 16 k x 32 q tile); each thread owns 2 x 2 points.  Cells of
// a run stream through shared memory in chunks of 32 (table rows e[u][k], (J, J - 1)[u][q] gathered
// by cell index, coalesced along k / q); per point 4 FMAs + 2 for F.  Mixed: FP32 chunk sums folded
// into float-float run totals (TwoSum); FP64: FP64 throughout.  Run totals go to FP64 running sums
// over the sorted bounds and each state's z is written once (FP64, [shell][state][point]).
// Phase 2 (k_vp_chain): one thread per point walks the shells: projection, alpha' = K^T alpha (or the
// stationary weights at s = 0) times exp(z - max Re z), renormalisation by max |alpha|, log scale;
// FP64, thread-private shared memory, no barriers.  The mixed path's chain (k_vp_chain_ff) is the same recursion in
// float-float; points where its range could tell are done over by k_vp_chain.
#include "kernels.cuh"

namespace sgl {

constexpr int kVpNS = 48;                 // latent states (Gauss-Hermite nodes)
constexpr int kZK = 16, kZQ = 32;         // phase-1 point tile (k x q)
constexpr int kZThreads = 128;            // 2 x 2 points per thread
constexpr int kZCh = 32;                  // cells per staged chunk
constexpr int kChPts = 56;                // phase-2 points per CTA (2 CTAs per SM with K staged)

template <typename TT> struct V2;
template <> struct V2<float> { using T = float2; };
template <> struct V2<double> { using T = double2; };

// e[u][i] = (cos - 1, sin)(k_i kap_u) from the half angle (no cancellation); Jt[u][j] = (J0, J0 - 1)
template <typename TT>
__global__ void k_vp_tables(const double* __restrict__ ku, const double* __restrict__ gu, int U,
                            const double* __restrict__ kv, int nk, const double* __restrict__ qv, int nq,
                            typename V2<TT>::T* __restrict__ e, typename V2<TT>::T* __restrict__ Jt) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long ne = (long long)U * nk;
    if (t < ne) {
        const int u = (int)(t / nk), i = (int)(t % nk);
        const double ph = kv[i] * ku[u];
        double s, c;
        sincos(0.5 * ph, &s, &c);
        e[t].x = (TT)(-2.0 * s * s);
        e[t].y = (TT)(2.0 * s * c);
    } else if (t < ne + (long long)U * nq) {
        const long long r = t - ne;
        const int u = (int)(r / nq), j = (int)(r % nq);
        const double jm = j0m1_d(qv[j] * gu[u]);
        Jt[r].x = (TT)(1.0 + jm);
        Jt[r].y = (TT)jm;
    }
}

__device__ __forceinline__ unsigned long long vz_add(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long vz_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// hi + lo += p  (Knuth TwoSum; no FMA contraction applies to additions)
__device__ __forceinline__ void ff_acc(float& hi, float& lo, float p) {
    const float s = hi + p;
    const float bb = s - hi;
    const float err = (hi - (s - bb)) + (p - bb);
    hi = s;
    lo += err;
}

// asynchronous global -> shared copies (zero-filled when !pred; the source address is then unused)
template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem, const void* gmem, bool pred) {
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(smem);
    const int n = pred ? BYTES : 0;
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(sa), "l"(gmem), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" :: "r"(sa), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

template <typename TT>
__global__ void __launch_bounds__(kZThreads)
k_vp_z(VpDevice d, const typename V2<TT>::T* __restrict__ e, const typename V2<TT>::T* __restrict__ Jt, int nk,
       int nq, int kb, int nkc, double2* __restrict__ zp, double2* __restrict__ alin, long long NP, int npieces) {
    using T2 = typename V2<TT>::T;
    __shared__ __align__(16) T2 s_e[2][kZCh][kZK];
    __shared__ __align__(16) T2 s_J[2][kZCh][kZQ];
    __shared__ __align__(16) T2 s_w[2][kZCh];
    constexpr bool MIX = sizeof(TT) == 4;
    constexpr int EB = (int)sizeof(T2);
    // blockIdx.z = (shell, piece): a piece is a contiguous part of the shell's run list.  Each run's
    // contribution to the states is additive, so pieces write partial z and A_lin (their own
    // slices of zp / alin) that the chain kernel sums in piece order.  More than one piece only
    // when the point tile grid alone would leave the GPU idle (the k-reach probes).
    const int s = blockIdx.z / npieces, piece = blockIdx.z % npieces;
    zp += (long long)piece * d.nsh * kVpNS * NP;
    alin += (long long)piece * d.nsh * NP;
    const int q0 = blockIdx.x * kZQ, k0 = kb + blockIdx.y * kZK, kend = kb + nkc;
    const int t = threadIdx.x, tq = t % 16, tk = t / 16;
    // my points: (k0 + tk + 8 m, q0 + tq + 16 i), index P = 2 m + i
    double SAr[4], SAi[4], SBr[4], SBi[4], ALr[4], ALi[4];
#pragma unroll
    for (int P = 0; P < 4; ++P) { SAr[P] = SAi[P] = SBr[P] = SBi[P] = ALr[P] = ALi[P] = 0.0; }
    long long pidx[4];
    bool live[4];
#pragma unroll
    for (int P = 0; P < 4; ++P) {
        const int k = k0 + tk + 8 * (P >> 1), q = q0 + tq + 16 * (P & 1);
        live[P] = k < kend && q < nq;
        pidx[P] = (long long)(k - kb) * nq + q;
    }
    int jcur = 0;
    auto emit_to = [&](int jend) {
        for (; jcur < jend; ++jcur) {
            const double uj = d.u[jcur];
            double2* row = zp + ((long long)s * kVpNS + jcur) * NP;
#pragma unroll
            for (int P = 0; P < 4; ++P)
                if (live[P]) row[pidx[P]] = make_double2(fma(uj, SAr[P], SBr[P]), fma(uj, SAi[P], SBi[P]));
        }
    };
    // chunks of <= 32 cells never straddle a run; the next chunk is copied (cp.async) into the other
    // buffer while the current one is summed
    auto issue = [&](int buf, long long base, long long c1) {
        const int cnt = (int)((c1 - base) < kZCh ? (c1 - base) : kZCh);
        for (int idx = t; idx < kZCh * kZK; idx += kZThreads) {
            const int c = idx / kZK, rr = idx % kZK, k = k0 + rr;
            const bool ok = c < cnt && k < kend;
            cp_async<EB>(&s_e[buf][c][rr], ok ? (const void*)(e + (long long)d.cu[base + c] * nk + k) : (const void*)e, ok);
        }
        for (int idx = t; idx < kZCh * kZQ; idx += kZThreads) {
            const int c = idx / kZQ, rr = idx % kZQ, q = q0 + rr;
            const bool ok = c < cnt && q < nq;
            cp_async<EB>(&s_J[buf][c][rr], ok ? (const void*)(Jt + (long long)d.cu[base + c] * nq + q) : (const void*)Jt, ok);
        }
        if (t < kZCh) {
            const bool ok = t < cnt;
            if constexpr (MIX) cp_async<EB>(&s_w[buf][t], ok ? (const void*)(d.wabf + base + t) : (const void*)d.wabf, ok);
            else cp_async<EB>(&s_w[buf][t], ok ? (const void*)(d.wab + base + t) : (const void*)d.wab, ok);
        }
        cp_async_commit();
    };
    const int rs0 = d.sh_run[s], rs1 = d.sh_run[s + 1];
    const int r0 = rs0 + (int)((long long)(rs1 - rs0) * piece / npieces);
    const int r1 = rs0 + (int)((long long)(rs1 - rs0) * (piece + 1) / npieces);
    int buf = 0;
    if (r0 < r1) issue(0, d.run_cell[r0], d.run_cell[r0 + 1]);
    for (int r = r0; r < r1; ++r) {
        const long long c0 = d.run_cell[r], c1 = d.run_cell[r + 1];
        // run totals: mixed = float-float (hi, lo), FP64 = plain
        TT hi[4][4], lo[4][4];
#pragma unroll
        for (int P = 0; P < 4; ++P)
#pragma unroll
            for (int v = 0; v < 4; ++v) { hi[P][v] = TT(0); lo[P][v] = TT(0); }
        for (long long base = c0; base < c1; base += kZCh) {
            const int cnt = (int)((c1 - base) < kZCh ? (c1 - base) : kZCh);
            // prefetch the next chunk (this run's, or the next run's first)
            const long long nb = base + kZCh;
            const bool has_next = nb < c1 || r + 1 < r1;
            if (has_next) {
                if (nb < c1) issue(buf ^ 1, nb, c1);
                else issue(buf ^ 1, d.run_cell[r + 1], d.run_cell[r + 2]);
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncthreads();
            TT p[4][4];
#pragma unroll
            for (int P = 0; P < 4; ++P)
#pragma unroll
                for (int v = 0; v < 4; ++v) p[P][v] = TT(0);
            for (int c = 0; c < cnt; ++c) {
                const T2 wv = s_w[buf][c];
                const T2 ev[2] = {s_e[buf][c][tk], s_e[buf][c][tk + 8]};
                const T2 jv[2] = {s_J[buf][c][tq], s_J[buf][c][tq + 16]};
#pragma unroll
                for (int P = 0; P < 4; ++P) {
                    const T2 ee = ev[P >> 1], jj = jv[P & 1];
                    const TT Fr = ee.x * jj.x + jj.y;          // (cos - 1) J + (J - 1)
                    const TT Fi = ee.y * jj.x;                 // sin J
                    p[P][0] += wv.x * Fr; p[P][1] += wv.x * Fi;
                    p[P][2] += wv.y * Fr; p[P][3] += wv.y * Fi;
                }
            }
#pragma unroll
            for (int P = 0; P < 4; ++P)
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    if constexpr (MIX) ff_acc(hi[P][v], lo[P][v], p[P][v]);
                    else hi[P][v] += p[P][v];
                }
            __syncthreads();                  // buffer `buf` is refilled by the next prefetch
            buf ^= 1;
        }
        const int kind = d.run_kind[r], bound = d.run_bound[r];
        if (kind == 0) {                                   // linear: u_j A (intercept dropped)
#pragma unroll
            for (int P = 0; P < 4; ++P) {
                ALr[P] += (double)hi[P][0] + (double)lo[P][0];
                ALi[P] += (double)hi[P][1] + (double)lo[P][1];
            }
        } else if (kind == 1) {                            // left: states >= lo, anchored at u_lo
            emit_to(bound);
            const double ub = d.u[bound];
#pragma unroll
            for (int P = 0; P < 4; ++P) {
                const double Ar = (double)hi[P][0] + (double)lo[P][0], Ai = (double)hi[P][1] + (double)lo[P][1];
                const double Br = (double)hi[P][2] + (double)lo[P][2], Bi = (double)hi[P][3] + (double)lo[P][3];
                SAr[P] += Ar; SAi[P] += Ai;
                SBr[P] += fma(-ub, Ar, Br); SBi[P] += fma(-ub, Ai, Bi);
            }
        } else {                                           // right: states <= hi, anchored at u_hi
            // = u_j A on every state (+ a dropped constant) minus [(u_j - u_hi) A + B] on states > hi
            emit_to(bound + 1);
            const double ub = d.u[bound];
#pragma unroll
            for (int P = 0; P < 4; ++P) {
                const double Ar = (double)hi[P][0] + (double)lo[P][0], Ai = (double)hi[P][1] + (double)lo[P][1];
                const double Br = (double)hi[P][2] + (double)lo[P][2], Bi = (double)hi[P][3] + (double)lo[P][3];
                ALr[P] += Ar; ALi[P] += Ai;
                SAr[P] -= Ar; SAi[P] -= Ai;
                SBr[P] += fma(ub, Ar, -Br); SBi[P] += fma(ub, Ai, -Bi);
            }
        }
    }
    emit_to(kVpNS);
#pragma unroll
    for (int P = 0; P < 4; ++P)
        if (live[P]) alin[(long long)s * NP + pidx[P]] = make_double2(ALr[P], ALi[P]);
}

// ---- phase 1 of the mixed path on a line of points (the k-reach probes)
// A warp takes a piece of a shell's cells for 32 points, a point per lane: cell indices and weights read 32 at a time and
// broadcast, the table entries of eight cells in flight; sums as in k_vp_z (FP32 over 32 cells of a run, float-float over
// the run, FP64 over the bounds).  Bound by the latency of the gathers from L2.  k_vp_z's 16 x 32 tiles hold a column or
// a row of such points: 20 points, 0.77 M cells 0.84 and 0.75 -> 0.13 ms.
constexpr int kZlThreads = 128;

__global__ void __launch_bounds__(kZlThreads)
k_vp_z_line(VpDevice d, const float2* __restrict__ e, const float2* __restrict__ Jt, int nk, int nq, int kb,
            double2* __restrict__ zp, double2* __restrict__ alin, long long NP, int npieces) {
    const int lane = threadIdx.x & 31, g = blockIdx.y * (kZlThreads / 32) + (threadIdx.x >> 5);
    if (g >= d.nsh * npieces) return;
    const int s = g / npieces, piece = g % npieces;
    zp += (long long)piece * d.nsh * kVpNS * NP;
    alin += (long long)piece * d.nsh * NP;
    const long long p = (long long)blockIdx.x * 32 + lane;
    const bool live = p < NP;
    const int pp = live ? (int)p : 0;
    const float2* ek = e + kb + pp / nq;                     // kb: first row of the pass
    const float2* jq = Jt + pp % nq;
    double SAr = 0.0, SAi = 0.0, SBr = 0.0, SBi = 0.0, ALr = 0.0, ALi = 0.0;
    int jcur = 0;
    auto emit_to = [&](int jend) {
        for (; jcur < jend; ++jcur) {
            const double uj = d.u[jcur];
            if (live) zp[((long long)s * kVpNS + jcur) * NP + p] = make_double2(fma(uj, SAr, SBr), fma(uj, SAi, SBi));
        }
    };
    // an equal part of the shell's cells (a run may span pieces: its contribution is additive), cut at 32 cells
    const int rs0 = d.sh_run[s], rs1 = d.sh_run[s + 1];
    const long long sc0 = d.run_cell[rs0], sn = d.run_cell[rs1] - sc0;
    const long long cb = sc0 + sn * piece / npieces, ce = sc0 + sn * (piece + 1) / npieces;
    int r0 = rs0, hi_r = rs1;                                // the run that holds cb
    while (hi_r - r0 > 1) {
        const int mid = (r0 + hi_r) >> 1;
        if (d.run_cell[mid] <= cb) r0 = mid; else hi_r = mid;
    }
    for (int r = r0; r < rs1; ++r) {
        const long long rc = d.run_cell[r], c0 = max(cb, rc), c1 = min(ce, d.run_cell[r + 1]);
        if (rc >= ce) break;
        if (c0 >= c1) continue;
        float hi[4] = {0.f, 0.f, 0.f, 0.f}, lo[4] = {0.f, 0.f, 0.f, 0.f};
        for (long long base = c0; base < c1; base += 32) {
            const int cnt = (int)min(32LL, c1 - base);
            const int cu = lane < cnt ? d.cu[base + lane] : 0;
            const float2 w = lane < cnt ? d.wabf[base + lane] : make_float2(0.f, 0.f);
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            for (int b = 0; b < cnt; b += 8) {
                float2 ev[8], jv[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const long long c = __shfl_sync(0xffffffffu, cu, b + i);      // (0 beyond the run's cells)
                    ev[i] = __ldg(ek + c * nk);
                    jv[i] = __ldg(jq + c * nq);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (b + i >= cnt) break;
                    const float wa = __shfl_sync(0xffffffffu, w.x, b + i), wb = __shfl_sync(0xffffffffu, w.y, b + i);
                    const float Fr = ev[i].x * jv[i].x + jv[i].y;                 // (cos - 1) J + (J - 1)
                    const float Fi = ev[i].y * jv[i].x;                           // sin J
                    v[0] += wa * Fr; v[1] += wa * Fi;
                    v[2] += wb * Fr; v[3] += wb * Fi;
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) ff_acc(hi[i], lo[i], v[i]);
        }
        const double Ar = (double)hi[0] + (double)lo[0], Ai = (double)hi[1] + (double)lo[1];
        const double Br = (double)hi[2] + (double)lo[2], Bi = (double)hi[3] + (double)lo[3];
        const int kind = d.run_kind[r], bound = d.run_bound[r];
        if (kind == 0) {                                   // linear: u_j A (intercept dropped)
            ALr += Ar; ALi += Ai;
        } else if (kind == 1) {                            // left: states >= lo, anchored at u_lo
            emit_to(bound);
            const double ub = d.u[bound];
            SAr += Ar; SAi += Ai;
            SBr += fma(-ub, Ar, Br); SBi += fma(-ub, Ai, Bi);
        } else {                                           // right: states <= hi, anchored at u_hi (as in k_vp_z)
            emit_to(bound + 1);
            const double ub = d.u[bound];
            ALr += Ar; ALi += Ai;
            SAr -= Ar; SAi -= Ai;
            SBr += fma(ub, Ar, -Br); SBi += fma(ub, Ai, -Bi);
        }
    }
    emit_to(kVpNS);
    if (live) alin[(long long)s * NP + p] = make_double2(ALr, ALi);
}

// ---- phase 1 of the mixed path on a grid of points
// F splits into e_c(k) J_c(q), of both axes, and J_c(q) - 1, of k_gamma alone: the second part of every run is summed
// once per q (k_vp_jm), and per (cell, point) only two packed FMAs remain, J times (w a e_re, w a e_im) and
// (w b e_re, w b e_im), the four products formed once per (cell, k) while staging (k_vp_z forms F and needs six scalar
// ones).  CTA: 16 k x 112 q of one shell (or a piece of its runs), 2 k x 7 q per thread, so that a cell costs a warp five
// shared-memory reads to 28 FMAs; FP32 sums over 32 cells, compensated (Kahan) over the run; the sums over the sorted
// bounds live in local memory, touched once per run.  Bound by the FP32 pipe; 409 x 109 points, 0.77 M cells:
// 21.9 -> 9.1 ms (issue 50% active, two warps per scheduler: the 56 pairs of compensated sums take 112 registers).
constexpr int kMzK = 16, kMzQ = 112, kMzThreads = 128, kMzCh = 32;

// J0 and J0 - 1 per unique cell with rows padded to whole q tiles (zeros), e as in k_vp_tables
__global__ void k_vp_tables_mixed(const double* __restrict__ ku, const double* __restrict__ gu, int U,
                                  const double* __restrict__ kv, int nk, const double* __restrict__ qv, int nq, int nqp,
                                  float2* __restrict__ e, float* __restrict__ J, float* __restrict__ Jm) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long ne = (long long)U * nk;
    if (t < ne) {
        const int u = (int)(t / nk), i = (int)(t % nk);
        const double ph = kv[i] * ku[u];
        double s, c;
        sincos(0.5 * ph, &s, &c);
        e[t] = make_float2((float)(-2.0 * s * s), (float)(2.0 * s * c));
    } else if (t < ne + (long long)U * nqp) {
        const long long r = t - ne;
        const int u = (int)(r / nqp), j = (int)(r % nqp);
        const double jm = j < nq ? j0m1_d(qv[j] * gu[u]) : -1.0;
        J[r] = (float)(1.0 + jm);
        Jm[r] = j < nq ? (float)jm : 0.f;
    }
}

// per run, part of its cells and q: sum_c (w a, w b)_c (J_c(q) - 1), FP32 over 32 cells, FP64 over the part; then the
// parts in order
constexpr int kJmParts = 16;
__global__ void __launch_bounds__(128) k_vp_jm(VpDevice d, const float* __restrict__ Jm, int nqp, double2* __restrict__ part) {
    const int r = blockIdx.x, q = blockIdx.z * 128 + threadIdx.x;
    if (q >= nqp) return;
    const long long n0 = d.run_cell[r], n1 = d.run_cell[r + 1];
    const long long per = ((n1 - n0 + kJmParts - 1) / kJmParts + 31) / 32 * 32;
    const long long c0 = min(n1, n0 + blockIdx.y * per), c1 = min(n1, c0 + per);
    double a = 0.0, b = 0.0;
    for (long long base = c0; base < c1; base += 32) {
        const int cnt = (int)min(32LL, c1 - base);
        float pa = 0.f, pb = 0.f;
#pragma unroll 8
        for (int c = 0; c < cnt; ++c) {
            const float2 w = d.wabf[base + c];
            const float j = Jm[(long long)d.cu[base + c] * nqp + q];
            pa = fmaf(w.x, j, pa);
            pb = fmaf(w.y, j, pb);
        }
        a += (double)pa;
        b += (double)pb;
    }
    part[((long long)blockIdx.y * d.nruns + r) * nqp + q] = make_double2(a, b);
}

__global__ void k_vp_jm_sum(const double2* __restrict__ part, long long n, double2* __restrict__ out) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    double a = 0.0, b = 0.0;
    for (int p = 0; p < kJmParts; ++p) { const double2 v = part[p * n + e]; a += v.x; b += v.y; }
    out[e] = make_double2(a, b);
}

__global__ void __launch_bounds__(kMzThreads, 2)
k_vp_z_mixed(VpDevice d, const float2* __restrict__ e, const float* __restrict__ J, const double2* __restrict__ jm, int nk,
             int nq, int nqp, int kb, int nkc, double2* __restrict__ zp, double2* __restrict__ alin, long long NP, int npieces) {
    __shared__ __align__(16) float s_J[2][kMzCh][kMzQ];
    __shared__ __align__(16) float4 s_we[2][kMzCh][kMzK];
    __shared__ int s_cu[4][kMzCh];             // unique-cell indices, two chunks ahead of the sums
    const int s = blockIdx.z / npieces, piece = blockIdx.z % npieces;
    zp += (long long)piece * d.nsh * kVpNS * NP;
    alin += (long long)piece * d.nsh * NP;
    const int q0 = blockIdx.x * kMzQ, k0 = kb + blockIdx.y * kMzK, kend = kb + nkc;
    const int t = threadIdx.x, lane = t & 31, tq = lane & 15;
    const int kl = (t >> 5) * 4 + (lane >> 4) * 2;                        // the thread's k: k0 + kl, + 1
    // its q: q0 + 4 tq + 0..3, 64 + 2 tq + 0..1, 96 + tq
    auto q_of = [&](int i) { return q0 + (i < 4 ? 4 * tq + i : (i < 6 ? 64 + 2 * tq + (i - 4) : 96 + tq)); };
    // sums over the bounds (A, B anchored at 0, linear A; re, im) in local memory: the opaque offset keeps them there
    double st[14][6];
    int z;
    asm volatile("mov.u32 %0, 0;" : "=r"(z));
#pragma unroll 1
    for (int P = 0; P < 14; ++P)
#pragma unroll 1
        for (int v = 0; v < 6; ++v) st[P + z][v + z] = 0.0;
    int jcur = 0;
    auto emit_to = [&](int jend) {
        for (; jcur < jend; ++jcur) {
            const double uj = d.u[jcur];
            double2* row = zp + ((long long)s * kVpNS + jcur) * NP;
#pragma unroll 1
            for (int P = 0; P < 14; ++P) {
                const int k = k0 + kl + P / 7, q = q_of(P % 7);
                const double* a = st[P + z];
                if (k < kend && q < nq)
                    row[(long long)(k - kb) * nq + q] = make_double2(fma(uj, a[0], a[2]), fma(uj, a[1], a[3]));
            }
        }
    };
    // the piece's cells: an equal part of the shell's (a run may span pieces: its contribution is additive), and the runs
    // that hold them
    const int rs0 = d.sh_run[s], rs1 = d.sh_run[s + 1];
    const long long sc0 = d.run_cell[rs0], sn = d.run_cell[rs1] - sc0;
    const long long cb = sc0 + sn * piece / npieces, ce = sc0 + sn * (piece + 1) / npieces;
    int r0 = rs0, r1 = rs1;
    while (r0 < r1 && d.run_cell[r0 + 1] <= cb) ++r0;
    while (r1 > r0 && d.run_cell[r1 - 1] >= ce) --r1;
    auto first = [&](int r) { return max(cb, d.run_cell[r]); };
    auto end = [&](int r) { return min(ce, d.run_cell[r + 1]); };
    // chunks of at most 32 cells that never straddle a run; (r, base) of the chunk after a given one
    auto next = [&](int& r, long long& base) {
        base += kMzCh;
        if (base >= end(r) && ++r < r1) base = first(r);
    };
    // staging: the indices of a chunk's cells (slot), then, one chunk later, its J by asynchronous 16-byte copies and its
    // e and weights into registers, whose products `place` writes
    auto fetch_cu = [&](int slot, int r, long long base) {
        if (r < r1 && t < kMzCh) {
            const bool ok = base + t < end(r);
            const uint32_t sa = (uint32_t)__cvta_generic_to_shared(&s_cu[slot][t]);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"(sa), "l"(ok ? d.cu + base + t : d.cu), "r"(ok ? 4 : 0) : "memory");
        }
    };
    float2 pe[4], pw[4];
    auto fetch = [&](int buf, int slot, int r, long long base) {
        const int cnt = (int)min((long long)kMzCh, end(r) - base);
#pragma unroll
        for (int x = 0; x < kMzCh * kMzQ / 4 / kMzThreads; ++x) {
            const int idx = t + x * kMzThreads, c = idx / (kMzQ / 4), o = (idx % (kMzQ / 4)) * 4;
            const bool ok = c < cnt;
            cp_async<16>(&s_J[buf][c][o], ok ? (const void*)(J + (long long)s_cu[slot][c] * nqp + q0 + o) : (const void*)J, ok);
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int idx = t + x * kMzThreads, c = idx / kMzK, k = k0 + idx % kMzK;
            const bool ok = c < cnt && k < kend;
            pe[x] = ok ? e[(long long)s_cu[slot][c] * nk + k] : make_float2(0.f, 0.f);
            pw[x] = ok ? d.wabf[base + c] : make_float2(0.f, 0.f);
        }
    };
    auto place = [&](int buf) {
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int idx = t + x * kMzThreads;
            s_we[buf][idx / kMzK][idx % kMzK] =
                make_float4(pw[x].x * pe[x].x, pw[x].x * pe[x].y, pw[x].y * pe[x].x, pw[x].y * pe[x].y);
        }
    };
    const unsigned long long m1 = f32x2_pack(-1.f, -1.f);
    int buf = 0, slot = 0;                     // the chunk being summed: its buffers, its slot of s_cu
    int rn = r0, r2 = r0;                      // the next chunk, and the one after it
    long long bn = 0, b2 = 0;
    if (r0 < r1) {
        bn = b2 = first(r0);
        fetch_cu(0, r0, bn);
        next(r2, b2);
        fetch_cu(1, r2, b2);
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        fetch(0, 0, r0, bn);
        cp_async_commit();
        place(0);
        cp_async_wait<0>();
        __syncthreads();
        rn = r2; bn = b2;
    }
    for (int r = r0; r < r1; ++r) {
        const long long c0 = first(r), c1 = end(r);
        unsigned long long hi[2][7][2], lo[2][7][2];                       // (k, q, a or b): (re, im), value hi - lo
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int i = 0; i < 7; ++i)
#pragma unroll
                for (int v = 0; v < 2; ++v) { hi[x][i][v] = 0ull; lo[x][i][v] = 0ull; }
        for (long long base = c0; base < c1; base += kMzCh) {
            const int cnt = (int)min((long long)kMzCh, c1 - base);
            const bool more = rn < r1;
            if (more) {
                fetch(buf ^ 1, (slot + 1) & 3, rn, bn);
                r2 = rn; b2 = bn;
                next(r2, b2);
                fetch_cu((slot + 2) & 3, r2, b2);
                cp_async_commit();
            }
            unsigned long long p[2][7][2];
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int i = 0; i < 7; ++i)
#pragma unroll
                    for (int v = 0; v < 2; ++v) p[x][i][v] = 0ull;
#pragma unroll 2
            for (int c = 0; c < cnt; ++c) {
                const float4 j4 = *reinterpret_cast<const float4*>(&s_J[buf][c][4 * tq]);
                const float2 j2 = *reinterpret_cast<const float2*>(&s_J[buf][c][64 + 2 * tq]);
                const float jv[7] = {j4.x, j4.y, j4.z, j4.w, j2.x, j2.y, s_J[buf][c][96 + tq]};
                const float4 w0 = s_we[buf][c][kl], w1 = s_we[buf][c][kl + 1];
                const unsigned long long wv[2][2] = {{f32x2_pack(w0.x, w0.y), f32x2_pack(w0.z, w0.w)},
                                                     {f32x2_pack(w1.x, w1.y), f32x2_pack(w1.z, w1.w)}};
#pragma unroll
                for (int i = 0; i < 7; ++i) {
                    const unsigned long long j = f32x2_pack(jv[i], jv[i]);
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        f32x2_fma(p[x][i][0], j, wv[x][0]);
                        f32x2_fma(p[x][i][1], j, wv[x][1]);
                    }
                }
            }
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int i = 0; i < 7; ++i)
#pragma unroll
                    for (int v = 0; v < 2; ++v) {
                        // Kahan: y = p - lo, sum = hi + y, lo = (sum - hi) - y
                        const unsigned long long y = vz_fma(lo[x][i][v], m1, p[x][i][v]);
                        const unsigned long long sum = vz_add(hi[x][i][v], y);
                        lo[x][i][v] = vz_fma(y, m1, vz_fma(hi[x][i][v], m1, sum));
                        hi[x][i][v] = sum;
                    }
            if (more) {
                place(buf ^ 1);
                cp_async_wait<0>();
            }
            __syncthreads();
            buf ^= 1;
            slot = (slot + 1) & 3;
            rn = r2; bn = b2;
        }
        const int kind = d.run_kind[r], bound = d.run_bound[r];
        const double ub = d.u[bound];
        const bool whole = c0 == d.run_cell[r];            // the piece with the run's first cell adds its J - 1 sums
        if (kind == 1) emit_to(bound);                     // left: states >= lo, anchored at u_lo
        else if (kind == 2) emit_to(bound + 1);            // right: as in k_vp_z
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int i = 0; i < 7; ++i) {
                double* a = st[x * 7 + i + z];
                const float2 ha = f32x2_unpack(hi[x][i][0]), la = f32x2_unpack(lo[x][i][0]);
                const float2 hb = f32x2_unpack(hi[x][i][1]), lb = f32x2_unpack(lo[x][i][1]);
                const double2 jq = whole ? jm[(long long)r * nqp + q_of(i)] : make_double2(0.0, 0.0);
                const double Ar = ((double)ha.x - (double)la.x) + jq.x, Ai = (double)ha.y - (double)la.y;
                const double Br = ((double)hb.x - (double)lb.x) + jq.y, Bi = (double)hb.y - (double)lb.y;
                if (kind == 0) {                           // linear: u_j A (intercept dropped)
                    a[4] += Ar; a[5] += Ai;
                } else if (kind == 1) {
                    a[0] += Ar; a[1] += Ai;
                    a[2] += fma(-ub, Ar, Br); a[3] += fma(-ub, Ai, Bi);
                } else {
                    a[4] += Ar; a[5] += Ai;
                    a[0] -= Ar; a[1] -= Ai;
                    a[2] += fma(ub, Ar, -Br); a[3] += fma(ub, Ai, -Bi);
                }
            }
    }
    emit_to(kVpNS);
#pragma unroll 1
    for (int P = 0; P < 14; ++P) {
        const int k = k0 + kl + P / 7, q = q_of(P % 7);
        if (k < kend && q < nq)
            alin[(long long)s * NP + (long long)(k - kb) * nq + q] = make_double2(st[P + z][4], st[P + z][5]);
    }
}

__global__ void __launch_bounds__(kChPts)
k_vp_chain(VpDevice d, const double2* __restrict__ zp, const double2* __restrict__ alin, long long NP, int nq, int kb,
           double* __restrict__ out_re, double* __restrict__ out_im, int npieces, const unsigned char* __restrict__ only) {
    extern __shared__ __align__(16) unsigned char vsm[];
    double (*ar)[kChPts] = (double (*)[kChPts])vsm;                       // alpha (normalised)
    double (*ai)[kChPts] = (double (*)[kChPts])(vsm + 1 * kVpNS * kChPts * 8);
    double (*br)[kChPts] = (double (*)[kChPts])(vsm + 2 * kVpNS * kChPts * 8);   // z, then alpha'
    double (*bi)[kChPts] = (double (*)[kChPts])(vsm + 3 * kVpNS * kChPts * 8);
    double* sK = (double*)(vsm + 4 * kVpNS * kChPts * 8);                    // K[s-1], 48 x 48
    const int t = threadIdx.x;
    const long long p = (long long)blockIdx.x * kChPts + t;
    bool live = p < NP;                        // dead threads only help stage K
    if (only) {                                // not NULL: the points marked there
        live = live && only[p] != 0;
        if (!__syncthreads_or(live)) return;
    }
    double scale = 0.0;
    for (int s = 0; s < d.nsh; ++s) {
        if (s > 0) {
            __syncthreads();
            const double* Ks = d.K + (long long)(s - 1) * kVpNS * kVpNS;
            for (int e = t; e < kVpNS * kVpNS; e += kChPts) sK[e] = Ks[e];
            __syncthreads();
        }
        if (!live) continue;
        double2 al = alin[(long long)s * NP + p];
        for (int pc = 1; pc < npieces; ++pc) {
            const double2 a2 = alin[((long long)pc * d.nsh + s) * NP + p];
            al.x += a2.x; al.y += a2.y;
        }
        double mr = 0.0, mi = 0.0;
        for (int j = 0; j < kVpNS; ++j) {
            double2 zz = zp[((long long)s * kVpNS + j) * NP + p];
            for (int pc = 1; pc < npieces; ++pc) {
                const double2 z2 = zp[(((long long)pc * d.nsh + s) * kVpNS + j) * NP + p];
                zz.x += z2.x; zz.y += z2.y;
            }
            const double uj = d.u[j], wj = d.w[j];
            const double zr = fma(uj, al.x, zz.x), zi = fma(uj, al.y, zz.y);
            br[j][t] = zr; bi[j][t] = zi;
            mr = fma(wj, zr, mr); mi = fma(wj, zi, mi);
        }
        double mx = -1e300;
        for (int j = 0; j < kVpNS; ++j) {
            const double zr = br[j][t] - mr;
            br[j][t] = zr; bi[j][t] -= mi;
            mx = fmax(mx, zr);
        }
        double nrm = 0.0;
        for (int j0 = 0; j0 < kVpNS; j0 += 4) {
            double gr[4], gi[4];
            if (s == 0) {
#pragma unroll
                for (int q = 0; q < 4; ++q) { gr[q] = d.w[j0 + q]; gi[q] = 0.0; }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) { gr[q] = 0.0; gi[q] = 0.0; }
#pragma unroll 4
                for (int i = 0; i < kVpNS; ++i) {
                    const double xr = ar[i][t], xi = ai[i][t];
                    const double2 k01 = *(const double2*)(sK + i * kVpNS + j0);
                    const double2 k23 = *(const double2*)(sK + i * kVpNS + j0 + 2);
                    gr[0] = fma(k01.x, xr, gr[0]); gi[0] = fma(k01.x, xi, gi[0]);
                    gr[1] = fma(k01.y, xr, gr[1]); gi[1] = fma(k01.y, xi, gi[1]);
                    gr[2] = fma(k23.x, xr, gr[2]); gi[2] = fma(k23.x, xi, gi[2]);
                    gr[3] = fma(k23.y, xr, gr[3]); gi[3] = fma(k23.y, xi, gi[3]);
                }
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int j = j0 + q;
                const double m = exp(br[j][t] - mx);
                double sn, cs;
                sincos(bi[j][t], &sn, &cs);
                const double er = m * cs, ei = m * sn;
                const double nr = gr[q] * er - gi[q] * ei, ni = gr[q] * ei + gi[q] * er;
                br[j][t] = nr; bi[j][t] = ni;
                nrm = fmax(nrm, nr * nr + ni * ni);
            }
        }
        nrm = sqrt(nrm);
        const double inv = 1.0 / nrm;
        for (int j = 0; j < kVpNS; ++j) { ar[j][t] = br[j][t] * inv; ai[j][t] = bi[j][t] * inv; }
        scale += mx + log(nrm);
    }
    if (!live) return;
    double sr = 0.0, si = 0.0;
    for (int j = 0; j < kVpNS; ++j) { sr += ar[j][t]; si += ai[j][t]; }
    const long long o = (long long)kb * nq + p;
    out_re[o] = scale + 0.5 * log(sr * sr + si * si);
    out_im[o] = atan2(si, sr);
}

// The chain of the mixed path in float-float on the FP32 pipe.  In FP64 a (point, shell) step is 4608 FMAs of the
// transition and 48 exponentials and sincos, some 10^4 operations on a pipe of 2 per clock and SM; here the transition
// takes 12 packed (re, im) FP32 operations per state pair at 64 lanes per clock, e^z about 200 FP32 operations per state, and
// FP64 stays where z comes in (projection, maximum, the logarithm of the scale).  The state is renormalised by a power of
// two, which is exact.  CTA: 32 points; phase A a thread per (point, 8 states): z, e^z into shared memory; phase B a thread
// per (4 states, 2 points): alpha' = K^T alpha, times e^z.  409 x 109 points, 24 shells: 19.7 -> 3.7 ms; ln R differs from the FP64
// path by the same 6e-12 (1 + |ln R|) as with the FP64 chain.
// Range: every operation is exact to 2^-48 or to a few 2^-149 of the largest state, and a state that is small now can be the
// largest later, when the others have been scaled down by 2^-E in all (E: the renormalisations' exponents, which only grow
// where z spreads).  The transitions conserve the sum of such errors, so they reach at most 48 x 8 x shells x 2^(E - 149) of
// the result: 5e-14 at E = 90 and 64 shells.  Points with more are marked, and k_vp_chain does them over in FP64.
constexpr int kCfPts = 32, kCfThreads = 192;

typedef unsigned long long P2;
__device__ __forceinline__ P2 p2_mul(P2 a, P2 b) { P2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ P2 p2_add(P2 a, P2 b) { return vz_add(a, b); }
__device__ __forceinline__ P2 p2_fma(P2 a, P2 b, P2 c) { return vz_fma(a, b, c); }
__device__ __forceinline__ P2 p2_sub(P2 a, P2 b, P2 m1) { return p2_fma(b, m1, a); }

__device__ __forceinline__ ff ff_two_sum(float a, float b) {
    ff r;
    r.hi = a + b;
    const float bb = r.hi - a;
    r.lo = (a - (r.hi - bb)) + (b - bb);
    return r;
}
__device__ __forceinline__ ff ff_quick(float a, float b) { ff r; r.hi = a + b; r.lo = b - (r.hi - a); return r; }   // |a| >= |b|
__device__ __forceinline__ ff ffx_add(ff a, ff b) {
    const ff s = ff_two_sum(a.hi, b.hi);
    return ff_quick(s.hi, s.lo + (a.lo + b.lo));
}
__device__ __forceinline__ ff ffx_mul(ff a, ff b) {
    const float p = a.hi * b.hi;
    return ff_quick(p, fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, fmaf(a.hi, b.hi, -p))));
}
__device__ __forceinline__ ff ff_neg(ff a) { a.hi = -a.hi; a.lo = -a.lo; return a; }

// x - q C, C = c1 + (c2h + c2l), q an integer: q c1 and x.hi - q c1 are exact (c1 of few bits)
__device__ __forceinline__ ff ff_reduce(ff x, float q, float c1, float c2h, float c2l) {
    const float r1 = fmaf(-q, c1, x.hi);
    const float p = q * c2h, e = fmaf(q, c2h, -p);
    const ff s = ff_two_sum(r1, -p);
    return ff_quick(s.hi, s.lo + ((x.lo - e) - q * c2l));
}

// e^x, x <= 0: x = n ln 2 + r with ln 2 as a short head and a tail (Cody & Waite, Software Manual for the Elementary
// Functions, 1980; the same for pi / 2 below), 1 + r + r^2 / 2 + r^3 / 6 in float-float, the rest (6e-4 of the value) in FP32; results down
// to the subnormal numbers, 0 below 2^-150
__device__ __forceinline__ ff ff_exp(ff x) {
    ff z = {0.f, 0.f};
    if (x.hi < -104.f) return z;
    const float n = rintf(x.hi * 1.44269504088896341f);
    const ff r = ff_reduce(x, n, 0.693359375f, -2.12194442e-4f, 1.64659497e-12f);
    float t = fmaf(r.hi, 1.f / 3628800.f, 1.f / 362880.f);
    t = fmaf(r.hi, t, 1.f / 40320.f);
    t = fmaf(r.hi, t, 1.f / 5040.f);
    t = fmaf(r.hi, t, 1.f / 720.f);
    t = fmaf(r.hi, t, 1.f / 120.f);
    t = fmaf(r.hi, t, 1.f / 24.f);
    const ff r2 = ffx_mul(r, r);
    const ff sixth = {0.166666672f, -4.96705388e-9f};
    const ff r3 = ffx_mul(ffx_mul(r2, r), sixth);
    const ff h = {0.5f * r2.hi, 0.5f * r2.lo}, one = {1.f, 0.f};
    ff v = ff_quick(r3.hi, fmaf(r2.hi * r2.hi, t, r3.lo));
    v = ffx_add(h, v);
    v = ffx_add(r, v);
    v = ffx_add(one, v);
    const int e1 = (int)n >> 1, e2 = (int)n - e1;                    // n >= -151: two normal factors
    const float s1 = __int_as_float((e1 + 127) << 23), s2 = __int_as_float((e2 + 127) << 23);
    v.hi = v.hi * s1 * s2;
    v.lo = v.lo * s1 * s2;
    return v;
}

// sin x and cos x, |x| <= 2e4: x = q pi/2 + r; r, r^3 / 6 and 1, r^2 / 2, r^4 / 24 in float-float, the rest in FP32
__device__ __forceinline__ void ff_sincos(ff x, ff& s, ff& c) {
    const float q = rintf(x.hi * 0.636619772367581343f);
    const ff r = ff_reduce(x, q, 1.5703125f, 4.83826792e-4f, 2.56334407e-12f);
    const ff r2 = ffx_mul(r, r), r3 = ffx_mul(r2, r), r4 = ffx_mul(r2, r2);
    const ff sixth = {0.166666672f, -4.96705388e-9f}, c24 = {0.0416666679f, -1.24176347e-9f}, one = {1.f, 0.f};
    float t = fmaf(r2.hi, -1.f / 39916800.f, 1.f / 362880.f);
    t = fmaf(r2.hi, t, -1.f / 5040.f);
    t = fmaf(r2.hi, t, 1.f / 120.f);
    const ff a = ff_neg(ffx_mul(r3, sixth));
    ff sn = ffx_add(r, ff_quick(a.hi, fmaf(r3.hi * r2.hi, t, a.lo)));
    t = fmaf(r2.hi, -1.f / 3628800.f, 1.f / 40320.f);
    t = fmaf(r2.hi, t, -1.f / 720.f);
    const ff b = ffx_mul(r4, c24), h = {-0.5f * r2.hi, -0.5f * r2.lo};
    ff cs = ffx_add(h, ff_quick(b.hi, fmaf(r4.hi * r2.hi, t, b.lo)));
    cs = ffx_add(one, cs);
    const int k = (int)q & 3;
    s = k & 1 ? cs : sn;
    c = k & 1 ? sn : cs;
    if (k & 2) s = ff_neg(s);
    if ((k + 1) & 2) c = ff_neg(c);
}

__global__ void k_vp_K_ff(const double* __restrict__ K, long long n, float2* __restrict__ out) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const ff f = ff_from_double(K[e]);
    out[e] = make_float2(f.hi, f.lo);
}

struct ChainShared {
    float4 alpha[kVpNS][kCfPts];               // (re hi, im hi, re lo, im lo)
    float4 ez[kVpNS][kCfPts];                  // e^{z - max}
    float4 K[kVpNS][kVpNS / 2];                // two states: (hi, lo, hi, lo)
    double red[6][kCfPts][2];
    double mean[kCfPts][2], mx[kCfPts], scale[kCfPts];
    unsigned big[kCfPts];
    int down[kCfPts];                          // E: exponents of the renormalisations, summed
};
constexpr int kCfMaxDown = 90;

__global__ void __launch_bounds__(kCfThreads, 2)
k_vp_chain_ff(VpDevice d, const float2* __restrict__ Kff, const double2* __restrict__ zp, const double2* __restrict__ alin,
              long long NP, int nq, int kb, double* __restrict__ out_re, double* __restrict__ out_im, int npieces,
              unsigned char* __restrict__ redo) {
    extern __shared__ __align__(16) unsigned char vsm[];
    ChainShared& S = *reinterpret_cast<ChainShared*>(vsm);
    const int t = threadIdx.x, pa = t % kCfPts, ja = t / kCfPts;             // phase A: point, states 8 ja .. 8 ja + 7
    const int pb = t % 16, jb = 4 * (t / 16);                                // phase B: points pb, pb + 16, states jb .. jb + 3
    const long long p0 = (long long)blockIdx.x * kCfPts, p = p0 + pa;
    const bool live = p < NP;
    if (t < kCfPts) { S.scale[t] = 0.0; S.down[t] = 0; }
    const P2 m1 = f32x2_pack(-1.f, -1.f);
    for (int s = 0; s < d.nsh; ++s) {
        __syncthreads();                       // the previous shell's readers of alpha, K and the reductions are done
        if (s > 0) {
            const float4* Ks = reinterpret_cast<const float4*>(Kff + (long long)(s - 1) * kVpNS * kVpNS);
            for (int e = t; e < kVpNS * kVpNS / 2; e += kCfThreads) (&S.K[0][0])[e] = Ks[e];
        }
        // ---- phase A: z with zero stationary mean
        double zr[8], zi[8];
        {
            double2 al = make_double2(0.0, 0.0);
            if (live)
                for (int pc = 0; pc < npieces; ++pc) {
                    const double2 a2 = alin[((long long)pc * d.nsh + s) * NP + p];
                    al.x += a2.x; al.y += a2.y;
                }
            double mr = 0.0, mi = 0.0;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int j = 8 * ja + q;
                double2 zz = make_double2(0.0, 0.0);
                if (live)
                    for (int pc = 0; pc < npieces; ++pc) {
                        const double2 z2 = zp[(((long long)pc * d.nsh + s) * kVpNS + j) * NP + p];
                        zz.x += z2.x; zz.y += z2.y;
                    }
                const double uj = d.u[j], wj = d.w[j];
                zr[q] = fma(uj, al.x, zz.x);
                zi[q] = fma(uj, al.y, zz.y);
                mr = fma(wj, zr[q], mr);
                mi = fma(wj, zi[q], mi);
            }
            S.red[ja][pa][0] = mr;
            S.red[ja][pa][1] = mi;
        }
        __syncthreads();
        if (t < 2 * kCfPts) {
            const int pp = t >> 1, c = t & 1;
            double v = 0.0;
#pragma unroll
            for (int g = 0; g < 6; ++g) v += S.red[g][pp][c];
            S.mean[pp][c] = v;
        }
        __syncthreads();
        {
            const double mr = S.mean[pa][0], mi = S.mean[pa][1];
            double mx = -1e300;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                zr[q] -= mr;
                zi[q] -= mi;
                mx = fmax(mx, zr[q]);
            }
            S.red[ja][pa][0] = mx;
        }
        __syncthreads();
        if (t < kCfPts) {
            double v = S.red[0][t][0];
#pragma unroll
            for (int g = 1; g < 6; ++g) v = fmax(v, S.red[g][t][0]);
            S.mx[t] = v;
            S.big[t] = 0u;
        }
        __syncthreads();
        {
            const double mx = S.mx[pa];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const ff m = ff_exp(ff_from_double(zr[q] - mx));
                ff sn, cs;
                if (fabs(zi[q]) <= 2e4) {
                    ff_sincos(ff_from_double(zi[q]), sn, cs);
                } else {
                    double ds, dc;
                    sincos(zi[q], &ds, &dc);
                    sn = ff_from_double(ds);
                    cs = ff_from_double(dc);
                }
                const ff er = ffx_mul(m, cs), ei = ffx_mul(m, sn);
                S.ez[8 * ja + q][pa] = make_float4(er.hi, ei.hi, er.lo, ei.lo);
            }
        }
        // ---- phase B: alpha' = K^T alpha (the stationary weights at the first shell)
        P2 gh[4][2], gl[4][2];
        if (s == 0) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const ff w = ff_from_double(d.w[jb + q]);
#pragma unroll
                for (int x = 0; x < 2; ++x) { gh[q][x] = f32x2_pack(w.hi, 0.f); gl[q][x] = f32x2_pack(w.lo, 0.f); }
            }
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int x = 0; x < 2; ++x) { gh[q][x] = 0ull; gl[q][x] = 0ull; }
#pragma unroll 2
            for (int i = 0; i < kVpNS; ++i) {
                const float4 k01 = S.K[i][jb / 2], k23 = S.K[i][jb / 2 + 1];
                const float4 a0 = S.alpha[i][pb], a1 = S.alpha[i][pb + 16];
                const P2 ah[2] = {f32x2_pack(a0.x, a0.y), f32x2_pack(a1.x, a1.y)};
                const P2 al2[2] = {f32x2_pack(a0.z, a0.w), f32x2_pack(a1.z, a1.w)};
                const float kh[4] = {k01.x, k01.z, k23.x, k23.z}, kl[4] = {k01.y, k01.w, k23.y, k23.w};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const P2 h = f32x2_pack(kh[q], kh[q]), nh = f32x2_pack(-kh[q], -kh[q]), l = f32x2_pack(kl[q], kl[q]);
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        const P2 pr = p2_mul(h, ah[x]), ne = p2_fma(nh, ah[x], pr);     // product, minus its error
                        const P2 sum = p2_add(gh[q][x], pr), bb = p2_sub(sum, gh[q][x], m1);
                        const P2 er = p2_add(p2_sub(gh[q][x], p2_sub(sum, bb, m1), m1), p2_sub(pr, bb, m1));
                        P2 lo = p2_add(gl[q][x], er);
                        lo = p2_sub(lo, ne, m1);
                        lo = p2_fma(l, ah[x], lo);
                        gl[q][x] = p2_fma(h, al2[x], lo);
                        gh[q][x] = sum;
                    }
                }
            }
        }
        __syncthreads();                       // e^z complete; every reader of alpha is done
        float4 na[4][2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            float big = 0.f;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 h = f32x2_unpack(gh[q][x]), l = f32x2_unpack(gl[q][x]);
                const ff gr = ff_quick(h.x, l.x), gi = ff_quick(h.y, l.y);
                const float4 e = S.ez[jb + q][pb + 16 * x];
                const ff er = {e.x, e.z}, ei = {e.y, e.w};
                const ff nr = ffx_add(ffx_mul(gr, er), ff_neg(ffx_mul(gi, ei)));
                const ff ni = ffx_add(ffx_mul(gr, ei), ffx_mul(gi, er));
                na[q][x] = make_float4(nr.hi, ni.hi, nr.lo, ni.lo);
                big = fmaxf(big, fabsf(nr.hi) + fabsf(ni.hi));
            }
            atomicMax(&S.big[pb + 16 * x], __float_as_uint(big));
        }
        __syncthreads();
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            // 2^-ex with the largest modulus in [1/2, 2): exact
            const int ex = (int)(S.big[pb + 16 * x] >> 23) - 126;
            const float sc = __int_as_float((127 - max(-126, min(126, ex))) << 23);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 v = na[q][x];
                S.alpha[jb + q][pb + 16 * x] = make_float4(v.x * sc, v.y * sc, v.z * sc, v.w * sc);
            }
        }
        if (t < kCfPts) {
            const int ex = max(-126, min(126, (int)(S.big[t] >> 23) - 126));
            S.scale[t] += S.mx[t] + ex * 0.6931471805599453;
            S.down[t] += max(0, -ex);
        }
    }
    __syncthreads();
    if (t < kCfPts && live) {
        double sr = 0.0, si = 0.0;
        for (int j = 0; j < kVpNS; ++j) {
            const float4 v = S.alpha[j][t];
            sr += (double)v.x + (double)v.z;
            si += (double)v.y + (double)v.w;
        }
        redo[p] = S.down[t] > kCfMaxDown;
        const long long o = (long long)kb * nq + p;
        out_re[o] = S.scale[t] + 0.5 * log(sr * sr + si * si);
        out_im[o] = atan2(si, sr);
    }
}

// z and A_lin of a shell's pieces into the first one's place, in piece order
__global__ void k_vp_sum_pieces(double2* __restrict__ zp, long long nz, double2* __restrict__ alin, long long na, int npieces) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nz + na) return;
    double2* x = t < nz ? zp + t : alin + (t - nz);
    const long long stride = t < nz ? nz : na;
    double2 v = x[0];
#pragma unroll 8
    for (int pc = 1; pc < npieces; ++pc) {
        const double2 a = x[pc * stride];
        v.x += a.x; v.y += a.y;
    }
    x[0] = v;
}

// The same chain for few points (the k-reach probe lines): one CTA per point, two threads per state, one for the real
// parts and one (in other warps) for the imaginary ones.  The per-state work (mat-vec over i in the same order, exp beside
// sincos, normalisation) runs in parallel; the ordered sums (the projection's weighted means, the final state sums) stay on
// one thread each in state order, and the maxima are order-free, so the results are those of k_vp_chain.  Bound by the
// FP64 instructions of a shell in sequence (a warp's takes 64 cycles): 20 points, 24 shells, 26 pieces 0.63 -> 0.21 ms
// (pieces summed, K fetched and both parts' products formed by the same 64 threads, in turn).
constexpr int kChHalf = 64, kChSmallThreads = 2 * kChHalf;

__global__ void __launch_bounds__(kChSmallThreads)
k_vp_chain_small(VpDevice d, const double2* __restrict__ zp, const double2* __restrict__ alin, long long NP, int nq,
                 int kb, double* __restrict__ out_re, double* __restrict__ out_im) {
    __shared__ __align__(16) double sK[2][kVpNS * kVpNS];
    __shared__ double sw[kVpNS], z_s[2][kVpNS], al_s[2][kVpNS], g_s[2][kVpNS], n_s[2][kVpNS], mn[2], ex_s[kVpNS];
    __shared__ double2 tr_s[kVpNS];
    __shared__ double red[kChHalf];
    const int h = threadIdx.x / kChHalf, j = threadIdx.x % kChHalf;      // h = 0: real parts, 1: imaginary
    const long long p = blockIdx.x;
    const bool st = j < kVpNS;
    auto fetch_K = [&](int s) {                                         // of the step from shell s - 1 to s
        const double* Ks = d.K + (long long)(s - 1) * kVpNS * kVpNS;
        for (int e = 2 * threadIdx.x; e < kVpNS * kVpNS; e += 2 * kChSmallThreads) cp_async<16>(&sK[s & 1][e], Ks + e, true);
        cp_async_commit();
    };
    auto max_of = [&](double v) {                                       // over the h = 0 threads
        if (h == 0) red[j] = v;
        __syncthreads();
        for (int o = kChHalf / 2; o > 0; o >>= 1) {
            if (h == 0 && j < o) red[j] = fmax(red[j], red[j + o]);
            __syncthreads();
        }
        const double m = red[0];
        __syncthreads();
        return m;
    };
    auto part = [&](const double2& v) { return h == 0 ? v.x : v.y; };
    if (h == 0 && st) sw[j] = d.w[j];
    const double uj = st ? d.u[j] : 0.0;
    double scale = 0.0;
    double zn = st ? part(zp[(long long)j * NP + p]) : 0.0, an = part(alin[p]);
    for (int s = 0; s < d.nsh; ++s) {
        if (st) z_s[h][j] = fma(uj, an, zn);
        if (s + 1 < d.nsh) {                                            // the next shell's inputs on their way
            fetch_K(s + 1);
            zn = st ? part(zp[((long long)(s + 1) * kVpNS + j) * NP + p]) : 0.0;
            an = part(alin[(long long)(s + 1) * NP + p]);
        }
        __syncthreads();
        if (j == 0) {
            double m = 0.0;
            for (int i = 0; i < kVpNS; ++i) m = fma(sw[i], z_s[h][i], m);
            mn[h] = m;
        }
        double g = 0.0;
        if (st) {
            if (s == 0) g = h == 0 ? sw[j] : 0.0;
            else
                for (int i = 0; i < kVpNS; ++i) g = fma(sK[s & 1][i * kVpNS + j], al_s[h][i], g);
            g_s[h][j] = g;
        }
        __syncthreads();
        const double z = st ? z_s[h][j] - mn[h] : 0.0;
        const double mx = max_of(st ? z : -1e300);
        if (st) {
            if (h == 0) ex_s[j] = exp(z - mx);
            else sincos(z, &tr_s[j].y, &tr_s[j].x);
        }
        __syncthreads();
        if (st) {
            const double er = ex_s[j] * tr_s[j].x, ei = ex_s[j] * tr_s[j].y, gr = g_s[0][j], gi = g_s[1][j];
            n_s[h][j] = h == 0 ? gr * er - gi * ei : gr * ei + gi * er;
        }
        __syncthreads();
        const double nrm = sqrt(max_of(h == 0 && st ? n_s[0][j] * n_s[0][j] + n_s[1][j] * n_s[1][j] : 0.0));
        const double inv = 1.0 / nrm;
        if (st) al_s[h][j] = n_s[h][j] * inv;
        if (threadIdx.x < 32) scale += mx + log(nrm);
        cp_async_wait<0>();
        __syncthreads();
    }
    if (j == 0) {
        double a = 0.0;
        for (int i = 0; i < kVpNS; ++i) a += al_s[h][i];
        mn[h] = a;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double sr = mn[0], si = mn[1];
        const long long o = (long long)kb * nq + p;
        out_re[o] = scale + 0.5 * log(sr * sr + si * si);
        out_im[o] = atan2(si, sr);
    }
}

// The mixed path's grid kernel works on 112 columns at a time, k_vp_z on 32, at 0.4 of its time per column: up to 32 columns
// k_vp_z is the faster one.  ln R on 6 shells, 193 k cells, grid kernel / k_vp_z in ms: 409 x 32 4.44 / 3.66, 409 x 33 4.43 /
// 5.04, 409 x 113 7.46 / 8.40, 8 x 33 0.80 / 0.87, 16 x 40 0.98 / 1.37
bool vp_mixed_grid(int precision, int nk, int nq) { return precision != SGL_FP64 && nk >= 8 && nq > 32; }
static int vp_nqp(int nq) { return ceil_div(nq, kMzQ) * kMzQ; }

size_t vp_table_bytes(int precision, int U, int nk, int nq, int nruns) {
    const size_t es = precision == SGL_FP64 ? 8 : 4;
    if (vp_mixed_grid(precision, nk, nq))
        return 8 * (size_t)U * nk + 8 * (size_t)U * vp_nqp(nq) +
               16 * (size_t)std::max(1, nruns) * vp_nqp(nq) * (kJmParts + 1) + 1024;
    return 2 * es * ((size_t)U * nk + (size_t)U * nq) + 256;
}

int vp_rows_per_pass(int nsh, int nk, int nq, size_t z_cap_bytes) {
    const size_t per_row = (size_t)nsh * (kVpNS + 1) * 16 * (size_t)nq;
    long long rows = (long long)(z_cap_bytes / (per_row > 0 ? per_row : 1));
    if (rows < 1) rows = 1;
    if (rows > nk) rows = nk;
    const long long passes = (nk + rows - 1) / rows;            // balanced passes (no thin last pass)
    return (int)((nk + passes - 1) / passes);
}

// lines of points of the mixed path (the grid kernel's tiles and k_vp_z's would be mostly empty)
static bool vp_line(int precision, int nk, int nq) { return precision != SGL_FP64 && (nk == 1 || nq == 1) && (long long)nk * nq <= 4LL * kNumSMs; }

int vp_pieces(int precision, int nsh, int rows, int nq) {
    if (vp_line(precision, rows, nq)) {
        // sixteen warps per SM
        const long long base = (long long)ceil_div((long long)rows * nq, 32) * nsh;
        return (int)std::max(1LL, std::min(128LL, 16LL * kNumSMs / base));
    }
    if (vp_mixed_grid(precision, rows, nq)) {
        // two CTAs per SM: at least four waves, so that the last one costs at most a fifth
        const long long base = (long long)(vp_nqp(nq) / kMzQ) * ceil_div(rows, kMzK) * nsh;
        return (int)std::max(1LL, std::min(8LL, (4LL * 2 * kNumSMs + base - 1) / base));
    }
    const long long base = (long long)ceil_div(nq, kZQ) * ceil_div(rows, kZK) * nsh;
    const long long want = 8LL * kNumSMs;                   // CTAs of 128 threads
    return (int)std::max(1LL, std::min(32LL, (want + base - 1) / base));
}

void launch_vp_lnR(int precision, const VpDevice& d, const double* kv, int nk, const double* qv, int nq, void* tables,
                   double2* zbuf, int rows_per_pass, double* out_re, double* out_im, cudaStream_t st, int npieces, float2* Kff,
                   unsigned char* redo) {
    const long long tot = (long long)d.U * (nk + nq);
    const size_t es = precision == SGL_FP64 ? 8 : 4;
    void* e = tables;
    void* Jt = (char*)tables + 2 * es * (size_t)d.U * nk;
    // mixed grid: e (float2), then the run sums of J - 1 (double2), J and J - 1 with padded rows
    const bool grid = vp_mixed_grid(precision, nk, nq);
    const int nqp = vp_nqp(nq);
    double2* jm = (double2*)(((uintptr_t)tables + 8 * (size_t)d.U * nk + 255) & ~(uintptr_t)255);
    double2* jm_part = jm + (size_t)std::max(1, d.nruns) * nqp;
    float* J = (float*)(jm_part + (size_t)std::max(1, d.nruns) * nqp * kJmParts);
    float* Jm = J + (size_t)d.U * nqp;
    if (grid) {
        k_vp_tables_mixed<<<ceil_div((long long)d.U * (nk + nqp), 256), 256, 0, st>>>(d.ku, d.gu, d.U, kv, nk, qv, nq, nqp,
                                                                                      (float2*)e, J, Jm);
        SGL_COUNT(1);
        if (d.nruns > 0) {
            k_vp_jm<<<dim3(d.nruns, kJmParts, ceil_div(nqp, 128)), 128, 0, st>>>(d, Jm, nqp, jm_part);
            k_vp_jm_sum<<<ceil_div((long long)d.nruns * nqp, 256), 256, 0, st>>>(jm_part, (long long)d.nruns * nqp, jm);
            SGL_COUNT(2);
        }
    } else if (precision == SGL_FP64) {
        k_vp_tables<double><<<ceil_div(tot, 256), 256, 0, st>>>(d.ku, d.gu, d.U, kv, nk, qv, nq, (double2*)e, (double2*)Jt);
        SGL_COUNT(1);
    } else {
        k_vp_tables<float><<<ceil_div(tot, 256), 256, 0, st>>>(d.ku, d.gu, d.U, kv, nk, qv, nq, (float2*)e, (float2*)Jt);
        SGL_COUNT(1);
    }
    const size_t chain_smem = (4 * (size_t)kVpNS * kChPts + (size_t)kVpNS * kVpNS) * sizeof(double);
    cudaFuncSetAttribute(k_vp_chain, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)chain_smem);
    if (Kff) {
        const long long nK = (long long)(d.nsh - 1) * kVpNS * kVpNS;
        if (nK > 0) { k_vp_K_ff<<<ceil_div(nK, 256), 256, 0, st>>>(d.K, nK, Kff); SGL_COUNT(1); }
        cudaFuncSetAttribute(k_vp_chain_ff, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ChainShared));
    }
    for (int kb = 0; kb < nk; kb += rows_per_pass) {
        const int nkc = nk - kb < rows_per_pass ? nk - kb : rows_per_pass;
        const long long NP = (long long)nkc * nq;
        double2* zp = zbuf;
        double2* al = zbuf + (long long)npieces * d.nsh * kVpNS * NP;
        dim3 g1(ceil_div(nq, kZQ), ceil_div(nkc, kZK), d.nsh * npieces);
        if (precision == SGL_FP64) {
            k_vp_z<double><<<g1, kZThreads, 0, st>>>(d, (const double2*)e, (const double2*)Jt, nk, nq, kb, nkc, zp, al, NP,
                                                     npieces);
            SGL_COUNT(1);
        } else if (grid) {
            k_vp_z_mixed<<<dim3(nqp / kMzQ, ceil_div(nkc, kMzK), d.nsh * npieces), kMzThreads, 0, st>>>(
                d, (const float2*)e, J, jm, nk, nq, nqp, kb, nkc, zp, al, NP, npieces);
            SGL_COUNT(1);
        } else if (vp_line(precision, nk, nq)) {
            const dim3 gl(ceil_div(NP, 32), ceil_div((long long)d.nsh * npieces, kZlThreads / 32));
            k_vp_z_line<<<gl, kZlThreads, 0, st>>>(d, (const float2*)e, (const float2*)Jt, nk, nq, kb, zp, al, NP, npieces);
            SGL_COUNT(1);
        } else {
            k_vp_z<float><<<g1, kZThreads, 0, st>>>(d, (const float2*)e, (const float2*)Jt, nk, nq, kb, nkc, zp, al, NP,
                                                    npieces);
            SGL_COUNT(1);
        }
        if (NP <= 4LL * kNumSMs) {
            const long long na = (long long)d.nsh * NP, nz = na * kVpNS;
            if (npieces > 1) {
                k_vp_sum_pieces<<<ceil_div(nz + na, 128), 128, 0, st>>>(zp, nz, al, na, npieces);
                SGL_COUNT(1);
            }
            k_vp_chain_small<<<(unsigned)NP, kChSmallThreads, 0, st>>>(d, zp, al, NP, nq, kb, out_re, out_im);
            SGL_COUNT(1);
        } else if (Kff) {
            k_vp_chain_ff<<<ceil_div(NP, kCfPts), kCfThreads, sizeof(ChainShared), st>>>(d, Kff, zp, al, NP, nq, kb, out_re,
                                                                                         out_im, npieces, redo);
            k_vp_chain<<<ceil_div(NP, kChPts), kChPts, chain_smem, st>>>(d, zp, al, NP, nq, kb, out_re, out_im, npieces, redo);
            SGL_COUNT(2);
        } else {
            k_vp_chain<<<ceil_div(NP, kChPts), kChPts, chain_smem, st>>>(d, zp, al, NP, nq, kb, out_re, out_im, npieces, nullptr);
            SGL_COUNT(1);
        }
    }
}

}  // namespace sgl
