// Fused gauss Psi_2 term of the mixed path (reference: Lam._Qxi_gauss, sgl_full.py:2869-2951).
//
// For xi_lin group g and a tile of jt <= 8 coarse k_gamma columns j0 .. j0 + jt - 1, one CTA forms
//   T[p, (jl, rr)] = sum_{entries e of p} rows[rr, e] J_m(gam_{q_e} kg_{j0 + jl})   CUDA cores, FP32
//   Gc[n, (jl, rr)] = sum_p Ec[n, p] T[p, (jl, rr)]                                  tcgen05, TMEM
//   Gs[n, (jl, rr)] = sum_p Es[n, p] T[p, (jl, rr)]
//   part[g, j, n]   = ( sum_rr (a^2 - b^2), sum_rr a b )                              epilogue
// with a = Gc + V (m = 0) or Gc + kg res / 2 (m = 1), b = Gs + kk res (m = 0) or Gs, and
// Ec = cos(kk_n kap_p) (cos - 1 for m = 0 groups), Es = sin(kk_n kap_p).  The k_kappa index n sits
// on the 128 TMEM lanes (nk <= 128), the (jl, rr) pairs on the accumulator columns, so each thread
// of the epilogue holds every row rr of its (n, j) and sums over them without communication.  T and
// G never reach global memory: the unfused form writes and re-reads about 2 GB of them per PDF.
//
// Columns c = jl xi_pad(r) + rr: rows padded to a multiple of four, so that four rows of an entry are one 16-byte load.
//
// Pipeline (kXfStages shared-memory stages of 64 KB: E 4 x 8 KB [part][cos | sin], T 2 x 16 KB [part]):
//   12 producer warps build the T tiles of 16-p K blocks from the CSR entries, each warp 4-p blocks of its own
//                     (every twelfth), eight lanes per p: lane = (p, row quads, column half) with the sums of up to
//                     12 rows x 4 columns in registers.  Rows and gamma-cell indices come straight from global memory
//                     (L2), four entries' loads in flight per lane; J_m of the CTA's columns is staged once; the
//                     sums are transposed among the four p's lanes, split into TF32 hi + lo and stored in the
//                     canonical K-major layout; fence.proxy.async, one arrival per block;
//   1 copy thread     brings the packed E block (both parts, both halves) with one bulk copy;
//   1 MMA thread      issues A0 B0 + A0 B1 + A1 B0 (TF32 hi/lo, ~2^-21 per product) into the cos and
//                     sin accumulators (TMEM columns 0 and 256) and commits each K block to its "empty"
//                     barrier.
// What bounds it: the producers, waiting for L2 (1.5-2k cycles per batch of loads, three warps per scheduler).  A CTA of
// the reference's z_s = 1 groups (35 rows, 254 p, 3,928 entries) takes 109k cycles: prologue 4k, tiles 95k (the MMAs 25k,
// hidden), last products 5k, squares 5k.  One launch: 1.55 -> 1.36 ms (three warps per 4-p block with a group barrier and
// a bulk copy per chunk of entries, squares with a test per column: 147k cycles a CTA).
// The summation order of T over entries and of the squares over rr is that of the unfused kernels.
// Every wait is bounded; a wait that runs out sets *err, and the CTA waits for its copies in flight and releases its TMEM.
#include "kernels.cuh"
#include "tcgen05.cuh"

namespace sgl {

constexpr int kXfStages = 2;
constexpr int kXfABytes = 4 * 8192;                  // E: [part][cos | sin] x 128 lanes x 16 p
constexpr int kXfBPart = 16384;                      // T: 256 columns x 16 p, per part
constexpr int kXfStageBytes = kXfABytes + 2 * kXfBPart;
constexpr int kXfRMax = 48;                          // rows per group: 3 row quads for each of 4 lanes
constexpr int kXfProdWarps = 12;
constexpr int kXfProd = kXfProdWarps * 32;
constexpr int kXfThreads = kXfProd + 64;             // + copy warp + MMA warp
constexpr int kXfParts = kXfProdWarps / 4;           // column parts of the epilogue
constexpr int kXfJt = 8;                             // k_gamma columns per CTA at most
constexpr int kXfBlocks = 4;                         // 4-p blocks of a K block
// A parity tells a barrier's phase from its neighbours only, and a producer warp's blocks are kXfProdWarps / kXfBlocks
// = 3 K blocks apart: with a barrier per stage it would meet one that is two phases behind and pass.  One per K block
// modulo 8: a waiter for kb is less than 8 K blocks from any K block that shares it.
constexpr int kXfEmpty = 8;
static_assert(kXfProdWarps / kXfBlocks + 2 * kXfStages < kXfEmpty, "waits for a K block's barrier are unambiguous");
constexpr int kXfBatch = 4;                          // entries whose loads are in flight per lane
constexpr int kXfSmemStages = kXfStages * kXfStageBytes;
constexpr int kXfTabBytes = kXfRMax * 128 * 8 + kXfRMax * kXfJt * 8;     // the epilogue's correction terms
constexpr int kXfSmemFixed = kXfSmemStages + kXfTabBytes;

__device__ __forceinline__ int xf_find(const long long* prefix, int ng, long long v) {
    int lo = 0, hi = ng - 1;                          // largest g with prefix[g] <= v
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ float xf_add_ff(float b, float2 hl) {   // round(b + (h + l)) in FP32
    const float s = b + hl.x, bp = s - b;
    const float err = (b - (s - bp)) + (hl.x - bp);
    return s + (err + hl.y);
}

// four columns of a warp's lanes, asynchronous; xf_ld_wait names the registers, so that nothing reads them before it
__device__ __forceinline__ void xf_ld4(uint32_t taddr, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "r"(taddr));
}
__device__ __forceinline__ void xf_ld_wait(uint32_t* v) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]),
                   "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]),
                   "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23])
                 :: "memory");
}

int xi_fused_jt(int r) { return r <= 0 ? 0 : std::min(kXfJt, 256 / xi_pad(r)); }

// stages, correction terms, J_m columns, then the mbarriers, the TMEM address and the failure flag
size_t xi_fused_smem(int n_gmc) { return (size_t)kXfSmemFixed + (size_t)n_gmc * kXfJt * 4 + 8 * (kXfStages + kXfEmpty + 1) + 32; }

bool xi_fused_fits(int r_max, int nk, int n_gmc) {
    return nk >= 1 && nk <= 128 && r_max >= 1 && r_max <= kXfRMax && xi_fused_smem(n_gmc) <= 227 * 1024;
}

// Packed E: per group, per 16-p K block, 4 blocks of 128 lanes x 16 p in the canonical layout,
// [part 0 cos][part 0 sin][part 1 cos][part 1 sin].  One CTA per padded p, one thread per lane n;
// lanes n >= nk and p >= nP are zero.  The phase path is that of k_xi_E_ff (float-float k kap,
// exact reduction, half-angle sin / cos).
__global__ void __launch_bounds__(128)
k_xi_E_pack(XiDevice x, const double* __restrict__ kk, int nk, const long long* __restrict__ pp_prefix,
            const long long* __restrict__ p_prefix, const long long* __restrict__ e_off, float* __restrict__ Epk) {
    const long long P = blockIdx.x;
    const int g = xf_find(pp_prefix, x.n_groups, P);
    const int p = (int)(P - pp_prefix[g]);
    const int n = threadIdx.x;
    float ec = 0.f, es = 0.f;
    if (p < x.g_nP[g] && n < nk) {
        const ff kap = ff_from_double(x.kmc[x.idx_p[p_prefix[g] + p]]);
        float s, c, ph_hi, ph_lo;
        halfangle_sincos_ff(ff_from_double(kk[n]), kap, s, c, ph_hi, ph_lo);
        ec = x.g_m[g] == 0 ? -2.f * s * s : (c - s) * (c + s);
        es = 2.f * s * c;
    }
    const int k = p & 15;
    float* base = Epk + e_off[g] + (long long)(p >> 4) * (kXfABytes / 4);
    const int o = (n >> 3) * 128 + (k >> 2) * 32 + (n & 7) * 4 + (k & 3);
    const float ch = tf32_rna(ec), sh = tf32_rna(es);
    base[o] = ch;
    base[2048 + o] = sh;
    base[4096 + o] = tf32_rna(ec - ch);
    base[6144 + o] = tf32_rna(es - sh);
}

struct XiFusedArgs {
    XiDevice x;
    const long long* p_prefix;      // [n_groups + 1] global index of each group's first p
    const long long* rowf_off;      // [n_groups] float offset of each group's padded rows
    const int* jt;                  // [n_groups] k_gamma columns per CTA
    const long long* cta_prefix;    // [n_groups + 1]
    const long long* e_off;         // [n_groups] packed E offsets (floats)
    const float* Epk;
    const float* J;                 // FP32 Bessel tables [4][n_gmc][nkg]
    const float* Vf;                // [rows][nkg]  U (J0 - 1), m = 0 rows
    const float2* kresT;            // [rows][nk]   kk_n res_R as float-float
    const float2* hq;               // [rows][nkg]  kg_j res_R / 2 as float-float
    int nk, nkg;
    float2* part;                   // [n_groups][nkg][nk]
    int* err;
};

// ( sum_rr (a^2 - b^2), sum_rr a b ) of one k_gamma column, rows in order: cos sums at TMEM column col, sin sums 256 on.
// Twelve rows' loads under one wait and the harmonic's form fixed at compile time: with a test per column this took 27k
// cycles of a CTA (5k now).
template <int M>
__device__ __forceinline__ float2 xf_square(uint32_t col, int nq, int r, bool any, const float2* __restrict__ cor,
                                            const float2* __restrict__ kres) {
    float gre = 0.f, gim = 0.f;
    for (int Q0 = 0; Q0 < nq; Q0 += 3) {
        uint32_t v[3][8];
#pragma unroll
        for (int i = 0; i < 3; ++i)
            if (any && Q0 + i < nq) {
                xf_ld4(col + (uint32_t)(4 * (Q0 + i)), v[i]);
                xf_ld4(col + 256u + (uint32_t)(4 * (Q0 + i)), v[i] + 4);
            } else {
#pragma unroll
                for (int k = 0; k < 8; ++k) v[i][k] = 0u;
            }
        if (any) xf_ld_wait(&v[0][0]);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int rr = 4 * (Q0 + i) + k;
                if (rr >= r) break;                          // (the padded rows)
                float av = __uint_as_float(v[i][k]), bv = __uint_as_float(v[i][4 + k]);
                if (M == 0) {
                    av += cor[rr * kXfJt].x;
                    bv = xf_add_ff(bv, kres[rr * 128]);
                } else if (M == 1) {
                    av = xf_add_ff(av, cor[rr * kXfJt]);
                }
                gre = fmaf(av, av, fmaf(-bv, bv, gre));
                gim = fmaf(av, bv, gim);
            }
    }
    return make_float2(gre, gim);
}

__global__ void __launch_bounds__(kXfThreads, 1)
k_xi_fused(XiFusedArgs a) {
    extern __shared__ __align__(1024) unsigned char xsm[];
    const XiDevice& x = a.x;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long long cta = blockIdx.x;
    const int g = xf_find(a.cta_prefix, x.n_groups, cta);
    const int jt = a.jt[g];
    const int j0 = (int)(cta - a.cta_prefix[g]) * jt;
    const int r = x.g_r[g], m = x.g_m[g], nP = x.g_nP[g];
    const int r4 = xi_pad(r), nq = r4 / 4;
    const int N = ((jt * r4 + 15) / 16) * 16;           // MMA N (<= 256)
    const int nkb = (nP + 15) / 16;
    const int nk = a.nk, nkg = a.nkg, n_gmc = x.n_gmc;
    float* s_J = (float*)(xsm + kXfSmemFixed);                           // [n_gmc][8]
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(xsm);
    const uint32_t boff = kXfSmemFixed + n_gmc * kXfJt * 4;
    const uint32_t bar = sbase + boff;                   // full[S], empty[kXfEmpty], done
    constexpr int kNBar = kXfStages + kXfEmpty + 1;
    const uint32_t tslot = bar + 8 * kNBar;
    volatile int* s_fail = (volatile int*)(xsm + boff + 8 * kNBar + 8);
    auto full = [&](int s) { return bar + 8 * s; };
    auto empty = [&](int kb) { return bar + 8 * (kXfStages + kb % kXfEmpty); };
    auto wait_consumed = [&](int kb) { return mbar_wait_sleep(empty(kb), (uint32_t)((kb / kXfEmpty) & 1)); };
    const uint32_t done = bar + 8 * (kXfStages + kXfEmpty);

    if (warp == kXfProdWarps + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(tslot), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < kXfStages; ++s) mbar_init(full(s), kXfBlocks + 1);
        for (int e = 0; e < kXfEmpty; ++e) mbar_init(empty(e), 1);
        mbar_init(done, 1);
        *s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    {
        const float* Jm = a.J + (long long)m * n_gmc * nkg;
        for (int i = tid; i < n_gmc * kXfJt; i += kXfThreads) {
            const int q = i / kXfJt, jl = i % kXfJt, j = j0 + jl;
            s_J[i] = (jl < jt && j < nkg) ? Jm[(long long)q * nkg + j] : 0.f;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *(volatile uint32_t*)(xsm + boff + 8 * kNBar);

    int issued = 0;                                      // K blocks whose E copy was issued
    if (warp < kXfProdWarps && nkb > 0) {
        // ---- T producers.  Lane (u, rg, jh): p = 4 b + u of block b, row quads rg, rg + 4, rg + 8, columns 4 jh .. + 3;
        // an entry's sums run over the entries in order
        const int u = lane & 3, rg = (lane >> 2) & 3, jh = lane >> 4;
        const int* pptr = x.p_ptr + a.p_prefix[g];
        const float4* rows4 = (const float4*)(x.rows_f + a.rowf_off[g]) + rg;
        const long long ent0 = x.g_ent_off[g];
        const float* sj = s_J + 4 * jh;
        const int nslot = (nq + 3) / 4;                     // row quads of a lane (the last for some lanes only)
        const int nblk = kXfBlocks * nkb;
        int e0 = pptr[min(4 * warp + u, nP)], e1 = pptr[min(4 * warp + u + 1, nP)];
        for (int b = warp; b < nblk; b += kXfProdWarps) {
            const int n = e1 - e0, nmax = __reduce_max_sync(0xffffffffu, n);
            const int* qg = x.ent_qg + e0;
            const float4* rp = rows4 + ((long long)e0 - ent0) * nq;
            const int bn = b + kXfProdWarps;                // the next block's bounds, while this one is summed
            e0 = pptr[min(4 * bn + u, nP)];
            e1 = pptr[min(4 * bn + u + 1, nP)];
            float acc[3][4][4];                             // [row quad][row][column]
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int w = 0; w < 4; ++w) acc[i][k][w] = 0.f;
            for (int s0 = 0; s0 < nmax; s0 += kXfBatch) {
                int q[kXfBatch];
                float4 v[kXfBatch][3];
#pragma unroll
                for (int k = 0; k < kXfBatch; ++k) {
                    const bool in = s0 + k < n;
                    q[k] = in ? __ldg(qg + s0 + k) * kXfJt : 0;
#pragma unroll
                    for (int i = 0; i < 3; ++i)
                        v[k][i] = in && rg + 4 * i < nq ? __ldg(rp + (s0 + k) * nq + 4 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
                }
#pragma unroll
                for (int k = 0; k < kXfBatch; ++k) {
                    if (s0 + k >= nmax) break;
                    const float4 j = *(const float4*)(sj + q[k]);
#pragma unroll
                    for (int i = 0; i < 3; ++i) {
                        if (i >= nslot) break;
                        const float vv[4] = {v[k][i].x, v[k][i].y, v[k][i].z, v[k][i].w};
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            acc[i][t][0] = fmaf(vv[t], j.x, acc[i][t][0]);
                            acc[i][t][1] = fmaf(vv[t], j.y, acc[i][t][1]);
                            acc[i][t][2] = fmaf(vv[t], j.z, acc[i][t][2]);
                            acc[i][t][3] = fmaf(vv[t], j.w, acc[i][t][3]);
                        }
                    }
                }
            }
            const int kb = b / kXfBlocks, pb = b % kXfBlocks, s = kb % kXfStages;
            // its stage must have been consumed by the MMAs of kb - S (the warp stops or goes on as one)
            if (!warp_all(!*s_fail && (kb < kXfStages || wait_consumed(kb - kXfStages)))) {
                *s_fail = 1;
                break;
            }
            float* Bst = (float*)(xsm + s * kXfStageBytes + kXfABytes);
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const int Q = rg + 4 * i;
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    // transpose among the four p's lanes: lane u gets row 4 Q + u of the p's 0 .. 3
                    float t0 = acc[i][0][w], t1 = acc[i][1][w], t2 = acc[i][2][w], t3 = acc[i][3][w];
                    const float x0 = __shfl_xor_sync(0xffffffffu, u & 1 ? t0 : t1, 1);
                    const float x1 = __shfl_xor_sync(0xffffffffu, u & 1 ? t2 : t3, 1);
                    if (u & 1) { t0 = x0; t2 = x1; } else { t1 = x0; t3 = x1; }
                    const float y0 = __shfl_xor_sync(0xffffffffu, u & 2 ? t0 : t2, 2);
                    const float y1 = __shfl_xor_sync(0xffffffffu, u & 2 ? t1 : t3, 2);
                    if (u & 2) { t0 = y0; t1 = y1; } else { t2 = y0; t3 = y1; }
                    const int jl = 4 * jh + w;
                    if (jl < jt && Q < nq) {
                        // column c = jl r4 + 4 Q + u, K index 4 pb + (0 .. 3)
                        const int cq = jl * nq + Q, o = (cq >> 1) * 128 + pb * 32 + (cq & 1) * 16 + u * 4;
                        const float4 h = make_float4(tf32_rna(t0), tf32_rna(t1), tf32_rna(t2), tf32_rna(t3));
                        *(float4*)(Bst + o) = h;
                        *(float4*)(Bst + kXfBPart / 4 + o) =
                            make_float4(tf32_rna(t0 - h.x), tf32_rna(t1 - h.y), tf32_rna(t2 - h.z), tf32_rna(t3 - h.w));
                    }
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(full(s));
        }
    } else if (warp == kXfProdWarps && lane == 0) {
        // ---- E: one bulk copy per K block (both parts, cos and sin halves)
        const float* Eg = a.Epk + a.e_off[g];
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = kb % kXfStages;
            if (kb >= kXfStages && (*s_fail || !wait_consumed(kb - kXfStages))) {
                *s_fail = 1;
                break;
            }
            issued = kb + 1;
            mbar_expect_tx(full(s), kXfABytes);
            bulk_g2s(sbase + s * kXfStageBytes, Eg + (long long)kb * (kXfABytes / 4), kXfABytes, full(s));
        }
    } else if (warp == kXfProdWarps + 1 && lane == 0 && nkb > 0) {
        // ---- MMA issuer: cos accumulator at TMEM column 0, sin at column 256
        constexpr int PA[3] = {0, 0, 1};
        constexpr int PB[3] = {0, 1, 0};
        const uint32_t idesc = tc_idesc_tf32(kTcBM, N);
        for (int kb = 0; kb < nkb; ++kb) {
            const int s = kb % kXfStages;
            if (*s_fail || !mbar_wait_sleep(full(s), (uint32_t)((kb / kXfStages) & 1))) { *s_fail = 1; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a0 = sbase + s * kXfStageBytes, b0 = a0 + kXfABytes;
#pragma unroll
            for (int ks = 0; ks < 2; ++ks) {
                const uint32_t o = ks * 2 * kTcLBO;
#pragma unroll
                for (int trig = 0; trig < 2; ++trig)
#pragma unroll
                    for (int t = 0; t < 3; ++t)
                        tc_mma(tmem + 256u * trig, tc_desc(a0 + (PA[t] * 2 + trig) * 8192 + o),
                               tc_desc(b0 + PB[t] * kXfBPart + o), idesc, (kb | ks | t) ? 1u : 0u);
            }
            tc_commit(empty(kb));
        }
        tc_commit(done);
    }

    // ---- epilogue.  The producers that are done stage the square's correction terms for this CTA's rows and columns
    // while the last tiles are built and the last MMAs run.
    const long long R0 = x.g_row_off[g];
    float2* s_kres = (float2*)(xsm + kXfSmemStages);                       // [r][128]  kk_n res (m = 0)
    float2* s_cor = (float2*)(xsm + kXfSmemStages + kXfRMax * 128 * 8);   // [r][8]    (V, 0) m = 0 / hq m = 1
    if (warp < kXfProdWarps) {
        for (int i = tid; i < r * 128; i += kXfProd) {
            const int rq = i >> 7, n = i & 127;
            s_kres[i] = (m == 0 && n < nk) ? a.kresT[(R0 + rq) * nk + n] : make_float2(0.f, 0.f);
        }
        for (int i = tid; i < r * kXfJt; i += kXfProd) {
            const int rq = i / kXfJt, jl = i % kXfJt, j = j0 + jl;
            float2 v = make_float2(0.f, 0.f);
            if (jl < jt && j < nkg) {
                if (m == 0) v.x = a.Vf[(R0 + rq) * nkg + j];
                else if (m == 1) v = a.hq[(R0 + rq) * nkg + j];
            }
            s_cor[i] = v;
        }
    }
    bool ok = true;
    if (nkb > 0) ok = mbar_wait_sleep(done, 0u);
    const int all_ok = __syncthreads_and((ok && !*s_fail) ? 1 : 0);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (all_ok) {
        if (warp < kXfProdWarps) {
            // warp w reads TMEM lanes 32 (w % 4) .. + 31 (k_kappa index n) and the column part w / 4
            // (of kXfParts) of the (jl, rr) pairs; the rows rr of one (n, j) are summed in registers
            const int quad = warp & 3, part_ = warp >> 2;
            const int n = quad * 32 + lane;
            const int jl_lo = (jt * part_) / kXfParts, jl_hi = (jt * (part_ + 1)) / kXfParts;
            const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
            for (int jl = jl_lo; jl < jl_hi; ++jl) {
                const uint32_t col = lane_base + (uint32_t)(jl * r4);
                const float2* cor = s_cor + jl;
                float2 s = make_float2(0.f, 0.f);
                if (m == 0) s = xf_square<0>(col, nq, r, nkb > 0, cor, s_kres + n);
                else if (m == 1) s = xf_square<1>(col, nq, r, nkb > 0, cor, nullptr);
                else s = xf_square<2>(col, nq, r, nkb > 0, cor, nullptr);
                const int j = j0 + jl;
                if (n < nk && j < nkg) a.part[((long long)g * nkg + j) * nk + n] = s;
            }
        }
    } else {
        if (tid == 0) atomicExch(a.err, 1);
        // no bulk copy may outlive the CTA: waits for those of the last stages, bounded (a barrier whose producers gave up
        // never completes, but by then its copy has long landed)
        for (int kb = max(0, issued - kXfStages); kb < issued; ++kb) mbar_wait_sleep(full(kb % kXfStages), (uint32_t)((kb / kXfStages) & 1));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kXfProdWarps + 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512) : "memory");
    }
}

// out(n, j) = sum_g sign_g / 2 (sum_rr (a^2 - b^2)) + i sign_g sum_rr a b, groups in order, FP64
__global__ void k_xi_fused_sum(const float2* __restrict__ part, const int* __restrict__ g_m, int n_groups, int nk,
                               int nkg, double* __restrict__ out_re, double* __restrict__ out_im) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long long)nk * nkg) return;
    const int j = (int)(e / nk), n = (int)(e % nk);
    const long long stride = (long long)nkg * nk;
    const float2* pp = part + (long long)j * nk + n;
    double re = 0.0, im = 0.0;
    auto add = [&](int m, float2 v) {
        const double sign = (m == 0) ? 1.0 : ((m & 1) ? -2.0 : 2.0);
        re = fma(0.5 * sign, (double)v.x, re);
        im = fma(0.5 * sign, 2.0 * (double)v.y, im);
    };
    int g = 0;
    for (; g + 8 <= n_groups; g += 8) {            // eight loads in flight, summed in group order
        float2 v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = pp[(long long)(g + k) * stride];
#pragma unroll
        for (int k = 0; k < 8; ++k) add(g_m[g + k], v[k]);
    }
    for (; g < n_groups; ++g) add(g_m[g], pp[(long long)g * stride]);
    out_re[(long long)n * nkg + j] = re;
    out_im[(long long)n * nkg + j] = im;
}

void launch_xi_E_pack(const XiDevice& x, const double* kk, int nk, const long long* pp_prefix, long long total_pp,
                      const long long* p_prefix, const long long* e_off, float* Epk, cudaStream_t st) {
    if (total_pp <= 0) return;
    k_xi_E_pack<<<(unsigned)total_pp, 128, 0, st>>>(x, kk, nk, pp_prefix, p_prefix, e_off, Epk);
    SGL_COUNT(1);
}

void launch_xi_fused(const XiDevice& x, const long long* p_prefix, const long long* rowf_off, const int* jt,
                     const long long* cta_prefix, long long ctas, const long long* e_off, const float* Epk,
                     const float* J, const float* Vf, const float2* kresT, const float2* hq, int nk, int nkg,
                     float2* part, int* err, double* out_re, double* out_im, cudaStream_t st) {
    if (ctas > 0) {
        XiFusedArgs a{x, p_prefix, rowf_off, jt, cta_prefix, e_off, Epk, J, Vf, kresT, hq, nk, nkg, part, err};
        const size_t sm = xi_fused_smem(x.n_gmc);
        cudaFuncSetAttribute(k_xi_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        k_xi_fused<<<(unsigned)ctas, kXfThreads, sm, st>>>(a);
        SGL_COUNT(1);
    }
    const long long tot = (long long)nk * nkg;
    k_xi_fused_sum<<<ceil_div(tot, 256), 256, 0, st>>>(part, x.g_m, x.n_groups, nk, nkg, out_re, out_im);
    SGL_COUNT(1);
}

}  // namespace sgl
