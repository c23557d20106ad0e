// Fused inference of the surrogate MLP (8 -> 256 -> 5 x (256 -> 256) -> 2, SiLU): one persistent
// kernel, one CTA per SM, 128-row tiles; the activations never leave the SM.
//
// Per tile, each layer is one accumulation in TMEM (128 lanes x 256 columns FP32) of
// tcgen05.mma.kind::f16 products.  The input layer (K = 8) takes the inputs as three BF16 parts (all
// 24 bits); a hidden layer's input is held in shared memory as two (hi = bf16(a), lo = bf16(a - hi):
// the FP32 activation to 2^-17), and its BF16 weights come through a 4-stage ring of 16 KB bulk copies
// (the same for every tile: L2-resident).  The epilogue warps read the accumulator with
// tcgen05.ld, add the bias, apply SiLU and write the next layer's hi / lo parts in the canonical
// K-major layout; after the last hidden layer they form the two outputs as FP32 dot products.  The
// arithmetic is that of the training forward (BF16 weights, split BF16 inputs, FP32 accumulation).
//
// Warps 0-15: epilogue (row = 32 x (warp & 3) + lane, columns 8 x (warp >> 2) of each K block), warp
// 16 lane 0: weight copies, warp 17: MMAs.  The layers alternate between two accumulators and
// each K block has a barrier of its own, so a layer's products start while the epilogue that makes
// its input is at the second K block; the next tile's input epilogue runs before the last epilogue of
// a tile, under which the next tile's first products run.  Of a layer's ~4,100 MMA cycles only the last
// block's are not under an epilogue.
//
// What bounds it: per tile and SM 20.5k MMA cycles (both parts, 4 x 128 per K block) and 6 x 4.1k cycles of the
// special-function unit (exp2 and reciprocal per value).  A tile takes 34k: a layer's epilogue 5.3k, then ~1.2k until
// the last K block's products are through.  700,001 rows: 4.34 -> 0.72 ms (four epilogue warps and one accumulator,
// epilogues and products in turn: 220k cycles a tile; input layer on the CUDA cores, 9k cycles of the tile: 0.84 ms).
//
// Every wait is bounded; a wait that runs out raises *err, and the CTA waits for its copies and
// products in flight and frees its TMEM before it returns.
#include <cuda_bf16.h>

#include <algorithm>

#include "cfterm.cuh"
#include "kernels.cuh"
#include "tcgen05.cuh"

namespace sgl {
namespace {

constexpr int kMfRows = 128;
constexpr int kMfW = 256;                          // hidden width
constexpr int kMfIn = 8;
constexpr int kMfHidden = 5;                       // 256 -> 256 layers on the tensor cores
constexpr int kMfKB = kMfW / 32;                   // 32-element K blocks per layer
constexpr int kMfABlock = kMfRows * 64;            // bytes of one K block of one activation part
constexpr int kMfWBlock = kMfW * 64;               // bytes of one K block of a weight matrix
constexpr int kMfStages = 4;
static_assert(kMfKB == 2 * kMfStages, "a layer takes each ring stage twice: its parities are constants");
constexpr int kMfEpiWarps = 16;
constexpr int kMfGroups = kMfEpiWarps / 4;         // column groups of a K block, 8 columns each
constexpr int kMfThreads = (kMfEpiWarps + 2) * 32;
static_assert(kMfGroups * 8 == 32, "a K block's columns over the groups");
constexpr int kMfOffAhi = 0;
constexpr int kMfOffAlo = kMfKB * kMfABlock;                         // 64 KB
constexpr int kMfOffRing = 2 * kMfKB * kMfABlock;                    // 128 KB
constexpr int kMfOffSmall = kMfOffRing + kMfStages * kMfWBlock;      // 192 KB
// small tables (floats): W0 (BF16, the K-major B operand of K = 16 with the 8 inputs twice), biases [6][256], W6 [256][2], b6 [2]
constexpr int kMfSmallFloats = kMfIn * kMfW + 6 * kMfW + 2 * kMfW + 2;
// partial outputs of the column groups 1 .. : [tile parity][group - 1][row][2]
constexpr int kMfOffY = kMfOffSmall + ((kMfSmallFloats * 4 + 127) / 128) * 128;
// the next tile's inputs, one K block of the layout of an activation part: x1 | x2 | x3 | 0 (8 elements each)
constexpr int kMfOffX = kMfOffY + 2 * (kMfGroups - 1) * kMfRows * 8;
constexpr int kMfOffBar = kMfOffX + kMfABlock;
constexpr int kMfSmem = kMfOffBar + 256;

// byte offset of (row r, k) of a K-major activation part: K blocks of 32, core matrices 8 x 16 B
__device__ __forceinline__ uint32_t mf_a_off(int r, int k) {
    return (uint32_t)((k >> 5) * kMfABlock + (r >> 3) * 512 + ((k & 31) >> 3) * 128 + (r & 7) * 16);
}

// z / (1 + exp(-z)) of two values, to a few 2^-23 of the value where |z| is a few (the exponent's rounding grows with
// |z| on the negative side, where the value itself decays); z below -88 gives 0 and a NaN or -inf a NaN, as the
// quotient does.  One reciprocal for both (1 / d0 = d1 / (d0 d1)) was no faster: the exponents need a bound then.
__device__ __forceinline__ unsigned long long mf_silu2(unsigned long long z) {
    const float2 p = f32x2_unpack(f32x2_mul(z, f32x2_dup(-1.44269504088896341f)));
    float e0, e1, r0, r1;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(p.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(p.y));
    const float2 d = f32x2_unpack(f32x2_add(f32x2_pack(e0, e1), f32x2_dup(1.f)));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(d.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r1) : "f"(d.y));
    return f32x2_mul(z, f32x2_pack(r0, r1));
}

// two activations as their BF16 parts
__device__ __forceinline__ void mf_split(unsigned long long a, uint32_t& hi, uint32_t& lo) {
    const float2 v = f32x2_unpack(a);
    const __nv_bfloat162 h = __floats2bfloat162_rn(v.x, v.y);
    hi = *(const uint32_t*)&h;
    const float2 d = f32x2_unpack(f32x2_fma3(f32x2_pack(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u)),
                                             f32x2_dup(-1.f), a));
    const __nv_bfloat162 l = __floats2bfloat162_rn(d.x, d.y);
    lo = *(const uint32_t*)&l;
}

// 8 consecutive activations of one row (k0 multiple of 8) into the hi / lo parts
__device__ __forceinline__ void mf_store8(unsigned char* sm, int r, int k0, const unsigned long long* a) {
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) mf_split(a[e], hi[e], lo[e]);
    const uint32_t o = mf_a_off(r, k0);
    *(uint4*)(sm + kMfOffAhi + o) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *(uint4*)(sm + kMfOffAlo + o) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
}

// the input weights as a B operand: K = 16, 8-row groups 256 bytes apart
__device__ __forceinline__ uint64_t mf_desc_w0(uint32_t saddr) {
    return (tc_desc(saddr) & ~((uint64_t)0x3FFF << 32)) | ((uint64_t)(256 >> 4) << 32);
}

// 8 columns of a warp's lanes, asynchronous; mf_ld8_wait names the registers, so that nothing reads them before it
__device__ __forceinline__ void mf_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void mf_ld8_wait(uint32_t* r) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7])
                 :: "memory");
}

__global__ void __launch_bounds__(kMfThreads, 1)
k_mlp_fused(int n, const float* __restrict__ X, const unsigned char* __restrict__ Wp, const float* __restrict__ small,
            float* __restrict__ Y, int* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char sm[];
    const uint32_t sb = (uint32_t)__cvta_generic_to_shared(sm);
    const uint32_t bar = sb + kMfOffBar;               // full[4], empty[4], layer_done, drain, y, x, in, ready[8]
    const uint32_t b_full = bar, b_empty = bar + 8 * kMfStages, b_done = bar + 16 * kMfStages, b_drain = b_done + 8,
                   b_y = b_done + 16, b_x = b_done + 24, b_in = b_done + 32, b_ready = b_done + 40;
    volatile int* s_fail = (volatile int*)(sm + kMfOffBar + 192);
    const uint32_t tslot = sb + kMfOffBar + 200;
    float* s_small = (float*)(sm + kMfOffSmall);
    const float* s_b = s_small + kMfIn * kMfW;          // [layer][n], layer 0 .. 5
    const float* s_W6 = s_b + 6 * kMfW;                 // [k][2]
    const float* s_b6 = s_W6 + 2 * kMfW;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n_tiles = (n + kMfRows - 1) / kMfRows;

    for (int e = tid; e < kMfSmallFloats; e += kMfThreads) s_small[e] = small[e];
    for (int r = tid; r < kMfRows; r += kMfThreads) *(uint4*)(sm + kMfOffX + (r >> 3) * 512 + 384 + (r & 7) * 16) = make_uint4(0, 0, 0, 0);
    fence_proxy_async_smem();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(tslot), "r"(2 * kMfW) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < 2 * kMfStages + 2; ++s) mbar_init(bar + 8 * s, 1);
        mbar_init(b_y, kMfEpiWarps - 4);
        mbar_init(b_x, kMfEpiWarps);
        mbar_init(b_in, 1);
        for (int kb = 0; kb < kMfKB; ++kb) mbar_init(b_ready + 8 * kb, kMfEpiWarps);
        *s_fail = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *(volatile uint32_t*)(sm + kMfOffBar + 200);

    if (warp == kMfEpiWarps) {
        if (lane == 0) {
            // weight copies: per tile, every hidden layer's 8 K blocks, through the ring
            long long it = 0;
            for (int t = blockIdx.x; t < n_tiles && !*s_fail; t += gridDim.x) {
                for (int q = 0; q < kMfHidden * kMfKB; ++q, ++it) {
                    const int s = (int)(it % kMfStages);
                    if (it >= kMfStages && !mbar_wait_bounded(b_empty + 8 * s, (uint32_t)(((it / kMfStages) - 1) & 1))) {
                        *s_fail = 1;
                        break;
                    }
                    mbar_expect_tx(b_full + 8 * s, kMfWBlock);
                    bulk_g2s(sb + kMfOffRing + s * kMfWBlock, Wp + (long long)q * kMfWBlock, kMfWBlock, b_full + 8 * s);
                }
                if (*s_fail) break;
            }
            // the copies issued last have landed before the CTA moves on (normally already consumed)
            for (long long j = it - 1; j >= 0 && j >= it - kMfStages; --j)
                if (!mbar_wait_bounded(b_full + 8 * (int)(j % kMfStages), (uint32_t)((j / kMfStages) & 1))) *s_fail = 1;
        }
    } else if (warp == kMfEpiWarps + 1) {
        // the whole warp runs the loop and lane 0 issues: descriptors and parities stay uniform values, the stage of
        // a K block is a constant (8 blocks a layer, 4 stages)
        const uint32_t idesc = tc_idesc_bf16(kMfRows, kMfW);
        const uint64_t d_ah = tc_desc(sb + kMfOffAhi), d_al = tc_desc(sb + kMfOffAlo), d_w = tc_desc(sb + kMfOffRing);
        uint32_t use = 0, inputs = 0;
        bool ok = true;
        // the input layer of a tile into the accumulator of its layer 0: (x1 + x2 + x3) W0, W0 the same for both steps
        auto input_mma = [&]() {
            ok = ok && mbar_wait_bounded(b_x, inputs & 1u);
            ++inputs;
            if (lane == 0 && ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + (use & 1u) * kMfW;
                const uint64_t d_x = tc_desc(sb + kMfOffX), d_w0 = mf_desc_w0(sb + kMfOffSmall);
                tc_mma_bf16(acc, d_x + (uint64_t)((2 * kTcLBO) >> 4), d_w0, idesc, 0u);
                tc_mma_bf16(acc, d_x, d_w0, idesc, 1u);
                tc_commit(b_in);
            }
        };
        if ((int)blockIdx.x < n_tiles) input_mma();
        for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
            for (int l = 0; l < kMfHidden && ok; ++l, ++use) {
                const uint32_t acc = tmem + (use & 1u) * kMfW;
                ok = !*s_fail;
                // layer 0 overwrites the accumulator its input is read from: all of it has to be read
                if (l == 0) ok = ok && mbar_wait_bounded(b_ready + 8 * (kMfKB - 1), use & 1u);
#pragma unroll
                for (int kb = 0; kb < kMfKB; ++kb) {
                    const int s = kb % kMfStages;
                    ok = ok && mbar_wait_bounded(b_ready + 8 * kb, use & 1u) &&
                         mbar_wait_bounded(b_full + 8 * s, (uint32_t)((kb / kMfStages) & 1));
                    if (lane == 0 && ok) {
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        // low parts first: each addition is truncated at the accumulator's magnitude, and the first
                        // block's meet a small one (30 truncations of a layer's 32 count)
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const uint64_t o = (uint64_t)((kb * kMfABlock + (q & 1) * 2 * kTcLBO) >> 4);
                            const uint64_t w = d_w + (uint64_t)((s * kMfWBlock + (q & 1) * 2 * kTcLBO) >> 4);
                            tc_mma_bf16(acc, (q < 2 ? d_al : d_ah) + o, w, idesc, (kb | q) ? 1u : 0u);
                        }
                        tc_commit(b_empty + 8 * s);
                        if (kb == kMfKB - 1) tc_commit(b_done);
                    }
                }
            }
            // layer 3's accumulator was read before layer 4's products began
            if (t + (int)gridDim.x < n_tiles) input_mma();
        }
        if (lane == 0) {
            // every product issued has finished before the TMEM is given back
            tc_commit(b_drain);
            ok = mbar_wait_bounded(b_drain, 0u) && ok;
        }
        if (!ok) *s_fail = 1;
    } else {
        // epilogue: row r of the tile, columns c .. c + 7 of each K block
        const int r = (warp & 3) * 32 + lane, g = warp >> 2, c = g * 8;
        const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c;
        long long use = 0;
        int par = 0;
        // the warp's part of K block kb is in shared memory (and the accumulator columns behind it are read)
        auto ready = [&](int kb) {
            fence_proxy_async_smem();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(b_ready + 8 * kb);
        };
        // inputs of a tile: two values per thread, read early, put into shared memory as three BF16 parts (all 24 bits)
        float xr[2];
        auto fetch_x = [&](int t) {
            const long long e0 = (long long)t * kMfRows * kMfIn;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const long long e = e0 + q * (kMfEpiWarps * 32) + tid;
                xr[q] = e < (long long)n * kMfIn ? X[e] : 0.f;
            }
        };
        auto put_x = [&]() {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int e = q * (kMfEpiWarps * 32) + tid, row = e >> 3, k = e & 7;
                unsigned char* p = sm + kMfOffX + (row >> 3) * 512 + (row & 7) * 16 + 2 * k;
                float v = xr[q];
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const __nv_bfloat16 h = __float2bfloat16_rn(v);
                    *(__nv_bfloat16*)(p + j * 128) = h;
                    v -= __bfloat162float(h);
                }
            }
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(b_x);
        };
        // bias and SiLU of an accumulator; store: into the next layer's input, else the outputs' dot products
        unsigned long long y = 0ull;
        auto epilogue = [&](uint32_t acc, const float* bl, bool store) {
            uint32_t v[8];
            mf_ld8(acc, v);
#pragma unroll 2
            for (int kb = 0; kb < kMfKB; ++kb) {
                mf_ld8_wait(v);
                const ulonglong2 b0 = *(const ulonglong2*)(bl + kb * 32), b1 = *(const ulonglong2*)(bl + kb * 32 + 4);
                unsigned long long z[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) z[j] = f32x2_pack(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
                if (kb + 1 < kMfKB) mf_ld8(acc + (kb + 1) * 32, v);
                z[0] = mf_silu2(f32x2_add(z[0], b0.x));
                z[1] = mf_silu2(f32x2_add(z[1], b0.y));
                z[2] = mf_silu2(f32x2_add(z[2], b1.x));
                z[3] = mf_silu2(f32x2_add(z[3], b1.y));
                if (store) {
                    mf_store8(sm, r, kb * 32 + c, z);
                    ready(kb);
                } else {
                    const ulonglong2* w6 = (const ulonglong2*)(s_W6 + 2 * (kb * 32 + c));
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 zj = f32x2_unpack(z[j]);
                        const ulonglong2 w = w6[j];
                        y = f32x2_fma3(f32x2_dup(zj.x), w.x, y);
                        y = f32x2_fma3(f32x2_dup(zj.y), w.y, y);
                    }
                }
            }
        };
        // waits of a whole warp: tcgen05.ld is warp-collective, so is the decision to stop
        bool bad = false;
        auto wait = [&](uint32_t bar_, uint32_t parity) {
            bad = *s_fail != 0 || !mbar_wait_bounded(bar_, parity);
            if (__any_sync(0xffffffffu, bad)) { bad = true; *s_fail = 1; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            return !bad;
        };
        if ((int)blockIdx.x < n_tiles) {
            fetch_x(blockIdx.x);
            put_x();
            if (wait(b_in, 0u)) epilogue(trow, s_b + c, true);
        }
        for (int t = blockIdx.x; t < n_tiles && !bad; t += gridDim.x, par ^= 1) {
            const bool more = t + (int)gridDim.x < n_tiles;
            if (more) fetch_x(t + gridDim.x);
            for (int l = 0; l < kMfHidden - 1; ++l, ++use) {
                // this tile's inputs were consumed before layer 0
                if (more && l == kMfHidden - 2) put_x();
                if (!wait(b_done, (uint32_t)(use & 1))) break;
                epilogue(trow + (uint32_t)((use & 1) * kMfW), s_b + (l + 1) * kMfW + c, true);
            }
            if (bad || !wait(b_done, (uint32_t)(use & 1))) { bad = true; break; }
            // the activations of this tile are consumed: the next tile's first products run under its last epilogue
            if (more) {
                if (!wait(b_in, (uint32_t)(par ^ 1))) break;
                epilogue(trow + (uint32_t)(((use + 1) & 1) * kMfW), s_b + c, true);
            }
            y = 0ull;
            epilogue(trow + (uint32_t)((use & 1) * kMfW), s_b + kMfHidden * kMfW + c, false);
            ++use;
            // the column groups' sums, added in order by group 0.  Two buffers: a group writes this one again two
            // tiles on, after layers whose inputs group 0 had to hand over
            unsigned long long* sy = (unsigned long long*)(sm + kMfOffY) + par * (kMfGroups - 1) * kMfRows + r;
            if (g) {
                sy[(g - 1) * kMfRows] = y;
                __syncwarp();
                if (lane == 0) mbar_arrive(b_y);
                continue;
            }
            bad = !mbar_wait_bounded(b_y, (uint32_t)par);
            if (__any_sync(0xffffffffu, bad)) { *s_fail = 1; break; }
#pragma unroll
            for (int q = 0; q < kMfGroups - 1; ++q) y = f32x2_add(y, sy[q * kMfRows]);
            const long long gr = (long long)t * kMfRows + r;
            if (gr < n) {
                const float2 o = f32x2_unpack(y);
                Y[2 * gr] = o.x + s_b6[0];
                Y[2 * gr + 1] = o.y + s_b6[1];
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0 && *s_fail) atomicExch(err, 1);
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(2 * kMfW) : "memory");
    }
}

// hidden weights W_l (FP32 [k][n], l = 1 .. 5) -> BF16 canonical K-major B blocks [l][kb][n rows][64 B]
__global__ void k_mlp_pack_hidden(const float* const* __restrict__ W, unsigned char* __restrict__ out) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;           // (layer, kb, n, chunk of 8 k)
    const int total = kMfHidden * kMfKB * kMfW * 4;
    if (e >= total) return;
    const int c = e & 3, nrow = (e >> 2) % kMfW, kb = ((e >> 2) / kMfW) % kMfKB, l = (e >> 2) / kMfW / kMfKB;
    const float* Wl = W[l];
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int k = kb * 32 + c * 8 + 2 * q;
        const __nv_bfloat162 b2 = __floats2bfloat162_rn(Wl[k * kMfW + nrow], Wl[(k + 1) * kMfW + nrow]);
        w[q] = *(const uint32_t*)&b2;
    }
    const long long o = (long long)(l * kMfKB + kb) * kMfWBlock + (nrow >> 3) * 512 + c * 128 + (nrow & 7) * 16;
    *(uint4*)(out + o) = make_uint4(w[0], w[1], w[2], w[3]);
}

// the small tables: input weights and last weights rounded to BF16 (as the training forward's GEMMs
// use them), biases FP32.  Input weights: 8-row groups of 256 bytes, two equal 128-byte core matrices each.
__global__ void k_mlp_pack_small(const float* __restrict__ W0, const float* const* __restrict__ b,
                                 const float* __restrict__ W6, const float* __restrict__ b6, float* __restrict__ out) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < kMfIn * kMfW) {
        const int nrow = (e >> 6) * 8 + ((e & 31) >> 2), k = 2 * (e & 3);
        const __nv_bfloat162 v = __floats2bfloat162_rn(W0[k * kMfW + nrow], W0[(k + 1) * kMfW + nrow]);
        out[e] = __uint_as_float(*(const uint32_t*)&v);
        return;
    }
    int f = e - kMfIn * kMfW;
    if (f < 6 * kMfW) { out[e] = b[f / kMfW][f % kMfW]; return; }
    f -= 6 * kMfW;
    if (f < 2 * kMfW) { out[e] = __bfloat162float(__float2bfloat16_rn(W6[f])); return; }
    f -= 2 * kMfW;
    if (f < 2) out[e] = b6[f];
}

}  // namespace

int mlp_fused_smem() { return kMfSmem; }
int mlp_fused_small_floats() { return kMfSmallFloats; }
long long mlp_fused_wp_bytes() { return (long long)kMfHidden * kMfKB * kMfWBlock; }

void launch_mlp_fused(int n, const float* X, const float* const* W_dev, const float* const* b_dev, unsigned char* Wp,
                      float* small, const float** ptrs, float* Y, int* err, int ctas, cudaStream_t st) {
    // ptrs (device): W_1 .. W_5, then b_0 .. b_5
    k_mlp_pack_hidden<<<ceil_div(kMfHidden * kMfKB * kMfW * 4, 256), 256, 0, st>>>(ptrs, Wp);
    k_mlp_pack_small<<<ceil_div(kMfSmallFloats, 256), 256, 0, st>>>(W_dev[0], ptrs + kMfHidden, W_dev[6], b_dev[6], small);
    const int n_tiles = (n + kMfRows - 1) / kMfRows;
    k_mlp_fused<<<std::max(1, std::min(ctas, n_tiles)), kMfThreads, kMfSmem, st>>>(n, X, Wp, small, Y, err);
    SGL_COUNT(3);
}

sgl_status mlp_fused_attr() {
    return cudaFuncSetAttribute(k_mlp_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, kMfSmem) == cudaSuccess
               ? SGL_OK : SGL_ERR_CUDA;
}

}  // namespace sgl
