// Grouped FP64 GEMM on the 5th-generation tensor cores by exact slicing (the scheme of Ozaki, Ogita, Oishi & Rump,
// Numer. Algorithms 59, 95 (2012), in fixed point with BF16 digits):
//   C(i, j) = alpha sum_k A(i, k) B(k, j) + beta C(i, j)
//
// A row of A (a column of B) is scaled by a power of two so that its largest element has 55 bits before the binary
// point, rounded to an integer and cut into 7 balanced base-256 digits, each exact in BF16 (|digit| <= 128):
//   A(i, k) = 2^(ea_i - 55) sum_s a_s(i, k) 256^(6 - s),   s = 0 .. 6,
// the largest element of a row exactly, smaller ones to 2^-56 of it.  Before that, column k of A is divided and row k of
// B multiplied by the power of two of the column's largest element: where large elements of A meet small ones of B (the
// separable expansion's weights against J0 - 1) the scales then follow the products; an empty column takes its row of B
// out of the scales.  The digit products of equal weight,
// D_d = sum_k sum_{s + t = d} a_s b_t, d = 0 .. 6, are formed by tcgen05.mma.kind::f16 in FP32 accumulators: over
// kOzDrainK = 128 k and at most 7 digit pairs every partial sum is an integer of at most 128 * 7 * 2^14 < 2^24, so no
// accumulation rounds.  Every 128 k the seven accumulators are drained into two 64-bit integers per output (exact), and
// the only roundings are the slicing, the dropped weights d >= 7 (at most 6 x 2^-56 = 8e-17 of max |row| max |column| per
// term, after the scales; rms about 2^-56) and the final conversion.  The bound is normwise: where a row's large elements
// meet zeros of a column and its small ones carry that output, FP64 FMAs keep more of it.  On the path's data the error is
// about a quarter of what they accumulate (2^-53 of the partial sum per term, half that on average; rms below).
//
// Why: the FP64 pipe does 2 FMA per clock and SM (0.95 TFLOP/s in this engine's SIMT GEMM); 28 digit products of BF16
// are 28 / 4096 of a clock per FP64 FMA.  A k block of 32 takes 2180 clocks, 1792 of them tensor work, with its 84 KB of
// operands from L2 underneath; with few k blocks (the xi groups: 17k of a tile's 44k clocks) the drains, the rounding and
// the set-up take the rest.  Measured (FP64 SIMT before -> with slicing): sep1 3366 x 580 x 6384 25.2 -> 1.01 ms,
// Hankel 3366 x 796 x 2687 11.0 -> 0.53, kappa 2400 x 798 x 3366 13.8 -> 0.57, sep2 3366 x 2687 x 446 6.8 -> 0.40, the xi
// groups (67 GFLOP, K about 300) 70.4 -> 5.0 (6.5 with row-wise scattered stores and FP64 conversions in the epilogue); rms error on such data 6e-17 .. 5e-16 against 6e-16 .. 3e-15.
//
// Layout: operands packed by k_oz_pack as [k block of 32][digit][row][64 B] in the canonical K-major core-matrix
// layout (as tc_gemm.cu), so that one bulk copy moves a tile's digit.  One CTA per 128 x 64 tile: the seven
// accumulators take 7 x 64 TMEM columns.  Digit s of A multiplies digits 0 .. 6 - s of B, which lie one after the other
// in shared memory as one operand of up to 448 columns and land on accumulators s .. 6: two MMAs (256 columns is an
// instruction's most) instead of 7 - s, and A is read that much less often.
// Warps 0-7: drains and epilogue (TMEM lanes 32 (w % 4) .., columns 32 (w / 4) .. of each accumulator); warp 8 lane 0:
// bulk copies; warp 9 lane 0: MMAs.  Every wait is bounded; a wait that runs out raises *err and the CTA frees its TMEM.
#include "kernels.cuh"
#include "tcgen05.cuh"

namespace sgl {

constexpr int kOzS = 7;                        // digits
constexpr int kOzBM = 128, kOzBN = 64, kOzKB = 32;
constexpr int kOzDrain = 4;                    // k blocks per drain (128 k)
constexpr int kOzThreads = 320;
constexpr int kOzStages = 2;
constexpr int kOzABytes = kOzBM * 64, kOzBBytes = kOzBN * 64;               // one digit of a k block
constexpr int kOzStageBytes = kOzS * (kOzABytes + kOzBBytes);               // 84 KB
constexpr int kOzBarOff = kOzStages * kOzStageBytes;
constexpr int kOzNBar = 2 * kOzStages + 3;                                  // full, empty, acc full, acc empty, done
constexpr int kOzSmem = kOzBarOff + 8 * kOzNBar + 32;
constexpr int kOzScaleRows = 256, kOzScaleK = 64;

namespace {

template <typename D, typename F>
__device__ __forceinline__ int find_desc(const D* d, int n, long long v, F begin) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (begin(d[mid]) <= v) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// Scales: the largest biased exponent of a row, each element's first shifted by the k scales' sign * (kexp - 1023), kept as
// kOzBias + exponent (0: a row of zeros); kOzNan: the row holds an infinity or a NaN (its outputs are summed by plain
// FMAs in the epilogue, so that infinities and NaN come out as of an FP64 product).  A k scale is that of the finite
// elements of A's column; where it has none but zeros, row k of B adds nothing to any finite output, so it is cut to zero
// digits and does not enter the scales of B's columns (unscaled, it would push the rows that count out of their digits).
constexpr int kOzBias = 8192, kOzNan = 1 << 20, kOzDead = 1 << 24;

__device__ __forceinline__ int oz_shift(const OzPackDesc& d, const int* scale, int k) {
    if (d.k_sign == 0) return 0;
    const int s = scale[d.k_off + k];
    return s == 0 ? kOzDead : d.k_sign * (s - kOzBias - 1023);
}

__global__ void __launch_bounds__(256) k_oz_scale(const OzPackDesc* __restrict__ descs, int n, int* __restrict__ scale) {
    const long long b = blockIdx.x;
    const OzPackDesc d = descs[find_desc(descs, n, b, [](const OzPackDesc& x) { return x.scale_begin; })];
    const long long local = b - d.scale_begin;
    const int nrb = (d.R + kOzScaleRows - 1) / kOzScaleRows;
    const int r0 = (int)(local % nrb) * kOzScaleRows, k0 = (int)(local / nrb) * kOzScaleK;
    const int k1 = min(d.K, k0 + kOzScaleK);
    auto exponent = [&](double v, int shift) {
        const int e = (__double2hiint(v) >> 20) & 0x7ff;
        if (e == 0x7ff) return d.k_sign == 0 ? 0 : kOzNan;
        return v == 0.0 || shift == kOzDead ? 0 : kOzBias + max(e, 1) + shift;
    };
    __shared__ int s_shift[kOzScaleK];
    for (int k = threadIdx.x; k < k1 - k0; k += 256) s_shift[k] = oz_shift(d, scale, k0 + k);
    __syncthreads();
    if (d.x_rs == 1 || d.x_cs != 1) {                        // consecutive threads, consecutive rows
        const int r = r0 + threadIdx.x;
        if (r >= d.R) return;
        int e = 0;
#pragma unroll 16
        for (int k = k0; k < k1; ++k)
            e = max(e, exponent(d.X[(long long)r * d.x_rs + (long long)k * d.x_cs], s_shift[k - k0]));
        if (e > 0) atomicMax(scale + d.scale_off + r, e);
    } else {                                                  // rows contiguous along k: a warp per row
        const int lane = threadIdx.x & 31;
#pragma unroll 4
        for (int r = r0 + (threadIdx.x >> 5); r < min(d.R, r0 + kOzScaleRows); r += 8) {
            int e = 0;
#pragma unroll 4
            for (int k = k0 + lane; k < k1; k += 32) e = max(e, exponent(d.X[(long long)r * d.x_rs + k], s_shift[k - k0]));
            e = __reduce_max_sync(0xffffffffu, e);
            if (lane == 0 && e > 0) atomicMax(scale + d.scale_off + r, e);
        }
    }
}

// One thread per (row, 8 consecutive k): the seven 16-byte core-matrix rows of BF16 digits.  All integer.
__global__ void __launch_bounds__(256) k_oz_pack(const OzPackDesc* __restrict__ descs, int n, const int* __restrict__ scale,
                                                 unsigned char* __restrict__ packed) {
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const OzPackDesc d = descs[find_desc(descs, n, t, [](const OzPackDesc& x) { return x.quad_begin; })];
    const long long q = t - d.quad_begin;
    if (q >= (long long)d.Rpad * d.nkb * 4) return;
    const int r = (int)(q % d.Rpad);
    const long long rest = q / d.Rpad;
    const int c = (int)(rest % 4), kb = (int)(rest / 4);
    uint32_t w[kOzS][4];
    const int emax = r < d.R ? scale[d.scale_off + r] : 0;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int k = kb * kOzKB + c * 8 + e;
        const double v = (r < d.R && k < d.K) ? __ldg(d.X + (long long)r * d.x_rs + (long long)k * d.x_cs) : 0.0;
        const long long bits = __double_as_longlong(v);
        const int ex = (int)((bits >> 52) & 0x7ff);
        long long m = bits & 0xfffffffffffffLL;
        if (ex > 0) m |= 1LL << 52;
        // to 55 bits for the row's largest exponent
        const int shift = k < d.K ? oz_shift(d, scale, k) : 0;
        const int sh = max(ex, 1) + shift + kOzBias - emax + 2;
        if (m == 0 || emax >= kOzNan || shift == kOzDead) m = 0;
        else if (sh >= 0) m <<= sh;                             // 0 .. 2
        else m = sh < -56 ? 0 : (m + (1LL << (-sh - 1))) >> -sh;
        if (bits < 0) m = -m;
        // balanced digits from the lowest up; the last one takes the carry (|m| <= 2^55: at most 128)
#pragma unroll
        for (int s = kOzS - 1; s >= 0; --s) {
            const int dig = s > 0 ? (int)(signed char)(m & 0xff) : (int)m;
            if (s > 0) m = (m - dig) >> 8;
            // small integers are exact in BF16: the upper half of the float
            const uint32_t f = __float_as_uint(__int_as_float(0x4b400000 + dig) - 12582912.f) >> 16;
            if (e & 1) w[s][e >> 1] |= f << 16; else w[s][e >> 1] = f;
        }
    }
    unsigned char* out = packed + d.out_off + (long long)kb * kOzS * d.Rpad * 64 + (long long)(r >> 3) * 512 + c * 128 + (r & 7) * 16;
#pragma unroll
    for (int s = 0; s < kOzS; ++s)
        *reinterpret_cast<uint4*>(out + (long long)s * d.Rpad * 64) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
}

// hi 2^24 + lo as a double, rounded to nearest even, times 2^(e - 2106): 2^48 of the digits' weights and 2^(e - 1077) of
// the two operands' integers, e their largest biased exponents.  On the integer pipe (an FP64 instruction, 64-bit
// conversions included, holds a scheduler for 64 cycles, also where its result is not selected) and without a branch, so
// that several outputs' chains interleave.  In the rare range outside the normal numbers: the unscaled value, *odd.
__device__ __forceinline__ double oz_value(long long hi, long long lo, int e, bool* odd) {
    // magnitude H 2^24 + L, L < 2^24
    hi += lo >> 24;
    const bool neg = hi < 0;
    unsigned int L = (unsigned int)lo & 0xffffffu;
    unsigned long long H = (unsigned long long)(neg ? ~hi : hi);
    H += neg && L == 0 ? 1 : 0;
    L = neg ? (0x1000000u - L) & 0xffffffu : L;
    const bool low = H == 0;
    H = low ? L : H;
    L = low ? 0u : L;
    const int top = low ? 63 : 87, lz = min(__clzll(H), 63);          // top: exponent of H's bit 63
    const unsigned long long l40 = (unsigned long long)L << 40;
    const unsigned long long x = (H << lz) | ((l40 >> 1) >> (63 - lz));
    const unsigned int rest = (unsigned int)(x & 0x3ff) | (unsigned int)((l40 << lz) != 0);
    unsigned long long m = x >> 11;                                   // 53 bits
    m += ((unsigned int)x >> 10) & ((rest != 0 ? 1u : 0u) | (unsigned int)m) & 1u;
    const int E = top - lz + 1023;                                    // biased exponent before the scale
    int s = e - 2106;
    const bool normal = E + s > 0 && E + s < 0x7fe;
    *odd = !normal && H != 0;
    s = normal ? s : 0;
    const long long v = (((long long)(E + s - 1) << 52) + (long long)m) | (neg ? (long long)(1ULL << 63) : 0);
    return __longlong_as_double(H == 0 ? 0 : v);
}

__device__ __noinline__ double oz_plain_sum(const double* a, long long a_cs, const double* b, long long b_rs, int K) {
    double acc = 0.0;
    for (int k = 0; k < K; ++k) acc = fma(a[(long long)k * a_cs], b[(long long)k * b_rs], acc);
    return acc;
}

__global__ void __launch_bounds__(kOzThreads, 1)
k_oz_gemm(const OzGemmDesc* __restrict__ descs, int nprob, const unsigned char* __restrict__ packed,
          const int* __restrict__ scale, int* __restrict__ err) {
    extern __shared__ __align__(1024) unsigned char tsm[];
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(tsm);
    const uint32_t bar = sbase + kOzBarOff;
    auto full = [&](int s) { return bar + 8 * s; };
    auto empty = [&](int s) { return bar + 8 * (kOzStages + s); };
    const uint32_t accf = bar + 8 * (2 * kOzStages), acce = accf + 8, done = accf + 16;
    const uint32_t tslot = bar + 8 * kOzNBar;
    volatile int* s_fail = (volatile int*)(tsm + kOzBarOff + 8 * kOzNBar + 8);
    volatile int* s_used = (volatile int*)(tsm + kOzBarOff + 8 * kOzNBar + 12);      // k blocks the MMAs took
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tile = blockIdx.x;
    // the last problem that begins at or before the tile: counted by all threads, one round trip to memory
    int before = 0;
    for (int p0 = 0; p0 < nprob; p0 += kOzThreads)
        before += __syncthreads_count(p0 + tid < nprob && descs[p0 + tid].tile_begin <= tile);
    const OzGemmDesc d = descs[before - 1];
    const int local = tile - d.tile_begin;
    const int i0 = (local / d.tiles_n) * kOzBM, j0 = (local % d.tiles_n) * kOzBN;
    const int nkb = (d.K + kOzKB - 1) / kOzKB;
    const int nblk = (nkb + kOzDrain - 1) / kOzDrain;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(tslot), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int s = 0; s < kOzStages; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        mbar_init(accf, 1);
        mbar_init(acce, 8);
        mbar_init(done, 1);
        *s_fail = 0;
        *s_used = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *(volatile uint32_t*)(tsm + kOzBarOff + 8 * kOzNBar);

    int issued = 0;                            // k blocks whose copies the producer issued
    if (warp == 8) {
        if (lane == 0) {
            const long long a_dig = (long long)d.Mpad * 64, b_dig = (long long)d.Npad * 64;
            for (int kb = 0; kb < nkb; ++kb) {
                const int s = kb % kOzStages;
                if (*s_fail || (kb >= kOzStages && !mbar_wait_bounded(empty(s), (uint32_t)(((kb / kOzStages) - 1) & 1)))) {
                    *s_fail = 1;
                    break;
                }
                issued = kb + 1;
                const uint32_t st = sbase + s * kOzStageBytes;
                mbar_expect_tx(full(s), kOzStageBytes);
                const unsigned char* a = packed + d.a_off + (long long)kb * kOzS * a_dig + (long long)i0 * 64;
                const unsigned char* b = packed + d.b_off + (long long)kb * kOzS * b_dig + (long long)j0 * 64;
#pragma unroll
                for (int q = 0; q < kOzS; ++q) {
                    bulk_g2s(st + q * kOzABytes, a + q * a_dig, kOzABytes, full(s));
                    bulk_g2s(st + kOzS * kOzABytes + q * kOzBBytes, b + q * b_dig, kOzBBytes, full(s));
                }
            }
        }
    } else if (warp == 9) {
        if (lane == 0) {
            for (int kb = 0; kb < nkb; ++kb) {
                const int blk = kb / kOzDrain;
                const bool first = kb % kOzDrain == 0;
                if (first && blk >= 1 && (*s_fail || !mbar_wait_bounded(acce, (uint32_t)((blk - 1) & 1)))) { *s_fail = 1; break; }
                const int s = kb % kOzStages;
                if (*s_fail || !mbar_wait_bounded(full(s), (uint32_t)((kb / kOzStages) & 1))) { *s_fail = 1; break; }
                *s_used = kb + 1;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a0 = sbase + s * kOzStageBytes, b0 = a0 + kOzS * kOzABytes;
#pragma unroll
                for (int ks = 0; ks < 2; ++ks) {
                    const uint32_t o = ks * 2 * kTcLBO;
#pragma unroll
                    for (int q = 0; q < kOzS; ++q) {
                        // digit q of A with digits 0 .. 6 - q of B, at most four (256 columns) per instruction;
                        // q = 0 touches every accumulator first
                        const uint32_t acc = (first && ks == 0 && q == 0) ? 0u : 1u;
                        constexpr int kMax = 256 / kOzBN;
                        const int nb = kOzS - q, n0 = nb < kMax ? nb : kMax;
                        tc_mma_bf16(tmem + q * kOzBN, tc_desc(a0 + q * kOzABytes + o), tc_desc(b0 + o),
                                    tc_idesc_bf16(kOzBM, n0 * kOzBN), acc);
                        if (nb > kMax)
                            tc_mma_bf16(tmem + (q + kMax) * kOzBN, tc_desc(a0 + q * kOzABytes + o),
                                        tc_desc(b0 + kMax * kOzBBytes + o), tc_idesc_bf16(kOzBM, (nb - kMax) * kOzBN), acc);
                    }
                }
                tc_commit(empty(s));
                if (kb % kOzDrain == kOzDrain - 1 || kb == nkb - 1) tc_commit(accf);
            }
            tc_commit(done);                   // every MMA issued above has completed before TMEM is freed
            if (!mbar_wait_bounded(done, 0u)) *s_fail = 1;
        }
    } else {
        // hi = sum_d<4 D_d 256^(3 - d), lo = sum_d>=4 D_d 256^(6 - d): 64-bit integers per output
        constexpr int kCols = kOzBN / 2;
        static_assert(kCols == 32, "a lane per column of a warp's outputs");
        long long hi[kCols], lo[kCols];
#pragma unroll
        for (int c = 0; c < kCols; ++c) { hi[c] = 0; lo[c] = 0; }
        const uint32_t base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * kCols);
        bool ok = true;
        for (int blk = 0; blk < nblk && ok; ++blk) {
            ok = warp_all(!*s_fail && mbar_wait_bounded(accf, (uint32_t)(blk & 1)));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int c0 = 0; c0 < kCols; c0 += 16) {
#pragma unroll
                for (int dd = 0; dd < kOzS; ++dd) {
                    float v[16];
                    tmem_ld16(base + (uint32_t)(dd * kOzBN + c0), v);
#pragma unroll
                    for (int x = 0; x < 16; ++x) {
                        const long long p = (long long)__float2int_rn(v[x]);
                        if (dd < 4) hi[c0 + x] += p * (1 << (8 * (3 - dd)));
                        else lo[c0 + x] += p * (1 << (8 * (6 - dd)));
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(acce);
        }
        if (!ok) *s_fail = 1;
        // through shared memory (the stages are free: every product has been taken), each warp its own 32 rows, so that
        // C is written, and read for beta, along its rows
        if (ok) {
            const int r0 = i0 + (warp & 3) * 32, j = j0 + (warp >> 2) * kCols + lane;
            double* s_out = (double*)tsm + warp * 32 * (kCols + 1);
            const int ea = r0 + lane < d.M ? scale[d.sa_off + r0 + lane] : 0;
            const int ebs = j < d.N ? scale[d.sb_off + j] : 0;
            uint32_t odd = 0;                                        // outputs left unscaled, a bit per column
#pragma unroll
            for (int c = 0; c < kCols; ++c) {
                bool o;
                s_out[lane * (kCols + 1) + c] = oz_value(hi[c], lo[c], ea + __shfl_sync(0xffffffffu, ebs, c) - 2 * kOzBias, &o);
                odd |= (uint32_t)o << c;
            }
            if (__any_sync(0xffffffffu, odd != 0 || ea >= kOzNan || ebs >= kOzNan))
                for (int c = 0; c < kCols; ++c) {
                    const int eb = __shfl_sync(0xffffffffu, ebs, c);
                    double* o = s_out + lane * (kCols + 1) + c;
                    if (odd >> c & 1) *o = scalbn(*o, ea + eb - 2 * kOzBias - 2106);
                    // an infinity or a NaN in the row or the column: the sum of products as FP64 FMAs form it
                    const int jc = j - lane + c;
                    if ((ea >= kOzNan || eb >= kOzNan) && r0 + lane < d.M && jc < d.N)
                        *o = oz_plain_sum(d.A + (long long)(r0 + lane) * d.a_rs, d.a_cs, d.B + (long long)jc * d.b_cs, d.b_rs, d.K);
                }
            __syncwarp();
            const int nr = j < d.N ? min(32, d.M - r0) : 0;
            double* C = d.C + (long long)r0 * d.ldc + j;
            if (d.alpha == 1.0 && d.beta == 0.0) {
                // a loop of its own: FP64 instructions whose results are not selected take their 64 cycles all the same
#pragma unroll 8
                for (int r = 0; r < nr; ++r) C[r * d.ldc] = s_out[r * (kCols + 1) + lane];
            } else {
                for (int rb = 0; rb < nr; rb += 8) {                 // eight rows' loads in flight
                    double c[8];
#pragma unroll
                    for (int r = 0; r < 8; ++r) c[r] = d.beta != 0.0 && rb + r < nr ? C[(rb + r) * d.ldc] : 0.0;
#pragma unroll
                    for (int r = 0; r < 8; ++r) {
                        const double v = d.alpha * s_out[(rb + r) * (kCols + 1) + lane];
                        if (rb + r < nr) C[(rb + r) * d.ldc] = d.beta != 0.0 ? fma(d.beta, c[r], v) : v;
                    }
                }
            }
        }
    }
    // the MMAs have completed (the issuer waited on its final commit); after a failure no bulk copy
    // may outlive the CTA: the producer waits (bounded) for the copies the MMAs never took
    __syncthreads();
    if (*s_fail && warp == 8 && lane == 0)
        for (int kb = *s_used; kb < issued; ++kb) mbar_wait_bounded(full(kb % kOzStages), (uint32_t)((kb / kOzStages) & 1));
    if (*s_fail && tid == 0) atomicExch(err, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(512) : "memory");
    }
}

}  // namespace

// pk: 2 n operands, then n columns of A (for the k scales)
void oz_gemm_plan(OzGemmDesc* d, int n, OzPackDesc* pk, OzPlan* out) {
    OzPlan P{};
    for (int i = 0; i < n; ++i) {
        OzGemmDesc& g = d[i];
        g.tiles_n = (g.N + kOzBN - 1) / kOzBN;
        g.tile_begin = P.tiles;
        P.tiles += g.tiles_n * ((g.M + kOzBM - 1) / kOzBM);
        const int nkb = (g.K + kOzKB - 1) / kOzKB;
        g.Mpad = (g.M + kOzBM - 1) / kOzBM * kOzBM;
        g.Npad = g.tiles_n * kOzBN;
        g.a_off = P.bytes;
        P.bytes += (long long)nkb * kOzS * g.Mpad * 64;
        g.b_off = P.bytes;
        P.bytes += (long long)nkb * kOzS * g.Npad * 64;
        g.sa_off = P.scales;
        P.scales += g.M;
        g.sb_off = P.scales;
        P.scales += g.N;
        const int k_off = P.scales;
        P.scales += g.K;
        OzPackDesc& pc = pk[2 * n + i];
        pc = OzPackDesc{};
        pc.X = g.A; pc.x_rs = g.a_cs; pc.x_cs = g.a_rs;
        pc.R = g.K; pc.K = g.M;
        pc.scale_off = k_off;
        pc.scale_begin = P.k_ctas;
        P.k_ctas += (long long)((pc.R + kOzScaleRows - 1) / kOzScaleRows) * ((pc.K + kOzScaleK - 1) / kOzScaleK);
        for (int b = 0; b < 2; ++b) {
            OzPackDesc& p = pk[2 * i + b];                    // A(i, k): rows i; B(k, j): rows j
            p.X = b ? g.B : g.A;
            p.x_rs = b ? g.b_cs : g.a_rs;
            p.x_cs = b ? g.b_rs : g.a_cs;
            p.R = b ? g.N : g.M;
            p.K = g.K;
            p.Rpad = b ? g.Npad : g.Mpad;
            p.nkb = nkb;
            p.out_off = b ? g.b_off : g.a_off;
            p.scale_off = b ? g.sb_off : g.sa_off;
            p.k_off = k_off;
            p.k_sign = b ? 1 : -1;
            p.quad_begin = P.quads;
            P.quads += 4LL * p.Rpad * nkb;
            p.scale_begin = P.scale_ctas;
            P.scale_ctas += (long long)((p.R + kOzScaleRows - 1) / kOzScaleRows) * ((p.K + kOzScaleK - 1) / kOzScaleK);
        }
    }
    *out = P;
}

void launch_oz_gemm(const OzGemmDesc* d_descs, int n, const OzPackDesc* d_pack, const OzPlan& P, unsigned char* packed,
                    int* scale, int* err, cudaStream_t st) {
    cudaMemsetAsync(scale, 0, sizeof(int) * (size_t)P.scales, st);
    k_oz_scale<<<(unsigned)P.k_ctas, 256, 0, st>>>(d_pack + 2 * n, n, scale);
    k_oz_scale<<<(unsigned)P.scale_ctas, 256, 0, st>>>(d_pack, 2 * n, scale);
    k_oz_pack<<<(unsigned)ceil_div(P.quads, 256), 256, 0, st>>>(d_pack, 2 * n, scale, packed);
    cudaFuncSetAttribute(k_oz_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, kOzSmem);
    k_oz_gemm<<<P.tiles, kOzThreads, kOzSmem, st>>>(d_descs, n, packed, scale, err);
    SGL_COUNT(4);
}

}  // namespace sgl
