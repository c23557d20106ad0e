// Element-wise kernels of the per-plane log-CF surrogate MLP (BF16 tensor-core GEMMs are in
// tc_gemm.cu): bias + SiLU forward, SiLU backward, column sums for the bias gradients, MSE loss
// gradient and AdamW.  FP32 storage, FP64 for the reductions.
#include "kernels.cuh"

namespace sgl {

// Zb = Z + bias[col]; A = silu(Zb) (or Zb when silu = 0)
__global__ void k_bias_act(int M, int N, const float* __restrict__ Z, const float* __restrict__ bias,
                           float* __restrict__ Zb, float* __restrict__ A, int silu) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long long)M * N) return;
    const float z = Z[e] + bias[e % N];
    Zb[e] = z;
    A[e] = silu ? z / (1.f + expf(-z)) : z;
}

// dZ = dA * silu'(Zb),  silu'(z) = s (1 + z (1 - s)),  s = 1 / (1 + e^-z)
__global__ void k_act_grad(int M, int N, const float* __restrict__ dA, const float* __restrict__ Zb,
                           float* __restrict__ dZ) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long long)M * N) return;
    const float z = Zb[e];
    const float sg = 1.f / (1.f + expf(-z));
    dZ[e] = dA[e] * sg * (1.f + z * (1.f - sg));
}

// out[j] = sum_i X[i, j] in FP64.  Up to kColDirect rows: one CTA per column, its reads N apart but in L2 (the operand was
// just written).  Above: a CTA per (128 columns, 64 rows) adds its rows column by column (coalesced), and a second pass the
// CTAs' sums in order.  Per call, direct / two passes in us: 64 x 256 4.6 / 12.8, 4096 x 256 10.6 / 14.0, 16384 x 256 23 / 28,
// 20 x 5000 19 / 25, 100000 x 256 259 / 111, 300000 x 8 269 / 59, 1000000 x 2 854 / 147.
constexpr int kColRows = 64, kColDirect = 1 << 15;
__global__ void __launch_bounds__(128) k_col_part(int M, int N, int rows, const float* __restrict__ X, double* __restrict__ part) {
    const int j = blockIdx.x * 128 + threadIdx.x;
    if (j >= N) return;
    const int i0 = min((long long)M, (long long)blockIdx.y * rows), i1 = min((long long)M, (long long)i0 + rows);
    double a0 = 0.0, a1 = 0.0;
    int i = i0;
#pragma unroll 4
    for (; i + 1 < i1; i += 2) {
        a0 += (double)X[(long long)i * N + j];
        a1 += (double)X[(long long)(i + 1) * N + j];
    }
    if (i < i1) a0 += (double)X[(long long)i * N + j];
    part[(long long)blockIdx.y * N + j] = a0 + a1;
}

template <typename T>
__global__ void __launch_bounds__(256) k_col_sum(int M, int N, const T* __restrict__ X, float* __restrict__ out) {
    __shared__ double sh[32];
    const int j = blockIdx.x;
    double a = 0.0;
    for (int i = threadIdx.x; i < M; i += blockDim.x) a += (double)X[(long long)i * N + j];
    a = block_sum(a, sh);
    if (threadIdx.x == 0) out[j] = (float)a;
}

// dpred = 2 (pred - target) / n; partial sums of (pred - target)^2 per CTA
__global__ void __launch_bounds__(256) k_mse(long long n, const float* __restrict__ pred, const float* __restrict__ tgt,
                                             float* __restrict__ dpred, double* __restrict__ part) {
    __shared__ double sh[32];
    double a = 0.0;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x) {
        const float d = pred[e] - tgt[e];
        dpred[e] = 2.f * d / (float)n;
        a += (double)d * d;
    }
    a = block_sum(a, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = a;
}

// AdamW (decoupled weight decay), bias-corrected moments
__global__ void k_adamw(long long n, float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                        float* __restrict__ v, float lr, float b1, float b2, float eps, float wd, float c1, float c2) {
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n) return;
    const float gr = g[e];
    const float mm = b1 * m[e] + (1.f - b1) * gr;
    const float vv = b2 * v[e] + (1.f - b2) * gr * gr;
    m[e] = mm;
    v[e] = vv;
    w[e] = w[e] - lr * (mm / c1 / (sqrtf(vv / c2) + eps) + wd * w[e]);
}

void launch_bias_act(int M, int N, const float* Z, const float* bias, float* Zb, float* A, int silu, cudaStream_t st) {
    const long long t = (long long)M * N;
    if (t > 0) { k_bias_act<<<ceil_div(t, 256), 256, 0, st>>>(M, N, Z, bias, Zb, A, silu); SGL_COUNT(1); }
}
void launch_act_grad(int M, int N, const float* dA, const float* Zb, float* dZ, cudaStream_t st) {
    const long long t = (long long)M * N;
    if (t > 0) { k_act_grad<<<ceil_div(t, 256), 256, 0, st>>>(M, N, dA, Zb, dZ); SGL_COUNT(1); }
}
static int col_sum_rows(int M) { return std::max(kColRows, ceil_div(M, 65535)); }      // rows per CTA: grid.y <= 65535
long long col_sum_parts(int M, int N) { return M <= kColDirect ? 0 : (long long)ceil_div(M, col_sum_rows(M)) * N; }
void launch_col_sum(int M, int N, const float* X, double* part, float* out, cudaStream_t st) {
    if (N <= 0) return;
    if (M <= kColDirect) { k_col_sum<<<N, 256, 0, st>>>(M, N, X, out); SGL_COUNT(1); return; }
    const int rows = col_sum_rows(M), np = ceil_div(M, rows);
    k_col_part<<<dim3(ceil_div(N, 128), np), 128, 0, st>>>(M, N, rows, X, part);
    k_col_sum<<<N, 256, 0, st>>>(np, N, part, out);
    SGL_COUNT(2);
}
int mse_blocks(long long n) { return (int)std::min<long long>(1024, std::max<long long>(1, ceil_div(n, 256))); }
void launch_mse(long long n, const float* pred, const float* tgt, float* dpred, double* part, cudaStream_t st) {
    k_mse<<<mse_blocks(n), 256, 0, st>>>(n, pred, tgt, dpred, part);
    SGL_COUNT(1);
}
void launch_adamw(long long n, float* w, const float* g, float* m, float* v, float lr, float b1, float b2, float eps,
                  float wd, float c1, float c2, cudaStream_t st) {
    if (n > 0) { k_adamw<<<ceil_div(n, 256), 256, 0, st>>>(n, w, g, m, v, lr, b1, b2, eps, wd, c1, c2); SGL_COUNT(1); }
}

}  // namespace sgl
