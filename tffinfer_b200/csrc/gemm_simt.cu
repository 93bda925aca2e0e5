// C[M, N] = A[M, K] * W[N, K]^T (+ residual) of bfloat16 operands that the tensor-core products do not take (K no multiple of 8,
// unaligned rows), accumulated in float32 with plain FMAs.
// Every output element adds its K products in the order k = 0 .. K-1, so its value does not depend on M, on the tile it
// falls in, or on what else is in the batch.  (The products of bfloat16 elements are exact, so a chain of FMAs is off by its sums'
// roundings alone, 1.1e-7 at K = 256 and 1.6e-7 at 512 in the 2-norm; through gemm_f32.cu, whose sums are cut off, by 2.3e-7.)
#include "common.cuh"

namespace {

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;   // 256 threads, 4x4 outputs each

template <typename TC>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const bf16* __restrict__ A, const bf16* __restrict__ W, TC* C, const float* residual, int M, int N, int K) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;          // tx -> N, ty -> M
    const int tiles_n = (N + BN - 1) / BN;
    const int m0 = blockIdx.x / tiles_n * BM, n0 = blockIdx.x % tiles_n * BN;
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        // 64 rows x 16 k per operand = 1024 elements, 4 per thread
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int idx = tid + e * 256;
            const int r = idx / BK, kk = idx % BK;
            const int gk = k0 + kk;
            float a = 0.f, w = 0.f;
            if (gk < K) {
                if (m0 + r < M) a = to_f32<bf16>(A[(size_t)(m0 + r) * K + gk]);
                if (n0 + r < N) w = to_f32<bf16>(W[(size_t)(n0 + r) * K + gk]);
            }
            As[kk][r] = a;
            Ws[kk][r] = w;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = Ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (residual) v = residual[(size_t)m * N + n] + v;
            C[(size_t)m * N + n] = from_f32<TC>(v);
        }
    }
}

template <typename TC>
int launch(const void* A, const void* W, void* C, const float* residual, int M, int N, int K, cudaStream_t s) {
    const long long tiles = (long long)((N + BN - 1) / BN) * ((M + BM - 1) / BM);
    if (tiles >= (1ll << 31)) return TFF_ERR_UNSUPPORTED;
    gemm_simt_kernel<TC><<<(unsigned)tiles, 256, 0, s>>>((const bf16*)A, (const bf16*)W, (TC*)C, residual, M, N, K);
    return tff_launch_status();
}

}  // namespace

// c_dt: 0 = float32, 1 = bfloat16.  ``residual`` (float32 [M, N], may alias C
// when C is float32) is added to the product when it is not null.
TFF_API int tff_gemm_simt(const void* A, const void* W, void* C, int c_dt, const float* residual, int M, int N, int K,
                          cudaStream_t stream) {
    if (M <= 0 || N <= 0) return TFF_OK;
    if (K <= 0 || (c_dt & ~1)) return TFF_ERR_BAD_ARGUMENT;
    return c_dt ? launch<bf16>(A, W, C, residual, M, N, K, stream) : launch<float>(A, W, C, residual, M, N, K, stream);
}
