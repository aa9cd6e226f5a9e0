// Plain matrix products  Y[M,N] = X[M,K] * W[N,K]^T  (both operands K-major, as every weight of
// the model is stored: [out_features, in_features]; the reference's GEMM wrapper has the same
// contract, src/model/llama.cpp:45-52).
//
// * bfloat16 operands with float accumulation: the plain twin that the fast bfloat16 kernels are checked
//   against; Y may be float or bfloat16.  Every output element is accumulated over k in ascending order by
//   one thread, so a row's result does not depend on how many other rows are in the batch.
// * batches of small products (one per head, say) of either type.
// Single products of float operands (the true 32-bit path) are gemm_f32.cu.
#include "common.cuh"
#include "pdl.cuh"

namespace kvcm {

constexpr int TM = 64, TN = 64, TK = 16;   // block tile; 256 threads, each a 4x4 micro-tile

template <typename TIn, typename TOut>
__global__ void __launch_bounds__(256)
gemm_plain_kernel(const TIn* __restrict__ X, const TIn* __restrict__ W, TOut* __restrict__ Y,
                  int M, int N, int K, int ldx, int ldw, int ldy, long long bx, long long bw, long long by) {
  // blockIdx.z: one product of a batch whose operands lie bx / bw / by elements apart
  X += blockIdx.z * bx;
  W += blockIdx.z * bw;
  Y += blockIdx.z * by;
  __shared__ float xs[TK][TM + 1];
  __shared__ float ws[TK][TN + 1];
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  float acc[4][4] = {};
  for (int k0 = 0; k0 < K; k0 += TK) {
    for (int i = threadIdx.x; i < TM * TK; i += 256) {
      const int r = i / TK, c = i % TK;
      const int gm = m0 + r, gk = k0 + c;
      xs[c][r] = (gm < M && gk < K) ? ldf(X + size_t(gm) * ldx + gk) : 0.f;
    }
    for (int i = threadIdx.x; i < TN * TK; i += 256) {
      const int r = i / TK, c = i % TK;
      const int gn = n0 + r, gk = k0 + c;
      ws[c][r] = (gn < N && gk < K) ? ldf(W + size_t(gn) * ldw + gk) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < TK; ++k) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = xs[k][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = ws[k][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + ty * 4 + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tx * 4 + j;
      if (gn < N) stf(Y + size_t(gm) * ldy + gn, acc[i][j]);
    }
  }
}

// A batch of products of a handful of rows (decode): one warp per output column n of one product,
// the lanes stride over k with float FMAs in a fixed order, at most 16 rows at a time.  The rows of
// X (for this product) are staged in shared memory as floats.
constexpr int kFewRows = 16;

template <typename T>
__global__ void __launch_bounds__(256)
gemm_few_rows_kernel(const T* X, const T* W, T* __restrict__ Y, int M, int N, int K,
                     int ldx, int ldw, int ldy, long long bx, long long bw, long long by) {
  pdl_launch_dependents();
  pdl_wait();
  extern __shared__ float xrows[];                 // [M][K]
  X += blockIdx.z * bx;
  W += blockIdx.z * bw;
  Y += blockIdx.z * by;
  for (int i = threadIdx.x; i < M * K; i += blockDim.x) xrows[i] = ldf(X + size_t(i / K) * ldx + i % K);
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = blockIdx.x * (blockDim.x >> 5) + warp;
  if (n >= N) return;
  float acc[kFewRows];
#pragma unroll
  for (int m = 0; m < kFewRows; ++m) acc[m] = 0.f;
  const T* wn = W + size_t(n) * ldw;
  for (int k = lane; k < K; k += 32) {
    const float w = ldf(wn + k);
#pragma unroll
    for (int m = 0; m < kFewRows; ++m)
      if (m < M) acc[m] = fmaf(xrows[m * K + k], w, acc[m]);
  }
#pragma unroll
  for (int m = 0; m < kFewRows; ++m) {
    if (m >= M) break;
    const float a = warp_sum(acc[m]);
    if (lane == 0) stf(Y + size_t(m) * ldy + n, a);
  }
}

template <typename TIn, typename TOut>
int launch_gemm_plain(const void* X, const void* W, void* Y, int M, int N, int K, int ldx, int ldw,
                      int ldy, cudaStream_t s, int batch = 1, long long bx = 0, long long bw = 0, long long by = 0) {
  if (M == 0 || N == 0 || batch == 0) return 0;
  if (batch < 0 || batch > 65535) return KVCM_ERR_UNSUPPORTED;
  dim3 grid((N + TN - 1) / TN, (M + TM - 1) / TM, batch);
  gemm_plain_kernel<TIn, TOut><<<grid, 256, 0, s>>>((const TIn*)X, (const TIn*)W, (TOut*)Y, M, N, K,
                                                    ldx, ldw, ldy, bx, bw, by);
  return KVCM_LAUNCH_RESULT();
}

}  // namespace kvcm

using namespace kvcm;

KVCM_API int kvcm_gemm_plain_bf16(const void* X, const void* W, void* Y, int M, int N, int K, int ldx,
                                  int ldw, int ldy, void* stream) {
  return launch_gemm_plain<bf16, bf16>(X, W, Y, M, N, K, ldx, ldw, ldy, (cudaStream_t)stream);
}
KVCM_API int kvcm_gemm_plain_bf16_f32out(const void* X, const void* W, void* Y, int M, int N, int K,
                                         int ldx, int ldw, int ldy, void* stream) {
  return launch_gemm_plain<bf16, float>(X, W, Y, M, N, K, ldx, ldw, ldy, (cudaStream_t)stream);
}

// A batch of such products in one launch (one per head, say): product z reads X + z*bx and
// W + z*bw and writes Y + z*by (element counts); rows ldx / ldw / ldy apart as above.
template <typename T>
int launch_gemm_few_rows(const void* X, const void* W, void* Y, int M, int N, int K, int ldx, int ldw, int ldy, int batch,
                         long long bx, long long bw, long long by, cudaStream_t s) {
  const size_t smem = size_t(M) * K * sizeof(float);
  return pdl_launch(gemm_few_rows_kernel<T>, dim3((N + 7) / 8, 1, batch), dim3(256), smem, s, (const T*)X, (const T*)W, (T*)Y, M,
                    N, K, ldx, ldw, ldy, bx, bw, by);
}
static bool few_rows(int M, int N, int K, int batch) {
  return M >= 1 && M <= kFewRows && size_t(M) * K * sizeof(float) <= 48 * 1024 && batch >= 1 && batch <= 65535 && N >= 1;
}

KVCM_API int kvcm_gemm_plain_batched_f32(const void* X, const void* W, void* Y, int M, int N, int K, int ldx, int ldw,
                                         int ldy, int batch, long long bx, long long bw, long long by, void* stream) {
  if (few_rows(M, N, K, batch))
    return launch_gemm_few_rows<float>(X, W, Y, M, N, K, ldx, ldw, ldy, batch, bx, bw, by, (cudaStream_t)stream);
  return launch_gemm_plain<float, float>(X, W, Y, M, N, K, ldx, ldw, ldy, (cudaStream_t)stream, batch, bx, bw, by);
}
KVCM_API int kvcm_gemm_plain_batched_bf16(const void* X, const void* W, void* Y, int M, int N, int K, int ldx, int ldw,
                                          int ldy, int batch, long long bx, long long bw, long long by, void* stream) {
  if (few_rows(M, N, K, batch))
    return launch_gemm_few_rows<bf16>(X, W, Y, M, N, K, ldx, ldw, ldy, batch, bx, bw, by, (cudaStream_t)stream);
  return launch_gemm_plain<bf16, bf16>(X, W, Y, M, N, K, ldx, ldw, ldy, (cudaStream_t)stream, batch, bx, bw, by);
}
