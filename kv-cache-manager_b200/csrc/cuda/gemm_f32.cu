// Products of the true 32-bit path:  Y[M,N] = X[M,K] W[N,K]^T, float operands, float FMAs only (no tensor
// cores, no reduced-precision mode).
//
// One order of summation for every size, so that a row's result does not depend on how many rows are beside it:
// K is cut into S contiguous segments (S from K alone: segments()); within a segment the even and the odd k are
// two chains of FMAs in ascending order, whose sums are added; the segments' sums are added in ascending order.
// Shorter chains than one over the whole of K, so the error is smaller too.
//
// What bounds it: a handful of rows reads every weight once (DRAM); many rows are bound by the FMA pipes.
// * The S segments of an output tile are the S blocks of a cluster: even a 2048 x 2048 product of two rows is
//   256 blocks, and the partial tiles meet in distributed shared memory, without scratch in global memory.
// * Operands come in by 16-byte asynchronous copies into a ring of stages of 32 k's, rows 36 floats apart
//   (conflict-free 16-byte reads of 8 consecutive rows); unaligned operands by 4-byte copies, the same sums.
// * The even and the odd chain are the halves of one packed FMA (fma.rn.f32x2): a 16-byte read is its operand
//   pair as it lies, and the issue slots needed are halved.
// * The weights of the first stages are requested before the dependency wait where the caller vouches for them.
// * A thread's addresses are formed once: a few warps an SM run the copies, and their instructions were the bound.
// Measured on B200 at the 1.1B shape, W [11264, 2048]: 2 rows 21 us (4.3 TB/s of weights; 35 us with the addresses formed
// piece by piece), 600 rows 688 us (40 TFLOP/s).  Before, one block per 64 x 64 outputs walked the whole of K, whatever the
// number of rows: 370 to 1,200 us a product of this model at 2 to 130 rows.  Error against 64 bits over a run of two
// prompts of 64 tokens, 8 steps and their score: 2.6e-6 before, 7.3e-7 now.
#include <cooperative_groups.h>

#include "common.cuh"
#include "pdl.cuh"

namespace kvcm {

constexpr int kF32K = 32, kF32Pitch = kF32K + 4;
constexpr int kF32MaxSegments = 8;

__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float halves_sum(unsigned long long v) {
  return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32));
}
template <int BYTES>
__device__ __forceinline__ void copy_async(float* dst, const float* src, bool valid) {      // zeros where not valid
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(valid ? 16 : 0));
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(d), "l"(src), "r"(valid ? 4 : 0));
}

// A block: BM x BN outputs of one segment; a thread TM x TN of them, BM/TM and BN/TN apart; a warp spans LN
// columns and 32/LN rows.
template <int BM_, int BN_, int TM_, int TN_, int LN_, int STAGES_>
struct F32Tile {
  static constexpr int BM = BM_, BN = BN_, TM = TM_, TN = TN_, LN = LN_, STAGES = STAGES_;
  static constexpr int THREADS = (BM / TM) * (BN / TN);
  static constexpr int SMEM = STAGES * (BM + BN) * kF32Pitch * int(sizeof(float));
  static_assert(THREADS % 32 == 0 && (BN / TN) % LN == 0 && (BM / TM) % (32 / LN) == 0, "warps tile the block");
  static_assert(BM * BN <= STAGES * (BM + BN) * kF32Pitch, "the partial tile fits into the stages");
};

template <typename C, bool VEC>
__global__ void __launch_bounds__(C::THREADS)
gemm_f32_kernel(const float* X, const float* __restrict__ W, float* __restrict__ Y, int M, int N, int K,
                int ldx, int ldw, int ldy, int S, int seg, int mtiles, int weights_ready) {
  extern __shared__ __align__(16) float f32_smem[];
  constexpr int BM = C::BM, BN = C::BN, TM = C::TM, TN = C::TN, STAGES = C::STAGES;
  constexpr int STAGE = (BM + BN) * kF32Pitch;
  constexpr int PIECE = VEC ? 4 : 1, PIECES = kF32K / PIECE;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = blockIdx.x % S, tile = blockIdx.x / S;
  const int m0 = (tile % mtiles) * BM, n0 = (tile / mtiles) * BN;
  const int k0 = min(rank * seg, K), k1 = min(k0 + seg, K);
  const int steps = (k1 - k0 + kF32K - 1) / kF32K;

  // This thread's piece of a row of a stage, and every RSTEP-th row from r0 on: addresses are formed once.
  constexpr int RSTEP = C::THREADS / PIECES;
  static_assert(C::THREADS % PIECES == 0 && BN % RSTEP == 0 && (BM % RSTEP == 0 || BM < RSTEP), "copies tile the stage");
  const int r0 = tid / PIECES, c0 = (tid % PIECES) * PIECE;
  const float* const w_from = W + size_t(n0 + r0) * ldw + k0 + c0;
  const float* const x_from = X + size_t(m0 + r0) * ldx + k0 + c0;
  const size_t w_rstep = size_t(RSTEP) * ldw, x_rstep = size_t(RSTEP) * ldx;
  const int w_live = N - n0 - r0, x_live = M - m0 - r0;           // rows i * RSTEP below these exist
  const auto load_w = [&](int step) {
    const bool in = k0 + step * kF32K + c0 < k1;
    float* dst = f32_smem + (step % STAGES) * STAGE + (BM + r0) * kF32Pitch + c0;
#pragma unroll
    for (int i = 0; i < BN / RSTEP; ++i) {
      const bool ok = in && i * RSTEP < w_live;
      copy_async<PIECE * 4>(dst + i * RSTEP * kF32Pitch, ok ? w_from + i * w_rstep + step * kF32K : W, ok);
    }
  };
  const auto load_x = [&](int step) {
    const bool in = k0 + step * kF32K + c0 < k1;
    float* dst = f32_smem + (step % STAGES) * STAGE + r0 * kF32Pitch + c0;
    if (BM % RSTEP != 0 && r0 >= BM) return;
#pragma unroll
    for (int i = 0; i < (BM + RSTEP - 1) / RSTEP; ++i) {
      const bool ok = in && i * RSTEP < x_live;
      copy_async<PIECE * 4>(dst + i * RSTEP * kF32Pitch, ok ? x_from + i * x_rstep + step * kF32K : X, ok);
    }
  };

  pdl_launch_dependents();
  if (!weights_ready) pdl_wait();
  for (int s = 0; s < STAGES - 1 && s < steps; ++s) load_w(s);
  if (weights_ready) pdl_wait();
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < steps) load_x(s);
    asm volatile("cp.async.commit_group;\n");
  }

  constexpr int WARPS_N = (BN / TN) / C::LN;
  const int tn = (warp % WARPS_N) * C::LN + lane % C::LN, tm = (warp / WARPS_N) * (32 / C::LN) + lane / C::LN;
  unsigned long long acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
    __syncthreads();                                  // this stage has landed; everyone is done with the one before
    if (step + STAGES - 1 < steps) { load_w(step + STAGES - 1); load_x(step + STAGES - 1); }
    asm volatile("cp.async.commit_group;\n");
    const float* xs = f32_smem + (step % STAGES) * STAGE + tm * kF32Pitch;
    const float* ws = f32_smem + (step % STAGES) * STAGE + (BM + tn) * kF32Pitch;
#pragma unroll
    for (int k = 0; k < kF32K; k += 4) {
      ulonglong2 a[TM];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(xs + i * (BM / TM) * kF32Pitch + k);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(ws + j * (BN / TN) * kF32Pitch + k);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
          fma2(acc[i][j], a[i].x, b.x);
          fma2(acc[i][j], a[i].y, b.y);
        }
      }
    }
  }
  if (S == 1) {
#pragma unroll
    for (int i = 0; i < TM; ++i) {
      const int m = m0 + tm + i * (BM / TM);
#pragma unroll
      for (int j = 0; j < TN; ++j) {
        const int n = n0 + tn + j * (BN / TN);
        if (m < M && n < N) Y[size_t(m) * ldy + n] = halves_sum(acc[i][j]);
      }
    }
    return;
  }
  // the segments' sums meet in shared memory; block r of the cluster adds up and writes the r-th part of the tile
  asm volatile("cp.async.wait_group 0;\n");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) f32_smem[(tm + i * (BM / TM)) * BN + tn + j * (BN / TN)] = halves_sum(acc[i][j]);
  const auto cluster = cooperative_groups::this_cluster();
  cluster.sync();
  const int part = BM * BN / S;
  for (int e = rank * part + tid; e < (rank + 1) * part; e += C::THREADS) {
    const int m = m0 + e / BN, n = n0 + e % BN;
    if (m >= M || n >= N) continue;
    float v[kF32MaxSegments];
#pragma unroll
    for (int r = 0; r < kF32MaxSegments; ++r) v[r] = r < S ? *cluster.map_shared_rank(f32_smem + e, r) : 0.f;
    float sum = v[0];
#pragma unroll
    for (int r = 1; r < kF32MaxSegments; ++r)
      if (r < S) sum += v[r];
    Y[size_t(m) * ldy + n] = sum;
  }
  cluster.sync();                                     // nobody leaves while its tile is being read
}

// Segments of K: from K alone.  A segment has at least 128 k's, or the cluster costs more than it splits.
static int segments(int K) { return K >= 1024 ? 8 : K >= 512 ? 4 : K >= 256 ? 2 : 1; }

template <typename C, bool VEC>
static int launch_tile(const float* X, const float* W, float* Y, int M, int N, int K, int ldx, int ldw, int ldy, int weights_ready,
                       cudaStream_t s) {
  static OncePerDevice once;
  const int rc = allow_shared_memory(once, gemm_f32_kernel<C, VEC>, C::SMEM);
  if (rc) return rc;
  const int S = segments(K), seg = ((K + S - 1) / S + 3) / 4 * 4;
  const long long mtiles = (M + C::BM - 1) / C::BM, blocks = mtiles * ((N + C::BN - 1) / C::BN) * S;
  if (blocks > 0x7fffffffll) return KVCM_ERR_UNSUPPORTED;
  return pdl_launch_cluster(gemm_f32_kernel<C, VEC>, dim3(unsigned(blocks)), dim3(C::THREADS), C::SMEM, s, S, X, W, Y, M, N, K,
                            ldx, ldw, ldy, S, seg, int(mtiles), weights_ready);
}

// Which tile.  Up to 16 rows read the weights once: a narrow N leaves few blocks, which then take small tiles and deep
// rings; a wide N makes more blocks than run at once, which then take little shared memory each.  Beyond, the smallest
// padding of the rows; tiles of 48 rows run at 0.85 of the rate of tiles of 64.  Measured in us on B200 (W [11264, 2048] | [2048,
// 5632]): 2 rows 21 | 12.5 (the other form 28 | 22), 8 rows 27.5 | 21.7 (30 | 30), 16 rows 32 | 24 (42 | 34), 32 rows 52 | 45, 64
// rows 87 | 48 (in tiles of 32: 90; in tiles of 64: 76), 72 rows 124 | 64 (in tiles of 64: 160 | 77), 600 rows 688 | 358.
template <bool VEC>
static int launch(const float* X, const float* W, float* Y, int M, int N, int K, int ldx, int ldw, int ldy, int weights_ready,
                  cudaStream_t s) {
#define KVCM_F32_TILE(...) return launch_tile<F32Tile<__VA_ARGS__>, VEC>(X, W, Y, M, N, K, ldx, ldw, ldy, weights_ready, s)
  const bool narrow = N <= 4096;
  if (M <= 4) { if (narrow) KVCM_F32_TILE(4, 32, 2, 1, 32, 8); else KVCM_F32_TILE(4, 64, 2, 1, 32, 3); }
  if (M <= 8) { if (narrow) KVCM_F32_TILE(8, 32, 4, 1, 16, 4); else KVCM_F32_TILE(8, 64, 4, 1, 16, 3); }
  if (M <= 16) { if (narrow) KVCM_F32_TILE(16, 64, 4, 2, 8, 5); else KVCM_F32_TILE(16, 64, 8, 2, 16, 3); }
  if (M <= 32 || (M > 48 && M <= 64 && narrow)) KVCM_F32_TILE(32, 64, 8, 4, 16, 4);
  if (M <= 48) KVCM_F32_TILE(48, 64, 6, 4, 16, 4);
  if ((M + 47) / 48 * 55 < (M + 63) / 64 * 64) KVCM_F32_TILE(48, 64, 6, 8, 8, 3);
  KVCM_F32_TILE(64, 64, 8, 8, 8, 3);
#undef KVCM_F32_TILE
}

}  // namespace kvcm

using namespace kvcm;

// weights_ready = 1: nothing that is still running on the stream writes W (a model's weights), so that it may be read
// before the launch's dependencies are done.
KVCM_API int kvcm_gemm_f32(const void* X, const void* W, void* Y, int M, int N, int K, int ldx, int ldw, int ldy,
                           int weights_ready, void* stream) {
  if (M == 0 || N == 0) return 0;
  const bool vec = K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(W) & 15) == 0;
  return (vec ? launch<true> : launch<false>)((const float*)X, (const float*)W, (float*)Y, M, N, K, ldx, ldw, ldy, weights_ready,
                                              (cudaStream_t)stream);
}
KVCM_API int kvcm_gemm_plain_f32(const void* X, const void* W, void* Y, int M, int N, int K, int ldx, int ldw, int ldy, void* stream) {
  return kvcm_gemm_f32(X, W, Y, M, N, K, ldx, ldw, ldy, 0, stream);
}
