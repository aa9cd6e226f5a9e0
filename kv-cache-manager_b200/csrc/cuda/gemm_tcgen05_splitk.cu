// Matrix product for a few dozen to a few hundred rows (decode at larger batches, short prompt
// portions) on the fifth-generation tensor cores:
//     Y[M, N] = X[M, K] * W[N, K]^T,  M <= 256, bfloat16 operands, float accumulation.
//
// With so few rows the product is bound by reading W once, so the roles of the operands are swapped:
// 128 rows of W are the 128-row operand of tcgen05.mma and the (padded) batch is its N, the
// accumulator [128 weight rows x M] sits in tensor memory.  N / 128 tiles alone would leave most of
// the 148 SMs idle, so K is split over the blocks of a thread-block cluster (1 to 8): every
// block streams its 128 x (K / S) slab of W (and the matching columns of X) through a TMA ring.  At the
// end every block puts its partial sums into its own shared memory, the cluster meets, and each block
// adds the S partial sums (always in block order: reproducible) of its share of the batch rows through
// distributed shared memory, a warp a row, and ends the row (see SplitkEpilogue).
//  * Two blocks share an SM (half of its shared memory and registers each).  Launched as programmatic dependents,
//    they fill their rings with W, where the caller vouches that it is a constant, while what lies before still runs; X
//    follows after the dependency wait.  (Blocks of 384 threads needed one SM each and were a quarter slower.)
//  * The residual stream and its norm ride along as in the weight-streaming kernel (gemm_stream.cu): a product
//    that ends a sublayer adds into the float residual and leaves bfloat16(w * x_new) and, per tile of 128
//    columns and row, the sum of squares; the product that begins the next one scales its sums by 1/rms.
// Roles per block: warp 0 one thread TMA, warp 1 one thread tcgen05.mma, warps 4-7 empty the accumulator; all eight
// end rows, two to four at a time.
// Measured on B200, 64 rows of the 1.1B shape: qkv 8.1 us, output and down product 6.5 and 10.8, gate/up 14.2 with their
// ends, 42 us a layer; the library's products with the norms, rotary encoding and activation as kernels of their own: 45.
// At 24 rows of the 7B shape 102 against 105 us; a step of 64 requests 1.26 -> 1.12 ms.
// Every wait on an mbarrier is bounded; a block whose wait ran out records it
// (kvcm_gemm_tcgen05_splitk_error), contributes nothing more, lets its copies land, still meets its cluster and
// frees its tensor memory.  The reference calls cuBLAS for these products (src/model/llama.cpp:45-52).
#include <cooperative_groups.h>

#include "gated_act.cuh"
#include "pdl.cuh"
#include "tcgen05_common.cuh"

namespace kvcm {

namespace cg = cooperative_groups;

constexpr int kSkThreads = 256, kSkWarps = kSkThreads / 32;
constexpr int kSkRows = 128;                 // weight rows per tile
constexpr int kSkBK = 64;                    // k elements per stage
constexpr int kSkMaxStages = 10;
constexpr int kSkMaxSplit = 8;
constexpr int kSkWBytes = kSkRows * kSkBK * 2;
constexpr size_t kSkSmemLimit = 200 * 1024;
constexpr size_t kSkSmemHalf = 108 * 1024;   // two such blocks share an SM
constexpr int kSkNormRows = 128;             // row stride of the partial sums of squares

__device__ int g_splitk_error = 0;

// What happens to a finished row of a tile (128 weight rows = output columns; a lane holds four neighbours).
//  kSkStore   : y[m][n] = sum.
//  kSkRope    : the tile is 128 / hd whole heads of [q | k | v]: the sums are rounded to bfloat16 as the plain
//               product would store them, q and k heads are rotated (rotate-half over the whole head) by the step's
//               table of cosines and sines, q goes to y, k and v go into the row's cache page slot.
//  kSkSilu    : the tile is 64 gate rows and the 64 up rows beside them: y[m][i] = the gated activation of the
//               rounded sums, as the separate kernel (SiLU).
//  kSkResidual: resid[m][n] += round(sum); ss_out[tile][m] = the sum of squares of the new values; h_out[m][n] =
//               bfloat16(next_w[n] * resid[m][n]) where next_w is given.
enum SplitkEpilogue { kSkStore = 0, kSkRope = 1, kSkSilu = 2, kSkResidual = 3 };

struct SplitkParams {
  void* Y; int M, N, K, ldy, Mp, stages, tmem_cols;
  int weights_ready;                          // nothing that may still be running writes W
  // SCALED: the sums of row m are multiplied by rsqrt(sum over t of ss_in[t][m] / K + eps) before the epilogue
  const float* ss_in; int ss_tiles; float eps;
  // kSkRope: table [M][hd] (hd/2 cosines, then hd/2 sines)
  const float* rope_table; const int* slot_mapping; bf16* k_cache; bf16* v_cache; int nh, nkv, hd, block_size;
  // kSkResidual
  float* resid; int ldr; float* ss_out; bf16* h_out; int ldh; const bf16* next_w;
};

__device__ __forceinline__ void store_bf16x4(bf16* p, float a, float b, float c, float d) {
  const __nv_bfloat162 lo = __floats2bfloat162_rn(a, b), hi = __floats2bfloat162_rn(c, d);
  uint2 raw;
  raw.x = *reinterpret_cast<const uint32_t*>(&lo);
  raw.y = *reinterpret_cast<const uint32_t*>(&hi);
  *reinterpret_cast<uint2*>(p) = raw;
}

// MAXS: the largest S that it runs with; fewer parts leave registers for more rows at a time.
template <typename OutT, int EPI, bool SCALED, int MAXS>
__global__ void __launch_bounds__(kSkThreads, 2)
gemm_tcgen05_splitk_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, SplitkParams p) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const int stages = p.stages;
  const int stage_bytes = kSkWBytes + p.Mp * kSkBK * 2;        // W piece, then X piece (both 1,024-byte multiples)
  __shared__ __align__(8) uint64_t full[kSkMaxStages], empty[kSkMaxStages], acc_full;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int abort_flag;
  __shared__ float norm_s[SCALED ? kSkNormRows : 1];           // SCALED: 1/rms of this block's rows

  cg::cluster_group cluster = cg::this_cluster();
  const int S = int(cluster.num_blocks()), rank = int(cluster.block_rank());
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = int(blockIdx.x) / S;
  const int n0 = tile * (EPI == kSkSilu ? kSkRows / 2 : kSkRows);        // first (gate) row of W
  const int nk = (p.K + kSkBK - 1) / kSkBK;
  const int k_begin = nk * rank / S, steps = nk * (rank + 1) / S - k_begin;   // k-steps of this block
  const bool aligned = (tc5::s32(smem_raw) & 1023) == 0;       // the swizzled tiles need this

  if (threadIdx.x == 0) {
    abort_flag = aligned ? 0 : 1;
    if (!aligned) atomicExch(&g_splitk_error, (7 << 16) | int(blockIdx.x & 0xffff));
    for (int s = 0; s < stages; ++s) { tc5::mbar_init(&full[s], 1); tc5::mbar_init(&empty[s], 1); }
    tc5::mbar_init(&acc_full, 1);
    tc5::mbar_init_fence();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc5::s32(&tmem_base)), "r"(p.tmem_cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  tc5::fence_before();
  __syncthreads();
  tc5::fence_after();
  const uint32_t tmem = tmem_base;
  // only now, with the tensor memory in hand: a dependent that takes some early would keep a block of this launch waiting
  // for it, and itself waits for this launch
  pdl_launch_dependents();

  auto fail = [&](int code) {
    atomicExch(&g_splitk_error, (code << 16) | int(blockIdx.x & 0xffff));
    abort_flag = 1;
  };

  if (warp == 0) {
    if (lane == 0 && !abort_flag) {
      const auto load_w = [&](int i, int s) {
        tc5::mbar_expect_tx(&full[s], uint32_t(stage_bytes));
        unsigned char* w_s = smem_raw + size_t(s) * stage_bytes;
        tc5::tma_load_2d(w_s, &map_w, &full[s], (k_begin + i) * kSkBK, n0);
        if constexpr (EPI == kSkSilu)                          // the map's box is 64 rows: the up rows follow
          tc5::tma_load_2d(w_s + kSkWBytes / 2, &map_w, &full[s], (k_begin + i) * kSkBK, p.N + n0);
      };
      const auto load_x = [&](int i, int s) {
        tc5::tma_load_2d(smem_raw + size_t(s) * stage_bytes + kSkWBytes, &map_x, &full[s], (k_begin + i) * kSkBK, 0);
      };
      const int first = min(steps, stages);
      if (!p.weights_ready) pdl_wait();
      for (int i = 0; i < first; ++i) load_w(i, i);
      pdl_wait();                                              // (X is the predecessor's in any case)
      for (int i = 0; i < first; ++i) load_x(i, i);
      int issued = first;
      for (int i = first, s = 0, round = 1; i < steps && !abort_flag; ++i) {
        if (!tc5::mbar_wait(&empty[s], (round - 1) & 1)) { fail(1); break; }
        load_w(i, s);
        load_x(i, s);
        ++issued;
        if (++s == stages) { s = 0; ++round; }
      }
      if (abort_flag)                                          // nothing of this block's may land after it has left
        for (int s = 0; s < stages; ++s) {
          const int fills = issued > s ? (issued - s - 1) / stages + 1 : 0;
          if (fills > 0) tc5::mbar_wait(&full[s], (fills - 1) & 1);
        }
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t instr = tc5::idesc(kSkRows, p.Mp);
      for (int i = 0, s = 0, phase = 0; i < steps && !abort_flag; ++i) {
        if (!tc5::mbar_wait(&full[s], phase)) { fail(2); break; }
        tc5::fence_after();
        const uint32_t w_addr = tc5::s32(smem_raw + size_t(s) * stage_bytes);
        const uint64_t da = tc5::smem_desc(w_addr), db = tc5::smem_desc(w_addr + kSkWBytes);
#pragma unroll
        for (int j = 0; j < kSkBK / 16; ++j)
          tc5::mma(tmem, da + uint64_t(2 * j), db + uint64_t(2 * j), instr, (i > 0 || j > 0) ? 1u : 0u);
        tc5::commit(&empty[s]);                                // the slot is free once these products have read it
        if (++s == stages) { s = 0; phase ^= 1; }
      }
      if (!abort_flag) tc5::commit(&acc_full);
    }
    __syncwarp();
  }
  pdl_wait();                                                  // what the epilogue reads is the predecessors' too
  if constexpr (SCALED) {                                      // while the ring streams
    const int m_end = p.M * (rank + 1) / S;
    for (int m = p.M * rank / S + warp - 2; warp >= 2 && m < m_end; m += kSkWarps - 2) {
      float ss = 0.f;
      for (int i = lane; i < p.ss_tiles; i += 32) ss += __ldcg(p.ss_in + i * kSkNormRows + m);
      ss = warp_sum(ss);
      if (lane == 0) norm_s[m] = rsqrtf(ss / float(p.K) + p.eps);
    }
  }

  // ---- the block's partial sums go to its shared memory as [M][128] floats (the ring is no longer
  // needed: every copy has landed and every product has read it once acc_full completes)
  float* partial = reinterpret_cast<float*>(smem_raw);
  if (warp >= 4) {
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;                       // weight row of the tile = lane of tensor memory
    bool have = steps > 0 && !abort_flag;
    if (have) have = tc5::mbar_wait(&acc_full, 0);
    if (!__all_sync(0xffffffffu, have)) {
      if (steps > 0 && !abort_flag && lane == 0) fail(3);
      have = false;
    }
    tc5::fence_after();
    if (have || steps == 0)                                    // (after a failure the ring may still be written)
      for (int c = 0; c < (p.Mp + 31) / 32; ++c) {
        uint32_t v[32];
        if (have) {
          // (loads of 32 columns; the allocation is a power of two >= Mp rounded up to 32, so the
          // columns beyond Mp exist and are simply not used)
          tc5::ld32(tmem + (uint32_t(quarter * 32) << 16) + uint32_t(c * 32), v);
          tc5::ld_wait();
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int m = c * 32 + i;
          if (m < p.M) partial[m * kSkRows + row] = have ? __uint_as_float(v[i]) : 0.f;
        }
      }
    tc5::fence_before();
  }
  if (S > 1) cluster.sync();                                   // every block's partial sums are in place
  else __syncthreads();

  if (!abort_flag) {
    constexpr int U = 16 / MAXS;                               // rows a warp ends at a time
    const float* parts[MAXS];
#pragma unroll
    for (int q = 0; q < MAXS; ++q) parts[q] = cluster.map_shared_rank(partial, q < S ? q : rank);
    const int m_end = p.M * (rank + 1) / S;
    const int c = lane * 4, n = n0 + c;                        // this lane's columns of the tile
    const bool whole = n + 4 <= p.N;
    const int head = EPI == kSkRope ? n / p.hd : 0, j = EPI == kSkRope ? n - head * p.hd : 0;
    for (int m0 = p.M * rank / S + warp; m0 < m_end; m0 += U * kSkWarps) {
      // everything the rows need is asked for before the first sum is waited for
      float4 before[U], cs[U], sn[U], t[U][MAXS];
      int slot[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int m = m0 + u * kSkWarps;
        slot[u] = -1;
        if (m >= m_end) break;
#pragma unroll
        for (int q = 0; q < MAXS; ++q)
          if (q < S) t[u][q] = *reinterpret_cast<const float4*>(parts[q] + m * kSkRows + c);
        if constexpr (EPI == kSkResidual)
          before[u] = whole ? __ldcg(reinterpret_cast<const float4*>(p.resid + size_t(m) * p.ldr + n)) : make_float4(0.f, 0.f, 0.f, 0.f);
        if constexpr (EPI == kSkRope) {
          const int half = p.hd / 2;
          cs[u] = sn[u] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (head < p.nh + p.nkv) {
            const float* row = p.rope_table + size_t(m) * p.hd + (j < half ? j : j - half);
            cs[u] = *reinterpret_cast<const float4*>(row);
            sn[u] = *reinterpret_cast<const float4*>(row + half);
          }
          if (head >= p.nh && whole) slot[u] = p.slot_mapping[m];
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int m = m0 + u * kSkWarps;
        if (m >= m_end) break;
        float r[4] = {t[u][0].x, t[u][0].y, t[u][0].z, t[u][0].w};
#pragma unroll
        for (int q = 1; q < MAXS; ++q)
          if (q < S) { r[0] += t[u][q].x; r[1] += t[u][q].y; r[2] += t[u][q].z; r[3] += t[u][q].w; }
        if constexpr (SCALED) {
          const float f = norm_s[m];
#pragma unroll
          for (int i = 0; i < 4; ++i) r[i] *= f;
        }
        if constexpr (EPI == kSkStore) {
          OutT* dst = reinterpret_cast<OutT*>(p.Y) + size_t(m) * p.ldy + n;
          if (whole && (p.ldy & 3) == 0 && (reinterpret_cast<uintptr_t>(p.Y) & 15) == 0) {
            if constexpr (sizeof(OutT) == 4) *reinterpret_cast<float4*>(dst) = make_float4(r[0], r[1], r[2], r[3]);
            else store_bf16x4(dst, r[0], r[1], r[2], r[3]);
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (n + i < p.N) stf(dst + i, r[i]);
          }
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) r[i] = Store<bf16>::round(r[i]);          // what the plain product stores
        }
        if constexpr (EPI == kSkResidual) {
          const float v[4] = {before[u].x + r[0], before[u].y + r[1], before[u].z + r[2], before[u].w + r[3]};
          if (whole) {
            *reinterpret_cast<float4*>(p.resid + size_t(m) * p.ldr + n) = make_float4(v[0], v[1], v[2], v[3]);
            if (p.next_w != nullptr)
              store_bf16x4(p.h_out + size_t(m) * p.ldh + n, ldf(p.next_w + n) * v[0], ldf(p.next_w + n + 1) * v[1],
                           ldf(p.next_w + n + 2) * v[2], ldf(p.next_w + n + 3) * v[3]);
          }
          const float ss = warp_sum(whole ? v[0] * v[0] + v[1] * v[1] + v[2] * v[2] + v[3] * v[3] : 0.f);
          if (lane == 0) p.ss_out[tile * kSkNormRows + m] = ss;
        }
        if constexpr (EPI == kSkSilu) {
          float up[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) up[i] = __shfl_down_sync(0xffffffffu, r[i], 16);
          if (lane < 16 && whole) {
            const GatedAct act{};
            store_bf16x4(reinterpret_cast<bf16*>(p.Y) + size_t(m) * p.ldy + n, gated_act<kGatedSilu, bf16>(r[0], up[0], act),
                         gated_act<kGatedSilu, bf16>(r[1], up[1], act), gated_act<kGatedSilu, bf16>(r[2], up[2], act),
                         gated_act<kGatedSilu, bf16>(r[3], up[3], act));
          }
        }
        if constexpr (EPI == kSkRope) {
          const bool low = j < p.hd / 2;
          float other[4], v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) other[i] = __shfl_xor_sync(0xffffffffu, r[i], p.hd / 8);   // the pair's other half
          const float csv[4] = {cs[u].x, cs[u].y, cs[u].z, cs[u].w}, snv[4] = {sn[u].x, sn[u].y, sn[u].z, sn[u].w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float a, b;
            rotate_pair(low ? r[i] : other[i], low ? other[i] : r[i], csv[i], snv[i], a, b);
            v[i] = head < p.nh + p.nkv ? (low ? a : b) : r[i];
          }
          if (whole && head < p.nh) {
            store_bf16x4(reinterpret_cast<bf16*>(p.Y) + size_t(m) * p.ldy + n, v[0], v[1], v[2], v[3]);
          } else if (slot[u] >= 0) {
            const int page = slot[u] / p.block_size, off = slot[u] - page * p.block_size;
            const bool is_k = head < p.nh + p.nkv;
            const int kvh = is_k ? head - p.nh : head - p.nh - p.nkv;
            store_bf16x4((is_k ? p.k_cache : p.v_cache) + ((size_t(page) * p.nkv + kvh) * p.block_size + off) * p.hd + j,
                         v[0], v[1], v[2], v[3]);
          }
        }
      }
    }
  }
  if (S > 1) cluster.sync();                                   // nobody leaves while its memory is read
  tc5::fence_before();
  __syncthreads();
  if (warp == 1) {
    tc5::fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(p.tmem_cols));
  }
}

// How K is split: as many blocks as run at once (two to an SM, less a tenth: clusters do not pack the GPCs without gaps; at
// 6,144 outputs of 4,096 240 blocks took 11.6 us and 288 took 19, at 12,288 outputs 192 took 19.7 and 288 took 31), at most
// 8 per tile, at least four k-steps each.
static int splitk_factor(int tiles, int K, int sm_count) {
  const int nk = (K + kSkBK - 1) / kSkBK;
  int S = 1;
  while (S < kSkMaxSplit && tiles * (S + 1) * 10 <= 18 * sm_count && nk / (S + 1) >= 4) ++S;
  return S;
}

template <typename OutT, int EPI, bool SCALED>
int launch_splitk(const void* X, const void* W, int ldx, int ldw, SplitkParams p, cudaStream_t s) {
  static int sm_count = 0;
  if (sm_count == 0) sm_count = tc5::current_sm_count();
  p.Mp = (p.M + 15) / 16 * 16;
  CUtensorMap mw, mx;
  int rc = tc5::make_map(&mw, W, EPI == kSkSilu ? 2 * p.N : p.N, p.K, ldw, EPI == kSkSilu ? kSkRows / 2 : kSkRows);
  if (rc) return rc;
  rc = tc5::make_map(&mx, X, p.M, p.K, ldx, p.Mp);
  if (rc) return rc;
  const int cols = EPI == kSkSilu ? kSkRows / 2 : kSkRows;
  const int tiles = (p.N + cols - 1) / cols;
  const int stage_bytes = kSkWBytes + p.Mp * kSkBK * 2;
  const size_t partial_bytes = size_t(p.M) * kSkRows * sizeof(float);
  const int S = splitk_factor(tiles, p.K, sm_count);
  const int nk = (p.K + kSkBK - 1) / kSkBK, per = (nk + S - 1) / S;
  int stages = int(kSkSmemHalf / stage_bytes);
  if (stages < 2) stages = 2;
  if (stages > kSkMaxStages) stages = kSkMaxStages;
  if (stages > per) stages = per;
  size_t smem = size_t(stages) * stage_bytes;
  if (smem < partial_bytes) smem = partial_bytes;
  if (smem > kSkSmemLimit) return KVCM_ERR_UNSUPPORTED;
  p.stages = stages;
  p.tmem_cols = 32;
  while (p.tmem_cols < p.Mp) p.tmem_cols *= 2;
  auto kernel = S <= 4 ? gemm_tcgen05_splitk_kernel<OutT, EPI, SCALED, 4> : gemm_tcgen05_splitk_kernel<OutT, EPI, SCALED, kSkMaxSplit>;
  static OncePerDevice once[2];
  rc = allow_shared_memory(once[S <= 4 ? 0 : 1], kernel, kSkSmemLimit);
  if (rc) return rc;
  return pdl_launch_cluster(kernel, dim3(tiles * S), dim3(kSkThreads), smem, s, S, mw, mx, p);
}

static bool aligned16(const void* a) { return (reinterpret_cast<uintptr_t>(a) & 15) == 0; }

}  // namespace kvcm

using namespace kvcm;

KVCM_API int kvcm_gemm_tcgen05_splitk_supports(int M, int N, int K, int ldx, int ldw) {
  return M >= 1 && M <= 256 && N >= 1 && K >= 8 && (K % 8) == 0 && (ldx % 8) == 0 && (ldw % 8) == 0;
}

// out_f32: 0 = bfloat16 result, 1 = float result.  weights_ready = 1: nothing that is still running on the stream writes W
// (a model's weights), so that it may be read before the launch's dependencies are done.
KVCM_API int kvcm_gemm_tcgen05_splitk_bf16(const void* X, const void* W, void* Y, int M, int N, int K, int ldx, int ldw,
                                           int ldy, int out_f32, int weights_ready, void* stream) {
  if (M == 0 || N == 0) return 0;
  if (!kvcm_gemm_tcgen05_splitk_supports(M, N, K, ldx, ldw) || !aligned16(X) || !aligned16(W)) return KVCM_ERR_UNSUPPORTED;
  SplitkParams p = {};
  p.Y = Y; p.M = M; p.N = N; p.K = K; p.ldy = ldy; p.weights_ready = weights_ready;
  cudaStream_t s = (cudaStream_t)stream;
  return out_f32 ? launch_splitk<float, kSkStore, false>(X, W, ldx, ldw, p, s) : launch_splitk<bf16, kSkStore, false>(X, W, ldx, ldw, p, s);
}

// The forms with a fused end (W is a model's weights: it is read ahead), for a step of M rows of a model of these sizes (at most 128 rows: the partial sums of
// squares are kSkNormRows rows wide).
KVCM_API int kvcm_splitk_fused_supports(int M, int N, int K) {
  return M >= 1 && M <= kSkNormRows && N >= 4 && (N % 4) == 0 && K >= 8 && (K % 8) == 0;
}
KVCM_API long long kvcm_splitk_norm_floats(int N) { return (long long)(N + kSkRows - 1) / kSkRows * kSkNormRows; }

// The product that ends a sublayer: resid[M, N] += round_bf16(X * W^T); ss_out (kvcm_splitk_norm_floats(N) floats) and,
// where next_w is given, h_out for the product that follows.
KVCM_API int kvcm_splitk_residual_bf16(const void* X, const void* W, float* resid, float* ss_out, void* h_out, const void* next_w,
                                       int M, int N, int K, int ldx, int ldw, int ldr, int ldh, void* stream) {
  if (M == 0) return 0;
  if (!kvcm_splitk_fused_supports(M, N, K) || (ldx % 8) || (ldw % 8) || (ldr % 4) || (ldh % 4) || !aligned16(X) || !aligned16(W) ||
      !aligned16(resid) || !aligned16(h_out) || ss_out == nullptr || (next_w != nullptr && h_out == nullptr))
    return KVCM_ERR_UNSUPPORTED;
  SplitkParams p = {};
  p.M = M; p.N = N; p.K = K; p.weights_ready = 1;
  p.resid = resid; p.ldr = ldr; p.ss_out = ss_out; p.h_out = (bf16*)h_out; p.ldh = ldh; p.next_w = (const bf16*)next_w;
  return launch_splitk<bf16, kSkResidual, false>(X, W, ldx, ldw, p, (cudaStream_t)stream);
}

// qkv = X * Wqkv^T (rows scaled by the norm's 1/rms where ss_in is given), rotary encoding by the table of the step's
// angles, q to Yq, k and v into the cache pages.  hd: 16, 32, 64 or 128 (a tile is whole heads).
KVCM_API int kvcm_splitk_qkv_bf16(const void* X, const float* ss_in, int ss_tiles, float eps, const void* Wqkv, void* Yq, int M,
                                  int K, int ldx, int ldw, int ldy, const float* rope_table, const int* slot_mapping, void* k_cache,
                                  void* v_cache, int nh, int nkv, int hd, int block_size, void* stream) {
  const int N = (nh + 2 * nkv) * hd;
  if (M == 0) return 0;
  if ((hd != 16 && hd != 32 && hd != 64 && hd != 128) || !kvcm_splitk_fused_supports(M, N, K) || (ldx % 8) || (ldw % 8) ||
      (ldy % 4) || !aligned16(X) || !aligned16(Wqkv) || !aligned16(Yq) || !aligned16(rope_table) || !aligned16(k_cache) || !aligned16(v_cache))
    return KVCM_ERR_UNSUPPORTED;
  SplitkParams p = {};
  p.Y = Yq; p.M = M; p.N = N; p.K = K; p.ldy = ldy; p.weights_ready = 1;
  p.ss_in = ss_in; p.ss_tiles = ss_tiles; p.eps = eps;
  p.rope_table = rope_table; p.slot_mapping = slot_mapping; p.k_cache = (bf16*)k_cache; p.v_cache = (bf16*)v_cache;
  p.nh = nh; p.nkv = nkv; p.hd = hd; p.block_size = block_size;
  cudaStream_t s = (cudaStream_t)stream;
  return ss_in ? launch_splitk<bf16, kSkRope, true>(X, Wqkv, ldx, ldw, p, s) : launch_splitk<bf16, kSkRope, false>(X, Wqkv, ldx, ldw, p, s);
}

// act[M, I] = silu(X Wg^T) * (X Wu^T), W [2I, K] with the gate rows first; rows scaled as above where ss_in is given.
KVCM_API int kvcm_splitk_gate_up_silu_bf16(const void* X, const float* ss_in, int ss_tiles, float eps, const void* W, void* Y, int M,
                                           int I, int K, int ldx, int ldw, int ldy, void* stream) {
  if (M == 0) return 0;
  if (!kvcm_splitk_fused_supports(M, I, K) || (ldx % 8) || (ldw % 8) || (ldy % 4) || !aligned16(X) || !aligned16(W) || !aligned16(Y))
    return KVCM_ERR_UNSUPPORTED;
  SplitkParams p = {};
  p.Y = Y; p.M = M; p.N = I; p.K = K; p.ldy = ldy; p.weights_ready = 1;
  p.ss_in = ss_in; p.ss_tiles = ss_tiles; p.eps = eps;
  cudaStream_t s = (cudaStream_t)stream;
  return ss_in ? launch_splitk<bf16, kSkSilu, true>(X, W, ldx, ldw, p, s) : launch_splitk<bf16, kSkSilu, false>(X, W, ldx, ldw, p, s);
}

// Device address of the error word (the sampling kernels copy it out with the step's tokens).
KVCM_API const int* kvcm_gemm_tcgen05_splitk_error_address(void) {
  int* p = nullptr;
  return cudaGetSymbolAddress((void**)&p, g_splitk_error) == cudaSuccess ? p : nullptr;
}

// Reads and clears the error word of the kernel (0 = no bounded wait ever ran out); else
// (code << 16) | block: 1 the producer waited for a free stage, 2 the products for data, 3 the
// epilogue for the accumulator, 7 shared memory not aligned to 1,024 bytes.
KVCM_API int kvcm_gemm_tcgen05_splitk_error(void) {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_splitk_error, sizeof v) != cudaSuccess) return -1;
  if (v != 0) cudaMemcpyToSymbol(g_splitk_error, &zero, sizeof zero);
  return v;
}
