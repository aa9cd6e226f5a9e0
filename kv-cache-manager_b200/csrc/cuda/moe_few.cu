// The experts' products of a routed feed-forward for a step of few rows (decode), bfloat16, float accumulation:
//     act[pair] = silu(h[row] Wg_e^T) * (h[row] Wu_e^T);   y[pair] = act[pair] Wd_e^T      (pair = row * top + choice)
//
// Such a step reads the matrices of the chosen experts once and multiplies each by a row or two, so it is bound by
// that read.  Tiles of 128 pairs (moe_tcgen05.cu) leave a handful of blocks per expert walking K one stage after
// another, behind a sort and a gather of their own.  Here a warp takes 16 rows of an expert's matrix as the 16-row
// operand of mma.sync (m16n8k16; the pairs are its 8 columns) straight from memory, several blocks of 32 k's in flight a
// thread and few enough registers for four blocks an SM.  A block of the grid's second axis takes the n-th of the chosen
// experts and looks through the step's choices itself for that expert's pairs, in their order: no sort, no gather, and y
// lies in the order of the pairs.
// Both products read the choices behind their own dependency wait: nothing else makes the router's writes visible to a
// kernel that was launched early, and a choice is an address here.  (So the down product cannot ask for weights before its
// wait.)  A choice that names no expert is passed over and reported through the error word of the experts' products.
// The k index inside a 32-wide block is permuted identically for both operands (thread t of a quad owns k = 8t..8t+7),
// which makes every load a 16-byte vector.  Partial sums of the warps are added in warp order: reproducible.
// Measured on B200 (32 experts of 512 x 2,048, 8 choices a row, launches back to back): 1 row 16 us, 4 rows 35, 8 rows 43, 16
// rows 50; the sorted form 30, 46, 50 and 50.  Several tiles a block and whole rows through shared memory by asynchronous copies
// were both slower.
#include "common.cuh"
#include "pdl.cuh"

namespace kvcm {

constexpr int kMfMaxRows = 16, kMfMaxPairs = 1024, kMfMaxExperts = 1024;
constexpr int kMfUp = 8, kMfDown = 4;                      // warps of a gate/up block (they share K) and of a down block (16 rows each)
constexpr int kMfUpAhead = 4, kMfDownAhead = 8;            // blocks of 32 k's a thread has in flight (gate/up: four blocks an SM)

__device__ __forceinline__ uint4 load_stream(const bf16* p) {          // read once: not kept in L1
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void mma_few(float (&d)[4], const uint4& a, const uint4& b, const uint4& x) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a.x), "r"(b.x), "r"(a.y), "r"(b.y), "r"(x.x), "r"(x.y));
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a.z), "r"(b.z), "r"(a.w), "r"(b.w), "r"(x.z), "r"(x.w));
}

struct FewPick {
  int list[kMfMaxPairs];                                   // the pairs of the block's expert, ascending
  unsigned chosen[kMfMaxExperts / 32];                     // bit per expert
  int expert, count;
};

constexpr int kMfNoExpert = 9;                              // code of a choice that names no expert

// The which-th of the chosen experts (ascending) and its pairs; count 0 where there are no more.  Whole block; ends with a
// barrier.
__device__ __forceinline__ void pick_expert(FewPick& s, const int* idx, int pairs, int E, int which, int* error) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    s.chosen[lane] = 0u;
    __syncwarp();
    for (int p = lane; p < pairs; p += 32) {
      const unsigned e = unsigned(idx[p]);
      if (e < unsigned(E)) atomicOr(&s.chosen[e >> 5], 1u << (e & 31));
      else if (error != nullptr) atomicExch(error, (kMfNoExpert << 16) | p);
    }
    __syncwarp();
    const unsigned word = s.chosen[lane];
    int upto = __popc(word);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += t;
    }
    const int before = upto - __popc(word);
    int e = -1;
    if (which >= before && which < upto) e = 32 * lane + int(__fns(word, 0, which - before + 1));
    e = __reduce_max_sync(0xffffffffu, e);
    int n = 0;
    for (int p0 = 0; e >= 0 && p0 < pairs; p0 += 32) {
      const int p = p0 + lane;
      const bool mine = p < pairs && idx[p] == e;
      const unsigned who = __ballot_sync(0xffffffffu, mine);
      if (mine) s.list[n + __popc(who & ((1u << lane) - 1u))] = p;
      n += __popc(who);
    }
    if (lane == 0) { s.expert = e; s.count = n; }
  }
  __syncthreads();
}

// acc[j] += 16 matrix rows (this thread: rows g and g + 8 from wa and wb) x the rows x[j] behind columns 8 j.., over the
// 32-wide blocks of k from kb by `stride` below K (K % 8 == 0; addresses already hold the thread's 8 * t4).
template <int NT, int AHEAD>
__device__ __forceinline__ void walk_k(float (&acc)[NT][4], const bf16* wa, const bf16* wb, const bf16* const (&x)[NT], int nt,
                                       int kb, int stride, int K, int t4) {
  const uint4 none = make_uint4(0u, 0u, 0u, 0u);
  for (; kb < K; kb += AHEAD * stride) {
    uint4 a[AHEAD], b[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int k = kb + u * stride;
      const bool in = k + 8 * t4 < K;
      a[u] = in ? load_stream(wa + k) : none;
      b[u] = in ? load_stream(wb + k) : none;
    }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      if (j >= nt) break;
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const int k = kb + u * stride;
        const uint4 v = k + 8 * t4 < K ? *reinterpret_cast<const uint4*>(x[j] + k) : none;
        mma_few(acc[j], a[u], b[u], v);
      }
    }
  }
}

// Block (tile of 8 gate rows and their 8 up rows, n-th chosen expert).  `place_of`: every pair's place is its own number (the
// readers of y look it up); written by the first block.
template <int NT>
__global__ void __launch_bounds__(32 * kMfUp, NT == 1 ? 4 : 2)
moe_few_gate_up_kernel(const bf16* h, int ldh, const bf16* __restrict__ wgu, const int* idx, int pairs, int top, int E, int F, int D,
                       bf16* act, int* place_of, int* error) {
  __shared__ FewPick pick;
  __shared__ __align__(16) float red[kMfUp][16][8 * NT];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
  const int f0 = 8 * blockIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  if (blockIdx.x == 0 && blockIdx.y == 0)
    for (int i = tid; i < pairs; i += 32 * kMfUp) place_of[i] = i;
  pick_expert(pick, idx, pairs, E, blockIdx.y, error);
  const int n = pick.count;
  const bf16* wa = wgu + (size_t(max(pick.expert, 0)) * 2 * F + f0 + g) * D + 8 * t4;      // (F % 8 == 0: the tile's rows exist)
  for (int n0 = 0; n0 < n; n0 += 8 * NT) {                               // (one trip unless a row chose an expert twice)
    const int here = min(8 * NT, n - n0);
    const bf16* x[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) x[j] = h + size_t(pick.list[n0 + min(8 * j + g, here - 1)] / top) * ldh + 8 * t4;
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    walk_k<NT, kMfUpAhead>(acc, wa, wa + size_t(F) * D, x, (here + 7) / 8, warp * 32, 32 * kMfUp, D, t4);
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      *reinterpret_cast<float2*>(&red[warp][g][8 * j + 2 * t4]) = make_float2(acc[j][0], acc[j][1]);
      *reinterpret_cast<float2*>(&red[warp][g + 8][8 * j + 2 * t4]) = make_float2(acc[j][2], acc[j][3]);
    }
    __syncthreads();
    for (int i = tid; i < 8 * here; i += 32 * kMfUp) {
      const int m = i >> 3, r = i & 7;
      float xg = 0.f, xu = 0.f;
#pragma unroll
      for (int w = 0; w < kMfUp; ++w) { xg += red[w][r][m]; xu += red[w][r + 8][m]; }
      act[size_t(pick.list[n0 + m]) * F + f0 + r] = __float2bfloat16_rn(xg / (1.f + expf(-xg)) * xu);
    }
    __syncthreads();
  }
}

// Block (tile of 64 output columns, n-th chosen expert): a warp 16 of them over the whole of K = F.
template <int NT>
__global__ void __launch_bounds__(32 * kMfDown)
moe_few_down_kernel(const bf16* act, const bf16* __restrict__ wd, const int* idx, int pairs, int E, int F, int D, float* y) {
  __shared__ FewPick pick;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  const int c0 = (blockIdx.x * kMfDown + warp) * 16;
  pdl_launch_dependents();
  pdl_wait();
  pick_expert(pick, idx, pairs, E, blockIdx.y, nullptr);                 // (gate/up has reported)
  const int n = pick.count;
  if (c0 >= D) return;
  const bf16* wa = wd + (size_t(max(pick.expert, 0)) * D + c0 + g) * F + 8 * t4;           // (D % 8 == 0: rows g exist)
  const bf16* wb = c0 + 8 < D ? wa + size_t(8) * F : wa;
  for (int n0 = 0; n0 < n; n0 += 8 * NT) {
    const int here = min(8 * NT, n - n0);
    const bf16* x[NT];
#pragma unroll
    for (int j = 0; j < NT; ++j) x[j] = act + size_t(pick.list[n0 + min(8 * j + g, here - 1)]) * F + 8 * t4;
    float acc[NT][4];
#pragma unroll
    for (int j = 0; j < NT; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;
    walk_k<NT, kMfDownAhead>(acc, wa, wb, x, (here + 7) / 8, 0, 32, F, t4);
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = 8 * j + 2 * t4 + (i & 1), c = c0 + g + 8 * (i >> 1);
        if (m < here && c < D) y[size_t(pick.list[n0 + m]) * D + c] = acc[j][i];
      }
  }
}

template <int NT>
int launch_moe_few(const bf16* h, int ldh, const bf16* wgu, const bf16* wd, const int* idx, int pairs, int top, int E, int F, int D,
                   int* place_of, int* error, bf16* act, float* y, cudaStream_t s) {
  const int most = pairs < E ? pairs : E;                                // as many experts can be chosen
  int rc = pdl_launch(moe_few_gate_up_kernel<NT>, dim3(F / 8, most), dim3(32 * kMfUp), 0, s, h, ldh, wgu, idx, pairs, top, E, F, D, act,
                      place_of, error);
  if (rc) return rc;
  return pdl_launch(moe_few_down_kernel<NT>, dim3((D + 16 * kMfDown - 1) / (16 * kMfDown), most), dim3(32 * kMfDown), 0, s,
                    (const bf16*)act, wd, idx, pairs, E, F, D, y);
}

}  // namespace kvcm

using namespace kvcm;

extern "C" const int* kvcm_moe_tcgen05_error_address(void);

KVCM_API int kvcm_moe_few_supports(int rows, int top, int E, int F, int D) {
  return rows >= 1 && rows <= kMfMaxRows && top >= 1 && rows * (long long)top <= kMfMaxPairs && E >= 1 && E <= kMfMaxExperts && F >= 8 &&
         (F % 8) == 0 && D >= 8 && (D % 8) == 0;
}

// `work`: the scratch of kvcm_moe_work_ints; y [pairs, D] in the order of the pairs; rows of y whose choice
// is not within [0, E) are left as they are.
KVCM_API int kvcm_moe_experts_few_bf16(const void* h, int ldh, const void* wgu, const void* wd, const int* idx, int rows, int top, int E,
                                       int F, int D, int* work, void* act, float* y, void* stream) {
  if (rows == 0) return 0;
  if (!kvcm_moe_few_supports(rows, top, E, F, D) || (ldh % 8) ||
      ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(wgu) | reinterpret_cast<uintptr_t>(wd) |
        reinterpret_cast<uintptr_t>(act)) & 15))
    return KVCM_ERR_UNSUPPORTED;
  const int pairs = rows * top;
  int* place_of = work + E + 2 + pairs;                                  // as moe.cu lays it out
  const auto run = rows <= 8 ? launch_moe_few<1> : launch_moe_few<2>;
  return run((const bf16*)h, ldh, (const bf16*)wgu, (const bf16*)wd, idx, pairs, top, E, F, D, place_of,
             const_cast<int*>(kvcm_moe_tcgen05_error_address()), (bf16*)act, y, (cudaStream_t)stream);
}
