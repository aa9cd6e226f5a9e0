// Plain paged attention: one block per (row, query head), keys walked through the page table in
// chunks with a running (max, sum, accumulator): softmax and P*V in float whatever the storage
// type.  Any head_dim up to 1024, any number of heads and groups, any page size, optional window.
// With float storage this is the attention of the true 32-bit path; with bfloat16 it is the twin
// that the fast kernels are checked against.  A row's result depends only on its own position,
// its keys and the window, never on the batch around it.
// Optional: scores capped as cap * tanh(score / cap); a sink per head, one more term exp(sink) in
// the softmax's denominator with neither a key nor a value behind it (the running maximum starts at the sink
// with a sum of one and an empty accumulator).
//
// Arithmetic as the reference's kernel (src/cuda/paged_attention.cu:80-182): q is scaled first,
// the causal mask is the loop bound ctx = position + 1, o = (sum_t p_t v_t) / sum_t p_t.
// With a window, `keep_first` > 0 keeps the first keep_first keys of the request visible to every row: the
// keys walked are [0, min(keep_first, lo)) followed by the window [lo, ctx).
// With `chunk` > 0 a row sees only the keys of its own chunk of positions (chunks counted from position 0).
//
// What bounds it: the latency of one row's chain of keys (a decode step has few rows), so a key's cache row is looked
// up once per chunk and kept, elements move four at a time, and the products with V are dealt out over groups of
// threads that take every n-th key each, joined at the end in the groups' order.  Measured on B200 (float32, 2 requests,
// 32 heads of 64, 64 to 80 keys): 17.9 us a launch before; eight tokens of two such requests through 22 layers, with the
// float products' tiles of the same change: 38.4 -> 27.2 ms.
#include "common.cuh"
#include "pdl.cuh"

namespace kvcm {

constexpr int kPlainThreads = 128;
constexpr int kPlainChunk = 512;
constexpr int kPlainMaxDimsPerThread = 8;     // head_dim <= 8 * 128

template <int VEC> __device__ __forceinline__ void load_n(const float* p, float (&v)[VEC]) {
  if constexpr (VEC == 4) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else {
    v[0] = *p;
  }
}
template <int VEC> __device__ __forceinline__ void load_n(const bf16* p, float (&v)[VEC]) {
  if constexpr (VEC == 4) {
    const uint2 t = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&t.y));
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
  } else {
    v[0] = ldf(p);
  }
}

template <typename T, int VEC>
__global__ void __launch_bounds__(kPlainThreads)
attention_plain_kernel(const T* q, int q_stride, T* __restrict__ out, int out_stride,
                       const T* k_cache, const T* v_cache,
                       const int* __restrict__ block_tables, int max_blocks,
                       const int* __restrict__ row_seq, const int* __restrict__ positions,
                       int nh, int nkv, int hd, int block_size, float scale, int window, float softcap,
                       const float* __restrict__ sink, int keep_first, int chunk) {
  constexpr int kUnits = kPlainMaxDimsPerThread / VEC;      // pieces of VEC elements a thread may own
  extern __shared__ __align__(16) float smem[];
  float* qs = smem;                     // [hd]
  float* sc = qs + (hd + 3) / 4 * 4;    // [kPlainChunk]
  unsigned* rows_s = reinterpret_cast<unsigned*>(sc + kPlainChunk);   // [kPlainChunk] cache row of each key of the chunk
  float* joined = reinterpret_cast<float*>(rows_s + kPlainChunk);   // [kPlainThreads * VEC]
  float* scratch = joined + kPlainThreads * VEC;            // [33]
  pdl_launch_dependents();
  pdl_wait();
  const int row = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int kvh = h / (nh / nkv);
  const int ctx = positions[row] + 1;
  const int lo = first_visible(ctx - 1, window, chunk);
  const int kept = min(keep_first, lo);          // keys [0, kept) come first, then [lo, ctx)
  const int total = kept + ctx - lo;
  const int* table = block_tables + size_t(row_seq[row]) * max_blocks;

  for (int d = tid; d < hd; d += kPlainThreads)
    qs[d] = ldf(q + size_t(row) * q_stride + size_t(h) * hd + d) * scale;
  __syncthreads();

  // P*V: piece `unit` (and every 128th after it) of the keys `group`, group + groups, ...
  const int units = hd / VEC, groups = max(1, kPlainThreads / units);
  const int group = groups > 1 ? tid / units : 0, unit = groups > 1 ? tid - group * units : tid;
  float m = sink ? sink[h] : -INFINITY, l = sink ? 1.f : 0.f;
  const float inv_cap = softcap > 0.f ? 1.f / softcap : 0.f;
  float acc[kUnits][VEC];
#pragma unroll
  for (int i = 0; i < kUnits; ++i)
#pragma unroll
    for (int e = 0; e < VEC; ++e) acc[i][e] = 0.f;

  for (int c0 = 0; c0 < total; c0 += kPlainChunk) {
    const int n = min(kPlainChunk, total - c0);
    float local_max = -INFINITY;
    for (int j = tid; j < n; j += kPlainThreads) {
      const int t = c0 + j < kept ? c0 + j : c0 + j - kept + lo;
      const int page = t / block_size;
      const unsigned cache_row = (unsigned(table[page]) * nkv + kvh) * block_size + t - page * block_size;
      rows_s[j] = cache_row;
      const T* kp = k_cache + size_t(cache_row) * hd;
      float s = 0.f;
#pragma unroll 4
      for (int d = 0; d < hd; d += VEC) {
        float kv[VEC];
        load_n<VEC>(kp + d, kv);
#pragma unroll
        for (int e = 0; e < VEC; ++e) s = fmaf(qs[d + e], kv[e], s);
      }
      if (softcap > 0.f) s = softcap * tanhf(s * inv_cap);
      sc[j] = s;
      local_max = fmaxf(local_max, s);
    }
    const float m_new = fmaxf(m, block_max(local_max, scratch));
    const float factor = (m == -INFINITY) ? 0.f : expf(m - m_new);
    float local_sum = 0.f;
    for (int j = tid; j < n; j += kPlainThreads) {
      const float p = expf(sc[j] - m_new);
      sc[j] = p;
      local_sum += p;
    }
    l = l * factor + block_sum(local_sum, scratch);   // the sums' barriers also publish sc[] and rows_s[]
    m = m_new;
#pragma unroll
    for (int i = 0; i < kUnits; ++i) {
      const int u = unit + i * kPlainThreads;
      if (u >= units || group >= groups) break;
#pragma unroll
      for (int e = 0; e < VEC; ++e) acc[i][e] *= factor;
#pragma unroll 4
      for (int j = group; j < n; j += groups) {
        float vv[VEC];
        load_n<VEC>(v_cache + size_t(rows_s[j]) * hd + u * VEC, vv);
#pragma unroll
        for (int e = 0; e < VEC; ++e) acc[i][e] = fmaf(sc[j], vv[e], acc[i][e]);
      }
    }
    __syncthreads();                    // sc[] is overwritten by the next chunk
  }
  if (groups > 1) {                     // (one piece a thread) the groups' sums, in their order
    if (group < groups)
#pragma unroll
      for (int e = 0; e < VEC; ++e) joined[(group * units + unit) * VEC + e] = acc[0][e];
    __syncthreads();
    if (group == 0)
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        for (int g = 1; g < groups; ++g) acc[0][e] += joined[(g * units + unit) * VEC + e];
    if (group > 0) return;
  }
#pragma unroll
  for (int i = 0; i < kUnits; ++i) {
    const int u = unit + i * kPlainThreads;
    if (u < units)
#pragma unroll
      for (int e = 0; e < VEC; ++e)
        stf(out + size_t(row) * out_stride + size_t(h) * hd + u * VEC + e, l > 0.f ? acc[i][e] / l : 0.f);
  }
}

template <typename T>
int launch_attention_plain(const void* q, int q_stride, void* out, int out_stride, const void* k_cache,
                           const void* v_cache, const int* block_tables, int max_blocks,
                           const int* row_seq, const int* positions, int rows, int nh, int nkv, int hd,
                           int block_size, float scale, int window, float softcap, const float* sink, int keep_first, int chunk,
                           cudaStream_t s) {
  if (rows == 0) return 0;
  if (hd > kPlainMaxDimsPerThread * kPlainThreads || nkv <= 0 || nh % nkv) return KVCM_ERR_UNSUPPORTED;
  // four elements at a time where every row of the cache starts on such a piece
  const uintptr_t bases = reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache);
  const bool vec = hd % 4 == 0 && bases % (4 * sizeof(T)) == 0;
  const size_t smem = (size_t(hd + 3) / 4 * 4 + 2 * kPlainChunk + kPlainThreads * (vec ? 4 : 1) + 33) * sizeof(float);
  dim3 grid(rows, nh);
  return pdl_launch(vec ? attention_plain_kernel<T, 4> : attention_plain_kernel<T, 1>, grid, dim3(kPlainThreads), smem, s,
                    (const T*)q, q_stride, (T*)out, out_stride, (const T*)k_cache, (const T*)v_cache, block_tables,
                    max_blocks, row_seq, positions, nh, nkv, hd, block_size, scale, window, softcap, sink,
                    window > 0 && keep_first > 0 ? keep_first : 0, chunk);
}

}  // namespace kvcm

using namespace kvcm;

#define KVCM_PLAIN_ARGS                                                                                              \
  const void *q, int q_stride, void *out, int out_stride, const void *k_cache, const void *v_cache,                  \
      const int *block_tables, int max_blocks, const int *row_seq, const int *positions, int rows, int nh, int nkv, \
      int hd, int block_size, float scale, int window, float softcap, const float *sink

KVCM_API int kvcm_attention_plain_keep_f32(KVCM_PLAIN_ARGS, int keep_first, int chunk, void* stream) {
  return launch_attention_plain<float>(q, q_stride, out, out_stride, k_cache, v_cache, block_tables, max_blocks, row_seq,
                                       positions, rows, nh, nkv, hd, block_size, scale, window, softcap, sink, keep_first,
                                       chunk, (cudaStream_t)stream);
}
KVCM_API int kvcm_attention_plain_keep_bf16(KVCM_PLAIN_ARGS, int keep_first, int chunk, void* stream) {
  return launch_attention_plain<bf16>(q, q_stride, out, out_stride, k_cache, v_cache, block_tables, max_blocks, row_seq,
                                      positions, rows, nh, nkv, hd, block_size, scale, window, softcap, sink, keep_first,
                                      chunk, (cudaStream_t)stream);
}
KVCM_API int kvcm_attention_plain_f32(KVCM_PLAIN_ARGS, void* stream) {
  return kvcm_attention_plain_keep_f32(q, q_stride, out, out_stride, k_cache, v_cache, block_tables, max_blocks, row_seq,
                                       positions, rows, nh, nkv, hd, block_size, scale, window, softcap, sink, 0, 0, stream);
}
KVCM_API int kvcm_attention_plain_bf16(KVCM_PLAIN_ARGS, void* stream) {
  return kvcm_attention_plain_keep_bf16(q, q_stride, out, out_stride, k_cache, v_cache, block_tables, max_blocks, row_seq,
                                        positions, rows, nh, nkv, hd, block_size, scale, window, softcap, sink, 0, 0, stream);
}
