// Plain attention over the paged cache, one block per (token row, query head), in
// fp32 arithmetic for fp32 or bf16 storage. It is the true-32-bit product path and the
// yardstick the tensor-core kernels are tested against.
//   s_j = scale * q_h . K[j, g],  j in [max(0, pos - window + 1), pos],  g = h / (H / KV)
//   out_h = sum_j softmax(s)_j V[j, g]
// as in the reference's split kernel (src/source/op/kernels/cuda/paged_kernels.cu:96-206)
// and its oracle form (cpu/mha_kernel.cpp:112-171). Causality inside a portion comes from
// all rows' K/V being stored before this kernel runs, each row reading up to its own
// position. The order of the reduction for a row depends only on its position, never on
// the rest of the batch: the warps take runs of KEYS keys in turn with a running max, and
// their partial results are merged at the end. Bound by latency: a warp's table entries, then all key and value loads of
// a run are in flight at once, so that a run costs two round trips instead of two a key.
// Measured at one row each of six sequences of up to 216 keys, 3 heads of 32: 7.8 us, where a key at a time took 36. Heads above 128 have
// runs of two keys, which leave room for more warps (1,000 rows of two heads of 256: four keys 554 us, two 357, a key at a time 448).
#include "common.cuh"
#include <math.h>

#define REF_WARPS 8
#define REF_MAX_PER_LANE 8   // head sizes up to 256

// PER: entries of a head that a lane holds (hs <= 32 * PER); KEYS: keys of a run.
template <typename T, int PER, int KEYS>
__global__ void __launch_bounds__(REF_WARPS * 32)
paged_attention_ref_kernel(const T* __restrict__ q, long long q_row_stride,
                           const T* __restrict__ k_cache, const T* __restrict__ v_cache,
                           const int* __restrict__ block_table, int table_width,
                           const int* __restrict__ row_seq, const int* __restrict__ positions,
                           T* __restrict__ out, long long out_row_stride, int num_pages,
                           int page_size, int num_seqs, int H, int KV, int hs, float scale,
                           int window, int* status) {
  extern __shared__ float smem[];   // [REF_WARPS][hs] accumulators, then m[REF_WARPS], l[REF_WARPS]
  pdl_prologue();
  const int t = blockIdx.x, h = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = h / (H / KV);
  const int pos = positions[t];
  const int seq = row_seq[t];
  T* o = out + (size_t)t * out_row_stride + (size_t)h * hs;
  if (seq < 0 || seq >= num_seqs) {      // seq < 0 marks a padding row of a fixed-shape step
    if (threadIdx.x == 0 && seq >= 0) set_status(status, SI_BAD_SEQ);
    for (int d = threadIdx.x; d < hs; d += blockDim.x) o[d] = from_f32<T>(0.f);
    return;
  }
  const int* table = block_table + (size_t)seq * table_width;
  const T* qh = q + (size_t)t * q_row_stride + (size_t)h * hs;

  float qr[PER], acc[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int d = lane + 32 * i;
    qr[i] = d < hs ? to_f32<T>(qh[d]) : 0.f;
    acc[i] = 0.f;
  }
  float m = -INFINITY, l = 0.f;
  const int j0 = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
  for (int jb = j0 + warp * KEYS; jb <= pos; jb += REF_WARPS * KEYS) {
    long long at = -1;                   // lane u: where key jb + u lies in the caches
    if (lane < KEYS && jb + lane <= pos) {
      const int j = jb + lane, slot = j / page_size;
      const int page = slot < table_width ? table[slot] : -1;
      if (page < 0 || page >= num_pages) set_status(status, SI_BAD_PAGE);
      else at = (((long long)page * KV + g) * page_size + (j - slot * page_size)) * hs;
    }
    float k[KEYS][PER], v[KEYS][PER], dot[KEYS];
    bool have[KEYS];
#pragma unroll
    for (int u = 0; u < KEYS; ++u) {
      const long long base = __shfl_sync(0xffffffffu, at, u);
      have[u] = base >= 0;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int d = lane + 32 * i;
        const bool in = have[u] && d < hs;
        k[u][i] = in ? to_f32<T>(k_cache[base + d]) : 0.f;
        v[u][i] = in ? to_f32<T>(v_cache[base + d]) : 0.f;
      }
    }
    float m_new = m;
#pragma unroll
    for (int u = 0; u < KEYS; ++u) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < PER; ++i) s += qr[i] * k[u][i];
      dot[u] = warp_sum(s) * scale;
      if (have[u]) m_new = fmaxf(m_new, dot[u]);
    }
    if (!__any_sync(0xffffffffu, at >= 0)) continue;      // no key of the run could be read
    const float corr = expf(m - m_new);
    l *= corr;
#pragma unroll
    for (int i = 0; i < PER; ++i) acc[i] *= corr;
#pragma unroll
    for (int u = 0; u < KEYS; ++u) {
      const float p = have[u] ? expf(dot[u] - m_new) : 0.f;
      l += p;
#pragma unroll
      for (int i = 0; i < PER; ++i) acc[i] += p * v[u][i];
    }
    m = m_new;
  }
  float* sacc = smem;
  float* sm = smem + REF_WARPS * hs;
  float* sl = sm + REF_WARPS;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int d = lane + 32 * i;
    if (d < hs) sacc[warp * hs + d] = acc[i];
  }
  if (lane == 0) { sm[warp] = m; sl[warp] = l; }
  __syncthreads();
  float M = -INFINITY;
#pragma unroll
  for (int w = 0; w < REF_WARPS; ++w) M = fmaxf(M, sm[w]);
  float L = 0.f, wgt[REF_WARPS];
#pragma unroll
  for (int w = 0; w < REF_WARPS; ++w) {
    wgt[w] = sm[w] == -INFINITY ? 0.f : expf(sm[w] - M);
    L += sl[w] * wgt[w];
  }
  for (int d = threadIdx.x; d < hs; d += blockDim.x) {
    float v = 0.f;
#pragma unroll
    for (int w = 0; w < REF_WARPS; ++w) v += sacc[w * hs + d] * wgt[w];
    o[d] = from_f32<T>(L > 0.f ? v / L : 0.f);
  }
}

SI_EXPORT int si_paged_attention_ref(const void* q, int dtype, long long q_row_stride,
                                     const void* k_cache, const void* v_cache,
                                     const int* block_table, int table_width, const int* row_seq,
                                     const int* positions, void* out, long long out_row_stride,
                                     int num_pages, int page_size, int num_tokens, int num_seqs,
                                     int H, int KV, int hs, float scale, int window, int* status,
                                     cudaStream_t stream) {
  if (num_tokens <= 0) return 0;
  if (hs > 32 * REF_MAX_PER_LANE || hs <= 0 || KV <= 0 || H % KV) return -2;
  dim3 grid(num_tokens, H);
  const size_t smem = (size_t)(REF_WARPS * hs + 2 * REF_WARPS) * sizeof(float);
#define REF_LAUNCH(T, PER, KEYS)                                                                                       \
  si_launch(paged_attention_ref_kernel<T, PER, KEYS>, grid, dim3(REF_WARPS * 32), smem, stream,                      \
      (const T*)q, q_row_stride, (const T*)k_cache, (const T*)v_cache, block_table, table_width, row_seq, positions, \
      (T*)out, out_row_stride, num_pages, page_size, num_seqs, H, KV, hs, scale, window, status)
#define REF_BY_SIZE(T)                          \
  if (hs <= 32) REF_LAUNCH(T, 1, 8);            \
  else if (hs <= 64) REF_LAUNCH(T, 2, 8);       \
  else if (hs <= 128) REF_LAUNCH(T, 4, 8);      \
  else REF_LAUNCH(T, REF_MAX_PER_LANE, 2)
  if (dtype == SI_BF16) { REF_BY_SIZE(__nv_bfloat16); }
  else { REF_BY_SIZE(float); }
#undef REF_BY_SIZE
#undef REF_LAUNCH
  return si_last_error();
}
