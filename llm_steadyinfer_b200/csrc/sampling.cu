// Token selection from fp32 logits: a row held on the chip by a cluster of blocks (sample_cluster_kernel; one block a row that
// reads it again and again, sample_kernel, for vocabularies beyond what a cluster holds), or, for batches that are greedy
// throughout, the vocabulary of a row split over 32 blocks (argmax_split_kernel).
//  * greedy: argmax, ties to the lowest index, as the reference's batch argmax
//    (src/source/op/kernels/cuda/argmax_kernel.cu:14-19, 93-117).
//  * temperature / top-k / top-p: p_i = exp((x_i - max) / T); keep the k largest logits
//    (all ties of the k-th kept), then the smallest set of largest logits whose mass reaches
//    top_p of what top-k kept (ties kept); draw by inverse CDF in index order with a uniform
//    from a counter-based generator keyed by (seed, index of the output token), so that a
//    request regenerates the same tokens after preemption. The reference samples greedily only.
// The thresholds are found by bisection over the order-preserving integer image of the
// logits, so no sort and no scratch memory is needed.
#include "common.cuh"
#include <cooperative_groups.h>
#include <math.h>

namespace cg = cooperative_groups;

#define SAMPLE_THREADS 1024

// Larger float, larger key; -0.0 and +0.0, equal as numbers, get the same key (they must tie like other equals).
__device__ __forceinline__ unsigned ordered_key(float x) {
  unsigned u = __float_as_uint(x);
  if (u == 0x80000000u) u = 0u;
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float block_reduce_sum_f(float v, float* sh) {
  return block_sum(v, sh);
}

__device__ __forceinline__ float block_reduce_max_f(float v, float* sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float s = lane < nw ? sh[lane] : -INFINITY;
    s = warp_max(s);
    if (lane == 0) sh[32] = s;
  }
  __syncthreads();
  return sh[32];
}

// splitmix64 finaliser over (seed, counter) -> uniform in [0, 1) with 24 bits
__device__ __forceinline__ float uniform01(unsigned long long seed, unsigned long long counter) {
  unsigned long long z = seed ^ (counter * 0x9E3779B97F4A7C15ull);
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (float)(z >> 40) * (1.0f / 16777216.0f);
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_kernel(const float* __restrict__ logits, long long row_stride, int vocab,
              const float* __restrict__ temperature, const int* __restrict__ top_k,
              const float* __restrict__ top_p, const unsigned long long* __restrict__ seed,
              const unsigned long long* __restrict__ counter, int* __restrict__ out) {
  __shared__ float sh[33];
  __shared__ float chunk_sum[SAMPLE_THREADS];
  __shared__ int s_idx;
  pdl_prologue();
  const int r = blockIdx.x;
  const float* x = logits + (size_t)r * row_stride;
  const int tid = threadIdx.x;

  // row maximum and its lowest index
  float best = -INFINITY;
  int best_i = 0x7fffffff;
  for (int i = tid; i < vocab; i += blockDim.x) {
    const float v = x[i];
    if (v > best) { best = v; best_i = i; }
  }
  const float mx = block_reduce_max_f(best, sh);
  if (tid == 0) s_idx = 0x7fffffff;
  __syncthreads();
  if (best == mx && best_i != 0x7fffffff) atomicMin(&s_idx, best_i);
  __syncthreads();
  const float T = temperature ? temperature[r] : 0.f;
  if (!(T > 0.f)) {
    if (tid == 0) out[r] = s_idx == 0x7fffffff ? 0 : s_idx;
    return;
  }
  const float invT = 1.f / T;
  const int k = top_k ? top_k[r] : 0;
  const float pp = top_p ? top_p[r] : 1.f;

  unsigned lo_key = 0;                       // keep logits whose key >= lo_key
  if (k > 0 && k < vocab) {
    // largest key u with count{key >= u} >= k
    unsigned lo = 0, hi = 0xffffffffu;
    while (lo < hi) {
      const unsigned mid = lo + ((hi - lo) >> 1) + 1;
      float c = 0.f;
      for (int i = tid; i < vocab; i += blockDim.x) c += ordered_key(x[i]) >= mid ? 1.f : 0.f;
      c = block_reduce_sum_f(c, sh);
      if (c >= (float)k) lo = mid; else hi = mid - 1;
    }
    lo_key = lo;
  }
  // mass kept by top-k
  float z = 0.f;
  for (int i = tid; i < vocab; i += blockDim.x)
    if (ordered_key(x[i]) >= lo_key) z += expf((x[i] - mx) * invT);
  z = block_reduce_sum_f(z, sh);
  if (pp < 1.f) {
    const float target = pp * z;
    unsigned lo = lo_key, hi = ordered_key(mx);
    while (lo < hi) {
      const unsigned mid = lo + ((hi - lo) >> 1) + 1;
      float s = 0.f;
      for (int i = tid; i < vocab; i += blockDim.x)
        if (ordered_key(x[i]) >= mid) s += expf((x[i] - mx) * invT);
      s = block_reduce_sum_f(s, sh);
      if (s >= target) lo = mid; else hi = mid - 1;
    }
    lo_key = lo;
    z = 0.f;
    for (int i = tid; i < vocab; i += blockDim.x)
      if (ordered_key(x[i]) >= lo_key) z += expf((x[i] - mx) * invT);
    z = block_reduce_sum_f(z, sh);
  }
  // inverse CDF in index order: thread i owns the contiguous chunk [i*c, (i+1)*c)
  const float u = uniform01(seed ? seed[r] : 0ull, counter ? counter[r] : 0ull);
  const float target = u * z;
  const int chunk = (vocab + blockDim.x - 1) / blockDim.x;
  const int b = tid * chunk, e = min(vocab, b + chunk);
  float mine = 0.f;
  for (int i = b; i < e; ++i)
    if (ordered_key(x[i]) >= lo_key) mine += expf((x[i] - mx) * invT);
  chunk_sum[tid] = mine;
  __syncthreads();
  if (tid == 0) {
    // the walk over per-thread sums is short (1024 entries) and keeps one summation order
    float run = 0.f;
    int owner = -1;
    float before = 0.f;
    int last_nonempty = -1;
    for (int i = 0; i < (int)blockDim.x; ++i) {
      if (chunk_sum[i] > 0.f) last_nonempty = i;
      if (owner < 0 && chunk_sum[i] > 0.f && run + chunk_sum[i] > target) { owner = i; before = run; }
      run += chunk_sum[i];
    }
    if (owner < 0) { owner = last_nonempty; before = run - chunk_sum[owner < 0 ? 0 : owner]; }
    s_idx = owner;
    sh[0] = before;
  }
  __syncthreads();
  if (tid == s_idx) {
    float run = sh[0];
    int pick = -1, last = -1;
    for (int i = b; i < e; ++i) {
      if (ordered_key(x[i]) >= lo_key) {
        last = i;
        run += expf((x[i] - mx) * invT);
        if (run > target) { pick = i; break; }
      }
    }
    out[r] = pick >= 0 ? pick : last;
  }
}

// The same choice with the row on the chip. A cluster of up to 8 blocks shares a row: a thread keeps the keys of its VPT groups of
// four logits in registers and their weights exp((x - max) / T) in its own places of shared memory, so the row is read from
// memory once. A threshold is bracketed by a histogram over 256 equal steps of the logit (counts, or masses as whole numbers, so
// that the order of the atomics changes nothing) and then found among the few keys of one step in rounds: a warp shows its keys
// between the bounds to its lanes one by one, every lane compares with a value of its own, a 33rd of the range is left. The blocks'
// numbers meet in each other's shared memory, one cluster barrier an exchange, and every block adds them in the same order and so
// decides alike. The range for top-p starts at max - T (ln(vocab / (1 - top_p)) + 1): what lies below weighs less than 1 - top_p
// of the maximum alone. A group of 128 logits (a warp's loads) without a key between the bounds is added up once and then left.
// Bound by the exchanges' latency (some ten of 1 to 2 us) and, from 37 rows of 128,256 logits on, by the second round of clusters
// over the SMs, not by memory. Rows of 128,256 logits, temperature 0.7, top_p 0.9, a launch behind a launch: 64 rows 1,142 us with a block a
// row that reads it some 40 times, 77 us here (86 with the rows in memory); 8 rows 30 us (47); top_k 50 instead 64 and 25 us; no restriction 31
// and 11 us.
#define SC_THREADS 512
#define SC_WARPS (SC_THREADS / 32)
#define SC_MAX_CLUSTER 8

struct SampleShared {
  float red[3][SC_WARPS];
  float slot[2][SC_MAX_CLUSTER][4];      // a round's sums of every block, two rounds in turn
  unsigned hist[256];
  float mass[256];
  int bins[2];
  float lanes[SC_WARPS][32];             // a fine round: per warp the sums of 32 thresholds, then every block's, two in turn
  float lane_slot[2][SC_MAX_CLUSTER][32];
  float part[16 * SC_WARPS];             // kept mass per (group, warp) in index order
  int pick;
};

// Sums of three values over the cluster, in the same order in every block. `turn` alternates from call to call.
__device__ __forceinline__ void cluster_sum3(cg::cluster_group& cl, SampleShared& sm, int& turn, float& a, float& b, float& c) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  a = warp_sum(a); b = warp_sum(b); c = warp_sum(c);
  if (lane == 0) { sm.red[0][warp] = a; sm.red[1][warp] = b; sm.red[2][warp] = c; }
  __syncthreads();
  const int blocks = (int)cl.num_blocks();
  if (warp == 0) {
    a = lane < SC_WARPS ? sm.red[0][lane] : 0.f;
    b = lane < SC_WARPS ? sm.red[1][lane] : 0.f;
    c = lane < SC_WARPS ? sm.red[2][lane] : 0.f;
    a = warp_sum(a); b = warp_sum(b); c = warp_sum(c);
    if (lane < blocks) {
      float* d = cl.map_shared_rank(&sm.slot[turn][0][0], lane) + 4 * (int)cl.block_rank();
      d[0] = a; d[1] = b; d[2] = c;
    }
  }
  cl.sync();                             // every block's sums are here; the next call writes the other slots
  a = b = c = 0.f;
  for (int r = 0; r < blocks; ++r) { a += sm.slot[turn][r][0]; b += sm.slot[turn][r][1]; c += sm.slot[turn][r][2]; }
  turn ^= 1;
}

__device__ __forceinline__ float key_value(unsigned u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u); }

// Narrows (lo, hi] to the keys of the histogram's step in which count or mass reaches `target` (two neighbouring steps where the
// masses' rounding leaves it open). `within`: keys of the row between the bounds, before and after; false: nothing was done.
template <int VPT, bool COUNT>
__device__ __forceinline__ bool cluster_narrow(cg::cluster_group& cl, SampleShared& sm, int& turn, const unsigned (&key)[VPT][4],
                                               const float4* weight, unsigned& lo, unsigned& hi, float target, float mx, float invT,
                                               float bottom, float& within) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, blocks = (int)cl.num_blocks();
  const float v_hi = key_value(hi), v_lo = fmaxf(key_value(lo), bottom), inv = 255.f / (v_hi - v_lo), step = (v_hi - v_lo) * (1.f / 255.f) * invT;
  if (!(inv > 0.f) || isinf(inv) || (!COUNT && !(step < 0.5f))) return false;
  auto bin_of = [&](unsigned u) { return (int)fminf((v_hi - key_value(u)) * inv, 255.f); };     // -infinity: the last one
  if (threadIdx.x < 256) sm.hist[threadIdx.x] = 0u;
  __syncthreads();
  float above = 0.f, z1 = 0.f, z2 = 0.f;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const float4 v = COUNT ? make_float4(1.f, 1.f, 1.f, 1.f) : weight[j * SC_THREADS];
    const float ww[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const unsigned u = key[j][i];
      if (u > hi) above += ww[i];
      else if (u > lo) {
        const int bin = bin_of(u);
        // a mass relative to its step's upper end, in 16 bits: rounding below 1e-5 of it; a block's sum stays below 2^31
        atomicAdd(&sm.hist[bin], COUNT ? 1u : (unsigned)(fminf(expf((key_value(u) - v_hi) * invT + (float)bin * step), 1.f) * 65536.f + 0.5f));
      }
    }
  }
  cluster_sum3(cl, sm, turn, above, z1, z2);             // (its barrier also stands between the histograms and their readers)
  if (threadIdx.x < 256) {
    unsigned long long n = 0;
    for (int b = 0; b < blocks; ++b) n += cl.map_shared_rank(&sm.hist[0], b)[threadIdx.x];
    sm.mass[threadIdx.x] = COUNT ? (float)n : (float)n * (1.f / 65536.f) * expf((v_hi - mx) * invT - (float)threadIdx.x * step);
  }
  __syncthreads();
  if (warp == 0) {
    float own = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) own += sm.mass[lane * 8 + i];
    float before = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float v = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += v;
    }
    before += above - own;
    const float slack = COUNT ? 0.f : 2e-5f;
    int may = 256, must = 256;                           // the first step that may, that must, reach the target
    for (int i = 0; i < 8; ++i) {
      before += sm.mass[lane * 8 + i];
      if (may == 256 && before * (1.f + slack) >= target) may = lane * 8 + i;
      if (must == 256 && before * (1.f - slack) >= target) must = lane * 8 + i;
    }
    may = __reduce_min_sync(0xffffffffu, may);
    must = __reduce_min_sync(0xffffffffu, must);
    if (lane == 0) { sm.bins[0] = may; sm.bins[1] = must; }
  }
  __syncthreads();
  const int may = sm.bins[0], must = sm.bins[1];
  unsigned least = 0xffffffffu, most = 0u, n = 0u;
#pragma unroll
  for (int j = 0; j < VPT; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const unsigned u = key[j][i];
      if (u > lo && u <= hi) {
        const int bin = bin_of(u);
        if (bin >= may && bin <= must) { least = min(least, u); most = max(most, u); ++n; }
      }
    }
  least = __reduce_min_sync(0xffffffffu, least);
  most = __reduce_max_sync(0xffffffffu, most);
  n = __reduce_add_sync(0xffffffffu, n);
  if (lane == 0) { sm.red[0][warp] = __uint_as_float(least); sm.red[1][warp] = __uint_as_float(most); sm.red[2][warp] = (float)n; }
  __syncthreads();
  if (warp == 0) {
    least = __reduce_min_sync(0xffffffffu, lane < SC_WARPS ? __float_as_uint(sm.red[0][lane]) : 0xffffffffu);
    most = __reduce_max_sync(0xffffffffu, lane < SC_WARPS ? __float_as_uint(sm.red[1][lane]) : 0u);
    const float c = warp_sum(lane < SC_WARPS ? sm.red[2][lane] : 0.f);
    if (lane < blocks) {
      float* d = cl.map_shared_rank(&sm.slot[turn][0][0], lane) + 4 * (int)cl.block_rank();
      d[0] = __uint_as_float(least); d[1] = __uint_as_float(most); d[2] = c;
    }
  }
  cl.sync();                                             // also: every block has read the histograms
  least = 0xffffffffu; most = 0u;
  float c = 0.f;
  for (int b = 0; b < blocks; ++b) {
    least = min(least, __float_as_uint(sm.slot[turn][b][0]));
    most = max(most, __float_as_uint(sm.slot[turn][b][1]));
    c += sm.slot[turn][b][2];
  }
  turn ^= 1;
  if (c == 0.f) { hi = lo; within = 0.f; return true; }  // nothing between the bounds reaches it: lo does
  if (must < 256) lo = least;                            // its step reaches the target
  hi = most;
  within = c;
  return true;
}

// The largest u in [lo, hi] whose keys >= u have at least `target` of count (COUNT) or mass; lo is taken to have it. `within`: how
// many keys of the row lie between the bounds, the same number in every block; `bottom`: the row's least logit.
#define SC_FINE 1024                     // keys between the bounds up to which the rounds begin
template <int VPT, bool COUNT>
__device__ __forceinline__ unsigned cluster_threshold(cg::cluster_group& cl, SampleShared& sm, int& turn, const unsigned (&key)[VPT][4],
                                                      const float4* weight, unsigned lo, unsigned hi, float target, float mx, float invT,
                                                      float bottom, float within) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, blocks = (int)cl.num_blocks();
  for (int level = 0; level < 3 && within > (float)SC_FINE && lo < hi; ++level)
    if (!cluster_narrow<VPT, COUNT>(cl, sm, turn, key, weight, lo, hi, target, mx, invT, bottom, within)) break;
  unsigned active = (1u << VPT) - 1u;
  float above = 0.f;                     // of groups that are done: what lies above the range
  auto retire = [&]() {                  // groups without a key between the bounds
#pragma unroll
    for (int j = 0; j < VPT; ++j)
      if (active >> j & 1u) {
        bool in = false;
#pragma unroll
        for (int i = 0; i < 4; ++i) in |= key[j][i] > lo && key[j][i] <= hi;
        if (!__any_sync(0xffffffffu, in)) {
          const float4 w = COUNT ? make_float4(1.f, 1.f, 1.f, 1.f) : weight[j * SC_THREADS];
          above += (key[j][0] > hi ? w.x : 0.f) + (key[j][1] > hi ? w.y : 0.f) + (key[j][2] > hi ? w.z : 0.f) + (key[j][3] > hi ? w.w : 0.f);
          active &= ~(1u << j);
        }
      }
  };
  int flip = 0;
  while (lo < hi) {
    retire();
    // lane l stands for lo + (l + 1) q, the last ones cut at hi; the 33 parts cover the range
    const unsigned w = hi - lo, q = w / 33u + (w % 33u != 0u);
    const unsigned mine = (unsigned)min((unsigned long long)lo + (unsigned long long)(lane + 1) * q, (unsigned long long)hi);
    float s = 0.f, over = above;
#pragma unroll
    for (int j = 0; j < VPT; ++j)
      if (active >> j & 1u) {
        const float4 v = COUNT ? make_float4(1.f, 1.f, 1.f, 1.f) : weight[j * SC_THREADS];
        const float ww[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (key[j][i] > hi) over += ww[i];                               // counts for every lane
          unsigned who = __ballot_sync(0xffffffffu, key[j][i] > lo && key[j][i] <= hi);
          while (who) {
            const int from = __ffs(who) - 1;
            who &= who - 1u;
            const unsigned u = __shfl_sync(0xffffffffu, key[j][i], from);
            const float f = __shfl_sync(0xffffffffu, ww[i], from);
            s += u >= mine ? f : 0.f;
          }
        }
      }
    sm.lanes[warp][lane] = s + warp_sum(over);
    __syncthreads();
    if (warp == 0) {
      s = 0.f;
#pragma unroll
      for (int i = 0; i < SC_WARPS; ++i) s += sm.lanes[i][lane];
      for (int b = 0; b < blocks; ++b) cl.map_shared_rank(&sm.lane_slot[flip][0][0], b)[32 * (int)cl.block_rank() + lane] = s;
    }
    cl.sync();
    s = 0.f;
    for (int b = 0; b < blocks; ++b) s += sm.lane_slot[flip][b][lane];
    flip ^= 1;
    const unsigned have = __ballot_sync(0xffffffffu, s >= target);
    // the largest threshold that has it; the next one (where there is one above) bounds the range
    const int top = have ? 31 - __clz(have) : -1;
    const unsigned next = __shfl_sync(0xffffffffu, mine, min(top + 1, 31)), at = __shfl_sync(0xffffffffu, mine, max(top, 0));
    if (top >= 0) lo = at;
    if (top < 31 && next > lo) hi = next - 1u;
  }
  return lo;
}

template <int VPT>
__global__ void __launch_bounds__(SC_THREADS, VPT <= 8 ? 2 : 1)
sample_cluster_kernel(const float* __restrict__ logits, long long row_stride, int vocab, int per_block, int vec,
                      const float* __restrict__ temperature, const int* __restrict__ top_k,
                      const float* __restrict__ top_p, const unsigned long long* __restrict__ seed,
                      const unsigned long long* __restrict__ counter, int* __restrict__ out) {
  extern __shared__ float4 weights[];    // [VPT][SC_THREADS]
  __shared__ SampleShared sm;
  cg::cluster_group cl = cg::this_cluster();
  const int blocks = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int r = blockIdx.x / blocks, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  cl.barrier_arrive();                   // waited for before the first store into another block's memory
  pdl_prologue();
  const float* x = logits + (size_t)r * row_stride;
  const int first = rank * per_block, end = min(vocab, first + per_block);     // this block's logits

  // four neighbouring logits a group; places behind the end get key 0 and weight 0
  unsigned key[VPT][4];
  float best = -INFINITY, least = INFINITY;
  int best_i = 0x7fffffff;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    const int at = first + 4 * (j * SC_THREADS + tid);
    float v[4];
    if (vec && at + 4 <= end) {
      const float4 f = __ldcs(reinterpret_cast<const float4*>(x + at));
      v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) v[i] = at + i < end ? x[at + i] : -INFINITY;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (v[i] > best) { best = v[i]; best_i = at + i; }
      if (v[i] > -INFINITY) least = fminf(least, v[i]);
      key[j][i] = at + i < end ? ordered_key(v[i]) : 0u;
    }
  }
  // the row's maximum and its lowest index, and its least finite logit
  auto better = [](float& m, int& i, float m2, int i2) { if (m2 > m || (m2 == m && i2 < i)) { m = m2; i = i2; } };
  auto warp_best = [&](float& m, int& i) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float m2 = __shfl_xor_sync(0xffffffffu, m, o);
      const int i2 = __shfl_xor_sync(0xffffffffu, i, o);
      better(m, i, m2, i2);
    }
  };
  warp_best(best, best_i);
  least = -warp_max(-least);
  if (lane == 0) { sm.red[0][warp] = best; sm.red[1][warp] = __int_as_float(best_i); sm.red[2][warp] = least; }
  __syncthreads();
  cl.barrier_wait();
  int turn = 0;
  if (warp == 0) {
    best = lane < SC_WARPS ? sm.red[0][lane] : -INFINITY;
    best_i = lane < SC_WARPS ? __float_as_int(sm.red[1][lane]) : 0x7fffffff;
    warp_best(best, best_i);
    least = -warp_max(lane < SC_WARPS ? -sm.red[2][lane] : -INFINITY);
    if (lane < blocks) {
      float* d = cl.map_shared_rank(&sm.slot[turn][0][0], lane) + 4 * rank;
      d[0] = best; d[1] = __int_as_float(best_i); d[2] = least;
    }
  }
  cl.sync();
  best = -INFINITY; best_i = 0x7fffffff; least = INFINITY;
  for (int b = 0; b < blocks; ++b) {
    better(best, best_i, sm.slot[turn][b][0], __float_as_int(sm.slot[turn][b][1]));
    least = fminf(least, sm.slot[turn][b][2]);
  }
  turn ^= 1;
  if (best_i == 0x7fffffff) best_i = 0;
  const float mx = best, T = temperature ? temperature[r] : 0.f;
  if (!(T > 0.f)) {                      // every block of the cluster comes here or none; nobody reads another's memory any more
    if (rank == 0 && tid == 0) out[r] = best_i;
    return;
  }
  const float invT = 1.f / T;
  const int k = top_k ? top_k[r] : 0;
  const float pp = top_p ? top_p[r] : 1.f;
  float4* weight = weights + tid;
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    float w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      w[i] = key[j][i] ? expf((key_value(key[j][i]) - mx) * invT) : 0.f;
    }
    weight[j * SC_THREADS] = make_float4(w[0], w[1], w[2], w[3]);      // read by this thread only
  }

  unsigned lo_key = 0;                   // keep logits whose key >= lo_key
  const unsigned hi_key = ordered_key(mx);
  if (k > 0 && k < vocab)                // largest key u with count{key >= u} >= k
    lo_key = cluster_threshold<VPT, true>(cl, sm, turn, key, weight, 0u, hi_key, (float)k, mx, invT, least, (float)vocab);
  if (pp < 1.f) {
    const float low = mx - T * (logf((float)vocab / (1.f - pp)) + 1.f);
    const unsigned low_key = max(lo_key, low < mx ? ordered_key(low) : 0u);      // (not a number or no step below the maximum: the whole range)
    float z = 0.f, n = 0.f, none = 0.f;  // mass kept by top-k, keys between the bounds
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const float4 w = weight[j * SC_THREADS];
#pragma unroll
      for (int i = 0; i < 4; ++i) n += key[j][i] > low_key && key[j][i] <= hi_key ? 1.f : 0.f;
      z += (key[j][0] >= lo_key ? w.x : 0.f) + (key[j][1] >= lo_key ? w.y : 0.f) + (key[j][2] >= lo_key ? w.z : 0.f) + (key[j][3] >= lo_key ? w.w : 0.f);
    }
    cluster_sum3(cl, sm, turn, z, n, none);
    lo_key = cluster_threshold<VPT, false>(cl, sm, turn, key, weight, low_key, hi_key, pp * z, mx, invT, least, n);
  }
  // inverse CDF in index order: blocks, then groups and warps, then lanes, then a lane's four
#pragma unroll
  for (int j = 0; j < VPT; ++j) {
    float4 w = weight[j * SC_THREADS];
    w.x = key[j][0] >= lo_key ? w.x : 0.f; w.y = key[j][1] >= lo_key ? w.y : 0.f;
    w.z = key[j][2] >= lo_key ? w.z : 0.f; w.w = key[j][3] >= lo_key ? w.w : 0.f;
    weight[j * SC_THREADS] = w;          // what is not kept weighs nothing from here on
    const float s = warp_sum(w.x + w.y + w.z + w.w);
    if (lane == 0) sm.part[j * SC_WARPS + warp] = s;
  }
  __syncthreads();
  constexpr int PARTS = VPT * SC_WARPS, PER = PARTS / 32;
  static_assert(PARTS % 32 == 0, "a lane takes the same number of parts");
  float before = 0.f, all = 0.f, share = 0.f;
  if (warp == 0) {
#pragma unroll
    for (int i = 0; i < PER; ++i) share += sm.part[lane * PER + i];
    before = share;                      // inclusive prefix over the lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float v = __shfl_up_sync(0xffffffffu, before, o);
      if (lane >= o) before += v;
    }
    const float total = __shfl_sync(0xffffffffu, before, 31);
    if (lane < blocks) cl.map_shared_rank(&sm.slot[turn][0][0], lane)[4 * rank] = total;
  }
  cl.sync();                             // the last exchange: from here on a block reads its own memory only
  for (int b = 0; b < blocks; ++b) all += sm.slot[turn][b][0];
  const float target = uniform01(seed ? seed[r] : 0ull, counter ? counter[r] : 0ull) * all;
  int owner = -1, last = -1;
  float run = 0.f, owner_before = 0.f, last_before = 0.f;
  for (int b = 0; b < blocks; ++b) {
    const float s = sm.slot[turn][b][0];
    if (s > 0.f) { last = b; last_before = run; }
    if (owner < 0 && s > 0.f && run + s > target) { owner = b; owner_before = run; }
    run += s;
  }
  if (owner < 0) { owner = last; owner_before = last_before; }
  if (owner < 0) {                       // no mass at all (not a number, or infinite logits): the maximum
    if (rank == 0 && tid == 0) out[r] = best_i;
    return;
  }
  if (owner != rank) return;
  if (warp == 0) {
    const unsigned over = __ballot_sync(0xffffffffu, share > 0.f && owner_before + before > target);
    const unsigned any = __ballot_sync(0xffffffffu, share > 0.f);
    const int from = over ? __ffs(over) - 1 : 31 - __clz(any);
    if (lane == from) {
      float at = owner_before + (before - share), keep = at;
      int pick = -1;
      for (int i = 0; i < PER; ++i) {
        const float s = sm.part[lane * PER + i];
        if (s > 0.f) {
          pick = lane * PER + i; keep = at;
          if (at + s > target) break;
        }
        at += s;
      }
      sm.pick = pick;
      sm.red[0][0] = keep;
    }
  }
  __syncthreads();
  const int pick = sm.pick;
  if (warp != pick % SC_WARPS) return;
  const float base = sm.red[0][0];
  const int group = (pick / SC_WARPS) * SC_THREADS;
  const float4 f = weight[group];
  const float mine = f.x + f.y + f.z + f.w;
  float upto = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float v = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += v;
  }
  const unsigned over = __ballot_sync(0xffffffffu, mine > 0.f && base + upto > target);
  const unsigned any = __ballot_sync(0xffffffffu, mine > 0.f);
  if (lane == (over ? __ffs(over) - 1 : 31 - __clz(any))) {
    float at = base + (upto - mine);
    int id = 0;
    if (f.x > 0.f) at += f.x;
    if (f.y > 0.f && !(at > target && f.x > 0.f)) { id = 1; at += f.y; }
    if (f.z > 0.f && !(at > target && (f.x > 0.f || f.y > 0.f))) { id = 2; at += f.z; }
    if (f.w > 0.f && !(at > target && (f.x > 0.f || f.y > 0.f || f.z > 0.f))) id = 3;
    out[r] = first + 4 * (group + tid) + id;
  }
}

// Greedy rows only: the vocabulary of a row is split over ARGMAX_SPLITS blocks, each leaves its
// (maximum, lowest index) in `scratch`, and the block that comes last (a ticket per row) merges them;
// it also puts the ticket back to zero for the next launch. One block per row, as in sample_kernel,
// leaves most of the SMs idle while a few of them read the whole row.
#define ARGMAX_SPLITS 32
#define ARGMAX_THREADS 256

__global__ void __launch_bounds__(ARGMAX_THREADS)
argmax_split_kernel(const float* __restrict__ logits, long long row_stride, int vocab, float* __restrict__ part_max,
                    int* __restrict__ part_idx, int* __restrict__ tickets, int* __restrict__ out) {
  __shared__ float sh[33];
  __shared__ int s_idx, s_last;
  pdl_prologue();
  const int r = blockIdx.y, sp = blockIdx.x;
  const float* x = logits + (size_t)r * row_stride;
  const int per = (vocab + ARGMAX_SPLITS - 1) / ARGMAX_SPLITS;
  const int b = sp * per, e = min(vocab, b + per);
  float best = -INFINITY;
  int best_i = 0x7fffffff;
  for (int i = b + threadIdx.x; i < e; i += ARGMAX_THREADS) {
    const float v = x[i];
    if (v > best) { best = v; best_i = i; }
  }
  const float mx = block_reduce_max_f(best, sh);
  if (threadIdx.x == 0) s_idx = 0x7fffffff;
  __syncthreads();
  if (best == mx && best_i != 0x7fffffff) atomicMin(&s_idx, best_i);
  __syncthreads();
  if (threadIdx.x == 0) {
    part_max[r * ARGMAX_SPLITS + sp] = mx;
    part_idx[r * ARGMAX_SPLITS + sp] = s_idx;
    __threadfence();
    s_last = atomicAdd(&tickets[r], 1) == ARGMAX_SPLITS - 1;
  }
  __syncthreads();
  if (!s_last || threadIdx.x >= 32) return;
  __threadfence();
  float m = __ldcg(part_max + r * ARGMAX_SPLITS + threadIdx.x);     // ARGMAX_SPLITS == 32: one per lane
  int idx = __ldcg(part_idx + r * ARGMAX_SPLITS + threadIdx.x);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, idx, o);
    if (m2 > m || (m2 == m && i2 < idx)) { m = m2; idx = i2; }
  }
  if (threadIdx.x == 0) {
    out[r] = idx == 0x7fffffff ? 0 : idx;
    tickets[r] = 0;
  }
}

// Words of scratch (4 bytes each) that si_argmax needs for up to `capacity` rows; the caller zeroes them
// once. The tickets stand first, so that they lie in the same place for every number of rows.
SI_EXPORT long long si_argmax_scratch_words(int capacity) { return (long long)capacity * (2 * ARGMAX_SPLITS + 1); }

SI_EXPORT int si_argmax(const float* logits, long long row_stride, int num_rows, int vocab, void* scratch, int capacity,
                        int* out, cudaStream_t stream) {
  if (num_rows <= 0) return 0;
  if (!scratch || num_rows > capacity || num_rows > 65535) return -2;
  int* tickets = (int*)scratch;
  float* part_max = (float*)scratch + capacity;
  int* part_idx = (int*)scratch + capacity + (size_t)capacity * ARGMAX_SPLITS;
  si_launch(argmax_split_kernel, dim3(ARGMAX_SPLITS, num_rows), dim3(ARGMAX_THREADS), 0, stream, logits, row_stride,
            vocab, part_max, part_idx, tickets, out);
  return si_last_error();
}

SI_EXPORT int si_sample(const float* logits, long long row_stride, int num_rows, int vocab,
                        const float* temperature, const int* top_k, const float* top_p,
                        const unsigned long long* seed, const unsigned long long* counter,
                        int* out, cudaStream_t stream) {
  if (num_rows <= 0) return 0;
  // A cluster holds 8 x 16 x 2,048 logits. One block is quicker than a cluster's barriers up to 4,096, and up to 16,384 where the rows'
  // clusters do not all run at once (128 rows of 4,100 logits: 66 us with eight blocks a row, 18 with one; 256 rows of 16,384: 131 and 36).
  const bool one_wave = (long long)num_rows * SC_MAX_CLUSTER <= 2LL * si_sm_count();
  const int blocks = vocab <= (one_wave ? 2 : 8) * 4 * SC_THREADS ? 1 : SC_MAX_CLUSTER;
  const int per_block = ((vocab + blocks - 1) / blocks + 3) / 4 * 4;
  const int groups = (per_block + 4 * SC_THREADS - 1) / (4 * SC_THREADS);
  if (groups > 16 || (long long)num_rows * blocks > 0x7fffffffLL) {
    si_launch(sample_kernel, dim3(num_rows), dim3(SAMPLE_THREADS), 0, stream, logits, row_stride, vocab, temperature,
              top_k, top_p, seed, counter, out);
    return si_last_error();
  }
  const int vec = row_stride % 4 == 0 && ((uintptr_t)logits & 15) == 0;
  auto go = [&](auto kernel, int vpt) {
    const size_t smem = (size_t)vpt * SC_THREADS * sizeof(float4);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(num_rows * blocks));
    cfg.blockDim = dim3(SC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = si_pdl_enabled() ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, kernel, logits, row_stride, vocab, per_block, vec, temperature, top_k, top_p, seed, counter, out);
    return e != cudaSuccess ? (int)e : si_last_error();
  };
  if (groups <= 2) return go(sample_cluster_kernel<2>, 2);
  if (groups <= 4) return go(sample_cluster_kernel<4>, 4);
  if (groups <= 8) return go(sample_cluster_kernel<8>, 8);
  return go(sample_cluster_kernel<16>, 16);
}
