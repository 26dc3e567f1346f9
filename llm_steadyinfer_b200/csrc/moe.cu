// Routed feed-forward ("mixture of experts"): every row chooses `top` of E small feed-forwards by a score and adds their
// results, weighted. Everything that depends on the choice happens on the device: no count travels to the host, so a
// step through these kernels can be recorded in a graph.
//   moe_route    scores z = W_r x (fp32 sums over the row in fp32), s = sigmoid(z) (or softmax over the experts), the `top`
//                largest (ties: the lower index), weights s * scale (optionally divided by their sum); rows of further
//                gate matrices behind the router's give sigmoid(w . x) for the same row (a gate on a shared expert).
//                With a choice bias the `top` largest of s + bias are chosen instead; the weights stay s. With groups the experts
//                fall into `groups` equal runs of neighbours; only those of the `keep` runs with the largest sum of their two best
//                choice scores can be chosen.
//   moe_plan     the (row, choice) pairs ordered by expert, rows in step order within an expert: offsets per expert, the
//                row of every place, the place of every pair. Counting ranks within chunks of 1,024 pairs, so the order
//                never depends on timing.
//   moe_gemm     C[place] = act(A[row of place] W_e^T) for every place of expert e: a grouped product whose row tiles are
//                found from the offsets by every block itself (blocks beyond the last tile leave). bf16 on mma.sync
//                m16n8k16 with fp32 sums: few places an expert stream its weights (moe_stream_kernel), more go by tiles of 64
//                rows x 64 columns, three cp.async stages (16 rows, four stages, where few are not in 16-byte pieces); fp32 on FFMA.
//                act "glu_limited": W_e holds gate and up rows in turn (row 2i the gate of entry i, row 2i + 1 its up), and
//                C[place, i] = g sigmoid(alpha g) (u + shift) with g = min(gate sum, limit), u = clamp(up sum, -limit, limit)
//                (no limit, alpha 1 and shift 0: silu(gate) * up).
//                A row's sums run over k in the same order wherever the row lies in its tile. (Many rows in bf16
//                go to the tcgen05 grouped product of gemm_tc05.cu instead, behind `moe_gather`.)
//   moe_combine  out[t] = sum_c weight[t, c] * Y[place(t, c)] (+ gate[t] * shared[t]), the choices in their own order.
//                A choice whose id is not below `real` names an identity expert: its result is the row x[t] itself.
#include "common.cuh"
#include <math.h>
#include <mma.h>

typedef __nv_bfloat16 bf16;

// ---- router -------------------------------------------------------------------------------------------------------------
// x [T, d]; w [E + extra, d] (router rows, then `extra` gate rows) in the compute dtype; ids int32 [T, top]; wts fp32
// [T, top]; gates fp32 [T, extra]. mode 0: sigmoid scores; 1: softmax over the experts. A block takes a row, a warp a weight row at a time.
// EARLY (no more rows than SMs): as many warps as weight rows, up to 32, and a warp's first 256 x ROUTE_AHEAD weights, which do not depend
// on the kernel before, are in flight before the block waits for x. A row's sums run over k in the same order either way. Bound by latency
// (a round trip for the weights, one for the row, the choice by one warp): four rows, a launch behind a launch, d = 2,048 and 64 experts
// 20.7 us with eight warps that read the weights behind the wait and 12.0 so, d = 1,536 and 32 experts 10.1 and 5.8. With more rows than
// SMs the eight warps serve (591 rows, d = 2,048, 64 experts: 31.0 us; four rows a block took 32.4, and 97 against 89 at 2,048 rows).
#define ROUTE_AHEAD 4
template <typename T, bool EARLY>
__global__ void __launch_bounds__(EARLY ? 1024 : 256) moe_route_kernel(const T* __restrict__ x, long long x_stride, const T* __restrict__ w,
    int E, int extra, int d, int top, float scale, int mode, int renorm, float renorm_eps, int groups, int keep,
    const float* __restrict__ choice_bias, int* __restrict__ ids, float* __restrict__ wts, float* __restrict__ gates, int trigger) {
  if (trigger) pdl_trigger();
  extern __shared__ float rsm[];                       // the row [d], scores [E + extra], used [E], choice keys [E] (and groups' scores)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const long long t = blockIdx.x;
  float* xr = rsm;
  float* sc = rsm + d;
  float* used = sc + E + extra;
  float* key = used + E;
  const bool wide = sizeof(T) == 2 && d % 8 == 0 && ((uintptr_t)w & 15) == 0;      // rows of 16-byte pieces: eight entries a load
  uint4 ahead[ROUTE_AHEAD];
  if (EARLY && wide && warp < E + extra) {
#pragma unroll
    for (int u = 0; u < ROUTE_AHEAD; ++u)
      if (lane * 8 + u * 256 < d) ahead[u] = *reinterpret_cast<const uint4*>(w + (size_t)warp * d + lane * 8 + u * 256);
  }
  pdl_wait();
  if (EARLY && wide && x_stride % 8 == 0 && ((uintptr_t)x & 15) == 0) {
    for (int at = threadIdx.x * 8; at < d; at += blockDim.x * 8) {
      const uint4 raw = *reinterpret_cast<const uint4*>(x + t * x_stride + at);
      const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
      for (int j = 0; j < 4; ++j) reinterpret_cast<float2*>(xr + at)[j] = __bfloat1622float2(h2[j]);
    }
  } else {
    for (int i = threadIdx.x; i < d; i += blockDim.x) xr[i] = to_f32<T>(x[t * x_stride + i]);
  }
  for (int e = threadIdx.x; e < E; e += blockDim.x) used[e] = 0.f;
  __syncthreads();
  for (int e = warp; e < E + extra; e += nwarps) {
    const T* we = w + (size_t)e * d;
    float acc = 0.f;
    if (wide) {
      int from = lane * 8;
      if (EARLY && e == warp) {
#pragma unroll
        for (int u = 0; u < ROUTE_AHEAD; ++u)
          if (lane * 8 + u * 256 < d) {
            const int i = lane * 8 + u * 256;
            const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&ahead[u]);
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
              const float2 f = __bfloat1622float2(h2[j]), h = __bfloat1622float2(h2[j + 1]);
              const float4 xv = *reinterpret_cast<const float4*>(xr + i + 2 * j);
              acc = fmaf(f.x, xv.x, acc); acc = fmaf(f.y, xv.y, acc);
              acc = fmaf(h.x, xv.z, acc); acc = fmaf(h.y, xv.w, acc);
            }
          }
        from += ROUTE_AHEAD * 256;
      }
      for (int i = from; i < d; i += 256) {
        const uint4 raw = *reinterpret_cast<const uint4*>(we + i);
        const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = __bfloat1622float2(h2[j]);
          acc = fmaf(f.x, xr[i + 2 * j], acc);
          acc = fmaf(f.y, xr[i + 2 * j + 1], acc);
        }
      }
    } else {
      for (int i = lane; i < d; i += 32) acc = fmaf(to_f32<T>(we[i]), xr[i], acc);
    }
    acc = warp_sum(acc);
    if (lane == 0) sc[e] = acc;
  }
  __syncthreads();
  if (warp != 0) return;                               // one warp chooses
  for (int e = lane; e < extra; e += 32) gates[t * extra + e] = 1.f / (1.f + expf(-sc[E + e]));
  float zmax = -INFINITY, zsum = 0.f;
  if (mode == 1) {
    for (int e = lane; e < E; e += 32) zmax = fmaxf(zmax, sc[e]);
    zmax = warp_max(zmax);
    for (int e = lane; e < E; e += 32) zsum += expf(sc[e] - zmax);
    zsum = warp_sum(zsum);
  }
  // what the choice goes by: the sums themselves (the scores rise with them), or score + bias where a bias is given
  for (int e = lane; e < E; e += 32) {
    float kv = sc[e];
    if (choice_bias) kv = (mode == 1 ? expf(sc[e] - zmax) / zsum : 1.f / (1.f + expf(-sc[e]))) + choice_bias[e];
    key[e] = kv;
  }
  __syncwarp();
  if (groups > 1 && keep < groups) {                     // experts of the groups that are not kept cannot be chosen
    float* gscore = key + E;
    const int size = E / groups;
    for (int g = lane; g < groups; g += 32) {
      float b1 = -INFINITY, b2 = -INFINITY;
      for (int e = g * size; e < (g + 1) * size; ++e) {
        const float kv = key[e];
        if (kv > b1) { b2 = b1; b1 = kv; } else if (kv > b2) { b2 = kv; }
      }
      gscore[g] = size > 1 ? b1 + b2 : b1;
    }
    __syncwarp();
    for (int g = lane; g < groups; g += 32) {
      int better = 0;                                    // groups before this one in the order of scores (ties: the lower index)
      for (int o = 0; o < groups; ++o) better += gscore[o] > gscore[g] || (gscore[o] == gscore[g] && o < g);
      if (better >= keep)
        for (int e = g * size; e < (g + 1) * size; ++e) used[e] = 1.f;
    }
    __syncwarp();
  }
  float total = 0.f, mine = 0.f;
  int my_id = 0;
  // up to 32 experts: a lane an expert, the largest of order-preserving whole numbers in one instruction
  unsigned held = 0u;
  if (E <= 32 && lane < E && used[lane] == 0.f) {
    unsigned u = __float_as_uint(key[lane] + 0.f);       // (-0 becomes 0: equal keys tie)
    held = max((u & 0x80000000u) ? ~u : (u | 0x80000000u), 1u);
  }
  for (int c = 0; c < top; ++c) {
    float best = -INFINITY;
    int idx = -1;
    if (E <= 32) {
      const unsigned most = __reduce_max_sync(0xffffffffu, held);
      if (most) idx = __ffs(__ballot_sync(0xffffffffu, held == most)) - 1;
      if (lane == idx) held = 0u;
    } else {
    for (int e = lane; e < E; e += 32)
      if (used[e] == 0.f && (idx < 0 || key[e] > best)) { best = key[e]; idx = e; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
      if (oi >= 0 && (idx < 0 || ob > best || (ob == best && oi < idx))) { best = ob; idx = oi; }
    }
    }
    if (idx < 0) idx = 0;                              // fewer experts than choices: never with a checked configuration
    const float z = sc[idx];
    const float s = mode == 1 ? expf(z - zmax) / zsum : 1.f / (1.f + expf(-z));
    total += s;
    if (lane == c % 32 && c < 32) { mine = s; my_id = idx; }
    if (lane == 0) used[idx] = 1.f;
    __syncwarp();
  }
  if (lane < top) {
    ids[t * top + lane] = my_id;
    wts[t * top + lane] = (renorm ? mine / (total + renorm_eps) : mine) * scale;
  }
}

SI_EXPORT int si_moe_route(const void* x, int dtype, long long x_stride, const void* w, int E, int extra, int d, int top,
                           float scale, int mode, int renorm, float renorm_eps, int groups, int keep, const float* choice_bias,
                           int* ids, float* wts, float* gates, int rows, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (E <= 0 || top <= 0 || top > E || top > 32 || extra < 0 || d <= 0 || mode < 0 || mode > 1) return -2;
  if (groups > 1 && (E % groups || keep < 1 || keep > groups || !choice_bias)) return -2;      // groups go by choice scores
  if (groups > 1 && (long long)keep * (E / groups) < top) return -2;
  const size_t smem = (size_t)(d + 3 * E + extra + (groups > 1 ? groups : 0)) * sizeof(float);
  if (smem > 160 * 1024) return -2;
  const bool early = rows <= si_sm_count();
  const int trigger = early ? si_pdl_trigger_mode(rows, si_sm_count()) : 0;
  const int warps = E + extra < 32 ? E + extra : 32;
  const dim3 grid(rows), block(early ? 32 * warps : E + extra >= 8 ? 256 : 128);
#define ROUTE_LAUNCH(T)                                                                                                \
  {                                                                                                                  \
    static size_t configured = 0;                                                                                    \
    if (smem > 48 * 1024 && smem > configured) {                                                                     \
      if (cudaFuncSetAttribute(moe_route_kernel<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess       \
          || cudaFuncSetAttribute(moe_route_kernel<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return -2; \
      configured = smem;                                                                                             \
    }                                                                                                                \
    si_launch(early ? moe_route_kernel<T, true> : moe_route_kernel<T, false>, grid, block, smem, stream, (const T*)x, x_stride, (const T*)w, E, extra, d, top, scale, \
              mode, renorm, renorm_eps, groups, keep, choice_bias, ids, wts, gates, trigger);                                                        \
  }
  if (dtype == SI_BF16) ROUTE_LAUNCH(bf16) else ROUTE_LAUNCH(float)
#undef ROUTE_LAUNCH
  return si_last_error();
}

// ---- plan ---------------------------------------------------------------------------------------------------------------
#define PLAN_CHUNK 1024

// One chunk of pairs: every pair's rank among the pairs of the same expert before it in the chunk, and the chunk's count
// per expert.
__device__ void plan_rank_chunk(const int* __restrict__ ids, int P, int E, int chunk, int* __restrict__ rank,
                                int* __restrict__ counts, int* sm_ids) {
  const int base = chunk * PLAN_CHUNK;
  const int n = min(PLAN_CHUNK, P - base);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    int e = ids[base + i];
    sm_ids[i] = (e < 0 || e >= E) ? 0 : e;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int e = sm_ids[i];
    int r = 0;
    for (int j = 0; j < i; ++j) r += sm_ids[j] == e;
    rank[base + i] = r;
  }
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int c = 0;
    for (int j = 0; j < n; ++j) c += sm_ids[j] == e;
    counts[(size_t)chunk * E + e] = c;
  }
}

// counts [chunks, E] become the first place of every (chunk, expert); offsets [E + 1] the first place of every expert.
__device__ void plan_offsets(int* __restrict__ counts, int chunks, int E, int* __restrict__ offsets, int* sm_tot) {
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int c = 0;
    for (int k = 0; k < chunks; ++k) c += counts[(size_t)k * E + e];
    sm_tot[e] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int e = 0; e < E; ++e) { const int c = sm_tot[e]; sm_tot[e] = acc; offsets[e] = acc; acc += c; }
    offsets[E] = acc;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < E; e += blockDim.x) {
    int acc = sm_tot[e];
    for (int k = 0; k < chunks; ++k) { const int c = counts[(size_t)k * E + e]; counts[(size_t)k * E + e] = acc; acc += c; }
  }
}

__device__ void plan_place(const int* __restrict__ ids, const int* __restrict__ rank, const int* __restrict__ counts, int P,
                           int E, int top, int first, int last, int* __restrict__ row_of, int* __restrict__ place_of) {
  for (int i = first + threadIdx.x; i < last; i += blockDim.x) {
    int e = ids[i];
    e = (e < 0 || e >= E) ? 0 : e;
    const int place = counts[(size_t)(i / PLAN_CHUNK) * E + e] + rank[i];
    row_of[place] = i / top;
    place_of[i] = place;
  }
}

__global__ void __launch_bounds__(1024) moe_plan_one_kernel(const int* __restrict__ ids, int P, int E, int top,
    int* __restrict__ rank, int* __restrict__ counts, int* __restrict__ offsets, int* __restrict__ row_of,
    int* __restrict__ place_of) {
  extern __shared__ int psm[];                         // ids of the chunk [PLAN_CHUNK], totals [E]
  pdl_prologue();
  plan_rank_chunk(ids, P, E, 0, rank, counts, psm);
  __syncthreads();
  plan_offsets(counts, 1, E, offsets, psm + PLAN_CHUNK);
  __syncthreads();
  plan_place(ids, rank, counts, P, E, top, 0, P, row_of, place_of);
}
__global__ void __launch_bounds__(1024) moe_plan_rank_kernel(const int* __restrict__ ids, int P, int E, int* __restrict__ rank,
                                                             int* __restrict__ counts) {
  extern __shared__ int psm[];
  pdl_prologue();
  plan_rank_chunk(ids, P, E, blockIdx.x, rank, counts, psm);
}
__global__ void __launch_bounds__(1024) moe_plan_offsets_kernel(int* __restrict__ counts, int chunks, int E, int* __restrict__ offsets) {
  extern __shared__ int psm[];
  pdl_prologue();
  plan_offsets(counts, chunks, E, offsets, psm);
}
__global__ void __launch_bounds__(1024) moe_plan_place_kernel(const int* __restrict__ ids, const int* __restrict__ rank,
    const int* __restrict__ counts, int P, int E, int top, int* __restrict__ row_of, int* __restrict__ place_of) {
  pdl_prologue();
  const int first = blockIdx.x * PLAN_CHUNK;
  plan_place(ids, rank, counts, P, E, top, first, min(P, first + PLAN_CHUNK), row_of, place_of);
}

SI_EXPORT long long si_moe_plan_ints(int P, int E) {        // scratch of the plan: ranks, then counts per chunk
  const long long chunks = (P + PLAN_CHUNK - 1) / PLAN_CHUNK;
  return (long long)P + chunks * E;
}

SI_EXPORT int si_moe_plan(const int* ids, int P, int E, int top, int* scratch, int* offsets, int* row_of, int* place_of,
                          cudaStream_t stream) {
  if (P <= 0) return 0;
  if (E <= 0 || E > 8192 || top <= 0 || P % top) return -2;
  const int chunks = (P + PLAN_CHUNK - 1) / PLAN_CHUNK;
  int* rank = scratch;
  int* counts = scratch + P;
  const int threads = P >= PLAN_CHUNK ? 1024 : ((P + 31) / 32) * 32;
  if (chunks == 1) {
    si_launch(moe_plan_one_kernel, dim3(1), dim3(threads), (size_t)(PLAN_CHUNK + E) * sizeof(int), stream, ids, P, E, top, rank,
              counts, offsets, row_of, place_of);
  } else {
    si_launch(moe_plan_rank_kernel, dim3(chunks), dim3(1024), (size_t)PLAN_CHUNK * sizeof(int), stream, ids, P, E, rank, counts);
    si_launch(moe_plan_offsets_kernel, dim3(1), dim3(E >= 512 ? 1024 : 256), (size_t)E * sizeof(int), stream, counts, chunks, E,
              offsets);
    si_launch(moe_plan_place_kernel, dim3(chunks), dim3(1024), 0, stream, ids, (const int*)rank, (const int*)counts, P, E, top,
              row_of, place_of);
  }
  return si_last_error();
}

// ---- grouped product ------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float moe_act(float v, int act) {
  if (act == 1) { const float r = fmaxf(v, 0.f); return r * r; }           // the square of relu
  if (act == 2) return v / (1.f + expf(-v));                               // silu
  if (act == 3) return 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));   // gelu_tanh
  return v;
}
#define MOE_ACT_GLU_LIMITED 4
// gate and up sums of one entry (neighbouring columns of the product): g sigmoid(alpha g) (u + shift) within the limit
__device__ __forceinline__ float moe_glu_limited(float gate, float up, float limit, float alpha, float shift) {
  const float g = fminf(gate, limit), u = fminf(fmaxf(up, -limit), limit);
  return g / (1.f + expf(-alpha * g)) * (u + shift);
}

// The tile a block takes: expert, first place, places. Thread 0 walks the offsets; false: no tile is left for this block.
__device__ __forceinline__ bool moe_find_tile(const int* __restrict__ offsets, int E, int BM, int tile, int* sm3) {
  if (threadIdx.x == 0) {
    int acc = 0, found = -1, first = 0, rows = 0;
    for (int e = 0; e < E; ++e) {
      const int a = offsets[e], cnt = offsets[e + 1] - a;
      const int tiles = (cnt + BM - 1) / BM;
      if (tile < acc + tiles) { found = e; first = a + (tile - acc) * BM; rows = min(BM, a + cnt - first); break; }
      acc += tiles;
    }
    sm3[0] = found; sm3[1] = first; sm3[2] = rows;
  }
  __syncthreads();
  return sm3[0] >= 0;
}

#define MOE_BN 64
// A tile row in shared memory holds BK + 8 bf16 entries (fragment loads without bank conflicts).

__device__ __forceinline__ void moe_cp16(void* dst, const void* src, int bytes) {       // bytes < 16: the rest is zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes));
}

// A [*, K] rows (row of place p: a_rows[p], or p itself when a_rows is absent); W [E, N, K]; C [places, N] (bf16 or fp32).
template <int BM, int BN, int MOE_BK, int MOE_STAGES>
__global__ void __launch_bounds__(128) moe_gemm_bf16_kernel(const bf16* __restrict__ A, long long a_stride,
    const int* __restrict__ a_rows, const bf16* __restrict__ W, void* __restrict__ C, long long c_stride, int c_f32,
    const int* __restrict__ offsets, int E, int N, int K, int act, int wide, float limit, float alpha, float shift) {
  constexpr int MOE_PITCH = MOE_BK + 8, KC = MOE_BK / 8;
  __shared__ __align__(16) bf16 As[MOE_STAGES][BM][MOE_PITCH];
  __shared__ __align__(16) bf16 Ws[MOE_STAGES][BN][MOE_PITCH];
  __shared__ int tile_info[3];
  __shared__ int src_row[BM];
  pdl_prologue();
  if (!moe_find_tile(offsets, E, BM, blockIdx.x, tile_info)) return;
  const int e = tile_info[0], first = tile_info[1], rows = tile_info[2];
  const int n0 = blockIdx.y * BN;
  for (int r = threadIdx.x; r < BM; r += blockDim.x) src_row[r] = r < rows ? (a_rows ? a_rows[first + r] : first + r) : -1;
  __syncthreads();
  const bf16* We = W + (size_t)e * N * K;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, tq = lane & 3;
  constexpr int NT = BM == 64 ? BN / 8 : BN / 32;    // n-tiles of 8 columns a warp: warps over the rows, or over the columns
  const int wr0 = BM == 64 ? warp * 16 : 0, wn0 = BM == 64 ? 0 : warp * (BN / 4);
  float acc[NT][4];
#pragma unroll
  for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
  const int ktiles = (K + MOE_BK - 1) / MOE_BK;
  auto load = [&](int kt, int buf) {
    const int k0 = kt * MOE_BK;
    if (wide) {
      for (int c = threadIdx.x; c < (BM + BN) * KC; c += blockDim.x) {
        const int r = c / KC, kc = (c % KC) * 8;
        const int left = K - (k0 + kc);
        const int bytes = left >= 8 ? 16 : (left > 0 ? left * 2 : 0);
        if (r < BM) {
          const int sr = src_row[r];
          const bf16* src = sr >= 0 ? A + (size_t)sr * a_stride + k0 + kc : A;
          moe_cp16(&As[buf][r][kc], bytes > 0 ? src : A, sr >= 0 ? bytes : 0);
        } else {
          const int n = n0 + r - BM;
          const bf16* src = We + (size_t)(n < N ? n : 0) * K + k0 + kc;
          moe_cp16(&Ws[buf][r - BM][kc], bytes > 0 ? src : We, n < N ? bytes : 0);
        }
      }
    } else {                                           // rows that are not 16-byte aligned: entry by entry
      for (int c = threadIdx.x; c < (BM + BN) * MOE_BK; c += blockDim.x) {
        const int r = c / MOE_BK, kk = c % MOE_BK;
        const bool kin = k0 + kk < K;
        if (r < BM) {
          const int sr = src_row[r];
          As[buf][r][kk] = (sr >= 0 && kin) ? A[(size_t)sr * a_stride + k0 + kk] : __float2bfloat16_rn(0.f);
        } else {
          const int n = n0 + r - BM;
          Ws[buf][r - BM][kk] = (n < N && kin) ? We[(size_t)n * K + k0 + kk] : __float2bfloat16_rn(0.f);
        }
      }
    }
    asm volatile("cp.async.commit_group;\n" ::);
  };
  for (int s = 0; s < MOE_STAGES - 1; ++s) {
    if (s < ktiles) load(s, s);
    else asm volatile("cp.async.commit_group;\n" ::);
  }
  for (int kt = 0; kt < ktiles; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(MOE_STAGES - 2) : "memory");
    __syncthreads();
    if (kt + MOE_STAGES - 1 < ktiles) load(kt + MOE_STAGES - 1, (kt + MOE_STAGES - 1) % MOE_STAGES);
    else asm volatile("cp.async.commit_group;\n" ::);
    const int buf = kt % MOE_STAGES;
#pragma unroll
    for (int kk = 0; kk < MOE_BK; kk += 16) {
      unsigned a0 = *reinterpret_cast<const unsigned*>(&As[buf][wr0 + g][kk + 2 * tq]);
      unsigned a1 = *reinterpret_cast<const unsigned*>(&As[buf][wr0 + g + 8][kk + 2 * tq]);
      unsigned a2 = *reinterpret_cast<const unsigned*>(&As[buf][wr0 + g][kk + 8 + 2 * tq]);
      unsigned a3 = *reinterpret_cast<const unsigned*>(&As[buf][wr0 + g + 8][kk + 8 + 2 * tq]);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int nn = wn0 + nt * 8 + g;
        unsigned b0 = *reinterpret_cast<const unsigned*>(&Ws[buf][nn][kk + 2 * tq]);
        unsigned b1 = *reinterpret_cast<const unsigned*>(&Ws[buf][nn][kk + 8 + 2 * tq]);
        asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                     : "+f"(acc[nt][0]), "+f"(acc[nt][1]), "+f"(acc[nt][2]), "+f"(acc[nt][3])
                     : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int r = wr0 + g + half * 8;
      if (r >= rows) continue;
      const size_t place = (size_t)(first + r);
      if (act == MOE_ACT_GLU_LIMITED) {                 // the thread's two columns are an entry's gate and up
        const int n = n0 + wn0 + nt * 8 + 2 * tq;
        if (n + 1 >= N) continue;
        const float v = moe_glu_limited(acc[nt][half * 2], acc[nt][half * 2 + 1], limit, alpha, shift);
        if (c_f32) reinterpret_cast<float*>(C)[place * c_stride + (n >> 1)] = v;
        else reinterpret_cast<bf16*>(C)[place * c_stride + (n >> 1)] = __float2bfloat16_rn(v);
        continue;
      }
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const int n = n0 + wn0 + nt * 8 + 2 * tq + c;
        if (n >= N) continue;
        const float v = moe_act(acc[nt][half * 2 + c], act);
        if (c_f32) reinterpret_cast<float*>(C)[place * c_stride + n] = v;
        else reinterpret_cast<bf16*>(C)[place * c_stride + n] = __float2bfloat16_rn(v);
      }
    }
  }
}

// Few places an expert (decode rows, short portions): a stream of the chosen experts' weights, as gemm_skinny.cu streams a
// matrix. A block takes 16 columns of one expert for up to 16 of its places; its eight warps take the 32-wide chunks of k in turn,
// with a warp's loads of four chunks (both operands, 16 bytes a lane) in flight at once, straight into the fragments of
// mma.sync m16n8k16 (the weights are its 16 rows, the places its 8 columns), and their sums are added in warp order. The places come
// from the plan (offsets and rows); steps of at most 32 (row, choice) pairs have a kernel of their own (moe_pairs_kernel).
__device__ __forceinline__ void moe_mma(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 moe_ld(const bf16* p, bool stream) {
  uint4 v;
  if (stream) asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  else asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}

#define STREAM_WARPS 8
template <int MT>
__device__ __forceinline__ void moe_stream_tile(const bf16* __restrict__ A, long long a_stride, const int* src_row, const bf16* __restrict__ We,
                                                int n0, int N, int K, float (*red)[2][32][4]) {
  constexpr int U = MT == 1 ? 4 : 2;     // three blocks an SM: one's start and end under the others' loads
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const bf16* w0 = We + (size_t)min(n0 + g, N - 1) * K + t * 8;          // rows beyond N stand for the last one: never stored
  const bf16* w1 = We + (size_t)min(n0 + 8 + g, N - 1) * K + t * 8;
  const bf16* xr[MT];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) xr[mt] = A + (size_t)src_row[mt * 8 + g] * a_stride + t * 8;
  float acc[MT][4];
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) acc[mt][0] = acc[mt][1] = acc[mt][2] = acc[mt][3] = 0.f;
  const int nchunks = (K + 31) >> 5;
  for (int c = warp; c < nchunks; c += STREAM_WARPS * U) {
    uint4 lo[U], hi[U], xb[U][MT];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (c + u * STREAM_WARPS) * 32;
      lo[u] = hi[u] = make_uint4(0, 0, 0, 0);
      if (k + t * 8 < K) { lo[u] = moe_ld(w0 + k, true); hi[u] = moe_ld(w1 + k, true); }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = (c + u * STREAM_WARPS) * 32;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        xb[u][mt] = make_uint4(0, 0, 0, 0);
        if (k + t * 8 < K) xb[u][mt] = moe_ld(xr[mt] + k, false);
      }
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (c + u * STREAM_WARPS < nchunks) {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          moe_mma(acc[mt], lo[u].x, hi[u].x, lo[u].y, hi[u].y, xb[u][mt].x, xb[u][mt].y);
          moe_mma(acc[mt], lo[u].z, hi[u].z, lo[u].w, hi[u].w, xb[u][mt].z, xb[u][mt].w);
        }
      }
  }
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int i = 0; i < 4; ++i) red[warp][mt][lane][i] = acc[mt][i];
}

__global__ void __launch_bounds__(STREAM_WARPS * 32, 3) moe_stream_kernel(const bf16* __restrict__ A, long long a_stride,
    const int* __restrict__ a_rows, const bf16* __restrict__ W, void* __restrict__ C,
    long long c_stride, int c_f32, const int* __restrict__ offsets, int E, int N, int K, int act, float limit, float alpha,
    float shift) {
  __shared__ float red[STREAM_WARPS][2][32][4];
  __shared__ int place[16], src_row[16], info[2];
  pdl_prologue();
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    int e = -1, rows = 0, mine = -1;                     // lane l < 16: the tile's place l
    int before = 0, first = 0;
    for (int base = 0; base < E && e < 0; base += 32) {
      const int x = base + lane;
      const int a = x < E ? offsets[x] : 0, n = x < E ? offsets[x + 1] - a : 0;
      const int tiles = (n + 15) / 16;
      int upto = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
      }
      upto += before;
      const unsigned past = __ballot_sync(0xffffffffu, (int)blockIdx.y < upto);
      if (past) {
        const int at = __ffs(past) - 1;
        const int skip = ((int)blockIdx.y - (upto - tiles)) * 16;      // of lane `at`: places of the expert before this tile
        first = __shfl_sync(0xffffffffu, a + skip, at);
        rows = __shfl_sync(0xffffffffu, min(n - skip, 16), at);
        e = base + at;
      }
      before = __shfl_sync(0xffffffffu, upto, 31);
    }
    if (e >= 0 && lane < rows) mine = first + lane;
    const int head = __shfl_sync(0xffffffffu, mine, 0);
    if (lane < 16) {                                     // places that are not there stand for the first one: never stored
      const int p = mine >= 0 ? mine : head;
      place[lane] = mine;
      src_row[lane] = p < 0 ? 0 : a_rows ? a_rows[p] : p;
    }
    if (lane == 0) { info[0] = e; info[1] = rows; }
  }
  __syncthreads();
  const int e = info[0], rows = info[1], n0 = blockIdx.x * 16;
  if (e < 0) return;
  const bf16* We = W + (size_t)e * N * K;
  if (rows <= 8) moe_stream_tile<1>(A, a_stride, src_row, We, n0, N, K, red);
  else moe_stream_tile<2>(A, a_stride, src_row, We, n0, N, K, red);
  __syncthreads();
  const bool pair = act == MOE_ACT_GLU_LIMITED;
  // a thread adds the warps' sums of one column (or of a gate and its up, neighbours) of one place
  const int per_place = pair ? 8 : 16;
  for (int i = threadIdx.x; i < rows * per_place; i += STREAM_WARPS * 32) {
    const int r = i / per_place, q = i % per_place, mt = r >> 3;
    auto sum = [&](int col) {                            // column of the 16: fragment (lane (col % 8, r % 8 / 2), element)
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < STREAM_WARPS; ++w) v += red[w][mt][(col & 7) * 4 + ((r & 7) >> 1)][(col >> 3) * 2 + (r & 1)];
      return v;
    };
    const size_t at = (size_t)place[r] * c_stride;
    float v;
    int n;
    if (pair) {
      n = n0 + 2 * q;
      if (n + 1 >= N) continue;
      v = moe_glu_limited(sum(2 * q), sum(2 * q + 1), limit, alpha, shift);
      n >>= 1;
    } else {
      n = n0 + q;
      if (n >= N) continue;
      v = moe_act(sum(q), act);
    }
    if (c_f32) reinterpret_cast<float*>(C)[at + n] = v;
    else reinterpret_cast<bf16*>(C)[at + n] = __float2bfloat16_rn(v);
  }
}

// ---- few pairs ------------------------------------------------------------------------------------------------------------
// A matrix that every row takes, beside the chosen ones (the shared expert's): C[t] = form(A[t] W^T) for `rows` rows, at most 16.
// form 0 the sum; 1 the square of relu; 2 silu(gate) * up; 3 the limited form with biases (fp32 in the rows' order, or null). The latter two
// have gates and ups in groups of 8 rows. The sums are rounded to bf16 before a form, as the few-row product does that serves it alone.
struct MoeShared {
  const bf16* A; long long a_stride;
  const bf16* W;
  bf16* C; long long c_stride;
  const float* bias;
  int rows, N, K, form;
  float limit, alpha;
};

__device__ __forceinline__ uint4 moe_ld_if(const bf16* p, bool take, bool stream) {      // without a branch; not taken: zeros
  uint4 v;
  if (stream)
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
                 "@q ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}\n"
                 : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w) : "l"(p), "r"((int)take) : "memory");
  else
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %5, 0;\n\tmov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\tmov.u32 %3, 0;\n\t"
                 "@q ld.global.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}\n"
                 : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w) : "l"(p), "r"((int)take) : "memory");
  return v;
}

// At most 32 (row, choice) pairs of at most 16 rows: a pair is a place of its own, and no plan is made; pair p reads row p / a_div of A.
// Tiles of 16 columns, first the shared matrix's, then expert by expert as they are first chosen, go in turn to two blocks an SM. A block's
// warps take the 32-wide chunks of k in turn, UP of them at once with both operands, straight into the fragments of mma.sync; the next
// round's loads (of this tile or the next) are on their way while the warps' sums are added, so that a block's start and the latency of a round
// are paid once, and blocks that begin with the shared matrix ask for its weights before the wait for the router. Bound by the stream of
// weights. Both products of 2,048 columns, in us, as launches of their own with a block a tile and the shared expert behind them, and so: one
// row of two experts of 1,408 and a shared one of 2,816 (69 MB) 23.1, 14.3; three rows of six without gates (69 MB) 28.4, 18.1; two rows of
// eight and none shared (138 MB) 31.3, 25.5.
template <int MT>
__global__ void __launch_bounds__(STREAM_WARPS * 32, 2) moe_pairs_kernel(const bf16* __restrict__ A, long long a_stride,
    const int* __restrict__ ids, int a_div, const bf16* __restrict__ W, void* __restrict__ C, long long c_stride, int c_f32, int P, int E,
    int N, int K, int act, float limit, float alpha, float shift, int trigger, const MoeShared sh) {
  constexpr int UP = MT == 1 ? 8 : 4, PLACES = MT * 8;  // places that a tile's sums have room for
  __shared__ float red[2][STREAM_WARPS][MT][32][4];
  __shared__ int place[32][PLACES], count[32], expert[32], entries;
  if (trigger) pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int nx = (N + 15) / 16, ns = (sh.N + 15) / 16;
  // The tiles go to the blocks forwards and backwards in turn: the first ones (the shared matrix's) may be the longer ones.
  int q = blockIdx.x, pass = 0, r = 0, y = 0, n0 = 0, width = 0, depth = 0;      // the tile and round whose loads were asked for last
  uint4 lo[UP], hi[UP], xb[UP][MT];
  auto load_w = [&]() {
    const bf16* w;
    if (q < ns) {
      n0 = q * 16; w = sh.W; width = sh.N; depth = sh.K;
    } else {
      y = (q - ns) / nx;
      n0 = (q - ns - y * nx) * 16; w = W + (size_t)expert[y] * N * K; width = N; depth = K;
    }
    const bf16* w0 = w + (size_t)min(n0 + g, width - 1) * depth;       // rows beyond the matrix stand for the last one: never stored
    const bf16* w1 = w + (size_t)min(n0 + 8 + g, width - 1) * depth;
#pragma unroll
    for (int u = 0; u < UP; ++u) {
      const int k = (warp + (r * UP + u) * STREAM_WARPS) * 32 + t * 8;
      lo[u] = moe_ld_if(w0 + k, k < depth, true);
      hi[u] = moe_ld_if(w1 + k, k < depth, true);
    }
  };
  auto load_x = [&]() {
    const bool shared = q < ns;
    const int rows = shared ? sh.rows : count[y];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      const int i = mt * 8 + g;
      const bool in = i < rows;
      const bf16* xr = shared ? sh.A + (long long)(in ? i : 0) * sh.a_stride : A + (long long)(place[y][in ? i : 0] / a_div) * a_stride;
#pragma unroll
      for (int u = 0; u < UP; ++u) {
        const int k = (warp + (r * UP + u) * STREAM_WARPS) * 32 + t * 8;
        xb[u][mt] = moe_ld_if(xr + k, in && k < depth, false);
      }
    }
  };
  if (q < ns) load_w();                                  // the shared matrix does not depend on the choice before this kernel
  pdl_wait();
  if (warp == 0) {
    int id = lane < P ? ids[lane] : -1;
    if (id < 0 || id >= E) id = -1;                      // (identity experts and none: no product)
    // An expert is one entry, as a row's choices are different experts; ids that name one more often than its rows make an entry of every
    // PLACES places.
    const unsigned same = __match_any_sync(0xffffffffu, id), below = (1u << lane) - 1;
    const int rank = __popc(same & below), first = rank - rank % PLACES;
    const unsigned leaders = __ballot_sync(0xffffffffu, id >= 0 && rank == first);
    if (id >= 0) {
      const int leader = first == 0 ? __ffs(same) - 1 : (int)__fns(same, 0, first + 1);
      const int at = __popc(leaders & ((1u << leader) - 1));
      place[at][rank - first] = lane;
      if (rank == first) { expert[at] = id; count[at] = min(__popc(same) - first, PLACES); }
    }
    if (lane == 0) entries = __popc(leaders);
  }
  __syncthreads();
  const int total = ns + entries * nx;
  if (q < total) {
    if (q >= ns) load_w();
    load_x();
  }
  int par = 0;
  while (q < total) {
    float acc[MT][4];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) acc[mt][0] = acc[mt][1] = acc[mt][2] = acc[mt][3] = 0.f;
    const bool shared = q < ns;
    const int rows = shared ? sh.rows : count[y], tile_y = y, tile_n0 = n0, tile_width = width;
    const int rounds = (depth + STREAM_WARPS * UP * 32 - 1) / (STREAM_WARPS * UP * 32);
    for (int round = 0; round < rounds; ++round) {
#pragma unroll
      for (int u = 0; u < UP; ++u)
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          moe_mma(acc[mt], lo[u].x, hi[u].x, lo[u].y, hi[u].y, xb[u][mt].x, xb[u][mt].y);
          moe_mma(acc[mt], lo[u].z, hi[u].z, lo[u].w, hi[u].w, xb[u][mt].z, xb[u][mt].w);
        }
      if (++r == rounds) {
        r = 0;
        ++pass;
        q = pass * gridDim.x + ((pass & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
      }
      if (q < total) { load_w(); load_x(); }
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
      *reinterpret_cast<float4*>(red[par][warp][mt][lane]) = make_float4(acc[mt][0], acc[mt][1], acc[mt][2], acc[mt][3]);
    __syncthreads();
    // a thread adds the warps' sums of one column (or of a gate and its up) of one place
    const bool gated = shared ? sh.form >= 2 : act == MOE_ACT_GLU_LIMITED;
    const int per_place = gated ? 8 : 16, gap = shared ? 8 : 1;        // the shared matrix has gates and ups in eights, the experts' in turn
    for (int i = threadIdx.x; i < rows * per_place; i += STREAM_WARPS * 32) {
      const int row = i / per_place, c = i % per_place, mt = row >> 3;
      auto sum = [&](int col) {                          // column of the 16: fragment (lane (col % 8, row % 8 / 2), element)
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < STREAM_WARPS; ++w) v += red[par][w][mt][(col & 7) * 4 + ((row & 7) >> 1)][(col >> 3) * 2 + (row & 1)];
        return v;
      };
      const int first = gated && !shared ? 2 * c : c;
      if (tile_n0 + first + (gated ? gap : 0) >= tile_width) continue;
      float v = sum(first), up = gated ? sum(first + gap) : 0.f;
      const int n = gated ? (tile_n0 >> 1) + c : tile_n0 + c;
      if (shared) {
        v = __bfloat162float(__float2bfloat16_rn(v));
        up = __bfloat162float(__float2bfloat16_rn(up));
        if (sh.form == 3) {
          if (sh.bias) { v += sh.bias[tile_n0 + c]; up += sh.bias[tile_n0 + 8 + c]; }
          v = moe_glu_limited(v, up, sh.limit, sh.alpha, 1.f);
        } else {
          v = sh.form == 2 ? silu_mul(v, up) : moe_act(v, sh.form);
        }
        sh.C[(size_t)row * sh.c_stride + n] = __float2bfloat16_rn(v);
      } else {
        v = gated ? moe_glu_limited(v, up, limit, alpha, shift) : moe_act(v, act);
        const size_t at = (size_t)place[tile_y][row] * c_stride + n;
        if (c_f32) reinterpret_cast<float*>(C)[at] = v;
        else reinterpret_cast<bf16*>(C)[at] = __float2bfloat16_rn(v);
      }
    }
    par ^= 1;
  }
}

// True 32-bit: tiles of 32 places x 64 columns, 16 entries of k at a time, a thread 2 x 4 results.
__global__ void __launch_bounds__(256) moe_gemm_f32_kernel(const float* __restrict__ A, long long a_stride,
    const int* __restrict__ a_rows, const float* __restrict__ W, float* __restrict__ C, long long c_stride,
    const int* __restrict__ offsets, int E, int N, int K, int act, float limit, float alpha, float shift) {
  constexpr int BM = 32, BK = 16;
  __shared__ float As[BK][BM + 1];
  __shared__ float Ws[BK][MOE_BN + 1];
  __shared__ int tile_info[3];
  __shared__ int src_row[BM];
  pdl_prologue();
  if (!moe_find_tile(offsets, E, BM, blockIdx.x, tile_info)) return;
  const int e = tile_info[0], first = tile_info[1], rows = tile_info[2];
  const int n0 = blockIdx.y * MOE_BN;
  for (int r = threadIdx.x; r < BM; r += blockDim.x) src_row[r] = r < rows ? (a_rows ? a_rows[first + r] : first + r) : -1;
  __syncthreads();
  const float* We = W + (size_t)e * N * K;
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
  float acc[2][4] = {};
  for (int k0 = 0; k0 < K; k0 += BK) {
    for (int c = threadIdx.x; c < (BM + MOE_BN) * BK; c += blockDim.x) {
      const int r = c / BK, kk = c % BK;
      const bool kin = k0 + kk < K;
      if (r < BM) {
        const int sr = src_row[r];
        As[kk][r] = (sr >= 0 && kin) ? A[(size_t)sr * a_stride + k0 + kk] : 0.f;
      } else {
        const int n = n0 + r - BM;
        Ws[kk][r - BM] = (n < N && kin) ? We[(size_t)n * K + k0 + kk] : 0.f;
      }
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      const float a0 = As[kk][ty * 2], a1 = As[kk][ty * 2 + 1];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float b = Ws[kk][tx * 4 + c];
        acc[0][c] = fmaf(a0, b, acc[0][c]);
        acc[1][c] = fmaf(a1, b, acc[1][c]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int rr = 0; rr < 2; ++rr) {
    const int r = ty * 2 + rr;
    if (r >= rows) continue;
    if (act == MOE_ACT_GLU_LIMITED) {
#pragma unroll
      for (int c = 0; c < 4; c += 2) {
        const int n = n0 + tx * 4 + c;
        if (n + 1 < N) C[(size_t)(first + r) * c_stride + (n >> 1)] = moe_glu_limited(acc[rr][c], acc[rr][c + 1], limit, alpha, shift);
      }
      continue;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int n = n0 + tx * 4 + c;
      if (n < N) C[(size_t)(first + r) * c_stride + n] = moe_act(acc[rr][c], act);
    }
  }
}

SI_EXPORT int si_moe_gemm(const void* A, int dtype, long long a_stride, const int* a_rows, const void* W, void* C, int c_dtype,
                          long long c_stride, const int* offsets, int P, int E, int N, int K, int act, float limit, float alpha,
                          float shift, cudaStream_t stream) {
  if (P <= 0) return 0;
  if (E <= 0 || N <= 0 || K <= 0 || act < 0 || act > MOE_ACT_GLU_LIMITED) return -2;
  if (act == MOE_ACT_GLU_LIMITED && (N % 2 || !(limit > 0.f))) return -2;
  const int ny = (N + MOE_BN - 1) / MOE_BN;
  if (ny > 65535) return -2;
  if (dtype == SI_F32) {
    if (c_dtype != SI_F32) return -2;
    const dim3 grid((P + 31) / 32 + E, ny), block(256);
    si_launch(moe_gemm_f32_kernel, grid, block, 0, stream, (const float*)A, a_stride, a_rows, (const float*)W, (float*)C, c_stride,
              offsets, E, N, K, act, limit, alpha, shift);
    return si_last_error();
  }
  const int wide = (K % 8 == 0 && a_stride % 8 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0) ? 1 : 0;
  if ((P < 32LL * E || P < 128) && wide) {              // few rows an expert, or few at all
    const long long tiles = P < (P + 15) / 16 + E ? P : (P + 15) / 16 + E;       // no more can there be
    if (tiles > 65535) return -2;
    si_launch(moe_stream_kernel, dim3((N + 15) / 16, (unsigned)tiles), dim3(STREAM_WARPS * 32), 0, stream, (const bf16*)A, a_stride, a_rows,
              (const bf16*)W, C, c_stride, c_dtype == SI_F32 ? 1 : 0, offsets, E, N, K, act, limit, alpha, shift);
  } else if (P < 32LL * E && !wide) {
    // few rows an expert, and sizes or rows that are not in 16-byte pieces: tiles of 16 places (one row of two experts of 1,408 x 1,034:
    // 134 us, 176 in tiles of 64)
    si_launch(moe_gemm_bf16_kernel<16, 64, 64, 4>, dim3((P + 15) / 16 + E, ny), dim3(128), 0, stream, (const bf16*)A, a_stride, a_rows,
              (const bf16*)W, C, c_stride, c_dtype == SI_F32 ? 1 : 0, offsets, E, N, K, act, wide, limit, alpha, shift);
  } else {
    const dim3 grid((P + 63) / 64 + E, ny), block(128);
    si_launch(moe_gemm_bf16_kernel<64, 64, 32, 3>, grid, block, 0, stream, (const bf16*)A, a_stride, a_rows, (const bf16*)W, C, c_stride,
              c_dtype == SI_F32 ? 1 : 0, offsets, E, N, K, act, wide, limit, alpha, shift);
  }
  return si_last_error();
}

// The grouped product without a plan: P = rows x choices pairs, at most 32 of at most 16 rows; pair p of expert ids[p] reads row
// p / a_div of A and writes row p of C. Pairs whose id is not below E are left alone. With sW the shared matrix's product (see MoeShared) for
// the P / choices rows of sA runs in the same launch. bf16; returns -2 for what it does not take.
SI_EXPORT int si_moe_gemm_pairs(const void* A, long long a_stride, int a_div, const int* ids, const void* W, void* C, int c_dtype,
                                long long c_stride, int P, int choices, int E, int N, int K, int act, float limit, float alpha,
                                float shift, const void* sA, long long sa_stride, const void* sW, void* sC, long long sc_stride,
                                int sN, int sK, int s_form, const float* s_bias, float s_limit, float s_alpha, cudaStream_t stream) {
  if (P <= 0) return 0;
  if (E <= 0 || N <= 0 || K <= 0 || act < 0 || act > MOE_ACT_GLU_LIMITED || choices <= 0 || P % choices || P > 32 || P / choices > 16 || a_div <= 0) return -2;
  if (act == MOE_ACT_GLU_LIMITED && (N % 2 || !(limit > 0.f))) return -2;
  if (K % 8 || a_stride % 8 || ((uintptr_t)A & 15) || ((uintptr_t)W & 15)) return -2;
  MoeShared sh = {};
  long long tiles = (long long)((N + 15) / 16) * (P < E ? P : E);
  const int T = P / choices;
  if (sW) {
    if (sN <= 0 || sK <= 0 || sK % 8 || sa_stride % 8 || ((uintptr_t)sA & 15) || ((uintptr_t)sW & 15) || s_form < 0 || s_form > 3 || !sC) return -2;
    if (s_form >= 2 && sN % 16) return -2;
    sh.A = (const bf16*)sA; sh.a_stride = sa_stride; sh.W = (const bf16*)sW; sh.C = (bf16*)sC; sh.c_stride = sc_stride;
    sh.bias = s_bias; sh.rows = T; sh.N = sN; sh.K = sK; sh.form = s_form; sh.limit = s_limit; sh.alpha = s_alpha;
    tiles += (sN + 15) / 16;
  }
  const long long slots = 2LL * si_sm_count(), grid = tiles < slots ? tiles : slots;
  si_launch(T <= 8 ? moe_pairs_kernel<1> : moe_pairs_kernel<2>, dim3((unsigned)grid), dim3(STREAM_WARPS * 32), 0, stream,
            (const bf16*)A, a_stride, ids, a_div, (const bf16*)W, C, c_stride, c_dtype == SI_F32 ? 1 : 0, P, E, N, K, act, limit, alpha, shift,
            si_pdl_trigger_mode(grid, slots), sh);
  return si_last_error();
}

// ---- rows in the order of their places ------------------------------------------------------------------------------------
// out[p, :] = a[rows[p], :] for every place p (what the TMA-fed grouped product reads as one matrix); 16 bytes a thread
// and step where rows are so aligned.
template <typename T>
__global__ void __launch_bounds__(256) moe_gather_kernel(const T* __restrict__ a, long long a_stride, const int* __restrict__ rows,
    T* __restrict__ out, long long out_stride, int num_rows, int K, int wide) {
  pdl_prologue();
  const long long p = blockIdx.x;
  int r = rows[p];
  if (r < 0 || r >= num_rows) r = 0;
  const T* src = a + (size_t)r * a_stride;
  T* dst = out + p * out_stride;
  if (wide) {
    constexpr int PER = 16 / sizeof(T);
    for (int i = threadIdx.x; i < K / PER; i += blockDim.x) reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
  } else {
    for (int i = threadIdx.x; i < K; i += blockDim.x) dst[i] = src[i];
  }
}

SI_EXPORT int si_moe_gather(const void* a, int dtype, long long a_stride, const int* rows, void* out, long long out_stride,
                            int P, int num_rows, int K, cudaStream_t stream) {
  if (P <= 0) return 0;
  if (K <= 0 || num_rows <= 0) return -2;
  const int es = dtype == SI_BF16 ? 2 : 4, per = 16 / es;
  const int wide = (K % per == 0 && a_stride % per == 0 && out_stride % per == 0 && ((uintptr_t)a & 15) == 0 && ((uintptr_t)out & 15) == 0) ? 1 : 0;
  const dim3 grid(P), block(K / per >= 256 ? 256 : 128);
  if (dtype == SI_BF16)
    si_launch(moe_gather_kernel<bf16>, grid, block, 0, stream, (const bf16*)a, a_stride, rows, (bf16*)out, out_stride, num_rows, K, wide);
  else
    si_launch(moe_gather_kernel<float>, grid, block, 0, stream, (const float*)a, a_stride, rows, (float*)out, out_stride, num_rows, K, wide);
  return si_last_error();
}

// ---- combine --------------------------------------------------------------------------------------------------------------
// out[t, :] = sum_c wts[t, c] * Y[place_of[t, c], :] + gate[t] * shared[t, :]   (gate absent: 1; shared absent: none)
// Y fp32 or the compute dtype; shared and out in the compute dtype. Sums in fp32, the choices in their own order. No place_of: a
// pair is its own place.
template <typename TY, typename T>
__global__ void __launch_bounds__(256) moe_combine_kernel(const TY* __restrict__ Y, long long y_stride, const int* __restrict__ place_of,
    const float* __restrict__ wts, int top, const T* __restrict__ shared, long long shared_stride, const float* __restrict__ gate,
    int gate_stride, T* __restrict__ out, long long out_stride, int d, const int* __restrict__ ids, int real,
    const T* __restrict__ x, long long x_stride, int trigger) {
  if (trigger) pdl_trigger();
  pdl_wait();
  const long long t = blockIdx.x;
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < d; i += blockDim.x * gridDim.y) {
    float acc = 0.f;
    for (int c = 0; c < top; ++c) {
      const bool same = ids && ids[t * top + c] >= real;           // an identity expert: the row itself
      const float y = same ? to_f32<T>(x[t * x_stride + i]) : to_f32<TY>(Y[(size_t)(place_of ? place_of[t * top + c] : t * top + c) * y_stride + i]);
      acc = fmaf(wts[t * top + c], y, acc);
    }
    if (shared) acc = fmaf(gate ? gate[t * gate_stride] : 1.f, to_f32<T>(shared[t * shared_stride + i]), acc);
    out[t * out_stride + i] = from_f32<T>(acc);
  }
}

SI_EXPORT int si_moe_combine(const void* Y, int y_dtype, long long y_stride, const int* place_of, const float* wts, int top,
                             const void* shared, long long shared_stride, const float* gate, int gate_stride, void* out,
                             int dtype, long long out_stride, int rows, int d, const int* ids, int real, const void* x,
                             long long x_stride, cudaStream_t stream) {
  if (rows <= 0) return 0;
  if (top <= 0 || d <= 0 || (ids && !x)) return -2;
  const dim3 block(d >= 1024 ? 256 : 128);
  const dim3 grid(rows, si_row_shares(rows, d, block.x));
  const int trigger = si_pdl_trigger_small((long long)grid.x * grid.y);
  if (dtype == SI_BF16 && y_dtype == SI_F32)
    si_launch(moe_combine_kernel<float, bf16>, grid, block, 0, stream, (const float*)Y, y_stride, place_of, wts, top,
              (const bf16*)shared, shared_stride, gate, gate_stride, (bf16*)out, out_stride, d, ids, real, (const bf16*)x, x_stride, trigger);
  else if (dtype == SI_BF16 && y_dtype == SI_BF16)
    si_launch(moe_combine_kernel<bf16, bf16>, grid, block, 0, stream, (const bf16*)Y, y_stride, place_of, wts, top,
              (const bf16*)shared, shared_stride, gate, gate_stride, (bf16*)out, out_stride, d, ids, real, (const bf16*)x, x_stride, trigger);
  else if (dtype == SI_F32 && y_dtype == SI_F32)
    si_launch(moe_combine_kernel<float, float>, grid, block, 0, stream, (const float*)Y, y_stride, place_of, wts, top,
              (const float*)shared, shared_stride, gate, gate_stride, (float*)out, out_stride, d, ids, real, (const float*)x, x_stride, trigger);
  else
    return -2;
  return si_last_error();
}
