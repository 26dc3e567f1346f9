// Attention for prompt portions on the 5th-generation tensor cores (tcgen05), bf16, over the
// paged cache. One block handles one work item (a run of consecutive query tokens of a sequence)
// for one KV head as TWO query tiles of 128 rows each (row r of a tile = token r / G of the tile,
// head r % G; a tile holds floor(128 / G) tokens), against key tiles of 128. The two query tiles
// share every K and V tile and take turns: while the rows of one are in the softmax, the tensor
// cores work for the other.
//
//   warp 8 (producer)  looks up the pages of a key tile and issues its K and V boxes by TMA
//                      (128-byte swizzle) into one of two stages;
//   warp 9 (issuer)    per query tile: S = Q K^T with tcgen05.mma into tensor memory (Q, K K-major) and,
//                      once the probabilities stand in tensor memory, O += P V with P as the
//                      tensor-memory A operand and V the MN-major B operand, as it lies in the cache.
//                      Its order of issue, P V and the next S of tile 0, then of tile 1, keeps the two
//                      tiles in opposite phases: one in the softmax while the tensor cores serve the other;
//   warps 0-3 / 4-7    one thread per row of query tile 0 / 1: reads the row of S (tcgen05.ld), takes its
//                      maximum, computes exp2 of the scaled scores in fp32 against a base that is raised
//                      only when the maximum has grown by more than 2^8 (then the row of O in tensor
//                      memory is rescaled first), and writes the bf16 probabilities over the first
//                      columns of S (tcgen05.st); at the end it reads O and divides by the row sum.
//
// The tensor cores run one thread's instructions in the order of issue, which is what keeps this
// simple: S of the next key tile is issued behind P V of the current one, so it overwrites P only
// after P has been read, and when S is complete so is every earlier product into O.
//
// Keys and values narrower than a tile's columns (multiples of 8): the tensor maps end at their sizes, so the boxes' further
// columns arrive as zeros; the queries are padded likewise and results beyond the value size are not stored.
//
// Instances: key size in NK halves of 64 columns (1 to 3), value size in NV (1 or 2); values beyond NV halves go to further blocks
// (blockIdx.z), which make the scores again. With 192-wide keys the values have one stage, so that all fits shared memory. MODE
// says what a score gets beside its scale: nothing, the extended form (slopes by distance, a query temperature, an output gate), a
// bias by distance from a table, or a soft limit (see AttnExtras). All of it is fp32 arithmetic on the scores in registers, which
// costs issue slots of the softmax threads: they, and their exponentials, bound the kernel, not the tensor cores.
// Measured, a portion of 2,048 tokens in place of the mma.sync kernel: bias by distance (16 query, 4 key heads of 128) 285 -> 59 us, 192-wide
// latent keys (16 heads) 297 -> 49, a soft limit over 64-wide keys and 128-wide values (32 query, 8 key heads) 501 -> 63, four key heads a
// 512-wide value head 752 -> 99; 32 tokens behind 16,000 with the bias 1,333 -> 279. Keys of one item cut over blocks (2,043 tokens at the end of
// 16,128, 24 query and 8 key heads, where 200 blocks were 1.4 waves of SMs): 622 -> 518 us with the merge.
//
// The reference computes prompt attention row by row with its scalar split kernel
// (src/source/op/kernels/cuda/paged_kernels.cu:96-206). Conditions here: key sizes up to 192 and value sizes in multiples of 8
// (the extended instance: 64 or 128, both alike), page size a power of two from 8 to 64 (or keys of one sequence in neighbouring
// rows of a matrix, `dense`), G <= 128; other layouts use the mma.sync kernel. Every mbarrier wait
// is bounded; when one runs out the block sets SI_WAIT_LIMIT and leaves without storing.
#include "attention_common.cuh"
#include "tma_common.cuh"
#include <algorithm>
#include <functional>
#include <new>
#include <vector>
#include <limits.h>

// Packed fp32 arithmetic of sm_100 in the softmax (two scores an instruction) and three-input maxima.
#ifndef SI_ATTN_PACKED
#define SI_ATTN_PACKED 1
#endif
__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
  unsigned long long v;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void unpack_f32x2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;\n" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long fma_f32x2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long add_f32x2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

template <int NROWS>
__device__ __forceinline__ bf16* half_ptr(bf16* base, int row, int chunk) {
  return base + (size_t)(chunk >> 3) * (NROWS * 64) + (size_t)row * 64 + (((chunk & 7) ^ (row & 7)) << 3);
}

// What a MODE adds to a score and to the result, all fp32 arithmetic in the softmax threads:
//   EXT   score(i, j) = scale * t(i) * q.k - slope[h] * (i - j),  t(i) = 1 + qt_coef * ln(floor((i + 1) / qt_every) + 1)  (qt_every 0: t = 1)
//         result(i, h, d) *= sigmoid(gate[i, h * hs + d])   (gate null: none)
//   BIAS  score(i, j) = scale * q.k + bias[min(i - j, nd - 1), h]
//   CAP   score(i, j) = cap * tanh(scale * q.k / cap)
//   GEN   score(i, j) = scale * q.k
// BIAS, CAP and GEN are the general form: key heads that share values, fp32 results, values in several blocks, dense rows. What its
// tiles hold behind an item's last key (a page's earlier owner's rows, another sequence's) is zeroed before it meets the probabilities:
// those are zeros there, but zero times a number that is not finite is none.
// CUT is PLAIN with items whose keys are cut over blocks (AttnExtras::shares). What only some forms have is decided when their instance is
// compiled: 2,048 tokens of 32 query and 8 key heads of 128 took 51.7 us where the plain form asked for shares, dense rows and the rest as
// it ran, and 50.0 so.
enum { MODE_PLAIN = 0, MODE_CUT = 1, MODE_EXT = 2, MODE_BIAS = 3, MODE_CAP = 4, MODE_GEN = 5 };
struct AttnExtras {
  const float* slopes;                           // fp32 [H] or nullptr
  float qt_coef; int qt_every;
  const bf16* gate; long long gate_stride;       // rows 16-byte aligned
  const float* bias; int nd;                     // fp32 [nd, H]
  float cap_log2, scale_over_cap;                // cap * log2(e), scale / cap
  int v_share;                                   // key heads that read one value head
  int out_f32;                                   // p.out is fp32
  int dense;                                     // keys and values [rows, KV * size]: a sequence's rows lie behind its table's first entry
  // MODE_CUT, one block of values: an item's keys may be cut into shares, a block each. Entry (item, share, shares of the item, slot of
  // its first share's partial results); a whole item has one share. Shares leave O, maximum and sum per row; a second kernel merges.
  const int4* shares;
  float* part_o;                                 // [slot][KV][256 rows][NV * 64]
  float* part_ml;                                // [slot][KV][256 rows][2]
};

// Floats of a bias window in shared memory: the distances that a query tile's rows have to a key tile's keys, per head. The
// pitch puts the lanes of a warp (G heads of neighbouring tokens) into different banks.
__host__ __device__ __forceinline__ int bias_pitch(int G) { return (128 / G + 128 + 31) / 32 * 32 + (G < 32 ? 32 / G : 0); }

// tanh for |z| <= 1/2: z + z^3 q(z^2), q a degree-3 polynomial fitted at Chebyshev points; absolute error 6e-8 in fp32 (the
// quotient form below: 1.2e-7). Two at a time.
__device__ __forceinline__ unsigned long long mul_f32x2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long tanh_small_f32x2(unsigned long long z) {
  const unsigned long long c3 = pack_f32x2(0.017993388697504997f, 0.017993388697504997f), c2 = pack_f32x2(-0.053373366594314575f, -0.053373366594314575f),
                           c1 = pack_f32x2(0.1333010345697403f, 0.1333010345697403f), c0 = pack_f32x2(-0.33333292603492737f, -0.33333292603492737f);
  const unsigned long long u = mul_f32x2(z, z);
  const unsigned long long q = fma_f32x2(fma_f32x2(fma_f32x2(c3, u, c2), u, c1), u, c0);
  return fma_f32x2(z, mul_f32x2(u, q), z);
}

template <int NK, int NV, int MODE>
__global__ void __launch_bounds__(320)
attn_portion_tc05_kernel(const AttnParams p, const __grid_constant__ CUtensorMap kmap,
                         const __grid_constant__ CUtensorMap vmap, int log2_page, const AttnExtras x) {
  constexpr bool CUT = MODE == MODE_CUT, EXT = MODE == MODE_EXT, GENERAL = MODE >= MODE_BIAS;
  const bool dense = GENERAL && x.dense;
  constexpr int BM = 128, BN = 128, DK = NK * 64, DV = NV * 64, STAGES = 2, VST = NK > 2 ? 1 : 2;
  constexpr int KTILE = NK * BN * 64, VTILE = NV * BN * 64;      // elements of a tile: halves of [128][64]
  constexpr int TM_S = 0, TM_O = 2 * BN;             // tensor-memory columns: S of tile q at TM_S + q*BN, O at TM_O + q*DV
  constexpr int TM_COLS = 512;
  extern __shared__ unsigned char smem_dyn[];
  __shared__ __align__(8) uint64_t k_full[STAGES], k_empty[STAGES], v_full[VST], v_empty[VST];
  __shared__ __align__(8) uint64_t s_full[2], p_full[2], o_full[2];   // per query tile
  __shared__ unsigned tmem_slot;
  __shared__ int s_abort;
  unsigned char* smem_raw = reinterpret_cast<unsigned char*>(((uintptr_t)smem_dyn + 1023) & ~(uintptr_t)1023);
  bf16* Qs = reinterpret_cast<bf16*>(smem_raw);     // [2 tiles][NK][128][64]
  bf16* Ks = Qs + 2 * BM * DK;                       // [STAGES][KTILE]
  bf16* Vs = Ks + STAGES * KTILE;                    // [VST][VTILE]
  float* Bs = reinterpret_cast<float*>(Vs + VST * VTILE);        // BIAS: [2 tiles][2 buffers][G][pitch]

  // Items of a prompt come in order of position, so the last ones have the most keys: start with those,
  // for all KV heads alike (blocks are handed out with x running fastest, and x is the KV head).
  // (With shares the entries come longest first.)
  const int4 share = CUT ? x.shares[blockIdx.y] : make_int4(gridDim.y - 1 - blockIdx.y, 0, 1, 0);
  const AttnItem item = p.items[share.x];
  if (item.ntok <= 0) return;
  const int g = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (item.seq < 0 || item.seq >= p.num_seqs) {
    if (threadIdx.x == 0) set_status(p.status, SI_BAD_SEQ);
    return;
  }
  const int* table = p.block_table + (size_t)item.seq * p.table_width;
  const int tile_tokens = BM / p.G;                  // tokens of one query tile
  const bool two = item.ntok > tile_tokens;          // the second query tile has rows
  int kv_end = item.pos0 + item.ntok;
  const int kv_lo = first_visible_key(item.pos0, p.window, p.chunk);
  int kv_begin = kv_lo / BN * BN;
  int ntiles = (kv_end - kv_begin + BN - 1) / BN;
  if (CUT && share.z > 1) {           // this share's tiles
    const int first = (int)((long long)ntiles * share.y / share.z), last = (int)((long long)ntiles * (share.y + 1) / share.z);
    kv_begin += first * BN;
    ntiles = last - first;
    kv_end = min(kv_end, kv_begin + ntiles * BN);
  }
  const int page_rows = 1 << log2_page;              // dense: rows of a box
  const int pages_per_tile = BN >> log2_page;
  const int v0 = GENERAL ? blockIdx.z * DV : 0;                    // first value column of this block

  pdl_trigger();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1);
      if (s < VST) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      mbar_init(&s_full[q], 1);
      mbar_init(&p_full[q], 4);                      // one arrival per warp of the tile's rows
      mbar_init(&o_full[q], 1);
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 9) tmem_alloc(&tmem_slot, TM_COLS);
  // rows that no copy fills must hold finite numbers (they meet zero probabilities): those behind the
  // last key in the last tile, and pages wholly before the window in the first
  // (dense tiles are fetched whole: what lies behind a sequence is another's rows, or zeros behind the last)
  auto clear_tile = [&](int t) {
    uint4* kz = reinterpret_cast<uint4*>(Ks + (size_t)(t % STAGES) * KTILE);
    uint4* vz = reinterpret_cast<uint4*>(Vs + (size_t)(t % VST) * VTILE);
    for (int i = threadIdx.x; i < KTILE / 8; i += blockDim.x) kz[i] = make_uint4(0, 0, 0, 0);
    for (int i = threadIdx.x; i < VTILE / 8; i += blockDim.x) vz[i] = make_uint4(0, 0, 0, 0);
  };
  if (!dense && (kv_end - kv_begin) % BN != 0) clear_tile(ntiles - 1);
  if (!dense && kv_begin + page_rows <= kv_lo) clear_tile(0);
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  tc05_fence_before_sync();
  __syncthreads();                                   // barriers, tensor memory and the zeroed rows stand
  // launched as a programmatic dependent, all of the above ran while the kernel before this one (which wrote the
  // queries and the newest keys and values) was ending; the items and the block table were copied in earlier
  pdl_wait();
  tc05_fence_after_sync();
  const unsigned tmem = tmem_slot;
  if (warp != 8) {
    // Query rows, while the producer already fetches the first keys: row r of tile q is token
    // q * tile_tokens + r / G, head g*G + r % G. All loads of a thread are issued before its stores.
    constexpr int NT = 288, PER = (2 * BM * (DK / 8) + NT - 1) / NT;
    const int tid = warp == 9 ? 256 + lane : threadIdx.x;
    const int rows = two ? 2 * BM : BM;              // the second tile is not read when it has no token
    uint4 v[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int id = tid + i * NT;
      const int row = id / (DK / 8), c = id % (DK / 8);
      const int q = row / BM, r = row % BM;
      const int tl = r / p.G, hh = r - tl * p.G;
      const int tok = q * tile_tokens + tl;
      v[i] = make_uint4(0, 0, 0, 0);
      if (row < rows && tl < tile_tokens && tok < item.ntok && c * 8 < p.hs)
        v[i] = *reinterpret_cast<const uint4*>(p.q + (size_t)(item.row0 + tok) * p.q_stride + (size_t)(g * p.G + hh) * p.hs + c * 8);
    }
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int id = tid + i * NT;
      const int row = id / (DK / 8), c = id % (DK / 8);
      if (row < rows) *reinterpret_cast<uint4*>(half_ptr<BM>(Qs + (size_t)(row / BM) * BM * DK, row % BM, c)) = v[i];
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    asm volatile("bar.sync 1, 288;\n" ::: "memory");   // warps 0-7 and 9
  }

  if (warp == 8) {
    // ---- producer: box b = (page, half, K or V) of each tile, boxes spread over the lanes. K and V
    // have barriers of their own: a K stage is free as soon as both S have been computed from it, long
    // before the V stage of the same tile, so the next keys arrive under the softmax.
    const int gv = GENERAL ? g / x.v_share : g, KVv = GENERAL ? p.KV / x.v_share : p.KV;
    const int first_row = dense ? table[0] : 0;    // of the sequence's rows in the matrices
    for (int t = 0; t < ntiles; ++t) {
      const int j = kv_begin + t * BN;
      int page = -1;                                 // lane l: the page of the tile's keys from l * page_rows on
      // pages past the last key, or wholly before the window, are not fetched
      if (!dense && lane < pages_per_tile && j + lane * page_rows < kv_end && j + (lane + 1) * page_rows > kv_lo) {
        const int slot = (j >> log2_page) + lane;
        page = slot < p.table_width ? table[slot] : -1;
        if (page < 0 || page >= p.num_pages) { set_status(p.status, SI_BAD_PAGE); page = -1; }
      }
      const int pages = dense ? pages_per_tile : __popc(__ballot_sync(0xffffffffu, page >= 0));
      auto fetch = [&](bool keys) {
        const int nh = keys ? NK : NV, st = keys ? STAGES : VST, stage = t % st;
        uint64_t* full = keys ? &k_full[stage] : &v_full[stage];
        uint64_t* empty = keys ? &k_empty[stage] : &v_empty[stage];
        bf16* tile = keys ? Ks + (size_t)stage * KTILE : Vs + (size_t)stage * VTILE;
        if (t >= st && !mbar_wait_warp(empty, (unsigned)(((t / st) - 1) & 1))) return false;
        if (lane == 0) mbar_expect_tx(full, (unsigned)(pages * nh * page_rows * 128));
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int b = lane + 32 * i, pg = b / nh, h = b % nh;
          const int of = __shfl_sync(0xffffffffu, page, pg & 31);
          if (pg >= pages_per_tile || (!dense && of < 0)) continue;
          bf16* to = tile + (size_t)h * (BN * 64) + (size_t)(pg * page_rows) * 64;
          const int col = (keys ? 0 : v0) + h * 64;
          if (dense) tma_load_3d(to, keys ? &kmap : &vmap, full, col, keys ? g : gv, first_row + j + pg * page_rows);
          else tma_load_2d(to, keys ? &kmap : &vmap, full, col, (of * (keys ? p.KV : KVv) + (keys ? g : gv)) << log2_page);
        }
        return true;
      };
      if (!fetch(true) || !fetch(false)) {
        if (lane == 0) { set_status(p.status, SI_WAIT_LIMIT); s_abort = 1; }
        break;
      }
    }
  } else if (warp == 9) {
    // ---- issuer: S_0(0) S_1(0) | P V_0(0) S_0(1) | P V_1(0) S_1(1) | P V_0(1) S_0(2) | ...
    // The whole warp runs this code and one elected lane issues: what an instruction needs (descriptors,
    // addresses) is then uniform over the warp. The descriptors are made once and only their address
    // fields (units of 16 bytes) advance. An instruction is accepted only as fast as the tensor cores
    // run, so whatever else this warp does between two of them leaves the tensor cores idle.
    constexpr unsigned idesc_s = umma_idesc_bf16(BM, BN, false);
    constexpr unsigned idesc_o = umma_idesc_bf16(BM, DV, true);
    constexpr unsigned U_KTILE = KTILE * 2 / 16, U_VTILE = VTILE * 2 / 16, U_QTILE = BM * DK * 2 / 16, U_HALF = BN * 64 * 2 / 16;
    const int nq = two ? 2 : 1;
    const unsigned long long qd0 = umma_desc_sw128(Qs, 16, 1024);
    const unsigned long long kd0 = umma_desc_sw128(Ks, 16, 1024);
    const unsigned long long vd0 = umma_desc_sw128(Vs, BN * 128, 1024);
    auto issue_s = [&](int q, int t) {  // S_q[128, 128] = Q_q[128, DK] K_t[128 keys, DK]^T: 4 steps per 64-column half
      const unsigned long long qd = qd0 + (unsigned)q * U_QTILE;
      const unsigned long long kd = kd0 + (unsigned)(t % STAGES) * U_KTILE;
      const unsigned sd = tmem + TM_S + q * BN;
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < DK / 16; ++kk)
          tc05_mma_bf16(sd, qd + ((kk >> 2) * U_HALF + 2 * (kk & 3)), kd + ((kk >> 2) * U_HALF + 2 * (kk & 3)), idesc_s, kk != 0 ? 1u : 0u);
        tc05_commit(&s_full[q]);
        if (q == nq - 1) tc05_commit(&k_empty[t % STAGES]);      // the keys of this tile are not needed again
      }
      __syncwarp();
    };
    bool ok = ntiles > 0 && mbar_wait_warp(&k_full[0], 0);
    if (ok) {
      tc05_fence_after_sync();
      for (int q = 0; q < nq; ++q) issue_s(q, 0);
    }
    for (int t = 0; t < ntiles && ok; ++t) {
      const int stage = t % VST;
      const bool more = t + 1 < ntiles;
      ok = mbar_wait_warp(&v_full[stage], (unsigned)((t / VST) & 1));
      if (GENERAL && ok && !more && (kv_end - kv_begin) % BN != 0) {      // a row is 128 bytes of each half, whatever the swizzle
        const int first = (kv_end - kv_begin) % BN;
        for (int i = lane; i < (BN - first) * NV * 8; i += 32) {
          const int half = i / ((BN - first) * 8), at = i - half * (BN - first) * 8;
          reinterpret_cast<uint4*>(Vs + (size_t)stage * VTILE + (size_t)half * (BN * 64) + (size_t)first * 64)[at] = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        __syncwarp();
      }
      for (int q = 0; q < nq && ok; ++q) {
        ok = mbar_wait_warp(&p_full[q], (unsigned)(t & 1));
        if (!ok) break;
        tc05_fence_after_sync();
        // O_q[128, DV] (+)= P_q[128, 128 keys] V_t[128 keys, DV]: 8 steps of 16 keys; P lies packed in the first
        // 64 columns of S_q, V rows are keys (MN-major B)
        const unsigned long long vd = vd0 + (unsigned)stage * U_VTILE;
        const unsigned sd = tmem + TM_S + q * BN, od = tmem + TM_O + q * DV;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < BN / 16; ++kk)
            tc05_mma_bf16_tmem_a(od, sd + 8 * kk, vd + 128 * kk, idesc_o, (t | kk) != 0 ? 1u : 0u);
          if (!more) tc05_commit(&o_full[q]);
          if (q == nq - 1) tc05_commit(&v_empty[stage]);
        }
        __syncwarp();
        if (more) {                        // behind P V in the order of issue: S overwrites P only after it was read
          if (q == 0) ok = mbar_wait_warp(&k_full[(t + 1) % STAGES], (unsigned)(((t + 1) / STAGES) & 1));
          if (!ok) break;
          tc05_fence_after_sync();
          issue_s(q, t + 1);
        }
      }
    }
    if (!ok && ntiles > 0 && lane == 0) { set_status(p.status, SI_WAIT_LIMIT); s_abort = 1; }
  } else if (warp < 4 || two) {
    // ---- one thread per row of query tile q
    const int q = warp >> 2;
    const int r = threadIdx.x & (BM - 1);            // tile row = tensor-memory lane
    const int tl = r / p.G, hh = r - tl * p.G;
    const int tok = q * tile_tokens + tl;
    const bool valid = tl < tile_tokens && tok < item.ntok;
    const int pos = valid ? item.pos0 + tok : -1;
    int lo = p.window > 0 ? pos - p.window + 1 : INT_MIN;           // visible keys: lo <= j <= pos
    if (p.chunk > 0) lo = max(lo, pos / p.chunk * p.chunk);
    const unsigned lane_base = (unsigned)((warp & 3) * 32) << 16;
    const unsigned ts = tmem + lane_base + TM_S + q * BN, to = tmem + lane_base + TM_O + q * DV;
    float m = -INFINITY, l = 0.f;                    // base of the exponentials (log2 domain), the row's sum
    bool alive = true;
    // EXT: the row's own scale (its query temperature) and its head's slope, base 2; the scores then carry scale and
    // penalty before the maximum is taken, and `sc` below is one
    float row_scale = p.scale_log2, sl2 = 0.f;
    if (EXT) {
      if (x.qt_every > 0 && pos >= 0) row_scale *= 1.f + x.qt_coef * logf((float)((pos + 1) / x.qt_every + 1));
      if (x.slopes) sl2 = x.slopes[g * p.G + (hh < p.G ? hh : 0)] * 1.4426950408889634f;
    }
    const float sc = EXT || MODE == MODE_BIAS || MODE == MODE_CAP ? 1.f : p.scale_log2;
    // BIAS: entry k of a head's window is the distance (last position of the query tile) - j0 - k; the tile's four warps
    // copy the next key tile's window while this one's is read
    const int pitch = MODE == MODE_BIAS ? bias_pitch(p.G) : 0, span = tile_tokens + BN - 1;
    const int last_pos = item.pos0 + (q + 1) * tile_tokens - 1;
    float* const window = Bs + (size_t)q * 2 * p.G * pitch;
    auto stage_bias = [&](int t) {
      float* dst = window + (size_t)(t & 1) * p.G * pitch;
      const int d0 = last_pos - (kv_begin + t * BN);
      for (int i = r; i < span * p.G; i += BM) {
        const int k = i / p.G, h = i - k * p.G;
        const int d = min(max(d0 - k, 0), x.nd - 1);
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_u32(dst + h * pitch + k)), "l"(x.bias + (size_t)d * p.H + g * p.G + h));
      }
      asm volatile("cp.async.commit_group;\n" ::);
    };
    if (MODE == MODE_BIAS && ntiles > 0) stage_bias(0);
    for (int t = 0; t < ntiles; ++t) {
      const int j0 = kv_begin + t * BN;
      if (MODE == MODE_BIAS) {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        asm volatile("bar.sync %0, 128;\n" ::"r"(2 + q) : "memory");      // this window stands; nobody reads the one before any more
        if (t + 1 < ntiles) stage_bias(t + 1);
      }
      alive = alive && mbar_wait_warp(&s_full[q], (unsigned)(t & 1));
      if (!alive) {
        if (MODE == MODE_BIAS) continue;             // the tile's other warps still count on this one at their barrier
        break;
      }
      tc05_fence_after_sync();
      float s[BN];
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) tmem_ld_32x32_issue(ts + 32 * c, s + 32 * c);
      tmem_ld_wait();
      if (MODE == MODE_BIAS) {
        const float* b = window + (size_t)(t & 1) * p.G * pitch + (hh < p.G ? hh : 0) * pitch + (tile_tokens - 1 - min(tl, tile_tokens - 1));
#pragma unroll
        for (int i = 0; i < BN; ++i) s[i] = fmaf(b[i], LOG2E, s[i] * p.scale_log2);
      }
      if (MODE == MODE_CAP) {
        float top = 0.f;
#pragma unroll
        for (int i = 0; i < BN; i += 2) top = max3(top, fabsf(s[i]), fabsf(s[i + 1]));
        if (__any_sync(0xffffffffu, !(top * x.scale_over_cap <= 0.5f))) {
          // tanh(y) = 1 - 2 / (exp(2 y) + 1): absolute error of some 1e-7, which is what counts for a score
          const float c2 = 2.f * LOG2E * x.scale_over_cap;
#pragma unroll
          for (int i = 0; i < BN; ++i) s[i] = x.cap_log2 * (1.f - __fdividef(2.f, exp2f(s[i] * c2) + 1.f));
        } else {
          const unsigned long long c2 = pack_f32x2(x.scale_over_cap, x.scale_over_cap), cap2 = pack_f32x2(x.cap_log2, x.cap_log2);
#pragma unroll
          for (int i = 0; i < BN; i += 2)
            unpack_f32x2(mul_f32x2(tanh_small_f32x2(mul_f32x2(pack_f32x2(s[i], s[i + 1]), c2)), cap2), s[i], s[i + 1]);
        }
      }
      // most tiles lie wholly inside every row's visible range: then nothing is masked
      if (__any_sync(0xffffffffu, !(j0 >= lo && j0 + BN - 1 <= pos))) {
#pragma unroll
        for (int i = 0; i < BN; ++i) {
          const int j = j0 + i;
          if (j < lo || j > pos) s[i] = -INFINITY;
        }
      }
      if (EXT) {                                           // masked scores stay -inf
        const float c0 = sl2 * (float)(j0 - pos);
#pragma unroll
        for (int i = 0; i < BN; ++i) s[i] = fmaf(s[i], row_scale, fmaf(sl2, (float)i, c0));
      }
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#if SI_ATTN_PACKED
#pragma unroll
      for (int i = 0; i < BN; i += 8) {                    // three-input maxima: half the instructions
        m4[0] = max3(m4[0], s[i], s[i + 1]); m4[1] = max3(m4[1], s[i + 2], s[i + 3]);
        m4[2] = max3(m4[2], s[i + 4], s[i + 5]); m4[3] = max3(m4[3], s[i + 6], s[i + 7]);
      }
#else
#pragma unroll
      for (int i = 0; i < BN; i += 4) {
        m4[0] = fmaxf(m4[0], s[i]); m4[1] = fmaxf(m4[1], s[i + 1]);
        m4[2] = fmaxf(m4[2], s[i + 2]); m4[3] = fmaxf(m4[3], s[i + 3]);
      }
#endif
      // the scale is positive, so the maximum may be taken before it
      const float mx = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])) * sc;
      // raise the base only when the maximum has outgrown it by 2^8; then O and l are rescaled. S being
      // complete, so is every earlier product into O.
      float factor = 1.f;
      const bool raise = mx > m + 8.f;
      if (raise) { factor = fast_exp2(m - mx); m = mx; }   // exp2(-inf) = 0 on the first keys
      if (t > 0 && __any_sync(0xffffffffu, raise)) {
#pragma unroll 1
        for (int c = 0; c < DV / 32; ++c) {
          float v[32];
          tmem_ld_32x32(to + c * 32, v);
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] *= factor;
          tmem_st_32x32(to + c * 32, v);
        }
      }
      const float base = m == -INFINITY ? 0.f : m;
#if SI_ATTN_PACKED
      // scale, subtraction of the base and the row's sum two scores at a time (fma.rn.f32x2, add.rn.f32x2: the
      // same roundings as the single instructions, half as many of them)
      const unsigned long long sc2 = pack_f32x2(sc, sc), nb2 = pack_f32x2(-base, -base);
      unsigned long long sum2[2] = {0ull, 0ull};
#pragma unroll
      for (int b = 0; b < BN / 64; ++b) {
        unsigned pk[32];
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
          float e[4];
#pragma unroll
          for (int w = 0; w < 2; ++w) {
            float x0, x1;
            unpack_f32x2(fma_f32x2(pack_f32x2(s[64 * b + i + 2 * w], s[64 * b + i + 2 * w + 1]), sc2, nb2), x0, x1);
            e[2 * w] = fast_exp2(x0);                      // exp2(-inf) = 0 for masked keys
            e[2 * w + 1] = fast_exp2(x1);
            sum2[w] = add_f32x2(sum2[w], pack_f32x2(e[2 * w], e[2 * w + 1]));
          }
          pk[i / 2] = pack_bf16(e[0], e[1]);
          pk[i / 2 + 1] = pack_bf16(e[2], e[3]);
        }
        // the probabilities of keys 64b .. 64b+63 go over columns 32b .. 32b+31 of S, which is in registers
        tmem_st_32x32_issue(ts + 32 * b, pk);
      }
      float s4[4];
      unpack_f32x2(sum2[0], s4[0], s4[1]);
      unpack_f32x2(sum2[1], s4[2], s4[3]);
      l = l * factor + ((s4[0] + s4[1]) + (s4[2] + s4[3]));
#else
      float s4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int b = 0; b < BN / 64; ++b) {
        unsigned pk[32];
#pragma unroll
        for (int i = 0; i < 64; i += 4) {
#pragma unroll
          for (int w = 0; w < 4; ++w) {
            const float e = fast_exp2(fmaf(s[64 * b + i + w], sc, -base));    // exp2(-inf) = 0 for masked keys
            s[64 * b + i + w] = e;
            s4[w] += e;
          }
          pk[i / 2] = pack_bf16(s[64 * b + i], s[64 * b + i + 1]);
          pk[i / 2 + 1] = pack_bf16(s[64 * b + i + 2], s[64 * b + i + 3]);
        }
        // the probabilities of keys 64b .. 64b+63 go over columns 32b .. 32b+31 of S, which is in registers
        tmem_st_32x32_issue(ts + 32 * b, pk);
      }
      l = l * factor + ((s4[0] + s4[1]) + (s4[2] + s4[3]));
#endif
      tmem_st_wait();
      tc05_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_full[q]);
    }
    if (alive && ntiles > 0) alive = mbar_wait_warp(&o_full[q], 0);
    if (!alive && lane == 0) { set_status(p.status, SI_WAIT_LIMIT); s_abort = 1; }
    if (CUT && share.z > 1) {                 // a share's results as they are
      const size_t row = (((size_t)(share.w + share.y) * p.KV + g) * 2 + q) * BM + r;
      if (alive && valid) {
        tc05_fence_after_sync();
        x.part_ml[row * 2] = m;
        x.part_ml[row * 2 + 1] = l;
      }
      if (alive)                                             // (the loads are the whole warp's)
#pragma unroll 1
        for (int c = 0; c < DV / 32; ++c) {
          float v[32];
          tc05_fence_after_sync();
          tmem_ld_32x32(to + c * 32, v);
          if (!valid) continue;
          float4* dst = reinterpret_cast<float4*>(x.part_o + row * DV + c * 32);
#pragma unroll
          for (int i = 0; i < 8; ++i) dst[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        }
      alive = false;                                         // nothing is stored here
    }
    if (alive) {
      tc05_fence_after_sync();
      float inv = l > 0.f ? 1.f / l : 0.f;
      if (p.sink) {                                          // exp(sink) joins the denominator once
        const float s2 = p.sink[g * p.G + (hh < p.G ? hh : 0)] * LOG2E, M = fmaxf(m, s2), f = fast_exp2(m - M);
        inv = f / (l * f + fast_exp2(s2 - M));
      }
      const size_t at = (size_t)(item.row0 + tok) * p.out_stride + (size_t)(g * p.G + hh) * p.vs + v0;
      bf16* dst = p.out + at;
#pragma unroll
      for (int c = 0; c < DV / 64; ++c) {
        float v[64];
        tmem_ld_32x32_issue(to + c * 64, v);
        tmem_ld_32x32_issue(to + c * 64 + 32, v + 32);
        tmem_ld_wait();
        if (valid) {
          if (EXT && x.gate) {                               // the output gate: sigmoid of this row's and head's gate sums
            const bf16* gr = x.gate + (size_t)(item.row0 + tok) * x.gate_stride + (size_t)(g * p.G + hh) * p.hs + c * 64;
#pragma unroll
            for (int q8 = 0; q8 < 8; ++q8) {
              const uint4 gz = *reinterpret_cast<const uint4*>(gr + q8 * 8);
              const __nv_bfloat162* g2 = reinterpret_cast<const __nv_bfloat162*>(&gz);
#pragma unroll
              for (int e2 = 0; e2 < 4; ++e2) {
                const float2 z = __bfloat1622float2(g2[e2]);
                v[8 * q8 + 2 * e2] *= 1.f / (1.f + __expf(-z.x));
                v[8 * q8 + 2 * e2 + 1] *= 1.f / (1.f + __expf(-z.y));
              }
            }
          }
          if (GENERAL && x.out_f32) {
            float* f = reinterpret_cast<float*>(p.out) + at;
#pragma unroll
            for (int q8 = 0; q8 < 16; ++q8)
              if (v0 + c * 64 + q8 * 4 < p.vs)
                *reinterpret_cast<float4*>(f + c * 64 + q8 * 4) = make_float4(v[4 * q8] * inv, v[4 * q8 + 1] * inv, v[4 * q8 + 2] * inv, v[4 * q8 + 3] * inv);
            continue;
          }
#pragma unroll
          for (int q8 = 0; q8 < 8; ++q8) {
            uint4 raw;
            raw.x = pack_bf16(v[8 * q8] * inv, v[8 * q8 + 1] * inv);
            raw.y = pack_bf16(v[8 * q8 + 2] * inv, v[8 * q8 + 3] * inv);
            raw.z = pack_bf16(v[8 * q8 + 4] * inv, v[8 * q8 + 5] * inv);
            raw.w = pack_bf16(v[8 * q8 + 6] * inv, v[8 * q8 + 7] * inv);
            if (v0 + c * 64 + q8 * 8 < p.vs) *reinterpret_cast<uint4*>(dst + c * 64 + q8 * 8) = raw;
          }
        }
      }
    }
  }
  tc05_fence_before_sync();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem, TM_COLS);
}

// Merge of the items whose keys were cut: entry (item, shares, slot of the first, -). A warp a row: the shares weighed by their maxima,
// the sink in the denominator once.
template <int NV>
__global__ void __launch_bounds__(256) attn_portion_merge_kernel(const AttnParams p, const int4* __restrict__ cut, const float* __restrict__ part_o,
                                                                 const float* __restrict__ part_ml) {
  constexpr int DV = NV * 64, PER = DV / 32;
  pdl_prologue();
  const int4 e = cut[blockIdx.y];
  const AttnItem item = p.items[e.x];
  const int g = blockIdx.x, row = blockIdx.z * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int tile_tokens = 128 / p.G, q = row >> 7, r = row & 127, tl = r / p.G, hh = r - tl * p.G, tok = q * tile_tokens + tl;
  if (tl >= tile_tokens || tok >= item.ntok) return;
  const size_t first = ((size_t)e.z * p.KV + g) * 256 + row, step = (size_t)p.KV * 256;
  const float m_own = lane < e.y ? part_ml[(first + lane * step) * 2] : -INFINITY, l_own = lane < e.y ? part_ml[(first + lane * step) * 2 + 1] : 0.f;
  const int head = g * p.G + hh;
  const float sk = p.sink ? p.sink[head] * LOG2E : -INFINITY;
  const float M = fmaxf(warp_max(m_own), sk);
  const float w_own = m_own == -INFINITY ? 0.f : fast_exp2(m_own - M);
  const float L = warp_sum(l_own * w_own) + (p.sink ? fast_exp2(sk - M) : 0.f);
  float acc[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) acc[i] = 0.f;
  for (int s = 0; s < e.y; ++s) {
    const float w = __shfl_sync(0xffffffffu, w_own, s);
    const float* src = part_o + (first + s * step) * DV + lane * PER;
#pragma unroll
    for (int i = 0; i < PER; i += 2) {
      const float2 v = *reinterpret_cast<const float2*>(src + i);
      acc[i] = fmaf(v.x, w, acc[i]); acc[i + 1] = fmaf(v.y, w, acc[i + 1]);
    }
  }
  const float inv = L > 0.f ? 1.f / L : 0.f;
  bf16* dst = p.out + (size_t)(item.row0 + tok) * p.out_stride + (size_t)head * p.vs;
#pragma unroll
  for (int i = 0; i < PER; i += 2)
    if (lane * PER + i < p.vs) *reinterpret_cast<__nv_bfloat162*>(dst + lane * PER + i) = __floats2bfloat162_rn(acc[i] * inv, acc[i + 1] * inv);
}

// ---- host side --------------------------------------------------------------------------------
// 1 when this kernel takes the layout.
SI_EXPORT int si_attn_portion_tc05_ok(int H, int KV, int hs, int vs, int page_size) {
  if (KV <= 0 || H % KV || H / KV > 128) return 0;
  if (hs <= 0 || vs <= 0 || hs > 128 || vs > 128 || hs % 8 || vs % 8) return 0;
  if (page_size != 8 && page_size != 16 && page_size != 32 && page_size != 64) return 0;
  return si_encode_fn() != nullptr;
}

// Tokens of one item: two query tiles of floor(128 / G) each.
SI_EXPORT int si_attn_portion_tc05_tokens(int H, int KV) { return 2 * (128 / (H / KV)); }

// Bytes of shared memory of a block: Q of both query tiles, the stages of K and of V, the biases. The block takes all of tensor
// memory, so a second block on the same SM could only wait for it: ask for more than half of the shared memory.
#define PORTION_SMEM_LIMIT (227 * 1024 - 256)            // beside the barriers
static size_t portion_smem(int nk, int nv, bool bias, int G) {
  size_t smem = (size_t)(2 * 128 * nk * 64 + 2 * nk * 128 * 64 + (nk > 2 ? 1 : 2) * nv * 128 * 64) * sizeof(bf16) + 1024;
  if (bias) smem += (size_t)4 * G * bias_pitch(G) * sizeof(float);
  return smem < 120 * 1024 ? 120 * 1024 : smem;
}

template <int NK, int NV, int MODE>
static int launch(const AttnParams& p, const CUtensorMap& km, const CUtensorMap& vm, int num_items, int log2_page,
                  cudaStream_t stream, const AttnExtras& x) {
  const size_t smem = portion_smem(NK, NV, MODE == MODE_BIAS, p.G);
  if (smem > PORTION_SMEM_LIMIT) return -2;
  auto k = attn_portion_tc05_kernel<NK, NV, MODE>;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  si_launch(k, dim3(p.KV, num_items, (p.vs + NV * 64 - 1) / (NV * 64)), dim3(320), smem, stream, p, km, vm, log2_page, x);
  return si_last_error();
}

// The cut of a step's items into shares (host arithmetic only; called before every long prompt step, so in native code: some 3,000 steps of
// a heap). `tiles[i]`: key tiles of item i, which runs for `copies` key/value heads; `blocks` run at once. Longest shares are tried from the
// longest item down and the shortest schedule is taken (longest share first to the block that is free first; a share costs its tiles and
// about two for its start, a cut item's share three more for handing over). No share is below `least` tiles; at most `most` shares are
// partial results. entries [cap][4] receives (item, share, shares, first slot), longest first, cut [n][4] (item, shares, first slot, 0),
// counts (entries, cut items, slots). Returns 1, 0 where whole items are within a twentieth of the best, or -2.
static int cut_portions(const int* tiles, int n, int copies, int blocks, int least, long long most, int* entries, int cap, int* cut, int* counts) {
  if (n <= 0 || copies <= 0 || blocks <= 0 || least <= 0) return -2;
  long long longest = 0, total = 0;
  for (int i = 0; i < n; ++i) {
    longest = std::max<long long>(longest, tiles[i]);
    total += (long long)tiles[i] * copies;
  }
  if (longest < 2LL * least || (long long)n * copies > 8LL * blocks) return 0;
  auto up = [](long long a, long long b) { return (a + b - 1) / b; };
  std::vector<long long> cost, heap;
  auto schedule = [&](long long limit) {
    cost.clear();
    for (int i = 0; i < n; ++i) {
      if (tiles[i] <= 0) continue;
      const long long shares = up(tiles[i], limit), each = up(tiles[i], shares) + 2 + (shares > 1 ? 3 : 0);
      cost.insert(cost.end(), (size_t)shares, each);
    }
    std::sort(cost.begin(), cost.end(), std::greater<long long>());
    heap.assign((size_t)blocks, 0);                        // every block's end, the earliest on top
    long long end = 0;
    for (const long long c : cost)
      for (int k = 0; k < copies; ++k) {
        const long long v = heap[0] + c;
        end = std::max(end, v);
        size_t at = 0;
        for (;;) {
          size_t kid = 2 * at + 1;
          if (kid >= heap.size()) break;
          if (kid + 1 < heap.size() && heap[kid + 1] < heap[kid]) ++kid;
          if (heap[kid] >= v) break;
          heap[at] = heap[kid];
          at = kid;
        }
        heap[at] = v;
      }
    return end;
  };
  const long long whole = schedule(longest);
  if ((double)whole * 0.95 <= (double)total / blocks) return 0;
  std::vector<long long> limits;
  for (const int k : {2, 3, 4, 6, 9, 13, 18}) {
    const long long limit = std::max<long long>(least, up(longest, k));
    long long shares = 0;
    for (int i = 0; i < n; ++i) shares += tiles[i] > limit ? up(tiles[i], limit) : 0;
    if ((k <= 6 || (long long)n * copies * k <= 4LL * blocks) && limit < longest && shares * copies <= most) limits.push_back(limit);
  }
  std::sort(limits.begin(), limits.end());
  limits.erase(std::unique(limits.begin(), limits.end()), limits.end());
  long long best = -1, limit = 0;
  for (const long long l : limits) {
    const long long end = schedule(l);
    if (best < 0 || end < best) { best = end; limit = l; }
  }
  if (best < 0 || (double)best > 0.95 * (double)whole) return 0;
  int num = 0, num_cut = 0, slots = 0;
  struct Share { long long length; int v[4]; };
  std::vector<Share> all;
  for (int i = 0; i < n; ++i) {
    if (tiles[i] <= 0) continue;
    const int shares = (int)up(tiles[i], limit);
    if (shares > 32 || num + shares > cap) return -2;      // (a merging warp's lanes; never with 18 shares at most)
    for (int k = 0; k < shares; ++k) all.push_back(Share{up(tiles[i], shares), {i, k, shares, shares > 1 ? slots : 0}});
    num += shares;
    if (shares > 1) {
      const int e[4] = {i, shares, slots, 0};
      std::copy(e, e + 4, cut + 4 * (num_cut++));
      slots += shares;
    }
  }
  std::stable_sort(all.begin(), all.end(), [](const Share& x, const Share& y) { return x.length > y.length; });
  for (int i = 0; i < num; ++i) std::copy(all[i].v, all[i].v + 4, entries + 4 * i);
  counts[0] = num; counts[1] = num_cut; counts[2] = slots;
  return 1;
}

SI_EXPORT int si_cut_portions(const int* tiles, int n, int copies, int blocks, int least, long long most, int* entries, int cap, int* cut, int* counts) {
  try {
    return cut_portions(tiles, n, copies, blocks, least, most, entries, cap, cut, counts);
  } catch (const std::bad_alloc&) {                        // no memory for the search: whole items serve as well
    return 0;
  }
}

// Floats of partial results of `slots` shares.
SI_EXPORT long long si_attn_portion_share_floats(int slots, int KV, int hs, int vs) {
  return (long long)slots * KV * 256 * ((hs <= 64 && vs <= 64 ? 64 : 128) + 2);
}

static AttnParams make_params(const void* q, long long q_stride, const int* block_table, int table_width, const void* items, void* out,
                              long long out_stride, int num_pages, int page_size, int num_seqs, int H, int KV, int hs, int vs,
                              float scale, int window, int chunk, const float* sink, int* status) {
  AttnParams p;
  p.q = (const bf16*)q; p.q_stride = q_stride;
  p.k_cache = nullptr; p.v_cache = nullptr;          // reached through the tensor maps
  p.block_table = block_table; p.table_width = table_width;
  p.items = (const AttnItem*)items;
  p.out = (bf16*)out; p.out_stride = out_stride;
  p.part_o = nullptr; p.part_ml = nullptr; p.counters = nullptr;
  p.num_pages = num_pages; p.page_size = page_size; p.num_seqs = num_seqs;
  p.H = H; p.KV = KV; p.G = H / KV; p.hs = hs; p.vs = vs;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.window = window; p.chunk = chunk; p.sink = sink; p.nsplit = 1; p.status = status;
  return p;
}
static int log2_of(int n) { int l = 0; while ((1 << l) < n) ++l; return l; }

// Same contract as si_attn_portion (attention_mma.cu) with the tensor maps of the layer's K and V cache
// (made by si_attn_encode_cache_map of attention_tma.cu); items hold at most si_attn_portion_tc05_tokens().
// `slopes`, the query temperature and `gate` (see AttnExtras) select the extended kernel; without them the plain one runs.
// Values that are the keys: pass the key cache and its map as the values too.
SI_EXPORT int si_attn_portion_tc05(const void* q, long long q_stride, const void* k_cache, const void* v_cache,
                                   const void* kmap, const void* vmap, const int* block_table, int table_width,
                                   const void* items, int num_items, void* out, long long out_stride, int num_pages,
                                   int page_size, int num_seqs, int H, int KV, int hs, int vs, float scale, int window,
                                   const float* slopes, float qt_coef, int qt_every, const void* gate, long long gate_stride,
                                   int chunk, const float* sink, const int* shares, int num_shares, const int* cut, int num_cut,
                                   int slots, float* scratch, int* status, cudaStream_t stream) {
  if (num_items <= 0) return 0;
  if (qt_every < 0 || chunk < 0 || (gate && (gate_stride % 8 || ((uintptr_t)gate % 16)))) return -2;
  // a temperature below zero would turn the order of the scores round: the plain kernels serve that
  AttnExtras x = {};
  x.slopes = slopes; x.qt_coef = qt_coef; x.qt_every = qt_every; x.gate = (const bf16*)gate; x.gate_stride = gate_stride; x.v_share = 1;
  const bool ext = slopes || qt_every > 0 || gate;
  if (num_items > 65535) return -2;                  // the grid's second dimension
  if (!si_attn_portion_tc05_ok(H, KV, hs, vs, page_size) || !kmap || !vmap) return -2;
  if ((q_stride % 8) || (out_stride % 8) || ((uintptr_t)q % 16) || ((uintptr_t)out % 16)) return -2;
  const AttnParams p = make_params(q, q_stride, block_table, table_width, items, out, out_stride, num_pages, page_size, num_seqs, H, KV,
                                   hs, vs, scale, window, chunk, sink, status);
  const int log2_page = log2_of(page_size);
  const CUtensorMap& km = *(const CUtensorMap*)kmap;
  const CUtensorMap& vm = *(const CUtensorMap*)vmap;
  if (ext && (hs != vs || (hs != 64 && hs != 128))) return -2;
  const bool narrow = hs <= 64 && vs <= 64;
  if (shares) {                                      // see AttnExtras
    if (ext || num_shares <= 0 || num_shares > 65535 || num_cut < 0 || num_cut > 65535 || (num_cut && (!cut || !scratch || slots <= 0))) return -2;
    if (((uintptr_t)shares | (uintptr_t)cut | (uintptr_t)scratch) & 15) return -2;
    const int dv = narrow ? 64 : 128;
    x.shares = (const int4*)shares;
    x.part_o = scratch;
    x.part_ml = scratch + (long long)slots * KV * 256 * dv;
    int rc = narrow ? launch<1, 1, MODE_CUT>(p, km, vm, num_shares, log2_page, stream, x) : launch<2, 2, MODE_CUT>(p, km, vm, num_shares, log2_page, stream, x);
    if (rc || !num_cut) return rc;
    const dim3 grid(KV, num_cut, 32);
    if (narrow) si_launch(attn_portion_merge_kernel<1>, grid, dim3(256), 0, stream, p, (const int4*)cut, (const float*)x.part_o, (const float*)x.part_ml);
    else si_launch(attn_portion_merge_kernel<2>, grid, dim3(256), 0, stream, p, (const int4*)cut, (const float*)x.part_o, (const float*)x.part_ml);
    return si_last_error();
  }
  if (ext) return narrow ? launch<1, 1, MODE_EXT>(p, km, vm, num_items, log2_page, stream, x) : launch<2, 2, MODE_EXT>(p, km, vm, num_items, log2_page, stream, x);
  return narrow ? launch<1, 1, MODE_PLAIN>(p, km, vm, num_items, log2_page, stream, x) : launch<2, 2, MODE_PLAIN>(p, km, vm, num_items, log2_page, stream, x);
}

// The general form: key size up to 192, values of any size (128 columns a block), key heads that share a value head, results in fp32,
// and one of a bias by distance (fp32 [nd, H]) and a soft limit, over pages or (dense) over matrices of one row a token
// [rows, KV * size] in which sequence s has the rows from block_table[s, 0] on. 1 when it takes the layout.
#define DENSE_BOX 64
SI_EXPORT int si_attn_portion_gen_ok(int H, int KV, int dk, int dv, int v_share, int page_size, int dense, int bias, int cap) {
  if (KV <= 0 || H % KV || H / KV > 128 || v_share < 1 || KV % v_share) return 0;
  if (dk <= 0 || dv <= 0 || dk > 192 || dk % 8 || dv % 8 || dv > 8192 || (bias && cap)) return 0;
  if ((bias || cap) && dk > 128) return 0;
  // a bias's windows stand beside the tiles in shared memory: up to 13 heads a key head with two halves of key columns
  if (bias && (H / KV > 16 || portion_smem((dk + 63) / 64, 2, true, H / KV) > PORTION_SMEM_LIMIT)) return 0;
  if (!dense && page_size != 8 && page_size != 16 && page_size != 32 && page_size != 64) return 0;
  return si_encode_fn() != nullptr;
}

// `keys`, `values`: the caches' tensor maps, or (dense) the matrices themselves, of `num_pages` rows.
SI_EXPORT int si_attn_portion_gen(const void* q, long long q_stride, const void* keys, const void* values, const int* block_table, int table_width,
                                  const void* items, int num_items, void* out, int out_f32, long long out_stride, int num_pages, int page_size,
                                  int dense, int num_seqs, int H, int KV, int dk, int dv, int v_share, float scale, int window, int chunk,
                                  const float* sink, const float* bias, int nd, float softcap, int* status, cudaStream_t stream) {
  if (num_items <= 0) return 0;
  if (num_items > 65535 || chunk < 0 || softcap < 0.f || !keys || !values || (bias && nd <= 0) || table_width <= 0) return -2;
  if (!si_attn_portion_gen_ok(H, KV, dk, dv, v_share, page_size, dense, bias != nullptr, softcap > 0.f)) return -2;
  if ((q_stride % 8) || (out_stride % 8) || ((uintptr_t)q % 16) || ((uintptr_t)out % 16)) return -2;
  AttnExtras x = {};
  x.v_share = v_share; x.out_f32 = out_f32; x.dense = dense; x.bias = bias; x.nd = nd;
  if (softcap > 0.f) { x.cap_log2 = softcap * 1.4426950408889634f; x.scale_over_cap = scale / softcap; }
  const AttnParams p = make_params(q, q_stride, block_table, table_width, items, out, out_stride, num_pages, page_size, num_seqs, H, KV,
                                   dk, dv, scale, window, chunk, sink, status);
  const int log2_page = log2_of(dense ? DENSE_BOX : page_size), nk = (dk + 63) / 64;
  alignas(64) CUtensorMap km, vm;
  if (dense) {
    if (num_pages <= 0 || ((uintptr_t)keys % 16) || ((uintptr_t)values % 16)) return -2;
    int rc = si_encode_bf16_heads(&km, keys, (unsigned long long)num_pages, KV, dk, DENSE_BOX);
    if (!rc) rc = si_encode_bf16_heads(&vm, values, (unsigned long long)num_pages, KV / v_share, dv, DENSE_BOX);
    if (rc) return rc;
  } else {
    km = *(const CUtensorMap*)keys;
    vm = *(const CUtensorMap*)values;
  }
#define GEN_LAUNCH(NK, MODE) return launch<NK, 2, MODE>(p, km, vm, num_items, log2_page, stream, x)
  if (bias) { if (nk == 1) GEN_LAUNCH(1, MODE_BIAS); GEN_LAUNCH(2, MODE_BIAS); }
  if (softcap > 0.f) { if (nk == 1) GEN_LAUNCH(1, MODE_CAP); GEN_LAUNCH(2, MODE_CAP); }
  if (nk == 1) GEN_LAUNCH(1, MODE_GEN);
  if (nk == 2) GEN_LAUNCH(2, MODE_GEN);
  GEN_LAUNCH(3, MODE_GEN);
#undef GEN_LAUNCH
}
