// Shared device helpers for every kernel file: element load/store through fp32,
// warp and block reductions, and the status word that kernels write instead of
// trapping. Each .cu file is compiled on its own into one shared library and
// exports plain C entry points that take raw device pointers and a stream.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdlib.h>

// A file that includes another .cu file to reuse its kernels defines SI_EXPORT first (hidden visibility),
// so that the included file's entry points are not exported a second time from its library.
#ifndef SI_EXPORT
#define SI_EXPORT extern "C" __attribute__((visibility("default")))
#endif

// Status codes written (atomicMax) into the engine's device status word.
enum SiStatus : int {
  SI_OK = 0,
  SI_BAD_TOKEN = 1,      // token id outside [0, vocab)
  SI_BAD_PAGE = 2,       // block table entry outside [0, num_pages)
  SI_BAD_SEQ = 3,        // row names a sequence outside the batch
  SI_WAIT_LIMIT = 4,     // a bounded wait inside a kernel ran out
};

// dtype codes shared with the Python binding
enum SiDtype : int { SI_F32 = 0, SI_BF16 = 1 };

template <typename T> __device__ __forceinline__ float to_f32(T v);
template <> __device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) {
  return __bfloat162float(v);
}
template <typename T> __device__ __forceinline__ T from_f32(float v);
template <> __device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) {
  return __float2bfloat16_rn(v);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// Sum over a block of up to 1024 threads; every thread gets the result.
// `scratch` holds 33 floats of shared memory.
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();                 // scratch may still be read from an earlier call
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  if (warp == 0) {
    float s = lane < nwarps ? scratch[lane] : 0.f;
    s = warp_sum(s);
    if (lane == 0) scratch[32] = s;
  }
  __syncthreads();
  return scratch[32];
}

// The feed-forward's gated activation: silu(g) * u in fp32.
__device__ __forceinline__ float silu_mul(float g, float u) { return (g / (1.f + expf(-g))) * u; }

__device__ __forceinline__ void set_status(int* status, int code) {
  if (status) atomicMax(status, code);
}

// Programmatic dependent launch: a kernel launched through si_launch() carries the attribute that lets its launch overlap the end
// of the kernel before it; it waits for that kernel's results (pdl_wait, or pdl_prologue at its start) before it touches what
// others write. Launched with <<<>>> the instruction does nothing. SI_PDL=0 in the environment turns the attribute off.
//
// Loads through the read-only path (ld.global.nc, which the compiler also makes of const __restrict__ pointers) may be moved across
// the wait, since they promise that nothing writes there while the kernel runs: a product's rows were read so before the kernel before
// had written them. Behind a branch on a value that comes with the wait they stay: a load is not made before it is known that it is to be.
__device__ __forceinline__ void pdl_wait() {
  unsigned sms;
  asm volatile("griddepcontrol.wait;\n\tmov.u32 %0, %%nsmid;\n" : "=r"(sms) :: "memory");
  if (sms == 0u) {                       // never
    asm volatile("exit;\n");
    __builtin_unreachable();
  }
}
__device__ __forceinline__ void pdl_prologue() { pdl_wait(); }

// A decode row's norm weights have left L2 since the step before (all weights passed through it): a hint at a thread's own, given before the wait
// for the kernel before, brings them while the row is still being made. Many rows find them in L2.
__device__ __forceinline__ void prefetch_l1(const void* p) { asm volatile("prefetch.global.L1 [%0];\n" :: "l"(p) : "memory"); }

// A hint that [base, base + bytes) will be streamed soon: block `part` of `parts` asks the memory system
// to bring its share into L2, one prefetch per 128-byte line. Kernels that wait on latency while HBM
// idles (the norms of a decode step) call this for the first weights of the matrix product after them.
__device__ __forceinline__ void l2_prefetch_share(const void* base, long long bytes, int part, int parts) {
  constexpr long long LINE = 128;
  const long long lines = bytes / LINE;
  const long long per = (lines + parts - 1) / parts;
  const long long c0 = (long long)part * per;
  const long long c1 = c0 + per < lines ? c0 + per : lines;
  for (long long c = c0 + threadIdx.x; c < c1; c += blockDim.x)
    asm volatile("prefetch.global.L2 [%0];\n" :: "l"(reinterpret_cast<const char*>(base) + c * LINE) : "memory");
}

// For kernels that let the next one launch early. A small kernel (a norm, the
// position encoding) calls pdl_trigger() at its start: the kernel after it may then become resident and do
// whatever does not depend on this one (set-up, the first loads of its weights) before its own pdl_wait().
// Kernels of more than one wave do not trigger: blocks of the next kernel that sit waiting would take the
// places of their own later blocks.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// SI_PDL_TRIGGER: 0 no kernel triggers but the tcgen05 ones, which always do; 1 the small kernels too; 2 (default; higher levels are the same)
// also every kernel of one wave of blocks, at its start.
static inline int si_pdl_trigger_level() {
  static int level = -1;
  if (level < 0) {
    const char* e = getenv("SI_PDL_TRIGGER");
    level = (e && (e[0] == '0' || e[0] == '1')) ? e[0] - '0' : 2;
  }
  return level;
}
static inline bool si_pdl_trigger_enabled() { return si_pdl_trigger_level() >= 1; }
// Whether a small kernel of `blocks` blocks, a handful as a decode step's rows make them, triggers: 1 or 0. For the norms, combines, gates,
// preparations and stores of decode rows, whose next kernel has weights or older keys to ask for meanwhile. Passes with and without, us: two
// Mivorax requests 9,990 and 10,245, 16 14,020 and 14,400, two Fevosun requests 14,840 and 15,230; a line at 148 blocks instead of 64 and batches of 100
// requests: no difference.
static inline int si_pdl_trigger_small(long long blocks) { return blocks <= 64 && si_pdl_trigger_enabled() ? 1 : 0; }
// Whether a kernel of `blocks` blocks, `slots` of which run at once, triggers at its start: 1 or 0.
static inline int si_pdl_trigger_mode(long long blocks, long long slots) { return blocks <= slots && si_pdl_trigger_level() >= 2 ? 1 : 0; }

// Streaming multiprocessors of the current device, asked once per device. Grid sizes that should fill the
// device once ("one wave") are derived from it; no kernel's result depends on it.
static inline int si_sm_count() {
  static int count[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (count[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 1;
    count[dev] = n;
  }
  return count[dev];
}

static inline bool si_pdl_enabled() {
  static int on = -1;
  if (on < 0) {
    const char* e = getenv("SI_PDL");
    on = (e && e[0] == '0') ? 0 : 1;
  }
  return on == 1;
}

template <typename... P, typename... A>
static inline void si_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = si_pdl_enabled() ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// Shares of a row's entries for kernels that take a block a row: one while the rows alone give every SM two blocks,
// else as many as bring the blocks there, each share at least one pass of the block's threads.
static inline int si_row_shares(long long rows, long long entries, int threads) {
  const long long want = 2LL * si_sm_count();
  if (rows >= want || rows <= 0) return 1;
  long long shares = (want + rows - 1) / rows;
  const long long most = (entries + threads - 1) / threads;
  if (shares > most) shares = most;
  if (shares > 64) shares = 64;
  return shares < 1 ? 1 : (int)shares;
}

static inline int si_last_error() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}
