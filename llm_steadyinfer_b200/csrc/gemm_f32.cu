// True 32-bit matrix product for the fp32 path: C[M, N] = A[M, K] * W[N, K]^T with plain
// FFMA and fp32 accumulation, no tensor cores and no reduced-precision mode. (The
// reference's "fp32" GEMM is cuBLAS TF32, src/source/op/kernels/cuda/matmul_kernel.cu:128-150;
// its exact fallback is the one-block-per-row kernel at :12-63.) The k loop runs in one
// fixed order for every output element, whatever M and the tile are, so a row's result does not depend
// on how many other rows share the step.
//
// Tiles of A and W lie in shared memory as rows of BK entries of k, fetched by cp.async STAGES - 1 tiles ahead; a thread reads four
// entries of k of its TM rows and TN columns as 16-byte words. Tiles of 64 x 64 where they give every SM one, tiles of 16 x 32 (a
// sixteenth and less of the work, so that a small product spreads over more SMs) where they do not: a small product is bound by one
// block's chain of K dependent sums and the first fetch.
// Measured at six rows, N and K of 96 to 1,000: 3.5 us a launch, where tiles of 64 x 64 alone, one k tile at a time, took 11.3.
// Rows that are not in 16-byte words go entry by entry, where a small tile's fetches outweigh its sums: large tiles from half the SMs on
// (700 x 780, K = 333: 44.3 us in small tiles, 26.3 in large ones; 300 x 1,700, K = 700, in words: 42.4 in small ones, where the large ones of
// before took 53.5).
#include "common.cuh"

template <int BM, int BN, int TM, int TN, int BK, int STAGES, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_kernel(const float* __restrict__ A, long long lda, const float* __restrict__ W,
                long long ldw, float* __restrict__ C, long long ldc, int M, int N, int K) {
  pdl_prologue();
  constexpr int THREADS = (BM / TM) * (BN / TN), PITCH = BK + 4;       // rows apart by 4 banks more than a multiple of 32
  __shared__ __align__(16) float tile[STAGES][BM + BN][PITCH];         // rows of A, then rows of W
  const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int ktiles = (K + BK - 1) / BK;
  auto fetch = [&](int kt) {
    const int k0 = kt * BK;
    float(*dst)[PITCH] = tile[kt % STAGES];
    constexpr int PER = VEC ? 4 : 1, PIECES = BK / PER;
    for (int i = threadIdx.x; i < (BM + BN) * PIECES; i += THREADS) {
      const int r = i / PIECES, c = (i % PIECES) * PER, k = k0 + c;
      const bool of_a = r < BM;
      const int row = of_a ? m0 + r : n0 + r - BM;
      const bool in = row < (of_a ? M : N) && k < K;
      const float* src = of_a ? A + (size_t)(in ? row : 0) * lda : W + (size_t)(in ? row : 0) * ldw;
      if (in) src += k;
      const unsigned to = (unsigned)__cvta_generic_to_shared(&dst[r][c]);
      if (VEC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(src), "r"(in ? 16 : 0));      // K is a multiple of 4
      else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(to), "l"(src), "r"(in ? 4 : 0));
    }
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < ktiles) fetch(s);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  for (int kt = 0; kt < ktiles; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();                     // this tile stands, and everyone is done with the one whose place is filled next
    if (kt + STAGES - 1 < ktiles) fetch(kt + STAGES - 1);
    asm volatile("cp.async.commit_group;\n" ::);
    const float(*t)[PITCH] = tile[kt % STAGES];
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      float4 a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(&t[ty + i * (BM / TM)][kk]);
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(&t[BM + tx + j * (BN / TN)][kk]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
          acc[i][j] = fmaf(a[i].x, w[j].x, acc[i][j]);
          acc[i][j] = fmaf(a[i].y, w[j].y, acc[i][j]);
          acc[i][j] = fmaf(a[i].z, w[j].z, acc[i][j]);
          acc[i][j] = fmaf(a[i].w, w[j].w, acc[i][j]);
        }
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + ty + i * (BM / TM);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + tx + j * (BN / TN);
      if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
    }
  }
}

SI_EXPORT int si_gemm_f32(const float* A, long long lda, const float* W, long long ldw, float* C,
                          long long ldc, int M, int N, int K, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
  const long long big = (long long)((N + 63) / 64) * ((M + 63) / 64);
  const bool large = big >= (vec ? si_sm_count() : si_sm_count() / 2);
  const dim3 grid = large ? dim3((N + 63) / 64, (M + 63) / 64) : dim3((N + 31) / 32, (M + 15) / 16);
  if (grid.y > 65535) return -2;
  if (large) {
    if (vec) si_launch(gemm_f32_kernel<64, 64, 4, 4, 32, 2, true>, grid, dim3(256), 0, stream, A, lda, W, ldw, C, ldc, M, N, K);
    else si_launch(gemm_f32_kernel<64, 64, 4, 4, 16, 3, false>, grid, dim3(256), 0, stream, A, lda, W, ldw, C, ldc, M, N, K);
  } else {
    if (vec) si_launch(gemm_f32_kernel<16, 32, 2, 2, 64, 3, true>, grid, dim3(128), 0, stream, A, lda, W, ldw, C, ldc, M, N, K);
    else si_launch(gemm_f32_kernel<16, 32, 2, 2, 64, 3, false>, grid, dim3(128), 0, stream, A, lda, W, ldw, C, ldc, M, N, K);
  }
  return si_last_error();
}
