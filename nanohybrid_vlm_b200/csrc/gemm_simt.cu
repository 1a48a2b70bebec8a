// C[M,N] = A[M,K] * W[N,K]^T on the CUDA cores with fp32 multiply-add: the matrix
// product of the true 32-bit path (no TF32 or other reduced-precision matrix mode) for sizes that
// gemm_f32_tcgen05.cu does not take, also usable with bf16 storage.  W is row-major [out, in] as in nanovllm/layers/linear.py:40,66.
//
// Each output element is two accumulators, of the products at even and at odd k, each in ascending k, added at the
// end; so the value of C[m,n] does not depend on M, on the tile that holds it or on the batch.
//
// Bound by the FP32 pipes (72 TFLOP/s) from some dozens of rows on, by reading W below that, and by the way from
// global to shared memory where a product has few tiles.  So:
//   - both operands lie in shared memory as they lie in global memory, 32 columns of k a stage, and reach it by
//     cp.async in pieces of 16 bytes, two or more stages ahead of the multiplying (one stage ahead through registers
//     left 0.8 us per 16 columns exposed: 155 us for 3 x 1024 x 3072);
//   - a thread reads four consecutive k of a row at once, two pairs, and one instruction multiplies and adds a pair
//     into the pair of accumulators of even and odd k: no transposing, no duplicating of operands;
//   - rows of 36 floats spread the eight (four) rows that a warp reads at once over all banks.
// A warp holds 4 x 8 threads of TM x TN outputs each, rows 4 apart, columns 8 apart.  Operands that cp.async cannot
// take (bf16, sizes or addresses that are no multiple of 16 bytes) go through registers into the same places.
// 370 x 6144 x 1024: 123 us (38 TFLOP/s); 370 x 1024 x 3072: 108 us; 3 x 1024 x 3072: 66 us.  Tiles of 64 x 64 outputs
// loaded 4 bytes at a time, without overlap, ran the four products of such a layer at about 13 TFLOP/s in all.
#include <type_traits>

#include "nhv_common.cuh"

constexpr int GK = 32;                                   // columns of k per stage
constexpr int GS = GK + 4;                               // floats of a row in shared memory

static __device__ __forceinline__ void copy16(float* smem, const float* gmem, bool there) {
  const int bytes = there ? 16 : 0;                      // what is not there arrives as zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem),
               "r"(bytes));
}

template <typename T, typename TO, int TM, int TN, int WM, int WN, int STAGES, bool ASYNC>
__global__ void __launch_bounds__(WM * WN * 32) gemm_nt_simt_kernel(
    TO* __restrict__ C, const T* __restrict__ A, const T* __restrict__ W, int M, int N, int K, int lda, int ldw, int ldc,
    long batch_a, long batch_w, long batch_c) {
  constexpr int THREADS = WM * WN * 32, GM = WM * 4 * TM, GN = WN * 8 * TN;
  extern __shared__ __align__(16) float smem[];          // [STAGES][GM + GN][GS]
  pdl_prologue();
  A += (size_t)blockIdx.z * batch_a;                     // one product per blockIdx.z, the operands a fixed step apart
  W += (size_t)blockIdx.z * batch_w;
  C += (size_t)blockIdx.z * batch_c;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int row0 = (warp / WN) * 4 * TM + (lane >> 3), col0 = (warp % WN) * 8 * TN + (lane & 7);
  const int m0 = blockIdx.y * GM, n0 = blockIdx.x * GN;

  auto fetch = [&](int c) {                              // stage c: columns [c * GK, (c + 1) * GK)
    float* to = smem + (c % STAGES) * (GM + GN) * GS;
#pragma unroll
    for (int e = tid; e < (GM + GN) * (GK / 4); e += THREADS) {
      const int r = e / (GK / 4), kk = 4 * (e % (GK / 4)), k = c * GK + kk;
      const bool a = r < GM;
      const int at = a ? m0 + r : n0 + r - GM;
      const bool row = at < (a ? M : N);
      const T* src = a ? A : W;
      const size_t base = row ? (size_t)at * (a ? lda : ldw) : 0;
      if constexpr (ASYNC) {
        const bool there = row && k < K;                 // K is a multiple of 4
        copy16(to + r * GS + kk, src + (there ? base + k : 0), there);
      } else {
        float v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = row && k + i < K ? to_f32<T>(src[base + k + i]) : 0.f;
        *reinterpret_cast<float4*>(to + r * GS + kk) = make_float4(v[0], v[1], v[2], v[3]);
      }
    }
  };

  f32x2 acc[TM][TN];                                     // sums over even k | over odd k
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;

  const int n_stages = (K + GK - 1) / GK;
#pragma unroll
  for (int c = 0; c < STAGES - 1; ++c) {
    if (c < n_stages) fetch(c);
    asm volatile("cp.async.commit_group;\n" ::);
  }
  for (int c = 0; c < n_stages; ++c) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
    __syncthreads();                                     // stage c is there; stage c - 1 has been read by all
    if (c + STAGES - 1 < n_stages) fetch(c + STAGES - 1);
    asm volatile("cp.async.commit_group;\n" ::);
    const float* as = smem + (c % STAGES) * (GM + GN) * GS + row0 * GS;
    const float* ws = smem + (c % STAGES) * (GM + GN) * GS + (GM + col0) * GS;
#pragma unroll
    for (int kk = 0; kk < GK; kk += 4) {
      ulonglong2 a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(as + 4 * i * GS + kk);
#pragma unroll
      for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(ws + 8 * j * GS + kk);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = f2_fma(a[i].x, w[j].x, acc[i][j]);
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = f2_fma(a[i].y, w[j].y, acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + row0 + 4 * i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int n = n0 + col0 + 8 * j;
      float even, odd;
      f2_unpack(acc[i][j], even, odd);
      if (n < N) C[(size_t)m * ldc + n] = from_f32<TO>(even + odd);
    }
  }
}

struct SimtGemm {
  void* C;
  const void *A, *W;
  int M, N, K, lda, ldw, ldc, batch;
  long batch_a, batch_w, batch_c;
  bool vec;
  cudaStream_t stream;
};

template <typename T, typename TO, int TM, int TN, int WM, int WN, int STAGES>
static cudaError_t launch_tile(const SimtGemm& g) {
  constexpr int GM = WM * 4 * TM, GN = WN * 8 * TN, SMEM = STAGES * (GM + GN) * GS * 4;
  const dim3 grid((g.N + GN - 1) / GN, (g.M + GM - 1) / GM, g.batch);
  static std::atomic<uint64_t> done[2];
  auto go = [&](auto kernel, int which) {
    const cudaError_t e = nhv_allow_smem((const void*)kernel, SMEM, done[which]);
    if (e != cudaSuccess) return e;
    return nhv_launch(kernel, grid, WM * WN * 32, SMEM, g.stream, (TO*)g.C, (const T*)g.A, (const T*)g.W, g.M, g.N, g.K,
                      g.lda, g.ldw, g.ldc, g.batch_a, g.batch_w, g.batch_c);
  };
  if constexpr (std::is_same<T, float>::value)
    if (g.vec) return go(gemm_nt_simt_kernel<T, TO, TM, TN, WM, WN, STAGES, true>, 1);
  return go(gemm_nt_simt_kernel<T, TO, TM, TN, WM, WN, STAGES, false>, 0);
}

// Which tile: an SM works through its share of the tiles, so the time goes with the tiles of the fullest SM times what
// one costs; the smaller tiles cost more per output (more reads of shared memory per multiply-add).  In us, tiles of
// 64 x 64, 32 x 64, 16 x 32: 123, 139, 181 for 370 x 6144 x 1024; 108, 117, 137 for 370 x 1024 x 3072; 186, 162, 168 for
// 600 x 1024 x 3072; 106, 80, 66 for 60 x 1024 x 3072.
template <typename T, typename TO>
static cudaError_t launch_simt(const SimtGemm& g) {
  auto cost = [&](int gm, int gn, float per_output) {
    const long tiles = (long)((g.M + gm - 1) / gm) * ((g.N + gn - 1) / gn) * g.batch;
    return (float)((tiles + 147) / 148) * gm * gn * per_output;
  };
  const float large = cost(64, 64, 1.0f), medium = cost(32, 64, 1.25f), small = cost(16, 32, 1.7f);
  // (M / 64 blocks fit the grid's second dimension, the caller checks; finer cuts of so many rows might not)
  if ((large <= medium && large <= small) || g.M > 16 * 65535) return launch_tile<T, TO, 8, 4, 2, 2, 3>(g);
  if (medium <= small) return launch_tile<T, TO, 4, 4, 2, 2, 4>(g);
  return launch_tile<T, TO, 4, 4, 1, 1, 6>(g);
}

// out_f32 != 0: C is fp32 whatever the storage type of A and W (logits).
// `batch` products in one launch: product b reads A + b * batch_a, W + b * batch_w and writes C + b * batch_c (in
// elements); the operands of different products may interleave (heads side by side in a row).
NHV_API int nhv_gemm_nt_simt_batched(int dtype, void* C, const void* A, const void* W, int M, int N, int K, int lda,
                                     int ldw, int ldc, int out_f32, int batch, long batch_a, long batch_w,
                                     long batch_c, cudaStream_t stream) {
  if (M == 0 || N == 0 || batch == 0) return 0;
  NHV_REQUIRE(M > 0 && N > 0 && K > 0 && lda >= K && ldw >= K && ldc >= N, "gemm: bad sizes M=%d N=%d K=%d", M, N, K);
  NHV_REQUIRE((M + 63) / 64 <= 65535 && batch > 0 && batch <= 65535, "gemm: M=%d or %d products are beyond the grid's reach",
              M, batch);
  const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && batch_a % 4 == 0 && batch_w % 4 == 0 &&
                   (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
  const SimtGemm g{C, A, W, M, N, K, lda, ldw, ldc, batch, batch_a, batch_w, batch_c, vec, stream};
  if (dtype == NHV_F32) NHV_CUDA((launch_simt<float, float>(g)), "gemm_nt_simt");
  else if (dtype == NHV_BF16 && out_f32) NHV_CUDA((launch_simt<__nv_bfloat16, float>(g)), "gemm_nt_simt");
  else if (dtype == NHV_BF16) NHV_CUDA((launch_simt<__nv_bfloat16, __nv_bfloat16>(g)), "gemm_nt_simt");
  else NHV_REQUIRE(false, "gemm: unknown dtype %d", dtype);
  NHV_CHECK_LAUNCH("gemm_nt_simt");
  return 0;
}

NHV_API int nhv_gemm_nt_simt(int dtype, void* C, const void* A, const void* W, int M, int N, int K, int lda, int ldw,
                             int ldc, int out_f32, cudaStream_t stream) {
  return nhv_gemm_nt_simt_batched(dtype, C, A, W, M, N, K, lda, ldw, ldc, out_f32, 1, 0, 0, 0, stream);
}
