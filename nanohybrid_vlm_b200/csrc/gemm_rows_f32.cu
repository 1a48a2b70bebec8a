// out[M, N] (fp32) = x[M, K] @ w[N, K]^T for bfloat16 operands and few outputs: the small projections whose results
// enter a recurrence or a gate in 32-bit (a handful of rows of w, a step of a few tokens).  One warp per output:
// the lanes walk K in 16-byte pieces, sum in fp32 in a fixed order and meet in a shuffle tree, so an output does
// not depend on what else is in the batch.  Large M goes to the library product instead (the caller decides).
// Bound by latency (a step's x and these rows are a few hundred kilobytes): a warp asks for up to eight pieces of its row of w before it
// waits for the kernel before, and for as many of x at once (read piece by piece behind the wait, a launch of 16 rows of K = 2,048 took
// 2.7 and 2.8 us for 8 and 48 tokens; 1.7 and 2.3 now).
#include "nhv_common.cuh"

constexpr int GR_WARPS = 4;

// AHEAD: pieces of a row on their way at once, 256 columns each
template <int AHEAD>
__global__ void __launch_bounds__(GR_WARPS * 32) gemm_rows_f32_kernel(float* __restrict__ out, int out_stride,
                                                                       const __nv_bfloat16* __restrict__ x, int x_stride,
                                                                       const __nv_bfloat16* __restrict__ w, int w_stride,
                                                                       int M, int N, int K) {
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long item = (long)blockIdx.x * GR_WARPS + warp;
  const bool there = item < (long)M * N;
  const int m = there ? (int)(item / N) : 0, n = there ? (int)(item - (long)m * N) : 0, pieces = K >> 3;
  const uint4* xr = reinterpret_cast<const uint4*>(x + (size_t)m * x_stride);
  const uint4* wr = reinterpret_cast<const uint4*>(w + (size_t)n * w_stride);
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 a[AHEAD], b[AHEAD];
#pragma unroll
  for (int i = 0; i < AHEAD; ++i) b[i] = lane + 32 * i < pieces ? wr[lane + 32 * i] : zero;
  pdl_wait();
  if (!there) return;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (int c0 = lane; c0 < pieces; c0 += 32 * AHEAD) {
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) a[i] = c0 + 32 * i < pieces ? xr[c0 + 32 * i] : zero;
    if (c0 != lane)
#pragma unroll
      for (int i = 0; i < AHEAD; ++i) b[i] = c0 + 32 * i < pieces ? wr[c0 + 32 * i] : zero;
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      if (c0 + 32 * i >= pieces) break;
      const __nv_bfloat162* ap = reinterpret_cast<const __nv_bfloat162*>(&a[i]);
      const __nv_bfloat162* bp = reinterpret_cast<const __nv_bfloat162*>(&b[i]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 fa = __bfloat1622float2(ap[e]), fb = __bfloat1622float2(bp[e]);
        acc[e] = fmaf(fa.x, fb.x, acc[e]);
        acc[e] = fmaf(fa.y, fb.y, acc[e]);
      }
    }
  }
  const float sum = warp_sum((acc[0] + acc[1]) + (acc[2] + acc[3]));
  if (lane == 0) out[(size_t)m * out_stride + n] = sum;
}

NHV_API int nhv_gemm_rows_f32(float* out, int out_stride, const void* x, int x_stride, const void* w, int w_stride, int M,
                              int N, int K, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  NHV_REQUIRE(M > 0 && N > 0 && K > 0 && K % 8 == 0 && x_stride % 8 == 0 && w_stride % 8 == 0 &&
                  ((uintptr_t)x % 16) == 0 && ((uintptr_t)w % 16) == 0,
              "gemm_rows_f32: K and the row strides must be multiples of 8 elements, the operands 16-byte aligned");
  const long items = (long)M * N;
  // As many pieces as a row has, up to eight; with eight a thread takes 120 registers, so for more outputs than fit on the SMs then, one:
  // 200 x 40 outputs of K = 1,024 5.4 us with eight, 4.0 with two and 3.6 with one, of 4,096 10.1, 9.6 and 8.1; 100 x 40 of 2,048 4.0, 4.2
  // and 4.1, 8 x 16 of 4,096 2.3, 3.4 and 2.9; 48 x 64 of 512 2.7 with eight and 1.9 with two.
  const int ahead = items > 5000 && K > 512 ? 1 : K > 1024 ? 8 : K > 512 ? 4 : K > 256 ? 2 : 1;
#define GO(AHEAD)                                                                                                            \
  nhv_launch(gemm_rows_f32_kernel<AHEAD>, (int)((items + GR_WARPS - 1) / GR_WARPS), GR_WARPS * 32, 0, stream, out, out_stride, \
             (const __nv_bfloat16*)x, x_stride, (const __nv_bfloat16*)w, w_stride, M, N, K)
  if (ahead == 8) GO(8);
  else if (ahead == 4) GO(4);
  else if (ahead == 2) GO(2);
  else GO(1);
#undef GO
  NHV_CHECK_LAUNCH("gemm_rows_f32");
  return 0;
}
