// Short causal convolution over time, one filter per channel, with SiLU, for packed steps of several requests.
//
//   y[t, c] = silu(bias[c] + sum_{j < K} w[c, j] * x[t - (K - 1) + j, c])
//
// where t counts within the request: inputs before the request's first token are zero, and inputs before this
// step's portion come from the request's state, which holds its last K - 1 inputs (fp32, [slot][K - 1][C], oldest
// first).  A first kernel computes all outputs (reading the old state), a second one moves the state on; in a step of
// single tokens (the caller says that every request brings exactly one) the first does both, since the thread of a
// channel then is the only one that reads the channel's state: one launch fewer per layer of a decode step, and no
// search for a token's request.  A request with q_start == 0 starts from zeros whatever its slot held.  Requests without a slot (slot < 0: the
// idle entries that pad a captured batch) read zeros and write nothing.
#include "nhv_common.cuh"

constexpr int SC_MAX_TAPS = 8;
constexpr int SC_TOKENS = 32;       // tokens per block of the output kernel in a long step (each input is read once for them);
                                    // a short step takes one token per block: finding a token's request is a chain of
                                    // dependent loads that the tokens of a block would go through one after another

// Entry j of the state that a window (the latest input last) leaves behind
__device__ __forceinline__ float keep(const float (&win)[SC_MAX_TAPS - 1], int j, int K) {
  float v = 0.f;
#pragma unroll
  for (int m = 0; m < SC_MAX_TAPS - 1; ++m)
    if (m == SC_MAX_TAPS - 1 - (K - 1) + j) v = win[m];
  return v;
}

// SINGLE: every request brings one token
template <typename T, typename TO, bool SINGLE>
__global__ void short_conv_silu_kernel(TO* __restrict__ y, int y_stride, const T* __restrict__ x, int x_stride,
                                       const T* __restrict__ w, const T* __restrict__ bias,
                                       float* __restrict__ state, long state_stride,
                                       const int* __restrict__ cu_q, const int* __restrict__ q_start,
                                       const int* __restrict__ slots, int n_seqs, int n_tokens, int C, int K,
                                       int tokens_per_block) {
  pdl_prologue();
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  const int t0 = blockIdx.x * tokens_per_block;
  if (c >= C || t0 >= n_tokens) return;
  // the filter right-aligned in 8 places (the last one is the current token's), zeros before it
  constexpr int M = SC_MAX_TAPS - 1;
  float wr[SC_MAX_TAPS];
#pragma unroll
  for (int m = 0; m < SC_MAX_TAPS; ++m) wr[m] = m >= SC_MAX_TAPS - K ? to_f32<T>(w[(size_t)c * K + (m - (SC_MAX_TAPS - K))]) : 0.f;
  const float b = bias ? to_f32<T>(bias[c]) : 0.f;
  // the request of the tile's first token (binary search over the starts), then walk on
  int lo = SINGLE ? t0 : 0, hi = SINGLE ? t0 : n_seqs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cu_q[mid] <= t0) lo = mid; else hi = mid - 1;
  }
  int s = lo;
  int seq_first = SINGLE ? t0 : cu_q[s], next_first = SINGLE ? t0 + 1 : cu_q[s + 1];
  float win[M];                                     // the inputs before the current token, the latest last
  // the window in front of token t of request s: earlier tokens of this portion, behind them the request's state
  auto fill = [&](int t) {
    const int i = t - seq_first;
    const int slot = slots[s];
    const bool has_past = slot >= 0 && q_start[s] > 0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      float v = 0.f;
      if (m >= M - (K - 1)) {
        const int rel = i - M + m;                  // index in the portion; negative: before it
        if (rel >= 0) v = to_f32<T>(x[(size_t)(t - M + m) * x_stride + c]);
        else if (has_past) v = state[(size_t)slot * state_stride + (size_t)(K - 1 + rel) * C + c];
      }
      win[m] = v;
    }
  };
  fill(t0);
  const int t_end = min(t0 + tokens_per_block, n_tokens);
  for (int t = t0; t < t_end; ++t) {
    if (t >= next_first) {                          // the next request begins (requests without tokens are passed over)
      while (s + 1 < n_seqs && cu_q[s + 1] <= t) ++s;
      seq_first = cu_q[s];
      next_first = cu_q[s + 1];
      fill(t);
    }
    const float xt = to_f32<T>(x[(size_t)t * x_stride + c]);
    float acc = fmaf(wr[M], xt, b);
#pragma unroll
    for (int m = 0; m < M; ++m) acc = fmaf(wr[m], win[m], acc);
#pragma unroll
    for (int m = 0; m + 1 < M; ++m) win[m] = win[m + 1];
    win[M - 1] = xt;
    if (SINGLE && slots[s] >= 0)
#pragma unroll
      for (int j = 0; j < M; ++j)
        if (j < K - 1) state[(size_t)slots[s] * state_stride + (size_t)j * C + c] = keep(win, j, K);
    y[(size_t)t * y_stride + c] = from_f32<TO>(acc / (1.0f + expf(-acc)));
  }
}

template <typename T>
__global__ void short_conv_state_kernel(const T* __restrict__ x, int x_stride, float* __restrict__ state,
                                        long state_stride, const int* __restrict__ cu_q,
                                        const int* __restrict__ q_start, const int* __restrict__ slots, int C, int K) {
  pdl_prologue();
  const int s = blockIdx.x;
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  const int slot = slots[s];
  if (c >= C || slot < 0) return;
  const int first = cu_q[s], n = cu_q[s + 1] - first;
  const bool has_past = q_start[s] > 0;
  float* st = state + (size_t)slot * state_stride;
  float keep[SC_MAX_TAPS];
#pragma unroll
  for (int j = 0; j < SC_MAX_TAPS - 1; ++j) {
    keep[j] = 0.f;
    if (j < K - 1) {
      const int rel = n - (K - 1) + j;              // the input that becomes entry j of the new state
      if (rel >= 0) keep[j] = to_f32<T>(x[(size_t)(first + rel) * x_stride + c]);
      else if (has_past) keep[j] = st[(size_t)(K - 1 + rel) * C + c];
    }
  }
#pragma unroll
  for (int j = 0; j < SC_MAX_TAPS - 1; ++j)
    if (j < K - 1) st[(size_t)j * C + c] = keep[j];
}

// The same filter without bias or activation, added to its own input, for one or two filters over one input:
//   y1[t, c] = x[t, c] + sum_{j < K} w1[c, j] * x[t - (K - 1) + j, c],   y2 likewise with w2 (y2, w2 may be null)
// Both read the same inputs, so one state (the request's last K - 1 inputs) serves both.
template <typename T, bool SINGLE>
__global__ void filter_add_kernel(T* __restrict__ y1, T* __restrict__ y2, int y_stride, const T* __restrict__ x,
                                  int x_stride, const T* __restrict__ w1, const T* __restrict__ w2,
                                  float* __restrict__ state, long state_stride, const int* __restrict__ cu_q,
                                  const int* __restrict__ q_start, const int* __restrict__ slots, int n_seqs,
                                  int n_tokens, int C, int K, int tokens_per_block) {
  pdl_prologue();
  const int c = blockIdx.y * blockDim.x + threadIdx.x;
  const int t0 = blockIdx.x * tokens_per_block;
  if (c >= C || t0 >= n_tokens) return;
  constexpr int M = SC_MAX_TAPS - 1;
  float wa[SC_MAX_TAPS], wb[SC_MAX_TAPS];
#pragma unroll
  for (int m = 0; m < SC_MAX_TAPS; ++m) {
    const bool in = m >= SC_MAX_TAPS - K;
    wa[m] = in ? to_f32<T>(w1[(size_t)c * K + (m - (SC_MAX_TAPS - K))]) : 0.f;
    wb[m] = in && w2 ? to_f32<T>(w2[(size_t)c * K + (m - (SC_MAX_TAPS - K))]) : 0.f;
  }
  int lo = SINGLE ? t0 : 0, hi = SINGLE ? t0 : n_seqs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cu_q[mid] <= t0) lo = mid; else hi = mid - 1;
  }
  int s = lo;
  int seq_first = SINGLE ? t0 : cu_q[s], next_first = SINGLE ? t0 + 1 : cu_q[s + 1];
  float win[M];
  auto fill = [&](int t) {
    const int i = t - seq_first;
    const int slot = slots[s];
    const bool has_past = slot >= 0 && q_start[s] > 0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      float v = 0.f;
      if (m >= M - (K - 1)) {
        const int rel = i - M + m;
        if (rel >= 0) v = to_f32<T>(x[(size_t)(t - M + m) * x_stride + c]);
        else if (has_past) v = state[(size_t)slot * state_stride + (size_t)(K - 1 + rel) * C + c];
      }
      win[m] = v;
    }
  };
  fill(t0);
  const int t_end = min(t0 + tokens_per_block, n_tokens);
  for (int t = t0; t < t_end; ++t) {
    if (t >= next_first) {
      while (s + 1 < n_seqs && cu_q[s + 1] <= t) ++s;
      seq_first = cu_q[s];
      next_first = cu_q[s + 1];
      fill(t);
    }
    const float xt = to_f32<T>(x[(size_t)t * x_stride + c]);
    float ra = 0.f, rb = 0.f;                           // oldest tap first, the current token last, then the input itself
#pragma unroll
    for (int m = 0; m < M; ++m) {
      ra = fmaf(wa[m], win[m], ra);
      rb = fmaf(wb[m], win[m], rb);
    }
#pragma unroll
    for (int m = 0; m + 1 < M; ++m) win[m] = win[m + 1];
    win[M - 1] = xt;
    if (SINGLE && slots[s] >= 0)
#pragma unroll
      for (int j = 0; j < M; ++j)
        if (j < K - 1) state[(size_t)slots[s] * state_stride + (size_t)j * C + c] = keep(win, j, K);
    y1[(size_t)t * y_stride + c] = from_f32<T>(xt + fmaf(wa[M], xt, ra));
    if (y2) y2[(size_t)t * y_stride + c] = from_f32<T>(xt + fmaf(wb[M], xt, rb));
  }
}

// Long steps, up to four taps, channels in steps of 4 on aligned rows: four channels a thread, the inputs of four tokens on
// their way together.  The kernels above fetch 2 bytes a thread and token, one after another, and carry eight taps whatever
// the filter has: 60 us for 4,096 tokens of 4,096 and 2,304 channels (90 MB in the mean; 35 here).  The same operations in the same order, so
// the same bits.  FILTER: filter_add (one or two filters, outputs of x's type), else silu (one, with a bias).
constexpr int SV_TOKENS = 16, SV_TAPS = 4;

__device__ __forceinline__ void sv_load(float (&o)[4], const float* p) {
  const float4 v = *reinterpret_cast<const float4*>(p);
  o[0] = v.x; o[1] = v.y; o[2] = v.z; o[3] = v.w;
}
__device__ __forceinline__ void sv_load(float (&o)[4], const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  o[0] = lo.x; o[1] = lo.y; o[2] = hi.x; o[3] = hi.y;
}
__device__ __forceinline__ void sv_store(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void sv_store(__nv_bfloat16* p, const float (&v)[4]) {
  uint2 raw;
  *reinterpret_cast<__nv_bfloat162*>(&raw.x) = __floats2bfloat162_rn(v[0], v[1]);
  *reinterpret_cast<__nv_bfloat162*>(&raw.y) = __floats2bfloat162_rn(v[2], v[3]);
  *reinterpret_cast<uint2*>(p) = raw;
}

template <typename T, typename TO, bool FILTER>
__global__ void __launch_bounds__(128) short_conv_vec_kernel(
    TO* __restrict__ y1, TO* __restrict__ y2, int y_stride, const T* __restrict__ x, int x_stride, const T* __restrict__ w1,
    const T* __restrict__ w2, const T* __restrict__ bias, const float* __restrict__ state, long state_stride,
    const int* __restrict__ cu_q, const int* __restrict__ q_start, const int* __restrict__ slots, int n_seqs, int n_tokens,
    int C, int K) {
  pdl_prologue();
  const int c = 4 * (blockIdx.y * blockDim.x + threadIdx.x);
  const int t0 = blockIdx.x * SV_TOKENS;
  if (c >= C || t0 >= n_tokens) return;
  constexpr int M = SV_TAPS - 1;
  float wa[SV_TAPS][4], wb[FILTER ? SV_TAPS : 1][4], b[4] = {0.f, 0.f, 0.f, 0.f};       // right-aligned, zeros before
#pragma unroll
  for (int m = 0; m < SV_TAPS; ++m)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = m - (SV_TAPS - K);
      wa[m][e] = k >= 0 ? to_f32<T>(w1[(size_t)(c + e) * K + k]) : 0.f;
      if (FILTER) wb[m][e] = k >= 0 && w2 ? to_f32<T>(w2[(size_t)(c + e) * K + k]) : 0.f;
    }
  if (!FILTER && bias)
#pragma unroll
    for (int e = 0; e < 4; ++e) b[e] = to_f32<T>(bias[c + e]);
  int lo = 0, hi = n_seqs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cu_q[mid] <= t0) lo = mid; else hi = mid - 1;
  }
  int s = lo;
  int seq_first = cu_q[s], next_first = cu_q[s + 1];
  float win[M][4];
  auto fill = [&](int t) {
    const int i = t - seq_first;
    const int slot = slots[s];
    const bool has_past = slot >= 0 && q_start[s] > 0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
#pragma unroll
      for (int e = 0; e < 4; ++e) win[m][e] = 0.f;
      if (m >= M - (K - 1)) {
        const int rel = i - M + m;
        if (rel >= 0) sv_load(win[m], x + (size_t)(t - M + m) * x_stride + c);
        else if (has_past) {
          const float* st = state + (size_t)slot * state_stride + (size_t)(K - 1 + rel) * C + c;
#pragma unroll
          for (int e = 0; e < 4; ++e) win[m][e] = st[e];
        }
      }
    }
  };
  fill(t0);
  const int t_end = min(t0 + SV_TOKENS, n_tokens);
  for (int tb = t0; tb < t_end; tb += 4) {
    float xs[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (tb + u < t_end) sv_load(xs[u], x + (size_t)(tb + u) * x_stride + c);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int t = tb + u;
      if (t >= t_end) break;
      if (t >= next_first) {
        while (s + 1 < n_seqs && cu_q[s + 1] <= t) ++s;
        seq_first = cu_q[s];
        next_first = cu_q[s + 1];
        fill(t);
      }
      float o1[4], o2[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float xt = xs[u][e];
        if (FILTER) {
          float ra = 0.f, rb = 0.f;
#pragma unroll
          for (int m = 0; m < M; ++m) {
            ra = fmaf(wa[m][e], win[m][e], ra);
            rb = fmaf(wb[FILTER ? m : 0][e], win[m][e], rb);
          }
          o1[e] = xt + fmaf(wa[M][e], xt, ra);
          o2[e] = xt + fmaf(wb[FILTER ? M : 0][e], xt, rb);
        } else {
          float acc = fmaf(wa[M][e], xt, b[e]);
#pragma unroll
          for (int m = 0; m < M; ++m) acc = fmaf(wa[m][e], win[m][e], acc);
          o1[e] = acc / (1.0f + expf(-acc));
        }
#pragma unroll
        for (int m = 0; m + 1 < M; ++m) win[m][e] = win[m + 1][e];
        win[M - 1][e] = xt;
      }
      sv_store(y1 + (size_t)t * y_stride + c, o1);
      if (FILTER && y2) sv_store(y2 + (size_t)t * y_stride + c, o2);
    }
  }
}

// Whether a step goes that way.  `item`: bytes of x's elements, `out_item` of the outputs'
static bool sv_takes(int n_tokens, int C, int K, const void* y1, const void* y2, int y_stride, int out_item, const void* x,
                     int x_stride, int item) {
  return n_tokens > 512 && K <= SV_TAPS && C % 4 == 0 && x_stride % 4 == 0 && y_stride % 4 == 0 &&
         (uintptr_t)x % (4 * item) == 0 && (uintptr_t)y1 % (4 * out_item) == 0 && (uintptr_t)y2 % (4 * out_item) == 0;
}

// y1 (and y2) [T, C] rows of y_stride; x [T, C] rows of x_stride; w1 (and w2) [C, K]; all of one type.  The state
// [slots][(K - 1) * C] fp32 is read and then moved on.
NHV_API int nhv_causal_filter_add(int dtype, void* y1, void* y2, int y_stride, const void* x, int x_stride, const void* w1,
                                  const void* w2, float* state, long state_stride, const int* cu_q, const int* q_start,
                                  const int* slots, int n_seqs, int n_tokens, int C, int K, int single, cudaStream_t stream) {
  if (n_tokens == 0 || n_seqs == 0) return 0;
  NHV_REQUIRE(C > 0 && K >= 1 && K <= SC_MAX_TAPS, "causal_filter: %d taps are beyond the supported %d", K, SC_MAX_TAPS);
  NHV_REQUIRE(K == 1 || (state && state_stride >= (long)(K - 1) * C), "causal_filter: the state holds fewer than (taps - 1) * channels floats");
  NHV_REQUIRE(y1 && w1 && (!y2) == (!w2), "causal_filter: a second output comes with a second filter");
  NHV_REQUIRE(!single || n_tokens == n_seqs, "causal_filter: %d requests of one token each do not have %d tokens", n_seqs, n_tokens);
  const int threads = 128;
  const int tokens_per_block = single || n_tokens <= 512 ? 1 : SC_TOKENS;
  dim3 grid((n_tokens + tokens_per_block - 1) / tokens_per_block, (C + threads - 1) / threads);
  dim3 grid2(n_seqs, (C + threads - 1) / threads);
  const int item = dtype == NHV_F32 ? 4 : 2;
  const bool vec = !single && sv_takes(n_tokens, C, K, y1, y2, y_stride, item, x, x_stride, item);
  const dim3 vgrid((n_tokens + SV_TOKENS - 1) / SV_TOKENS, (C / 4 + threads - 1) / threads);
#define LAUNCH(T)                                                                                                  \
  do {                                                                                                             \
    if (vec)                                                                                                       \
      nhv_launch(short_conv_vec_kernel<T, T, true>, vgrid, threads, 0, stream, (T*)y1, (T*)y2, y_stride, (const T*)x, \
                 x_stride, (const T*)w1, (const T*)w2, (const T*)nullptr, (const float*)state, state_stride, cu_q, \
                 q_start, slots, n_seqs, n_tokens, C, K);                                                          \
    else                                                                                                           \
    nhv_launch(single ? filter_add_kernel<T, true> : filter_add_kernel<T, false>, grid, threads, 0, stream, (T*)y1,  \
               (T*)y2, y_stride, (const T*)x, x_stride, (const T*)w1, (const T*)w2, state, state_stride, cu_q,     \
               q_start, slots, n_seqs, n_tokens, C, K, tokens_per_block);                                          \
    if (K > 1 && !single)                                                                                          \
      nhv_launch(short_conv_state_kernel<T>, grid2, threads, 0, stream, (const T*)x, x_stride, state, state_stride, \
                 cu_q, q_start, slots, C, K);                                                                      \
  } while (0)
  if (dtype == NHV_F32) LAUNCH(float);
  else if (dtype == NHV_BF16) LAUNCH(__nv_bfloat16);
  else NHV_REQUIRE(false, "causal_filter: unknown dtype %d", dtype);
#undef LAUNCH
  NHV_CHECK_LAUNCH("causal_filter");
  return 0;
}

// dtype: of x, the filters and the bias; out_dtype: of y (fp32 where a recurrence reads it next)
NHV_API int nhv_short_conv_silu(int dtype, int out_dtype, void* y, int y_stride, const void* x, int x_stride, const void* w,
                                const void* bias, float* state, long state_stride, const int* cu_q,
                                const int* q_start, const int* slots, int n_seqs, int n_tokens, int C, int K,
                                int single, cudaStream_t stream) {
  if (n_tokens == 0 || n_seqs == 0) return 0;
  NHV_REQUIRE(out_dtype == dtype || out_dtype == NHV_F32, "short_conv: the output is of the input's type or fp32");
  NHV_REQUIRE(C > 0 && K >= 1 && K <= SC_MAX_TAPS, "short_conv: %d taps are beyond the supported %d", K, SC_MAX_TAPS);
  NHV_REQUIRE(!single || n_tokens == n_seqs, "short_conv: %d requests of one token each do not have %d tokens", n_seqs, n_tokens);
  NHV_REQUIRE(K == 1 || (state && state_stride >= (long)(K - 1) * C), "short_conv: the state holds fewer than (taps - 1) * channels floats");
  const int threads = 128;
  const int tokens_per_block = single || n_tokens <= 512 ? 1 : SC_TOKENS;
  dim3 grid((n_tokens + tokens_per_block - 1) / tokens_per_block, (C + threads - 1) / threads);
  dim3 grid2(n_seqs, (C + threads - 1) / threads);
  const int item = dtype == NHV_F32 ? 4 : 2;
  const bool vec = !single && sv_takes(n_tokens, C, K, y, nullptr, y_stride, out_dtype == NHV_F32 ? 4 : 2, x, x_stride, item);
  const dim3 vgrid((n_tokens + SV_TOKENS - 1) / SV_TOKENS, (C / 4 + threads - 1) / threads);
#define OUT(T, TO)                                                                                                 \
  if (vec)                                                                                                         \
    nhv_launch(short_conv_vec_kernel<T, TO, false>, vgrid, threads, 0, stream, (TO*)y, (TO*)nullptr, y_stride,     \
               (const T*)x, x_stride, (const T*)w, (const T*)nullptr, (const T*)bias, (const float*)state,         \
               state_stride, cu_q, q_start, slots, n_seqs, n_tokens, C, K);                                        \
  else                                                                                                             \
  nhv_launch(single ? short_conv_silu_kernel<T, TO, true> : short_conv_silu_kernel<T, TO, false>, grid, threads, 0, \
             stream, (TO*)y, y_stride, (const T*)x, x_stride, (const T*)w, (const T*)bias, state, state_stride,    \
             cu_q, q_start, slots, n_seqs, n_tokens, C, K, tokens_per_block)
#define LAUNCH(T)                                                                                                  \
  do {                                                                                                             \
    if (out_dtype == NHV_F32) { OUT(T, float); }                                                                   \
    else { OUT(T, T); }                                                                                            \
    if (K > 1 && !single)                                                                                          \
      nhv_launch(short_conv_state_kernel<T>, grid2, threads, 0, stream, (const T*)x, x_stride, state, state_stride, \
                 cu_q, q_start, slots, C, K);                                                                      \
  } while (0)
  if (dtype == NHV_F32) LAUNCH(float);
  else if (dtype == NHV_BF16) LAUNCH(__nv_bfloat16);
  else NHV_REQUIRE(false, "short_conv: unknown dtype %d", dtype);
#undef LAUNCH
#undef OUT
  NHV_CHECK_LAUNCH("short_conv");
  return 0;
}
