// Recurrences with one decay per head, a chunk of 32 tokens at a time.
//
//   S_t = g_t S_(t-1) + k_t w_t u_t^T,   o_t = S_t^T q_t,   0 <= g_t <= 1
//
// per head, S [d, dv] fp32.  With s0 the state before the chunk, D(i, t) = g_(i+1) .. g_t and gam_t = g_1 .. g_t:
//   o_t = gam_t (s0^T q_t) + sum_{i <= t} P(t, i) u_i,   P(t, i) = D(i, t) w_i (q_t . k_i)
//   s_end = gam_C s0 + sum_i E_i k_i u_i^T,              E_i = D(i, C) w_i
// u_t is the token's value, or for the delta rule (w = 1)
//   u_t = beta_t (v_t - gam_t (s0^T k_t) - sum_{i < t} D(i, t) (k_i . k_t) u_i):   U = T' (V - diag(gam) K s0)
// with T' = (I + A)^-1 diag(beta), A(t, i) = beta_t D(i, t) (k_t . k_i) below the diagonal.  Token by token a recurrence
// is a chain of n rounds of sums over lanes and a write (delta rule, 16 heads of 128 x 128, one request of 4,096 tokens:
// 1,042 us); chunk by chunk the chain is n / 32 rounds of small matrix products.  Those are fp32 on the CUDA cores (fused
// multiply-add, two at a time).  What every chunk is made from, the products q . k and k . k and the decays between
// tokens (running products, never quotients), is summed and multiplied in 64 bits and rounded once to fp32, so that the error
// against 64 bits is no larger than token by token.
//
// Two kernels.  The first has a block per (chunk, q/k head) and no chain: the products q . k and k . k, the decays, the
// inverse.  It leaves per (chunk, head) CS_WORK floats.  The second has a block per (request, head, 16 columns of S) and
// walks the request's chunks; K and Q of the next chunk, and P and T' of this one, arrive by cp.async meanwhile.  It is
// bound by reading shared memory (eight values for sixteen multiply-adds in the largest product) and, between its barriers
// (six a chunk for the delta rule, five for the others), by latency; chunks of 32 tokens let two blocks share an SM, so
// that one computes while the other waits.
// Chunks are numbered over the step: chunk c of request s (first token `first`) is number first / 32 + s + c, which
// leaves no two requests the same number.
#pragma once
#include "nhv_common.cuh"

constexpr int CS_C = 32;                                  // tokens of a chunk
constexpr int CS_COLS = 16;                               // columns of S per block
constexpr int CS_THREADS = 256;
constexpr int CS_PS = CS_C + 4;                           // floats of a row of P, T', V, U in shared memory
// per (chunk, head): P, T' below their diagonals [32][32]; gam, E, the diagonals of P and of T' [32]
constexpr int CS_P = 0, CS_T = CS_C * CS_C, CS_GAM = 2 * CS_C * CS_C, CS_E = CS_GAM + CS_C, CS_PD = CS_E + CS_C,
              CS_TD = CS_PD + CS_C, CS_VECS = 4, CS_WORK = CS_GAM + CS_VECS * CS_C;

static inline long cs_chunks(int n_tokens, int n_seqs) { return (long)n_tokens / CS_C + n_seqs; }

static __device__ __forceinline__ void cs_copy16(float* smem, const float* gmem, bool there) {
  const int bytes = there ? 16 : 0;                       // what is not there arrives as zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem),
               "r"(bytes));
}
static __device__ __forceinline__ void cs_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> static __device__ __forceinline__ void cs_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// 32 rows of d floats (zeros from row cn on and from column d on) into [32][D + 4]
template <int D>
static __device__ __forceinline__ void cs_fetch_rows(float* to, const float* from, long stride, int cn, int d) {
  for (int e = threadIdx.x; e < CS_C * (D / 4); e += CS_THREADS) {
    const int r = e / (D / 4), c = 4 * (e % (D / 4));
    const bool there = r < cn && c < d;
    cs_copy16(to + r * (D + 4) + c, from + (there ? r * stride + c : 0), there);
  }
}

// The request and chunk with this number: false if there is none.
static __device__ __forceinline__ bool cs_find(int number, const int* cu_q, int n_seqs, int& s, int& c, int& first, int& n) {
  int lo = 0, hi = n_seqs - 1;                            // the last request whose chunks start at or before `number`
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (cu_q[mid] / CS_C + mid <= number) lo = mid;
    else hi = mid - 1;
  }
  s = lo;
  first = cu_q[s];
  n = cu_q[s + 1] - first;
  c = number - (first / CS_C + s);
  return c >= 0 && c * CS_C < n;
}

// Products of rows of two tiles [32][D + 4] in shared memory, out[t][i] = a_t . b_i for i <= t (and what else lies in the 8 x 8
// tiles on the diagonal): a warp takes the eight rows from 8 `band` on.  Summed in 64 bits, on the matrix instruction for
// them, and rounded once: every output of a chunk is made from these products, and with 32-bit sums (two chains of D / 2)
// theirs was most of the error of a scan by chunks (state space 1.68e-7 in all, 1.06e-7 by tokens).
template <int D>
static __device__ __forceinline__ void cs_products(float* out, const float* a, const float* b, int band) {
  const int lane = threadIdx.x & 31;
  const float* ar = a + (8 * band + (lane >> 2)) * (D + 4) + (lane & 3);       // element (lane >> 2, lane & 3) of an 8 x 4 tile
  const float* br = b + (lane >> 2) * (D + 4) + (lane & 3);
  double acc[4][2];
#pragma unroll
  for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = 0.0;
#pragma unroll 4
  for (int k = 0; k < D; k += 4) {
    const double av = ar[k];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j <= band) {
        const double bv = br[8 * j * (D + 4) + k];
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
            : "+d"(acc[j][0]), "+d"(acc[j][1])
            : "d"(av), "d"(bv));
      }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j <= band)
      *reinterpret_cast<float2*>(out + (8 * band + (lane >> 2)) * CS_PS + 8 * j + 2 * (lane & 3)) =
          make_float2((float)acc[j][0], (float)acc[j][1]);
}

// Sums of 32 rows times 16 columns over 4 K4 elements (contiguous in both, in shared memory) by a warp: a lane's rows
// (lane >> 2) + 8 i, columns (lane & 3) + 4 j, i, j < 4.
template <int K4>
static __device__ __forceinline__ void cs_rows_by_cols(float out[4][4], const float* rows, int row_stride, const float* cols,
                                                       int col_stride) {
  const int lane = threadIdx.x & 31;
  const float* rp = rows + (lane >> 2) * row_stride;
  const float* cp = cols + (lane & 3) * col_stride;
  f32x2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll 4
  for (int k = 0; k < K4; ++k) {
    ulonglong2 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(rp + 8 * i * row_stride + 4 * k);
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(cp + 4 * j * col_stride + 4 * k);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] = f2_fma(a[i].x, b[j].x, acc[i][j]);
        acc[i][j] = f2_fma(a[i].y, b[j].y, acc[i][j]);
      }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float even, odd;
      f2_unpack(acc[i][j], even, odd);
      out[i][j] = even + odd;
    }
}

// out += the same for 4 rows of a matrix [32][CS_PS] with zeros on and above its diagonal and 16 columns per warp (warp w:
// rows 4 w to 4 w + 3; row lane >> 3, columns (lane & 7) + 8 j, j < 2), then += diagonal[row] times the row's own token, most
// of the sum: last, in one rounding.  A value that is no number would reach the rows before its own through the zeros:
// MASKED leaves out what a row may not see, for chunks that hold such a value (selects in all chunks cost up to 10 % of a scan).
template <bool MASKED>
static __device__ __forceinline__ void cs_triangle(float out[2], const float* rows, const float* cols, const float* diagonal,
                                                   int warp) {
  const int lane = threadIdx.x & 31, row = lane >> 3;
  const float* rp = rows + (4 * warp + row) * CS_PS;
  const float* cp = cols + (lane & 7) * CS_PS;
  f32x2 acc[2][2] = {{0ull, 0ull}, {0ull, 0ull}};
#pragma unroll 4
  for (int k = 0; k <= warp; ++k) {
    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(rp + 4 * k);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      ulonglong2 b = *reinterpret_cast<const ulonglong2*>(cp + 8 * j * CS_PS + 4 * k);
      if (MASKED && k == warp) {
        b.x &= row > 1 ? ~0ull : row > 0 ? 0xffffffffull : 0ull;
        b.y &= row > 2 ? 0xffffffffull : 0ull;
      }
      acc[j][0] = f2_fma(a.x, b.x, acc[j][0]);
      acc[j][1] = f2_fma(a.y, b.y, acc[j][1]);
    }
  }
  const float d = diagonal[4 * warp + row];
#pragma unroll
  for (int j = 0; j < 2; ++j) out[j] = fmaf(d, cp[8 * j * CS_PS + 4 * warp + row], out[j] + f2_sum(acc[j][0], acc[j][1]));
}
static __device__ __forceinline__ bool cs_no_number(float v) { return !(fabsf(v) < INFINITY); }

// What kind of recurrence the second kernel walks
enum CsKind { CS_DELTA, CS_PLAIN, CS_NORMED };           // u from T'; u = v; u = v and o divided by its normaliser

struct CsPairs {
  const float *q, *k;                // row t, q/k head g: at t * qk_stride + g * d
  long qk_stride;
  float* work;                       // [chunks][H][CS_WORK]
  float* extra;                      // CS_NORMED: [chunks][H][2 * 32 + d]: sums of a row of P, exp(-m) per token, sum of E k
  const int *cu_q, *slots;
  int n_seqs, G, H, d;
};

template <int D, int KIND>
constexpr int cs_pairs_smem_floats() {
  return 2 * CS_C * (D + 4) + (KIND == CS_DELTA ? 3 : 1) * CS_C * CS_PS + 4 * CS_C;
}

// Gates: decay, weight and what else a kind needs of token t (of the packed step) and head h
template <int D, int KIND, typename Gates>
__global__ void __launch_bounds__(CS_THREADS) chunk_pairs_kernel(const CsPairs p, const Gates gates) {
  constexpr bool DELTA = KIND == CS_DELTA, NORMED = KIND == CS_NORMED;
  extern __shared__ __align__(16) float smem[];
  float* Ks = smem;                                       // [32][D + 4]
  float* Qs = Ks + CS_C * (D + 4);
  float* QK = Qs + CS_C * (D + 4);                        // [32][CS_PS]
  float* KK = QK + CS_C * CS_PS;                          // DELTA: the same of k . k, then A
  float* As = KK + (DELTA ? CS_C * CS_PS : 0);
  double* gd = reinterpret_cast<double*>(As + (DELTA ? CS_C * CS_PS : 0));     // decay of the token
  float* ws = reinterpret_cast<float*>(gd + CS_C);        // weight of the token (DELTA: beta)
  float* Es = ws + CS_C;
  pdl_wait();                                             // (the scan behind it takes whole SMs: it is let in at the end)
  int s, c, first, n;
  if (!cs_find(blockIdx.x, p.cu_q, p.n_seqs, s, c, first, n) || p.slots[s] < 0) return;
  const int tid = threadIdx.x, g = blockIdx.y, t0 = first + c * CS_C, cn = min(CS_C, n - c * CS_C);
  cs_fetch_rows<D>(Ks, p.k + (size_t)t0 * p.qk_stride + (size_t)g * p.d, p.qk_stride, cn, p.d);
  cs_fetch_rows<D>(Qs, p.q + (size_t)t0 * p.qk_stride + (size_t)g * p.d, p.qk_stride, cn, p.d);
  cs_commit();
  cs_wait<0>();
  __syncthreads();
  // (a band of eight rows has one to four tiles: warps that share a quarter of the SM have five between them)
  const int warp = tid >> 5;
  if (warp < 4) cs_products<D>(QK, Qs, Ks, warp);
  else if (DELTA) cs_products<D>(KK, Ks, Ks, 7 - warp);

  const int per = p.H / p.G, share = (per + gridDim.z - 1) / gridDim.z;       // heads of the group, of this block
  const int h_end = min((int)(blockIdx.z + 1) * share, per) + g * per;
  for (int h = g * per + blockIdx.z * share; h < h_end; ++h) {
    float* out = p.work + ((size_t)blockIdx.x * p.H + h) * CS_WORK;
    float* ex = NORMED ? p.extra + ((size_t)blockIdx.x * p.H + h) * (2 * CS_C + p.d) : nullptr;
    __syncthreads();
    if (tid < CS_C) {
      float gate = 1.f, weight = 0.f, em = 0.f;           // behind the last token: nothing is added, nothing decays
      if (tid < cn) gates(t0 + tid, h, gate, weight, em);
      gd[tid] = gate;
      ws[tid] = weight;
      if (NORMED) ex[CS_C + tid] = em;
    }
    __syncthreads();
    {
      const int i = tid & 31, ta = 4 * (tid >> 5);        // a column of the triangle, four of its rows
      // (products of 64 bits, rounded once: where states last, those of 32 bits were most of what was left of the error)
      double dec = 1.0;                                   // g_(i+1) .. g_t
      for (int t = i + 1; t < ta; ++t) dec *= gd[t];
      const double wi = DELTA ? 1.0 : (double)ws[i];
#pragma unroll
      for (int t = ta; t < ta + 4; ++t) {
        if (t > i) dec *= gd[t];
        const float pv = t >= i ? (float)(dec * wi * QK[t * CS_PS + i]) : 0.f;
        out[CS_P + t * CS_C + i] = t > i ? pv : 0.f;
        if (t == i) out[CS_PD + t] = pv;
        if (DELTA) As[t * CS_PS + i] = t > i ? (float)(dec * ws[t] * KK[t * CS_PS + i]) : 0.f;
        if (i == 0) out[CS_GAM + t] = (float)(gd[0] * dec);
        if (NORMED) {
          const float sum = warp_sum(pv);
          if (i == 0) ex[t] = sum;
        }
      }
      if (ta == CS_C - 4) {
        const float e = (float)(dec * wi);
        out[CS_E + i] = e;
        if (NORMED) Es[i] = e;
      }
    }
    __syncthreads();
    if (NORMED) {
      if (tid < p.d) {
        float sum = 0.f;
        for (int t = 0; t < cn; ++t) sum = fmaf(Es[t], Ks[t * (D + 4) + tid], sum);
        ex[2 * CS_C + tid] = sum;
      }
    }
    if (DELTA) {
      if (tid < CS_C) {                                   // (I + A)^-1, a column a thread
        float x[CS_C];
#pragma unroll
        for (int t = 0; t < CS_C; ++t) {
          float sum[4] = {t == tid ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int i = 0; i < t; ++i) sum[i & 3] = fmaf(-As[t * CS_PS + i], x[i], sum[i & 3]);
          x[t] = (sum[0] + sum[1]) + (sum[2] + sum[3]);
          out[CS_T + t * CS_C + tid] = t > tid ? x[t] * ws[tid] : 0.f;
        }
        out[CS_TD + tid] = ws[tid];                       // the inverse has ones there
      }
    }
  }
}

template <int D, int KIND, typename Gates>
static cudaError_t cs_launch_pairs(const CsPairs& p, const Gates& gates, int n_tokens, cudaStream_t stream) {
  constexpr int smem = cs_pairs_smem_floats<D, KIND>() * 4;
  auto kernel = chunk_pairs_kernel<D, KIND, Gates>;
  static std::atomic<uint64_t> done{0};
  const cudaError_t e = nhv_allow_smem((const void*)kernel, smem, done);
  if (e != cudaSuccess) return e;
  // many heads on one product of q and k: several blocks compute it, each for four of them
  const int per = p.H / p.G;
  return nhv_launch(kernel, dim3((unsigned)cs_chunks(n_tokens, p.n_seqs), p.G, (per + 3) / 4), CS_THREADS, smem, stream, p, gates);
}

struct CsScan {
  float* y;                          // [T, H * dv] fp32
  const float *q, *k;                // row t, q/k head g: at t * qk_stride + g * d
  long qk_stride;
  const void* v;                     // row t, head h: at t * v_stride + h * dv, of the kernel's type TV
  long v_stride;
  const float* work;                 // [chunks][H][CS_WORK]
  const float* skip;                 // CS_PLAIN: y gets skip[h] * v besides, if given
  const float* extra;                // CS_NORMED: what chunk_pairs_kernel left there
  const float* top;                  // CS_NORMED: [T][H] the running maximum, whose last value the state keeps
  float* state;
  long state_stride;
  const int *cu_q, *q_start, *slots;
  int G, H, d, dv;
};

constexpr int CS_PARTIAL = 8 * 32 * 20;                  // rows of 20 floats, 32 a warp, for partial sums

template <int D, int KIND>
constexpr int cs_smem_floats() {
  return CS_COLS * (D + 4) + 4 * CS_C * (D + 4) + (KIND == CS_DELTA ? 2 : 1) * CS_C * CS_PS + 2 * CS_COLS * CS_PS +
         2 * CS_VECS * CS_C + CS_PARTIAL + CS_C * 20 + (KIND == CS_NORMED ? D + 2 * (2 * CS_C) + CS_C : 0);
}

static __device__ __forceinline__ float4 cs_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
static __device__ __forceinline__ float4 cs_load4(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}

template <int D, int KIND, typename TV>
__global__ void __launch_bounds__(CS_THREADS, 2) chunk_scan_kernel(const CsScan p) {
  constexpr bool DELTA = KIND == CS_DELTA, NORMED = KIND == CS_NORMED;
  constexpr int RS = D + 4;
  constexpr int GROUPS = DELTA ? 2 : 1, SPLIT = 8 / GROUPS;         // the 32 rows of K and those of Q (Q alone); warps that share them
  extern __shared__ __align__(16) float smem[];
  float* Ss = smem;                                       // [16 columns][RS]
  float* KQ = Ss + CS_COLS * RS;                          // [2 stages][K, Q][32][RS]
  float* Ps = KQ + 4 * CS_C * RS;                         // [32][CS_PS]
  float* Ts = Ps + CS_C * CS_PS;                          // DELTA: [32][CS_PS]
  float* Rs = Ts + (DELTA ? CS_C * CS_PS : 0);            // [16 columns][CS_PS]: V, for DELTA then V - diag(gam) K s0
  float* Us = Rs + CS_COLS * CS_PS;                       // DELTA: [16 columns][CS_PS]
  float* Vec = Us + CS_COLS * CS_PS;                      // [2 stages][gam, E, P's diagonal, T' 's][32]
  float* Xs = Vec + 2 * CS_VECS * CS_C;                   // partial sums
  float* Os = Xs + CS_PARTIAL;       // [32][20]: diag(gam) Q s0
  float* Ns = Os + CS_C * 20;                             // NORMED: [D] n, [2 stages][sum of P's row, exp(-m)][32], [32] the division
  pdl_wait();
  const int s = blockIdx.x, h = blockIdx.y, cb = blockIdx.z, col0 = cb * CS_COLS;
  const int g = h / (p.H / p.G), d = p.d, dv = p.dv;
  const int first = p.cu_q[s], n = p.cu_q[s + 1] - first, slot = p.slots[s];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ncol = min(CS_COLS, dv - col0);               // a multiple of 4
  float* yb = p.y + (size_t)first * p.H * dv + (size_t)h * dv + col0;
  if (slot < 0) {
    for (int i = tid; i < n * ncol; i += CS_THREADS) yb[(size_t)(i / ncol) * p.H * dv + i % ncol] = 0.f;
    return;
  }
  if (n <= 0) return;
  const bool fresh = p.q_start[s] == 0;
  float* base = p.state + (size_t)slot * p.state_stride;
  float* st = base + ((size_t)h * dv + col0) * d;
  float* nm = NORMED ? base + (size_t)p.H * dv * d + ((size_t)h * gridDim.z + cb) * (d + 1) : nullptr;
  const float* qb = p.q + (size_t)first * p.qk_stride + (size_t)g * d;
  const float* kb = p.k + (size_t)first * p.qk_stride + (size_t)g * d;
  const TV* vb = (const TV*)p.v + (size_t)first * p.v_stride + (size_t)h * dv + col0;
  const long number0 = first / CS_C + s;
  const int n_chunks = (n + CS_C - 1) / CS_C;

  auto work_of = [&](int c) { return p.work + ((number0 + c) * p.H + h) * CS_WORK; };
  auto fetch_kq = [&](int c) {                            // K, Q and the vectors of chunk c
    const int cn = min(CS_C, n - c * CS_C), stage = c & 1;
    cs_fetch_rows<D>(KQ + (2 * stage) * CS_C * RS, kb + (size_t)c * CS_C * p.qk_stride, p.qk_stride, cn, d);
    cs_fetch_rows<D>(KQ + (2 * stage + 1) * CS_C * RS, qb + (size_t)c * CS_C * p.qk_stride, p.qk_stride, cn, d);
    if (tid < (DELTA ? 4 : 3) * CS_C / 4) cs_copy16(Vec + stage * CS_VECS * CS_C + 4 * tid, work_of(c) + CS_GAM + 4 * tid, true);
    if (NORMED && tid < 2 * CS_C / 4)
      cs_copy16(Ns + D + stage * 2 * CS_C + 4 * tid, p.extra + ((number0 + c) * p.H + h) * (2 * CS_C + d) + 4 * tid, true);
  };
  auto fetch_pt = [&](int c) {
    const float* w = work_of(c);
    for (int e = tid; e < CS_C * CS_C / 4; e += CS_THREADS) {
      const int r = e / (CS_C / 4), k = 4 * (e % (CS_C / 4));
      cs_copy16(Ps + r * CS_PS + k, w + CS_P + r * CS_C + k, true);
      if (DELTA) cs_copy16(Ts + r * CS_PS + k, w + CS_T + r * CS_C + k, true);
    }
  };
  const int vt = (tid >> 2) & (CS_C - 1), vc = 4 * (tid & 3);       // the four values of a chunk that this thread brings in
  auto load_v = [&](int c) {
    const int t = c * CS_C + vt;
    return tid < 4 * CS_C && t < n && vc < ncol ? cs_load4(vb + (size_t)t * p.v_stride + vc) : make_float4(0.f, 0.f, 0.f, 0.f);
  };

  fetch_kq(0);
  cs_commit();
  const bool st_vec = ((uintptr_t)st % 16) == 0;
  for (int e = tid; e < CS_COLS * (D / 4); e += CS_THREADS) {
    const int c = e / (D / 4), i = 4 * (e % (D / 4));
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!fresh && c < ncol && i < d) {
      const float* at = st + (size_t)c * d + i;
      v = st_vec ? *reinterpret_cast<const float4*>(at) : make_float4(at[0], at[1], at[2], at[3]);
    }
    *reinterpret_cast<float4*>(Ss + c * RS + i) = v;
  }
  if (NORMED)
    for (int i = tid; i < D; i += CS_THREADS) Ns[i] = !fresh && i < d ? nm[i] : 0.f;
  const float skip = KIND == CS_PLAIN && p.skip ? p.skip[h] : 0.f;
  float4 v_next = load_v(0);
  // the part of the state that this thread moves on: four rows, four columns, its share of the tokens
  constexpr int QUADS = D / 4, TGROUPS = CS_THREADS / (QUADS * 4);
  const int quad = tid % QUADS, cg = (tid / QUADS) % 4, tg = tid / (QUADS * 4);

  for (int c = 0; c < n_chunks; ++c) {
    const int stage = c & 1, cn = min(CS_C, n - c * CS_C);
    const float* Ks = KQ + (2 * stage) * CS_C * RS;
    const float *gam = Vec + stage * CS_VECS * CS_C, *E = gam + CS_C, *Pd = E + CS_C, *Td = Pd + CS_C;
    cs_wait<0>();
    // whether the chunk holds a value that is no number (DELTA: asked of V - diag(gam) K s0 and of U, below)
    bool odd = !DELTA && (cs_no_number(v_next.x) || cs_no_number(v_next.y) || cs_no_number(v_next.z) || cs_no_number(v_next.w));
    if (tid < 4 * CS_C) {
      Rs[(vc + 0) * CS_PS + vt] = v_next.x; Rs[(vc + 1) * CS_PS + vt] = v_next.y;
      Rs[(vc + 2) * CS_PS + vt] = v_next.z; Rs[(vc + 3) * CS_PS + vt] = v_next.w;
    }
    if (DELTA) __syncthreads();
    else odd = __syncthreads_or(odd);
    fetch_pt(c);
    cs_commit();
    if (c + 1 < n_chunks) {
      fetch_kq(c + 1);
      v_next = load_v(c + 1);
    }
    cs_commit();

    // K s0 and Q s0 (Q s0 alone), each sum split over SPLIT warps
    {
      const int group = warp % GROUPS, part = warp / GROUPS;
      const float* rows = (DELTA ? Ks : Ks + CS_C * RS) + group * 32 * RS + part * (D / SPLIT);
      float x[4][4];
      cs_rows_by_cols<D / SPLIT / 4>(x, rows, RS, Ss + part * (D / SPLIT), RS);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) Xs[(part * 32 * GROUPS + group * 32 + (lane >> 2) + 8 * i) * 20 + (lane & 3) + 4 * j] = x[i][j];
      if (NORMED) {                                       // q . n0 and the division, four tokens a warp
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int t = warp * 4 + i;
          const float* qr = Ks + (CS_C + t) * RS;
          float dot = 0.f;
          for (int e = lane; e < D; e += 32) dot = fmaf(qr[e], Ns[e], dot);
          dot = warp_sum(dot);
          const float* ex = Ns + D + stage * 2 * CS_C;
          if (lane == 0) Ns[D + 4 * CS_C + t] = fmaxf(fabsf(gam[t] * dot + ex[t]), ex[CS_C + t]) + 1e-6f;
        }
      }
      cs_wait<1>();                                       // P and T' are there
      __syncthreads();
#pragma unroll
      for (int e = tid; e < 32 * GROUPS * CS_COLS; e += CS_THREADS) {
        const int r = e / CS_COLS, col = e % CS_COLS, t = r % CS_C;
        float sum = 0.f;
#pragma unroll
        for (int o = 0; o < SPLIT; ++o) sum += Xs[(o * 32 * GROUPS + r) * 20 + col];
        if (DELTA && r < CS_C) {
          const float v = Rs[col * CS_PS + t] - gam[t] * sum;
          odd |= cs_no_number(v);
          Rs[col * CS_PS + t] = v;
        } else {
          Os[t * 20 + col] = gam[t] * sum;
        }
      }
      if (DELTA) odd = __syncthreads_or(odd);
      else __syncthreads();
    }
    const float* U = Rs;
    if (DELTA) {
      float u[2] = {0.f, 0.f};
      if (warp * 4 < cn) {
        if (odd) cs_triangle<true>(u, Ts, Rs, Td, warp);
        else cs_triangle<false>(u, Ts, Rs, Td, warp);
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) Us[((lane & 7) + 8 * j) * CS_PS + warp * 4 + (lane >> 3)] = u[j];
      U = Us;
      odd = __syncthreads_or(cs_no_number(u[0]) || cs_no_number(u[1]));
    }
    if (warp * 4 < cn) {
      const int t = warp * 4 + (lane >> 3);
      float o[2] = {Os[t * 20 + (lane & 7)], Os[t * 20 + (lane & 7) + 8]};
      if (odd) cs_triangle<true>(o, Ps, U, Pd, warp);
      else cs_triangle<false>(o, Ps, U, Pd, warp);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int col = (lane & 7) + 8 * j;
        float out = o[j];
        if (KIND == CS_PLAIN) out = fmaf(skip, U[col * CS_PS + t], out);
        if (NORMED) out /= Ns[D + 4 * CS_C + t];
        if (t < cn && col < ncol) yb[(size_t)(c * CS_C + t) * p.H * dv + col] = out;
      }
    }
    // s_end = gam_C s0 + sum_t E_t k_t u_t^T
    {
      f32x2 acc[4][2];
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = 0ull;
      const int t0 = tg * (CS_C / TGROUPS), t1 = min(t0 + CS_C / TGROUPS, (cn + 3) & ~3);
#pragma unroll 2
      for (int t = t0; t < t1; t += 4) {
        const float4 e4 = *reinterpret_cast<const float4*>(E + t);
        const float ee[4] = {e4.x, e4.y, e4.z, e4.w};
        ulonglong2 k4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) k4[i] = *reinterpret_cast<const ulonglong2*>(Ks + (t + i) * RS + 4 * quad);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 u4 = *reinterpret_cast<const float4*>(U + (4 * cg + j) * CS_PS + t);
          const float uu[4] = {u4.x, u4.y, u4.z, u4.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float w = ee[i] * uu[i];
            const f32x2 ww = f2_pack(w, w);
            acc[j][0] = f2_fma(k4[i].x, ww, acc[j][0]);
            acc[j][1] = f2_fma(k4[i].y, ww, acc[j][1]);
          }
        }
      }
      // the groups of tokens after the first leave their sums in Xs (read last before the barrier above)
      if (TGROUPS > 1 && tg > 0)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          *reinterpret_cast<ulonglong2*>(Xs + (((tg - 1) * 4 + cg) * 4 + j) * D + 4 * quad) = make_ulonglong2(acc[j][0], acc[j][1]);
      if (NORMED && tid < D && tid < d) {
        const float add = p.extra[((number0 + c) * p.H + h) * (2 * CS_C + d) + 2 * CS_C + tid];
        Ns[tid] = fmaf(gam[CS_C - 1], Ns[tid], add);
      }
      if (TGROUPS > 1) __syncthreads();
      if (tg == 0) {
        const float keep = gam[CS_C - 1];
        const f32x2 kk = f2_pack(keep, keep);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          ulonglong2* at = reinterpret_cast<ulonglong2*>(Ss + (4 * cg + j) * RS + 4 * quad);
          const f32x2 one = f2_pack(1.f, 1.f);
#pragma unroll
          for (int o = 1; o < TGROUPS; ++o) {
            const ulonglong2 more = *reinterpret_cast<const ulonglong2*>(Xs + (((o - 1) * 4 + cg) * 4 + j) * D + 4 * quad);
            acc[j][0] = f2_fma(more.x, one, acc[j][0]);
            acc[j][1] = f2_fma(more.y, one, acc[j][1]);
          }
          const ulonglong2 old = *at;
          *at = make_ulonglong2(f2_fma(old.x, kk, acc[j][0]), f2_fma(old.y, kk, acc[j][1]));
        }
      }
    }
    __syncthreads();                                      // S, Rs, Us, Xs, Ps are free for the next chunk
  }
  pdl_launch_dependents();
  for (int e = tid; e < ncol * (D / 4); e += CS_THREADS) {
    const int c = e / (D / 4), i = 4 * (e % (D / 4));
    if (i >= d) continue;
    const float4 v = *reinterpret_cast<const float4*>(Ss + c * RS + i);
    float* at = st + (size_t)c * d + i;
    if (st_vec) *reinterpret_cast<float4*>(at) = v;
    else { at[0] = v.x; at[1] = v.y; at[2] = v.z; at[3] = v.w; }
  }
  if (NORMED)
    for (int i = tid; i <= d; i += CS_THREADS) nm[i] = i < d ? Ns[i] : p.top[(size_t)(first + n - 1) * p.H + h];
}

template <int D, int KIND, typename TV>
static cudaError_t cs_launch_scan(const CsScan& p, int n_seqs, cudaStream_t stream) {
  constexpr int smem = cs_smem_floats<D, KIND>() * 4;
  static_assert(smem <= 115712, "two blocks an SM");
  static std::atomic<uint64_t> done{0};
  const cudaError_t e = nhv_allow_smem((const void*)chunk_scan_kernel<D, KIND, TV>, smem, done);
  if (e != cudaSuccess) return e;
  return nhv_launch(chunk_scan_kernel<D, KIND, TV>, dim3(n_seqs, p.H, (p.dv + CS_COLS - 1) / CS_COLS), CS_THREADS, smem, stream, p);
}
