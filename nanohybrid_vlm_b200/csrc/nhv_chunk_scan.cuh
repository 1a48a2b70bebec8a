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
// 1,042 us); chunk by chunk the chain is n / 32 rounds of small matrix products.  What every chunk is made from, the products
// q . k and k . k and the decays between tokens (running products, never quotients), is summed and multiplied in 64 bits and
// rounded once to fp32, so that the error against 64 bits is no larger than token by token.
//
// The chain's products run on the tensor cores (mma.sync).  All operands are fp32: each is cut into three bfloat16 of eight
// bits, which hold it exactly, and a product is the six products of their parts down to 2^-16 of the largest; what is left
// out is below 2^-24, half a unit of fp32's last place.  The products of the two first parts have sums of their own, apart
// from the small ones (CS_CUT_OFF).
//
// Two kernels.  The first has a block per (chunk, q/k head) and no chain: the products q . k and k . k, the decays, the
// inverse; it leaves all operands cut, in the order in which the second one's shared memory and registers take them: per
// (chunk, q/k head) K and Q (cs_image_floats), per (chunk, head) P and T' (CS_WORK).  The second has a group of warps per
// (request, head, 16 columns of S) and walks the request's chunks, the next one on its way by cp.async.
//
// Everything in it is transposed, the 16 columns of S and of the values on the M axis: then the fragments in which a warp holds
// a result are those in which the next product takes it.  S^T [16 x d] stays in registers over all chunks, 16 rows of S in
// each warp; what these parts add up to goes through shared memory, lane by lane as it lies, and so does what four of the
// warps make of the values of eight tokens each, and four of the outputs.  (tcgen05 would want 64 to 128 rows of M, both operands of one product from
// shared memory and a trip through tensor memory between the products of the chain.)
//
// What bounds it, one long request: per chunk and SM 1,344 cycles of mma.sync (8 a product and quarter of the SM), some 2,000 of
// reading and writing shared memory, and the latencies of the chain S -> K S -> U -> S with four barriers (two where U is the
// value), 3,800 in all.  Fp32 multiply-adds on the CUDA cores with six barriers a chunk took 7,000.  In us, one request of
// 4,096 tokens with heads of 128 rows and 2,048 columns in all, before and now: delta rule 485 and 262, state space 340
// and 184, mLSTM 500 and 264 (both kernels and what prepares them: 531 and 317, 368 and 214, 575 and 330).  Not faster: four
// warps with 32 rows each (262); the outputs a chunk later, beside the next K S (279); operands cut in the chain itself (505).
// Chunks are numbered over the step: chunk c of request s (first token `first`) is number first / 32 + s + c, which
// leaves no two requests the same number.
#pragma once
#include "nhv_common.cuh"

constexpr int CS_C = 32;                                  // tokens of a chunk
constexpr int CS_COLS = 16;                               // columns of S per group of warps
constexpr int CS_THREADS = 256;                           // of the first kernel
constexpr int CS_PS = CS_C + 4;                           // floats of a row of 32 in shared memory
// per (chunk, head): gam, E, the diagonals of P and of T' [32]; P, T' below their diagonals, cut: the right operand of a product
// over 32 tokens with 8 tokens' outputs, [4 tiles of outputs][3 parts][32 lanes][4 registers]
constexpr int CS_GAM = 0, CS_E = CS_C, CS_PD = 2 * CS_C, CS_TD = 3 * CS_C, CS_VECS = 4, CS_P = CS_VECS * CS_C,
              CS_TRI = 4 * 3 * 32 * 4, CS_T = CS_P + CS_TRI, CS_WORK = CS_T + CS_TRI;
// per (chunk, q/k head), in floats: K and Q [3 parts][32 tokens][D] bfloat16, the pieces of 16 bytes of a row in the order
// piece ^ (row & 7), so that the rows of a column of pieces lie in different banks
constexpr int cs_image_floats(int D) { return 2 * 3 * CS_C * D / 2; }
static inline int cs_width(int d) { return d <= 64 ? 64 : 128; }             // D for heads of d rows
// floats of the scratch of a step (the images of all chunks come first)
static inline long cs_floats(long chunks, int G, int H, int d) {
  return chunks * ((long)G * cs_image_floats(cs_width(d)) + (long)H * CS_WORK);
}

static inline long cs_chunks(int n_tokens, int n_seqs) { return (long)n_tokens / CS_C + n_seqs; }

static __device__ __forceinline__ void cs_copy16(float* smem, const float* gmem, bool there) {
  const int bytes = there ? 16 : 0;                       // what is not there arrives as zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem),
               "r"(bytes));
}
static __device__ __forceinline__ void cs_copy16_all(float* smem, const float* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
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

// Two floats as the three bfloat16 each that they consist of: what is left, rounded to eight bits, three times.  Exact (to the
// nearest: cut off, the parts would all have the value's sign, and what the products leave out would add up) from 7.7e-34 on; above
// bfloat16's largest number, 3.39e38, the first part is that; infinities turn into values that are no number.
struct CsParts { uint32_t part[3]; };
static __device__ __forceinline__ CsParts cs_cut(float x, float y) {
  CsParts c;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    if (i == 0) asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;\n" : "=r"(c.part[i]) : "f"(y), "f"(x));
    else asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(c.part[i]) : "f"(y), "f"(x));
    x -= __uint_as_float(c.part[i] << 16);
    y -= __uint_as_float(c.part[i] & 0xffff0000u);
  }
  return c;
}
static __device__ __forceinline__ float cs_half(uint32_t pair, int which) {
  return __uint_as_float(which ? pair & 0xffff0000u : pair << 16);
}
// Where M(t, i) of a cut triangle lies: the register of part 0 (the others 32 lanes of four registers on), its half i & 1
static __device__ __forceinline__ int cs_tri_at(int t, int i) {
  return (((t >> 3) * 3) * 32 + (t & 7) * 4 + ((i & 7) >> 1)) * 4 + (i >> 4) * 2 + ((i >> 3) & 1);
}
static __device__ __forceinline__ bool cs_no_number(float v) { return !(fabsf(v) < INFINITY); }

// What kind of recurrence the second kernel walks
enum CsKind { CS_DELTA, CS_PLAIN, CS_NORMED };           // u from T'; u = v; u = v and o divided by its normaliser

struct CsPairs {
  const float *q, *k;                // row t, q/k head g: at t * qk_stride + g * d
  long qk_stride;
  float* images;                     // [chunks][G][cs_image_floats(D)]
  float* work;                       // [chunks][H][CS_WORK]
  float* extra;                      // CS_NORMED: [chunks][H][2 * 32 + d]: sums of a row of P, exp(-m) per token, sum of E k
  const int *cu_q, *slots;
  int n_seqs, G, H, d;
};

template <int D, int KIND>
constexpr int cs_pairs_smem_floats() {
  return 2 * CS_C * (D + 4) + (KIND == CS_DELTA ? 4 : 2) * CS_C * CS_PS + 4 * CS_C;
}

// A triangle [32][CS_PS] in shared memory, cut, by 128 threads: each the four registers of a lane, three times
static __device__ __forceinline__ void cs_store_triangle(float* M, const float* from, int thread) {
  const int tile = thread >> 5, lane = thread & 31;
  const float* row = from + (8 * tile + (lane >> 2)) * CS_PS + 2 * (lane & 3);
  CsParts c[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 v = *reinterpret_cast<const float2*>(row + 8 * i);
    c[i] = cs_cut(v.x, v.y);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
    reinterpret_cast<uint4*>(M)[(tile * 3 + i) * 32 + lane] = make_uint4(c[0].part[i], c[1].part[i], c[2].part[i], c[3].part[i]);
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
  float* Ms = Es + CS_C;                                  // [32][CS_PS]: P
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
  if (blockIdx.z == 0) {                                  // K and Q, cut
    uint4* image = reinterpret_cast<uint4*>(p.images + ((size_t)blockIdx.x * p.G + g) * cs_image_floats(D));
    constexpr int PIECES = D / 8;                         // of a row
    for (int e = tid; e < 2 * CS_C * PIECES; e += CS_THREADS) {
      const int which = e / (CS_C * PIECES), r = e / PIECES % CS_C, piece = e % PIECES;
      const float* at = (which ? Qs : Ks) + r * (D + 4) + 8 * piece;
      const float4 lo = *reinterpret_cast<const float4*>(at), hi = *reinterpret_cast<const float4*>(at + 4);
      const CsParts c[4] = {cs_cut(lo.x, lo.y), cs_cut(lo.z, lo.w), cs_cut(hi.x, hi.y), cs_cut(hi.z, hi.w)};
#pragma unroll
      for (int i = 0; i < 3; ++i)
        image[((which * 3 + i) * CS_C + r) * PIECES + (piece ^ (r & 7))] = make_uint4(c[0].part[i], c[1].part[i], c[2].part[i], c[3].part[i]);
    }
  }

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
        Ms[t * CS_PS + i] = t > i ? pv : 0.f;
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
        }
        __syncwarp();                                     // (no other warp reads A)
#pragma unroll
        for (int t = 0; t < CS_C; ++t) As[t * CS_PS + tid] = t > tid ? x[t] * ws[tid] : 0.f;
        out[CS_TD + tid] = ws[tid];                       // the inverse has ones there
      }
      __syncthreads();
    }
    if (tid < 128) cs_store_triangle(out + CS_P, Ms, tid);
    else if (DELTA) cs_store_triangle(out + CS_T, As, tid - 128);
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
  const void* v;                     // row t, head h: at t * v_stride + h * dv, of the kernel's type TV
  long v_stride;
  const float* images;               // [chunks][G][cs_image_floats(D)]
  const float* work;                 // [chunks][H][CS_WORK]
  const float* skip;                 // CS_PLAIN: y gets skip[h] * v besides, if given
  const float* extra;                // CS_NORMED: what chunk_pairs_kernel left there
  const float* top;                  // CS_NORMED: [T][H] the running maximum, whose last value the state keeps
  float* state;
  long state_stride;
  const int *cu_q, *q_start, *slots;
  int G, H, d, dv;
};

// The tensor cores cut off what lies below a sum's last place instead of rounding it, which makes a sum smaller by this part of
// itself on the mean; it is given back.  (Half a unit of the last place would be 4.3e-8; measured, as the part with which the
// error against 64 bits of no recurrence, head size or decay is larger than with fp32 multiply-adds throughout: 1.2e-8 and 2.8e-8 are
// worse at long and at short memories; with nothing given back, states that last were 10 to 30 % further off.)  Never as much as
// half a unit of the last place, 2.98e-8 of the largest significands: sums that are exact, as of one token alone, stay so.
constexpr float CS_CUT_OFF = 2e-8f;

static __device__ __forceinline__ void cs_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// 8 x 8 matrices of bfloat16 from shared memory, a row of 16 bytes from each lane's address (lanes 8 i to 8 i + 7: matrix i)
static __device__ __forceinline__ void cs_ldmatrix(uint32_t (&r)[4], uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
static __device__ __forceinline__ void cs_ldmatrix_t(uint32_t (&r)[4], uint32_t at) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
// The barrier with this number, for THREADS threads; the second form tells whether any of them asks for it.
template <int THREADS>
static __device__ __forceinline__ void cs_sync(int barrier) {
  asm volatile("bar.sync %0, %1;\n" ::"r"(barrier), "n"(THREADS) : "memory");
}
template <int THREADS>
static __device__ __forceinline__ bool cs_sync_any(int barrier, bool mine) {
  uint32_t any;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbar.red.or.pred q, %2, %3, p;\nselp.u32 %0, 1, 0, q;\n}\n"
               : "=r"(any) : "r"((uint32_t)mine), "r"(barrier), "n"(THREADS) : "memory");
  return any != 0;
}
// The six products of two operands' parts: (part of the left, part of the right one), the products of first parts last
constexpr int CS_TERMS = 6;
static __device__ __forceinline__ constexpr int cs_left_part(int term) { return term == 0 ? 2 : term == 2 || term == 3 ? 1 : 0; }
static __device__ __forceinline__ constexpr int cs_right_part(int term) { return term == 1 ? 2 : term == 2 || term == 4 ? 1 : 0; }
struct CsSum {                       // of 16 x 8 outputs: the products of first parts, and the small ones
  float big[4], small[4];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int r = 0; r < 4; ++r) big[r] = small[r] = 0.f;
  }
  __device__ __forceinline__ float operator[](int r) const { return big[r] + fmaf(CS_CUT_OFF, big[r], small[r]); }
  // the same where two steps of 16 added up
  __device__ __forceinline__ float of_two(int r) const { return big[r] + fmaf(1.45f * CS_CUT_OFF, big[r], small[r]); }
};

// 16 x 8 floats of a warp as a left operand's half, for all warps of the group: [part][tile][lane]
static __device__ __forceinline__ void cs_share(uint2* X, const float (&v)[4], int tile, int lane) {
  const CsParts lo = cs_cut(v[0], v[1]), hi = cs_cut(v[2], v[3]);
#pragma unroll
  for (int i = 0; i < 3; ++i) X[(i * 4 + tile) * 32 + lane] = make_uint2(lo.part[i], hi.part[i]);
}
struct CsLeft { uint32_t part[2][3][4]; };              // left operands over 32 tokens, two steps of 16
static __device__ __forceinline__ void cs_take(CsLeft& a, const uint2* X, int lane) {
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint2 v = X[(i * 4 + j) * 32 + lane];
      a.part[j >> 1][i][2 * (j & 1)] = v.x;
      a.part[j >> 1][i][2 * (j & 1) + 1] = v.y;
    }
}

// Adds to out (16 columns of the values, the eight tokens of `tile`) a cut triangle M times U^T, out[v][t] += sum over
// i < t of M(t, i) U[i][v].  A value that is no number would reach the tokens before its own through the zeros: where U holds
// one (`odd`), it was shared as zero, and it is added by itself, from `raw`, to what may see it.
static __device__ __forceinline__ void cs_triangle(float (&out)[4], const float* M, const CsLeft& U, const float4* raw, bool odd,
                                                   int tile, int lane) {
  CsSum sum[2];                                          // of 16 tokens each
  float more[2][4];                                      // (the small products in two chains)
  sum[0].clear();
  sum[1].clear();
#pragma unroll
  for (int r = 0; r < 4; ++r) more[0][r] = more[1][r] = 0.f;
  uint4 b[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) b[i] = reinterpret_cast<const uint4*>(M)[(tile * 3 + i) * 32 + lane];
#pragma unroll
  for (int term = 0; term < CS_TERMS; ++term) {
    const uint4 right = b[cs_right_part(term)];
    cs_mma(term == 5 ? sum[0].big : term & 1 ? more[0] : sum[0].small, U.part[0][cs_left_part(term)], right.x, right.y);
    cs_mma(term == 5 ? sum[1].big : term & 1 ? more[1] : sum[1].small, U.part[1][cs_left_part(term)], right.z, right.w);
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    sum[0].small[r] += more[0][r];
    sum[1].small[r] += more[1][r];
    out[r] += sum[0][r] + sum[1][r];
  }
  if (odd)
    for (int i = 0; i < CS_C; ++i) {
      const float4 x = raw[(i >> 3) * 32 + (lane & ~3) + ((i & 7) >> 1)];    // columns g and g + 8 of the tokens i & ~1, i | 1
      const float u[2] = {i & 1 ? x.y : x.x, i & 1 ? x.w : x.z};
      for (int e = 0; e < 2; ++e) {
        const int t = 8 * tile + 2 * (lane & 3) + e;
        if (i >= t) continue;
        const uint32_t* at = reinterpret_cast<const uint32_t*>(M) + cs_tri_at(t, i);
        const float m = cs_half(at[0], i & 1) + (cs_half(at[128], i & 1) + cs_half(at[256], i & 1));
        if (cs_no_number(u[0])) out[e] = fmaf(m, u[0], out[e]);
        if (cs_no_number(u[1])) out[2 + e] = fmaf(m, u[1], out[2 + e]);
      }
    }
}

// floats of shared memory: two chunks on their way; per group its values, the parts of Q s0 (and K s0), what is shared
// of U (and of U times E, of R): cut and as it is
template <int D, int KIND>
constexpr int cs_stage_floats() {
  return cs_image_floats(D) + (KIND == CS_DELTA ? CS_WORK : CS_T) + (KIND == CS_NORMED ? 2 * CS_C : 0);
}
template <int D, int KIND>
constexpr int cs_group_floats() {
  constexpr int CUT = 3 * 4 * 32 * 2, RAW = CS_COLS * CS_C, PARTS = D / 16 * RAW;
  return CS_COLS * CS_PS + (KIND == CS_DELTA ? 2 * PARTS + 3 * CUT + 2 * RAW : PARTS + 2 * CUT + RAW) +
         (KIND == CS_NORMED ? D / 16 * CS_C + D : 0);
}
template <int D, int KIND, int GROUPS>
constexpr int cs_smem_floats() {
  return 2 * cs_stage_floats<D, KIND>() + GROUPS * cs_group_floats<D, KIND>();
}

static __device__ __forceinline__ float4 cs_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
static __device__ __forceinline__ float4 cs_load4(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}

// Fragments: lane (g, t) = (lane >> 2, lane & 3) holds of a result of 16 x 8 the rows g (elements 0, 1) and g + 8 (2, 3),
// columns 2 t and 2 t + 1.
template <int D, int KIND, int GROUPS, typename TV>
__global__ void __launch_bounds__(2 * D * GROUPS, 1) chunk_scan_kernel(const CsScan p) {
  constexpr bool DELTA = KIND == CS_DELTA, NORMED = KIND == CS_NORMED;
  constexpr int WARPS = D / 16, GROUP_THREADS = 32 * WARPS, THREADS = GROUP_THREADS * GROUPS;
  constexpr int IMAGE = cs_image_floats(D), WORK = DELTA ? CS_WORK : CS_T, STAGE = cs_stage_floats<D, KIND>();
  constexpr int PLANE = CS_C * D * 2, Q_PLANES = 3 * PLANE;      // bytes of a part of K or Q; where Q's parts start
  constexpr int CUT = 3 * 4 * 32, RAW = 4 * 32;           // elements of uint2, of float4
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int group = tid / GROUP_THREADS, gt = tid % GROUP_THREADS, warp = gt >> 5;
  float* Vs = smem + 2 * STAGE + group * cs_group_floats<D, KIND>();         // [16 columns][CS_PS]
  float4* Xq = reinterpret_cast<float4*>(Vs + CS_COLS * CS_PS);              // [warp][tile of tokens][lane]: parts of Q s0
  float4* Xk = Xq + WARPS * RAW;                          // DELTA: of K s0
  uint2* Xu = reinterpret_cast<uint2*>(Xk + (DELTA ? WARPS * RAW : 0));      // U cut, U times E cut, DELTA: R cut
  uint2 *Xe = Xu + CUT, *Xr = Xe + CUT;
  float4* raw_u = reinterpret_cast<float4*>(Xr + (DELTA ? CUT : 0));         // [tile of tokens][lane]: U, DELTA: R
  float4* raw_r = raw_u + RAW;
  float* Xn = reinterpret_cast<float*>(raw_u + RAW);      // NORMED: [warp][32 tokens] parts of Q n0
  float* Ns = Xn + WARPS * CS_C;                          // NORMED: [D] n
  pdl_wait();
  const int s = blockIdx.x, h = blockIdx.y, cb = blockIdx.z * GROUPS + group, col0 = cb * CS_COLS;
  const int gk = h / (p.H / p.G), d = p.d, dv = p.dv;
  const int first = p.cu_q[s], n = p.cu_q[s + 1] - first, slot = p.slots[s];
  const int ncol = max(0, min(CS_COLS, dv - col0));       // a multiple of 4 (0: a group behind the last column)
  float* yb = p.y + (size_t)first * p.H * dv + (size_t)h * dv + col0;
  if (slot < 0) {
    for (int i = gt; i < n * ncol; i += GROUP_THREADS) yb[(size_t)(i / ncol) * p.H * dv + i % ncol] = 0.f;
    return;
  }
  if (n <= 0) return;
  const bool fresh = p.q_start[s] == 0;
  float* base = p.state + (size_t)slot * p.state_stride;
  float* st = base + ((size_t)h * dv + col0) * d;
  const int n_blocks = (dv + CS_COLS - 1) / CS_COLS;      // NORMED: a copy of n and m per 16 columns
  const TV* vb = (const TV*)p.v + (size_t)first * p.v_stride + (size_t)h * dv + col0;
  const long number0 = first / CS_C + s;
  const int n_chunks = (n + CS_C - 1) / CS_C;
  const float* extra = NORMED ? p.extra + (number0 * p.H + h) * (2 * CS_C + d) : nullptr;
  const long extra_step = (long)p.H * (2 * CS_C + d);

  auto fetch = [&](int c) {                               // all of chunk c but its values
    float* to = smem + (c & 1) * STAGE;
    const float* image = p.images + ((number0 + c) * p.G + gk) * IMAGE;
#pragma unroll
    for (int e = 4 * tid; e < IMAGE; e += 4 * THREADS) cs_copy16_all(to + e, image + e);
    const float* w = p.work + ((number0 + c) * p.H + h) * CS_WORK;
#pragma unroll
    for (int e = 4 * tid; e < WORK; e += 4 * THREADS) cs_copy16_all(to + IMAGE + e, w + e);
    if (NORMED && tid < 2 * CS_C / 4) cs_copy16_all(to + IMAGE + WORK + 4 * tid, extra + c * extra_step + 4 * tid);
    cs_commit();
  };
  const int vt = gt >> 2, vc = 4 * (gt & 3);              // the four values of a chunk that this thread brings in
  auto load_v = [&](int c) {
    const int at = c * CS_C + vt;
    return vt < CS_C && at < n && vc < ncol ? cs_load4(vb + (size_t)at * p.v_stride + vc) : make_float4(0.f, 0.f, 0.f, 0.f);
  };

  fetch(0);
  const bool st_vec = ((uintptr_t)st % 8) == 0;
  const int row0 = warp * 16 + 2 * t;                     // (the first of) this lane's rows of S
  float S[2][4];
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int c = g + 8 * half, i = row0 + 8 * j;
      float2 v = make_float2(0.f, 0.f);
      if (!fresh && c < ncol && i < d) {
        const float* at = st + (size_t)c * d + i;
        v = st_vec ? *reinterpret_cast<const float2*>(at) : make_float2(at[0], at[1]);
      }
      S[j][2 * half] = v.x;
      S[j][2 * half + 1] = v.y;
    }
  if (NORMED) {
    const float* nm = base + (size_t)p.H * dv * d + ((size_t)h * n_blocks + blockIdx.z * GROUPS) * (d + 1);
    for (int i = gt; i < D; i += GROUP_THREADS) Ns[i] = !fresh && i < d ? nm[i] : 0.f;
  }
  const float skip = KIND == CS_PLAIN && p.skip ? p.skip[h] : 0.f;
  float4 v_next = load_v(0);
  // this lane's row of the matrices that it points ldmatrix to, as bytes from the start of a part: two tiles of tokens and the
  // two pieces of the warp's rows of S for K and Q as they are, row `lane` for K transposed
  const uint32_t smem0 = (uint32_t)__cvta_generic_to_shared(smem);
  const uint32_t at_rows = (uint32_t)(((lane & 7) + 8 * (lane >> 4)) * D * 2 + (((2 * warp + ((lane >> 3) & 1)) ^ (lane & 7)) << 4));
  const uint32_t at_cols = (uint32_t)(lane * D * 2);
  // a chunk's tokens in tiles of eight: the first four warps make U (the chain), the last four the outputs
  const bool makes_u = warp < 4, makes_o = warp >= WARPS - 4;
  const int tile_o = warp - (WARPS - 4), all_of_group = 1 + 2 * group, makers_of_u = 2 + 2 * group;
  bool odd = false;                                       // whether the chunk's U holds a value that is no number
  CsLeft left;

  auto sum_parts = [&](const float4* X, int tile) {
    float4 a = X[tile * 32 + lane];
#pragma unroll
    for (int w = 1; w < WARPS; ++w) {
      const float4 x = X[(w * 4 + tile) * 32 + lane];
      a.x += x.x; a.y += x.y; a.z += x.z; a.w += x.w;
    }
    return a;
  };
  auto outputs = [&](int c) {
    const int cn = min(CS_C, n - c * CS_C);
    if (8 * tile_o >= cn) return;
    const float *stage = smem + (c & 1) * STAGE, *vec = stage + IMAGE;
    const int t0 = 8 * tile_o + 2 * t;                    // this lane's two tokens
    const float4 qs = sum_parts(Xq, tile_o), u4 = raw_u[tile_o * 32 + lane];
    const float2 ga = *reinterpret_cast<const float2*>(vec + CS_GAM + t0), pd = *reinterpret_cast<const float2*>(vec + CS_PD + t0);
    const float u[4] = {u4.x, u4.y, u4.z, u4.w};
    float o[4] = {ga.x * qs.x, ga.y * qs.y, ga.x * qs.z, ga.y * qs.w};
    cs_take(left, Xu, lane);
    cs_triangle(o, vec + CS_P, left, raw_u, odd, tile_o, lane);
    float den[2] = {1.f, 1.f};
    if (NORMED) {
      const float* ex = vec + WORK;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        float dot = Xn[t0 + e];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) dot += Xn[w * CS_C + t0 + e];
        den[e] = fmaxf(fabsf((e ? ga.y : ga.x) * dot + ex[t0 + e]), ex[CS_C + t0 + e]) + 1e-6f;
      }
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int e = r & 1, col = g + 4 * (r & 2);
      float out = fmaf(e ? pd.y : pd.x, u[r], o[r]);
      if (KIND == CS_PLAIN) out = fmaf(skip, u[r], out);
      if (NORMED) out /= den[e];
      if (t0 + e < cn && col < ncol) yb[(size_t)(c * CS_C + t0 + e) * p.H * dv + col] = out;
    }
  };

  for (int c = 0; c < n_chunks; ++c) {
    const float *stage = smem + (c & 1) * STAGE, *vec = stage + IMAGE;
    const uint32_t image = smem0 + (uint32_t)((c & 1) * STAGE * 4);
    if (makes_u) {
      Vs[(vc + 0) * CS_PS + vt] = v_next.x; Vs[(vc + 1) * CS_PS + vt] = v_next.y;
      Vs[(vc + 2) * CS_PS + vt] = v_next.z; Vs[(vc + 3) * CS_PS + vt] = v_next.w;
    }
    cs_wait<0>();
    __syncthreads();                                      // chunk c is there, and what chunk c - 1 lay in is free
    float n_add = 0.f;
    if (NORMED && gt < d) n_add = extra[c * extra_step + 2 * CS_C + gt];
    if (c + 1 < n_chunks) {
      fetch(c + 1);
      v_next = load_v(c + 1);
    }
    float own[4];                                         // the values of this warp's tokens
    if (makes_u)
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const float2 v = *reinterpret_cast<const float2*>(Vs + (g + 8 * half) * CS_PS + 8 * warp + 2 * t);
        own[2 * half] = v.x;
        own[2 * half + 1] = v.y;
      }
    // shares U (this warp's tokens of it) with the group, and U times E
    auto share_u = [&]() {
      bool mine = false;
      float clean[4], scaled[4];
      const float2 e = *reinterpret_cast<const float2*>(vec + CS_E + 8 * warp + 2 * t);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const bool no = cs_no_number(own[r]);
        mine |= no;
        clean[r] = no ? 0.f : own[r];
        scaled[r] = (r & 1 ? e.y : e.x) * clean[r];
      }
      cs_share(Xe, scaled, warp, lane);
      cs_share(Xu, clean, warp, lane);
      raw_u[warp * 32 + lane] = make_float4(own[0], own[1], own[2], own[3]);
      return mine;
    };

    // parts of (rows s0)^T over this warp's rows of S, for the chunk's 32 tokens
    uint32_t s_left[3][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const CsParts x = cs_cut(S[r >> 1][2 * (r & 1)], S[r >> 1][2 * (r & 1) + 1]);
#pragma unroll
      for (int i = 0; i < 3; ++i) s_left[i][r] = x.part[i];
    }
    uint32_t b[3][4][2];                                  // [part][tile of tokens][half]
    auto times_state = [&](CsSum (&sum)[4], uint32_t planes) {
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          uint32_t r[4];
          cs_ldmatrix(r, planes + at_rows + i * PLANE + 8 * j * D * 2);
          b[i][j][0] = r[0]; b[i][j][1] = r[1]; b[i][j + 1][0] = r[2]; b[i][j + 1][1] = r[3];
        }
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[j].clear();
#pragma unroll
      for (int term = 0; term < CS_TERMS; ++term)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          cs_mma(term == 5 ? sum[j].big : sum[j].small, s_left[cs_left_part(term)], b[cs_right_part(term)][j][0],
                 b[cs_right_part(term)][j][1]);
    };
    auto leave = [&](float4* X, const CsSum (&sum)[4]) {
#pragma unroll
      for (int j = 0; j < 4; ++j) X[(warp * 4 + j) * 32 + lane] = make_float4(sum[j][0], sum[j][1], sum[j][2], sum[j][3]);
    };
    auto times_n = [&]() {                                // parts of Q n0 (with Q in `b`)
      // the three parts of n as three rows of a left operand, so that one product makes three of them
      const CsParts lo = cs_cut(Ns[row0], Ns[row0 + 1]), hi = cs_cut(Ns[row0 + 8], Ns[row0 + 9]);
      const uint32_t n_left[4] = {g == 0 ? lo.part[0] : g == 1 ? lo.part[1] : g == 2 ? lo.part[2] : 0u, 0u,
                                  g == 0 ? hi.part[0] : g == 1 ? hi.part[1] : g == 2 ? hi.part[2] : 0u, 0u};
      CsSum sum[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) sum[j].clear();
#pragma unroll
      for (int i = 2; i >= 0; --i)
#pragma unroll
        for (int j = 0; j < 4; ++j) cs_mma(i ? sum[j].small : sum[j].big, n_left, b[i][j][0], b[i][j][1]);
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          // row 0: n's first part times Q's first (big) and others (small); rows 1 and 2: small altogether
          const float big = sum[j].big[e], rest = sum[j].small[e] + (g == 0 ? CS_CUT_OFF * big : big);
          const float dot = big + (rest + (__shfl_down_sync(0xffffffffu, rest, 4) + __shfl_down_sync(0xffffffffu, rest, 8)));
          if (g == 0) Xn[warp * CS_C + 8 * j + 2 * t + e] = dot;
        }
    };
    bool mine = false;
    CsSum sums[4];
    if (DELTA) {
      times_state(sums, image);
      leave(Xk, sums);
    } else if (makes_u) {
      mine = share_u();
    }
    times_state(sums, image + Q_PLANES);
    leave(Xq, sums);
    if (NORMED) times_n();
    if (DELTA) cs_sync<GROUP_THREADS>(all_of_group);
    if (DELTA && makes_u) {                               // R = V - diag(gam) K s0, of this warp's tokens
      const float4 ks = sum_parts(Xk, warp);
      const float2 ga = *reinterpret_cast<const float2*>(vec + CS_GAM + 8 * warp + 2 * t);
      own[0] -= ga.x * ks.x; own[1] -= ga.y * ks.y; own[2] -= ga.x * ks.z; own[3] -= ga.y * ks.w;
      float clean[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const bool no = cs_no_number(own[r]);
        mine |= no;
        clean[r] = no ? 0.f : own[r];
      }
      cs_share(Xr, clean, warp, lane);
      raw_r[warp * 32 + lane] = make_float4(own[0], own[1], own[2], own[3]);
      const bool odd_r = cs_sync_any<128>(makers_of_u, mine);
      cs_take(left, Xr, lane);                            // U = T' R; the token's own term, most of the sum, last
      float u[4] = {0.f, 0.f, 0.f, 0.f};
      cs_triangle(u, vec + CS_T, left, raw_r, odd_r, warp, lane);
      const float2 td = *reinterpret_cast<const float2*>(vec + CS_TD + 8 * warp + 2 * t);
#pragma unroll
      for (int r = 0; r < 4; ++r) own[r] = fmaf(r & 1 ? td.y : td.x, own[r], u[r]);
    }
    if (DELTA) mine = makes_u && share_u();
    // K transposed, [part][tile of S's rows][step, half]
    uint32_t k_cols[3][2][4];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) cs_ldmatrix_t(k_cols[i][j], image + at_cols + i * PLANE + (((2 * warp + j) ^ (lane & 7)) << 4));
    const float keep = vec[CS_GAM + CS_C - 1];
    odd = cs_sync_any<GROUP_THREADS>(all_of_group, mine);
    if (NORMED && gt < d) Ns[gt] = fmaf(keep, Ns[gt], n_add);
    // s_end = gam_C s0 + sum_t E_t k_t u_t^T
    {
      cs_take(left, Xe, lane);
      CsSum sum[2];
      float more[2][4];                                   // (the small products in two chains)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        sum[j].clear();
#pragma unroll
        for (int r = 0; r < 4; ++r) more[j][r] = 0.f;
      }
#pragma unroll
      for (int term = 0; term < CS_TERMS; ++term)
#pragma unroll
        for (int kk = 0; kk < 2; ++kk)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            cs_mma(term == 5 ? sum[j].big : kk ? more[j] : sum[j].small, left.part[kk][cs_left_part(term)],
                   k_cols[cs_right_part(term)][j][2 * kk], k_cols[cs_right_part(term)][j][2 * kk + 1]);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          sum[j].small[r] += more[j][r];
          S[j][r] = fmaf(S[j][r], keep, sum[j].of_two(r));
        }
      if (odd)                                            // the values that are no numbers, by themselves
        for (int i = 0; i < CS_C; ++i) {
          const float4 x = raw_u[(i >> 3) * 32 + (lane & ~3) + ((i & 7) >> 1)];
          const float u[2] = {i & 1 ? x.y : x.x, i & 1 ? x.w : x.z};
          const unsigned char* row = reinterpret_cast<const unsigned char*>(stage) + i * D * 2;
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int at = (((2 * warp + j) ^ (i & 7)) << 4) + 4 * t;
            uint32_t k[3];
#pragma unroll
            for (int e = 0; e < 3; ++e) k[e] = *reinterpret_cast<const uint32_t*>(row + e * PLANE + at);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
              const float k1 = cs_half(k[0], r & 1) + (cs_half(k[1], r & 1) + cs_half(k[2], r & 1));
              if (cs_no_number(u[r >> 1])) S[j][r] = fmaf(k1, vec[CS_E + i] * u[r >> 1], S[j][r]);
            }
          }
        }
    }
    if (makes_o) outputs(c);
  }
  pdl_launch_dependents();
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int c = g + 8 * half, i = row0 + 8 * j;
      if (c >= ncol || i >= d) continue;
      float* at = st + (size_t)c * d + i;
      if (st_vec) *reinterpret_cast<float2*>(at) = make_float2(S[j][2 * half], S[j][2 * half + 1]);
      else { at[0] = S[j][2 * half]; at[1] = S[j][2 * half + 1]; }
    }
  if (NORMED && ncol > 0) {
    float* nm = base + (size_t)p.H * dv * d + ((size_t)h * n_blocks + cb) * (d + 1);
    for (int i = gt; i <= d; i += GROUP_THREADS) nm[i] = i < d ? Ns[i] : p.top[(size_t)(first + n - 1) * p.H + h];
  }
}

template <int D, int KIND, int GROUPS, typename TV>
static cudaError_t cs_launch_groups(const CsScan& p, int n_seqs, cudaStream_t stream) {
  constexpr int smem = cs_smem_floats<D, KIND, GROUPS>() * 4;
  static_assert(smem <= 232448, "an SM's shared memory");
  static std::atomic<uint64_t> done{0};
  auto kernel = chunk_scan_kernel<D, KIND, GROUPS, TV>;
  const cudaError_t e = nhv_allow_smem((const void*)kernel, smem, done);
  if (e != cudaSuccess) return e;
  const int blocks = (p.dv + CS_COLS * GROUPS - 1) / (CS_COLS * GROUPS);
  return nhv_launch(kernel, dim3(n_seqs, p.H, blocks), 2 * D * GROUPS, smem, stream, p);
}
// A block takes an SM.  One group a block while all of them find an SM of their own, else two, which share a chunk's operands: 8
// requests of 512 tokens, 1,024 groups, delta rule 217 us (the CUDA-core form's two blocks an SM: 330).
template <int D, int KIND, typename TV>
static cudaError_t cs_launch_scan(const CsScan& p, int n_seqs, cudaStream_t stream) {
  const long groups = (long)n_seqs * p.H * ((p.dv + CS_COLS - 1) / CS_COLS);
  return groups <= 148 ? cs_launch_groups<D, KIND, 1, TV>(p, n_seqs, stream) : cs_launch_groups<D, KIND, 2, TV>(p, n_seqs, stream);
}
