// C[M,N] = A[M,K] * W[N,K]^T in fp32 on the 5th-generation tensor cores (tcgen05.mma), with no less precision than fp32
// multiply-adds: each operand is cut into three bfloat16 of eight bits, which hold it exactly (7.7e-34 and more), and a product is
// the six products of their parts down to 2^-16 of the largest (what is left out is below 2^-24 of it and of either sign).
// Rows of smaller values, sums below 1.2e-35 and sums that are no finite number are multiplied again on the CUDA cores, by
// themselves: infinities and the whole range of fp32 give what they give there.  Looking for them costs up to 4 % for 1 to 16 rows
// (6144 x 1024 14.2 and 14.4 us, 43392 x 1024 65.8 and 68.5); ordinary rows show a larger value in their last stage.
//
// Sums.  The tensor cores cut off what lies below a sum's last place.  So the products of first parts are added up over 64
// columns only (four MMAs) in tensor memory and then added to a sum in registers, rounded to the nearest; the five kinds of
// small products, 2^-8 of it and less, stay in a sum of their own in tensor memory over the whole run of columns.  Error
// against 64 bits (relative, 2-norm, unit normal operands), K = 1,024, 2,048, 3,072, 4,096: 9.4e-8, 9.9e-8, 1.06e-7, 1.7e-7; fp32
// multiply-adds in two sums per output (gemm_simt.cu): 4.1e-7, 5.7e-7, 7.0e-7, 8.1e-7.
//
// A value of C does not depend on M, on the tile that holds it or on the batch: the columns of K are cut into runs (one or
// SPLIT of them, by N and K alone), each run goes through its stages in order, and the runs are added in order.
//
// A block takes 128 rows of W (M axis of the MMA, lanes of tensor memory) by 128 rows of A, or by 32 where A has no more (N axis).
// Warps 8-15 fetch both operands from global memory, one stage of 64 columns ahead in registers (W four stages ahead into L2),
// cut them and write the parts to shared memory in the 128-byte swizzle (two stages of six tiles of 128 x 64; three where A's
// tiles are small); lane 0 of warp 16 issues the MMAs; warps 0-7, two for each quarter of the lanes, add the stages' sums to
// their registers, two sums alternating in tensor memory so that the next stage's MMAs run meanwhile.  Where K has more than
// one run, a cluster of blocks takes a tile, a run each, and adds the runs through its shared memory.
//
// What bounds it: the way of a stage from global memory to its parts, about 2 us for 64 columns of both operands (1.1 where A
// has up to 32 rows), beside 1,536 cycles of the tensor pipe, whose MMAs read all that shared memory gives.  In us, on the CUDA cores
// and here, weights from memory, for 370 rows: N x K = 4096 x 1024 88 and 37, 1024 x 2048 159 and 19, 6144 x 1024 115 and 38, 1024 x 3072
// 238 and 25; for 16 rows 28 and 14, 42 and 14, 34 and 15, 62 and 18; 43392 x 1024, 3 and 33 rows: 65 and 69, 140 and 89.  Not faster: W two stages
// ahead in registers with the MMAs issued by an adding warp (41 against 37 for 370 x 4096 x 1024 in one run).
#define NHV_WAIT_LIMIT (1u << 22)
#include "nhv_async.cuh"

namespace {

constexpr int TILE = 128;              // rows of W per block
constexpr int BK = 64;                 // columns per stage = one 128-byte swizzle row of bfloat16
constexpr int ADD_WARPS = 8, CUT_WARPS = 8;
constexpr int THREADS = 32 * (2 + ADD_WARPS + CUT_WARPS);
constexpr int FIRST_CUT = ADD_WARPS, MMA_WARP = ADD_WARPS + CUT_WARPS, ALLOC_WARP = MMA_WARP + 1;
constexpr int W_PART = TILE * 128;     // bytes of a part's tile
constexpr int stages_of(int nt) { return nt == 128 ? 2 : 3; }
constexpr int stage_bytes(int nt) { return 3 * (W_PART + nt * 128); }       // W's three parts, then A's
constexpr uint32_t tmem_cols(int nt) { return nt == 128 ? 512 : 128; }      // two alternating sums and the small products'
constexpr int MAX_SPLIT = 4;

__device__ __forceinline__ void tmem_alloc(uint32_t* slot_in_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(slot_in_smem)), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
// D[tmem] (+)= A[smem] * B[smem]^T, both operands K-major bfloat16
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_ld16(float (&v)[16], uint32_t taddr) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// Shared-memory matrix descriptor of a K-major bf16 operand tile in the 128-byte swizzle (rows of 128 bytes, groups of
// 8 rows 1024 bytes apart; the tile starts on a 1024-byte boundary; `addr` may point 32, 64 or 96 bytes into the
// first row to select the K=16 slice).
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
  uint64_t d = 0;
  d |= (uint64_t)((addr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
// Instruction descriptor: bf16 x bf16 -> fp32, both K-major, M x N.
__device__ __forceinline__ uint32_t instr_desc(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ float4 cluster_load4(const float* mine, uint32_t rank) {       // the same place in another block
  uint32_t at;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(smem_u32(mine)), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
  return v;
}

__device__ __forceinline__ uint32_t cluster_load(const uint32_t* mine, uint32_t rank) {
  uint32_t at, v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(at) : "r"(smem_u32(mine)), "r"(rank));
  asm volatile("ld.shared::cluster.u32 %0, [%1];\n" : "=r"(v) : "r"(at) : "memory");
  return v;
}

// Eight floats as three times eight bfloat16 (16 bytes each): what is left, rounded to eight bits, three times (above bfloat16's
// largest, 3.39e38, the first part is that).  Exact down to 7.7e-34, below which the last bits are less than bfloat16's smallest
// number; an infinity has a part that is no number.  What that leaves wrong is done again: `by_multiply_adds`.
__device__ __forceinline__ void cut8(uint4 (&part)[3], const float (&x)[8]) {
  float v[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = x[j];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    uint32_t p[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (i == 0) asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;\n" : "=r"(p[j]) : "f"(v[2 * j + 1]), "f"(v[2 * j]));
      else asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(p[j]) : "f"(v[2 * j + 1]), "f"(v[2 * j]));
      v[2 * j] -= __uint_as_float(p[j] << 16);
      v[2 * j + 1] -= __uint_as_float(p[j] & 0xffff0000u);
    }
    part[i] = make_uint4(p[0], p[1], p[2], p[3]);
  }
}

// The largest of eight floats (what is no number does not count).
__device__ __forceinline__ float largest_of8(const float (&x)[8]) {
  float a, b;
  asm("max.abs.f32 %0, %1, %2, %3;\n" : "=f"(a) : "f"(x[0]), "f"(x[1]), "f"(x[2]));
  asm("max.abs.f32 %0, %1, %2, %3;\n" : "=f"(b) : "f"(x[3]), "f"(x[4]), "f"(x[5]));
  asm("max.abs.f32 %0, %1, %2, %3;\n" : "=f"(a) : "f"(x[6]), "f"(x[7]), "f"(a));
  return fmaxf(a, b);
}
constexpr float SMALL_ROW = 0x1p-101f, SMALL_SUM = 0x1p-116f;
// Whether the tensor cores' sum is to be done again: no finite number, or so small that fp32's last place is 2^-149 (cut off there
// in each step, K / 64 times over); not where it is zero.
__device__ __forceinline__ bool doubtful(float v) {
  const uint32_t size = __float_as_uint(v) & 0x7fffffffu, least = __float_as_uint(SMALL_SUM);
  return size - least >= 0x7f800000u - least && size != 0;
}

// One value of C on the CUDA cores, as gemm_simt.cu adds it up.  For what the tensor cores cannot give: a sum that is `doubtful` (no
// finite number: an operand is none, or some of the parts' products are beyond fp32's range, of either sign), and rows of A
// or W whose largest value is below SMALL_ROW (their last bits are lost in bfloat16; beside a larger value in the row they
// are below 2^-30 of it).
__device__ __noinline__ float by_multiply_adds(const float* a, const float* w, int K) {
  float even = 0.f, odd = 0.f;
  for (int k = 0; k < K; k += 4) {
    const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(w + k);
    even = fmaf(x.z, y.z, fmaf(x.x, y.x, even));
    odd = fmaf(x.w, y.w, fmaf(x.y, y.y, odd));
    if (isnan(even) || isnan(odd)) break;                        // stays one
  }
  return even + odd;
}

// Order of a stage's products: (part of W, part of A), the products of first parts by themselves
__device__ __forceinline__ constexpr int w_part(int term) { return term == 0 ? 2 : term == 2 || term == 3 ? 1 : 0; }
__device__ __forceinline__ constexpr int a_part(int term) { return term == 1 ? 2 : term == 2 || term == 4 ? 1 : 0; }

struct Params {
  float* C;
  const float *A, *W;
  int M, N, K, lda, ldc;
  int split, run;                      // runs of K; columns of a run (a multiple of BK; the last one may be shorter)
};

template <int NT>                                                 // rows of A per block
__global__ void __launch_bounds__(THREADS, 1) gemm_f32_tcgen05_kernel(const Params p) {
  constexpr int STAGES = stages_of(NT), STAGE_BYTES = stage_bytes(NT), A_PART = NT * 128, PER = NT / 2;    // PER: rows of A an adding warp
  constexpr uint32_t SMALL_COL = 2 * NT;
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = smem_unaligned + ((1024 - (smem_u32(smem_unaligned) & 1023)) & 1023);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)STAGES * STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* sum_full = empty + STAGES;           // the alternating sums
  uint64_t* sum_empty = sum_full + 2;
  uint64_t* small_full = sum_empty + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(small_full + 1);
  __shared__ int s_abort;
  // rows of W, then of A: 1 where the run holds a value of SMALL_ROW or more, 256 where one that is not zero; whether a row is small
  __shared__ uint32_t s_size[TILE + NT], s_small[TILE + NT];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = p.split > 1 ? cluster_rank() : 0;
  const int n0 = (int)(blockIdx.x / p.split) * TILE, m0 = blockIdx.y * NT;
  const int k0 = (int)rank * p.run, k1 = min(p.K, k0 + p.run);
  const int stages = (k1 - k0 + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], CUT_WARPS);
      mbar_init(&empty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&sum_full[s], 1);
      mbar_init(&sum_empty[s], ADD_WARPS);
    }
    mbar_init(small_full, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == ALLOC_WARP) tmem_alloc(tmem_slot, tmem_cols(NT));
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();

  const bool adds = warp < ADD_WARPS;
  const int col = (warp & 3) * 32 + lane, row0 = warp / 4 * PER;   // an adding lane's row of W; (the first of) its rows of A
  float acc[PER];
  if (warp >= FIRST_CUT && warp < MMA_WARP) {
    // ------------------------------------------------------------------ fetch and cut: eight floats of a row a task
    const int t = threadIdx.x - 32 * FIRST_CUT, c = t & 7, r0 = t >> 3;      // piece of the row; rows r0 + 32 i
    float w[4][8], a[NT / 32][8];
    auto load = [&](auto& v, const float* X, int rows, long ld, int base, int stage) {
      const int k = k0 + stage * BK + 8 * c;
#pragma unroll
      for (int i = 0; i < (int)(sizeof(v) / sizeof(v[0])); ++i) {
        const int r = base + r0 + 32 * i;
        const float* at = X + (size_t)r * ld + k;
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] = 0.f;
        if (r < rows && k < k1) {                                // K is a multiple of 4
          if (k + 4 < k1 && ((uintptr_t)at & 31) == 0)
            asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                         : "=f"(v[i][0]), "=f"(v[i][1]), "=f"(v[i][2]), "=f"(v[i][3]), "=f"(v[i][4]), "=f"(v[i][5]),
                           "=f"(v[i][6]), "=f"(v[i][7]) : "l"(at) : "memory");
          else {
            const float4 x = *reinterpret_cast<const float4*>(at);
            v[i][0] = x.x; v[i][1] = x.y; v[i][2] = x.z; v[i][3] = x.w;
            if (k + 4 < k1) {
              const float4 y = *reinterpret_cast<const float4*>(at + 4);
              v[i][4] = y.x; v[i][5] = y.y; v[i][6] = y.z; v[i][7] = y.w;
            }
          }
        }
      }
    };
    // bits 0 to 3: this thread's rows of W that hold a value of SMALL_ROW or more, 4 to 7: of A; 8 to 15: any that is not zero
    constexpr unsigned ROWS = NT == 128 ? 0xff : 0x1f;
    unsigned sizes = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (n0 + r0 + 32 * i >= p.N) sizes |= 1u << i;
      if (i < NT / 32 && m0 + r0 + 32 * i >= p.M) sizes |= 16u << i;
    }
    auto look = [&](const auto& v, unsigned bit) {
#pragma unroll
      for (int i = 0; i < (int)(sizeof(v) / sizeof(v[0])); ++i) {
        const float top = largest_of8(v[i]);
        if (top >= SMALL_ROW) sizes |= bit << i;
        if (top > 0.f) sizes |= bit << (8 + i);
      }
    };
    auto put = [&](const auto& v, unsigned char* tiles, int part_bytes) {
#pragma unroll
      for (int i = 0; i < (int)(sizeof(v) / sizeof(v[0])); ++i) {
        const int r = r0 + 32 * i;
        uint4 part[3];
        cut8(part, v[i]);
#pragma unroll
        for (int e = 0; e < 3; ++e)
          *reinterpret_cast<uint4*>(tiles + e * part_bytes + r * 128 + ((c ^ (r & 7)) << 4)) = part[e];
      }
    };
    // W two and more stages ahead into L2: thread t asks for the line t & 1 of row t >> 1
    auto hint = [&](int stage) {
      const int r = n0 + (t >> 1), k = k0 + stage * BK + 32 * (t & 1);
      if (r < p.N && k < k1) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p.W + (size_t)r * p.K + k));
    };
    load(w, p.W, p.N, p.K, n0, 0);
    for (int s = 1; s < 4; ++s) hint(s);
    pdl_wait();                                                  // A is the work of kernels before
    load(a, p.A, p.M, p.lda, m0, 0);
    for (int s = 0; s < stages; ++s) {
      const int slot = s % STAGES;
      if (s >= STAGES && !mbar_wait(&empty[slot], (uint32_t)((s / STAGES) - 1) & 1, 1)) { s_abort = 1; break; }
      unsigned char* to = smem + (size_t)slot * STAGE_BYTES;
      hint(s + 4);
      put(w, to, W_PART);
      if (s + 1 < stages) load(w, p.W, p.N, p.K, n0, s + 1);
      put(a, to + 3 * W_PART, A_PART);
      if (s + 1 < stages) load(a, p.A, p.M, p.lda, m0, s + 1);
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[slot]);
    }
    // The rows' sizes: the last stage, still in registers, says enough of ordinary rows, while its products are made; where a row
    // has nothing but small values there, the others are read again.
    for (int s = -1; s + 1 < stages; ++s) {
      if (s >= 0) {
        load(w, p.W, p.N, p.K, n0, s);
        load(a, p.A, p.M, p.lda, m0, s);
      }
      look(w, 1u);
      look(a, 16u);
#pragma unroll
      for (int d = 1; d < 8; d <<= 1) sizes |= __shfl_xor_sync(0xffffffffu, sizes, d);
      if (__all_sync(0xffffffffu, (sizes & ROWS) == ROWS)) break;
    }
    if (c == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i) s_size[r0 + 32 * i] = sizes >> i & 0x101;
#pragma unroll
      for (int i = 0; i < NT / 32; ++i) s_size[TILE + r0 + 32 * i] = sizes >> (4 + i) & 0x101;
    }
  } else if (warp == MMA_WARP) {
    // ------------------------------------------------------------------ MMA issuer
    if (lane == 0) {
      const uint32_t idesc = instr_desc(TILE, NT);
      bool ok = true;
      for (int s = 0; s < stages && ok; ++s) {
        const int slot = s % STAGES, sum = s & 1;
        ok = (s < 2 || mbar_wait(&sum_empty[sum], (uint32_t)((s / 2) - 1) & 1, 2)) && mbar_wait(&full[slot], (uint32_t)(s / STAGES) & 1, 3);
        if (!ok) break;
        tc_fence_after();
        const uint32_t w_addr = smem_u32(smem + (size_t)slot * STAGE_BYTES), a_addr = w_addr + 3 * W_PART;
#pragma unroll
        for (int term = 0; term < 6; ++term)
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            tc_mma(tmem_base + (term == 5 ? (uint32_t)(sum * NT) : SMALL_COL),
                   smem_desc_sw128(w_addr + w_part(term) * W_PART + kk * 32),
                   smem_desc_sw128(a_addr + a_part(term) * A_PART + kk * 32), idesc,
                   term == 5 ? (kk == 0 ? 0u : 1u) : (s == 0 && term == 0 && kk == 0 ? 0u : 1u));
        tc_commit(&empty[slot]);
        tc_commit(&sum_full[sum]);
      }
      if (ok) tc_commit(small_full);
      else s_abort = 1;
    }
    __syncwarp();
    pdl_wait();
  } else if (adds) {
    // ------------------------------------------------------------------ the sums: a row of W a lane, half the rows of A a warp
    const uint32_t taddr = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)row0;
#pragma unroll
    for (int i = 0; i < PER; ++i) acc[i] = 0.f;
    auto add = [&](uint32_t at) {
#pragma unroll
      for (int q = 0; q < PER; q += 16) {
        float v[16];
        tmem_ld16(v, at + q);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[q + i] += v[i];
      }
    };
    bool ok = true;
    for (int s = 0; s < stages && ok; ++s) {
      ok = __all_sync(0xffffffffu, mbar_wait(&sum_full[s & 1], (uint32_t)(s / 2) & 1, 4));
      if (!ok) break;
      tc_fence_after();
      add(taddr + (s & 1) * NT);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sum_empty[s & 1]);
    }
    ok = ok && __all_sync(0xffffffffu, mbar_wait(small_full, 0, 5));
    if (!ok) s_abort = 1;
    else {
      tc_fence_after();
      add(taddr + SMALL_COL);
      tc_fence_before();
    }
    pdl_wait();                                                  // C may be read by kernels before
  } else {
    pdl_wait();
  }
  // ------------------------------------------------------------------ out: a lane holds a row of W, neighbours in a row of C
  __syncthreads();                                               // (the ring is free: the last MMAs have read it)
  bool again = false;                                            // whether this thread has met a value that is to be done again
  const int share = NT / p.split, first = (int)rank * share;     // each block of the cluster its share of the tile's rows
  if (p.split == 1) {
    if (adds && !s_abort && n0 + col < p.N)
#pragma unroll
      for (int i = 0; i < PER; ++i)
        if (m0 + row0 + i < p.M) {
          p.C[(size_t)(m0 + row0 + i) * p.ldc + n0 + col] = acc[i];
          again |= doubtful(acc[i]);
        }
    if (const int t = THREADS - 1 - (int)threadIdx.x; t < TILE + NT) {
      s_small[t] = s_size[t] == 0x100;
      again |= s_small[t] != 0;
    }
  } else {
    float* tile = reinterpret_cast<float*>(smem);                // [rows of A][128 rows of W]
    if (adds)
#pragma unroll
      for (int i = 0; i < PER; ++i) tile[(row0 + i) * TILE + col] = s_abort ? __int_as_float(0x7fc00000) : acc[i];
    cluster_sync();
    if (const int t = THREADS - 1 - (int)threadIdx.x; t < TILE + NT) {      // (threads that have the least to do below)
      uint32_t size[MAX_SPLIT];                                  // (all runs' on their way at once)
#pragma unroll
      for (int q = 0; q < MAX_SPLIT; ++q) size[q] = q < p.split ? cluster_load(&s_size[t], (uint32_t)q) : 0u;
      s_small[t] = (size[0] | size[1] | size[2] | size[3]) == 0x100;
      again = s_small[t];
    }
    // the runs in order
    for (int e = threadIdx.x; e < share * (TILE / 4); e += THREADS) {
      const int r = first + e / (TILE / 4), c = 4 * (e % (TILE / 4));
      if (m0 + r >= p.M || n0 + c >= p.N) continue;
      float4 run[MAX_SPLIT];
#pragma unroll
      for (int q = 0; q < MAX_SPLIT; ++q)
        if (q < p.split) run[q] = cluster_load4(tile + r * TILE + c, (uint32_t)q);
      float4 sum = run[0];
#pragma unroll
      for (int q = 1; q < MAX_SPLIT; ++q)
        if (q < p.split) { sum.x += run[q].x; sum.y += run[q].y; sum.z += run[q].z; sum.w += run[q].w; }
      float* at = p.C + (size_t)(m0 + r) * p.ldc + n0 + c;
      const float v[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (n0 + c + i < p.N) {
          at[i] = v[i];
          again |= doubtful(v[i]);
        }
    }
    cluster_sync();                                              // the others read in here
  }
  if (__syncthreads_or(again) && !s_abort)                       // by the row's and the column's own values: any batch, the same bits
    for (int e = threadIdx.x; e < share * TILE; e += THREADS) {
      const int r = first + e / TILE, c = e % TILE, m = m0 + r, n = n0 + c;
      if (m >= p.M || n >= p.N) continue;
      float* at = p.C + (size_t)m * p.ldc + n;
      if (s_small[c] || s_small[TILE + r] || doubtful(*at)) *at = by_multiply_adds(p.A + (size_t)m * p.lda, p.W + (size_t)n * p.K, p.K);
    }
  if (s_abort) give_up_delay();
  tc_fence_after();
  if (warp == ALLOC_WARP) tmem_dealloc(tmem_base, tmem_cols(NT));
}

constexpr size_t smem_bytes(int nt) { return 1024 + (size_t)stages_of(nt) * stage_bytes(nt) + (2 * stages_of(nt) + 5) * 8 + 16; }

template <int NT>
cudaError_t launch(const Params& p, cudaStream_t stream) {
  static std::atomic<uint64_t> done{0};
  const cudaError_t e = nhv_allow_smem((const void*)gemm_f32_tcgen05_kernel<NT>, (int)smem_bytes(NT), done);
  if (e != cudaSuccess) return e;
  return nhv_launch_cluster(gemm_f32_tcgen05_kernel<NT>, dim3((p.N + TILE - 1) / TILE * p.split, (p.M + NT - 1) / NT), THREADS,
                            smem_bytes(NT), stream, p.split, p);
}

}  // namespace

NHV_API int nhv_gemm_f32_tcgen05_error() { return nhv_wait_error_take(); }
NHV_API void* nhv_gemm_f32_tcgen05_error_word() { return nhv_wait_error_address(); }

// C [M, N] (rows ldc apart) = A [M, K] (rows lda apart) W [N, K]^T, all fp32; K and lda multiples of 4, A and W on 16-byte
// boundaries.
NHV_API int nhv_gemm_f32_tcgen05(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldc, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  NHV_REQUIRE(M > 0 && N > 0 && K > 0 && lda >= K && ldc >= N, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
  NHV_REQUIRE(K % 4 == 0 && lda % 4 == 0 && ((uintptr_t)A % 16) == 0 && ((uintptr_t)W % 16) == 0,
              "gemm_f32: rows of %d elements do not start on 16-byte boundaries", K);
  const int tiles_n = (N + TILE - 1) / TILE;
  NHV_REQUIRE((M + 127) / 128 <= 65535, "gemm_f32: M=%d is beyond the grid's reach", M);
  Params p{C, A, W, M, N, K, lda, ldc, 1, 0};
  // Runs of K: by N and K alone, so that a value does not depend on M.  Narrow matrices leave SMs idle: 128 rows, one run / two
  // (four for N = 1,024): 4096 x 1024 36 / 23 us, 6144 x 1024 37 / 23; for 370 rows, where the SMs are full, 37 / 43 and 39 / 43.
  const int all = (K + BK - 1) / BK;
  while (p.split < MAX_SPLIT && tiles_n * p.split < 50 && all >= 8 * p.split) p.split *= 2;
  p.run = (all + p.split - 1) / p.split * BK;
  NHV_CUDA(M <= 32 ? launch<32>(p, stream) : launch<128>(p, stream), "gemm_f32");
  return 0;
}
