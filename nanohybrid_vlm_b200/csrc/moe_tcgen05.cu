// The experts' products of a mixture of experts over rows ordered by expert, for prompts, on the 5th-generation
// tensor cores: tcgen05.mma by pairs of SMs with the accumulators in tensor memory, operands brought by TMA.
//
// Rows are those of moe_align (csrc/moe.cu) with tiles of 256 rows: every tile belongs to one expert.  A pair of blocks (a
// cluster of two) takes one tile of rows and 256 rows of that expert's weights, as one tcgen05.mma.cta_group::2 of
// 256 x 256 x 16: the tile's rows sit on the M axis, 128 in each block, the weight rows on the N axis, 128 brought by each
// block and read by both.  D is 128 lanes x 256 columns (fp32) per block: one row of the ordering per lane, and so per
// thread of the epilogue.
//   first:  block 0 brings 128 rows of the gate matrix, block 1 the 128 rows of the up matrix of the same output columns, so
//           that a thread finds gate and up of its row in two columns of its lane: act[row, c] = glu(gate, up);
//   second: y[row, c] = act[row] . Wd[e][c], 256 output columns;
//   for experts without a gate, first: act[row, c] = relu(x[token(row)] . Wu[e][c])^2, 256 output columns.
// The first product reads its A rows from a copy of x gathered into the order of the rows (moe_gather_rows below), so
// that a tile of rows is one TMA box.  Rows behind the middle of a tile that are padding altogether are not brought; what the
// MMAs make of them is not read.
//
// What bounds it: what the SMs take in from L2.  A product of 128 x 128 x 64 by one block brings 32 KB for 256 cycles of the
// tensor pipe, one of 256 x 256 x 64 by a pair 32 KB a block for 512: 16,300 rows of 16 experts, 2,048 columns to 1,024 and
// back, 259 + 97 us by tiles of 128 x 128, 141 + 72 by pairs (970 and 950 TFLOP/s).  At 85 rows an expert, where half of a
// pair's tile is empty and the weights' 201 MB from memory weigh most, 47 + 20 and 43 + 20.
// Two blocks share an SM (96 KB of ring and 256 of its 512 columns each), so that one's epilogue runs beside the other's
// products; one block with six stages was slower where the grid leaves SMs to one block (27 against 21 us).
//
// Warp roles: warp 0 lane 0 issues the block's TMA loads into a ring of stages (64 columns of K each, 128-byte swizzle), all
// counted on the pair's "full" barrier in block 0, which arms it for both; warp 1 allocates tensor memory, and in block 0
// its lane 0 issues the MMAs and commits them to the stage's "empty" barrier of both blocks, at the end to both
// accumulators' barriers; warps 2-9, two for each quarter of the lanes, read with tcgen05.ld and write the outputs (a
// division of the gated unit holds a warp up for some hundred cycles: with four warps the first product took 166 us instead
// of 141).  Every wait is bounded; one that runs out sets the file's error word and the block leaves through the common exit,
// where the pair meets before either frees its tensor memory.
#include <mutex>
#include <unordered_map>

#define NHV_WAIT_LIMIT (1u << 22)
#include "nhv_async.cuh"
#include "nhv_glu.cuh"

namespace {

typedef __nv_bfloat16 bf16;
constexpr int HALF = 128;              // rows of the ordering, and rows of the weights, that a block brings
constexpr int ROWS = 2 * HALF;         // rows of the ordering per pair = MMA M
constexpr int COLS = 2 * HALF;         // weight rows per pair = MMA N = columns of tensor memory
constexpr int BK = 64;                 // columns per stage = one 128-byte swizzle row
constexpr int UMMA_K = 16;
constexpr int STAGES = 3;
constexpr int THREADS = 320;           // producer warp, MMA warp, eight epilogue warps
constexpr uint32_t OPERAND_BYTES = HALF * 128, STAGE_BYTES = 2 * OPERAND_BYTES;

__device__ __forceinline__ void tmem_alloc(uint32_t* slot_in_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(slot_in_smem)), "r"(ncols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// The address of a shared variable in block 0 of the pair.
__device__ __forceinline__ uint32_t in_block0(const void* p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
// A tile of a 2-D tensor map into this block's shared memory, counted on a barrier of either block of the pair.
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n"
               ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// The pair's MMAs so far, on the barrier at this place in both blocks.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
// D[tmem of both] (+)= A[smem of both] * B[smem of both]^T, both operands K-major bfloat16
__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t (&r)[32], uint32_t taddr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }
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
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

struct alignas(64) Params {
  CUtensorMap w0_map;   // first: gate [E * N, K]; second: down [E * N, K]; boxes of 64 columns x 128 rows in all three
  CUtensorMap w1_map;   // first: up, as gate
  CUtensorMap a_map;    // the rows [rows, K]
  bf16* out;            // [rows, N]
  const int* sorted_slots;
  const int* tile_expert;
  int N, K;
  float limit, alpha, up_shift;
  const float* row_scale;     // a factor on the expert's input per (token, choice) slot, or null
};

// 32 outputs of a row, columns n to n + 31 of N: pieces of 32 bytes where the rows allow it (a whole sector a thread), else
// of 16, else one by one.
__device__ __forceinline__ void store_row(bf16* at, const float (&v)[32], int n, int N) {
  uint32_t w[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    w[i] = *reinterpret_cast<const uint32_t*>(&h);
  }
  if (n + 32 <= N && ((uintptr_t)at & 31) == 0) {
#pragma unroll
    for (int i = 0; i < 16; i += 8)
      asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(at + 2 * i), "r"(w[i]), "r"(w[i + 1]),
                   "r"(w[i + 2]), "r"(w[i + 3]), "r"(w[i + 4]), "r"(w[i + 5]), "r"(w[i + 6]), "r"(w[i + 7]) : "memory");
  } else if (n + 32 <= N && ((uintptr_t)at & 15) == 0) {
#pragma unroll
    for (int i = 0; i < 16; i += 4) *reinterpret_cast<uint4*>(at + 2 * i) = make_uint4(w[i], w[i + 1], w[i + 2], w[i + 3]);
  } else {
#pragma unroll
    for (int i = 0; i < 32; ++i)
      if (n + i < N) at[i] = __float2bfloat16_rn(v[i]);
  }
}

template <int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS, 2) moe_tcgen05_kernel(const __grid_constant__ Params p) {
  constexpr bool FIRST = MODE == 1;
  constexpr int WIDTH = FIRST ? HALF : COLS;                    // output columns of a pair
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* smem = smem_unaligned + ((1024 - (smem_u32(smem_unaligned) & 1023)) & 1023);
  unsigned char* ring = smem;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)STAGES * STAGE_BYTES);      // used in block 0, for both
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_full + 1);
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  // panels of one tile of rows are neighbours in the grid: they run together and share the tile's rows in L2, and the
  // tiles of one expert follow one another, so its weights stay there too
  const int tile = blockIdx.y;
  const int n0 = (int)(blockIdx.x >> 1) * WIDTH;
  const int kb_n = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, COLS);
  tc_fence_before();
  __syncthreads();
  cluster_sync();                                                // both blocks' barriers are there
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  pdl_launch_dependents();
  pdl_wait();                                                   // the ordering and the rows are the work of kernels before
  const int e = p.tile_expert[tile];                            // the pair's: a tile without an expert has no work
  const int row0 = tile * ROWS + (int)rank * HALF;              // this block's rows
  const bool upper = e >= 0 && p.sorted_slots[(size_t)tile * ROWS + HALF] >= 0;     // padding lies behind the slots

  if (e >= 0) {
    if (warp == 0) {
      // ------------------------------------------------------------------ TMA producer
      if (lane == 0) {
        const CUtensorMap* w_map = FIRST && rank ? &p.w1_map : &p.w0_map;
        const int w_row = e * p.N + n0 + (FIRST ? 0 : (int)rank * HALF);
        const uint32_t pair_bytes = (upper ? 4 : 3) * OPERAND_BYTES;      // zero-filled parts of a box count too
        // (STAGES rounds more than there are stages to fill: no block leaves before the last commits have reached it)
        for (int kb = 0; kb < kb_n + STAGES; ++kb) {
          const int s = kb % STAGES;
          if (kb >= STAGES && !mbar_wait(&empty[s], (uint32_t)((kb / STAGES) - 1) & 1, 1)) { s_abort = 1; break; }
          if (kb >= kb_n) continue;
          unsigned char* dst = ring + (size_t)s * STAGE_BYTES;
          const uint32_t bar = in_block0(&full[s]);
          if (rank == 0) mbar_expect_tx(&full[s], pair_bytes);
          tma_load_2d_pair(dst + OPERAND_BYTES, w_map, kb * BK, w_row, bar);
          if (rank == 0 || upper) tma_load_2d_pair(dst, &p.a_map, kb * BK, row0, bar);
        }
      }
      __syncwarp();
    } else if (warp == 1) {
      // ------------------------------------------------------------------ MMA issuer, for the pair
      if (rank == 0 && lane == 0) {
        const uint32_t idesc = instr_desc(ROWS, COLS);
        bool ok = true;
        for (int kb = 0; kb < kb_n && ok; ++kb) {
          const int s = kb % STAGES;
          ok = mbar_wait(&full[s], (uint32_t)(kb / STAGES) & 1, 2);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a_addr = smem_u32(ring + (size_t)s * STAGE_BYTES);
          const uint32_t b_addr = a_addr + OPERAND_BYTES;
#pragma unroll
          for (int kk = 0; kk < BK / UMMA_K; ++kk)
            tc_mma(tmem_base, smem_desc_sw128(a_addr + kk * UMMA_K * 2), smem_desc_sw128(b_addr + kk * UMMA_K * 2), idesc,
                   (kb == 0 && kk == 0) ? 0u : 1u);
          tc_commit(&empty[s]);                                 // the stage is free in both blocks once these MMAs have read it
        }
        if (ok) tc_commit(acc_full);
        else s_abort = 1;
      }
      __syncwarp();
    } else {
      // ------------------------------------------------------------------ epilogue (warps 2..9): half a row a thread
      const int quarter = warp & 3;                             // the tensor-memory lanes this warp may read
      const int row = row0 + quarter * 32 + lane;
      const int slot = rank == 0 || upper ? p.sorted_slots[row] : -1;
      const float scale = MODE != 0 && p.row_scale && slot >= 0 ? p.row_scale[slot] : 1.f;
      const bool ok = mbar_wait(acc_full, 0, 4);
      if (!ok) s_abort = 1;
      tc_fence_after();
      if (__all_sync(0xffffffffu, ok) && (rank == 0 || upper)) {
        const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
        bf16* out = p.out + (size_t)row * p.N;
        for (int c0 = warp >= 6 ? 32 : 0; c0 < WIDTH && n0 + c0 < p.N; c0 += 64) {
          uint32_t g[32], u[32];
          float v[32];
          tmem_ld32(g, taddr + c0);
          if (FIRST) tmem_ld32(u, taddr + HALF + c0);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            // sums rounded to the storage type before the unit, as a separate product would leave them
            const float a = __uint_as_float(g[j]);
            if (FIRST)
              v[j] = nhv_glu(round_bf16(scale * a), round_bf16(scale * __uint_as_float(u[j])), p.limit, p.alpha, p.up_shift);
            else
              v[j] = MODE == 2 ? nhv_relu_squared_unit(round_bf16(scale * a)) : a;
          }
          if (slot >= 0) store_row(out + n0 + c0, v, n0 + c0, p.N);
        }
      }
      tc_fence_before();
    }
  }
  // ------------------------------------------------------------------ common exit
  __syncthreads();
  if (s_abort) give_up_delay();                                 // let copies that may still be in flight land
  cluster_sync();                                               // the other block's MMAs, commits and copies reach in here
  tc_fence_after();
  if (warp == 1) tmem_dealloc(tmem_base, COLS);
}

constexpr size_t SMEM_BYTES = 1024 + (size_t)STAGES * STAGE_BYTES + (2 * STAGES + 1) * 8 + 16;

struct MapKey {
  const void* base;
  long long rows;
  int cols, box_rows;
  bool operator==(const MapKey& o) const { return base == o.base && rows == o.rows && cols == o.cols && box_rows == o.box_rows; }
};
struct MapKeyHash {
  size_t operator()(const MapKey& k) const {
    return std::hash<const void*>()(k.base) ^ ((size_t)k.rows * 1000003u) ^ ((size_t)k.cols << 20) ^ (size_t)k.box_rows;
  }
};
std::unordered_map<MapKey, CUtensorMap, MapKeyHash> g_weight_maps;   // weights do not move: one map per stack
std::mutex g_maps_mutex;

bool weight_map(CUtensorMap* out, const void* base, long long rows, int cols, int box_rows) {
  std::lock_guard<std::mutex> lock(g_maps_mutex);
  const MapKey key{base, rows, cols, box_rows};
  auto it = g_weight_maps.find(key);
  if (it == g_weight_maps.end()) {
    CUtensorMap m;
    if (!nhv_make_map_bf16(&m, base, rows, cols, cols, BK, box_rows)) return false;
    it = g_weight_maps.emplace(key, m).first;
  }
  *out = it->second;
  return true;
}

// A warp per row of the ordering: the token's row of x.  Padding is left as it is: what the products make of such a row
// is not written.
constexpr int GATHER_WARPS = 8;
__global__ void __launch_bounds__(GATHER_WARPS * 32) moe_gather_rows_kernel(uint4* __restrict__ out, const uint4* __restrict__ x,
                                                                           const int* __restrict__ sorted_slots, int rows,
                                                                           int top, int pieces) {
  pdl_prologue();
  const int row = blockIdx.x * GATHER_WARPS + (threadIdx.x >> 5);
  const int slot = row < rows ? sorted_slots[row] : -1;
  if (slot < 0) return;
  uint4* dst = out + (size_t)row * pieces;
  const uint4* src = x + (size_t)(slot / top) * pieces;
#pragma unroll 8
  for (int i = threadIdx.x & 31; i < pieces; i += 32) dst[i] = src[i];
}

}  // namespace

NHV_API int nhv_moe_tcgen05_error() { return nhv_wait_error_take(); }
NHV_API void* nhv_moe_tcgen05_error_word() { return nhv_wait_error_address(); }
NHV_API int nhv_moe_tcgen05_tile() { return ROWS; }

// out [rows, width] (bfloat16) = x[sorted_slots[row] / top]; rows of padding are not written.
NHV_API int nhv_moe_gather_rows(void* out, const void* x, const int* sorted_slots, int rows, int top, int width,
                                cudaStream_t stream) {
  if (rows == 0) return 0;
  NHV_REQUIRE(width % 8 == 0 && ((uintptr_t)out % 16) == 0 && ((uintptr_t)x % 16) == 0 && top > 0,
              "moe_gather_rows: rows of %d elements do not start on 16-byte boundaries", width);
  NHV_CUDA(nhv_launch(moe_gather_rows_kernel, dim3((rows + GATHER_WARPS - 1) / GATHER_WARPS), dim3(GATHER_WARPS * 32), 0, stream,
                      (uint4*)out, (const uint4*)x, sorted_slots, rows, top, width / 8), "moe_gather_rows");
  return 0;
}

// mode 1: out [rows, N] = glu(A W0[e]^T, A W1[e]^T) with A [rows, K] (the gathered rows) and W0 / W1 [E, N, K]; 2: out =
// relu(A W0[e]^T)^2 of the same rows; 0: out [rows, N] = A W0[e]^T.  rows = tiles * 256, the ordering of moe_align with tiles of 256 rows.
NHV_API int nhv_moe_gemm_tcgen05(int mode, void* out, const void* A, const void* W0, const void* W1, int n_experts,
                                 const int* sorted_slots, const int* tile_expert, int tiles, int N, int K, float limit,
                                 float alpha, float up_shift, const float* row_scale, cudaStream_t stream) {
  if (tiles == 0) return 0;
  NHV_REQUIRE(tiles > 0 && N > 0 && K > 0 && K % 8 == 0 && n_experts > 0, "moe_gemm (tcgen05): K must be a multiple of 8 (N=%d K=%d)", N, K);
  NHV_REQUIRE(((uintptr_t)A % 16) == 0 && ((uintptr_t)W0 % 16) == 0 && (mode != 1 || ((uintptr_t)W1 % 16) == 0),
              "moe_gemm (tcgen05): operands must be 16-byte aligned");
  NHV_REQUIRE((long long)n_experts * N < (1LL << 31) && (long long)tiles * ROWS < (1LL << 31), "moe_gemm (tcgen05): too many rows");
  Params p;
  NHV_REQUIRE(weight_map(&p.w0_map, W0, (long long)n_experts * N, K, HALF), "moe_gemm (tcgen05): cannot encode the weights' tensor map");
  if (mode == 1) NHV_REQUIRE(weight_map(&p.w1_map, W1, (long long)n_experts * N, K, HALF), "moe_gemm (tcgen05): cannot encode the weights' tensor map");
  else p.w1_map = p.w0_map;
  NHV_REQUIRE(nhv_make_map_bf16(&p.a_map, A, (long long)tiles * ROWS, K, K, BK, HALF), "moe_gemm (tcgen05): cannot encode the rows' tensor map");
  p.out = (bf16*)out;
  p.sorted_slots = sorted_slots;
  p.tile_expert = tile_expert;
  p.N = N;
  p.K = K;
  p.limit = limit;
  p.alpha = alpha;
  p.up_shift = up_shift;
  p.row_scale = row_scale;
  const int width = mode == 1 ? HALF : COLS;
  dim3 grid(2 * ((N + width - 1) / width), tiles);
  NHV_REQUIRE(grid.y <= 65535, "moe_gemm (tcgen05): %d tiles of rows are beyond the grid's reach", tiles);
  const int m = mode == 1 ? 1 : mode == 2 ? 2 : 0;
  auto kernel = m == 1 ? moe_tcgen05_kernel<1> : m == 2 ? moe_tcgen05_kernel<2> : moe_tcgen05_kernel<0>;
  static std::atomic<uint64_t> allowed[3];
  NHV_CUDA(nhv_allow_smem((const void*)kernel, (int)SMEM_BYTES, allowed[m]), "moe_gemm (tcgen05)");
  NHV_CUDA(nhv_launch(kernel, grid, dim3(THREADS), SMEM_BYTES, stream, p), "moe_gemm (tcgen05)");
  return 0;
}
