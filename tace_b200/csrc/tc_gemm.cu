// FP32-accurate dense GEMM on the 5th-generation tensor cores (tcgen05 + TMEM + TMA): every fp32 linear whose widths are
// multiples of 64 and 32 - per-rank and per-species linears (tace/models/linear.py:377-481), the SO(2) linears of the edge
// block, and the layers of the radial MLP where they are evaluated per edge (tace/models/linear.py:267-276).
//
//   C[M, N] = A[M, K] @ B[N, K]^T        (both operands K-major, C row-major, all fp32)
//
// Plain TF32 (10-bit mantissa) is too coarse for the 1e-5 eV/atom parity target, so every
// operand is split into a TF32-exact high part and a residual, x = hi + lo, and the product is
// accumulated as hi*hi + hi*lo + lo*hi in the FP32 TMEM accumulator (the dropped lo*lo term is
// ~2^-22 relative).  Linears whose callers know the largest element of every row take FP16 parts of scaled operands
// instead (tc_gemm_fp16.cuh).  The weight operand B is split once on the host.  The activation operand A is split by the kernel
// right after its TMA load: one thread per row reads the row's 128 bytes (in the swizzled order the TMA engine wrote)
// and stores the high parts and the residuals to tensor memory, from where the tensor core takes its A operand
// (`tcgen05.mma` with A in TMEM, B from shared memory).
//
// One persistent CTA per SM walks its share of 128 x BN output tiles with specialised warps: a TMA
// producer fills a ring of {A, B_hi, B_lo} per 32-wide K step (four stages at BN = 128, six at BN = 64),
// four warps split A, one warp (through its elected lane) issues the tcgen05.mma instructions into one of two TMEM
// accumulators, and eight epilogue warps drain the other accumulator (tcgen05.ld of their 32 lanes, rows stored whole), so
// loads, splitting, tensor-core work and stores overlap.  The tensor core adds into its accumulator with truncation, an error that
// grows linearly with the number of accumulated instructions; long K loops are therefore cut
// into chunks of kChunk steps whose partial sums are drained from TMEM and added in FP32
// registers with round-to-nearest.  Every mbarrier wait is bounded: on expiry the CTA records an error code in
// global memory, stops waiting, drains and frees its TMEM, and returns.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include <cstring>
#include <cstdlib>

#include "../../include/tace_b200.h"
#include "kernels.h"

namespace tace {

namespace {

constexpr int kBM = 128;      // rows per tile = TMEM lanes
constexpr int kBK = 32;       // fp32 elements per K step = one 128-byte swizzle row
constexpr int kChunk = 8;     // K steps accumulated inside TMEM before draining into FP32 registers
constexpr int kTileABytes = kBM * kBK * 4;  // 16 KB
constexpr uint32_t kSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred P1;\n mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n selp.b32 %0, 1, 0, P1;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok;
}
// Bounded wait.  Returns false (and raises the CTA-wide abort flag) when the limit is hit.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* error, int code,
                                          uint32_t limit) {
  if (mbar_try_wait(bar, parity)) return !*abort_flag;  // the common case costs one probe
  for (uint32_t it = 0; it < limit; ++it) {
    if (mbar_try_wait(bar, parity)) return !*abort_flag;
    if ((it & 1023u) == 0u && *abort_flag) return false;
  }
  *abort_flag = 1;
  atomicCAS(error, 0, code);
  return false;
}
// The same for a warp whose lanes go on together: the lanes may read the abort flag at different times, and what follows a wait
// are instructions for all of them (tcgen05.ld / st, __syncwarp), so all leave when one does.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* error, int code, uint32_t limit) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, error, code, limit));
}
// K-major operand tile with 128-byte rows and 128-byte swizzle: 8-row groups are 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);  // start address
  d |= (uint64_t)1 << 16;                          // leading byte offset (unused for this layout)
  d |= (uint64_t)(1024 >> 4) << 32;                // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                          // descriptor version of sm_100
  d |= (uint64_t)2 << 61;                          // SWIZZLE_128B
  return d;
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n .reg .pred P1;\n elect.sync _|P1, 0xffffffff;\n selp.b32 %0, 1, 0, P1;\n}\n" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void umma_tf32_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n}\n"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}

// One linear problem of a launch: C[(atom, m), :] = A[(atom, m), 0:K] @ B[0:N, 0:K]^T (+ bias).
// Rows are (atom, component) pairs; the 3-D tensor map of A is {K, q, atoms} with box {32, q, R},
// R = 128 / q atoms per tile, so a tile's rows land in shared memory in (atom, m) order.
// Several products can share a result: their K ranges are walked one after the other in the same accumulators.
struct TcSegment {
  CUtensorMap tmA, tmBhi, tmBlo;  // B maps are 3-D {K, N, groups}; FP16: A {32, q, atoms, K/32}, tmBhi {32, N, K/32, groups} over packed weights
  const float* b_inv;    // FP16: inverse scales of the weights' columns, [groups][N]
  const unsigned* a_top; // FP16: bits of the largest |element| of the rows of atom i at [i * a_top_stride]
  int a_top_stride;
  int num_k;             // 32-wide K steps
  int b_tiled;           // B maps are 4-D {32, N, K/32, groups} over K-tile-major weights
};
struct TcProblem {
  float* C;
  const float* bias;     // [N] (per group) or nullptr
  long long c_s1, c_s2;  // atom stride / component stride of C rows (elements)
  long long bias_group_stride;
  int q, R, n_atoms, N;
  int seg0, n_seg, num_k;  // first of its segments, their number, K steps of all of them
  int row_tiles;         // of a plain problem
  // per-species problems: atoms are sorted by species, group g owns atoms [group_ptr[g], group_ptr[g+1]) and
  // R-atom tiles [tile_ptr[g], tile_ptr[g+1]); both arrays live in device memory.  n_groups == 0: one group.
  int n_groups;
  const int* group_ptr;
  const int* tile_ptr;
  const int* atom_map;   // row of C for sorted atom a is atom_map[a]; nullptr: identity
  int accumulate;        // C += instead of C =
  int table;             // offset of its row pointers in the kernel's shared-memory tables, -1: read from global memory
  int copy_table;        // not yet copied for an earlier problem
};
constexpr int kTcMaxProblems = kMaxLinears;
struct TcBatch {
  TcSegment seg[kTcMaxProblems];
  TcProblem p[kTcMaxProblems];
  int n_problems, n_segments;
  int tile_start[kTcMaxProblems + 1];  // prefix sum of the problems' tile counts
  int* error;
  uint32_t spin_limit;   // polls per wait before a role gives up (kSpinLimit; smaller in the test mode)
  uint32_t extra_tx;     // test mode: bytes added to what the first load barrier expects, so that it never completes
};

// Warp roles (448 threads): warp 0 = TMA producer, warp 1 = MMA issuer, warps 2, 3, 8, 9 = operand splitters (one per TMEM lane
// quarter), warps 4..7 and 10..13 = epilogue (warp w owns the TMEM lanes 32 * (w % 4) .. + 31; the second four take the right
// half of the columns, so that 64 running sums per thread fit its registers and a tile drains in half the time).
//
// The activation operand of the tensor-core instructions lives in tensor memory.  The splitters read the tile the TMA
// unit wrote and store its high part and residual to TMEM (one thread per row = TMEM lane), so a stage needs no room for
// them in shared memory: 48 KB at BN = 128, i.e. four K-steps in flight (six at BN = 64), and the tensor core reads only the weight
// operand from shared memory.
template <int BN>
struct TcSmem {
  static constexpr int kStages = BN == 128 ? 4 : 6;
  static constexpr int kTileBBytes = BN * kBK * 4;
  static constexpr int kStageBytes = kTileABytes + 2 * kTileBBytes;
  static constexpr int kThreads = 448, kSplitWarps = 4, kEpilogueThreads = 256;
  static constexpr int kTmemCols = 512;                  // accumulators [0, 2 BN) | per stage 32 columns high part, 32 residual
  static constexpr int kTmemA = 2 * BN;                  // first activation column
  static constexpr int kBarrierBytes = 256;  // and the tile counts of the problems
  // result staging: per epilogue warp sixteen rows x 32 columns, and the addresses of its 32 rows
  static constexpr int kStoreBytes = 8 * 16 * 128, kRowBytes = 8 * 32 * 8;
  // row pointers of the species and tile tables of the grouped problems, copied in once (a tile is found by a search over them)
  static constexpr int kTableInts = 1536;
  static constexpr int kTotal = kStages * kStageBytes + kStoreBytes + kRowBytes + kBarrierBytes + 4 * kTableInts + 1024;  // + alignment slack
};

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z)
      : "memory");
}

__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z, int w) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}

// Result path of an epilogue warp: lane r holds 32 consecutive columns of row r.  Sixteen rows at a time go through shared
// memory (16-byte chunk j of row r at chunk j ^ (r & 7)) and leave as whole 128-byte rows, eight lanes per row: stored straight
// from the registers, every 16-byte store touched 32 rows, and that, not the tensor core, bounded the linears with few K steps.
__device__ __forceinline__ void store_slab(unsigned char* slab, const uint32_t (&rr)[32], const float* bias, float* const* rows, int col,
                                           bool accumulate, int lane) {
  const int sub = lane & 7;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if ((lane >> 4) == h) {
      float4* row = reinterpret_cast<float4*>(slab + (lane & 15) * 128);
#pragma unroll
      for (int q4 = 0; q4 < 8; ++q4)
        row[q4 ^ (lane & 7)] = make_float4(__uint_as_float(rr[4 * q4]), __uint_as_float(rr[4 * q4 + 1]), __uint_as_float(rr[4 * q4 + 2]),
                                           __uint_as_float(rr[4 * q4 + 3]));
    }
    __syncwarp();
    float* dst[4];
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = 4 * i + (lane >> 3);
      dst[i] = rows[16 * h + r];
      v[i] = *reinterpret_cast<const float4*>(slab + r * 128 + ((sub ^ (r & 7)) << 4));
    }
    if (bias) {
      const float4 b = *reinterpret_cast<const float4*>(bias + 4 * sub);
#pragma unroll
      for (int i = 0; i < 4; ++i) { v[i].x += b.x; v[i].y += b.y; v[i].z += b.z; v[i].w += b.w; }
    }
    if (accumulate) {  // every load before the first store: a load that follows a store to its line waits for it
      float4 o[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) o[i] = dst[i] ? *reinterpret_cast<const float4*>(dst[i] + col + 4 * sub) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) { v[i].x += o[i].x; v[i].y += o[i].y; v[i].z += o[i].z; v[i].w += o[i].w; }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (dst[i]) *reinterpret_cast<float4*>(dst[i] + col + 4 * sub) = v[i];
    __syncwarp();
  }
}

struct TileInfo {
  int prob, atom0, atom_end, group, n0, num_k;
};
// tile_start: prefix sums of the problems' tile counts (in shared memory: grouped problems only know
// their tile count on the device); tables: per grouped problem its tile_ptr, then group_ptr (P.table: offset, -1: not copied)
template <int BN>
__device__ __forceinline__ TileInfo decode_tile(const TcBatch& b, const int* tile_start, const int* tables, int tile) {
  int pi = 0;
  while (pi + 1 < b.n_problems && tile >= tile_start[pi + 1]) ++pi;
  const TcProblem& P = b.p[pi];
  const int local = tile - tile_start[pi];
  const int tiles_n = P.N / BN;
  const int mt = local / tiles_n;
  TileInfo t;
  t.prob = pi;
  t.n0 = (local - mt * tiles_n) * BN;
  t.num_k = P.num_k;
  if (P.n_groups > 0) {
    const int* tile_ptr = P.table >= 0 ? tables + P.table : P.tile_ptr;
    const int* group_ptr = P.table >= 0 ? tables + P.table + P.n_groups + 1 : P.group_ptr;
    int lo = 0, hi = P.n_groups;  // largest g with tile_ptr[g] <= mt
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tile_ptr[mid] <= mt) lo = mid; else hi = mid;
    }
    t.group = lo;
    t.atom0 = group_ptr[lo] + (mt - tile_ptr[lo]) * P.R;
    t.atom_end = group_ptr[lo + 1];
  } else {
    t.group = 0;
    t.atom0 = mt * P.R;
    t.atom_end = P.n_atoms;
  }
  return t;
}

// ONE_CHUNK: every K loop of the launch fits one TMEM accumulation chunk, so the epilogue stores
// straight from the drained registers and needs no running sums.
template <int BN, bool ONE_CHUNK>
__global__ void __launch_bounds__(TcSmem<BN>::kThreads, 1) tc_gemm_kernel(const __grid_constant__ TcBatch batch) {
  using S = TcSmem<BN>;
  constexpr int kStages = S::kStages;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;  // 128-byte-swizzled tiles need 1024-byte alignment
  unsigned char* base_ptr = smem_raw + (base - raw);
  const uint32_t store_base = base + kStages * S::kStageBytes;  // 1024-byte aligned: stage sizes are multiples of 1024
  const uint32_t bars = store_base + S::kStoreBytes + S::kRowBytes;
  float** row_addr = reinterpret_cast<float**>(base_ptr + kStages * S::kStageBytes + S::kStoreBytes);  // [8 warps][32]
  int* tables = reinterpret_cast<int*>(base_ptr + kStages * S::kStageBytes + S::kStoreBytes + S::kRowBytes + S::kBarrierBytes);
  // barriers: raw[s] TMA landed | ready[s] operands split | empty[s] MMAs done reading | acc_full[a] | acc_empty[a]
  auto raw_bar = [&](int s) { return bars + 8u * s; };
  auto ready_bar = [&](int s) { return bars + 8u * (kStages + s); };
  auto empty_bar = [&](int s) { return bars + 8u * (2 * kStages + s); };
  auto acc_full = [&](int a) { return bars + 8u * (3 * kStages + a); };
  auto acc_empty = [&](int a) { return bars + 8u * (3 * kStages + 2 + a); };
  const uint32_t drain_bar = bars + 8u * (3 * kStages + 4);  // abort path only: issued tensor-core work has retired
  unsigned char* misc = base_ptr + kStages * S::kStageBytes + S::kStoreBytes + S::kRowBytes + 8 * (3 * kStages + 5);
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(misc);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(misc + 8);
  int* tile_start = reinterpret_cast<int*>(misc + 16);  // [n_problems + 1]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // The prologue is a third of a launch with one tile per SM (5.3 us for 288 rows of K = N = 64), so its parts run side by side:
  // warp 0 counts the tiles, a lane per problem, and has the tensor maps fetched; warp 1 allocates; warp 2 sets the barriers up;
  // the others copy the tables.
  if (warp == 0) {
    const TcProblem& P = batch.p[lane < batch.n_problems ? lane : 0];
    int count = 0;
    if (lane < batch.n_problems) count = (P.n_groups > 0 ? P.tile_ptr[P.n_groups] : P.row_tiles) * (P.N / BN);
    int sum = count;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    if (lane <= kTcMaxProblems) tile_start[lane] = sum - count;  // past the last problem: the total
    for (int m = lane; m < 3 * batch.n_segments; m += 32) {
      const TcSegment& G = batch.seg[m / 3];
      prefetch_map(m % 3 == 0 ? &G.tmA : m % 3 == 1 ? &G.tmBhi : &G.tmBlo);
    }
  }
  if (warp > 2)
    for (int i = 0; i < batch.n_problems; ++i) {
      const TcProblem& P = batch.p[i];
      if (P.n_groups > 0 && P.copy_table)
        for (int k = tid - 96; k <= P.n_groups; k += S::kThreads - 96) {
          tables[P.table + k] = P.tile_ptr[k];
          tables[P.table + P.n_groups + 1 + k] = P.group_ptr[k];
        }
    }
  if (tid == 64) {  // `ready` takes one arrival per splitter warp
    for (int s = 0; s < kStages; ++s) { mbar_init(raw_bar(s), 1); mbar_init(ready_bar(s), S::kSplitWarps); mbar_init(empty_bar(s), 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(acc_full(a), 1); mbar_init(acc_empty(a), S::kEpilogueThreads); }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {  // two accumulators of BN fp32 columns
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)tmem_slot)), "r"(S::kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;

  const int n_tiles = tile_start[batch.n_problems];
  // instruction descriptor: D = F32, A = B = TF32, both K-major, N = BN, M = 128
  const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
  auto stage_a = [&](int s) { return base + s * S::kStageBytes; };
  constexpr int kBOff = kTileABytes;  // weights follow the activation tile
  auto stage_bhi = [&](int s) { return base + s * S::kStageBytes + kBOff; };
  auto stage_blo = [&](int s) { return base + s * S::kStageBytes + kBOff + S::kTileBBytes; };

  if (warp == 0) {
    // ---- TMA producer
    if (lane == 0) {
      int step = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
        const TileInfo t = decode_tile<BN>(batch, tile_start, tables, tile);
        const TcProblem& P = batch.p[t.prob];
        const uint32_t a_bytes = (uint32_t)P.R * P.q * kBK * 4;
        const TcSegment* G = &batch.seg[P.seg0];
        int left = G->num_k, ks = 0;  // K steps left in the segment, position in it
        for (int k = 0; k < t.num_k; ++k, ++ks, --left, ++step) {
          if (left == 0) { ++G; left = G->num_k; ks = 0; }
          const int s = step % kStages, ph = (step / kStages) & 1;
          if (!mbar_wait(empty_bar(s), ph ^ 1, abort_flag, batch.error, 1, batch.spin_limit)) { ok = false; break; }
          mbar_expect_tx(raw_bar(s), a_bytes + 2 * S::kTileBBytes + batch.extra_tx);
          tma_load_3d(stage_a(s), &G->tmA, raw_bar(s), ks * kBK, 0, t.atom0);
          if (G->b_tiled) {  // weights stored K-tile-major: one contiguous block per (k-step, n-tile)
            tma_load_4d(stage_bhi(s), &G->tmBhi, raw_bar(s), 0, t.n0, ks, t.group);
            tma_load_4d(stage_blo(s), &G->tmBlo, raw_bar(s), 0, t.n0, ks, t.group);
          } else {
            tma_load_3d(stage_bhi(s), &G->tmBhi, raw_bar(s), ks * kBK, t.n0, t.group);
            tma_load_3d(stage_blo(s), &G->tmBlo, raw_bar(s), ks * kBK, t.n0, t.group);
          }
        }
      }
      if (*abort_flag) {  // loads already issued must land before the CTA exits
        for (int j = step > kStages ? step - kStages : 0; j < step; ++j) {
          const int s = j % kStages, ph = (j / kStages) & 1;
          for (uint32_t it = 0; it < batch.spin_limit; ++it)
            if (mbar_try_wait(raw_bar(s), ph)) break;
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer.  One thread issues every tensor-core instruction of the SM, and its own instruction stream is part of
    // what the ring waits for.  The whole warp walks the loop, so that control flow is warp-uniform and descriptors, addresses and
    // counters can live in uniform registers, where the tensor-core instructions take them from; only those instructions are
    // guarded by the elected lane.  Descriptors are built once (only their 14-bit start-address field, in 16-byte units, changes
    // from stage to stage and from one 8-wide K slice to the next), stage index and phase are counted instead of divided.
    // 75 776 x 512 x 1 024: 388 -> 365 us, with K = 256: 684 -> 621 us at 526 000 rows, against a loop inside `if (lane == 0)`.
    {
      const bool leader = elect_one();
      const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
      const uint64_t dB0 = umma_desc(stage_bhi(0)), dBl0 = umma_desc(stage_blo(0));
      int chunk = 0, s = 0, ph = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
        const int num_k = __shfl_sync(0xffffffffu, decode_tile<BN>(batch, tile_start, tables, tile).num_k, 0);
        for (int ks = 0; ks < num_k; ++ks, ph ^= (s == kStages - 1), s = (s == kStages - 1) ? 0 : s + 1) {
          const int a = chunk & 1;
          const bool chunk_begin = (ks % kChunk) == 0;
          const bool chunk_end = (ks % kChunk) == kChunk - 1 || ks == num_k - 1;
          if (chunk_begin) ok = mbar_wait(acc_empty(a), ((chunk >> 1) & 1) ^ 1, abort_flag, batch.error, 4, batch.spin_limit);
          ok = ok && mbar_wait(ready_bar(s), ph, abort_flag, batch.error, 2, batch.spin_limit);
          if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }  // as in warp_wait, one vote for both waits
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t d = tmem + a * BN;
          const uint64_t stage_off = (uint64_t)((uint32_t)(s * S::kStageBytes) >> 4);
          if (leader) {
#pragma unroll
            for (int k8 = 0; k8 < kBK / 8; ++k8) {
              const uint64_t off = stage_off + (uint64_t)(k8 * 2);  // 8 fp32 = 32 bytes along K inside the swizzled row
              const uint64_t db = dB0 + off, dbl = dBl0 + off;
              // activations: 8 TMEM columns per slice, high part at +0, residual at +32 of the stage
              const uint32_t ta = tmem + (uint32_t)(S::kTmemA + s * 64 + k8 * 8);
              umma_tf32_ts(d, ta, db, idesc, (!chunk_begin || k8 > 0) ? 1u : 0u);
              umma_tf32_ts(d, ta, dbl, idesc, 1u);
              umma_tf32_ts(d, ta + 32, db, idesc, 1u);
            }
            umma_commit(empty_bar(s));  // ring slot reusable once these MMAs have read it
            if (chunk_end) umma_commit(acc_full(a));  // partial sum of this chunk complete
          }
          __syncwarp();
          if (chunk_end) ++chunk;
        }
      }
      if (leader && *abort_flag) {  // tensor-core work already issued must retire before the tensor memory is given back
        umma_commit(drain_bar);
        for (uint32_t it = 0; it < batch.spin_limit; ++it)
          if (mbar_try_wait(drain_bar, 0)) break;
      }
    }
  } else if (warp < 4 || warp == 8 || warp == 9) {
    // ---- operand splitters: A = hi + lo with hi exact in TF32
    int step = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
      const TileInfo t = decode_tile<BN>(batch, tile_start, tables, tile);
      for (int ks = 0; ks < t.num_k; ++ks, ++step) {
        const int s = step % kStages, ph = (step / kStages) & 1;
        if (!warp_wait(raw_bar(s), ph, abort_flag, batch.error, 3, batch.spin_limit)) { ok = false; break; }
        // one thread per row (= TMEM lane): the row's eight 16-byte pieces sit at positions j ^ (row & 7) of its 128 bytes
        // (the swizzle the TMA unit wrote); high parts go to 32 TMEM columns of the stage, residuals to the next 32
        const int row = (warp & 3) * 32 + lane;
        const float4* arow = reinterpret_cast<const float4*>(base_ptr + s * S::kStageBytes + row * 128);
        uint32_t hi[32], lo[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 v = arow[j ^ (row & 7)];
          const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint32_t h = __float_as_uint(x[q]) & 0xFFFFE000u;
            hi[4 * j + q] = h;
            lo[4 * j + q] = __float_as_uint(x[q] - __uint_as_float(h));
          }
        }
        const uint32_t ta = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(S::kTmemA + s * 64);
        tmem_st32(ta, hi);
        tmem_st32(ta + 32, lo);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(ready_bar(s));
      }
    }
  } else {
    // ---- epilogue: drain each chunk's partial sum from TMEM, add in FP32 registers, store at tile end
    const int ew = warp & 3;  // a warp may only touch TMEM lanes 32 * (warp % 4) .. + 31
    const int half = warp >= 10 ? 1 : 0;
    constexpr int HN = BN / 2;  // columns of this warp: [half * HN, half * HN + HN)
    unsigned char* slab = base_ptr + kStages * S::kStageBytes + (half * 4 + ew) * 16 * 128;
    float** rows = row_addr + (half * 4 + ew) * 32;
    float accr[ONE_CHUNK ? 1 : HN];
    int chunk = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
      const TileInfo t = decode_tile<BN>(batch, tile_start, tables, tile);
      const TcProblem& P = batch.p[t.prob];
      {  // addresses of this warp's 32 rows (every warp keeps its own: no barrier that a warp giving up could leave others at)
        const int r = ew * 32 + lane;
        const int al = r / P.q, m = r - al * P.q;
        const bool valid = r < P.R * P.q && t.atom0 + al < t.atom_end;
        long long atom = t.atom0 + al;
        if (valid && P.atom_map) atom = P.atom_map[atom];
        __syncwarp();
        rows[lane] = valid ? P.C + atom * P.c_s1 + (long long)m * P.c_s2 + t.n0 : nullptr;
        __syncwarp();
      }
      const float* bias = P.bias ? P.bias + t.group * P.bias_group_stride + t.n0 : nullptr;
      const bool accumulate = P.accumulate != 0;
      const int n_chunks = (t.num_k + kChunk - 1) / kChunk;
      for (int cin = 0; cin < n_chunks; ++cin, ++chunk) {
        const int a = chunk & 1;
        if (!warp_wait(acc_full(a), (chunk >> 1) & 1, abort_flag, batch.error, 5, batch.spin_limit)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int c = 0; c < HN / 32; ++c) {
          uint32_t rr[32];
          const int col = half * HN + c * 32;
          tmem_ld32(tmem_base + ((uint32_t)(ew * 32) << 16) + a * BN + col, rr);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if constexpr (ONE_CHUNK) {
            store_slab(slab, rr, bias ? bias + col : nullptr, rows, col, accumulate, lane);
          } else {
#pragma unroll
            for (int q = 0; q < 32; ++q) accr[c * 32 + q] = cin == 0 ? __uint_as_float(rr[q]) : accr[c * 32 + q] + __uint_as_float(rr[q]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        mbar_arrive(acc_empty(a));  // the issuer may overwrite this accumulator
        if constexpr (!ONE_CHUNK) {
          if (cin == n_chunks - 1) {
#pragma unroll
            for (int c = 0; c < HN / 32; ++c) {
              uint32_t rr[32];
#pragma unroll
              for (int q = 0; q < 32; ++q) rr[q] = __float_as_uint(accr[c * 32 + q]);
              const int col = half * HN + c * 32;
              store_slab(slab, rr, bias ? bias + col : nullptr, rows, col, accumulate, lane);
            }
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(S::kTmemCols));
}

#include "tc_gemm_fp16.cuh"

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  }
  return fn;
}

// 3-D fp32 weight tensor [groups][N][K]; box = [1][box_rows][32], 128-byte swizzle.
bool make_map_b(CUtensorMap* map, const float* ptr, int groups, long long N, long long K, long long group_stride, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)N, (cuuint64_t)groups};
  const cuuint64_t strides[2] = {(cuuint64_t)K * sizeof(float), (cuuint64_t)(groups > 1 ? group_stride : N * K) * sizeof(float)};
  const cuuint32_t box[3] = {(cuuint32_t)kBK, (cuuint32_t)box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(ptr), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// The same weights stored K-tile-major, [groups][K/32][N][32]: the 128-byte rows of one (k-step, n-tile) operand block are
// adjacent in memory, so a block that is read once from DRAM (per-species weights) streams as whole pages.
bool make_map_b_tiled(CUtensorMap* map, const float* ptr, int groups, long long N, long long K, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)kBK, (cuuint64_t)N, (cuuint64_t)(K / kBK), (cuuint64_t)groups};
  const cuuint64_t strides[3] = {(cuuint64_t)kBK * sizeof(float), (cuuint64_t)N * kBK * sizeof(float), (cuuint64_t)N * K * sizeof(float)};
  const cuuint32_t box[4] = {(cuuint32_t)kBK, (cuuint32_t)box_rows, 1, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(ptr), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// 3-D fp32 tensor [atoms][q][K]; box = [R atoms][q][32], 128-byte swizzle.
bool make_map_3d(CUtensorMap* map, const float* ptr, long long atoms, int q, long long K, long long atom_stride,
                 long long comp_stride, int R) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)q, (cuuint64_t)atoms};
  const cuuint64_t strides[2] = {(cuuint64_t)(q == 1 ? atom_stride : comp_stride) * sizeof(float),
                                 (cuuint64_t)atom_stride * sizeof(float)};
  const cuuint32_t box[3] = {(cuuint32_t)kBK, (cuuint32_t)q, (cuuint32_t)R};
  const cuuint32_t estr[3] = {1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(ptr), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Two K steps per load: {32, rows..., K/32} maps with a box of two in the last K dimension.  A: [K/32][atoms][q][32], box [2][R][q][32]
bool make_map_a_pairs(CUtensorMap* map, const float* ptr, long long atoms, int q, long long K, long long atom_stride, long long comp_stride, int R) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[4] = {kBK, (cuuint64_t)q, (cuuint64_t)atoms, (cuuint64_t)(K / kBK)};
  const cuuint64_t strides[3] = {(cuuint64_t)(q == 1 ? atom_stride : comp_stride) * sizeof(float), (cuuint64_t)atom_stride * sizeof(float),
                                 kBK * sizeof(float)};
  const cuuint32_t box[4] = {kBK, (cuuint32_t)q, (cuuint32_t)R, 2};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(ptr), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// B: [groups][N][K] or, tiled, [groups][K/32][N][32]; box [1][2][box_rows][32]
bool make_map_b_pairs(CUtensorMap* map, const float* ptr, int groups, long long N, long long K, long long group_stride, bool tiled, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return false;
  const cuuint64_t dims[4] = {kBK, (cuuint64_t)N, (cuuint64_t)(K / kBK), (cuuint64_t)groups};
  const cuuint64_t strides[3] = {(cuuint64_t)(tiled ? kBK : K) * sizeof(float), (cuuint64_t)(tiled ? N * kBK : kBK) * sizeof(float),
                                 (cuuint64_t)(groups > 1 ? group_stride : N * K) * sizeof(float)};
  const cuuint32_t box[4] = {kBK, (cuuint32_t)box_rows, 2, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(ptr), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Function attributes and the SM count belong to a device, not to the process: one slot per device ordinal.
constexpr int kMaxDevices = 64;

template <int BN, bool ONE_CHUNK>
cudaError_t launch_tc(const TcBatch& b, int dev, int sms, cudaStream_t s) {
  static bool configured[kMaxDevices] = {};
  using S = TcSmem<BN>;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(tc_gemm_kernel<BN, ONE_CHUNK>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int tiles = b.tile_start[b.n_problems];  // upper bound for per-species problems
  const int grid = tiles < sms ? tiles : sms;
  tc_gemm_kernel<BN, ONE_CHUNK><<<grid, S::kThreads, S::kTotal, s>>>(b);
  return cudaGetLastError();
}

template <int BN>
cudaError_t launch_tc_fp16(const TcBatch& b, int dev, int sms, cudaStream_t s) {
  static bool configured[kMaxDevices] = {};
  using S = Fp16Smem<BN>;
  if (!configured[dev]) {
    cudaError_t e = cudaFuncSetAttribute(tc_gemm_fp16_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kTotal);
    if (e != cudaSuccess) return e;
    configured[dev] = true;
  }
  const int tiles = b.tile_start[b.n_problems];
  tc_gemm_fp16_kernel<BN><<<tiles < sms ? tiles : sms, S::kThreads, S::kTotal, s>>>(b);
  return cudaGetLastError();
}

}  // namespace

// Test mode of the bounded waits (tace_tc_gemm_set_test_mode): a short poll limit, and a byte count added to what the
// load barriers expect so that they never complete; both 0 in normal operation.
static uint32_t g_test_spin_limit = 0, g_test_extra_tx = 0;
void tc_gemm_set_test_mode(uint32_t spin_limit, uint32_t extra_tx) { g_test_spin_limit = spin_limit; g_test_extra_tx = extra_tx; }

// FP16 where the results of a launch take more than three K steps on average: 75 776 x 512 rows with K = 96 take 48.0 us as TF32 and 47.9 as FP16, with
// K = 128 55.5 and 48.1, 526 336 x 128 with K = 128 98.6 and 85.2.
bool tc_fp16_pays(long long results, long long steps) { return steps > 3 * results; }
bool tc_linear_supported(int N, int K) { return N % 64 == 0 && K % kBK == 0; }

cudaError_t launch_tc_linear(const TcLinearProblem* probs, int n_problems, int* error_flag, cudaStream_t s, bool any_length) {
  if (n_problems <= 0) return cudaSuccess;
  if (n_problems > kTcMaxProblems || !error_flag) return cudaErrorInvalidValue;
  static int sms_of[kMaxDevices] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidValue;
  if (!sms_of[dev] && cudaDeviceGetAttribute(&sms_of[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return cudaErrorInvalidValue;
  const int sms = sms_of[dev];
  bool all128 = true, one = true, fp16 = true;
  int first[kTcMaxProblems + 1], n_results = 0, steps_of[kTcMaxProblems];  // results: runs of problems joined to their first one
  for (int i = 0; i < n_problems; ++i) {
    const TcLinearProblem& h = probs[i];
    if (!tc_linear_supported(h.N, h.K) || h.q < 1 || h.q > 128 || (h.a_atom_stride & 3) || (h.a_comp_stride & 3) || (h.c_s1 & 3) ||
        (h.c_s2 & 3))
      return cudaErrorInvalidValue;
    fp16 = fp16 && h.a_top && h.B && h.b_inv && !(reinterpret_cast<uintptr_t>(h.b_inv) & 15);
    if (h.join) {
      if (i == 0 || h.q != probs[i - 1].q || h.N != probs[i - 1].N || h.n_atoms != probs[i - 1].n_atoms || h.n_groups != probs[i - 1].n_groups)
        return cudaErrorInvalidValue;
      steps_of[n_results - 1] += h.K / kBK;
    } else {
      first[n_results] = i;
      steps_of[n_results++] = h.K / kBK;
    }
    all128 = all128 && (h.N % 128 == 0);
  }
  first[n_results] = n_problems;
  for (int i = 0; i < n_results; ++i) { one = one && steps_of[i] <= kChunk; fp16 = fp16 && first[i + 1] - first[i] <= kTcJoined; }
  // From the shapes alone: with a count of tiles, the last of them rounded up, one row more could change the kernel, and a replayed pass, whose
  // rows are those of its capacity, could take another one than the direct pass.
  long long results = 0, all_steps = 0;
  for (int i = 0; i < n_results; ++i) {
    const long long per_atom = (long long)probs[first[i]].q * probs[first[i]].N;
    results += per_atom;
    all_steps += per_atom * steps_of[i];
  }
  fp16 = fp16 && (any_length || tc_fp16_pays(results, all_steps));
  const int bn = all128 ? 128 : 64;
  TcBatch b;
  memset(&b, 0, sizeof(b));
  b.n_problems = 0;
  b.error = error_flag;
  b.spin_limit = g_test_spin_limit ? g_test_spin_limit : kSpinLimit;
  b.extra_tx = g_test_extra_tx;
  // long K loops first: tiles are dealt round robin, and the short ones fill what the long ones leave of the last round
  int order[kTcMaxProblems];
  for (int i = 0; i < n_results; ++i) {
    int j = i;
    for (; j > 0 && steps_of[order[j - 1]] < steps_of[i]; --j) order[j] = order[j - 1];
    order[j] = i;
  }
  int tiles = 0, table = 0, segs = 0;
  for (int i = 0; i < n_results; ++i) {
    const TcLinearProblem& h = probs[first[order[i]]];
    if (h.n_atoms <= 0) continue;
    TcProblem& P = b.p[b.n_problems];
    P.q = h.q; P.R = kBM / h.q; P.n_atoms = (int)h.n_atoms; P.N = h.N;
    P.C = h.C; P.bias = h.bias; P.c_s1 = h.c_s1; P.c_s2 = h.c_s2; P.bias_group_stride = h.bias_group_stride;
    P.n_groups = h.n_groups; P.group_ptr = h.group_ptr; P.tile_ptr = h.tile_ptr; P.atom_map = h.atom_map;
    P.accumulate = h.accumulate;
    P.table = -1;
    for (int k = 0; k < b.n_problems && h.n_groups > 0; ++k)  // the tables of an earlier problem
      if (b.p[k].n_groups == h.n_groups && b.p[k].tile_ptr == h.tile_ptr && b.p[k].group_ptr == h.group_ptr) P.table = b.p[k].table;
    if (h.n_groups > 0 && P.table < 0 && table + 2 * (h.n_groups + 1) <= TcSmem<128>::kTableInts) { P.table = table; P.copy_table = 1; table += 2 * (h.n_groups + 1); }
    const int groups = h.n_groups > 0 ? h.n_groups : 1;
    if (h.n_groups > 0 && (!h.group_ptr || !h.tile_ptr)) return cudaErrorInvalidValue;
    P.seg0 = segs; P.n_seg = first[order[i] + 1] - first[order[i]];
    for (int k = first[order[i]]; k < first[order[i] + 1]; ++k) {
      const TcLinearProblem& g = probs[k];
      TcSegment& G = b.seg[segs++];
      G.num_k = g.K / kBK;
      G.b_tiled = g.b_tiled;
      P.num_k += G.num_k;
      if (g.b_tiled && groups > 1 && g.b_group_stride != (long long)g.N * g.K) return cudaErrorInvalidValue;
      if (fp16) {
        G.b_inv = g.b_inv; G.a_top = g.a_top; G.a_top_stride = g.a_top_stride;
        if (!make_map_a_pairs(&G.tmA, g.A, g.n_atoms, g.q, g.K, g.a_atom_stride, g.a_comp_stride, P.R) ||
            !make_map_b_pairs(&G.tmBhi, g.B, groups, g.N, g.K, g.b_group_stride, g.b_tiled != 0, bn))
          return cudaErrorInvalidValue;
        continue;
      }
      if (!make_map_3d(&G.tmA, g.A, g.n_atoms, g.q, g.K, g.a_atom_stride, g.a_comp_stride, P.R)) return cudaErrorInvalidValue;
      if (g.b_tiled ? (!make_map_b_tiled(&G.tmBhi, g.Bhi, groups, g.N, g.K, bn) || !make_map_b_tiled(&G.tmBlo, g.Blo, groups, g.N, g.K, bn))
                    : (!make_map_b(&G.tmBhi, g.Bhi, groups, g.N, g.K, g.b_group_stride, bn) ||
                       !make_map_b(&G.tmBlo, g.Blo, groups, g.N, g.K, g.b_group_stride, bn)))
        return cudaErrorInvalidValue;
    }
    b.tile_start[b.n_problems] = tiles;
    P.row_tiles = (int)((h.n_atoms + P.R - 1) / P.R);
    tiles += (P.row_tiles + h.n_groups) * (h.N / bn);
    ++b.n_problems;
  }
  b.n_segments = segs;
  for (int i = b.n_problems; i <= kTcMaxProblems; ++i) b.tile_start[i] = tiles;
  if (tiles == 0) return cudaSuccess;
  if (fp16) return bn == 128 ? launch_tc_fp16<128>(b, dev, sms, s) : launch_tc_fp16<64>(b, dev, sms, s);
  if (bn == 128) return one ? launch_tc<128, true>(b, dev, sms, s) : launch_tc<128, false>(b, dev, sms, s);
  return one ? launch_tc<64, true>(b, dev, sms, s) : launch_tc<64, false>(b, dev, sms, s);
}

cudaError_t launch_tc_gemm(const float* A, long long lda, const float* Bhi, const float* Blo, float* C, long long ldc, int M,
                           int N, int K, int* error_flag, cudaStream_t s, const float* bias) {
  if (M <= 0) return cudaSuccess;
  TcLinearProblem h;
  memset(&h, 0, sizeof(h));
  h.A = A; h.a_atom_stride = lda; h.a_comp_stride = lda; h.q = 1; h.n_atoms = M; h.K = K;
  h.Bhi = Bhi; h.Blo = Blo; h.N = N; h.C = C; h.c_s1 = ldc; h.c_s2 = 0; h.bias = bias;
  return launch_tc_linear(&h, 1, error_flag, s);
}

cudaError_t launch_tc_pack(const float* hi, const float* lo, int groups, int N, int K, bool tiled, float* packed, float* inv, cudaStream_t s) {
  if (!hi || !lo || !packed || !inv || groups <= 0 || N <= 0 || K <= 0 || K % kBK) return cudaErrorInvalidValue;
  const long long columns = (long long)groups * N;
  tc_pack_kernel<<<(unsigned)((columns + 7) / 8), 256, 0, s>>>(hi, lo, columns, N, K / kBK, tiled, reinterpret_cast<__half*>(packed), inv);
  return cudaGetLastError();
}

}  // namespace tace

extern "C" int tace_tc_gemm_f32(const float* A, int64_t lda, const float* B_hi, const float* B_lo, float* C, int64_t ldc,
                                int32_t M, int32_t N, int32_t K, int32_t* error_flag, tace_stream_t stream) {
  if (!A || !B_hi || !B_lo || !C) return TACE_ERR_INVALID_ARGUMENT;
  cudaError_t e = tace::launch_tc_gemm(A, lda, B_hi, B_lo, C, ldc, M, N, K, error_flag, static_cast<cudaStream_t>(stream), nullptr);
  if (e == cudaErrorInvalidValue) return TACE_ERR_INVALID_ARGUMENT;
  return e == cudaSuccess ? TACE_OK : TACE_ERR_CUDA;
}

extern "C" int tace_tc_gemm_set_test_mode(uint32_t spin_limit, uint32_t extra_expected_bytes) {
  tace::tc_gemm_set_test_mode(spin_limit, extra_expected_bytes);
  return TACE_OK;
}

extern "C" int tace_tc_gemm_fp16_f32(const TaceTcOperands* operands, int32_t n_operands, int32_t n_atoms, int32_t q, int32_t N, int32_t n_groups,
                                     const int32_t* group_ptr, const int32_t* tile_ptr, float* C, const float* bias, int32_t accumulate,
                                     int32_t* error_flag, tace_stream_t stream) {
  constexpr int kMost = tace::kTcJoined;
  if (!operands || n_operands < 1 || n_operands > kMost || n_atoms < 0 || q < 1 || q > 128 || N < 64 || n_groups < 0 || !C || !error_flag ||
      (n_groups > 0 && (!group_ptr || !tile_ptr)))
    return TACE_ERR_INVALID_ARGUMENT;
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  tace::TcLinearProblem probs[kMost];
  memset(probs, 0, sizeof(probs));
  for (int i = 0; i < n_operands; ++i) {
    const TaceTcOperands& o = operands[i];
    if (!o.A || !o.A_top || !o.B_hi || !o.B_lo || !o.B_packed || o.K < 32 || !tace::tc_linear_supported(N, o.K)) return TACE_ERR_INVALID_ARGUMENT;
    const long long n = (long long)(n_groups > 0 ? n_groups : 1) * N * o.K;
    const cudaError_t e = tace::launch_tc_pack(o.B_hi, o.B_lo, n_groups > 0 ? n_groups : 1, N, o.K, n_groups > 0, o.B_packed, o.B_packed + n, s);
    if (e != cudaSuccess) return TACE_ERR_CUDA;
    tace::TcLinearProblem& h = probs[i];
    h.A = o.A; h.a_atom_stride = (long long)q * o.K; h.a_comp_stride = o.K; h.q = q; h.n_atoms = n_atoms; h.K = o.K; h.N = N;
    h.Bhi = o.B_hi; h.Blo = o.B_lo; h.B = o.B_packed; h.b_inv = o.B_packed + n; h.a_top = o.A_top; h.a_top_stride = 1;
    h.C = C; h.c_s1 = (long long)q * N; h.c_s2 = N; h.bias = bias;
    h.n_groups = n_groups; h.group_ptr = group_ptr; h.tile_ptr = tile_ptr; h.b_group_stride = (long long)N * o.K; h.bias_group_stride = N;
    h.b_tiled = n_groups > 0; h.accumulate = accumulate != 0; h.join = i > 0;
  }
  const cudaError_t e = tace::launch_tc_linear(probs, n_operands, error_flag, s, true);
  if (e == cudaErrorInvalidValue) return TACE_ERR_INVALID_ARGUMENT;
  return e == cudaSuccess ? TACE_OK : TACE_ERR_CUDA;
}
