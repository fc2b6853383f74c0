// The GEMM of tc_gemm.cu on FP16 operands, for linears whose caller knows the largest element of an operand's rows of every atom or edge
// (TcLinearProblem::a_top): the SO(2) linears over edges and, of larger models without the edge block, the per-species linears and linear_down.
// Included by tc_gemm.cu, whose barriers, tile search and tensor maps it uses.
//
// FP16 has the eleven mantissa bits of TF32 at twice its rate and half its bytes, and five exponent bits instead of eight; what those
// lack is given back by powers of two: the rows that an operand has of an atom (edge) are scaled so that their largest element lies in [2^13,
// 2^14), the weights likewise, every column of the result (of every element) by a power of its own; what shares a scale is the components of
// one rank or order.  x = hi + lo with both parts rounded to nearest, and hi*hi + hi*lo + lo*hi is accumulated as in TF32: an element keeps its 22 bits
// down to 2^-16 of the largest one of its row or column, and the error of a smaller one is 2^-39 of that.  The epilogue takes the scales out of
// the sums, which is exact.  Relative error (2-norm) of normal numbers 5.4e-7 with K = 128, 1.9e-6 with K = 512 and more; as TF32 1.4e-6 and 2.3e-6.
//
// What it had to solve besides: the TF32 kernel takes .72 us per K step of a CTA with the tensor pipe busy 69 % of it, and with FP16 parts in the
// same arrangement it still took .76.  Counted with clock64 per role: an epilogue of some 6 000 cycles a tile (each role decoding its
// tiles, results stored through shared memory), 680 cycles per step in the splitters, some 550 in the issuer around 94 of instructions.
// Hence schedulers that describe tiles ahead, two sets of splitters, results that go from registers to their rows, and two K steps per
// stage (one wait, one commit, two loads).  Times beside the TF32 kernel's (us): 75 776 x 512 x 1 024 362 and 215, x 512 192 and 119, x 256 92 and 76, x 128
// 56 and 48; 526 336 x 128 x 128 99 and 85; 2 048 x 128 x 384 13.3 and 9.6.  What bounds it now: at K >= 512 the ring (192 KB in flight against some
// 4 000 cycles from a freed stage to its next products; the pipe is busy 47 to 54 % of it), at K <= 128 the memory (5.9 TB/s).  Separate rings for A and
// B (228 -> 284 us at K = 1 024), L2 prefetch of A eight steps ahead (228 -> 239), weights as one linear copy per step (no change) and pairs of SMs
// with half of the weights each (cta_group::2, 223 -> 285) were tried.
//
// One persistent CTA per SM.  Warp roles (640 threads, five warpgroups): warp 0 = TMA producer, warp 1 = MMA issuer, warps 2, 3 = tile schedulers;
// warps 4..7 and 8..11 = operand splitters, warps 12..15 and 16..19 = epilogue (warp w works on the TMEM lanes 32 * (w % 4) .. + 31; the
// second four of the epilogue take the right half of the columns, so that 64 running sums per thread fit its registers).  Registers move from
// the first warpgroup to the others: 40 + 2 * 104 + 2 * 112 of the 5 * 96 of the launch.  Every wait is bounded, as in tc_gemm.cu.
#pragma once

// Stages accumulated inside TMEM before draining into FP32 registers: 96 instructions, as in TF32, which are 512 elements of K here and 256 there.
// With four stages the error at K >= 512 is 9.8e-7 instead of 1.9e-6 (2.3e-6 as TF32), and 75 776 x 512 x 1 024 take 226.5 us instead of 220.5, the
// linears of the edge block (526 k edges) 27.5 ms instead of 27.0.
constexpr int kFp16Chunk = 8;
constexpr int kInfo = 6;       // tiles the schedulers are ahead
constexpr int kTableInts = TcSmem<128>::kTableInts;

__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
// 16 TMEM lanes (rows) x 32 columns: lane t holds, for every 8-column block b, columns 2 (t % 4) and + 1 of row t / 4 in
// r[4 b], r[4 b + 1], and of row t / 4 + 8 in r[4 b + 2], r[4 b + 3].
__device__ __forceinline__ void tmem_ld_rows(uint32_t taddr, float (&r)[16]) {
  uint32_t u[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
        "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 16; ++i) r[i] = __uint_as_float(u[i]);
}

// Power of two that brings the largest element of a row or an array into [2^13, 2^14), and its inverse.
__device__ __forceinline__ float fp16_scale(float top, float& inv) {
  const int b = min(267 - (int)(__float_as_uint(top) >> 23), 253);  // biased exponent; the limit keeps the inverse a normal number
  inv = __uint_as_float((uint32_t)(254 - b) << 23);
  return __uint_as_float((uint32_t)b << 23);
}
__device__ __forceinline__ uint32_t pack_fp16(float x0, float x1) {
  const __half2 h = __floats2half2_rn(x0, x1);
  return *reinterpret_cast<const uint32_t*>(&h);
}
// High parts of two elements times `scale`, packed; the elements become their residuals.  Both parts are rounded to nearest: 22 bits and
// a sign.
__device__ __forceinline__ uint32_t split_fp16(float& x0, float& x1, float scale) {
  const __half2 h = __floats2half2_rn(x0 * scale, x1 * scale);
  const float2 f = __half22float2(h);
  x0 = fmaf(x0, scale, -f.x);
  x1 = fmaf(x1, scale, -f.y);
  return *reinterpret_cast<const uint32_t*>(&h);
}

// Two neighbouring 8-column blocks of one row, as tmem_ld_rows left them: lanes exchange pairs so that each holds four consecutive columns, and
// four lanes write 64 consecutive bytes of the row, eight rows per store.  (Through shared memory, in rows of 128 bytes, a tile took 3 700
// cycles; stored straight from a row per lane every store touched 32 rows.)
__device__ __forceinline__ float4 gather_columns(const float* v, int odd) {  // v[0..1]: first block, v[4..5]: second block
  const float s0 = odd ? v[0] : v[4], s1 = odd ? v[1] : v[5];
  const float r0 = __shfl_xor_sync(0xffffffffu, s0, 1), r1 = __shfl_xor_sync(0xffffffffu, s1, 1);
  return odd ? make_float4(r0, r1, v[4], v[5]) : make_float4(v[0], v[1], r0, r1);
}

// What the scheduler tells the other roles about a tile; num_k = 0 ends the list.
struct alignas(64) TileSlot {
  const float* bias;
  int num_k, seg0, atom0, n0, group, rows, accumulate;
};
template <int BN>
struct Fp16Smem {
  static constexpr int kSteps = 2;  // K steps of a stage
  static constexpr int kStages = BN == 128 ? 3 : 4;
  static constexpr int kTileBBytes = BN * kBK * 4;  // both parts of a step's weights
  static constexpr int kStageBytes = kSteps * (kTileABytes + kTileBBytes);
  static constexpr int kThreads = 640, kSplitWarps = 4, kEpilogueThreads = 256;
  static constexpr int kTmemCols = 512;                  // accumulators [0, 2 BN) | per stage and step 16 columns of high parts, 16 of residuals
  static constexpr int kTmemA = 2 * BN, kTmemStage = 64, kTmemStep = kTmemStage / kSteps;
  static constexpr int kBarrierBytes = 576;              // and the tile counts of the problems
  static constexpr int kInfoBytes = kInfo * (64 + kBM * 8);  // tile descriptions and the addresses of their rows
  static constexpr int kTopBytes = kInfo * kTcJoined * (kBM + BN) * 4;  // largest elements of the tiles' rows, inverse scales of their columns
  static constexpr int kTotal = kStages * kStageBytes + kInfoBytes + kBarrierBytes + 4 * kTableInts + kTopBytes + 1024;  // + alignment slack
  static_assert(kTmemA + kTmemStage * kStages <= kTmemCols && kTotal <= 232448, "on-chip memory");
};

template <int BN>
__global__ void __launch_bounds__(Fp16Smem<BN>::kThreads, 1) tc_gemm_fp16_kernel(const __grid_constant__ TcBatch batch) {
  using S = Fp16Smem<BN>;
  constexpr int kStages = S::kStages, kSteps = S::kSteps;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;  // 128-byte-swizzled tiles need 1024-byte alignment
  unsigned char* base_ptr = smem_raw + (base - raw);
  unsigned char* after = base_ptr + kStages * S::kStageBytes;
  float** row_addr = reinterpret_cast<float**>(after);                                   // [kInfo][kBM]
  TileSlot* info = reinterpret_cast<TileSlot*>(after + kInfo * kBM * 8);                 // [kInfo]
  const uint32_t bars = base + kStages * S::kStageBytes + S::kInfoBytes;
  int* tables = reinterpret_cast<int*>(after + S::kInfoBytes + S::kBarrierBytes);
  unsigned* row_top = reinterpret_cast<unsigned*>(tables + kTableInts);  // [kInfo][kTcJoined][kBM]: largest element of a row of every segment
  float* col_inv = reinterpret_cast<float*>(row_top + kInfo * kTcJoined * kBM);  // [kInfo][kTcJoined][BN]: inverse scale of a column
  // barriers: ready[s] operands split | empty[s] MMAs done reading | raw[s] operands landed | acc_full[a] | acc_empty[a] | info_full[i] | info_empty[i] |
  // rows_full[i] addresses and scales of a tile's rows known | cols_full[i] scales of its columns
  constexpr int kRing = 3 * kStages, kBars = kRing + 5 + 4 * kInfo;
  auto ready_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (kStages + s); };
  auto raw_bar = [&](int s) { return bars + 8u * (2 * kStages + s); };
  auto acc_full = [&](int a) { return bars + 8u * (kRing + a); };
  auto acc_empty = [&](int a) { return bars + 8u * (kRing + 2 + a); };
  const uint32_t drain_bar = bars + 8u * (kRing + 4);  // abort path only: issued tensor-core work has retired
  auto info_full = [&](int i) { return bars + 8u * (kRing + 5 + i); };
  auto info_empty = [&](int i) { return bars + 8u * (kRing + 5 + kInfo + i); };
  auto rows_full = [&](int i) { return bars + 8u * (kRing + 5 + 2 * kInfo + i); };
  auto cols_full = [&](int i) { return bars + 8u * (kRing + 5 + 3 * kInfo + i); };
  unsigned char* misc = after + S::kInfoBytes + 8 * kBars;
  static_assert(8 * kBars + 16 + 4 * (kTcMaxProblems + 1) <= S::kBarrierBytes, "barriers");
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
    for (int m = lane; m < 2 * batch.n_segments; m += 32) prefetch_map(m & 1 ? &batch.seg[m >> 1].tmBhi : &batch.seg[m >> 1].tmA);
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
    for (int s = 0; s < kStages; ++s) { mbar_init(raw_bar(s), 1); mbar_init(ready_bar(s), kSteps * S::kSplitWarps); mbar_init(empty_bar(s), 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(acc_full(a), 1); mbar_init(acc_empty(a), S::kEpilogueThreads / 32); }
    mbar_init(drain_bar, 1);
    for (int i = 0; i < kInfo; ++i) { mbar_init(info_full(i), 1); mbar_init(rows_full(i), 33); mbar_init(cols_full(i), 32); mbar_init(info_empty(i), 2 + 2 * S::kSplitWarps + S::kEpilogueThreads / 32); }
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
  // instruction descriptor: D = F32, A = B = F16, both K-major, N = BN, M = 128
  const uint32_t idesc = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
  auto stage_a = [&](int s) { return base + s * S::kStageBytes; };
  auto stage_b = [&](int s) { return stage_a(s) + kSteps * kTileABytes; };  // weights follow the activations

  // every role walks the scheduler's list: slot and phase of its i-th tile
  auto slot_of = [](int i) { return i % kInfo; };
  auto phase_of = [](int i) { return (uint32_t)(i / kInfo) & 1u; };
  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
  }
  if (warp == 2 || warp == 3) {
    // -- tile schedulers, every other tile each
    bool ok = true;
    for (int i = warp - 2, tile = blockIdx.x + i * gridDim.x; ok; i += 2, tile += 2 * gridDim.x) {
      const int slot = slot_of(i);
      if (!warp_wait(info_empty(slot), phase_of(i) ^ 1u, abort_flag, batch.error, 6, batch.spin_limit)) break;
      TileSlot& d = info[slot];
      if (tile < n_tiles) {
        const TileInfo t = decode_tile<BN>(batch, tile_start, tables, tile);
        const TcProblem& P = batch.p[t.prob];
        const int rows = P.R * P.q;
        if (lane == 0) {
          d.bias = P.bias ? P.bias + t.group * P.bias_group_stride + t.n0 : nullptr;
          d.num_k = P.num_k; d.seg0 = P.seg0; d.atom0 = t.atom0; d.n0 = t.n0; d.group = t.group;
          d.rows = rows; d.accumulate = P.accumulate;
          mbar_arrive(info_full(slot));  // the producer and the issuer can begin
        }
        // A tile's description is the longest step of tiles with few rows and K steps, so two warps work on it in turn, and nothing here waits
        // for memory before all of it has been asked for: the map of the result rows, the largest elements of the rows, the scales of the columns.
        // The last two come in asynchronously and count as arrivals of their own; the splitters do not wait for the scales of the columns, which may
        // come from DRAM.  89 elements, way back through the coefficients, K = 128 (1 480 atoms): 85 us with one warp, 63 with two.
        int atom[kBM / 32], comp[kBM / 32], to[kBM / 32];
        bool valid[kBM / 32];
#pragma unroll
        for (int k = 0; k < kBM / 32; ++k) {
          const int r = k * 32 + lane, al = r / P.q;
          comp[k] = r - al * P.q;
          atom[k] = to[k] = t.atom0 + al;
          valid[k] = r < rows && atom[k] < t.atom_end;
          if (valid[k] && P.atom_map) to[k] = P.atom_map[atom[k]];
        }
        for (int g = 0; g < P.n_seg; ++g) {
          const unsigned* from = batch.seg[P.seg0 + g].a_top;
          const int stride = batch.seg[P.seg0 + g].a_top_stride;
          unsigned* top = row_top + (slot * kTcJoined + g) * kBM + lane;
#pragma unroll
          for (int k = 0; k < kBM / 32; ++k) {
            if (valid[k]) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(top + 32 * k)), "l"(from + (long long)atom[k] * stride) : "memory");
            else top[32 * k] = 0u;
          }
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(rows_full(slot)) : "memory");
        if (lane < BN / 4) {
          const long long column = (long long)t.group * P.N + t.n0 + 4 * lane;
          for (int g = 0; g < P.n_seg; ++g)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(col_inv + (slot * kTcJoined + g) * BN + 4 * lane)),
                         "l"(batch.seg[P.seg0 + g].b_inv + column) : "memory");
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(cols_full(slot)) : "memory");
#pragma unroll
        for (int k = 0; k < kBM / 32; ++k)
          row_addr[slot * kBM + k * 32 + lane] = valid[k] ? P.C + (long long)to[k] * P.c_s1 + (long long)comp[k] * P.c_s2 + t.n0 : nullptr;
      } else {
        if (lane == 0) {
          d.num_k = 0;
          mbar_arrive(info_full(slot));
        }
        ok = false;
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(rows_full(slot)) : "memory");
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(rows_full(slot));
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else if (warp == 0) {
    // -- TMA producer
    if (lane == 0) {
      int s = 0, ph = 0, stages = 0;
      bool ok = true;
      for (int i = 0; ok; ++i) {
        if (!mbar_wait(info_full(slot_of(i)), phase_of(i), abort_flag, batch.error, 6, batch.spin_limit)) break;
        const TileSlot t = info[slot_of(i)];
        mbar_arrive(info_empty(slot_of(i)));
        const TcSegment* G = &batch.seg[t.seg0];
        for (int left = t.num_k; left > 0 && ok; ++G) {
          const int num_k = G->num_k;
          left -= num_k;
          for (int ks = 0; ks < num_k; ks += kSteps) {
            if (!mbar_wait(empty_bar(s), ph ^ 1, abort_flag, batch.error, 1, batch.spin_limit)) { ok = false; break; }
            const uint32_t bar = raw_bar(s);
            mbar_expect_tx(bar, kSteps * (uint32_t)t.rows * (kBK * 4) + 2 * S::kTileBBytes + batch.extra_tx);
            // both steps in one load each; past the end of the segment they are filled with zeros
            tma_load_4d(stage_a(s), &G->tmA, bar, 0, 0, t.atom0, ks);
            tma_load_4d(stage_b(s), &G->tmBhi, bar, 0, t.n0, ks, t.group);
            ++stages;
            if (++s == kStages) { s = 0; ph ^= 1; }
          }
        }
        if (t.num_k == 0) break;
      }
      if (*abort_flag) {  // loads already issued must land before the CTA exits
        for (int j = stages > kStages ? stages - kStages : 0; j < stages; ++j)
          for (uint32_t it = 0; it < batch.spin_limit; ++it)
            if (mbar_try_wait(raw_bar(j % kStages), (j / kStages) & 1)) break;
      }
    }
  } else if (warp == 1) {
    // -- MMA issuer, as in tc_gemm_kernel: the whole warp walks the loop, the elected lane issues
    {
      const bool leader = elect_one();
      const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
      const uint64_t dB0 = umma_desc(stage_b(0));
      int chunk = 0, s = 0, ph = 0;
      bool ok = true;
      for (int i = 0; ok; ++i) {
        if (!warp_wait(info_full(slot_of(i)), phase_of(i), abort_flag, batch.error, 6, batch.spin_limit)) break;
        const int num_k = __shfl_sync(0xffffffffu, info[slot_of(i)].num_k, 0);
        int seg = __shfl_sync(0xffffffffu, info[slot_of(i)].seg0, 0);
        if (lane == 0) mbar_arrive(info_empty(slot_of(i)));
        if (num_k == 0) break;
        for (int left = num_k; left > 0 && ok;) {
          const int steps = batch.seg[seg++].num_k;  // every segment has its scale and ends a chunk
          left -= steps;
          int in_chunk = 0;
          for (int ks = 0; ks < steps; ks += kSteps) {
            const int a = chunk & 1;
            const bool chunk_begin = in_chunk == 0;
            const bool chunk_end = ++in_chunk == kFp16Chunk || ks + kSteps >= steps;
            if (chunk_begin) ok = mbar_wait(acc_empty(a), ((chunk >> 1) & 1) ^ 1, abort_flag, batch.error, 4, batch.spin_limit);
            ok = ok && mbar_wait(ready_bar(s), ph, abort_flag, batch.error, 2, batch.spin_limit);
            if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }  // as in warp_wait, one vote for both waits
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t d = tmem + a * BN;
            const uint64_t stage_off = (uint64_t)((uint32_t)(s * S::kStageBytes) >> 4);
            if (leader) {
#pragma unroll
              for (int j = 0; j < kSteps; ++j)
#pragma unroll
                for (int k = 0; k < 2; ++k) {  // 16 elements = 32 bytes along K (the residuals are the other half of the 128-byte row), 8 TMEM columns
                  const uint64_t db = dB0 + stage_off + (uint64_t)((j * S::kTileBBytes >> 4) + k * 2);
                  const uint32_t ta = tmem + (uint32_t)(S::kTmemA + s * S::kTmemStage + j * S::kTmemStep + k * 8);
                  umma_f16_ts(d, ta, db, idesc, (!chunk_begin || j > 0 || k > 0) ? 1u : 0u);
                  umma_f16_ts(d, ta, db + 4, idesc, 1u);
                  umma_f16_ts(d, ta + S::kTmemStep / 2, db, idesc, 1u);
                }
              umma_commit(empty_bar(s));  // ring slot reusable once these MMAs have read it
              if (chunk_end) umma_commit(acc_full(a));  // partial sum of this chunk complete
            }
            __syncwarp();
            if (chunk_end) { ++chunk; in_chunk = 0; }
            ph ^= (s == kStages - 1);
            s = (s == kStages - 1) ? 0 : s + 1;
          }
        }
      }
      if (leader && *abort_flag) {  // tensor-core work already issued must retire before the tensor memory is given back
        umma_commit(drain_bar);
        for (uint32_t it = 0; it < batch.spin_limit; ++it)
          if (mbar_try_wait(drain_bar, 0)) break;
      }
    }
  } else if (warp >= 4 && warp < 12) {
    // -- operand splitters: A * scale = hi + lo, both FP16; a set of four warps takes its step of every stage
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    const int set = (warp >> 2) - 1;
    int s = 0, ph = 0;
    bool ok = true;
    const int row = (warp & 3) * 32 + lane;  // one thread per row (= TMEM lane)
    for (int i = 0; ok; ++i) {
      const int slot = slot_of(i);
      if (!warp_wait(rows_full(slot), phase_of(i), abort_flag, batch.error, 6, batch.spin_limit)) break;
      const int num_k = info[slot].num_k, seg0 = num_k ? info[slot].seg0 : 0;
      const int at = set * info[slot].rows + row;  // row of the stage: the steps follow each other without a gap
      unsigned tops[kTcJoined];  // (those of segments that the tile does not have are not used)
#pragma unroll
      for (int g = 0; g < kTcJoined; ++g) tops[g] = row_top[(slot * kTcJoined + g) * kBM + row];
      __syncwarp();
      if (lane == 0) mbar_arrive(info_empty(slot));
      if (num_k == 0) break;
      int seg = seg0, left = num_k, stages = 0;  // stages: left of the segment, its steps in pairs
      float scale = 0.f;
      while (left > 0 || stages > 0) {
        if (stages == 0) {
          const int steps = batch.seg[seg].num_k, g = seg - seg0;
          stages = (steps + 1) / kSteps;
          left -= steps;
          ++seg;
          float inv;
          scale = fp16_scale(__uint_as_float(g == 0 ? tops[0] : g == 1 ? tops[1] : tops[2]), inv);
        }
        --stages;
        if (!warp_wait(raw_bar(s), ph, abort_flag, batch.error, 3, batch.spin_limit)) { ok = false; break; }
        // the row's eight 16-byte pieces sit at positions j ^ (at & 7) of its 128 bytes (the swizzle the TMA unit wrote); the columns of the
        // residuals follow those of the high parts
        const float4* arow = reinterpret_cast<const float4*>(base_ptr + s * S::kStageBytes + at * 128);
        const uint32_t ta = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(S::kTmemA + s * S::kTmemStage + set * S::kTmemStep);
        uint32_t hi[16], lo[16];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float4 v = arow[j ^ (at & 7)];
          hi[2 * j] = split_fp16(v.x, v.y, scale);
          hi[2 * j + 1] = split_fp16(v.z, v.w, scale);
          lo[2 * j] = pack_fp16(v.x, v.y);
          lo[2 * j + 1] = pack_fp16(v.z, v.w);
        }
        tmem_st16(ta, hi);
        tmem_st16(ta + 16, lo);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(ready_bar(s));
        ph ^= (s == kStages - 1);
        s = (s == kStages - 1) ? 0 : s + 1;
      }
    }
  } else if (warp >= 12) {
    // -- epilogue: drain each chunk's partial sum from TMEM, add in FP32 registers, store at tile end
    asm volatile("setmaxnreg.inc.sync.aligned.u32 112;");
    const int ew = warp & 3;  // a warp may only touch TMEM lanes 32 * (warp % 4) .. + 31
    const int half = warp >= 16 ? 1 : 0;
    constexpr int HN = BN / 2;  // columns of this warp: [half * HN, half * HN + HN)
    const int r0 = ew * 32 + (lane >> 2);  // rows of this lane: r0, + 8, + 16, + 24
    const int odd = lane & 1, c0 = half * HN + (lane & 1) * 8 + (lane & 2) * 2;  // first of its four columns in every 16
    float sum[2][HN / 32][16];  // [rows 0..15 / 16..31][32 columns], as tmem_ld_rows leaves them
    int chunk = 0;
    bool ok = true;
    for (int i = 0; ok; ++i) {
      const int slot = slot_of(i);
      if (!warp_wait(rows_full(slot), phase_of(i), abort_flag, batch.error, 6, batch.spin_limit)) break;
      const int num_k = info[slot].num_k;
      if (num_k == 0) break;
      if (!warp_wait(cols_full(slot), phase_of(i), abort_flag, batch.error, 6, batch.spin_limit)) break;
      const float* bias = info[slot].bias;
      const bool accumulate = info[slot].accumulate != 0;
      const TcSegment* G = &batch.seg[info[slot].seg0];
      const unsigned* tops = row_top + slot * kTcJoined * kBM + r0;
      int left = G->num_k;
      const float* w_inv = col_inv + slot * kTcJoined * BN + half * HN + 2 * (lane & 3);  // from this lane's first column on, as tmem_ld_rows leaves them
      for (int ks = 0; ks < num_k; ++chunk) {
        if (left == 0) { left = (++G)->num_k; tops += kBM; w_inv += BN; }
        const int n = left < kSteps * kFp16Chunk ? left : kSteps * kFp16Chunk;
        const bool first = ks == 0;
        ks += n; left -= n;
        const int a = chunk & 1;
        if (!warp_wait(acc_full(a), (chunk >> 1) & 1, abort_flag, batch.error, 5, batch.spin_limit)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t acc = tmem_base + ((uint32_t)(ew * 32) << 16) + a * BN + half * HN;
        float f[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) fp16_scale(__uint_as_float(tops[8 * k]), f[k]);
#pragma unroll
        for (int c = 0; c < HN / 32; ++c) {
          float v[2][16];
          float2 w[4];
#pragma unroll
          for (int h = 0; h < 2; ++h) tmem_ld_rows(acc + ((uint32_t)(16 * h) << 16) + 32 * c, v[h]);
#pragma unroll
          for (int k = 0; k < 4; ++k) w[k] = *reinterpret_cast<const float2*>(w_inv + 32 * c + 8 * k);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 16; ++q) {
              const float x = v[h][q] * f[2 * h + (q >> 1 & 1)];  // exact, as the other product: powers of two
              sum[h][c][q] = fmaf(x, q & 1 ? w[q >> 2].y : w[q >> 2].x, first ? 0.f : sum[h][c][q]);
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(acc_empty(a));  // the issuer may overwrite this accumulator
      }
      if (!ok) break;
      // What the stores need of the slot goes to registers first: the arrival that hands the slot back then comes after every load from
      // it, and before this tile's stores (an arrival after them waits until they have been acknowledged, some 1 000 cycles).
      float* rows[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) rows[k] = row_addr[slot * kBM + r0 + 8 * k];
      __syncwarp();
      if (lane == 0) mbar_arrive(info_empty(slot));
#pragma unroll
      for (int c = 0; c < HN / 32; ++c) {
#pragma unroll
        for (int pair = 0; pair < 2; ++pair) {
          const int col = c0 + 32 * c + 16 * pair;
          const float4 b = bias ? *reinterpret_cast<const float4*>(bias + col) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int h = 0; h < 2; ++h) {  // rows r0 + 16 h and + 8
            float* dst[2];
            float4 o[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const float4 v = gather_columns(&sum[h][c][8 * pair + 2 * k], odd);
              o[k] = make_float4(v.x + b.x, v.y + b.y, v.z + b.z, v.w + b.w);
              dst[k] = rows[2 * h + k];
            }
            if (accumulate) {  // both loads before the first store
              float4 p[2];
#pragma unroll
              for (int k = 0; k < 2; ++k) p[k] = dst[k] ? *reinterpret_cast<const float4*>(dst[k] + col) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
              for (int k = 0; k < 2; ++k) { o[k].x += p[k].x; o[k].y += p[k].y; o[k].z += p[k].z; o[k].w += p[k].w; }
            }
#pragma unroll
            for (int k = 0; k < 2; ++k)
              if (dst[k]) *reinterpret_cast<float4*>(dst[k] + col) = o[k];
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(S::kTmemCols));
}

// ---- packed weights: run when weights are set ------------------------------------------------------------------
// Every run of 32 weights (128 bytes) becomes 32 FP16 high parts and 32 residuals of the scaled weights, in place of the 32 floats: strides
// and tensor maps are those of an fp32 array, and one load brings both parts of a K step.
// A warp per column of the result; blocks of the array: [column][K / 32], or [group][K / 32][column of the group].
__global__ void __launch_bounds__(256) tc_pack_kernel(const float* __restrict__ hi, const float* __restrict__ lo, long long columns, int N, int steps, bool tiled,
                                                      __half* out, float* inv) {
  const long long col = blockIdx.x * 8LL + (threadIdx.x >> 5);
  if (col >= columns) return;
  const int lane = threadIdx.x & 31;
  const long long g = col / N, first = tiled ? g * steps * N + (col - g * N) : col * steps, stride = tiled ? N : 1;
  unsigned m = 0;
  for (int k = 0; k < steps; ++k) {
    const long long i = (first + k * stride) * 32 + lane;
    const unsigned b = __float_as_uint(hi[i] + lo[i]) & 0x7FFFFFFFu;
    if (b < 0x7F800000u && b > m) m = b;  // infinities and NaN keep what they are under any scale
  }
  float back;
  const float sc = fp16_scale(__uint_as_float(__reduce_max_sync(0xffffffffu, m)), back);
  if (lane == 0) inv[col] = back;
  for (int k = 0; k < steps; ++k) {
    const long long run = first + k * stride, i = run * 32 + lane;
    const float v = (hi[i] + lo[i]) * sc;
    const __half h = __float2half_rn(v);
    out[run * 64 + lane] = h;
    out[run * 64 + 32 + lane] = __float2half_rn(v - __half2float(h));
  }
}
