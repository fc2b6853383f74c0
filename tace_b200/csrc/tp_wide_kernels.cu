// Interaction tensor product for fp32 models with tabulated radial weights and 64 or 128 channels: a thread owns 2 NV channels of
// an edge instead of one (NV = 1; with a scalar source, where a warp takes all channels, NV = channels / 64).  (tp_kernels.cu keeps the general kernels: fp64, weights in memory, other channel counts.)
//
// What bounds the contraction is FP32 work and, just below it, the shared-memory / L1 path, so both are what this layout
// saves.  A coupling entry G is read from shared memory once per warp and edge (a broadcast 128-bit read costs two
// wavefronts) and then serves 2 NV x 32 channels; packed fp32 arithmetic (F2) takes half the issue slots; the backward pass
// sums the products x gM over a thread's channels before it applies the coupling coefficients to them (353 multiply-adds per
// thread instead of per channel at rank 3); paths are walked source rank by source rank, so neither all weights nor all
// source components are live together.  NV = 1 (16 warps per SM backward) beat NV = 2 (12 warps, half the shared-memory
// reads): 1.04 against 1.18 ms for the rank-3 backward pass below.
//
// Measured against one channel per thread, on B200 at rank 3, 128 channels, 2 283 targets, 142 222 edges: backward 1.51 -> 1.04 ms
// (0.98 since; FMA pipe 67 % busy, LSU 71 % of its wavefronts), forward 0.80 -> 0.54 ms (LSU 80 %: of 848 wavefronts per edge 368 are table
// entries, 320 coupling rows, 64 source rows; 14.4 TB/s out of L2, of 19.6 that all SMs together can read), scalar source forward 0.11 -> 0.08 ms; rank 2, 64 channels, 131 072 targets,
// 5.5 M edges: 10.4 -> 7.2 and 5.1 -> 3.9 ms; 32 targets of 42 edges: 51 -> 10 and 31 -> 13 us.
#include <cstdint>
#include "kernels.h"
#include "tp_gen.cuh"

namespace tace {

namespace {

constexpr int kWideBatch = 16;  // edges whose coupling rows are in shared memory at a time
constexpr int kWideListRows = 8;
constexpr int kPairs = 1;       // pairs of channels of a thread where source features have a rank (NV = 1 in the text above)

// Entry `it` of the part of a partial pass' row list this launch works on, -1 past its end (see tp_row in tp_kernels.cu).
__device__ __forceinline__ int wide_row(const TPArgs<float>& a, int it) {
  const int n0 = *a.row_split;
  if (a.row_part == 0) { if (it >= n0) return -1; }
  else { it += n0; if (it >= a.n_seg) return -1; }
  return a.row_ids[it];
}

__device__ __forceinline__ void interval_of(const TPArgs<float>& a, float d, int& k, float& t) {
  const float u = d * a.rt_inv_h;
  k = (int)u;
  k = k < 0 ? 0 : (k > a.rt_K - 1 ? a.rt_K - 1 : k);
  t = u - (float)k;
}

template <int D>
__device__ __forceinline__ void load_Y(const float* __restrict__ Y, long long e, float (&y)[D]) {
  const float* p = Y + e * D;
  if constexpr (D % 4 == 0) {
#pragma unroll
    for (int k = 0; k < D; k += 4) ld4(p + k, y[k], y[k + 1], y[k + 2], y[k + 3]);
  } else {
#pragma unroll
    for (int k = 0; k < D; ++k) y[k] = p[k];
  }
}

// A lane's pairs are neighbouring channels, c0 + 64 v + 2 lane and the next, and travel in one 8-byte access (the same wavefronts as
// two channels 32 apart in two accesses, half the instructions: rank 3, 128 channels, 142 222 edges backward 1 028 -> 991 us, forward
// 531 -> 521).
__device__ __forceinline__ F2 ldg_pair(const float* p) { const float2 r = __ldg(reinterpret_cast<const float2*>(p)); return F2{r.x, r.y}; }
__device__ __forceinline__ F2 ld_pair(const float* p) { const float2 r = *reinterpret_cast<const float2*>(p); return F2{r.x, r.y}; }
__device__ __forceinline__ void st_pair(float* p, const F2& v) { *reinterpret_cast<float2*>(p) = make_float2(v.x, v.y); }

// Source row of one edge and its gradient row: component k, this lane's channels.
template <int NV, int C>
struct WideRow {
  const float* x;
  float* dx;
  template <int K> __device__ __forceinline__ void load(F2 (&r)[NV]) const {
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] = ldg_pair(x + K * C + 64 * v);
  }
  template <int K> __device__ __forceinline__ void store(const F2 (&r)[NV]) const {
#pragma unroll
    for (int v = 0; v < NV; ++v) st_pair(dx + K * C + 64 * v, r[v]);
  }
};
// Message gradient of the target in shared memory, [row][C].
template <int NV, int C>
struct WideMsg {
  const float* g;
  template <int K> __device__ __forceinline__ void load(F2 (&r)[NV]) const {
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] = ld_pair(g + K * C + 64 * v);
  }
};

// Path weights of one edge from the table: per (path, pair of channels) two 16-byte pieces (a, a', b, b'), (c, c', d, d') of the
// cubics a + t (b + t (c + t d)), so that both halves of a pair arrive in neighbouring registers (tp_wide_table).  DIST paths
// are in flight ahead of the one being worked on, across the end of an edge into the next one.
template <typename TP, int P0, int NP, int NV, int C, bool ENV, bool BWD, int DIST>
struct WideWeights {
  static_assert(NP >= DIST, "ring longer than the walk");
  const float* row;       // this edge's interval, this thread's first channels: path p at row + 4 C p
  const float* row_next;  // the next edge's
  float t, u;
  float4 q[DIST][2 * NV];
  F2 wd[NV], w0[NV];      // BWD: dw/dt and (ENV) the bare weight of the path in flight
  F2 dr, du;
  template <int O> __device__ __forceinline__ void fetch(const float* r) {
#pragma unroll
    for (int j = 0; j < 2 * NV; ++j)
      q[O % DIST][j] = __ldg(reinterpret_cast<const float4*>(r + 4 * C * TP::template v_order<P0 + O>() + 128 * j));
  }
  template <int O = 0> __device__ __forceinline__ void start(const float* r) {
    if constexpr (O < DIST) { fetch<O>(r); start<O + 1>(r); }
  }
  template <int ORD> __device__ __forceinline__ void get(F2 (&w)[NV]) {
    constexpr int O = ORD - P0;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const float4 lo = q[O % DIST][2 * v], hi = q[O % DIST][2 * v + 1];
      const F2 a{lo.x, lo.y}, b{lo.z, lo.w}, c{hi.x, hi.y}, d{hi.z, hi.w};
      const F2 e = fma2s(t, d, c), f = fma2s(t, e, b);
      w[v] = fma2s(t, f, a);
      if constexpr (BWD) wd[v] = fma2s(t, fma2s(t, d, e), f);
      if constexpr (BWD && ENV) w0[v] = w[v];
      if constexpr (ENV) w[v] = mul2s(u, w[v]);
    }
    if constexpr (O + DIST < NP) fetch<O + DIST>(row);
    else if constexpr (NP % DIST == 0) fetch<O + DIST - NP>(row_next);
    else if constexpr (O == NP - 1) start(row_next);  // the ring does not line up with the walk: refill it at the end
  }
  template <int ORD> __device__ __forceinline__ void put(const F2 (&dw)[NV]) {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      dr = fma2(dw[v], wd[v], dr);
      if constexpr (ENV) du = fma2(dw[v], w0[v], du);
    }
  }
};

// ---- forward ------------------------------------------------------------------------------------------------------
// One warp per (target, path group, 64 NV channels), no barrier: lane e builds the group's coupling row of edge e of a batch
// in the warp's own shared memory, then the warp walks over the batch, the source components of the next edge and the table
// entries of the next paths on their way.  ES warps share the edges of a target when there are too few targets to fill the
// chip; their sums are added in a fixed order.
template <typename TP, int C, bool ENV, int GRP>
__device__ __forceinline__ void wide_fwd_warp(const TPArgs<float>& a, int beg, int end, int c0, float* Gs, F2 (&acc)[TP::OUTMAX][kPairs]) {
  constexpr int GS = TP::GVMAX, NX = TP::v_nx(GRP);
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < TP::OUTMAX; ++k)
#pragma unroll
    for (int v = 0; v < kPairs; ++v) acc[k][v] = F2{0.0f, 0.0f};
  if (beg >= end) return;
  const float* table = a.rtab + 4 * c0 + 4 * lane;
  const float* x0 = a.x + TP::v_x0(GRP) * C + c0 + 2 * lane;
  constexpr int ROW = 4 * C * TP::NP;
  WideWeights<TP, TP::v_p0(GRP), TP::v_np(GRP), kPairs, C, ENV, false, 2> wf;
  auto load_x = [&](int src, F2 (&x)[TP::INMAX][kPairs]) {
    const float* p = x0 + (long long)src * (TP::NX * C);
#pragma unroll
    for (int k = 0; k < NX; ++k)
#pragma unroll
      for (int v = 0; v < kPairs; ++v) x[k][v] = ldg_pair(p + k * C + 64 * v);
  };
  for (int e0 = beg; e0 < end; e0 += kWideBatch) {
    const int nb = min(kWideBatch, end - e0);
    int src = 0, k = 0;
    float t = 0.0f, u = 1.0f;
    __syncwarp();
    if (lane < nb) {
      src = a.e_src[e0 + lane];
      interval_of(a, a.dlen[e0 + lane], k, t);
      if constexpr (ENV) u = a.env[e0 + lane];
    }
    F2 xn[TP::INMAX][kPairs];
    load_x(__shfl_sync(0xffffffffu, src, 0), xn);
    wf.row_next = table + (long long)__shfl_sync(0xffffffffu, k, 0) * ROW;
    wf.start(wf.row_next);
    if (lane < nb) {
      float y[TP::D];
      load_Y<TP::D>(a.Y, e0 + lane, y);
      TP::template build_v<GRP>(y, Gs + lane * GS);
    }
    __syncwarp();
    for (int e = 0; e < nb; ++e) {
      F2 x[TP::INMAX][kPairs];
#pragma unroll
      for (int k2 = 0; k2 < NX; ++k2)
#pragma unroll
        for (int v = 0; v < kPairs; ++v) x[k2][v] = xn[k2][v];
      const int nxt = e + 1 < nb ? e + 1 : e;
      load_x(__shfl_sync(0xffffffffu, src, nxt), xn);
      wf.row = wf.row_next;
      wf.row_next = table + (long long)__shfl_sync(0xffffffffu, k, nxt) * ROW;
      wf.t = __shfl_sync(0xffffffffu, t, e);
      if constexpr (ENV) wf.u = __shfl_sync(0xffffffffu, u, e);
      TP::template fwd_v<GRP, kPairs>(x, Gs + e * GS, wf, acc);
    }
  }
}

template <typename TP, int C>
struct WideFwdShape {
  static constexpr int CW = C / (64 * kPairs);                             // channel shares of a target (gridDim.y)
  static constexpr int TPB = TP::NGV >= 3 ? 1 : 4 / TP::NGV;          // targets per block
  static constexpr int kGBytes = kWideBatch * TP::GVMAX * 4;          // coupling rows of one warp
  static constexpr int kAccBytes = TP::OUTMAX * 2 * kPairs * 32 * 4;      // sums of one warp
};

template <typename TP, int C, bool ENV, int ES, int GRP>
__device__ __forceinline__ void wide_fwd_group(const TPArgs<float>& a, int i, int es, unsigned char* smem, float* Gs) {
  using S = WideFwdShape<TP, C>;
  const int lane = threadIdx.x & 31, c0 = blockIdx.y * 64 * kPairs;
  F2 acc[TP::OUTMAX][kPairs];
  int beg = 0, end = 0;
  if (i >= 0) { beg = a.rowptr[i]; end = a.rowptr[i + 1]; }
  const int deg = end - beg;
  const int lo = ES == 1 ? beg : beg + deg * es / ES, hi = ES == 1 ? end : beg + deg * (es + 1) / ES;
  wide_fwd_warp<TP, C, ENV, GRP>(a, lo, hi, c0, Gs, acc);
  constexpr int NOUT = TP::v_nout(GRP);
  if constexpr (ES > 1) {
    float* buf = reinterpret_cast<float*>(smem) + lane;
    for (int s = 1; s < ES; ++s) {
      __syncthreads();
      if (es == s) {
#pragma unroll
        for (int k = 0; k < NOUT; ++k)
#pragma unroll
          for (int v = 0; v < kPairs; ++v) { buf[(2 * (k * kPairs + v)) * 32] = acc[k][v].x; buf[(2 * (k * kPairs + v) + 1) * 32] = acc[k][v].y; }
      }
      __syncthreads();
      if (es == 0) {
#pragma unroll
        for (int k = 0; k < NOUT; ++k)
#pragma unroll
          for (int v = 0; v < kPairs; ++v) { acc[k][v].x += buf[(2 * (k * kPairs + v)) * 32]; acc[k][v].y += buf[(2 * (k * kPairs + v) + 1) * 32]; }
      }
    }
    if (es != 0) return;
  }
  if (i < 0) return;
  float* Mi = a.M + (long long)i * TP::NM * C + c0 + 2 * lane;
#pragma unroll
  for (int k = 0; k < NOUT; ++k)
#pragma unroll
    for (int v = 0; v < kPairs; ++v) st_pair(Mi + TP::template vmap<GRP>(k) * C + 64 * v, acc[k][v]);
  if (a.top) {  // (a uniform branch: all lanes of the warp are here)
    float most[TP::L + 1];  // per rank
#pragma unroll
    for (int l = 0; l <= TP::L; ++l) most[l] = 0.0f;
#pragma unroll
    for (int k = 0; k < NOUT; ++k)
#pragma unroll
      for (int v = 0; v < kPairs; ++v) {
        const int l = TP::rank_of(TP::template vmap<GRP>(k));
        most[l] = fmaxf(most[l], fmaxf(fabsf(acc[k][v].x), fabsf(acc[k][v].y)));
      }
    unsigned mine = 0u;
#pragma unroll
    for (int l = 0; l <= TP::L; ++l) {
      const unsigned b = __reduce_max_sync(0xffffffffu, __float_as_uint(most[l]));
      if (lane == l) mine = b;
    }
    if (lane <= TP::L) atomicMax(a.top + (long long)i * (TP::L + 1) + lane, mine);
  }
}

template <typename TP, int C, bool ENV, int ES, bool LIST>
__global__ void __maxnreg__(168) tp_fwd_wide_kernel(const TPArgs<float> a) {
  using S = WideFwdShape<TP, C>;
  extern __shared__ __align__(16) unsigned char smem[];
  const int warp = threadIdx.x >> 5;
  const int grp = ES == 1 ? warp % TP::NGV : (int)blockIdx.z, es = ES == 1 ? 0 : warp, tgt = ES == 1 ? warp / TP::NGV : 0;
  constexpr int NT = ES == 1 ? S::TPB : 1;
  float* Gs = reinterpret_cast<float*>(smem + warp * S::kGBytes);
  constexpr int ROWS = LIST ? kWideListRows : 1;
  for (int r = 0; r < ROWS; ++r) {
    const int it = (blockIdx.x * ROWS + r) * NT + tgt;
    int i = it < a.n_seg ? it : -1;
    if constexpr (LIST) i = wide_row(a, it);
    if (ES == 1 && i < 0) break;
    if (grp == 0) wide_fwd_group<TP, C, ENV, ES, 0>(a, i, es, smem, Gs);
    else if (grp == 1) { if constexpr (TP::NGV > 1) wide_fwd_group<TP, C, ENV, ES, 1>(a, i, es, smem, Gs); }
    else { if constexpr (TP::NGV > 2) wide_fwd_group<TP, C, ENV, ES, 2>(a, i, es, smem, Gs); }
  }
}

// ---- backward -----------------------------------------------------------------------------------------------------
// One block per target (and, with gridDim.y > 1, per share of its edges): the message gradient of the target sits in shared
// memory, the coupling rows of a batch are built by all warps together (warp g: path group g, lane: edge), then CW warps work
// on an edge at a time.  Everything the pass produces belongs to one edge, so edges can be dealt to warps and blocks freely.
template <typename TP, int C>
struct WideBwdShape {
  static constexpr int CW = C / (64 * kPairs);       // warps per edge
  static constexpr int kWarps = CW > 1 ? 8 : 4, EW = kWarps / CW;  // edges in flight per block
  static constexpr int NRED = TP::D + 2;          // dY | dE/d(length) | dE/d(envelope)
  static constexpr int kMsgFloats = TP::NM * C, kEdgeFloats = TP::GVS + (CW > 1 ? CW * NRED : 0);
  // Edges of a batch, which costs the block two barriers: 32, so that a whole warp of lanes builds rows, where the 16 warps that fit
  // an SM by their registers then still fit its shared memory (rank 3, 128 channels: two blocks of 96 KB).  Against 16 (runs of one side
  // within 0.2 %): 64 crystals 2 641 -> 2 632 us, 1 372 atoms 563 -> 558, water box of 32 400 atoms 44 932 -> 44 610, eight of 192 atoms
  // 2 451 -> 2 439, MD step of 131 072 atoms 22 981 -> 22 928.
  static constexpr int kBatch = (16 / kWarps) * ((kMsgFloats + 32 * kEdgeFloats) * 4 + 2048) <= 224 * 1024 ? 32 : 16;
  static constexpr int kGFloats = kBatch * TP::GVS, kRedFloats = CW > 1 ? kBatch * CW * NRED : 0;
  static constexpr int kBytes = (kMsgFloats + kGFloats + kRedFloats) * 4;
};

template <int GRP, typename TP>
__device__ __forceinline__ void wide_build(int grp, const float (&y)[TP::D], float* G) {
  if constexpr (GRP < TP::NGV) {
    if (grp == GRP) TP::template build_v<GRP>(y, G + TP::v_goff(GRP));
    else wide_build<GRP + 1, TP>(grp, y, G);
  }
}

// Sums of N per-lane values over a warp in a halving exchange (warp_sums in tp_kernels.cu); N <= 16.
template <int N>
__device__ __forceinline__ float wide_warp_sums(const float (&in)[N], int lane, int& k) {
  constexpr int NP2 = N <= 1 ? 1 : N <= 2 ? 2 : N <= 4 ? 4 : N <= 8 ? 8 : 16;
  static_assert(N <= 16, "at most 16 values");
  float v[NP2];
#pragma unroll
  for (int j = 0; j < NP2; ++j) v[j] = j < N ? in[j] : 0.0f;
  k = 0;
  int off = 16;
#pragma unroll
  for (int n = NP2; n > 1; n >>= 1, off >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int j = 0; j < n / 2; ++j) {
      const float send = upper ? v[j] : v[j + n / 2];
      const float keep = upper ? v[j + n / 2] : v[j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
    if (upper) k += n / 2;
  }
  for (; off > 0; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
  if ((lane & (32 / NP2 - 1)) != 0 || k >= N) k = N;
  return v[0];
}
__device__ __forceinline__ float wide_warp_sum(float v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

template <typename TP, int C, bool ENV>
__device__ __forceinline__ void wide_bwd_row(const TPArgs<float>& a, int i, unsigned char* smem, int* esrc, int* ek, float* et, float* eu) {
  using S = WideBwdShape<TP, C>;
  constexpr int D = TP::D, ROW = 4 * C * TP::NP;
  float* gMs = reinterpret_cast<float*>(smem);
  float* Gs = gMs + S::kMsgFloats;
  float* red = Gs + S::kGFloats;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cw = warp % S::CW, ew = warp / S::CW, c0 = cw * 64 * kPairs;
  int beg = a.rowptr[i], end = a.rowptr[i + 1];
  if (gridDim.y > 1) {
    const int deg = end - beg, lo = beg + deg * (int)blockIdx.y / (int)gridDim.y;
    end = beg + deg * ((int)blockIdx.y + 1) / (int)gridDim.y;
    beg = lo;
  }
  if (beg >= end) return;
  __syncthreads();  // a previous row's readers are done
  {
    const float* gMi = a.gM + (long long)i * S::kMsgFloats;
    for (int k = tid * 4; k < S::kMsgFloats; k += S::kWarps * 32 * 4)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(gMs + k)), "l"(gMi + k) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const float* table = a.rtab + 4 * c0 + 4 * lane;
  WideMsg<kPairs, C> gm;
  gm.g = gMs + c0 + 2 * lane;
  for (int e0 = beg; e0 < end; e0 += S::kBatch) {
    const int nb = min(S::kBatch, end - e0);
    if (e0 != beg) __syncthreads();
    if (lane < nb) {
      if (warp == 0) {
        esrc[lane] = a.e_src[e0 + lane];
        interval_of(a, a.dlen[e0 + lane], ek[lane], et[lane]);
        if constexpr (ENV) eu[lane] = a.env[e0 + lane];
      }
      if (warp < TP::NGV) {
        float y[D];
        load_Y<D>(a.Y, e0 + lane, y);
        wide_build<0, TP>(warp, y, Gs + lane * TP::GVS);
      }
    }
    if (e0 == beg) asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    WideWeights<TP, 0, TP::NP, kPairs, C, ENV, true, 1> wf;
    if (ew < nb) {
      wf.row_next = table + (long long)ek[ew] * ROW;
      wf.start(wf.row_next);
    }
    for (int e = ew; e < nb; e += S::EW) {
      WideRow<kPairs, C> xs;
      xs.x = a.x + (long long)esrc[e] * (TP::NX * C) + c0 + 2 * lane;
      xs.dx = a.dxe + (long long)(e0 + e - a.e_base) * (TP::NX * C) + c0 + 2 * lane;
      wf.row = wf.row_next;
      wf.row_next = table + (long long)ek[e + S::EW < nb ? e + S::EW : e] * ROW;
      wf.t = et[e];
      if constexpr (ENV) wf.u = eu[e];
      wf.dr = F2{0.0f, 0.0f};
      wf.du = F2{0.0f, 0.0f};
      float dY[D];
#pragma unroll
      for (int k = 0; k < D; ++k) dY[k] = 0.0f;
      TP::template bwd_v<kPairs>(xs, gm, Gs + e * TP::GVS, wf, dY);
      int k;
      const float v = wide_warp_sums<D>(dY, lane, k);
      float dr = wide_warp_sum(wf.dr.x + wf.dr.y) * a.rt_inv_h, du = 0.0f;
      if constexpr (ENV) { du = wide_warp_sum(wf.du.x + wf.du.y); dr *= wf.u; }
      if constexpr (S::CW == 1) {
        if (k < D) {
          float* dst = a.dY + (long long)(e0 + e) * D + k;
          *dst = a.accumulate_dY ? *dst + v : v;
        }
        if (lane == 0) {
          float* dl = a.ddlen + (e0 + e);
          *dl = a.accumulate_ddlen ? *dl + dr : dr;
          if constexpr (ENV) {
            float* de = a.denv + (e0 + e);
            *de = a.accumulate_denv ? *de + du : du;
          }
        }
      } else {
        float* r = red + (e * S::CW + cw) * S::NRED;
        if (k < D) r[k] = v;
        if (lane == 0) { r[D] = dr; r[D + 1] = du; }
      }
    }
    if constexpr (S::CW > 1) {
      __syncthreads();
      for (int idx = tid; idx < nb * S::NRED; idx += S::kWarps * 32) {
        const int e = idx / S::NRED, k = idx - e * S::NRED;
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < S::CW; ++w) v += red[(e * S::CW + w) * S::NRED + k];
        if (k < D) {
          float* dst = a.dY + (long long)(e0 + e) * D + k;
          *dst = a.accumulate_dY ? *dst + v : v;
        } else if (k == D) {
          float* dl = a.ddlen + (e0 + e);
          *dl = a.accumulate_ddlen ? *dl + v : v;
        } else if (ENV) {
          float* de = a.denv + (e0 + e);
          *de = a.accumulate_denv ? *de + v : v;
        }
      }
    }
  }
}

template <typename TP, int C, bool ENV, bool LIST>
__global__ void __maxnreg__(128) tp_bwd_wide_kernel(const TPArgs<float> a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int esrc[32], ek[32];
  __shared__ float et[32], eu[32];
  if constexpr (LIST) {
    for (int it = blockIdx.x * kWideListRows; it < ((int)blockIdx.x + 1) * kWideListRows; ++it) {
      const int i = wide_row(a, it);
      if (i < 0) break;
      wide_bwd_row<TP, C, ENV>(a, i, smem, esrc, ek, et, eu);
    }
  } else {
    wide_bwd_row<TP, C, ENV>(a, blockIdx.x, smem, esrc, ek, et, eu);
  }
}

// ---- backward, scalar source (the first interaction) --------------------------------------------------------------------
// The message gradient of a target is D rows only, so a warp keeps it in registers over the edges it works on, for all of its C
// channels, and nothing but the sums over the channels remains to be exchanged: the D - 1 derivatives that count (that of Y_00
// does not, sh_grad), dE/d(length) and dE/d(envelope) leave one halving exchange together.  No barrier; lane e of a batch
// builds edge e's coupling row, the next edge's source row is on its way. Shares of a target's edges go to neighbouring warps.
// With the gradient rows in shared memory, two warps per edge at 128 channels and two exchanges, the LSU was 73 % busy with them;
// what is left are the table entries.  Rank 2, 64 channels, 5.5 M edges: 2.82 -> 1.94 ms; rank 3, 64 channels, 1 372 targets of 42 edges:
// 47 -> 36 us; rank 3, 128 channels, 2.8 M edges: 2.56 -> 2.16 ms, 142 222 edges: 148 -> 125 us.
template <int NV, int D>
struct WideMsgRegs {
  F2 g[D][NV];
  template <int K> __device__ __forceinline__ void load(F2 (&r)[NV]) const {
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] = g[K][v];
  }
};
template <int NV>
struct WideRowRegs {
  F2 x[NV];
  template <int K> __device__ __forceinline__ void load(F2 (&r)[NV]) const {
#pragma unroll
    for (int v = 0; v < NV; ++v) r[v] = x[v];
  }
};
template <typename TP, int C, bool ENV>
__global__ void __launch_bounds__(128, C == 64 ? 5 : 3) tp_bwd_scalar_wide_kernel(const TPArgs<float> a, int shares) {
  static_assert(TP::NX == 1 && TP::NM == TP::D, "one source component, one path per rank");
  constexpr int NV = C / 64, D = TP::D, ROW = 4 * C * TP::NP, NSUM = D + (ENV && D < 16 ? 1 : 0);
  __shared__ __align__(16) float coupling[4][kWideBatch * TP::GVS];
  __shared__ __align__(16) float4 meta[4][kWideBatch];  // source, table interval, place in it, envelope
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit = blockIdx.x * 4 + warp, i = unit / shares, share = unit - i * shares;
  if (i >= a.n_seg) return;
  int beg = a.rowptr[i], end = a.rowptr[i + 1];
  const int deg = end - beg, lo = beg + deg * share / shares;
  end = beg + deg * (share + 1) / shares;
  beg = lo;
  if (beg >= end) return;
  WideMsgRegs<NV, D> gm;
  const float* gMi = a.gM + (long long)i * (D * C) + 2 * lane;
#pragma unroll
  for (int k = 0; k < D; ++k)
#pragma unroll
    for (int v = 0; v < NV; ++v) gm.g[k][v] = ld_pair(gMi + k * C + 64 * v);
  float* Gs = coupling[warp];
  float4* ms = meta[warp];
  const float* table = a.rtab + 4 * lane;
  auto load_x = [&](int src, WideRowRegs<NV>& x) {
    const float* p = a.x + (long long)src * C + 2 * lane;
#pragma unroll
    for (int v = 0; v < NV; ++v) x.x[v] = ldg_pair(p + 64 * v);
  };
  for (int e0 = beg; e0 < end; e0 += kWideBatch) {
    const int nb = min(kWideBatch, end - e0);
    __syncwarp();
    if (lane < nb) {
      int k;
      float t, u = 1.0f;
      interval_of(a, a.dlen[e0 + lane], k, t);
      if constexpr (ENV) u = a.env[e0 + lane];
      ms[lane] = make_float4(__int_as_float(a.e_src[e0 + lane]), __int_as_float(k), t, u);
      float y[D];
      load_Y<D>(a.Y, e0 + lane, y);
      TP::template build_v<0>(y, Gs + lane * TP::GVS);
    }
    __syncwarp();
    WideWeights<TP, 0, TP::NP, NV, C, ENV, true, (NV == 1 ? TP::NP : 2)> wf;
    WideRowRegs<NV> xn;
    float4 m = ms[0];
    load_x(__float_as_int(m.x), xn);
    wf.row_next = table + (long long)__float_as_int(m.y) * ROW;
    wf.start(wf.row_next);
    for (int e = 0; e < nb; ++e) {
      const float4 mn = ms[e + 1 < nb ? e + 1 : e];
      WideRowRegs<NV> xs = xn;
      load_x(__float_as_int(mn.x), xn);
      wf.row = wf.row_next;
      wf.row_next = table + (long long)__float_as_int(mn.y) * ROW;
      wf.t = m.z;
      if constexpr (ENV) wf.u = m.w;
      m = mn;
      wf.dr = F2{0.0f, 0.0f};
      wf.du = F2{0.0f, 0.0f};
      float dY[D], sum[NSUM];
#pragma unroll
      for (int k = 0; k < D; ++k) dY[k] = 0.0f;
      TP::template bwd_v<NV>(xs, gm, Gs + e * TP::GVS, wf, dY);
#pragma unroll
      for (int k = 1; k < D; ++k) sum[k] = dY[k];
      sum[0] = (wf.dr.x + wf.dr.y) * (ENV ? wf.u * a.rt_inv_h : a.rt_inv_h);
      float du = wf.du.x + wf.du.y;
      if constexpr (NSUM > D) sum[D] = du;
      else if constexpr (ENV) du = wide_warp_sum(du);
      int k;
      const float v = wide_warp_sums<NSUM>(sum, lane, k);
      float* dst = k == 0 ? a.ddlen + (e0 + e) : a.dY + (long long)(e0 + e) * D + k;
      bool add = k == 0 ? a.accumulate_ddlen : a.accumulate_dY;
      if constexpr (NSUM > D) { if (k == D) { dst = a.denv + (e0 + e); add = a.accumulate_denv; } }
      if (k < NSUM) *dst = add ? *dst + v : v;
      if constexpr (ENV && NSUM == D) {
        if (lane == 31) { float* de = a.denv + (e0 + e); *de = a.accumulate_denv ? *de + du : du; }
      }
    }
  }
}

// ---- launchers ----------------------------------------------------------------------------------------------------
constexpr int kWideMaxDevices = 64;

// Opt-in shared memory beyond 48 KB, once per kernel and device.
template <typename K>
cudaError_t allow_smem(K kernel, int bytes, bool (&done)[kWideMaxDevices]) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kWideMaxDevices) return cudaErrorInvalidValue;
  if (done[dev] || bytes <= 48 * 1024) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done[dev] = true;
  return e;
}

template <typename TP, int C, bool ENV, int ES, bool LIST>
cudaError_t launch_wide_fwd_k(const TPArgs<float>& a, cudaStream_t s) {
  using S = WideFwdShape<TP, C>;
  static bool done[kWideMaxDevices] = {};
  constexpr int warps = ES == 1 ? TP::NGV * S::TPB : ES, nt = ES == 1 ? S::TPB : 1;
  constexpr int g = warps * S::kGBytes, acc = ES > 1 ? S::kAccBytes : 0, bytes = g > acc ? g : acc;
  auto kernel = tp_fwd_wide_kernel<TP, C, ENV, ES, LIST>;
  const cudaError_t e = allow_smem(kernel, bytes, done);
  if (e != cudaSuccess) return e;
  const int per = nt * (LIST ? kWideListRows : 1);
  kernel<<<dim3((a.n_seg + per - 1) / per, S::CW, ES == 1 ? 1 : TP::NGV), warps * 32, bytes, s>>>(a);
  return cudaGetLastError();
}
// Few targets: four warps share the edges of a (target, group), so that a cell of some dozen atoms does not walk its edge lists
// with one warp per SM.  What a share costs besides its edges (coupling rows, sums through shared memory) weighs more the fewer
// edges it has, so the line moves with their number: at 62 edges per target and 128 channels shares win up to 864 blocks
// (126 -> 115 us, 576: 76 -> 72) and are even at 1 152, at 42 edges and 64 channels up to 500 (42 -> 40 us; 864: 50 -> 57).
template <typename TP, int C, bool ENV>
cudaError_t launch_wide_fwd(const TPArgs<float>& a, cudaStream_t s) {
  if (a.row_ids) return launch_wide_fwd_k<TP, C, ENV, 1, true>(a, s);
  const long long blocks = (long long)a.n_seg * (C / 64);
  if (a.split_sums && blocks * a.n_seg <= 15LL * a.n_edges && a.n_edges >= 16LL * a.n_seg) return launch_wide_fwd_k<TP, C, ENV, 4, false>(a, s);
  return launch_wide_fwd_k<TP, C, ENV, 1, false>(a, s);
}
template <typename TP, int C, bool ENV, bool LIST>
cudaError_t launch_wide_bwd_k(const TPArgs<float>& a, cudaStream_t s) {
  using S = WideBwdShape<TP, C>;
  static bool done[kWideMaxDevices] = {};
  auto kernel = tp_bwd_wide_kernel<TP, C, ENV, LIST>;
  const cudaError_t e = allow_smem(kernel, S::kBytes, done);
  if (e != cudaSuccess) return e;
  // Blocks per target: as many as it takes to give every SM several rounds of blocks (a last round that is nearly empty
  // costs a whole one), while a share keeps at least eight edges to pay for loading the message gradient again.
  int split = 1;
  if (!LIST)
    while ((long long)a.n_seg * split < 4 * kSMs * (16 / S::kWarps) && a.n_edges >= 16LL * split * a.n_seg && split < 16) split *= 2;
  kernel<<<dim3(LIST ? (a.n_seg + kWideListRows - 1) / kWideListRows : a.n_seg, split), S::kWarps * 32, S::kBytes, s>>>(a);
  return cudaGetLastError();
}
template <typename TP, int C, bool ENV>
cudaError_t launch_wide_bwd(const TPArgs<float>& a, cudaStream_t s) {
  if constexpr (TP::NX == 1) {
    if (a.row_ids) return cudaErrorInvalidValue;  // partial passes exist where source features are exchanged, not here
    // Shares per target: warps for three rounds of what the chip holds, while a share keeps at least eight edges; down to two
    // edges while there are fewer than eight warps per SM, because then the walk over a share is all that is waited for
    // (32 targets of 42 edges: 10.5 -> 4.6 us; with 500 targets such shares cost 15 -> 19 us).
    int shares = 1;
    while (shares < 16 && (((long long)a.n_seg * shares < 3 * kSMs * 16 && a.n_edges >= 16LL * shares * a.n_seg) ||
                           ((long long)a.n_seg * shares < 8 * kSMs && a.n_edges >= 4LL * shares * a.n_seg)))
      shares *= 2;
    tp_bwd_scalar_wide_kernel<TP, C, ENV><<<(unsigned)(((long long)a.n_seg * shares + 3) / 4), 128, 0, s>>>(a, shares);
    return cudaGetLastError();
  } else {
    return a.row_ids ? launch_wide_bwd_k<TP, C, ENV, true>(a, s) : launch_wide_bwd_k<TP, C, ENV, false>(a, s);
  }
}
template <typename TP>
cudaError_t wide_fwd_t(const TPArgs<float>& a, cudaStream_t s) {
  if (a.C == 64) return a.env ? launch_wide_fwd<TP, 64, true>(a, s) : launch_wide_fwd<TP, 64, false>(a, s);
  return a.env ? launch_wide_fwd<TP, 128, true>(a, s) : launch_wide_fwd<TP, 128, false>(a, s);
}
template <typename TP>
cudaError_t wide_bwd_t(const TPArgs<float>& a, cudaStream_t s) {
  if (TP::NX > 1 && !a.dxe) return cudaErrorInvalidValue;
  if (a.C == 64) return a.env ? launch_wide_bwd<TP, 64, true>(a, s) : launch_wide_bwd<TP, 64, false>(a, s);
  return a.env ? launch_wide_bwd<TP, 128, true>(a, s) : launch_wide_bwd<TP, 128, false>(a, s);
}

}  // namespace

bool tp_wide_supported(const TPArgs<float>& a) { return a.rtab && tp_wide_channels(a.C); }

// [intervals * paths][C][4] -> per 64 channels and lane: (a, a', b, b') then (c, c', d, d') of channels 2 lane and 2 lane + 1
void tp_wide_table(const float* in, float* out, long long rows, int C) {
  for (long long r = 0; r < rows; ++r)
    for (int c = 0; c < C; ++c)
      for (int k = 0; k < 4; ++k)
        out[r * 4 * C + (c >> 6) * 256 + (k >> 1) * 128 + ((c & 63) >> 1) * 4 + (k & 1) * 2 + (c & 1)] = in[(r * C + c) * 4 + k];
}

#define TACE_TP_WIDE_DISPATCH(FN)                                         \
  if (a.n_seg <= 0) return cudaSuccess;                                   \
  if (!a.dlen || a.rt_K < 1) return cudaErrorInvalidValue;                \
  if (a.L == 1 && a.scalar_src) return FN<TPX_L1_S>(a, s);                \
  if (a.L == 1 && a.Lin == 1) return FN<TPX_L1_F>(a, s);                  \
  if (a.L == 2 && a.scalar_src) return FN<TPX_L2_S>(a, s);                \
  if (a.L == 2 && a.Lin == 1) return FN<TPX_L2_N1>(a, s);                 \
  if (a.L == 2 && a.Lin == 2) return FN<TPX_L2_F>(a, s);                  \
  if (a.L == 3 && a.scalar_src) return FN<TPX_L3_S>(a, s);                \
  if (a.L == 3 && a.Lin == 1) return FN<TPX_L3_N1>(a, s);                 \
  if (a.L == 3 && a.Lin == 2) return FN<TPX_L3_N2>(a, s);                 \
  if (a.L == 3 && a.Lin == 3) return FN<TPX_L3_F>(a, s);                  \
  return cudaErrorInvalidValue;

cudaError_t launch_tp_fwd_wide(const TPArgs<float>& a, cudaStream_t s) { TACE_TP_WIDE_DISPATCH(wide_fwd_t) }
cudaError_t launch_tp_bwd_wide(const TPArgs<float>& a, cudaStream_t s) {
  if (!a.ddlen || (a.env && !a.denv)) return cudaErrorInvalidValue;
  TACE_TP_WIDE_DISPATCH(wide_bwd_t)
}

}  // namespace tace
