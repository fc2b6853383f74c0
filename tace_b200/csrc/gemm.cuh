// Grouped, irreps-aware GEMM used for every channel-mixing linear layer.
//
//   C[row, :] (+)= A[row, 0:K] @ B[0:K, 0:N] (+ bias)
//
// Rows are (atom, m) pairs of one rank-l block: row r of a problem maps to atom r / q and
// component r % q, and its address is base + atom * s1 + (r % q) * s2, with K (resp. N)
// contiguous.  This lets one kernel read the per-rank slices of the [atom][component][channel]
// feature layout without any transposition.  A launch carries up to kMaxProblems such
// problems (one per rank l) and, for per-species weights (the reference's e3nnElementLinear,
// tace/models/linear.py:377-481), one group per chemical species: atoms are visited through
// a species-sorted permutation and group g uses B + g * b_group_stride.
//
// FP64 runs on the double-precision tensor instruction (mma.sync m8n8k4): 32 x 32 tiles, four warps of 16 x 16, K in steps of
// 16 through a ring of three cp.async stages.  The tiles are small because the systems are (a 256-atom cell has 2 304 rows in
// all ranks of a linear together: 144 tiles for 148 SMs), and what bound the former 64 x 64 CUDA-core tiles was one block per
// four SMs walking its K loop with nothing in flight: K = N = 64 on those rows 18 -> 5 us, the 10 944 x 704 x 64 GEMMs of the
// radial MLP 139 / 255 -> 48 / 45 us (64 x 64 tiles of the tensor instruction 50 / 69: too few blocks).  The layers of the radial MLP
// have their activation, or the derivative of the one before, in the epilogue (act_out, act_in): eight launches of 5 us less per
// evaluation of 256 atoms against 1 to 6 us more in the products they leave.
// FP32 runs on the CUDA cores in the same tiles: linears with so little work that a launch of the tcgen05 kernel is nothing but its
// latency, and shapes which that kernel does not take.
//
// Problems can be joined to the one before them: their products are summed in the same accumulators.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>
#include "tace_common.cuh"

namespace tace {

constexpr int kMaxProblems = 12;

template <typename T>
struct GemmProblem {
  const T* A;
  const T* B;
  T* C;
  const T* bias;        // [N] per group, or nullptr
  int q;                // components per atom in this block (2l+1)
  int N, K;
  long long a_s1, a_s2; // atom stride / component stride of A rows
  long long c_s1, c_s2; // same for C rows
  long long b_group_stride, bias_group_stride;
  int accumulate;       // 0: C = ..., 1: C += ...
  int join;             // the product is added to that of the problem before (same rows and result)
  // double precision: silu(C) stored as well, or C = result * silu'(act_in), both laid out like C; or nullptr
  T* act_out;
  const T* act_in;
  const int* tile_ptr;  // grouped launches: [n_groups+1] prefix sum of ceil(atoms_g * q / 32)
};

template <typename T>
struct GemmBatch {
  GemmProblem<T> p[kMaxProblems];
  int first[kMaxProblems + 1];  // first problem of result i (set by launch_gemm)
  int n_problems;
  int n_groups;          // 1 unless per-species
  const int* group_ptr;  // [n_groups+1] atom ranges in `atom_map` order, or nullptr (=> all atoms)
  const int* atom_map;   // row position -> atom index of A, or nullptr (identity)
  const int* c_atom_map; // row position -> atom index of C, or nullptr (identity)
  int n_atoms;           // used when group_ptr == nullptr
};

constexpr int kGemmBM = 32;  // rows per tile

// Row tile of this block: group, first row inside the group and the group's atoms; false: nothing to do.
template <typename T>
__device__ __forceinline__ bool gemm_tile(const GemmBatch<T>& batch, const GemmProblem<T>& P, int& group, int& row0, int& M, int& a_begin) {
  int tile = blockIdx.x, a_end = batch.n_atoms;
  group = 0; a_begin = 0;
  if (batch.group_ptr) {
    // blockIdx.x enumerates the (species, row tile) pairs that exist; find ours.
    const int* tp = P.tile_ptr;
    if ((int)blockIdx.x >= tp[batch.n_groups]) return false;
    int lo = 0, hi = batch.n_groups;  // largest g with tp[g] <= blockIdx.x
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (tp[mid] <= (int)blockIdx.x) lo = mid; else hi = mid;
    }
    group = lo;
    tile = blockIdx.x - tp[lo];
    a_begin = batch.group_ptr[group];
    a_end = batch.group_ptr[group + 1];
  }
  M = (a_end - a_begin) * P.q;
  row0 = tile * kGemmBM;
  return row0 < M;
}
// Element offsets of row r of the tile in A and C, -1 past the last row.
template <typename T>
__device__ __forceinline__ void gemm_row(const GemmBatch<T>& batch, const GemmProblem<T>& P, int a_begin, int row, int M, long long& ao, long long& co) {
  ao = co = -1;
  if (row >= M) return;
  const int pos = a_begin + row / P.q, m = row % P.q;
  const long long a_atom = batch.atom_map ? batch.atom_map[pos] : pos;
  const long long c_atom = batch.c_atom_map ? batch.c_atom_map[pos] : pos;
  ao = a_atom * P.a_s1 + m * P.a_s2;
  co = c_atom * P.c_s1 + m * P.c_s2;
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool ok) {
  const int size = ok ? 16 : 0;  // 0: the destination is zero-filled
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(size) : "memory");
}

static __global__ void __launch_bounds__(128) gemm_f64_kernel(const GemmBatch<double> batch) {
  constexpr int BM = kGemmBM, BN = 32, BK = 16, ST = 3;
  constexpr int LA = BK + 4, LB = BN + 4;  // leading dimensions: a fragment's rows start four 8-byte banks apart
  const int first = batch.first[blockIdx.z], last = batch.first[blockIdx.z + 1];
  const GemmProblem<double>& P = batch.p[first];
  int group, row0, M, a_begin;
  const int col0 = blockIdx.y * BN;
  if (col0 >= P.N || !gemm_tile(batch, P, group, row0, M, a_begin)) return;
  __shared__ __align__(16) double As[ST][BM * LA];
  __shared__ __align__(16) double Bs[ST][BK * LB];
  __shared__ long long c_off[BM];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // this thread's pieces of a stage: two 16-byte pieces of A (row tid / 4, pieces tid % 4 and + 4), two of B (k row tid / 8 ...)
  const int ar = tid >> 2, ap = tid & 3;
  long long ao, co;
  gemm_row(batch, P, a_begin, row0 + ar, M, ao, co);
  if (ap == 0) c_off[ar] = co;
  const int bk = tid >> 3, bp = tid & 7;
  const double *Ag = P.A, *Bg = P.B + group * P.b_group_stride + col0;
  const int N = P.N;
  int steps = 0;
  for (int i = first; i < last; ++i) steps += (batch.p[i].K + BK - 1) / BK;
  int cur = first, k0 = 0, K = P.K;  // problem and place in its K range that the next load is for
  auto load = [&](int step) {
    const int s = step % ST;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = k0 + 2 * (ap + 4 * h);
      const bool ok = ao >= 0 && k < K;
      cp_async16(&As[s][ar * LA + 2 * (ap + 4 * h)], ok ? Ag + ao + k : Ag, ok);
      const int c = 2 * (bp + 8 * h);
      const bool okb = k0 + bk < K && col0 + c < N;
      cp_async16(&Bs[s][bk * LB + c], okb ? Bg + (long long)(k0 + bk) * N + c : P.B, okb);
    }
    k0 += BK;
    if (k0 >= K && cur + 1 < last) {
      const GemmProblem<double>& Q = batch.p[++cur];
      long long unused;
      gemm_row(batch, Q, a_begin, row0 + ar, M, ao, unused);
      Ag = Q.A; Bg = Q.B + group * Q.b_group_stride + col0; K = Q.K; k0 = 0;
    }
  };
#pragma unroll
  for (int i = 0; i < ST - 1; ++i) {
    if (i < steps) load(i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  const int wr = (warp & 1) * 16, wc = (warp >> 1) * 16, fr = lane >> 2, fk = lane & 3;
  double acc[2][2][2] = {};
  for (int i = 0; i < steps; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
    __syncthreads();  // stage i has landed for everybody, and everybody is done with the stage the next load overwrites
    if (i + ST - 1 < steps) load(i + ST - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const double* A = As[i % ST];
    const double* B = Bs[i % ST];
#pragma unroll
    for (int k4 = 0; k4 < BK; k4 += 4) {
      double a[2], b[2];
#pragma unroll
      for (int m = 0; m < 2; ++m) a[m] = A[(wr + 8 * m + fr) * LA + k4 + fk];
#pragma unroll
      for (int n = 0; n < 2; ++n) b[n] = B[(k4 + fk) * LB + wc + 8 * n + fr];
#pragma unroll
      for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n)
          asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                       : "+d"(acc[m][n][0]), "+d"(acc[m][n][1]) : "d"(a[m]), "d"(b[n]));
    }
  }
  const double* bias = P.bias ? P.bias + group * P.bias_group_stride : nullptr;
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const long long at = c_off[wr + 8 * m + fr];
    if (at < 0) continue;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int col = col0 + wc + 8 * n + 2 * fk;
      if (col >= N) continue;
      double2 v = make_double2(acc[m][n][0], acc[m][n][1]);
      double2* dst = reinterpret_cast<double2*>(P.C + at + col);
      if (bias) { v.x += bias[col]; v.y += bias[col + 1]; }
      if (P.accumulate) { const double2 o = *dst; v.x += o.x; v.y += o.y; }
      if (P.act_in) {
        const double2 z = *reinterpret_cast<const double2*>(P.act_in + at + col);
        v.x *= silu_grad_(z.x); v.y *= silu_grad_(z.y);
      }
      *dst = v;
      if (P.act_out) *reinterpret_cast<double2*>(P.act_out + at + col) = make_double2(silu_(v.x), silu_(v.y));
    }
  }
}

// 32 x 32 tiles, K in steps of 32 through a ring of four cp.async stages; four sets of 64 threads with 4 x 4 outputs each take a quarter
// of every step and their sums are added at the end (with one output row per thread and no such sets, shared-memory reads bounded
// the longer K loops: 10.6 against 7.2 us for the joined products of 32 atoms, rank 2, 64 channels).  What is left is latency: 2.9 us for
// 288 rows of K = N = 64, of which a third is the launch; the tensor-core kernel takes 5.5.
static __global__ void __launch_bounds__(256) gemm_f32_kernel(const GemmBatch<float> batch) {
  constexpr int BM = kGemmBM, BN = 32, BK = 32, ST = 4, LA = BK + 4;  // rows of A start four banks apart
  const int first = batch.first[blockIdx.z], last = batch.first[blockIdx.z + 1];
  const GemmProblem<float>& P = batch.p[first];
  int group, row0, M, a_begin;
  const int col0 = blockIdx.y * BN;
  if (col0 >= P.N || !gemm_tile(batch, P, group, row0, M, a_begin)) return;
  __shared__ __align__(16) float As[ST][BM * LA];
  __shared__ __align__(16) float Bs[ST][BK * BN];
  // this thread's piece of a stage: four values of A (row r, k 4 p ...) and of B (k r, columns 4 p ...)
  const int r = threadIdx.x >> 3, p = threadIdx.x & 7, N = P.N;
  long long ao, co;
  gemm_row(batch, P, a_begin, row0 + r, M, ao, co);
  const float *Ag = P.A, *Bg = P.B + group * P.b_group_stride + col0;
  int steps = 0;
  for (int i = first; i < last; ++i) steps += (batch.p[i].K + BK - 1) / BK;
  int cur = first, k0 = 0, K = P.K;  // problem and place in its K range that the next load is for
  auto load = [&](int step) {
    float* a = &As[step % ST][r * LA + 4 * p];
    float* b = &Bs[step % ST][r * BN + 4 * p];
    const int k = k0 + 4 * p, kb = k0 + r, c = col0 + 4 * p;
    const bool ok = ao >= 0 && k < K, okb = kb < K && c < N;
    cp_async16(a, ok ? Ag + ao + k : Ag, ok);
    cp_async16(b, okb ? Bg + (long long)kb * N + 4 * p : P.B, okb);
    k0 += BK;
    if (k0 >= K && cur + 1 < last) {
      const GemmProblem<float>& Q = batch.p[++cur];
      long long unused;
      gemm_row(batch, Q, a_begin, row0 + r, M, ao, unused);
      Ag = Q.A; Bg = Q.B + group * Q.b_group_stride + col0; K = Q.K; k0 = 0;
    }
  };
#pragma unroll
  for (int i = 0; i < ST - 1; ++i) {
    if (i < steps) load(i);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  // outputs of this thread: rows tr + 8 i, columns 4 p .. 4 p + 3, summed over k = 8 set .. 8 set + 7 of every step
  const int set = threadIdx.x >> 6, tr = (threadIdx.x >> 3) & 7;
  float acc[4][4] = {};
  for (int i = 0; i < steps; ++i) {
    asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
    __syncthreads();  // stage i has landed for everybody, and everybody is done with the stage the next load overwrites
    if (i + ST - 1 < steps) load(i + ST - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* A = &As[i % ST][tr * LA + 8 * set];
    const float* B = &Bs[i % ST][8 * set * BN + 4 * p];
#pragma unroll
    for (int k = 0; k < 8; k += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        a[j] = *reinterpret_cast<const float4*>(A + 8 * j * LA + k);
        b[j] = *reinterpret_cast<const float4*>(B + (k + j) * BN);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          const float x = j == 0 ? a[m].x : j == 1 ? a[m].y : j == 2 ? a[m].z : a[m].w;
          acc[m][0] = fmaf(x, b[j].x, acc[m][0]); acc[m][1] = fmaf(x, b[j].y, acc[m][1]);
          acc[m][2] = fmaf(x, b[j].z, acc[m][2]); acc[m][3] = fmaf(x, b[j].w, acc[m][3]);
        }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* sums = &As[0][0];  // [set][32][32]: the ring is done with
  static_assert(sizeof(As) >= 4 * BM * BN * sizeof(float), "the sums of the sets reuse the ring");
#pragma unroll
  for (int m = 0; m < 4; ++m)
    *reinterpret_cast<float4*>(sums + (set * BM + tr + 8 * m) * BN + 4 * p) = make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
  __syncthreads();
  const int col = col0 + 4 * p;
  if (co < 0 || col >= N) return;
  float4 v = *reinterpret_cast<const float4*>(sums + r * BN + 4 * p);
#pragma unroll
  for (int q = 1; q < 4; ++q) {
    const float4 o = *reinterpret_cast<const float4*>(sums + (q * BM + r) * BN + 4 * p);
    v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
  }
  const float* bias = P.bias ? P.bias + group * P.bias_group_stride + col : nullptr;
  float* dst = P.C + co + col;
  if (bias) { v.x += bias[0]; v.y += bias[1]; v.z += bias[2]; v.w += bias[3]; }
  if (P.accumulate) { const float4 o = *reinterpret_cast<const float4*>(dst); v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
  *reinterpret_cast<float4*>(dst) = v;
}

// n_atoms_total: atoms covered by the launch (all groups together); sizes grid.x.
template <typename T>
inline cudaError_t launch_gemm(GemmBatch<T>& b, long long n_atoms_total, cudaStream_t stream) {
  int maxN = 0, maxq = 0, n_results = 0;
  constexpr int V = 16 / sizeof(T);
  for (int i = 0; i < b.n_problems; ++i) {
    const GemmProblem<T>& p = b.p[i];
    maxN = p.N > maxN ? p.N : maxN;
    maxq = p.q > maxq ? p.q : maxq;
    // whole 16-byte pieces everywhere: channels come in multiples of 32, other widths of four, buffers from arenas
    if (((reinterpret_cast<uintptr_t>(p.A) | reinterpret_cast<uintptr_t>(p.B) | reinterpret_cast<uintptr_t>(p.C)) & 15) != 0 ||
        (p.a_s1 | p.a_s2 | p.c_s1 | p.c_s2 | p.b_group_stride | p.K | p.N) % V != 0)
      return cudaErrorInvalidValue;
    if (p.join && (i == 0 || p.q != b.p[i - 1].q || p.N != b.p[i - 1].N)) return cudaErrorInvalidValue;
    if (!p.join) b.first[n_results++] = i;
  }
  b.first[n_results] = b.n_problems;
  if (n_atoms_total <= 0 || maxN <= 0 || b.n_problems <= 0) return cudaSuccess;
  long long tiles = (n_atoms_total * maxq + kGemmBM - 1) / kGemmBM;
  if (b.group_ptr) tiles += b.n_groups;  // every group may end with a partial tile
  const dim3 grid((unsigned)tiles, (maxN + 31) / 32, n_results);
  if constexpr (std::is_same<T, double>::value) gemm_f64_kernel<<<grid, 128, 0, stream>>>(b);
  else gemm_f32_kernel<<<grid, 256, 0, stream>>>(b);
  return cudaGetLastError();
}

}  // namespace tace
