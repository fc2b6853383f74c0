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
// radial MLP 139 / 255 -> 48 / 45 us.
// FP32 shapes that the tcgen05 kernel does not take: CUDA cores, 32 x 64 x 16 tiles, 256 threads, 2 x 4 outputs per thread.
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
  const int* tile_ptr;  // grouped launches: [n_groups+1] prefix sum of ceil(atoms_g * q / 32)
};

template <typename T>
struct GemmBatch {
  GemmProblem<T> p[kMaxProblems];
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
  const GemmProblem<double>& P = batch.p[blockIdx.z];
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
  const double* Bg = P.B + group * P.b_group_stride + col0;
  const int K = P.K, N = P.N, steps = (K + BK - 1) / BK;
  auto load = [&](int step) {
    const int s = step % ST, k0 = step * BK;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int k = k0 + 2 * (ap + 4 * h);
      const bool ok = ao >= 0 && k < K;
      cp_async16(&As[s][ar * LA + 2 * (ap + 4 * h)], ok ? P.A + ao + k : P.A, ok);
      const int c = 2 * (bp + 8 * h);
      const bool okb = k0 + bk < K && col0 + c < N;
      cp_async16(&Bs[s][bk * LB + c], okb ? Bg + (long long)(k0 + bk) * N + c : P.B, okb);
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
      *dst = v;
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) gemm_kernel(const GemmBatch<T> batch) {
  constexpr int BM = kGemmBM, BN = 64, BK = 16;
  const GemmProblem<T>& P = batch.p[blockIdx.z];
  int group, row0, M, a_begin;
  const int col0 = blockIdx.y * BN;
  if (col0 >= P.N || !gemm_tile(batch, P, group, row0, M, a_begin)) return;

  __shared__ T As[BK][BM + 4];
  __shared__ T Bs[BK][BN + 4];
  __shared__ long long a_off[BM];
  __shared__ long long c_off[BM];

  const int tid = threadIdx.x;
  if (tid < BM) gemm_row(batch, P, a_begin, row0 + tid, M, a_off[tid], c_off[tid]);
  __syncthreads();

  const T* __restrict__ Bg = P.B + group * P.b_group_stride;
  const int tx = tid % 16, ty = tid / 16;  // 16 x 16 thread grid, 2x4 outputs each
  T acc[2][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = T(0);

  for (int k0 = 0; k0 < P.K; k0 += BK) {
    // A tile: 32 rows x 16 k  (512 elements, 2 per thread); k fastest for coalescing
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int idx = tid + i * 256;
      const int r = idx / BK, kk = idx % BK;
      const long long ao = a_off[r];
      T v = T(0);
      if (ao >= 0 && k0 + kk < P.K) v = P.A[ao + k0 + kk];
      As[kk][r] = v;
    }
    // B tile: 16 k x 64 cols
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int idx = tid + i * 256;
      const int kk = idx / BN, cc = idx % BN;
      T v = T(0);
      if (k0 + kk < P.K && col0 + cc < P.N) v = Bg[(long long)(k0 + kk) * P.N + col0 + cc];
      Bs[kk][cc] = v;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      T a[2], b[4];
#pragma unroll
      for (int i = 0; i < 2; ++i) a[i] = As[kk][ty * 2 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] += a[i] * b[j];
    }
    __syncthreads();
  }

  const T* bias = P.bias ? P.bias + group * P.bias_group_stride : nullptr;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const long long co = c_off[ty * 2 + i];
    if (co < 0) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int col = col0 + tx * 4 + j;
      if (col >= P.N) continue;
      T v = acc[i][j];
      if (bias) v += bias[col];
      if (P.accumulate) v += P.C[co + col];
      P.C[co + col] = v;
    }
  }
}

// n_atoms_total: atoms covered by the launch (all groups together); sizes grid.x.
template <typename T>
inline cudaError_t launch_gemm(const GemmBatch<T>& b, long long n_atoms_total, cudaStream_t stream) {
  int maxN = 0, maxq = 0;
  for (int i = 0; i < b.n_problems; ++i) {
    maxN = b.p[i].N > maxN ? b.p[i].N : maxN;
    maxq = b.p[i].q > maxq ? b.p[i].q : maxq;
  }
  if (n_atoms_total <= 0 || maxN <= 0 || b.n_problems <= 0) return cudaSuccess;
  long long tiles = (n_atoms_total * maxq + kGemmBM - 1) / kGemmBM;
  if (b.group_ptr) tiles += b.n_groups;  // every group may end with a partial tile
  if constexpr (std::is_same<T, double>::value)
    gemm_f64_kernel<<<dim3((unsigned)tiles, (maxN + 31) / 32, b.n_problems), 128, 0, stream>>>(b);
  else
    gemm_kernel<T><<<dim3((unsigned)tiles, (maxN + 63) / 64, b.n_problems), 256, 0, stream>>>(b);
  return cudaGetLastError();
}

}  // namespace tace
