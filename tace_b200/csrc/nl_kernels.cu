// Cell-list neighbour list for a batch of periodic (or partly periodic) structures.
//
// Semantics follow the reference's get_neighborhood (tace/dataset/neighbour_list.py:195-298,
// which wraps matscipy's "ijS" list): full list, edge vector r_target - r_source + S @ cell,
// strict |v| < cutoff evaluated in fp64, self pairs kept unless S = 0, no shift along
// non-periodic axes.  Cells narrower than the cutoff are handled by visiting several periodic
// images of the (single) bin along that axis.
//
// Atoms are binned per structure in fractional coordinates (bins at least cutoff / r wide, r
// bins searched on either side), sorted by bin with a stable radix sort, and every target atom
// walks its neighbouring bins in a fixed order, so the output order is deterministic: grouped
// by target, then by bin, then by source index.  The distance test uses the unwrapped input
// positions and explicit round-to-nearest multiplies/adds (no FMA contraction), so the edge set
// is bit-identical to a brute-force fp64 enumeration evaluated in the same order.
#include <cub/cub.cuh>
#include <thrust/iterator/transform_iterator.h>
#include <cuda_runtime.h>
#include <cstdint>

#include "../../include/tace_b200.h"

namespace tace {
namespace {

struct GraphBins {
  double inv[9];   // frac = pos @ inv
  double cell[9];
  double fmin[3], fext[3];
  int nb[3], r[3], pbc[3];
  int bin_offset, n_bins;
};

__device__ __forceinline__ void cell_inverse(const double* __restrict__ c, double (&inv)[9]) {
  const double det = c[0] * (c[4] * c[8] - c[5] * c[7]) - c[1] * (c[3] * c[8] - c[5] * c[6]) + c[2] * (c[3] * c[7] - c[4] * c[6]);
  const double id = 1.0 / det;
  inv[0] = (c[4] * c[8] - c[5] * c[7]) * id; inv[1] = (c[2] * c[7] - c[1] * c[8]) * id; inv[2] = (c[1] * c[5] - c[2] * c[4]) * id;
  inv[3] = (c[5] * c[6] - c[3] * c[8]) * id; inv[4] = (c[0] * c[8] - c[2] * c[6]) * id; inv[5] = (c[2] * c[3] - c[0] * c[5]) * id;
  inv[6] = (c[3] * c[7] - c[4] * c[6]) * id; inv[7] = (c[1] * c[6] - c[0] * c[7]) * id; inv[8] = (c[0] * c[4] - c[1] * c[3]) * id;
}
// Bins of one structure from its inverse cell and the range of its fractional coordinates (used on open axes only).
__device__ __forceinline__ void bins_of(const double* __restrict__ c, const double (&inv)[9], const uint8_t* __restrict__ pbc, int n_atoms,
                                        const double (&lo)[3], const double (&hi)[3], double cutoff, GraphBins& gb) {
  for (int k = 0; k < 9; ++k) { gb.inv[k] = inv[k]; gb.cell[k] = c[k]; }
  double width[3];
  for (int k = 0; k < 3; ++k) {
    // perpendicular height of the cell along axis k = 1 / |column k of inv|
    const double h = 1.0 / sqrt(inv[k] * inv[k] + inv[3 + k] * inv[3 + k] + inv[6 + k] * inv[6 + k]);
    gb.pbc[k] = pbc[k] ? 1 : 0;
    if (gb.pbc[k]) { gb.fmin[k] = 0.0; gb.fext[k] = 1.0; width[k] = h; }
    else {
      gb.fmin[k] = n_atoms ? lo[k] : 0.0;
      gb.fext[k] = n_atoms ? fmax(hi[k] - lo[k], 1e-12) : 1.0;
      width[k] = gb.fext[k] * h;
    }
    int nb = (int)floor(width[k] / cutoff);
    gb.nb[k] = nb < 1 ? 1 : (nb > 1024 ? 1024 : nb);
  }
  // keep the number of bins of a structure below ~2 per atom
  const long long cap = n_atoms > 0 ? 2LL * n_atoms : 1;
  while ((long long)gb.nb[0] * gb.nb[1] * gb.nb[2] > cap) {
    int k = 0;
    if (gb.nb[1] > gb.nb[k]) k = 1;
    if (gb.nb[2] > gb.nb[k]) k = 2;
    gb.nb[k] = (gb.nb[k] + 1) / 2;
  }
  for (int k = 0; k < 3; ++k) {
    const double bin_h = width[k] / gb.nb[k];
    int r = (int)ceil(cutoff / bin_h);
    if (r < 1) r = 1;
    if (!gb.pbc[k] && r > gb.nb[k] - 1) r = gb.nb[k] - 1;
    gb.r[k] = r;
  }
  gb.n_bins = gb.nb[0] * gb.nb[1] * gb.nb[2];
  gb.bin_offset = 0;
}
__device__ __forceinline__ void frac_range(const double* __restrict__ pos, int i, const double (&inv)[9], double (&lo)[3], double (&hi)[3]) {
  const double x = pos[3LL * i], y = pos[3LL * i + 1], z = pos[3LL * i + 2];
  for (int k = 0; k < 3; ++k) {
    const double f = x * inv[k] + y * inv[3 + k] + z * inv[6 + k];
    lo[k] = fmin(lo[k], f); hi[k] = fmax(hi[k], f);
  }
}

__global__ void nl_setup_kernel(const double* __restrict__ pos, const double* __restrict__ lattice,
                                const uint8_t* __restrict__ pbc, const int* __restrict__ graph_ptr, double cutoff,
                                GraphBins* bins) {
  const int g = blockIdx.x;
  __shared__ double smin[3][128], smax[3][128];
  const double* c = lattice + 9LL * g;
  double inv[9];
  cell_inverse(c, inv);
  double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
  const int a0 = graph_ptr[g], a1 = graph_ptr[g + 1];
  for (int i = a0 + threadIdx.x; i < a1; i += blockDim.x) frac_range(pos, i, inv, lo, hi);
  for (int k = 0; k < 3; ++k) { smin[k][threadIdx.x] = lo[k]; smax[k][threadIdx.x] = hi[k]; }
  __syncthreads();
  for (int off = 64; off > 0; off >>= 1) {
    if (threadIdx.x < off)
      for (int k = 0; k < 3; ++k) {
        smin[k][threadIdx.x] = fmin(smin[k][threadIdx.x], smin[k][threadIdx.x + off]);
        smax[k][threadIdx.x] = fmax(smax[k][threadIdx.x], smax[k][threadIdx.x + off]);
      }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    GraphBins gb;
    for (int k = 0; k < 3; ++k) { lo[k] = smin[k][0]; hi[k] = smax[k][0]; }
    bins_of(c, inv, pbc + 3LL * g, a1 - a0, lo, hi, cutoff, gb);
    bins[g] = gb;
  }
}

__global__ void nl_offsets_kernel(GraphBins* bins, int n_graphs, int* total) {
  if (blockIdx.x || threadIdx.x) return;
  int acc = 0;
  for (int g = 0; g < n_graphs; ++g) { bins[g].bin_offset = acc; acc += bins[g].n_bins; }
  *total = acc;
}

__device__ __forceinline__ int graph_of(const int* __restrict__ graph_ptr, int n_graphs, int i) {
  int lo = 0, hi = n_graphs;
  while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (graph_ptr[mid] <= i) lo = mid; else hi = mid; }
  return lo;
}
__device__ __forceinline__ int bin_of(const double* __restrict__ pos, int i, const GraphBins& gb, int* img) {
  const double x = pos[3LL * i], y = pos[3LL * i + 1], z = pos[3LL * i + 2];
  int b[3];
  for (int k = 0; k < 3; ++k) {
    const double f = x * gb.inv[k] + y * gb.inv[3 + k] + z * gb.inv[6 + k];
    int fl = 0;
    double t;
    if (gb.pbc[k]) { const double ff = floor(f); fl = (int)ff; t = f - ff; }
    else t = (f - gb.fmin[k]) / gb.fext[k];
    int bk = (int)(t * gb.nb[k]);
    bk = bk < 0 ? 0 : (bk >= gb.nb[k] ? gb.nb[k] - 1 : bk);
    b[k] = bk;
    img[3LL * i + k] = fl;
  }
  return gb.bin_offset + (b[0] * gb.nb[1] + b[1]) * gb.nb[2] + b[2];
}
__global__ void nl_bin_kernel(const double* __restrict__ pos, const GraphBins* __restrict__ bins,
                              const int* __restrict__ graph_ptr, int n_graphs, int n_atoms, int* keys, int* vals, int* img) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_atoms) return;
  keys[i] = bin_of(pos, i, bins[graph_of(graph_ptr, n_graphs, i)], img);
  vals[i] = i;
}

// Exclusive scan of one value per thread over a block of 1 024; `total` is the block's sum.
template <typename V>
__device__ __forceinline__ V scan_1024(V v, V* warp_sums, V& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  V x = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const V o = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += o;
  }
  __syncthreads();  // warp_sums may still be read from an earlier scan
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    V w = warp_sums[lane];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const V o = __shfl_up_sync(0xffffffffu, w, off);
      if (lane >= off) w += o;
    }
    warp_sums[lane] = w;
  }
  __syncthreads();
  total = warp_sums[31];
  return x - v + (warp ? warp_sums[warp - 1] : V(0));
}

// The whole preparation of a small batch (bins, atoms sorted by bin in index order, bin starts) in one block: five launches, one
// of them a device-wide sort, took 43 us of which half were gaps (32 atoms); this takes 8.
constexpr int kSmallAtoms = 8192, kSmallGraphs = 1024;
__global__ void __launch_bounds__(1024) nl_small_prepare_kernel(const double* __restrict__ pos, const double* __restrict__ lattice,
                                                                const uint8_t* __restrict__ pbc, const int* __restrict__ graph_ptr,
                                                                int n_graphs, int n_atoms, double cutoff, GraphBins* bins, int* keys,
                                                                int* tmp, int* atoms_sorted, int* img, int* cell_start, int* cursor,
                                                                int* found_valid, int found) {
  __shared__ int warp_sums[32];
  __shared__ int n_bins_s[kSmallGraphs];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) *found_valid = found;
  for (int g = warp; g < n_graphs; g += 32) {
    const double* c = lattice + 9LL * g;
    const uint8_t* p = pbc + 3LL * g;
    double inv[9];
    cell_inverse(c, inv);
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    const int a0 = graph_ptr[g], a1 = graph_ptr[g + 1];
    if (!(p[0] && p[1] && p[2])) {
      for (int i = a0 + lane; i < a1; i += 32) frac_range(pos, i, inv, lo, hi);
      for (int off = 16; off > 0; off >>= 1)
        for (int k = 0; k < 3; ++k) {
          lo[k] = fmin(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], off));
          hi[k] = fmax(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], off));
        }
    }
    if (lane == 0) {
      GraphBins gb;
      bins_of(c, inv, p, a1 - a0, lo, hi, cutoff, gb);
      bins[g] = gb;
      n_bins_s[g] = gb.n_bins;
    }
  }
  __syncthreads();
  int n_cells;
  const int off = scan_1024(tid < n_graphs ? n_bins_s[tid] : 0, warp_sums, n_cells);
  if (tid < n_graphs) bins[tid].bin_offset = off;
  for (int c = tid; c < n_cells; c += 1024) cell_start[c] = 0;
  __syncthreads();
  for (int i = tid; i < n_atoms; i += 1024) {
    const int key = bin_of(pos, i, bins[graph_of(graph_ptr, n_graphs, i)], img);
    keys[i] = key;
    atomicAdd(cell_start + key, 1);
  }
  __syncthreads();
  const int per = (n_cells + 1023) / 1024, c0 = tid * per, c1 = min(c0 + per, n_cells);
  int sum = 0, total;
  for (int c = c0; c < c1; ++c) sum += cell_start[c];
  int at = scan_1024(sum, warp_sums, total);
  for (int c = c0; c < c1; ++c) { const int n = cell_start[c]; cell_start[c] = at; cursor[c] = at; at += n; }
  if (tid == 0) cell_start[n_cells] = n_atoms;
  __syncthreads();
  for (int i = tid; i < n_atoms; i += 1024) tmp[atomicAdd(cursor + keys[i], 1)] = i;
  __syncthreads();
  for (int i = tid; i < n_atoms; i += 1024) {
    const int b = cell_start[keys[i]], e = cell_start[keys[i] + 1];
    int r = 0;
    for (int k = b; k < e; ++k) r += tmp[k] < i ? 1 : 0;
    atoms_sorted[b + r] = i;
  }
}
// row_ptr[i] = counts[0] + ... + counts[i - 1], i = 0..n, in one block.  Summed in 64 bits: 46 342 atoms that all see each other
// have 2^31 edges.
__global__ void __launch_bounds__(1024) nl_row_ptr_kernel(const int* __restrict__ counts, int n, int64_t* row_ptr) {
  __shared__ int64_t warp_sums[32];
  const int per = (n + 1023) / 1024, i0 = threadIdx.x * per, i1 = min(i0 + per, n);
  int64_t sum = 0, total;
  for (int i = i0; i < i1; ++i) sum += counts[i];
  int64_t at = scan_1024(sum, warp_sums, total);
  for (int i = i0; i < i1; ++i) { row_ptr[i] = at; at += counts[i]; }
  if (threadIdx.x == 0) row_ptr[n] = total;
}
__global__ void nl_zero_first_kernel(int64_t* row_ptr) { row_ptr[0] = 0; }

__global__ void nl_cell_start_kernel(const int* __restrict__ sorted_keys, int n_keys, int* cell_start, int n_cells) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > n_cells) return;
  int lo = 0, hi = n_keys;
  while (lo < hi) { const int mid = (lo + hi) >> 1; if (sorted_keys[mid] < c) lo = mid + 1; else hi = mid; }
  cell_start[c] = lo;
}

__device__ __forceinline__ int floordiv(int a, int b) { return (a >= 0) ? a / b : -((-a + b - 1) / b); }

// FILL = false: counts[i] = number of sources of target i; FILL = true: write them at row_ptr[i].
// One warp per target atom.  The neighbouring bins come 32 at a time (lane = bin, in the fixed order d0, d1, d2 of the
// offsets); a scan of their sizes numbers their atoms consecutively, and the lanes then test 32 candidates at a time, so that
// a few full bins (small cells: one bin seen 27 times) and many sparse ones keep all lanes busy alike.  A ballot turns hits
// into output positions: by bin, then by source index.
//
// W = 4: the four warps of a block share an atom, each testing a run of candidates at a time (small batches, where the walk over an
// atom's candidates is all there is to wait for).
// `found` (small batches): the count also leaves the first kFound sources of every target and their shifts in the workspace, and
// the fill copies them instead of searching again where the target has no more; `found_valid` says that the count did.
// 32 atoms of 42 edges (864 candidates each): count 10.7 -> 4.9 us, fill 9.2 -> 2.3; 570 atoms of 62: 20 -> 10 and 16 -> 3.
constexpr int kFound = 128;
__device__ __forceinline__ void nl_put(int64_t at, int64_t n_edges, int i, const int4& f, int64_t* edge_index, void* shifts, int shift_type) {
  if (at >= n_edges) return;
  edge_index[at] = f.x;
  edge_index[n_edges + at] = i;
  if (shift_type == TACE_F32) { float* p = static_cast<float*>(shifts) + 3 * at; p[0] = (float)f.y; p[1] = (float)f.z; p[2] = (float)f.w; }
  else if (shift_type == TACE_F64) { double* p = static_cast<double*>(shifts) + 3 * at; p[0] = f.y; p[1] = f.z; p[2] = f.w; }
  else { int32_t* p = static_cast<int32_t*>(shifts) + 3 * at; p[0] = f.y; p[1] = f.z; p[2] = f.w; }
}
template <bool FILL, int W>
__global__ void __launch_bounds__(128) nl_search_kernel(const double* __restrict__ pos, const GraphBins* __restrict__ bins,
                                 const int* __restrict__ graph_ptr, int n_graphs, int n_atoms, int n_targets, double cutoff,
                                 const int* __restrict__ keys_of_atom, const int* __restrict__ sorted_atoms,
                                 const int* __restrict__ cell_start, const int* __restrict__ img, int* counts,
                                 const int64_t* __restrict__ row_ptr, int64_t n_edges, int64_t* edge_index, void* shifts, int shift_type,
                                 int4* found, const int* __restrict__ found_valid) {
  __shared__ int hits_of[2][4];
  const int warp = threadIdx.x >> 5, part = W == 1 ? 0 : warp;
  const int i = W == 1 ? (int)(blockIdx.x * 4LL + warp) : (int)blockIdx.x;
  const int lane = threadIdx.x & 31;
  if (i >= n_atoms) return;  // whole warps (W = 4: the whole block) leave together
  if (i >= n_targets) {      // a ghost: no row of its own
    if (!FILL && lane == 0) counts[i] = 0;
    return;
  }
  if (FILL && found && *found_valid) {
    const int64_t beg = row_ptr[i];
    const int n = (int)(row_ptr[i + 1] - beg);
    if (n <= kFound) {
      for (int k = part * 32 + lane; k < n; k += 32 * W) nl_put(beg + k, n_edges, i, found[(int64_t)i * kFound + k], edge_index, shifts, shift_type);
      return;
    }
  }
  int turn = 0;
  const GraphBins& gb = bins[graph_of(graph_ptr, n_graphs, i)];
  const double c2 = __dmul_rn(cutoff, cutoff);
  const double xi = pos[3LL * i], yi = pos[3LL * i + 1], zi = pos[3LL * i + 2];
  double cell[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) cell[k] = gb.cell[k];
  const int nb0 = gb.nb[0], nb1 = gb.nb[1], nb2 = gb.nb[2];
  const int key = keys_of_atom[i] - gb.bin_offset;
  const int b2 = key % nb2, b1 = (key / nb2) % nb1, b0 = key / (nb2 * nb1);
  const int fi0 = img[3LL * i], fi1 = img[3LL * i + 1], fi2 = img[3LL * i + 2];
  const int w1 = 2 * gb.r[1] + 1, w2 = 2 * gb.r[2] + 1;
  const int n_cells = (2 * gb.r[0] + 1) * w1 * w2;
  int64_t out = FILL ? row_ptr[i] : 0;
  int count = 0;
  for (int cb = 0; cb < n_cells; cb += 32) {
    const int c = cb + lane;
    int k_beg = 0, size = 0, s0 = 0, s1 = 0, s2 = 0;
    if (c < n_cells) {
      const int d0 = c / (w1 * w2) - gb.r[0], d1 = (c / w2) % w1 - gb.r[1], d2 = c % w2 - gb.r[2];
      int c0 = b0 + d0, c1 = b1 + d1, c2i = b2 + d2;
      bool inside = true;
      if (gb.pbc[0]) { s0 = floordiv(c0, nb0); c0 -= s0 * nb0; } else if (c0 < 0 || c0 >= nb0) inside = false;
      if (gb.pbc[1]) { s1 = floordiv(c1, nb1); c1 -= s1 * nb1; } else if (c1 < 0 || c1 >= nb1) inside = false;
      if (gb.pbc[2]) { s2 = floordiv(c2i, nb2); c2i -= s2 * nb2; } else if (c2i < 0 || c2i >= nb2) inside = false;
      if (inside) {
        const int at = gb.bin_offset + (c0 * nb1 + c1) * nb2 + c2i;
        k_beg = cell_start[at]; size = cell_start[at + 1] - k_beg;
      }
    }
    int incl = size;  // inclusive scan over the lanes
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += t;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31), excl = incl - size;
    // four rounds of 32 candidates in flight: the chain shuffle -> index -> coordinates is latency, not work
    constexpr int U = 4;
    for (int t0 = 32 * U * part; t0 < (total + 32 * U * W - 1) / (32 * U * W) * (32 * U * W); t0 += 32 * U * W) {
      int j[U], S0[U], S1[U], S2[U];
      bool in[U], hit[U];
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int t = t0 + 32 * q + lane;
        int src = 0;  // bin (lane) of candidate t: the last one that starts at or before t (empty bins share a start: the last wins)
#pragma unroll
        for (int step = 16; step > 0; step >>= 1) {
          const int at = __shfl_sync(0xffffffffu, excl, src + step);
          if (at <= t) src += step;
        }
        const int k = __shfl_sync(0xffffffffu, k_beg, src) + t - __shfl_sync(0xffffffffu, excl, src);
        S0[q] = __shfl_sync(0xffffffffu, s0, src); S1[q] = __shfl_sync(0xffffffffu, s1, src); S2[q] = __shfl_sync(0xffffffffu, s2, src);
        in[q] = t < total;
        j[q] = in[q] ? sorted_atoms[k] : i;
      }
#pragma unroll
      for (int q = 0; q < U; ++q) {
        // wrapped image (s0,s1,s2) of source j seen from target i:  r_j - r_i + S' @ cell with S' = s - fl_j + fl_i;
        // the edge (source j -> target i) carries shift S = -S'.
        const int jj = j[q];
        S0[q] = -(S0[q] - img[3LL * jj] + fi0); S1[q] = -(S1[q] - img[3LL * jj + 1] + fi1); S2[q] = -(S2[q] - img[3LL * jj + 2] + fi2);
        const double a0 = (double)S0[q], a1 = (double)S1[q], a2 = (double)S2[q];
        const double v0 = __dadd_rn(__dadd_rn(__dmul_rn(a0, cell[0]), __dmul_rn(a1, cell[3])), __dmul_rn(a2, cell[6]));
        const double v1 = __dadd_rn(__dadd_rn(__dmul_rn(a0, cell[1]), __dmul_rn(a1, cell[4])), __dmul_rn(a2, cell[7]));
        const double v2 = __dadd_rn(__dadd_rn(__dmul_rn(a0, cell[2]), __dmul_rn(a1, cell[5])), __dmul_rn(a2, cell[8]));
        const double dx = __dadd_rn(__dadd_rn(xi, -pos[3LL * jj]), v0);
        const double dy = __dadd_rn(__dadd_rn(yi, -pos[3LL * jj + 1]), v1);
        const double dz = __dadd_rn(__dadd_rn(zi, -pos[3LL * jj + 2]), v2);
        const double dsq = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
        hit[q] = in[q] && dsq < c2 && !(jj == i && S0[q] == 0 && S1[q] == 0 && S2[q] == 0);
      }
      unsigned hits[U];
      int own = 0, all = 0, at = FILL ? 0 : count;  // at: of this warp's first hit in the target's row (FILL: from `out`)
#pragma unroll
      for (int q = 0; q < U; ++q) { hits[q] = __ballot_sync(0xffffffffu, hit[q]); own += __popc(hits[q]); }
      if constexpr (W > 1) {  // the runs of the warps before this one come first
        if (lane == 0) hits_of[turn][warp] = own;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < W; ++w) { const int n = hits_of[turn][w]; all += n; if (w < warp) at += n; }
        turn ^= 1;
      } else {
        all = own;
      }
#pragma unroll
      for (int q = 0; q < U; ++q) {
        const int k = at + __popc(hits[q] & ((1u << lane) - 1u));
        if (hit[q]) {
          const int4 f = make_int4(j[q], S0[q], S1[q], S2[q]);
          if (FILL) nl_put(out + k, n_edges, i, f, edge_index, shifts, shift_type);
          else if (found && k < kFound) found[(int64_t)i * kFound + k] = f;
        }
        at += __popc(hits[q]);
      }
      out += all;
      count += all;
    }
  }
  if (!FILL && lane == 0 && part == 0) counts[i] = count;
}

// Counts as 64-bit numbers: a device-wide scan adds up in the type of what it reads.
struct Widen { __host__ __device__ int64_t operator()(int x) const { return x; } };
inline auto widened(const int* counts) { return thrust::make_transform_iterator(counts, Widen()); }

inline size_t al256(size_t x) { return (x + 255) & ~size_t(255); }
inline int nl_max_cells(int n_atoms, int n_graphs) { return 2 * n_atoms + n_graphs + 1; }
size_t nl_cub_bytes(int n_atoms) {
  size_t sort = 0, scan = 0;
  if (n_atoms <= 0) return 0;
  cub::DeviceRadixSort::SortPairs(nullptr, sort, (const int*)nullptr, (int*)nullptr, (const int*)nullptr, (int*)nullptr, n_atoms);
  cub::DeviceScan::InclusiveSum(nullptr, scan, widened(nullptr), (int64_t*)nullptr, n_atoms);
  return sort > scan ? sort : scan;
}
size_t nl_workspace_bytes(int n_atoms, int n_graphs) {
  return al256(sizeof(GraphBins) * n_graphs) + al256(sizeof(int)) + 4 * al256(sizeof(int) * (size_t)n_atoms) +
         al256(sizeof(int) * 3 * (size_t)n_atoms) + 2 * al256(sizeof(int) * (size_t)(nl_max_cells(n_atoms, n_graphs) + 1)) +
         al256(nl_cub_bytes(n_atoms)) + 256;
}

// The first sources of every target, kept between the count and the fill of a small batch (at the end of a workspace that has room).
inline size_t nl_found_bytes(int n_atoms, int n_graphs) {
  return n_atoms <= kSmallAtoms && n_graphs <= kSmallGraphs ? sizeof(int4) * kFound * (size_t)n_atoms : 0;
}

// The scratch of one list, cut from its first 256-byte boundary.
struct NlScratch {
  GraphBins* bins;
  int4* found = nullptr;
  int *total, *keys, *vals, *keys_sorted, *atoms_sorted, *img, *cell_start, *cursor;
  void* cub;
  NlScratch(unsigned char* p, int n_atoms, int n_graphs) {
    auto take = [&p](size_t bytes) { unsigned char* r = p; p += al256(bytes); return r; };
    const size_t n = (size_t)n_atoms, cells = (size_t)nl_max_cells(n_atoms, n_graphs) + 1;
    bins = reinterpret_cast<GraphBins*>(take(sizeof(GraphBins) * n_graphs));
    total = reinterpret_cast<int*>(take(sizeof(int)));
    keys = reinterpret_cast<int*>(take(sizeof(int) * n)); vals = reinterpret_cast<int*>(take(sizeof(int) * n));
    keys_sorted = reinterpret_cast<int*>(take(sizeof(int) * n)); atoms_sorted = reinterpret_cast<int*>(take(sizeof(int) * n));
    img = reinterpret_cast<int*>(take(sizeof(int) * 3 * n));
    cell_start = reinterpret_cast<int*>(take(sizeof(int) * cells)); cursor = reinterpret_cast<int*>(take(sizeof(int) * cells));
    cub = p;
  }
};

// bins, sorted atoms and bin starts
cudaError_t nl_prepare(const NlScratch& w, const double* pos, const double* lattice, const uint8_t* pbc, const int32_t* graph_ptr,
                       int n_graphs, int n_atoms, double cutoff, cudaStream_t s) {
  if (n_atoms <= kSmallAtoms && n_graphs <= kSmallGraphs) {
    nl_small_prepare_kernel<<<1, 1024, 0, s>>>(pos, lattice, pbc, graph_ptr, n_graphs, n_atoms, cutoff, w.bins, w.keys, w.vals,
                                               w.atoms_sorted, w.img, w.cell_start, w.cursor, w.total, w.found ? 1 : 0);
    return cudaGetLastError();
  }
  nl_setup_kernel<<<n_graphs, 128, 0, s>>>(pos, lattice, pbc, graph_ptr, cutoff, w.bins);
  nl_offsets_kernel<<<1, 1, 0, s>>>(w.bins, n_graphs, w.total);
  nl_bin_kernel<<<(n_atoms + 127) / 128, 128, 0, s>>>(pos, w.bins, graph_ptr, n_graphs, n_atoms, w.keys, w.vals, w.img);
  const int max_cells = nl_max_cells(n_atoms, n_graphs);
  int bits = 1;
  while (bits < 31 && (1LL << bits) <= max_cells) ++bits;
  size_t cub_bytes = nl_cub_bytes(n_atoms);
  const cudaError_t err = cub::DeviceRadixSort::SortPairs(w.cub, cub_bytes, w.keys, w.keys_sorted, w.vals, w.atoms_sorted, n_atoms, 0, bits, s);
  if (err != cudaSuccess) return err;
  nl_cell_start_kernel<<<(max_cells + 128) / 128, 128, 0, s>>>(w.keys_sorted, n_atoms, w.cell_start, max_cells);
  return cudaGetLastError();
}
template <bool FILL>
cudaError_t nl_search(const NlScratch& w, const double* pos, const int32_t* graph_ptr, int n_graphs, int n_atoms, int n_targets,
                      double cutoff, int* counts, const int64_t* row_ptr, int64_t n_edges, int64_t* edge_index, void* shifts, int shift_type, cudaStream_t s) {
  auto run = [&](auto kernel, int blocks) {
    kernel<<<blocks, 128, 0, s>>>(pos, w.bins, graph_ptr, n_graphs, n_atoms, n_targets, cutoff, w.keys, w.atoms_sorted, w.cell_start, w.img, counts,
                                  row_ptr, n_edges, edge_index, shifts, shift_type, w.found, w.total);
  };
  if (n_atoms <= 2048) run(nl_search_kernel<FILL, 4>, n_atoms);
  else run(nl_search_kernel<FILL, 1>, (n_atoms + 3) / 4);
  return cudaGetLastError();
}
// counts -> row pointers; `cub` scratch only for large lists
cudaError_t nl_row_ptr(const int* counts, int n_atoms, int64_t* row_ptr, void* cub_temp, cudaStream_t s) {
  if (n_atoms <= (1 << 16) || !cub_temp) {
    nl_row_ptr_kernel<<<1, 1024, 0, s>>>(counts, n_atoms, row_ptr);
    return cudaGetLastError();
  }
  nl_zero_first_kernel<<<1, 1, 0, s>>>(row_ptr);
  size_t bytes = nl_cub_bytes(n_atoms);
  return cub::DeviceScan::InclusiveSum(cub_temp, bytes, widened(counts), row_ptr + 1, n_atoms, s);
}

// prepared: the workspace still holds what a count of the same structures left there
int nl_run(bool fill, bool prepared, const double* pos, const double* lattice, const uint8_t* pbc, const int32_t* graph_ptr, int32_t n_graphs,
           int64_t n_atoms64, int64_t n_targets, double cutoff, int32_t* counts, int64_t* row_ptr_out, const int64_t* row_ptr, int64_t n_edges,
           int64_t* edge_index, void* shifts, int shift_type, void* workspace, size_t workspace_bytes, cudaStream_t s) {
  if (!pos || !lattice || !pbc || !graph_ptr || n_graphs <= 0 || n_atoms64 < 0 || !(cutoff > 0.0)) return TACE_ERR_INVALID_ARGUMENT;
  if (n_atoms64 >= (1LL << 30)) return TACE_ERR_CAPACITY;
  if (fill ? (!row_ptr || (n_edges > 0 && (!edge_index || !shifts))) : !counts) return TACE_ERR_INVALID_ARGUMENT;
  const int n_atoms = (int)n_atoms64;
  if (n_atoms == 0) {
    if (row_ptr_out) nl_zero_first_kernel<<<1, 1, 0, s>>>(row_ptr_out);
    return TACE_OK;
  }
  if (!workspace) return TACE_ERR_INVALID_ARGUMENT;
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(workspace) + 255) & ~uintptr_t(255));
  const size_t lead = (size_t)(base - static_cast<unsigned char*>(workspace));
  if (workspace_bytes < lead || workspace_bytes - lead + 256 < nl_workspace_bytes(n_atoms, n_graphs)) return TACE_ERR_CAPACITY;
  NlScratch w(base, n_atoms, n_graphs);
  const size_t found_at = nl_workspace_bytes(n_atoms, n_graphs), found = nl_found_bytes(n_atoms, n_graphs);
  if (found && (prepared || !fill) && workspace_bytes - lead >= found_at + found) w.found = reinterpret_cast<int4*>(base + found_at);
  const int targets = n_targets < 0 || n_targets > n_atoms ? n_atoms : (int)n_targets;
  cudaError_t err = prepared ? cudaSuccess : nl_prepare(w, pos, lattice, pbc, graph_ptr, n_graphs, n_atoms, cutoff, s);
  if (err == cudaSuccess)
    err = fill ? nl_search<true>(w, pos, graph_ptr, n_graphs, n_atoms, targets, cutoff, nullptr, row_ptr, n_edges, edge_index, shifts, shift_type, s)
               : nl_search<false>(w, pos, graph_ptr, n_graphs, n_atoms, targets, cutoff, counts, nullptr, 0, nullptr, nullptr, -1, s);
  if (err == cudaSuccess && row_ptr_out) err = nl_row_ptr(counts, n_atoms, row_ptr_out, w.cub, s);
  return err == cudaSuccess ? TACE_OK : TACE_ERR_CUDA;
}

// ---- neighbour list without any allocation -------------------------------------------------------
// Scratch for tace_nl_build_noalloc lives in this file-scope device array (2 MiB per GPU that loads
// the library, held until the process exits).  In host code the name `nl_static_scratch` is only a
// handle for the runtime, not a device address: the address is looked up once per device with
// cudaGetSymbolAddress and that pointer is what the kernels receive.
constexpr int kNoAllocMaxAtoms = 16384;
constexpr int kNoAllocMaxGraphs = 1024;
constexpr size_t kNoAllocScratchBytes = size_t(2) << 20;
static __device__ __align__(256) unsigned char nl_static_scratch[kNoAllocScratchBytes];

int nl_build_noalloc(const double* pos, const double* lattice, const uint8_t* pbc, const int32_t* graph_ptr, int32_t n_graphs,
                     int64_t n_atoms64, double cutoff, int64_t max_edges, int64_t* row_ptr, int64_t* edge_index, int32_t* shifts,
                     cudaStream_t s) {
  if (!pos || !lattice || !pbc || !graph_ptr || !row_ptr || n_graphs <= 0 || n_atoms64 < 0 || max_edges < 0 || !(cutoff > 0.0) ||
      (max_edges > 0 && (!edge_index || !shifts)))
    return TACE_ERR_INVALID_ARGUMENT;
  if (n_atoms64 > kNoAllocMaxAtoms || n_graphs > kNoAllocMaxGraphs) return TACE_ERR_CAPACITY;
  const int n_atoms = (int)n_atoms64;
  // one-time, per-device lookup of the scratch array's device address (with that device current)
  constexpr int kMaxDevices = 64;
  static unsigned char* scratch_of_device[kMaxDevices] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return TACE_ERR_NO_DEVICE;
  if (!scratch_of_device[dev]) {
    unsigned char* ptr = nullptr;
    if (cudaGetSymbolAddress((void**)&ptr, nl_static_scratch) != cudaSuccess || !ptr) return TACE_ERR_CUDA;
    scratch_of_device[dev] = ptr;
  }
  unsigned char* p = scratch_of_device[dev];
  const NlScratch w(p, n_atoms, n_graphs);
  unsigned char* q = static_cast<unsigned char*>(w.cub);
  int* counts = reinterpret_cast<int*>(q + al256(n_atoms > kSmallAtoms ? nl_cub_bytes(n_atoms) : 0));
  if (reinterpret_cast<unsigned char*>(counts + n_atoms + 1) > p + kNoAllocScratchBytes) return TACE_ERR_CAPACITY;

  cudaError_t err = cudaSuccess;
  if (n_atoms > 0) {
    err = nl_prepare(w, pos, lattice, pbc, graph_ptr, n_graphs, n_atoms, cutoff, s);
    if (err == cudaSuccess) err = nl_search<false>(w, pos, graph_ptr, n_graphs, n_atoms, n_atoms, cutoff, counts, nullptr, 0, nullptr, nullptr, -1, s);
  }
  if (err == cudaSuccess) err = nl_row_ptr(counts, n_atoms, row_ptr, nullptr, s);
  if (err == cudaSuccess && n_atoms > 0)
    err = nl_search<true>(w, pos, graph_ptr, n_graphs, n_atoms, n_atoms, cutoff, nullptr, row_ptr, max_edges, edge_index, shifts, -1, s);
  return err == cudaSuccess ? TACE_OK : TACE_ERR_CUDA;
}

}  // namespace
}  // namespace tace

extern "C" {

int tace_nl_build_noalloc(const double* positions, const double* lattice, const uint8_t* pbc, const int32_t* graph_ptr,
                          int32_t n_graphs, int64_t n_atoms, double cutoff, int64_t max_edges, int64_t* row_ptr,
                          int64_t* edge_index, int32_t* edge_shifts, tace_stream_t stream) {
  return tace::nl_build_noalloc(positions, lattice, pbc, graph_ptr, n_graphs, n_atoms, cutoff, max_edges, row_ptr, edge_index,
                                edge_shifts, static_cast<cudaStream_t>(stream));
}

int tace_nl_workspace_bytes(int64_t n_atoms, int32_t n_graphs, size_t* bytes) {
  if (!bytes || n_atoms < 0 || n_graphs <= 0) return TACE_ERR_INVALID_ARGUMENT;
  if (n_atoms >= (1LL << 30)) return TACE_ERR_CAPACITY;
  *bytes = tace::nl_workspace_bytes((int)n_atoms, n_graphs) + tace::nl_found_bytes((int)n_atoms, n_graphs) + 256;
  return TACE_OK;
}

int tace_nl_count(const double* positions, const double* lattice, const uint8_t* pbc, const int32_t* graph_ptr,
                  int32_t n_graphs, int64_t n_atoms, double cutoff, int32_t* counts, void* workspace, size_t workspace_bytes,
                  tace_stream_t stream) {
  return tace::nl_run(false, false, positions, lattice, pbc, graph_ptr, n_graphs, n_atoms, -1, cutoff, counts, nullptr, nullptr, 0, nullptr,
                      nullptr, -1, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}

int tace_nl_rows(const double* positions, const double* lattice, const uint8_t* pbc, const int32_t* graph_ptr, int32_t n_graphs,
                 int64_t n_atoms, int64_t n_targets, double cutoff, int32_t* counts, int64_t* row_ptr, void* workspace,
                 size_t workspace_bytes, tace_stream_t stream) {
  if (!row_ptr) return TACE_ERR_INVALID_ARGUMENT;
  return tace::nl_run(false, false, positions, lattice, pbc, graph_ptr, n_graphs, n_atoms, n_targets, cutoff, counts, row_ptr, nullptr, 0,
                      nullptr, nullptr, -1, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}

int tace_nl_fill_rows(const double* positions, const double* lattice, const uint8_t* pbc, const int32_t* graph_ptr, int32_t n_graphs,
                      int64_t n_atoms, int64_t n_targets, double cutoff, const int64_t* row_ptr, int64_t n_edges, int64_t* edge_index,
                      void* edge_shifts, int32_t shift_type, void* workspace, size_t workspace_bytes, tace_stream_t stream) {
  return tace::nl_run(true, true, positions, lattice, pbc, graph_ptr, n_graphs, n_atoms, n_targets, cutoff, nullptr, nullptr, row_ptr,
                      n_edges, edge_index, edge_shifts, shift_type, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}

int tace_nl_fill(const double* positions, const double* lattice, const uint8_t* pbc, const int32_t* graph_ptr,
                 int32_t n_graphs, int64_t n_atoms, double cutoff, const int64_t* row_ptr, int64_t n_edges,
                 int64_t* edge_index, int32_t* edge_shifts, void* workspace, size_t workspace_bytes, tace_stream_t stream) {
  return tace::nl_run(true, false, positions, lattice, pbc, graph_ptr, n_graphs, n_atoms, -1, cutoff, nullptr, nullptr, row_ptr, n_edges,
                      edge_index, edge_shifts, -1, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
