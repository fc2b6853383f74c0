// Graph preparation: from the caller's edge_index (any order) to target-sorted and
// source-sorted CSR views, the atom -> graph map, and the species-sorted atom permutation used
// by the per-species linear layers.  The edge views are counting sorts: every bin (the edges of one
// atom) is filled through an atomic cursor and then put into ascending order by one warp, so the
// result is the stable order whatever the arrival order, and the segmented sums downstream are
// bit-reproducible.
//
// Five short kernels replaced two device-wide radix sorts with their row-pointer searches (21 launches
// and eight memset nodes): 2 407 atoms, 150 400 edges, as part of a replayed graph, 160 -> 30 us, most of
// it gaps around the memset nodes; 131 072 atoms, 5.5 M edges 0.45 -> 0.26 ms.
#include <cub/cub.cuh>
#include "kernels.h"

namespace tace {

namespace {

__global__ void iota_and_key32_kernel(const int* __restrict__ key_src, int* keys, int* vals, long long n) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  keys[i] = key_src[i];
  vals[i] = (int)i;
}
// keys[i] = 1 if any edge into target i comes from a ghost atom (index >= n_local), else 0; vals[i] = i
__global__ void ghost_row_key_kernel(const int* __restrict__ rowptr, const int* __restrict__ e_src, int n_local, int* keys, int* vals) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_local) return;
  int flag = 0;
  for (int e = rowptr[i]; e < rowptr[i + 1]; ++e) flag |= (e_src[e] >= n_local) ? 1 : 0;
  keys[i] = flag;
  vals[i] = i;
}
// rowptr[i] = number of sorted keys < i, i = 0..n_rows
__global__ void lower_bound_kernel(const int* __restrict__ sorted_keys, long long n_keys, int* rowptr, int n_rows) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > n_rows) return;
  long long lo = 0, hi = n_keys;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (sorted_keys[mid] < i) lo = mid + 1; else hi = mid;
  }
  rowptr[i] = (int)lo;
}
// tile_ptr: 32-row tiles of gemm.cuh; tc_tile_ptr: (128 / q)-atom tiles of the tensor-core GEMM; q = 1, 3, 5, 7.  One warp per
// table (`which` = 0..7), a warp scan over the species.
__device__ __forceinline__ void tile_table(const int* species_ptr, int n_el, int which, int* tile_ptr, int* tc_tile_ptr) {
  const int qi = which & 3, lane = threadIdx.x & 31;
  const bool tc = which >= 4;
  int* tp = (tc ? tc_tile_ptr : tile_ptr) + qi * (n_el + 1);
  int carry = 0;
  for (int g0 = 0; g0 <= n_el; g0 += 32) {
    const int g = g0 + lane;
    int tiles = 0;
    if (g < n_el) {
      const int cnt = species_ptr[g + 1] - species_ptr[g];
      if (!tc) tiles = (cnt * (2 * qi + 1) + 31) >> 5;
      else tiles = qi == 0 ? (cnt + 127) >> 7 : qi == 1 ? (cnt + 41) / 42 : qi == 2 ? (cnt + 24) / 25 : (cnt + 17) / 18;
    }
    int x = tiles;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, x, off);
      if (lane >= off) x += o;
    }
    if (g <= n_el) tp[g] = carry + x - tiles;
    carry += __shfl_sync(0xffffffffu, x, 31);
  }
}
__global__ void tile_ptr_kernel(const int* __restrict__ species_ptr, int n_el, int* tile_ptr, int* tc_tile_ptr) {
  tile_table(species_ptr, n_el, threadIdx.x >> 5, tile_ptr, tc_tile_ptr);
}

// ---- edge views ---------------------------------------------------------------------------------------------------
struct EdgeSort {
  const int64_t* src; const int64_t* dst;  // [E]; an edge with an index outside [0, n) belongs to no view (padding)
  long long E; int n;
  int *cur_dst, *cur_src;                  // [n + 1] counts, then cursors
  int *rowptr_dst, *rowptr_src;            // [n + 1]
  int *block_sums;                         // [2][blocks of the scan]
  int *by_dst, *by_src;                    // [E] bins in arrival order
  int *e_src, *e_dst, *e_orig, *perm_src;
};
struct SpeciesSort {
  const int* species; int n, n_el;  // species: inside [0, n_el)
  int *perm, *rank, *ptr, *tile_ptr, *tc_tile_ptr;  // rank: place of every atom in perm
};
constexpr int kCountThreads = 1024, kScanItems = 4, kScanBlock = 1024 * kScanItems;
constexpr int kSpeciesBlockAtoms = 8192;  // up to here one block sorts the atoms by species beside the edge count
constexpr int kSpeciesBlockElements = 256;

// Also copies the species, with 0 in the place of an index outside the element list: everything downstream addresses tables,
// counters and sorted rows with them.  (The read-out sees the caller's own index and gives such an atom a NaN.)
__global__ void edge_sort_init_kernel(EdgeSort a, const int* __restrict__ graph_ptr, int n_graphs, int* atom_graph,
                                      const int* __restrict__ species_in, int n_el, int* __restrict__ species) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i > a.n) return;
  a.cur_dst[i] = 0;
  a.cur_src[i] = 0;
  if (i == a.n) return;
  const int z = species_in[i];
  species[i] = (unsigned)z < (unsigned)n_el ? z : 0;
  int lo = 0, hi = n_graphs;  // largest g with graph_ptr[g] <= i
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (graph_ptr[mid] <= i) lo = mid; else hi = mid;
  }
  atom_graph[i] = lo;
}

// Stable counting sort of the atoms by species in one block of kCountThreads: counts, row pointers and tile tables, then the
// atoms in chunks of one per thread (rank inside the warp by match, warps in order).
__device__ void species_block(const SpeciesSort& a, int* smem) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, n_el = a.n_el;
  int* base = smem;                 // [n_el + 1]
  int* hist = smem + n_el + 1;      // [32][n_el]
  for (int k = tid; k <= n_el; k += kCountThreads) base[k] = 0;
  for (int k = tid; k < 32 * n_el; k += kCountThreads) hist[k] = 0;
  __syncthreads();
  for (int i = tid; i < a.n; i += kCountThreads) atomicAdd(&base[a.species[i] + 1], 1);
  __syncthreads();
  if (warp == 0) {
    int carry = 0;
    for (int k0 = 0; k0 <= n_el; k0 += 32) {
      const int k = k0 + lane;
      int v = k <= n_el ? base[k] : 0;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= off) v += o;
      }
      if (k <= n_el) base[k] = carry + v;
      carry += __shfl_sync(0xffffffffu, v, 31);
    }
  }
  __syncthreads();
  for (int k = tid; k <= n_el; k += kCountThreads) a.ptr[k] = base[k];
  if (warp < 8) tile_table(base, n_el, warp, a.tile_ptr, a.tc_tile_ptr);
  __syncthreads();
  for (int i0 = 0; i0 < a.n; i0 += kCountThreads) {
    const int i = i0 + tid;
    const int z = i < a.n ? a.species[i] : -1;
    const unsigned same = __match_any_sync(0xffffffffu, z);
    const int rank = __popc(same & ((1u << lane) - 1u));
    if (z >= 0 && rank == 0) hist[warp * n_el + z] = __popc(same);
    __syncthreads();
    for (int k = tid; k < n_el; k += kCountThreads) {
      int b = base[k], c[32];  // all counts read before the first offset is written: one shared-memory latency, not 32
#pragma unroll
      for (int w = 0; w < 32; ++w) c[w] = hist[w * n_el + k];
#pragma unroll
      for (int w = 0; w < 32; ++w) { hist[w * n_el + k] = b; b += c[w]; }
      base[k] = b;
    }
    __syncthreads();
    if (z >= 0) {
      const int at = hist[warp * n_el + z] + rank;
      a.perm[at] = i;
      a.rank[i] = at;
    }
    __syncthreads();
    for (int k = tid; k < 32 * n_el; k += kCountThreads) hist[k] = 0;
    __syncthreads();
  }
}

__device__ __forceinline__ bool edge_at(const EdgeSort& a, long long e, int& src, int& dst) {
  if (e >= a.E) return false;
  const int64_t s = a.src[e], d = a.dst[e];
  src = (int)s; dst = (int)d;
  return s >= 0 && s < a.n && d >= 0 && d < a.n;
}
// Adds to counter `key` for every lane with ok set, one atomic per run of equal keys of neighbouring lanes (edge lists mostly
// come grouped by target); returns the value before the run's addition plus the lane's place in the run.
__device__ __forceinline__ int run_add(int* counter, int key, bool ok) {
  const int lane = threadIdx.x & 31;
  if (!ok) key = -1 - lane;  // never part of a run
  const int prev = __shfl_up_sync(0xffffffffu, key, 1);
  const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || key != prev);
  const int head = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
  const unsigned later = head == 31 ? 0u : heads & (0xffffffffu << (head + 1));
  const int end = later ? __ffs(later) - 1 : 32;
  int base = 0;
  if (ok && lane == head) base = atomicAdd(counter + key, end - head);
  base = __shfl_sync(0xffffffffu, base, head);
  return base + lane - head;
}

__global__ void __launch_bounds__(kCountThreads) edge_count_kernel(EdgeSort a, SpeciesSort sp, int with_species) {
  extern __shared__ int smem[];
  int block = blockIdx.x, blocks = gridDim.x;
  if (with_species) {
    if (block == 0) { species_block(sp, smem); return; }
    --block; --blocks;
  }
  for (long long e0 = (long long)block * kCountThreads; e0 < a.E; e0 += (long long)blocks * kCountThreads) {
    int src = 0, dst = 0;
    const bool ok = edge_at(a, e0 + threadIdx.x, src, dst);
    run_add(a.cur_dst, dst, ok);
    if (ok) atomicAdd(a.cur_src + src, 1);
  }
}

// Exclusive scan of the counts into row pointers and cursors; blockIdx.y: target / source view.  With more than one block per
// view the block sums come from edge_block_sum_kernel.
__device__ __forceinline__ int block_exclusive_scan(int v, int* warp_sums, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += o;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int w = warp_sums[lane];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, w, off);
      if (lane >= off) w += o;
    }
    warp_sums[lane] = w;
  }
  __syncthreads();
  total = warp_sums[31];
  return x - v + (warp ? warp_sums[warp - 1] : 0);
}
__global__ void __launch_bounds__(1024) edge_block_sum_kernel(EdgeSort a) {
  __shared__ int warp_sums[32];
  const int* cnt = blockIdx.y ? a.cur_src : a.cur_dst;
  const long long i0 = (long long)blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
  int v = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) if (i0 + k < a.n) v += cnt[i0 + k];
  int total;
  block_exclusive_scan(v, warp_sums, total);
  if (threadIdx.x == 0) a.block_sums[blockIdx.y * gridDim.x + blockIdx.x] = total;
}
__global__ void __launch_bounds__(1024) edge_scan_kernel(EdgeSort a) {
  __shared__ int warp_sums[32];
  __shared__ int before;
  int* cur = blockIdx.y ? a.cur_src : a.cur_dst;
  int* rowptr = blockIdx.y ? a.rowptr_src : a.rowptr_dst;
  if (threadIdx.x < 32) {
    int v = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += 32) v += a.block_sums[blockIdx.y * gridDim.x + b];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    if (threadIdx.x == 0) before = v;
  }
  const long long i0 = (long long)blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
  int c[kScanItems], v = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) { c[k] = i0 + k < a.n ? cur[i0 + k] : 0; v += c[k]; }
  int total;
  int at = block_exclusive_scan(v, warp_sums, total) + before;  // `before` is visible after the scan's barriers
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (i0 + k <= a.n) rowptr[i0 + k] = at;
    if (i0 + k < a.n) cur[i0 + k] = at;
    at += c[k];
  }
}

__global__ void edge_scatter_kernel(EdgeSort a) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  int src = 0, dst = 0;
  const bool ok = edge_at(a, e, src, dst);
  const int at = run_add(a.cur_dst, dst, ok);
  if (ok) a.by_dst[at] = (int)e;
  // rows behind the last edge: an edge that exists, for the per-edge kernels (no atom's segment contains these rows)
  const long long tail = a.rowptr_dst[a.n] + e;
  if (tail < a.E) { a.e_src[tail] = 0; a.e_dst[tail] = 0; a.e_orig[tail] = 0; a.perm_src[tail] = 0; }
}

// Position of list[beg + j] in ascending order among the d (distinct) values of its bin.
__device__ __forceinline__ int rank_in_bin(const int* list, int beg, int d, int v) {
  int r = 0;
#pragma unroll 4
  for (int k = 0; k < d; ++k) r += list[beg + k] < v ? 1 : 0;
  return r;
}
__device__ __forceinline__ bool bin_sorted(const int* list, int beg, int d) {
  bool ok = true;
  for (int j = threadIdx.x & 31; j + 1 < d; j += 32) ok = ok && list[beg + j] < list[beg + j + 1];
  return __all_sync(0xffffffffu, ok);
}
// one warp per target: its edges in ascending order of the caller's index; every edge enters its source's bin
__global__ void edge_order_dst_kernel(EdgeSort a) {
  const int i = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  if (i >= a.n) return;
  const int beg = a.rowptr_dst[i], d = a.rowptr_dst[i + 1] - beg;
  const bool sorted = bin_sorted(a.by_dst, beg, d);
  for (int j = threadIdx.x & 31; j < d; j += 32) {
    const int v = a.by_dst[beg + j];
    const int at = beg + (sorted ? j : rank_in_bin(a.by_dst, beg, d, v));
    const int src = (int)a.src[v];
    a.e_orig[at] = v; a.e_dst[at] = i; a.e_src[at] = src;
    a.by_src[atomicAdd(a.cur_src + src, 1)] = at;
  }
}
// one warp per source: its edges in ascending order of their place in the target-sorted list
__global__ void edge_order_src_kernel(EdgeSort a) {
  const int i = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  if (i >= a.n) return;
  const int beg = a.rowptr_src[i], d = a.rowptr_src[i + 1] - beg;
  for (int j = threadIdx.x & 31; j < d; j += 32) {
    const int v = a.by_src[beg + j];
    a.perm_src[beg + rank_in_bin(a.by_src, beg, d, v)] = v;
  }
}

__global__ void chunk_bounds_kernel(const int* __restrict__ rowptr, int n_local, long long target, int n_chunks, int* atom_ptr,
                                    int* edge_ptr) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > n_chunks) return;
  int a = n_local;
  if (c < n_chunks) {  // first atom whose edge offset is >= c * target
    const long long want = c * target;
    int lo = 0, hi = n_local;
    while (lo < hi) { const int mid = (lo + hi) >> 1; if (rowptr[mid] < want) lo = mid + 1; else hi = mid; }
    a = lo;
  }
  atom_ptr[c] = a;
  edge_ptr[c] = rowptr[a];
}
__global__ void chunk_key_kernel(const int* __restrict__ e_src, long long E, int n_atoms, const int* __restrict__ edge_ptr,
                                 int n_chunks, int* keys, int* vals) {
  const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (e >= E) return;
  int lo = 0, hi = n_chunks;  // largest c with edge_ptr[c] <= e
  while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (edge_ptr[mid] <= e) lo = mid; else hi = mid; }
  keys[e] = lo * n_atoms + e_src[e];
  vals[e] = (int)e;
}

inline size_t align_up(size_t x) { return (x + 255) & ~size_t(255); }

size_t cub_sort_bytes(long long n) {
  size_t bytes = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, bytes, (const int*)nullptr, (int*)nullptr, (const int*)nullptr, (int*)nullptr,
                                  (int)n);
  return bytes;
}

}  // namespace

// The scratch serves, one after another: the edge sort (two lists of E, cursors and block sums), the sorts by species or ghost flag of
// large systems (three lists of n_atoms), and launch_chunk_src_sort (three lists of E).
size_t graph_prep_temp_bytes(long long E, int n_atoms) {
  const long long n = E > n_atoms ? E : n_atoms;
  const size_t edge = 2 * align_up(sizeof(int) * (size_t)E) + 2 * align_up(sizeof(int) * ((size_t)n_atoms + 1)) +
                      align_up(sizeof(int) * 2 * ((size_t)n_atoms / kScanBlock + 1));
  const size_t sorts = 3 * align_up(sizeof(int) * (size_t)n) + align_up(cub_sort_bytes(n));
  return (edge > sorts ? edge : sorts) + 256;
}

// Sorts that follow the edge sort reuse its scratch, which the view by sources reads.
static bool src_deferred(const GraphPrepArgs& a) {
  return a.defer_src && !a.split_rows && a.n_local <= kSpeciesBlockAtoms && a.n_elements <= kSpeciesBlockElements;
}
int graph_prep_launches(const GraphPrepArgs& a) {
  return 6 - (src_deferred(a) ? 1 : 0) + (a.n_atoms >= kScanBlock ? 1 : 0) + (a.split_rows && a.n_local > 0 ? 2 : 0) +
         (a.n_local > kSpeciesBlockAtoms || a.n_elements > kSpeciesBlockElements ? 4 : 0);
}

__global__ void invert_kernel(const int* __restrict__ perm, int n, int* __restrict__ rank) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) rank[perm[i]] = i;
}

// Arrays of the edge sort, its scratch in a.temp.
static EdgeSort edge_sort_of(const GraphPrepArgs& a) {
  unsigned char* p = static_cast<unsigned char*>(a.temp);
  auto take = [&p](size_t count) { int* r = reinterpret_cast<int*>(p); p += align_up(sizeof(int) * (count ? count : 1)); return r; };
  EdgeSort es;
  es.src = a.edge_index; es.dst = a.edge_index + a.E; es.E = a.E; es.n = a.n_atoms;
  es.by_dst = take(a.E); es.by_src = take(a.E); es.cur_dst = take((size_t)a.n_atoms + 1); es.cur_src = take((size_t)a.n_atoms + 1);
  es.block_sums = take(2 * (size_t)(a.n_atoms / kScanBlock + 1));
  es.rowptr_dst = a.rowptr_dst; es.rowptr_src = a.rowptr_src;
  es.e_src = a.e_src; es.e_dst = a.e_dst; es.e_orig = a.e_orig; es.perm_src = a.perm_src;
  return es;
}
static void order_by_source(const GraphPrepArgs& a, cudaStream_t s) {
  edge_order_src_kernel<<<(unsigned)(((long long)a.n_atoms + 7) / 8), 256, 0, s>>>(edge_sort_of(a));
}
cudaError_t launch_edge_order_src(const GraphPrepArgs& a, cudaStream_t s) {
  if (!src_deferred(a) || a.E <= 0) return cudaSuccess;
  order_by_source(a, s);
  return cudaGetLastError();
}

cudaError_t launch_graph_prep(const GraphPrepArgs& a, cudaStream_t s) {
  if (a.temp_bytes < graph_prep_temp_bytes(a.E, a.n_atoms)) return cudaErrorInvalidValue;
  const int scan_blocks = a.n_atoms / kScanBlock + 1;
  const EdgeSort es = edge_sort_of(a);
  SpeciesSort sp{a.species_safe, a.n_local, a.n_elements, a.species_perm, a.species_rank, a.species_ptr, a.tile_ptr, a.tc_tile_ptr};
  const bool small_species = a.n_local <= kSpeciesBlockAtoms && a.n_elements <= kSpeciesBlockElements;

  edge_sort_init_kernel<<<(a.n_atoms + 256) / 256, 256, 0, s>>>(es, a.graph_ptr, a.n_graphs, a.atom_graph, a.species, a.n_elements,
                                                                a.species_safe);
  long long blocks = (a.E + kCountThreads - 1) / kCountThreads;
  if (blocks > 2 * kSMs) blocks = 2 * kSMs;
  const size_t smem = small_species ? sizeof(int) * (33 * (size_t)a.n_elements + 1) : 0;
  if (blocks + small_species > 0)
    edge_count_kernel<<<(unsigned)(blocks + small_species), kCountThreads, smem, s>>>(es, sp, small_species ? 1 : 0);
  if (scan_blocks > 1) edge_block_sum_kernel<<<dim3(scan_blocks, 2), 1024, 0, s>>>(es);
  edge_scan_kernel<<<dim3(scan_blocks, 2), 1024, 0, s>>>(es);
  if (a.E > 0) {
    edge_scatter_kernel<<<(unsigned)((a.E + 255) / 256), 256, 0, s>>>(es);
    const unsigned wb = (unsigned)(((long long)a.n_atoms + 7) / 8);
    edge_order_dst_kernel<<<wb, 256, 0, s>>>(es);
    if (!src_deferred(a)) order_by_source(a, s);
  }
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;

  // sorts whose scratch overlays the edge sort's
  const long long n = a.E > a.n_atoms ? a.E : a.n_atoms;
  unsigned char* p = static_cast<unsigned char*>(a.temp);
  auto take = [&p](size_t count) { int* r = reinterpret_cast<int*>(p); p += align_up(sizeof(int) * (count ? count : 1)); return r; };
  int* keys_in = take(n); int* vals_in = take(n); int* keys_out = take(n);
  void* cub_temp = p;
  size_t cub_bytes = cub_sort_bytes(n);
  if (a.split_rows && a.n_local > 0) {  // stable one-bit sort: targets without a ghost source first
    ghost_row_key_kernel<<<(a.n_local + 255) / 256, 256, 0, s>>>(a.rowptr_dst, a.e_src, a.n_local, keys_in, vals_in);
    err = cub::DeviceRadixSort::SortPairs(cub_temp, cub_bytes, keys_in, keys_out, vals_in, a.row_ids, a.n_local, 0, 1, s);
    if (err != cudaSuccess) return err;
    lower_bound_kernel<<<1, 32, 0, s>>>(keys_out, a.n_local, a.row_split, 1);
  }
  if (!small_species) {  // species-sorted permutation of the local atoms
    int sbits = 1;
    while ((1 << sbits) < a.n_elements + 1 && sbits < 31) ++sbits;
    iota_and_key32_kernel<<<(a.n_local + 255) / 256, 256, 0, s>>>(a.species_safe, keys_in, vals_in, a.n_local);
    err = cub::DeviceRadixSort::SortPairs(cub_temp, cub_bytes, keys_in, keys_out, vals_in, a.species_perm, a.n_local, 0, sbits, s);
    if (err != cudaSuccess) return err;
    lower_bound_kernel<<<(a.n_elements + 256) / 256, 256, 0, s>>>(keys_out, a.n_local, a.species_ptr, a.n_elements);
    invert_kernel<<<(a.n_local + 255) / 256, 256, 0, s>>>(a.species_perm, a.n_local, a.species_rank);
    tile_ptr_kernel<<<1, 256, 0, s>>>(a.species_ptr, a.n_elements, a.tile_ptr, a.tc_tile_ptr);
  }
  return cudaGetLastError();
}

cudaError_t launch_chunk_bounds(const int* rowptr_dst, int n_local, long long target_edges, int n_chunks, int* atom_ptr,
                                int* edge_ptr, cudaStream_t s) {
  chunk_bounds_kernel<<<(n_chunks + 128) / 128, 128, 0, s>>>(rowptr_dst, n_local, target_edges, n_chunks, atom_ptr, edge_ptr);
  return cudaGetLastError();
}

cudaError_t launch_chunk_src_sort(const int* e_src, long long E, int n_atoms, const int* edge_ptr, int n_chunks, int* keys,
                                  int* perm, void* temp, size_t temp_bytes, cudaStream_t s) {
  if (E <= 0) return cudaSuccess;
  if ((long long)n_chunks * n_atoms >= (1LL << 31)) return cudaErrorInvalidValue;
  unsigned char* p = static_cast<unsigned char*>(temp);
  int* keys_in = reinterpret_cast<int*>(p); p += align_up(sizeof(int) * (size_t)E);
  int* vals_in = reinterpret_cast<int*>(p); p += align_up(sizeof(int) * (size_t)E);
  p += align_up(sizeof(int) * (size_t)E);
  size_t cub_bytes = cub_sort_bytes(E);
  if ((size_t)(p - static_cast<unsigned char*>(temp)) + cub_bytes > temp_bytes) return cudaErrorInvalidValue;
  int bits = 1;
  while ((1LL << bits) < (long long)n_chunks * n_atoms + 1 && bits < 31) ++bits;
  chunk_key_kernel<<<(unsigned)((E + 255) / 256), 256, 0, s>>>(e_src, E, n_atoms, edge_ptr, n_chunks, keys_in, vals_in);
  return cub::DeviceRadixSort::SortPairs(p, cub_bytes, keys_in, keys, vals_in, perm, (int)E, 0, bits, s);
}

}  // namespace tace
