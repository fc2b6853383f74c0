// Host-side engine behind the C ABI (include/tace_b200.h): model plan, weight arena,
// workspace layout and the forward / hand-written backward schedule of one
// energy + forces + virial evaluation.
//
// Schedule of one call (reference: TensorModel.forward, tace/models/adapter.py:32-41, over
// Representation.forward, tace/models/_e3nn/representation.py:302-429):
//   graph prep -> edge features + radial MLP hidden layers -> per layer:
//   [linear_up, last radial layer (GEMM), tensor-product message passing, linear_down,
//    gate, linear, product basis, per-species coefficient linears, linear (+ skip)]
//   -> read-out -> the same chain in reverse with transposed weights -> edge-vector gradients
//   -> forces / virials / stress.
#include <cuda_runtime.h>
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <type_traits>
#include <unordered_map>
#include <vector>

#include "../../include/tace_b200.h"
#include "gemm.cuh"
#include "kernels.h"
#include "tp_gen.cuh"

namespace tace {

namespace {

struct TPMeta { int NP, NX, NM, NG; const int* k; const int* base; };
struct PBMeta { int NP, NB; const int* k; const int* base; };

// L: rank of the angular features and messages; Lin: rank of the source features (< 0: scalar source)
bool tp_meta(int L, int Lin, TPMeta& m) {
#define TPM(TAG) { m = {TPX_##TAG::NP, TPX_##TAG::NX, TPX_##TAG::NM, TPX_##TAG::NG, tp_##TAG##_k, tp_##TAG##_base}; return true; }
  if (L == 1 && Lin < 0) TPM(L1_S)
  if (L == 1 && Lin == 1) TPM(L1_F)
  if (L == 2 && Lin < 0) TPM(L2_S)
  if (L == 2 && Lin == 1) TPM(L2_N1)
  if (L == 2 && Lin == 2) TPM(L2_F)
  if (L == 3 && Lin < 0) TPM(L3_S)
  if (L == 3 && Lin == 1) TPM(L3_N1)
  if (L == 3 && Lin == 2) TPM(L3_N2)
  if (L == 3 && Lin == 3) TPM(L3_F)
#undef TPM
  return false;
}
// L: rank of A; Lout: highest output rank (< 0: scalar outputs only)
bool pb_meta(int L, int Lout, PBMeta& m) {
#define PBM(TAG) { m = {PB_##TAG::NP, PB_##TAG::NB, pb_##TAG##_k, pb_##TAG##_base}; return true; }
  if (L == 1 && Lout < 0) PBM(L1_T)
  if (L == 1 && Lout == 1) PBM(L1_A)
  if (L == 2 && Lout < 0) PBM(L2_T)
  if (L == 2 && Lout == 1) PBM(L2_N1)
  if (L == 2 && Lout == 2) PBM(L2_A)
  if (L == 3 && Lout < 0) PBM(L3_T)
  if (L == 3 && Lout == 1) PBM(L3_N1)
  if (L == 3 && Lout == 2) PBM(L3_N2)
  if (L == 3 && Lout == 3) PBM(L3_A)
#undef PBM
  return false;
}

// gated bilinear product (two different factors, the second extended by a block of ones)
bool pbl_meta(int L, int Lout, PBMeta& m) {
#define PBM(TAG) { m = {PBL_##TAG::NP, PBL_##TAG::NB, pbl_##TAG##_k, pbl_##TAG##_base}; return true; }
  if (L == 1 && Lout < 0) PBM(L1_T)
  if (L == 1 && Lout == 1) PBM(L1_A)
  if (L == 2 && Lout < 0) PBM(L2_T)
  if (L == 2 && Lout == 1) PBM(L2_N1)
  if (L == 2 && Lout == 2) PBM(L2_A)
  if (L == 3 && Lout < 0) PBM(L3_T)
  if (L == 3 && Lout == 1) PBM(L3_N1)
  if (L == 3 && Lout == 2) PBM(L3_N2)
  if (L == 3 && Lout == 3) PBM(L3_A)
#undef PBM
  return false;
}

// third-order basis (correlation 3): L = rank of A, Lout as above
bool pb3_meta(int L, int Lout, PBMeta& m) {
#define PBM(TAG) { m = {PB3_##TAG::NP, PB3_##TAG::NB, pb3_##TAG##_k, pb3_##TAG##_base}; return true; }
  if (L == 1 && Lout < 0) PBM(L1_T)
  if (L == 1 && Lout == 1) PBM(L1_A)
  if (L == 2 && Lout < 0) PBM(L2_T)
  if (L == 2 && Lout == 1) PBM(L2_N1)
  if (L == 2 && Lout == 2) PBM(L2_A)
  if (L == 3 && Lout < 0) PBM(L3_T)
  if (L == 3 && Lout == 1) PBM(L3_N1)
  if (L == 3 && Lout == 2) PBM(L3_N2)
  if (L == 3 && Lout == 3) PBM(L3_A)
#undef PBM
  return false;
}

struct WeightEntry {
  std::string name;
  long long numel;
  long long offset;  // elements into the arena
  bool set;
};

struct LayerPlan {
  bool scalar_src, last, has_res;
  bool tece = false;        // the interaction is the TECE edge block (atomic_basis.type = uv_so2) instead of the tensor product
  TPMeta tp;
  PBMeta pb;                // second-order product basis (all ranks <= L when a third order follows)
  PBMeta pb3;               // third-order product basis (correlation 3)
  int pb_lout;              // output-rank argument of the second-order kernels
  int Din;                  // components per atom of the layer input (1 or D)
  int Dout;                 // components per atom of the layer output (D or 1)
  std::vector<int> in_ls;   // ranks present in the input
  std::vector<int> out_ls;  // ranks present in the output
};

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Bump allocator over the caller's workspace; in "measure" mode it only counts.
struct Arena {
  unsigned char* base = nullptr;
  size_t used = 0;
  template <typename U>
  U* take(size_t count) {
    U* p = base ? reinterpret_cast<U*>(base + used) : nullptr;
    used += align256(sizeof(U) * (count ? count : 1));
    return p;
  }
};

}  // namespace

struct ModelBase {
  TaceConfig cfg;
  virtual ~ModelBase() {
    if (ev_fork) cudaEventDestroy(ev_fork);
    if (ev_join) cudaEventDestroy(ev_join);
    if (ev_branch) cudaEventDestroy(ev_branch);
    if (ev_merge) cudaEventDestroy(ev_merge);
  }
  // Branches of a pass that is being captured: `branch` gives the stream for work that depends on what `s` has so far and that
  // nothing on `s` needs before the next `merge`.  In a pass that is launched kernel by kernel both do nothing and the work
  // goes to `s`.
  bool branches = false;  // the running pass is captured and has branch_stream at its disposal
  bool branch_open = false;
  cudaStream_t branch_stream = nullptr;
  cudaEvent_t ev_branch = nullptr, ev_merge = nullptr;
  int branch(cudaStream_t s, cudaStream_t* side) {
    *side = s;
    if (!branches) return TACE_OK;
    if (cudaEventRecord(ev_branch, s) != cudaSuccess || cudaStreamWaitEvent(branch_stream, ev_branch, 0) != cudaSuccess) return TACE_ERR_CUDA;
    *side = branch_stream;
    branch_open = true;
    return TACE_OK;
  }
  int merge(cudaStream_t s) {
    if (!branch_open) return TACE_OK;
    branch_open = false;
    if (cudaEventRecord(ev_merge, branch_stream) != cudaSuccess || cudaStreamWaitEvent(s, ev_merge, 0) != cudaSuccess) return TACE_ERR_CUDA;
    return TACE_OK;
  }
  // Branches end where a pass fills the chip by itself; the line is the last size at which no kind of model loses by them.  One pass
  // without -> with them, in us.  Edge block (rank 3, 128 channels): 8 200 edges 1 760 -> 1 646, 28 000: 4 457 -> 4 412, 66 000: 10 018 ->
  // 9 927, 94 000: 13 663 -> 13 685, 128 000: 18 634 -> 18 824, 526 000: 74 207 -> 75 390.  Radial table: rank 2, 64 channels, 11 000: 205 ->
  // 201, 59 000: 409 -> 407, 88 000: 525 -> 523, 469 000: 1 972 -> 1 975; rank 3, 128 channels, 21 000: 643 -> 641, even above.  fp32 with
  // weights in memory (rank 3, 128 channels): 21 000: 1 375 -> 1 356, 59 000: 2 818 -> 2 808, even above.  Double precision (rank 2, 64
  // channels) gains above the line too: 11 000: 535 -> 497, 59 000: 1 961 -> 1 888, 88 000: 2 609 -> 2 542, 171 000: 4 877 -> 4 762.
  static constexpr int64_t kBranchEdges = 1 << 16;
  // Streams and events of a captured pass.  With the fp64 products of the radial MLPs (thousands of blocks) on a branch, the main line
  // takes the higher priority, so that its small kernels do not stand in line behind them (two frames of 256 atoms 1 439 -> 1 374 us).  The edge
  // block's main line is large products with small kernels on the branch; there it loses (two frames of 128 atoms 3 671 us without, 3 745 with).
  virtual bool main_line_first() const = 0;
  bool capture_streams() {
    if (capture_stream) return true;
    int least = 0, greatest = 0;
    if (main_line_first() && cudaDeviceGetStreamPriorityRange(&least, &greatest) != cudaSuccess) return false;
    if (!ev_branch && cudaEventCreateWithFlags(&ev_branch, cudaEventDisableTiming) != cudaSuccess) return false;
    if (!ev_merge && cudaEventCreateWithFlags(&ev_merge, cudaEventDisableTiming) != cudaSuccess) return false;
    if (!branch_stream && cudaStreamCreateWithPriority(&branch_stream, cudaStreamNonBlocking, least) != cudaSuccess) return false;
    return cudaStreamCreateWithPriority(&capture_stream, cudaStreamNonBlocking, greatest) == cudaSuccess;
  }
  // Runs the exchange callback.  Without an exchange stream: on the stream of the pass (after a host synchronisation when
  // the callback asks for one).  With one: everything enqueued on `s` so far happens before the callback's work, which
  // runs on the exchange stream; the pass goes on with `s` and calls exchange_join before it touches the callback's output.
  bool exchange_on_side() const { return exchange_stream != nullptr && !exchange_sync; }
  int exchange_begin(int reverse, const void* in, void* out, long long n_rows, int row, cudaStream_t s) {
    const bool side = exchange_on_side();
    if (side) {
      if (!ev_fork && (cudaEventCreateWithFlags(&ev_fork, cudaEventDisableTiming) != cudaSuccess ||
                       cudaEventCreateWithFlags(&ev_join, cudaEventDisableTiming) != cudaSuccess))
        return TACE_ERR_CUDA;
      if (cudaEventRecord(ev_fork, s) != cudaSuccess || cudaStreamWaitEvent(exchange_stream, ev_fork, 0) != cudaSuccess)
        return TACE_ERR_CUDA;
    } else if (exchange_sync && cudaStreamSynchronize(s) != cudaSuccess) {
      return TACE_ERR_CUDA;
    }
    if (exchange_fn(exchange_user, reverse, in, out, n_rows, row) != 0) return TACE_ERR_INVALID_ARGUMENT;
    if (side && cudaEventRecord(ev_join, exchange_stream) != cudaSuccess) return TACE_ERR_CUDA;
    return TACE_OK;
  }
  int exchange_join(cudaStream_t s) {
    if (exchange_on_side() && cudaStreamWaitEvent(s, ev_join, 0) != cudaSuccess) return TACE_ERR_CUDA;
    return TACE_OK;
  }
  virtual int weight_count() const = 0;
  virtual int weight_info(int i, const char** name, int64_t* numel) const = 0;
  virtual int set_weight(const char* name, const void* host, int64_t numel) = 0;
  virtual int workspace_bytes(int64_t n_atoms, int64_t n_local, int64_t n_edges, int32_t n_graphs, size_t* bytes) = 0;
  virtual int forward(const TaceBatch* b, const TaceOutputs* o, void* ws, size_t ws_bytes, cudaStream_t s) = 0;
  virtual int64_t debug_read(const char* name, void* dst, int64_t numel, cudaStream_t s) = 0;

  // kernel-launch counter and optional per-phase CUDA-event timing
  long long launches = 0;
  // Batches with more edges than this are evaluated in chunks of target atoms: the per-edge tensors (radial-MLP
  // activations, path weights, per-edge source gradients) then exist for one chunk at a time and the backward pass
  // recomputes them, so memory per edge drops from kilobytes to about two hundred bytes.
  long long max_chunk_edges = 1LL << 21;
  tace_exchange_fn exchange_fn = nullptr;  // ghost-row exchange between layers (edge-vector mode)
  void* exchange_user = nullptr;
  bool exchange_sync = true;                // synchronise the stream before every exchange callback (tace_set_exchange_sync)
  // Stream on which the exchange callback enqueues its work (tace_set_exchange_stream).  The pass then orders the callback
  // against its own stream with events and keeps computing what does not need the ghost rows while they travel.
  cudaStream_t exchange_stream = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  int* dev_error = nullptr;  // device word written by kernels whose bounded waits expire
  bool profile = false;
  std::vector<std::string> phase_names;
  std::vector<cudaEvent_t> phase_events;
  size_t phase_used = 0;
  void phase(const char* name, cudaStream_t s) {
    if (!profile) return;
    if (phase_used == phase_events.size()) {
      cudaEvent_t e;
      if (cudaEventCreate(&e) != cudaSuccess) return;
      phase_events.push_back(e);
      phase_names.push_back("");
    }
    phase_names[phase_used] = name;
    cudaEventRecord(phase_events[phase_used], s);
    ++phase_used;
  }
  int phase_count() const { return phase_used > 0 ? (int)phase_used - 1 : 0; }
  int phase_read(int i, const char** name, float* ms) {
    if (i < 0 || i >= phase_count()) return TACE_ERR_INVALID_ARGUMENT;
    if (cudaEventSynchronize(phase_events[i + 1]) != cudaSuccess) return TACE_ERR_CUDA;
    if (cudaEventElapsedTime(ms, phase_events[i], phase_events[i + 1]) != cudaSuccess) return TACE_ERR_CUDA;
    *name = phase_names[i].c_str();
    return TACE_OK;
  }
  void release_events() {
    for (auto e : phase_events) cudaEventDestroy(e);
    phase_events.clear();
  }

  // ---- CUDA-graph replay ------------------------------------------------------------------------
  // A forward pass is several hundred short launches whose arguments depend only on the batch
  // sizes and the workspace address.  The second call with the same sizes is captured into a CUDA
  // graph on a private stream; from then on inputs are copied into a staging area at the end of
  // the workspace, the graph is launched on the caller's stream, and results are copied out, so
  // the caller's input and output pointers may change freely between calls.
  // The edge count of a structure that moves changes with every evaluation, so graphs are captured for a capacity: the
  // count rounded up to a multiple of 64 (up to 2 048 edges) or of a power of two between 1/32 and 1/16 of it, the staged edge
  // list padded with edges that belong to no atom.  Above 131 072 edges a pass is long enough for its launches to hide and the padding rows would
  // cost more than they save: exact counts there.
  static int64_t round_edges(int64_t E) {  // a multiple of its own step, so rounding it again changes nothing
    if (E <= 0 || E > (1 << 17)) return E;
    int64_t step = 64;
    while (step * 32 < E) step *= 2;
    return (E + step - 1) / step * step;
  }
  int64_t edge_capacity(int64_t E) const { return graph_mode && round_edges(E) <= max_chunk_edges ? round_edges(E) : E; }
  struct GraphKey {
    int64_t n_atoms, n_local, n_edges;  // n_edges: the capacity
    int32_t n_graphs, vec_mode;  // vec_mode bit 0: edge-vector input; bit 1: a fidelity array is given
    uint32_t out_mask;
    void* ws;
    size_t ws_bytes;
    bool operator==(const GraphKey& o) const {
      return n_atoms == o.n_atoms && n_local == o.n_local && n_edges == o.n_edges && n_graphs == o.n_graphs &&
             vec_mode == o.vec_mode && out_mask == o.out_mask && ws == o.ws && ws_bytes == o.ws_bytes;
    }
  };
  struct GraphEntry { GraphKey key; cudaGraphExec_t exec; long long launches; unsigned long long last_use; };
  static constexpr size_t kMaxGraphs = 4, kMaxSeen = 16;
  int graph_mode = 1;
  std::vector<GraphKey> seen, rejected;
  std::vector<GraphEntry> graphs;
  cudaStream_t capture_stream = nullptr;
  unsigned long long graph_clock = 0;
  long long graph_replays = 0;

  struct Stage {  // byte offsets (from the staging base) of the copies of every input and output
    size_t positions, lattice, species, graph_ptr, edge_index, edge_shifts, edge_vector, fidelity;
    size_t energy, node_energy, forces, virials, stress, edge_forces, total;
  };
  Stage stage_layout(int64_t N, int64_t NL, int64_t E, int32_t B) const {
    const size_t ts = cfg.dtype == TACE_F32 ? 4 : 8;
    Stage st;
    size_t off = 0;
    auto take = [&off](size_t bytes) { const size_t at = off; off += align256(bytes ? bytes : 1); return at; };
    st.positions = take(ts * 3 * N); st.lattice = take(ts * 9 * B); st.species = take(4 * (size_t)N);
    st.graph_ptr = take(4 * (size_t)(B + 1)); st.edge_index = take(16 * (size_t)E); st.edge_shifts = take(ts * 3 * E);
    st.edge_vector = take(ts * 3 * E); st.fidelity = take(4 * (size_t)B);
    st.energy = take(ts * B); st.node_energy = take(ts * NL); st.forces = take(ts * 3 * N); st.virials = take(ts * 9 * B);
    st.stress = take(ts * 9 * B); st.edge_forces = take(ts * 3 * E);
    st.total = off;
    return st;
  }
  void release_graphs() {
    for (auto& g : graphs) cudaGraphExecDestroy(g.exec);
    graphs.clear(); seen.clear(); rejected.clear();
    if (capture_stream) { cudaStreamDestroy(capture_stream); capture_stream = nullptr; }
    if (branch_stream) { cudaStreamDestroy(branch_stream); branch_stream = nullptr; }
  }

  int forward_entry(const TaceBatch* bt, const TaceOutputs* o, void* ws, size_t ws_bytes, cudaStream_t s) {
    if (!bt || !o || !ws) return TACE_ERR_INVALID_ARGUMENT;
    const int64_t N = bt->n_atoms, NL = bt->n_local, E = bt->n_edges;
    const int32_t B = bt->n_graphs;
    if (!graph_mode || profile || exchange_fn || N <= 0 || E <= 0 || B <= 0 || NL < 0 || NL > N || E > max_chunk_edges)
      return forward(bt, o, ws, ws_bytes, s);
    const int64_t Ecap = edge_capacity(E);
    const Stage st = stage_layout(N, NL, Ecap, B);
    if (ws_bytes < st.total + 256) return forward(bt, o, ws, ws_bytes, s);
    const size_t body_bytes = (ws_bytes - st.total) & ~size_t(255);
    unsigned char* sb = static_cast<unsigned char*>(ws) + body_bytes;
    GraphKey key{N, NL, Ecap, B, (bt->edge_vector ? 1 : 0) | (bt->fidelity ? 2 : 0), 0u, ws, ws_bytes};
    const bool vec_in = bt->edge_vector != nullptr;
    const void* outs[6] = {o->energy, o->node_energy, o->forces, o->virials, o->stress, o->edge_forces};
    for (int k = 0; k < 6; ++k) if (outs[k]) key.out_mask |= 1u << k;
    // inputs the pass reads (all must be present for the staged path)
    if (!bt->species || !bt->graph_ptr || !bt->edge_index) return forward(bt, o, ws, ws_bytes, s);
    if (!vec_in && (!bt->positions || !bt->lattice || !bt->edge_shifts)) return forward(bt, o, ws, ws_bytes, s);

    GraphEntry* hit = nullptr;
    for (auto& g : graphs) if (g.key == key) hit = &g;
    if (!hit) {
      for (const auto& r : rejected) if (r == key) return forward(bt, o, ws, ws_bytes, s);
      bool was_seen = false;
      for (const auto& k : seen) if (k == key) was_seen = true;
      if (!was_seen) {  // first call with these sizes: run it directly (also configures kernel attributes)
        if (seen.size() >= kMaxSeen) seen.erase(seen.begin());
        seen.push_back(key);
        return forward(bt, o, ws, ws_bytes, s);
      }
      // second call: capture a pass that works on the staged copies
      if (!capture_streams()) return forward(bt, o, ws, ws_bytes, s);
      TaceBatch sbt = *bt;
      sbt.n_edges = Ecap;
      TaceOutputs so;
      const size_t ts = cfg.dtype == TACE_F32 ? 4 : 8;
      (void)ts;
      sbt.species = reinterpret_cast<const int32_t*>(sb + st.species);
      sbt.graph_ptr = reinterpret_cast<const int32_t*>(sb + st.graph_ptr);
      sbt.edge_index = reinterpret_cast<const int64_t*>(sb + st.edge_index);
      sbt.positions = vec_in ? nullptr : sb + st.positions;
      sbt.lattice = vec_in ? nullptr : sb + st.lattice;
      sbt.edge_shifts = vec_in ? nullptr : sb + st.edge_shifts;
      sbt.edge_vector = vec_in ? sb + st.edge_vector : nullptr;
      sbt.fidelity = bt->fidelity ? reinterpret_cast<const int32_t*>(sb + st.fidelity) : nullptr;
      so.energy = o->energy ? sb + st.energy : nullptr;
      so.node_energy = o->node_energy ? sb + st.node_energy : nullptr;
      so.forces = o->forces ? sb + st.forces : nullptr;
      so.virials = o->virials ? sb + st.virials : nullptr;
      so.stress = o->stress ? sb + st.stress : nullptr;
      so.edge_forces = o->edge_forces ? sb + st.edge_forces : nullptr;
      const long long before = launches;
      cudaGraph_t graph = nullptr;
      cudaGraphExec_t exec = nullptr;
      bool ok = cudaStreamBeginCapture(capture_stream, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
      if (ok) {
        branches = Ecap <= kBranchEdges;
        const int status = forward(&sbt, &so, ws, body_bytes, capture_stream);
        branches = branch_open = false;
        const cudaError_t ce = cudaStreamEndCapture(capture_stream, &graph);
        ok = status == TACE_OK && ce == cudaSuccess && graph != nullptr;
      }
      const long long per_pass = launches - before;
      launches = before;
      if (ok) ok = cudaGraphInstantiate(&exec, graph, main_line_first() ? cudaGraphInstantiateFlagUseNodePriority : 0) == cudaSuccess;
      if (graph) cudaGraphDestroy(graph);
      if (!ok) {
        cudaGetLastError();  // a failed capture leaves a sticky-free error behind; this sizes runs without a graph
        rejected.push_back(key);
        return forward(bt, o, ws, ws_bytes, s);
      }
      if (graphs.size() >= kMaxGraphs) {
        size_t oldest = 0;
        for (size_t k = 1; k < graphs.size(); ++k) if (graphs[k].last_use < graphs[oldest].last_use) oldest = k;
        cudaGraphExecDestroy(graphs[oldest].exec);
        graphs.erase(graphs.begin() + oldest);
      }
      graphs.push_back({key, exec, per_pass, 0});
      hit = &graphs.back();
    }
    hit->last_use = ++graph_clock;
    const size_t ts = cfg.dtype == TACE_F32 ? 4 : 8;
    // one kernel gathers the caller's inputs, one hands out the results (eleven separate copies left about 4 us of idle GPU each)
    CopySegments in, out;
    in.add(sb + st.species, bt->species, 4 * (size_t)N);
    in.add(sb + st.graph_ptr, bt->graph_ptr, 4 * (size_t)(B + 1));
    in.add(sb + st.edge_index, bt->edge_index, 8 * (size_t)E);
    in.add(sb + st.edge_index + 8 * (size_t)Ecap, bt->edge_index + E, 8 * (size_t)E);
    in.pad = reinterpret_cast<int64_t*>(sb + st.edge_index); in.pad_from = E; in.pad_to = Ecap;
    if (bt->fidelity) in.add(sb + st.fidelity, bt->fidelity, 4 * (size_t)B);
    if (vec_in) {
      in.add(sb + st.edge_vector, bt->edge_vector, ts * 3 * E);
    } else {
      in.add(sb + st.positions, bt->positions, ts * 3 * N);
      in.add(sb + st.lattice, bt->lattice, ts * 9 * B);
      in.add(sb + st.edge_shifts, bt->edge_shifts, ts * 3 * E);
    }
    if (o->energy) out.add(o->energy, sb + st.energy, ts * B);
    if (o->node_energy) out.add(o->node_energy, sb + st.node_energy, ts * NL);
    if (o->forces) out.add(o->forces, sb + st.forces, ts * 3 * N);
    if (o->virials) out.add(o->virials, sb + st.virials, ts * 9 * B);
    if (o->stress) out.add(o->stress, sb + st.stress, ts * 9 * B);
    if (o->edge_forces) out.add(o->edge_forces, sb + st.edge_forces, ts * 3 * E);
    const bool ok = launch_copy_segments(in, s) == cudaSuccess && cudaGraphLaunch(hit->exec, s) == cudaSuccess &&
                    launch_copy_segments(out, s) == cudaSuccess;
    launches += hit->launches + 2;
    ++graph_replays;
    return ok ? TACE_OK : TACE_ERR_CUDA;
  }
};

template <typename T>
struct Model : ModelBase {
  int L, Ln, D, C, NL_, n_el, H;
  int nh = 3;                 // hidden layers of the radial MLP (radial_basis.hidden)
  bool mlp_bias = false;      // radial_basis.bias
  bool env_after = false;     // radial_basis.apply_cutoff = False: envelope multiplies the MLP output
  bool element2 = false;      // edge_update.type = element2
  int n_fid = 1;              // read-out heads (entries of `statistics`)
  int zbl = 0;                // 0 off, 1 ZBL repulsion inside the species scale, 2 outside it
  int density = 0;            // atomic_basis.scatter_norm: 0 avg_num_neighbors, 1 density, 2 no_cutoff_density
  bool res_identity = false;  // resnet.linear_type = identity: the skip connection copies the matching ranks, no weights
  bool bilinear = false;      // product_basis.nonlinear = silu_bilineargate: gated product of two linear images of A
  // TECE edge block: layers (bit t), orders kept, heads, width of the cluster expansion, activation (0 sigmoid, 1 SiLU)
  int tece_mask = 0, mmax = 2, heads = 1, Ca = 0, edge_act = 0;
  int rt_K = 0;               // > 0: path weights interpolated from per-layer tables with rt_K intervals (TaceConfig.radial_table)
  int t_NR = 0, t_NC = 0, t_NF = 0, t_G = 0, t_np = 0, t_WN = 0;  // rows (order-major / per weight / full), gates, paths, coefficients
  int t_k[4] = {1, 1, 1, 1}, t_base[4] = {0, 1, 4, 9};            // message layout of a TECE layer: one block of C per rank
  int t_wg = 0;  // packed Wigner entries per edge
  double t_row_scale[16], t_p_scale[12];
  int m0 = 1;  // 1: every rank gated (gate_m0 = True); 0: e3nn Gate, scalars through SiLU (gate_m0 = False)
  std::vector<LayerPlan> layers;
  std::vector<WeightEntry> weights;  // the first n_listed are the caller's, n_unset of them not set yet; the others are folded from them
  int n_listed = 0, n_unset = 0;
  bool folded = true;
  int device = 0;  // holds the arena
  std::unordered_map<std::string, int> weight_index;
  T* arena = nullptr;
  long long arena_numel = 0;
  // perm: the `row` elements of atom i are row perm[i] (nullptr: atom order)
  struct DebugBuf { std::string name; const void* ptr; long long numel; const int* perm = nullptr; long long row = 0; };
  std::vector<DebugBuf> debug;
  T host_bessel[kNumBessel + 1];  // host copies of the radial frequencies and prefactor

  ~Model() override {
    if (arena) cudaFree(arena);
    if (dev_error) cudaFree(dev_error);
    release_events();
  }
  static constexpr bool kTensorCore = sizeof(T) == 4;  // fp32 models run the radial GEMMs on tcgen05

  void add_weight(const std::string& name, long long numel) {
    weight_index.emplace(name, (int)weights.size());
    weights.push_back({name, numel, arena_numel, false});
    arena_numel += (numel + 63) / 64 * 64;
  }
  // a channel-mixing matrix used by the tensor-core path also comes as its TF32 high part and residual
  void add_linear_weight(const std::string& name, long long numel) {
    add_weight(name, numel);
    if (kTensorCore) { add_weight(name + "_hi", numel); add_weight(name + "_lo", numel); }
  }
  // The same for a [K][N] matrix per group, X, which the linears of the backward pass read, and its transpose, which those of the forward pass do;
  // backward, forward: whether they may take FP16 parts.  Every other array would be packed for nothing.
  void add_packed_weight(const std::string& name, const std::string& nameT, int groups, long long K, long long N, bool tiled, bool backward, bool forward) {
    add_linear_weight(name, groups * K * N);
    add_linear_weight(nameT, groups * K * N);
    if (kTensorCore && backward && tc_linear_supported((int)K, (int)N)) pack_shapes[name] = {groups, (int)K, (int)N, tiled};
    if (kTensorCore && forward && tc_linear_supported((int)N, (int)K)) pack_shapes[nameT] = {groups, (int)N, (int)K, tiled};
  }
  // What the tensor cores read of them: "X_pk", FP16 parts of X_hi + X_lo with every column of the result scaled by a power of two, and behind
  // them the inverse scales.
  struct Packed { const float* B; const float* inv; };
  struct PackShape { int groups, N, K; bool tiled; };
  std::map<std::string, PackShape> pack_shapes;  // by the name of the array, X
  Packed packed(const std::string& name) const {
    const auto it = weight_index.find(name + "_pk");
    if (it == weight_index.end()) return {nullptr, nullptr};
    const WeightEntry& e = weights[it->second];
    const float* B = reinterpret_cast<const float*>(arena + e.offset);
    const PackShape& sh = pack_shapes.at(name);
    return {B, B + (long long)sh.groups * sh.N * sh.K};
  }
  cudaError_t pack_weight(const std::string& name) {
    const auto it = weight_index.find(name + "_pk");
    if (it == weight_index.end()) return cudaSuccess;
    const WeightEntry& e = weights[it->second];
    float* B = reinterpret_cast<float*>(arena + e.offset);
    const PackShape& sh = pack_shapes.at(name);
    return launch_tc_pack(reinterpret_cast<const float*>(w(name + "_hi")), reinterpret_cast<const float*>(w(name + "_lo")), sh.groups, sh.N, sh.K, sh.tiled,
                          B, B + (long long)sh.groups * sh.N * sh.K, cudaStream_t(0));
  }
  const T* w(const std::string& name) const {
    const auto it = weight_index.find(name);
    return it == weight_index.end() ? nullptr : arena + weights[it->second].offset;
  }

  int init(const TaceConfig& c) {
    cfg = c;
    L = c.L; D = (L + 1) * (L + 1); C = c.num_channel; NL_ = c.num_layers; n_el = c.num_elements; H = c.readout_hidden;
    m0 = c.gate_m0_off ? 0 : 1;
    nh = (c.mlp_layers > 0) ? c.mlp_layers : 3;  // hidden layers of the radial MLP
    if (nh < 1 || nh > 3) return TACE_ERR_UNSUPPORTED_CONFIG;
    mlp_bias = c.mlp_bias != 0; env_after = c.env_after_mlp != 0; element2 = c.edge_update_element2 != 0;
    n_fid = c.num_fidelities > 0 ? c.num_fidelities : 1;
    zbl = c.zbl;
    density = c.scatter_norm_density;
    res_identity = c.resnet_identity != 0;
    bilinear = c.product_bilinear != 0;
    tece_mask = c.tece_layers; folded = tece_mask == 0; mmax = c.mmax; heads = c.num_head > 0 ? c.num_head : 1;
    rt_K = c.radial_table;
    if (rt_K < 0 || (rt_K > 0 && (!std::is_same<T, float>::value || element2 || tece_mask || rt_K > (1 << 16))))
      return TACE_ERR_UNSUPPORTED_CONFIG;
    Ca = c.edge_ace_hidden > 0 ? c.edge_ace_hidden : c.num_channel; edge_act = c.edge_act;
    if (tece_mask) {
      // the block needs ranks above 0 on its input (not the first layer), node rank = edge rank, orders <= 2
      if ((tece_mask & 1) || (c.Lnode > 0 && c.Lnode != c.L) || mmax < 0 || mmax > 2 || mmax > c.L || heads > 16 || C % heads ||
          Ca % 4 || density || (edge_act != 0 && edge_act != 1))
        return TACE_ERR_UNSUPPORTED_CONFIG;
      const int n = L + 1;
      t_NR = 0; t_NC = 0;
      for (int m = 0; m <= mmax; ++m) {
        for (int sign = 1; sign >= (m ? -1 : 1); sign -= 2)
          for (int l = m; l <= L; ++l) t_row_scale[t_NR++] = l > mmax ? std::sqrt((2.0 * l + 1.0) / (2.0 * mmax + 1.0)) : 1.0;
        t_NC += L + 1 - m;
      }
      t_NF = n + 2 * n * mmax;
      t_G = n * (mmax + 1 - (m0 ? 0 : 1));
      // cluster-expansion paths, output order major (oam_2026_07_05.py:331-369 with m1 >= m2)
      t_np = 0;
      for (int m3 = 0; m3 <= mmax; ++m3) {
        const int first = t_np;
        for (int m1 = 0; m1 <= mmax; ++m1)
          for (int m2 = 0; m2 <= m1; ++m2) {
            const bool sum = (m1 + m2 == m3), diff = !sum && (m1 - m2 == m3);
            if (!sum && !diff) continue;
            ++t_np;
          }
        for (int q = first; q < t_np; ++q) t_p_scale[q] = 1.0 / std::sqrt((double)(t_np - first));
      }
      t_WN = t_np * n * Ca;
      t_wg = tece_wigner_stride(L, mmax);
    }
    if (bilinear && c.correlation != 2) return TACE_ERR_UNSUPPORTED_CONFIG;
    if (zbl < 0 || zbl > 2 || density < 0 || density > 2 || (density && element2)) return TACE_ERR_UNSUPPORTED_CONFIG;
    Ln = (c.Lnode > 0) ? c.Lnode : L;  // node features between layers carry ranks 0..Ln; A, Y and the messages 0..L
    if (Ln > L || (Ln < L && c.correlation < 2)) return TACE_ERR_UNSUPPORTED_CONFIG;
    const int Dn = (Ln + 1) * (Ln + 1);
    layers.resize(NL_);
    for (int t = 0; t < NL_; ++t) {
      LayerPlan& p = layers[t];
      p.scalar_src = (t == 0);
      p.last = (t == NL_ - 1);
      p.has_res = (t > 0);
      const int lout = p.last ? -1 : Ln;
      p.pb_lout = (c.correlation == 3) ? L : lout;  // with a third order the second keeps every rank (prod.py:216-266)
      p.pb3 = PBMeta{0, 0, nullptr, nullptr};
      if (!tp_meta(L, p.scalar_src ? -1 : Ln, p.tp) || !(bilinear ? pbl_meta(L, p.pb_lout, p.pb) : pb_meta(L, p.pb_lout, p.pb)))
        return TACE_ERR_UNSUPPORTED_CONFIG;
      if (c.correlation == 3 && !pb3_meta(L, lout, p.pb3)) return TACE_ERR_UNSUPPORTED_CONFIG;
      p.tece = (tece_mask >> t) & 1;
      if (p.tece) p.tp = TPMeta{2 * t_NC, D, D, 0, t_k, t_base};  // radial weights [NC][2C]; messages one C-block per rank
      p.Din = p.scalar_src ? 1 : Dn;
      p.Dout = p.last ? 1 : Dn;
      p.in_ls.clear(); p.out_ls.clear();
      for (int l = 0; l <= (p.scalar_src ? 0 : Ln); ++l) p.in_ls.push_back(l);
      for (int l = 0; l <= (p.last ? 0 : Ln); ++l) p.out_ls.push_back(l);
    }
    add_weight("emb", (long long)n_el * C);
    add_weight("bessel", kNumBessel);
    add_weight("bessel_pref", 1);
    for (int t = 0; t < NL_; ++t) {
      const LayerPlan& p = layers[t];
      const std::string pre = "t" + std::to_string(t) + ".";
      for (int l : p.in_ls) { add_linear_weight(pre + "up.l" + std::to_string(l), (long long)C * C); add_linear_weight(pre + "upT.l" + std::to_string(l), (long long)C * C); }
      add_weight(pre + "up.b", C);
      if (rt_K) add_weight(pre + "rtab", (long long)rt_K * p.tp.NP * C * 4);
      add_weight(pre + "A0", kNumBessel * kHidden);
      if (nh >= 2) { add_linear_weight(pre + "A1", kHidden * kHidden); add_linear_weight(pre + "A1t", kHidden * kHidden); }
      if (nh >= 3) { add_linear_weight(pre + "A2", kHidden * kHidden); add_linear_weight(pre + "A2t", kHidden * kHidden); }
      if (mlp_bias) {
        add_weight(pre + "b0", kHidden);
        if (nh >= 2) add_weight(pre + "b1", kHidden);
        if (nh >= 3) add_weight(pre + "b2", kHidden);
        add_weight(pre + "b3", (long long)p.tp.NP * C);
      }
      if (p.tece) {
        for (int i = 0; i < 6; ++i) {
          const So2Shape sh = so2_shape(i);
          for (int m = 0; m <= sh.mm; ++m) {
            add_packed_weight(pre + "so2." + sh.name + ".m" + std::to_string(m), pre + "so2." + sh.name + "T.m" + std::to_string(m), 1,
                              (long long)sh.n_in[m] * sh.c_in, (long long)sh.n_out[m] * sh.c_out, false, true, true);
          }
          add_weight(pre + "so2." + sh.name + ".b", (long long)sh.n_out[0] * sh.c_out);
        }
        add_weight(pre + "att.temp", heads); add_weight(pre + "att.rw", (long long)kNumBessel * 2 * heads); add_weight(pre + "att.rb", 2 * heads);
      }
      if (density) {  // edge-density MLP 8 -> 64 -> 1 and the affine parameters {alpha, beta}
        add_weight(pre + "dA0", (long long)kNumBessel * kHidden); add_weight(pre + "dw1", kHidden); add_weight(pre + "dab", 2);
        if (mlp_bias) { add_weight(pre + "db0", kHidden); add_weight(pre + "db1", 1); }
      }
      if (element2) {
        add_weight(pre + "tdst", (long long)n_el * kHidden); add_weight(pre + "tsrc", (long long)n_el * kHidden);
        // edge features wider than the radial basis put a LayerNorm before every hidden activation of the radial MLP
        // (tace/models/_e3nn/base.py:183-185, tace/models/mlp.py:172-176): affine weights per hidden layer
        for (int j = 0; j < nh; ++j) {
          add_weight(pre + "ln" + std::to_string(j) + "g", kHidden); add_weight(pre + "ln" + std::to_string(j) + "b", kHidden);
        }
      }
      add_weight(pre + "W3", (long long)kHidden * p.tp.NP * C);
      add_weight(pre + "W3t", (long long)kHidden * p.tp.NP * C);
      if (kTensorCore) {  // TF32 high parts and residuals of both orientations
        add_weight(pre + "W3_hi", (long long)kHidden * p.tp.NP * C);
        add_weight(pre + "W3_lo", (long long)kHidden * p.tp.NP * C);
        add_weight(pre + "W3t_hi", (long long)kHidden * p.tp.NP * C);
        add_weight(pre + "W3t_lo", (long long)kHidden * p.tp.NP * C);
      }
      for (int l = 0; l <= L; ++l) {
        const long long outl = (l == 0) ? (long long)(L + 1 + m0) * C : C;
        add_packed_weight(pre + "down.l" + std::to_string(l), pre + "downT.l" + std::to_string(l), 1, (long long)p.tp.k[l] * C, outl, false,
                          fp16_down(true), fp16_down(false));
        add_linear_weight(pre + "nl.l" + std::to_string(l), (long long)C * C);
        add_linear_weight(pre + "nlT.l" + std::to_string(l), (long long)C * C);
      }
      add_weight(pre + "down.b", (long long)(L + 1 + m0) * C);
      add_weight(pre + "nl.b", C);
      for (size_t i = 0; i < p.out_ls.size(); ++i) {
        const int l = p.out_ls[i];
        const std::string ls = std::to_string(l);
        add_packed_weight(pre + "c0.l" + ls, pre + "c0T.l" + ls, n_el, C, C, true, fp16_species(true), fp16_species(false));
        if (cfg.correlation >= 2)
          add_packed_weight(pre + "c1.l" + ls, pre + "c1T.l" + ls, n_el, (long long)p.pb.k[i] * C, C, true, fp16_species(true), fp16_species(false));
        if (cfg.correlation >= 3) {
          add_linear_weight(pre + "c2.l" + ls, (long long)n_el * p.pb3.k[i] * C * C);
          add_linear_weight(pre + "c2T.l" + ls, (long long)n_el * p.pb3.k[i] * C * C);
        }
        add_linear_weight(pre + "lin.l" + ls, (long long)C * C);
        add_linear_weight(pre + "linT.l" + ls, (long long)C * C);
        if (p.has_res && !res_identity) {
          add_packed_weight(pre + "res.l" + ls, pre + "resT.l" + ls, n_el, C, C, true, fp16_species(true), fp16_species(false));
        }
      }
      if (bilinear) {  // linear_up of the product: every rank to both factors, the scalars also to the gates
        for (int l = 0; l <= L; ++l) {
          add_linear_weight(pre + "pu.l" + std::to_string(l), (long long)C * 2 * C);
          add_linear_weight(pre + "puT.l" + std::to_string(l), (long long)C * 2 * C);
        }
        add_linear_weight(pre + "pg", (long long)C * p.pb.NP * C);
        add_linear_weight(pre + "pgT", (long long)C * p.pb.NP * C);
        add_weight(pre + "pu.b", 2 * C);
        add_weight(pre + "pg.b", (long long)p.pb.NP * C);
      }
      add_weight(pre + "c.b", (long long)n_el * C);
      add_weight(pre + "lin.b", C);
      if (p.has_res && !res_identity) add_weight(pre + "res.b", (long long)n_el * C);
    }
    add_weight("ro.W1", (long long)n_fid * C * H);
    add_weight("ro.W2", (long long)n_fid * H);
    if (c.use_alllayer)
      for (int t = 0; t + 1 < NL_; ++t) add_weight("ro.lin" + std::to_string(t), (long long)n_fid * C);
    add_weight("scale", (long long)n_fid * n_el);
    add_weight("e0", (long long)n_fid * n_el);
    if (zbl) { add_weight("zbl.z", n_el); add_weight("zbl.rcov", n_el); add_weight("zbl.par", 2); }
    n_listed = n_unset = (int)weights.size();
    for (const auto& e : pack_shapes) add_weight(e.first + "_pk", (long long)e.second.groups * e.second.N * (e.second.K + 1));
    if (folded) add_weight("emb_up", (long long)n_el * C);
    for (int t = 0; t < NL_ && folded; ++t)
      for (int l : layers[t].out_ls) {
        for (int j = 0; j < c.correlation; ++j) add_weight(coef_name(t, j, "f", l), (long long)n_el * coef_rows(t, j, l) * C);
        if (l == 0) add_weight("t" + std::to_string(t) + ".cf.b", (long long)n_el * C);
      }
    if (cudaGetDevice(&device) != cudaSuccess) return TACE_ERR_CUDA;
    if (cudaMalloc(&arena, sizeof(T) * (size_t)arena_numel) != cudaSuccess) return TACE_ERR_CUDA;
    if (cudaMemset(arena, 0, sizeof(T) * (size_t)arena_numel) != cudaSuccess) return TACE_ERR_CUDA;
    if (cudaMalloc(&dev_error, sizeof(int)) != cudaSuccess || cudaMemset(dev_error, 0, sizeof(int)) != cudaSuccess)
      return TACE_ERR_CUDA;
    return TACE_OK;
  }

  bool main_line_first() const override { return rt_K == 0 && !tece_mask; }
  int weight_count() const override { return n_listed; }
  int weight_info(int i, const char** name, int64_t* numel) const override {
    if (i < 0 || i >= n_listed) return TACE_ERR_INVALID_ARGUMENT;
    if (name) *name = weights[i].name.c_str();
    if (numel) *numel = weights[i].numel;
    return TACE_OK;
  }
  // ---- folded weights ----------------------------------------------------------------------
  // Two linears that follow each other without anything in between are one: the final linear of the product goes into the
  // per-species coefficients before it (every order and rank: c0, c1, c2, and their bias, to which the skip connection's is added),
  // the first linear_up into the species embedding.  The products are taken here, once, when the weights are set, with sums in
  // double precision.  Per layer and pass one linear less, and the skip connection joins the sum of the coefficients: two launches
  // of 3 to 20 us each way and a pass over the rows per linear: 1 372 atoms 588 -> 570 us, 64 crystals 2 681 -> 2 639, 256 atoms in
  // double precision 749 -> 730.  Models with the edge block keep their linears apart: their energies feel the rounding of a linear
  // most (2.2e-5 between the two forms, where the others move by 3e-6).
  //   cJ.lL [n_el][K][C] stays as it was set; cJf.lL is the folded matrix, cJT.lL its transpose, cJ.lL_hi/_lo and cJT.lL_hi/_lo the
  //   K-tile-major TF32 parts of both, from which the packed ones are taken (what the caller sets under these names is the same before folding, and is not kept).
  static std::string coef_name(int t, int order, const char* form, int l) {
    return "t" + std::to_string(t) + ".c" + std::to_string(order) + form + ".l" + std::to_string(l);
  }
  long long coef_rows(int t, int order, int l) const {  // out_ls holds 0..lmax, so l is also the index
    const LayerPlan& p = layers[t];
    return (long long)C * (order == 0 ? 1 : order == 1 ? p.pb.k[l] : p.pb3.k[l]);
  }
  T* w_mut(const std::string& name) {
    const auto it = weight_index.find(name);
    return it == weight_index.end() ? nullptr : arena + weights[it->second].offset;
  }
  cudaError_t fold_coefs(int t, int order, int l) {
    const std::string lin = "t" + std::to_string(t) + ".lin.l" + std::to_string(l), c = coef_name(t, order, "", l), cT = coef_name(t, order, "T", l);
    const cudaError_t e = launch_fold_linear(w(c), w(lin), w_mut(coef_name(t, order, "f", l)), w_mut(cT), w_mut(c + "_hi"), w_mut(c + "_lo"), w_mut(cT + "_hi"),
                              w_mut(cT + "_lo"), n_el, (int)coef_rows(t, order, l), C, cudaStream_t(0));
    if (e != cudaSuccess) return e;
    const cudaError_t p = pack_weight(c);
    return p != cudaSuccess ? p : pack_weight(cT);
  }
  cudaError_t fold_bias(int t) {
    const std::string pre = "t" + std::to_string(t) + ".";
    return launch_fold_rows(w(pre + "c.b"), w(pre + "lin.l0"), w(pre + "lin.b"), w(pre + "res.b"), w_mut(pre + "cf.b"), n_el, C, cudaStream_t(0));
  }
  cudaError_t fold_embedding() {
    return launch_fold_rows(w("emb"), w("t0.up.l0"), w("t0.up.b"), (const T*)nullptr, w_mut("emb_up"), n_el, C, cudaStream_t(0));
  }
  // Order and form of a coefficient name "tN.cJ...": J and true where its content is derived, -1 for every other name.
  static int coef_order(const std::string& name, bool& derived) {
    const size_t dot = name.find('.');
    if (name[0] != 't' || dot == std::string::npos || name.size() < dot + 5 || name[dot + 1] != 'c' || name[dot + 2] < '0' || name[dot + 2] > '2') return -1;
    derived = name[dot + 3] == 'T' || name.back() < '0' || name.back() > '9';
    return name[dot + 2] - '0';
  }
  // Takes the folded weights again that depend on `name`; all of them when the last weight has arrived.
  // The packed form of what was set; of everything when the last weight has arrived.
  cudaError_t derive_after(const std::string& name, bool all) {
    const size_t dot = name.find('.');
    const int layer = name[0] == 't' && dot != std::string::npos ? atoi(name.c_str() + 1) : -1;
    const std::string stem = layer >= 0 ? name.substr(dot + 1) : "";
    bool derived = false, any = false;
    const int order = coef_order(name, derived);
    int current = 0;  // the weights may be set with another device current than the one that holds them
    cudaError_t e = cudaGetDevice(&current);
    if (e == cudaSuccess && current != device) e = cudaSetDevice(device);
    if (e != cudaSuccess) return e;
    const bool part = name.size() > 3 && (name.compare(name.size() - 3, 3, "_hi") == 0 || name.compare(name.size() - 3, 3, "_lo") == 0);
    for (int i = 0; i < n_listed && e == cudaSuccess && all && kTensorCore; ++i) {
      const std::string& nm = weights[i].name;
      bool of_coefs = false;
      if (nm.size() > 3 && nm.compare(nm.size() - 3, 3, "_hi") == 0 && !(folded && coef_order(nm, of_coefs) >= 0)) { e = pack_weight(nm.substr(0, nm.size() - 3)); any = true; }
    }
    if (!all && part && kTensorCore) { e = pack_weight(name.substr(0, name.size() - 3)); any = true; }
    if (e == cudaSuccess && folded && (all || name == "emb" || name == "t0.up.l0" || name == "t0.up.b")) { e = fold_embedding(); any = true; }
    for (int t = 0; t < NL_ && e == cudaSuccess && folded; ++t) {
      if (!all && t != layer) continue;
      for (int l : layers[t].out_ls) {
        const std::string ls = ".l" + std::to_string(l);
        for (int j = 0; j < cfg.correlation && e == cudaSuccess; ++j)
          if (all || stem == "lin" + ls || (order == j && stem == "c" + std::to_string(j) + ls)) { e = fold_coefs(t, j, l); any = true; }
      }
      if (e == cudaSuccess && (all || stem == "lin.l0" || stem == "lin.b" || stem == "c.b" || stem == "res.b")) { e = fold_bias(t); any = true; }
    }
    if (e == cudaSuccess && any) e = cudaStreamSynchronize(cudaStream_t(0));  // a later pass may run on any stream
    const cudaError_t back = current != device ? cudaSetDevice(current) : cudaSuccess;
    return e != cudaSuccess ? e : back;
  }

  int set_weight(const char* name, const void* host, int64_t numel) override {
    if (!name || !host) return TACE_ERR_INVALID_ARGUMENT;
    for (int i = 0; i < n_listed; ++i) {
      WeightEntry& e = weights[i];
      if (e.name == name) {
        if (numel != e.numel) return TACE_ERR_INVALID_ARGUMENT;
        std::vector<T> cubic;
        if (e.name.size() > 5 && e.name.compare(e.name.size() - 5, 5, ".rtab") == 0) {
          // the table arrives as (value, h slope) at both ends of every interval; the kernels evaluate the same cubic in its
          // power basis (three multiply-adds for the weight, two more for its derivative, instead of four and four)
          const T* in = static_cast<const T*>(host);
          cubic.resize((size_t)numel);
          for (int64_t k = 0; k + 3 < numel; k += 4) {
            const double v0 = in[k], m0 = in[k + 1], v1 = in[k + 2], m1 = in[k + 3];
            cubic[k] = in[k]; cubic[k + 1] = in[k + 1];
            cubic[k + 2] = T(3.0 * (v1 - v0) - 2.0 * m0 - m1);
            cubic[k + 3] = T(2.0 * (v0 - v1) + m0 + m1);
          }
          if constexpr (std::is_same<T, float>::value) {
            if (tp_wide_channels(C)) {
              std::vector<float> pairs(cubic.size());
              tp_wide_table(cubic.data(), pairs.data(), numel / (4 * C), C);
              cubic.swap(pairs);
            }
          }
          host = cubic.data();
        }
        bool derived = false;
        if (!folded || coef_order(e.name, derived) < 0) derived = false;
        if (!derived && cudaMemcpy(arena + e.offset, host, sizeof(T) * (size_t)numel, cudaMemcpyHostToDevice) != cudaSuccess)
          return TACE_ERR_CUDA;
        if (e.name == "bessel") memcpy(host_bessel, host, sizeof(T) * kNumBessel);
        if (e.name == "bessel_pref") memcpy(host_bessel + kNumBessel, host, sizeof(T));
        const bool last = !e.set && n_unset == 1;
        if (!e.set) --n_unset;
        e.set = true;
        if (n_unset == 0 && (last || !derived) && derive_after(e.name, last) != cudaSuccess) return TACE_ERR_CUDA;
        return TACE_OK;
      }
    }
    return TACE_ERR_UNKNOWN_WEIGHT;
  }

  // ---- workspace ---------------------------------------------------------------------------
  static constexpr long long kChunkSlack = 8192;  // a chunk ends at an atom boundary: room for one atom's edges beyond the target
  struct LayerBufs {
    T *h_in, *x, *xx, *gxx, *W, *H3, *Z1, *Z2, *Z3, *Hact, *M, *Gt, *gGt, *a, *B2, *out, *h_out;
    T *gh_out, *ga, *gx, *gh_in;
    T *As, *gAs, *gout_s, *hs;  // species-sorted copies used by the per-species linears
    // largest elements per rank; nullptr: not taken
    unsigned *top, *gtop;       // of those rows, forward [NL][3][L + 1] (As, B2, hs) and backward [NL][L + 1] (gout_s)
    unsigned *mtop, *dtop;      // of the rows that linear_down reads, forward (M) and backward (gGt), [NL][L + 1]
    T *B3, *gB2;                // third-order basis (reused for its gradient) and the gradient of the second-order one
    T *inv_density, *gdens;     // learned edge density: 1 / density_i and dE / d density_i
    T *XY, *gXY, *Zg, *gZg;     // gated bilinear product: both factors per (atom, component), gate pre-activations, gradients
    // TECE edge block (layouts at the top of tece_kernels.cu); gradients that may overwrite their forward buffer do
    T *tKs, *tQt, *tMw, *tKp, *tQp, *tlogit, *talpha, *tup, *tglu, *tcoef, *tU, *tdown;
    T *tgdown, *tgalpha, *tglogit, *tgcut, *tgproj, *tproj, *tgQp, *tgKp, *tgKs, *tgQt, *tddlen;
    unsigned* ttop;  // largest elements per edge (TeceTop), fp32 models
  };
  struct Bufs {
    int *row_ids, *row_split;  // owned targets without / with a ghost source (passes split around the exchange)
    int *e_src, *e_dst, *e_orig, *perm_src, *rowptr_dst, *rowptr_src, *atom_graph, *species, *species_perm, *species_rank, *species_ptr, *tile_ptr, *tc_tile_ptr;
    int *chunk_atom_ptr, *chunk_edge_ptr, *keys_cs, *perm_cs;  // edge chunks; (chunk, source)-sorted edge list
    int n_chunks; long long chunk_rows;                        // rows held by the per-edge chunk buffers
    void* prep_temp; size_t prep_temp_bytes;
    T *energy_partial;  // slice sums of the per-graph energies (graph_energy_slices)
    T *vec, *Y, *dY, *g, *e_scaled, *atom_virial, *dxe, *dlen, *ddlen, *ro_factor, *env, *denv, *zbl_node;
    T *tWg, *tgWg, *tgvec;  // TECE: Wigner rows of every edge (shared by the layers), their gradient (a share per 32 channels), dE/d(edge vector) through them
    std::vector<LayerBufs> lay;
  };

  size_t layout(Arena& ar, Bufs& b, long long N, long long NL, long long E, int B) {
    b.e_src = ar.take<int>(E); b.e_dst = ar.take<int>(E); b.e_orig = ar.take<int>(E); b.perm_src = ar.take<int>(E);
    b.rowptr_dst = ar.take<int>(N + 1); b.rowptr_src = ar.take<int>(N + 1); b.atom_graph = ar.take<int>(N);
    b.species = ar.take<int>(N); b.row_ids = ar.take<int>(NL); b.row_split = ar.take<int>(2);
    b.species_perm = ar.take<int>(NL); b.species_rank = ar.take<int>(NL); b.species_ptr = ar.take<int>(n_el + 1); b.tile_ptr = ar.take<int>(4 * (n_el + 1));
    b.tc_tile_ptr = ar.take<int>(4 * (n_el + 1));
    b.prep_temp_bytes = graph_prep_temp_bytes(E, (int)N);
    b.prep_temp = ar.take<unsigned char>(b.prep_temp_bytes);
    b.vec = ar.take<T>(3 * E); b.Y = ar.take<T>((size_t)D * E); b.dY = ar.take<T>((size_t)D * E); b.g = ar.take<T>(3 * E);
    b.energy_partial = ar.take<T>((size_t)B * graph_energy_slices(NL, B));
    b.e_scaled = ar.take<T>(NL); b.atom_virial = ar.take<T>(9 * NL); b.ro_factor = ar.take<T>(NL); b.zbl_node = zbl ? ar.take<T>(NL) : nullptr;
    b.tWg = b.tgWg = b.tgvec = nullptr;
    if (tece_mask) { b.tWg = ar.take<T>((size_t)E * t_wg); b.tgWg = ar.take<T>((size_t)E * t_wg * (C / 32)); b.tgvec = ar.take<T>(3 * (size_t)E); }
    b.dlen = ar.take<T>(E); b.ddlen = ar.take<T>(E);
    b.env = env_after ? ar.take<T>(E) : nullptr; b.denv = env_after ? ar.take<T>(E) : nullptr;
    const bool chunked = E > max_chunk_edges;
    b.n_chunks = chunked ? (int)((E + max_chunk_edges - 1) / max_chunk_edges) : 1;
    b.chunk_rows = chunked ? max_chunk_edges + kChunkSlack : E;
    const long long Ec = b.chunk_rows;
    b.chunk_atom_ptr = ar.take<int>(b.n_chunks + 1); b.chunk_edge_ptr = ar.take<int>(b.n_chunks + 1);
    b.keys_cs = chunked ? ar.take<int>(E) : nullptr; b.perm_cs = chunked ? ar.take<int>(E) : nullptr;
    b.dxe = NL_ > 1 ? ar.take<T>((size_t)Ec * D * C) : nullptr;  // per-edge gradient rows of the source features
    T* shared_edge[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
    T* shared_W = nullptr;
    if (chunked && !rt_K) {  // one set of chunk-sized per-edge buffers serves every layer
      for (int k = 0; k < 5; ++k) shared_edge[k] = ar.take<T>((size_t)Ec * kHidden);
      int np_max = 0;
      for (const auto& p : layers) np_max = p.tp.NP > np_max ? p.tp.NP : np_max;
      shared_W = ar.take<T>((size_t)Ec * np_max * C);
    }
    b.lay.resize(NL_);
    T* prev_h = folded ? nullptr : ar.take<T>((size_t)N * C);  // the species embedding, where it is not folded into linear_up
    T* prev_gh = nullptr;
    for (int t = 0; t < NL_; ++t) {
      const LayerPlan& p = layers[t];
      LayerBufs& lb = b.lay[t];
      lb.h_in = prev_h;
      lb.gh_in = prev_gh;
      lb.x = ar.take<T>((size_t)N * p.tp.NX * C);
      lb.gx = p.scalar_src ? nullptr : ar.take<T>((size_t)N * p.tp.NX * C);
      const bool ghosts = (N != NL) && !p.scalar_src;  // exchanged copies of x and of its gradient
      lb.xx = ghosts ? ar.take<T>((size_t)N * p.tp.NX * C) : nullptr;
      lb.gxx = ghosts ? ar.take<T>((size_t)N * p.tp.NX * C) : nullptr;
      if (rt_K) {  // tabulated radial weights: no per-edge activation or weight exists
        lb.H3 = lb.Z1 = lb.Z2 = lb.Z3 = lb.Hact = lb.W = nullptr;
      } else {
        lb.H3 = chunked ? shared_edge[0] : ar.take<T>((size_t)E * kHidden);
        lb.Z1 = chunked ? shared_edge[1] : ar.take<T>((size_t)E * kHidden);
        lb.Z2 = chunked ? shared_edge[2] : ar.take<T>((size_t)E * kHidden);
        lb.Z3 = chunked ? shared_edge[3] : ar.take<T>((size_t)E * kHidden);
        lb.Hact = chunked ? shared_edge[4] : ar.take<T>((size_t)E * kHidden);
        lb.W = chunked ? shared_W : ar.take<T>((size_t)E * p.tp.NP * C);
      }
      lb.M = ar.take<T>((size_t)NL * p.tp.NM * C);
      lb.Gt = ar.take<T>((size_t)NL * (L + 1 + D) * C);
      lb.gGt = ar.take<T>((size_t)NL * (L + 1 + D) * C);
      lb.inv_density = density ? ar.take<T>(NL) : nullptr; lb.gdens = density ? ar.take<T>(NL) : nullptr;
      lb.XY = lb.gXY = lb.Zg = lb.gZg = nullptr;
      if (p.tece) {
        const size_t Es = (size_t)E;
        lb.tKs = ar.take<T>(Es * t_NR * C); lb.tQt = ar.take<T>(Es * t_NR * C); lb.tMw = ar.take<T>(Es * t_NR * 2 * C);
        lb.tKp = ar.take<T>(Es * t_NR * C); lb.tQp = ar.take<T>(Es * t_NR * C);
        lb.tlogit = ar.take<T>(Es * heads); lb.talpha = ar.take<T>(Es * heads);
        lb.tup = ar.take<T>(Es * (t_G + t_NF) * Ca); lb.tglu = ar.take<T>(Es * t_NF * Ca); lb.tcoef = ar.take<T>(Es * t_WN);
        lb.tU = ar.take<T>(Es * t_NF * Ca); lb.tdown = ar.take<T>(Es * t_NR * C);
        lb.tgdown = ar.take<T>(Es * t_NR * C); lb.tgalpha = ar.take<T>(Es * heads); lb.tglogit = ar.take<T>(Es * heads);
        lb.tgcut = ar.take<T>(Es * heads); lb.tgproj = ar.take<T>(Es * 2 * heads); lb.tproj = ar.take<T>(Es * 2 * heads);
        lb.ttop = kTensorCore ? ar.take<unsigned>(Es * kTeceTops) : nullptr;
        lb.tgQp = ar.take<T>(Es * t_NR * C); lb.tgKp = ar.take<T>(Es * t_NR * C);
        lb.tgKs = ar.take<T>(Es * t_NR * C); lb.tgQt = ar.take<T>(Es * t_NR * C);
        lb.tddlen = ar.take<T>(Es);
      }
      if (bilinear) {
        lb.XY = ar.take<T>((size_t)NL * D * 2 * C); lb.gXY = ar.take<T>((size_t)NL * D * 2 * C);
        lb.Zg = ar.take<T>((size_t)NL * p.pb.NP * C); lb.gZg = ar.take<T>((size_t)NL * p.pb.NP * C);
      }
      lb.a = ar.take<T>((size_t)NL * D * C);
      lb.ga = ar.take<T>((size_t)NL * D * C);
      lb.B2 = ar.take<T>((size_t)NL * p.pb.NB * C);
      lb.B3 = cfg.correlation >= 3 ? ar.take<T>((size_t)NL * p.pb3.NB * C) : nullptr;
      lb.gB2 = cfg.correlation >= 3 ? ar.take<T>((size_t)NL * p.pb.NB * C) : nullptr;
      lb.As = ar.take<T>((size_t)NL * D * C);
      lb.gAs = ar.take<T>((size_t)NL * D * C);
      lb.gout_s = ar.take<T>((size_t)NL * p.Dout * C);
      lb.top = fp16_species(false) ? ar.take<unsigned>((size_t)NL * 3 * (L + 1)) : nullptr;
      lb.gtop = fp16_species(true) ? ar.take<unsigned>((size_t)NL * (L + 1)) : nullptr;
      lb.mtop = fp16_down(false) ? ar.take<unsigned>((size_t)NL * (L + 1)) : nullptr;
      lb.dtop = fp16_down(true) ? ar.take<unsigned>((size_t)NL * (L + 1)) : nullptr;
      lb.hs = p.has_res ? ar.take<T>((size_t)NL * p.Din * C) : nullptr;
      lb.out = folded ? nullptr : ar.take<T>((size_t)NL * p.Dout * C);
      lb.h_out = ar.take<T>((size_t)N * p.Dout * C);
      lb.gh_out = ar.take<T>((size_t)N * p.Dout * C);
      prev_h = lb.h_out;
      prev_gh = lb.gh_out;
    }
    return ar.used;
  }

  int workspace_bytes(int64_t n_atoms, int64_t n_local, int64_t n_edges, int32_t n_graphs, size_t* bytes) override {
    if (!bytes || n_atoms < 0 || n_local < 0 || n_local > n_atoms || n_edges < 0 || n_graphs < 0) return TACE_ERR_INVALID_ARGUMENT;
    if (n_edges >= (1LL << 31) - 64 || n_atoms >= (1LL << 31) - 64) return TACE_ERR_CAPACITY;
    Arena ar; Bufs b;
    *bytes = layout(ar, b, n_atoms, n_local, this->edge_capacity(n_edges), n_graphs) + 512 +
             this->stage_layout(n_atoms, n_local, this->edge_capacity(n_edges), n_graphs).total;
    return TACE_OK;
  }

  // ---- GEMM helpers ----------------------------------------------------------------------------
  static void add_problem(GemmBatch<T>& gb, const T* A, long long a_s1, long long a_s2, int q, int K, const T* Bm, int N,
                          T* Cm, long long c_s1, long long c_s2, const T* bias, int accumulate, int join = 0, long long b_gs = 0,
                          long long bias_gs = 0, const int* tile_ptr = nullptr) {
    GemmProblem<T>& p = gb.p[gb.n_problems++];
    p.A = A; p.B = Bm; p.C = Cm; p.bias = bias; p.q = q; p.N = N; p.K = K;
    p.a_s1 = a_s1; p.a_s2 = a_s2; p.c_s1 = c_s1; p.c_s2 = c_s2;
    p.b_group_stride = b_gs; p.bias_group_stride = bias_gs; p.accumulate = accumulate; p.join = join; p.tile_ptr = tile_ptr;
  }
  static GemmBatch<T> plain_batch(long long n_atoms) {
    GemmBatch<T> gb;
    memset(&gb, 0, sizeof(gb));
    gb.n_groups = 1; gb.n_atoms = (int)n_atoms;
    return gb;
  }
  const int* tiles(const Bufs& b, int l) const { return b.tile_ptr + l * (n_el + 1); }

  // One per-rank linear of a launch: rows (atom, m) of A times the [K][N] matrix `wname`;
  // `wname_t` names the same matrix transposed ([N][K]), which is what the tensor-core path reads.
  struct LinSpec {
    const T* A; long long a_s1, a_s2; int q, K;
    std::string wname, wname_t; int N;
    T* Cm; long long c_s1, c_s2; const T* bias;
    int accumulate = 0;          // Cm += instead of Cm =
    T* act_out = nullptr;        // fused activations of GemmProblem (double precision)
    const T* act_in = nullptr;
    const unsigned* a_top = nullptr; int a_top_stride = 0;  // those of TcLinearProblem
  };
  // the layers of the radial MLP of fp64 models apply their activations themselves (a LayerNorm in between needs whole rows)
  bool fused_activations() const { return !kTensorCore && !element2; }

  // accumulate = kJoin: the product is added to that of the spec before it (same rows and result), in one pass over both K ranges
  // where the tensor-core path takes them.
  static constexpr int kJoin = 2;
  // The specs of one call, a run of joined ones at a time: tcgen05 for fp32 models where every shape of the run fits and there is
  // enough work, the kernels of gemm.cuh for the rest.
  //
  // kSmallLinear: multiply-adds of a call up to which the CUDA cores are done before a launch of the tensor-core kernel has set up its
  // tensor memory, barriers and tiles: one evaluation of 32 atoms at rank 2, 64 channels 216 -> 173 us, at rank 3, 128 channels
  // 356 -> 279; 108 atoms 226 -> 187 and 420 -> 380; a limit of 64 Mi loses at 256 and 1 372 atoms (232 against 227 us, 446 against
  // 437), one of 16 Mi at 128 channels (518 against 503 at 256 atoms).  Models with the edge block keep one path for the linears of the forward
  // pass: their energies feel the rounding of the linears most (3e-5 between the two paths), and that is not to show between systems
  // of different size.
  // Four times as many where the tensor cores have at most kFewTiles tiles, each walking a long K loop on one SM (128 rows,
  // K = 4 352: 73 -> 43 us).  A per-species launch has tiles for every element present, which the host does not know, and that keeps
  // the tensor cores ahead from some number of elements on: evaluations of 24 and 48 atoms at rank 3, 128 channels, with the limit as it
  // is -> fourfold, 8 elements in the model 301 -> 292 us and 323 -> 316, 16 elements 305 -> 300 and even, 32 elements 318 -> 321 and
  // 345 -> 350, 89 elements 340 -> 346 and 389 -> 385 (40 atoms 373 -> 377).  So it ends at kFewElements.
  static constexpr long long kSmallLinear = 32LL << 20, kFewTiles = 8, kFewElements = 16;
  bool backward_pass = false;  // what forward() is enqueuing
  template <typename Spec>
  static bool small_call(const std::vector<Spec>& specs, long long counted, int n_groups) {
    long long work = 0, tiles = 0;  // tiles: of the tensor-core kernel, all elements taken together
    for (const Spec& sp : specs) {
      work += counted * sp.q * sp.K * sp.N;
      if (sp.accumulate != kJoin) tiles += (counted * sp.q + 127) / 128 * ((sp.N + 127) / 128);
    }
    const bool few = tiles <= kFewTiles && n_groups <= kFewElements;
    return work <= (few ? 4 : 1) * kSmallLinear;
  }
  // counted: rows for which the kernels are chosen.
  template <typename Spec, typename FillTc, typename Add>
  cudaError_t run_specs(const std::vector<Spec>& specs, long long n_atoms, long long counted, cudaStream_t s, const GemmBatch<T>& empty, FillTc&& fill,
                        Add&& add) {
    TcLinearProblem probs[kMaxLinears];
    int n_tc = 0;
    GemmBatch<T> gb = empty;
    cudaError_t err = cudaSuccess;
    const bool small = small_call(specs, counted, empty.n_groups);
    for (size_t i = 0, j; i < specs.size() && err == cudaSuccess; i = j) {
      bool tc = kTensorCore && ((tece_mask && !backward_pass) || !small);
      for (j = i; j < specs.size() && (j == i || specs[j].accumulate == kJoin); ++j) tc = tc && tc_linear_supported(specs[j].N, specs[j].K);
      if (!tc) {
        if (gb.n_problems + (int)(j - i) > kMaxProblems) { err = launch_gemm(gb, n_atoms, s); gb = empty; }
        for (size_t k = i; k < j; ++k) add(gb, specs[k], specs[k].accumulate == 1, specs[k].accumulate == kJoin);
        continue;
      }
      if (n_tc + (int)(j - i) > kMaxLinears) { err = launch_tc_linear(probs, n_tc, dev_error, s); n_tc = 0; }
      for (size_t k = i; k < j; ++k) {
        const Spec& sp = specs[k];
        TcLinearProblem& h = probs[n_tc++];
        memset(&h, 0, sizeof(h));
        h.A = reinterpret_cast<const float*>(sp.A); h.a_atom_stride = sp.a_s1; h.a_comp_stride = sp.a_s2; h.q = sp.q;
        h.n_atoms = n_atoms; h.K = sp.K; h.N = sp.N;
        h.Bhi = reinterpret_cast<const float*>(w(sp.wname_t + "_hi")); h.Blo = reinterpret_cast<const float*>(w(sp.wname_t + "_lo"));
        h.C = reinterpret_cast<float*>(sp.Cm); h.c_s1 = sp.c_s1; h.c_s2 = sp.c_s2; h.bias = reinterpret_cast<const float*>(sp.bias);
        h.accumulate = sp.accumulate == 1; h.join = sp.accumulate == kJoin;
        fill(h, sp);
      }
    }
    if (err == cudaSuccess && n_tc > 0) err = launch_tc_linear(probs, n_tc, dev_error, s);
    if (err == cudaSuccess && gb.n_problems > 0) err = launch_gemm(gb, n_atoms, s);
    return err;
  }
  // Plain (not per-species) linears.  c_map: row a of the results belongs to atom c_map[a] (nullptr: the same order).
  cudaError_t run_linear(const std::vector<LinSpec>& specs, long long n_atoms, cudaStream_t s, const int* c_map = nullptr) {
    return run_linear(specs, n_atoms, n_atoms, s, c_map);
  }
  // Linears whose rows are edges: a captured pass has the edges of its capacity where a direct one has those of the list, and both are to
  // take the same kernels.
  cudaError_t run_edge_linear(const std::vector<LinSpec>& specs, long long n_edges, cudaStream_t s) {
    return run_linear(specs, n_edges, round_edges(n_edges), s, nullptr);
  }
  cudaError_t run_linear(const std::vector<LinSpec>& specs, long long n_atoms, long long counted, cudaStream_t s, const int* c_map) {
    GemmBatch<T> gb = plain_batch(n_atoms);
    gb.c_atom_map = c_map;
    return run_specs(specs, n_atoms, counted, s, gb, [&](TcLinearProblem& h, const LinSpec& sp) {
                       h.atom_map = c_map;
                       if (!sp.a_top) return;
                       const Packed pk = packed(sp.wname_t);
                       h.a_top = sp.a_top; h.a_top_stride = sp.a_top_stride; h.B = pk.B; h.b_inv = pk.inv;
                     },
                     [&](GemmBatch<T>& g, const LinSpec& sp, int accumulate, int join) {
                       add_problem(g, sp.A, sp.a_s1, sp.a_s2, sp.q, sp.K, w(sp.wname), sp.N, sp.Cm, sp.c_s1, sp.c_s2, sp.bias, accumulate, join);
                       g.p[g.n_problems - 1].act_out = sp.act_out; g.p[g.n_problems - 1].act_in = sp.act_in;
                     });
  }

  // Per-species linears (the reference's e3nnElementLinear, tace/models/linear.py:377-481).  A holds rows of the
  // species-sorted atoms, so species g owns the contiguous rows [species_ptr[g], species_ptr[g+1]) and uses the g-th
  // matrix of `wname` ([n_el][K][N]); `mapped` sends row a of the result to atom species_perm[a].
  struct SpeciesSpec {
    const T* A; long long a_s1, a_s2; int q, K;
    std::string wname, wname_t; int N;
    T* Cm; long long c_s1, c_s2; const T* bias; bool mapped; int accumulate;
    int rank = 0, operand = 0;  // of A: l, and 0..2 for As, B2, hs (species_tops)
    const unsigned* a_top = nullptr; int a_top_stride = 0;  // those of TcLinearProblem, in species-sorted order
  };
  // Whether FP16 parts pay for the tensor-core call (tc_fp16_pays): the largest elements are not looked for in vain.
  template <typename Spec>
  static bool long_loops(const std::vector<Spec>& specs) {
    long long steps = 0, results = 0;
    for (const Spec& sp : specs) {
      steps += (long long)sp.q * sp.N * (sp.K / 32);
      if (sp.accumulate != kJoin) results += (long long)sp.q * sp.N;
    }
    return tc_fp16_pays(results, steps);
  }
  // Which linears of the nodes take FP16 parts.  Those of models with the edge block do not: their energies move by 4e-5 with the rounding.  Nor do
  // those of the forward pass with few elements: that line is drawn to keep the results, not for time or exactness.  Energies of such models move by
  // more with the kernel (rank 3, 128 channels, alloy of 2 048 atoms: 3.6e-5 off double precision, 2.1e-5 with FP16 for both kinds of linears) than
  // from one build to the next.  On the other side of it FP16 would be a little faster and closer to double precision: 64 random crystals with
  // 2, 5, 8, 16 elements 2 340, 2 343, 2 349, 2 366 us as it is and 2 299, 2 302, 2 308, 2 319 with FP16, energies off by 8e-9, 2e-9, 1e-9, 1e-9 eV an atom
  // and 3e-9, 9e-10, 6e-10, 5e-10.  With 64 channels most K loops of the backward pass are too short; above 128 the kernels that note largest
  // elements do not apply (pb_tops).
  bool fp16_nodes(bool backward) const { return folded && (backward ? C >= 128 : n_el > kFewElements); }
  // What can reach the two kinds of them: the kernels that note the largest elements are those of the second-order product and of the tables of
  // radial weights.
  bool fp16_species(bool backward) const { return kTensorCore && fp16_nodes(backward) && !bilinear && cfg.correlation == 2 && pb_tops(C); }
  bool fp16_down(bool backward) const {
    return kTensorCore && fp16_nodes(backward) && rt_K && !density && pb_tops(C) && (backward || tp_wide_channels(C));
  }
  // linear_down of a layer (1/avg_num_neighbors folded into the weights) and the way back through it, where the gradient of the messages
  // overwrites the messages
  std::vector<LinSpec> down_specs(const LayerPlan& p, const LayerBufs& lb, const std::string& pre, bool backward) const {
    std::vector<LinSpec> sp;
    for (int l = 0; l <= L; ++l) {
      const int Nk = p.tp.k[l] * C, Ng = (l == 0) ? (L + 1 + m0) * C : C;
      const std::string ls = std::to_string(l);
      T* M = lb.M + (long long)p.tp.base[l] * C;
      T* g = (backward ? lb.gGt : lb.Gt) + (l == 0 ? 0 : (long long)(L + m0 + l * l) * C);
      if (!backward)
        sp.push_back({M, (long long)p.tp.NM * C, Nk, 2 * l + 1, Nk, pre + "down.l" + ls, pre + "downT.l" + ls, Ng, g, (long long)(L + 1 + D) * C, C,
                      l == 0 ? w(pre + "down.b") : nullptr});
      else
        sp.push_back({g, (long long)(L + 1 + D) * C, C, 2 * l + 1, Ng, pre + "downT.l" + ls, pre + "down.l" + ls, Nk, M, (long long)p.tp.NM * C, Nk, nullptr});
    }
    return sp;
  }
  // Their rows' largest elements where these linears take FP16 parts, rank by rank (figures: species_tops).
  unsigned* down_tops(std::vector<LinSpec>& sp, unsigned* top, long long n_atoms, bool backward) const {
    if (!top || !fp16_down(backward) || small_call(sp, n_atoms, 1) || !long_loops(sp)) return nullptr;
    for (int l = 0; l <= L; ++l) { sp[l].a_top = top + l; sp[l].a_top_stride = L + 1; }
    return top;
  }
  // Largest elements of the atoms' rows for the per-species linears, by operand and rank (`top`, or nullptr where they are not wanted): those read
  // their weights from DRAM, and FP16 parts are half the bytes of TF32 parts.  These linears and linear_down together, random crystals of 89 elements at
  // rank 3, 128 channels (395 MB of weights as TF32 parts): 64 of them 2 641 -> 2 500 us, 16 1 121 -> 1 032, energies of 33 772 -> 722; backward only, two
  // elements: 1 536 atoms 2 447 -> 2 407, 32 400 45.1 -> 44.6 ms.
  unsigned* species_tops(std::vector<SpeciesSpec>& sp, unsigned* top, long long n_atoms, bool backward) const {
    if (!top || !fp16_species(backward) || small_call(sp, n_atoms, n_el) || !long_loops(sp)) return nullptr;
    set_tops(sp, top, backward ? 1 : 3);
    return top;
  }
  void set_tops(std::vector<SpeciesSpec>& sp, const unsigned* top, int operands) const {
    for (auto& q : sp) { q.a_top = top ? top + q.operand * (L + 1) + q.rank : nullptr; q.a_top_stride = operands * (L + 1); }
  }
  // Rows of D ranks
  cudaError_t gather_rows(const T* src, const int* perm, T* dst, long long n, int rows, unsigned* top, int top_stride, cudaStream_t s) const {
    if constexpr (kTensorCore) {
      if (top) return launch_gather_rows_top(src, perm, dst, n, rows == 1 ? 0 : Ln, C, top, top_stride, s);
    }
    return launch_gather_rows(src, perm, dst, n, rows * C, s);
  }
  cudaError_t run_species_linear(const std::vector<SpeciesSpec>& specs, const Bufs& b, long long n_atoms, cudaStream_t s) {
    if (specs.empty()) return cudaSuccess;
    GemmBatch<T> gb;
    memset(&gb, 0, sizeof(gb));
    gb.n_groups = n_el; gb.group_ptr = b.species_ptr;
    gb.c_atom_map = specs[0].mapped ? b.species_perm : nullptr;
    for (const auto& sp : specs)
      if (sp.mapped != specs[0].mapped) return cudaErrorInvalidValue;
    return run_specs(specs, n_atoms, n_atoms, s, gb,
                     [&](TcLinearProblem& h, const SpeciesSpec& sp) {
                       h.n_groups = n_el; h.group_ptr = b.species_ptr; h.tile_ptr = b.tc_tile_ptr + (sp.q / 2) * (n_el + 1);
                       h.atom_map = gb.c_atom_map;
                       h.b_group_stride = (long long)sp.K * sp.N; h.bias_group_stride = sp.N;
                       h.b_tiled = 1;  // the packed per-species hi / lo parts are K-tile-major (read once per pass, straight from DRAM)
                       if (!sp.a_top) return;
                       const Packed pk = packed(sp.wname_t);
                       h.a_top = sp.a_top; h.a_top_stride = sp.a_top_stride; h.B = pk.B; h.b_inv = pk.inv;
                     },
                     [&](GemmBatch<T>& g, const SpeciesSpec& sp, int accumulate, int join) {
                       add_problem(g, sp.A, sp.a_s1, sp.a_s2, sp.q, sp.K, w(sp.wname), sp.N, sp.Cm, sp.c_s1, sp.c_s2, sp.bias, accumulate, join,
                                   (long long)sp.K * sp.N, sp.N, tiles(b, sp.q / 2));
                     });
  }

#define CK(expr)                                                                                 \
  do {                                                                                           \
    cudaError_t err__ = (expr);                                                                  \
    if (err__ != cudaSuccess) {                                                                  \
      fprintf(stderr, "tace_b200: CUDA error %s at %s:%d\n", cudaGetErrorString(err__), __FILE__, __LINE__); \
      return TACE_ERR_CUDA;                                                                      \
    }                                                                                            \
  } while (0)

#define CKL(expr) do { CK(expr); ++launches; } while (0)
#define CKS(expr) do { const int st__ = (expr); if (st__ != TACE_OK) return st__; } while (0)
#define PH(name) phase(name, s)

  // Arguments of the per-edge MLP kernels for layers `ts` over edges [e0, e0 + Ec); row r of every [.][64] buffer is edge e0 + r.
  EdgeArgs<T> edge_range(const EdgeArgs<T>& ea, const Bufs& b, const std::vector<int>& ts, long long e0, long long Ec) const {
    EdgeArgs<T> r = ea;
    r.E = Ec; r.n_layers = (int)ts.size(); r.dlen = ea.dlen + e0; r.ddlen = ea.ddlen + e0;
    r.e_src = ea.e_src + e0; r.e_dst = ea.e_dst + e0;
    if (ea.env) r.env = ea.env + e0;
    if (ea.denv) r.denv = ea.denv + e0;
    for (size_t i = 0; i < ts.size(); ++i) {
      r.mlp[i] = ea.mlp[ts[i]];
      r.Z1[i] = b.lay[ts[i]].Z1;
      // activation of the first hidden layer; the last one's has to end up in H3, and fused layers go back and forth between the two
      r.H1[i] = nh == 1 || (nh == 3 && fused_activations()) ? b.lay[ts[i]].H3 : b.lay[ts[i]].Hact;
      r.dH1[i] = dh1_buffer(b.lay[ts[i]]);
    }
    return r;
  }
  // ---- TECE edge block --------------------------------------------------------------------------------------
  // the six SO(2) linears of the block (oam_2026_07_05.py:612-676): channel counts and rows per order on both sides
  struct So2Shape { const char* name; int mm, c_in, c_out, n_in[3], n_out[3]; };
  So2Shape so2_shape(int i) const {
    const int n = L + 1;
    So2Shape s{};
    const int red[3] = {n, n - 1, n - 2}, full[3] = {n, n, n};
    auto set = [&](const char* nm, int mm, int ci, int co, const int* in, const int* out) {
      s.name = nm; s.mm = mm; s.c_in = ci; s.c_out = co;
      for (int m = 0; m < 3; ++m) { s.n_in[m] = in[m]; s.n_out[m] = out[m]; }
    };
    const int up_out[3] = {t_G + n, n, n}, coef_out[3] = {t_np * n * Ca, 0, 0};
    switch (i) {
      case 0: set("key", mmax, C, C, red, red); break;
      case 1: set("query", mmax, C, C, red, red); break;
      case 2: set("up", mmax, 2 * C, Ca, red, up_out); break;
      case 3: set("glu", mmax, 2 * C, Ca, red, full); break;
      case 4: set("coefs", 0, 2 * C, 1, red, coef_out); break;
      default: set("down", mmax, Ca, C, full, red); break;
    }
    return s;
  }
  // GEMM problems of SO(2) linears over the E edges: `in` [E][in_rows][c_in] -> `out` [E][out_rows][c_out] (forward), or the
  // gradient of the output back to the gradient of the input (backward; `out` is then the input gradient, and linears of the
  // call with the same input gradient add up)
  struct So2Run { int which; const T* in; int in_rows; T* out; int out_rows; int top = 0; };  // top: first of its largest elements of an edge
  // Where the largest elements of what the linears of the call read are, per edge and order
  struct Tops { const unsigned* first; int stride; };
  void so2_specs(std::vector<LinSpec>& sp, const std::string& pre, const std::vector<So2Run>& runs, bool backward, Tops tops) const {
    std::vector<int> off_in(runs.size(), 0), off_out(runs.size(), 0);
    for (int m = 0; m <= mmax; ++m) {
      for (size_t i = 0; i < runs.size(); ++i) {
        const So2Run& r = runs[i];
        const So2Shape sh = so2_shape(r.which);
        if (m > sh.mm) continue;
        const int K = sh.n_in[m] * sh.c_in, Nn = sh.n_out[m] * sh.c_out;
        const std::string nm = pre + "so2." + sh.name + ".m" + std::to_string(m), nmT = pre + "so2." + sh.name + "T.m" + std::to_string(m);
        if (!backward)
          sp.push_back({r.in + (long long)off_in[i] * sh.c_in, (long long)r.in_rows * sh.c_in, K, m ? 2 : 1, K, nm, nmT, Nn,
                        r.out + (long long)off_out[i] * sh.c_out, (long long)r.out_rows * sh.c_out, Nn, m == 0 ? w(pre + "so2." + sh.name + ".b") : nullptr, 0});
        else  // `in` holds the gradient of the forward output, `out` receives the gradient of the forward input
          sp.push_back({r.in + (long long)off_out[i] * sh.c_out, (long long)r.out_rows * sh.c_out, Nn, m ? 2 : 1, Nn, nmT, nm, K,
                        r.out + (long long)off_in[i] * sh.c_in, (long long)r.in_rows * sh.c_in, K, nullptr,
                        i > 0 && r.out == runs[i - 1].out ? kJoin : 0});
        if (tops.first) { sp.back().a_top = tops.first + r.top + m; sp.back().a_top_stride = tops.stride; }
        // the order-0 block of the input always spans L + 1 rows (oam_2026_07_05.py:211)
        off_in[i] += (m == 0) ? (L + 1) : 2 * sh.n_in[m];
        off_out[i] += (m == 0) ? sh.n_out[0] : 2 * sh.n_out[m];
      }
    }
  }
  TeceArgs<T> tece_args(const EdgeArgs<T>& ea, const Bufs& b, const LayerBufs& lb, const std::string& pre, const T* x_src, long long N,
                        long long NL, long long E) const {
    TeceArgs<T> a;
    memset(&a, 0, sizeof(a));
    a.E = E; a.n_atoms = (int)N; a.n_local = (int)NL; a.C = C; a.Ca = Ca; a.L = L; a.mmax = mmax; a.H = heads; a.NR = t_NR;
    a.gate_m0 = m0; a.act = edge_act;
    for (int r = 0; r < t_NR; ++r) a.row_scale[r] = T(t_row_scale[r]);
    for (int q = 0; q < t_np; ++q) a.p_scale[q] = T(t_p_scale[q]);
    a.rp = ea.rp; a.vec = b.vec; a.dlen = b.dlen; a.env = env_after ? b.env : nullptr;
    a.e_src = b.e_src; a.e_dst = b.e_dst; a.rowptr = b.rowptr_dst;
    a.x = x_src; a.W = lb.W; a.Wg = b.tWg; a.Ks = lb.tKs; a.Qt = lb.tQt; a.Mw = lb.tMw; a.Kp = lb.tKp; a.Qp = lb.tQp;
    a.logit = lb.tlogit; a.alpha = lb.talpha; a.temp = w(pre + "att.temp"); a.rproj_w = w(pre + "att.rw"); a.rproj_b = w(pre + "att.rb");
    a.up = lb.tup; a.glu = lb.tglu; a.coefZ = lb.tcoef; a.U = lb.tU; a.down = lb.tdown; a.M = lb.M;
    a.gM = lb.M; a.gdown = lb.tgdown; a.galpha = lb.tgalpha; a.glogit = lb.tglogit; a.gcut = lb.tgcut; a.gproj = lb.tgproj; a.proj = lb.tproj;
    a.gQp = lb.tgQp; a.gKp = lb.tgKp; a.gKs = lb.tgKs; a.gQt = lb.tgQt; a.gMw = lb.tMw;
    a.gU = lb.tU; a.gup = lb.tup; a.gglu = lb.tglu; a.gcoefZ = lb.tcoef; a.gWg = b.tgWg; a.gvec = b.tgvec;
    a.dxe = b.dxe; a.gx = lb.gx; a.ddlen_extra = lb.tddlen;
    a.top = lb.ttop;
    return a;
  }
  // forward of the block for one layer: lb.W holds the radial weights, the result lands in lb.M
  int tece_forward(const TeceArgs<T>& ta, const LayerBufs& lb, const std::string& pre, long long E, cudaStream_t s) {
    std::vector<LinSpec> sp;
    auto top = [&](TeceTop k) { return Tops{lb.ttop ? lb.ttop + k * E : nullptr, tece_top_width(k)}; };
    if (lb.ttop && E > 0) CK(cudaMemsetAsync(lb.ttop, 0, sizeof(unsigned) * (size_t)(kTeceTops * E), s));
    CKL(launch_tece(ta, TECE_ROTATE_IN, s));
    so2_specs(sp, pre, {{0, lb.tKs, t_NR, lb.tKp, t_NR}, {1, lb.tQt, t_NR, lb.tQp, t_NR, 3}}, false, top(TECE_TOP_IN));
    CKL(run_edge_linear(sp, E, s)); sp.clear();
    cudaStream_t side;  // the attention weights, beside the linears and the cluster expansion of the messages
    CKS(branch(s, &side));
    CKL(launch_tece(ta, TECE_LOGIT, side));
    CKL(launch_tece(ta, TECE_SOFTMAX, side));
    so2_specs(sp, pre, {{2, lb.tMw, t_NR, lb.tup, t_G + t_NF}, {3, lb.tMw, t_NR, lb.tglu, t_NF}, {4, lb.tMw, t_NR, lb.tcoef, t_WN}}, false, top(TECE_TOP_MW));
    CKL(run_edge_linear(sp, E, s)); sp.clear();
    CKL(launch_tece(ta, TECE_MIX, s));
    so2_specs(sp, pre, {{5, lb.tU, t_NF, lb.tdown, t_NR}}, false, top(TECE_TOP_MIX));
    CKL(run_edge_linear(sp, E, s)); sp.clear();
    CKS(merge(s));
    CKL(launch_tece(ta, TECE_ROTATE_OUT, s));
    return TACE_OK;
  }
  // backward: lb.M holds dE/d(messages); leaves dE/d(radial weights) in lb.W, the per-edge source rows in dxe, the target part
  // added to lb.gx by the caller's order (source sum first), and this layer's share of dE/d(edge vector) in tgvec / tddlen
  int tece_backward(TeceArgs<T> ta, const Bufs& b, const LayerBufs& lb, const std::string& pre, long long N, long long E, bool first_tece,
                    cudaStream_t s, cudaStream_t* after) {
    std::vector<LinSpec> sp;
    auto top = [&](TeceTop k) { return Tops{lb.ttop ? lb.ttop + k * E : nullptr, tece_top_width(k)}; };
    cudaStream_t side;
    CKL(launch_tece(ta, TECE_ROTATE_OUT_BWD, s));
    // the attention weights down to the rotated rows, beside the way back through the messages (cluster expansion and linears)
    CKS(branch(s, &side));
    CKL(launch_tece(ta, TECE_ALPHA_BWD, side));
    CKL(launch_tece(ta, TECE_SOFTMAX_BWD, side));
    CKL(launch_tece(ta, TECE_LOGIT_BWD, side));
    CKL(launch_tece(ta, TECE_EDGE_SCALAR_BWD, side));
    so2_specs(sp, pre, {{5, lb.tgdown, t_NF, lb.tU, t_NR}}, true, top(TECE_TOP_DOWN));   // gU over U
    CKL(run_edge_linear(sp, E, s)); sp.clear();
    CKL(launch_tece(ta, TECE_MIX_BWD, s));                           // gup / gglu / gcoef over their forward buffers
    // gMw over Mw: the three linears that read Mw add up in one pass per order
    so2_specs(sp, pre, {{2, lb.tup, t_NR, lb.tMw, t_G + t_NF}, {3, lb.tglu, t_NR, lb.tMw, t_NF, 3}, {4, lb.tcoef, t_NR, lb.tMw, t_WN, 6}}, true, top(TECE_TOP_GMIX));
    CKL(run_edge_linear(sp, E, s)); sp.clear();
    CKS(merge(s));
    so2_specs(sp, pre, {{0, lb.tgKp, t_NR, lb.tgKs, t_NR}, {1, lb.tgQp, t_NR, lb.tgQt, t_NR, 3}}, true, top(TECE_TOP_GPROJ));
    CKL(run_edge_linear(sp, E, s)); sp.clear();
    CKL(launch_tece(ta, TECE_ROTATE_IN_BWD, s));
    ta.accumulate_gvec = first_tece ? 0 : 1;
    CKS(branch(s, after));  // what only the end of the pass needs
    CKL(launch_tece(ta, TECE_WIGNER_BWD, *after));
    CKL(launch_segment_sum_rows(b.dxe, b.rowptr_src, b.perm_src, lb.gx, 0, (int)N, D * C, s, /*accumulate=*/1));
    return TACE_OK;
  }

  DensityArgs<T> density_args(const EdgeArgs<T>& ea, const Bufs& b, const LayerBufs& lb, const std::string& pre, long long NL,
                              long long E) const {
    DensityArgs<T> da;
    memset(&da, 0, sizeof(da));
    da.rowptr_dst = b.rowptr_dst; da.e_dst = b.e_dst; da.dlen = b.dlen; da.rp = ea.rp;
    da.A0 = w(pre + "dA0"); da.w1 = w(pre + "dw1"); da.ab = w(pre + "dab");
    if (mlp_bias) { da.b0 = w(pre + "db0"); da.b1 = w(pre + "db1"); }
    da.use_env = (env_after && density == 1) ? 1 : 0;
    da.n = (int)NL; da.E = E; da.inv_density = lb.inv_density;
    return da;
  }
  // where the backward pass leaves dE/d(first hidden activation): it ping-pongs through the activation buffers
  T* dh1_buffer(const LayerBufs& lb) const { return nh == 3 ? lb.Z3 : nh == 2 ? lb.Hact : lb.H3; }
  // radial MLP hidden layers 8 -> 64 -> 64 -> 64 (tace/models/mlp.py:136-191): the first layer per edge, the
  // two 64 x 64 layers as GEMMs over the edges (all layers of `ts` in one launch), SiLU in between
  int radial_forward(const EdgeArgs<T>& ea, const Bufs& b, const std::vector<int>& ts, long long e0, long long Ec, cudaStream_t s) {
    if (Ec <= 0 || rt_K) return TACE_OK;  // tabulated weights: the radial MLP never runs
    const EdgeArgs<T> er = edge_range(ea, b, ts, e0, Ec);
    CKL(launch_edge_mlp_in(er, s));
    const long long n64 = Ec * kHidden;
    const bool ln = element2;  // LayerNorm before every hidden activation
    const bool fused = fused_activations();
    for (int j = 0; j < nh; ++j) {  // hidden layer j: activation, then (unless it is the last) the next 64 x 64 layer
      const bool last_hidden = (j == nh - 1);
      for (int t : ts) {
        if (fused || (!ln && j == 0)) break;  // launch_edge_mlp_in or the layer before wrote the activation already
        const LayerBufs& lb = b.lay[t];
        const T* z = j == 0 ? lb.Z1 : j == 1 ? lb.Z2 : lb.Z3;
        T* h = last_hidden ? lb.H3 : lb.Hact;
        if (ln) {
          const std::string pre = "t" + std::to_string(t) + ".ln" + std::to_string(j);
          CKL(launch_ln_silu_fwd(z, w(pre + "g"), w(pre + "b"), h, Ec, s));
        } else {
          CKL(launch_silu(z, h, n64, s));
        }
      }
      if (last_hidden) break;
      std::vector<LinSpec> sp;
      for (int t : ts) {
        const std::string pre = "t" + std::to_string(t) + ".";
        const std::string an = j == 0 ? "A1" : "A2";
        const LayerBufs& lb = b.lay[t];
        T* const in = fused && (nh - 1 - j) % 2 == 0 ? lb.H3 : lb.Hact;
        LinSpec spec{in, kHidden, 0, 1, kHidden, pre + an, pre + an + "t", kHidden, j == 0 ? lb.Z2 : lb.Z3, kHidden,
                     0, mlp_bias ? w(pre + (j == 0 ? "b1" : "b2")) : nullptr};
        if (fused) spec.act_out = in == lb.H3 ? lb.Hact : lb.H3;
        sp.push_back(spec);
      }
      CKL(run_edge_linear(sp, Ec, s));
    }
    return TACE_OK;
  }
  // back through the hidden layers: lay[t].H3 holds dE/dh3 on entry; ddlen receives dE/d(edge length)
  int radial_backward(const EdgeArgs<T>& ea, const Bufs& b, const std::vector<int>& ts, long long e0, long long Ec, int accumulate,
                      cudaStream_t s) {
    if (Ec <= 0) return TACE_OK;
    if (rt_K) {
      // Tabulated weights: the tensor-product backward passes added their dE/d(edge length) to ddlen already; what is
      // left of this stage is the envelope's own derivative (apply_cutoff = False), once, with the last layer processed.
      const bool last_call = ts.size() > 1 || NL_ == 1 || ts[0] == 0;
      if (!last_call || !ea.denv) return TACE_OK;
      EdgeArgs<T> er = edge_range(ea, b, std::vector<int>{}, e0, Ec);
      er.accumulate_ddlen = 1; er.add_denv = 1;
      CKL(launch_edge_mlp_out(er, s));
      return TACE_OK;
    }
    const long long n64 = Ec * kHidden;
    // gradient buffer chain: H3 -> Hact -> Z3 (three hidden layers), H3 -> Hact (two), H3 (one); the first layer's
    // activation derivative is applied by launch_edge_mlp_out
    const bool ln = element2;
    for (int j = nh - 1; j >= 1; --j) {
      for (int t : ts) {
        const LayerBufs& lb = b.lay[t];
        T* g = (j == nh - 1) ? lb.H3 : lb.Hact;
        if (fused_activations()) break;  // the product that made g applied the derivative
        if (ln) {
          const std::string pre = "t" + std::to_string(t) + ".ln" + std::to_string(j);
          CKL(launch_ln_silu_bwd(g, j == 1 ? lb.Z2 : lb.Z3, w(pre + "g"), w(pre + "b"), Ec, s));
        } else {
          CKL(launch_silu_grad_mul(g, j == 1 ? lb.Z2 : lb.Z3, n64, s));
        }
      }
      std::vector<LinSpec> sp;
      for (int t : ts) {
        const std::string pre = "t" + std::to_string(t) + ".";
        const std::string an = j == 1 ? "A1" : "A2";
        const LayerBufs& lb = b.lay[t];
        const T* g = (j == nh - 1) ? lb.H3 : lb.Hact;
        T* dst = (j == nh - 1) ? lb.Hact : lb.Z3;
        LinSpec spec{g, kHidden, 0, 1, kHidden, pre + an + "t", pre + an, kHidden, dst, kHidden, 0, nullptr};
        if (fused_activations() && j == 2) spec.act_in = lb.Z2;  // (j == 1: launch_edge_mlp_out applies the first layer's)
        sp.push_back(spec);
      }
      CKL(run_edge_linear(sp, Ec, s));
    }
    EdgeArgs<T> er = edge_range(ea, b, ts, e0, Ec);
    if (ln) {  // through the first hidden layer's LayerNorm and activation; launch_edge_mlp_out then starts from dE/dz1
      for (int t : ts) {
        const std::string pre = "t" + std::to_string(t) + ".ln0";
        CKL(launch_ln_silu_bwd(dh1_buffer(b.lay[t]), b.lay[t].Z1, w(pre + "g"), w(pre + "b"), Ec, s));
      }
      er.dz1_given = 1;
    }
    er.accumulate_ddlen = accumulate;
    // the envelope term enters once: with the whole batch in one call, or with the last layer processed (layer 0)
    er.add_denv = (ts.size() > 1 || NL_ == 1 || ts[0] == 0) ? 1 : 0;
    CKL(launch_edge_mlp_out(er, s));
    return TACE_OK;
  }
  // last radial-MLP layer for edges [e0, e0 + Ec): W[e, :] = H3[e, :] @ W3 (forward) or dH3[e, :] = dW[e, :] @ W3^T
  int radial_last(const LayerPlan& p, const LayerBufs& lb, const std::string& pre, long long Ec, bool backward, cudaStream_t s) {
    if (Ec <= 0 || rt_K) return TACE_OK;  // tabulated weights: the radial MLP never runs
    const int NW = p.tp.NP * C;
    if (kTensorCore && NW % 64 == 0) {
      if (!backward)
        CKL(launch_tc_gemm(reinterpret_cast<const float*>(lb.H3), kHidden, reinterpret_cast<const float*>(w(pre + "W3t_hi")),
                           reinterpret_cast<const float*>(w(pre + "W3t_lo")), reinterpret_cast<float*>(lb.W), (long long)NW, (int)Ec,
                           NW, kHidden, dev_error, s, mlp_bias ? reinterpret_cast<const float*>(w(pre + "b3")) : nullptr));
      else
        CKL(launch_tc_gemm(reinterpret_cast<const float*>(lb.W), (long long)NW, reinterpret_cast<const float*>(w(pre + "W3_hi")),
                           reinterpret_cast<const float*>(w(pre + "W3_lo")), reinterpret_cast<float*>(lb.H3), kHidden, (int)Ec,
                           kHidden, NW, dev_error, s));
    } else {
      GemmBatch<T> gb = plain_batch(Ec);
      if (!backward) add_problem(gb, lb.H3, kHidden, 0, 1, kHidden, w(pre + "W3"), NW, lb.W, (long long)NW, 0,
                                 mlp_bias ? w(pre + "b3") : nullptr, 0);
      else add_problem(gb, lb.W, (long long)NW, 0, 1, NW, w(pre + "W3t"), kHidden, lb.H3, kHidden, 0, nullptr, 0);
      if (backward && fused_activations() && nh > 1) gb.p[0].act_in = nh == 3 ? lb.Z3 : lb.Z2;
      CKL(launch_gemm(gb, Ec, s));
    }
    return TACE_OK;
  }

  // Buffers of a layer's backward pass that are added to, or written only where the output has a rank.  Captured passes clear them on the
  // branch: rank 3 with features of rank 2, 64 channels, 32 atoms 175.7 -> 173.6 us, 256: 253.4 -> 251.3, 1 372: 567.0 -> 565.1; rank 2,
  // 108 atoms 166.3 -> 165.1 (runs of one side within 0.2 to 1.2 us); edge block, 54 atoms 1 037 -> 1 035, nothing beyond the spread above.
  int zero_gradients(const LayerPlan& p, const LayerBufs& lb, long long NL, cudaStream_t s) {
    if (bilinear) CKL(launch_fill_zero(lb.gXY, NL * D * 2 * C, s));
    else if ((int)p.out_ls.size() != L + 1) CKL(launch_fill_zero(lb.gAs, NL * D * C, s));
    if (cfg.correlation >= 3) CKL(launch_fill_zero(lb.gB2, NL * p.pb.NB * C, s));  // ranks above the output ranks only receive third-order terms
    return TACE_OK;
  }

  int forward(const TaceBatch* bt, const TaceOutputs* o, void* ws, size_t ws_bytes, cudaStream_t s) override {
    if (!bt || !o || !ws) return TACE_ERR_INVALID_ARGUMENT;
    backward_pass = false;
    if (n_unset != 0) return TACE_ERR_WEIGHTS_MISSING;
    const long long N = bt->n_atoms, NL = bt->n_local, E = bt->n_edges;
    const int B = bt->n_graphs;
    if (N < 0 || NL < 0 || NL > N || E < 0 || B <= 0 || !bt->species || !bt->graph_ptr || (E > 0 && !bt->edge_index))
      return TACE_ERR_INVALID_ARGUMENT;
    const bool vec_mode = bt->edge_vector != nullptr;
    if (!vec_mode && E > 0 && (!bt->positions || !bt->lattice || !bt->edge_shifts)) return TACE_ERR_INVALID_ARGUMENT;
    // ghost atoms need a feature exchange between layers (tace_set_exchange)
    if (NL != N && NL_ > 1 && (!exchange_fn || !vec_mode)) return TACE_ERR_UNSUPPORTED_CONFIG;
    if ((reinterpret_cast<uintptr_t>(ws) & 255) != 0) return TACE_ERR_INVALID_ARGUMENT;
    Arena ar; ar.base = static_cast<unsigned char*>(ws);
    Bufs b;
    if (layout(ar, b, N, NL, E, B) > ws_bytes) return TACE_ERR_CAPACITY;
    debug.clear();
    const bool need_grad = o->forces || o->virials || o->stress || o->edge_forces;

    phase_used = 0;
    if (NL == 0) {
      // A rank that owns no atom (a block of vacuum in a domain decomposition): nothing to evaluate, results are
      // zero, but the exchange callback still runs once per exchanged layer and direction, with zero rows, so that
      // the point-to-point pattern of the other ranks stays matched.
      if (o->energy) CKL(launch_fill_zero(static_cast<T*>(o->energy), (long long)B, s));
      if (o->forces) CKL(launch_fill_zero(static_cast<T*>(o->forces), 3 * N, s));
      if (o->virials) CKL(launch_fill_zero(static_cast<T*>(o->virials), 9LL * B, s));
      if (o->stress) CKL(launch_fill_zero(static_cast<T*>(o->stress), 9LL * B, s));
      if (o->edge_forces) CKL(launch_fill_zero(static_cast<T*>(o->edge_forces), 3 * E, s));
      for (int pass = 0; pass < (need_grad ? 2 : 1); ++pass)
        for (int k = 0; k < NL_; ++k) {
          const int t = pass == 0 ? k : NL_ - 1 - k;
          LayerBufs& lb = b.lay[t];
          const long long row = (long long)layers[t].tp.NX * C;
          if (pass == 0 && lb.xx) {
            CKL(launch_fill_zero(lb.x, N * row, s));
            CKS(exchange_begin(0, lb.x, lb.xx, N, (int)row, s));
            CKS(exchange_join(s));
          }
          if (pass == 1 && lb.gxx) {
            CKL(launch_fill_zero(lb.gx, N * row, s));
            CKS(exchange_begin(1, lb.gx, lb.gxx, N, (int)row, s));
            CKS(exchange_join(s));
          }
        }
      return TACE_OK;
    }
    PH("graph_prep");
    // ---- graph preparation
    GraphPrepArgs gp;
    gp.E = E; gp.n_atoms = (int)N; gp.n_local = (int)NL; gp.n_graphs = B; gp.n_elements = n_el;
    gp.edge_index = bt->edge_index; gp.species = bt->species; gp.graph_ptr = bt->graph_ptr;
    gp.e_src = b.e_src; gp.e_dst = b.e_dst; gp.e_orig = b.e_orig; gp.rowptr_dst = b.rowptr_dst;
    gp.perm_src = b.perm_src; gp.rowptr_src = b.rowptr_src; gp.atom_graph = b.atom_graph;
    gp.species_safe = b.species; gp.species_perm = b.species_perm; gp.species_rank = b.species_rank; gp.species_ptr = b.species_ptr; gp.tile_ptr = b.tile_ptr; gp.tc_tile_ptr = b.tc_tile_ptr;
    gp.temp = b.prep_temp; gp.temp_bytes = b.prep_temp_bytes;
    // edge chunks: one chunk (all atoms) unless the batch exceeds max_chunk_edges
    const bool chunked = E > max_chunk_edges;
    // With an exchange stream the tensor-product passes of the exchanged layers run in two parts: the target atoms none
    // of whose sources is a ghost while the ghost rows travel, the others afterwards (forward), and the other way round
    // for the gradients.  Every target is still summed in one piece, so the numbers do not depend on the schedule.
    const bool overlap = exchange_on_side() && !chunked && NL != N && NL_ > 1;
    gp.split_rows = overlap ? 1 : 0; gp.row_ids = b.row_ids; gp.row_split = b.row_split;
    gp.defer_src = branches || !need_grad;  // the view by sources is read by the backward pass only
    CK(launch_graph_prep(gp, s));
    launches += graph_prep_launches(gp);
    if (branches && need_grad) {
      cudaStream_t side;
      CKS(branch(s, &side));
      CKL(launch_edge_order_src(gp, side));
      for (int t = 0; t < NL_; ++t) CKS(zero_gradients(layers[t], b.lay[t], NL, side));
    }
    std::vector<int> chunk_atom{0, (int)NL}, chunk_edge{0, (int)E};
    if (chunked) {
      const int nc = b.n_chunks;
      CKL(launch_chunk_bounds(b.rowptr_dst, (int)NL, max_chunk_edges, nc, b.chunk_atom_ptr, b.chunk_edge_ptr, s));
      chunk_atom.assign(nc + 1, 0); chunk_edge.assign(nc + 1, 0);
      CK(cudaMemcpyAsync(chunk_atom.data(), b.chunk_atom_ptr, sizeof(int) * (nc + 1), cudaMemcpyDeviceToHost, s));
      CK(cudaMemcpyAsync(chunk_edge.data(), b.chunk_edge_ptr, sizeof(int) * (nc + 1), cudaMemcpyDeviceToHost, s));
      CK(cudaStreamSynchronize(s));
      for (int c = 0; c < nc; ++c)
        if (chunk_edge[c + 1] - chunk_edge[c] > b.chunk_rows) return TACE_ERR_CAPACITY;  // an atom with more than kChunkSlack edges
      if (need_grad && NL_ > 1) {
        CKL(launch_chunk_src_sort(b.e_src, E, (int)N, b.chunk_edge_ptr, nc, b.keys_cs, b.perm_cs, b.prep_temp, b.prep_temp_bytes, s));
        ++launches;
      }
    }
    const int n_chunks = (int)chunk_atom.size() - 1;
    PH("edge_fwd");

    // ---- edge features
    EdgeArgs<T> ea;
    memset(&ea, 0, sizeof(ea));
    ea.L = L; ea.n_layers = NL_; ea.E = E;
    ea.e_src = b.e_src; ea.e_dst = b.e_dst; ea.e_orig = b.e_orig;
    ea.positions = static_cast<const T*>(bt->positions); ea.lattice = static_cast<const T*>(bt->lattice);
    ea.atom_graph = b.atom_graph; ea.shifts = static_cast<const T*>(bt->edge_shifts);
    ea.edge_vector = static_cast<const T*>(bt->edge_vector);
    {
      // the radial parameters travel by value inside the kernel arguments
      for (int k = 0; k < kNumBessel; ++k) ea.rp.w[k] = host_bessel[k];
      ea.rp.pref = host_bessel[kNumBessel];
      ea.rp.rc = T(cfg.cutoff); ea.rp.p = cfg.envelope_p;
    }
    for (int t = 0; t < NL_; ++t) {
      const std::string pre = "t" + std::to_string(t) + ".";
      memset(&ea.mlp[t], 0, sizeof(ea.mlp[t]));
      ea.mlp[t].A0 = w(pre + "A0");
      if (mlp_bias) ea.mlp[t].b0 = w(pre + "b0");
      if (element2) { ea.mlp[t].tbl_dst = w(pre + "tdst"); ea.mlp[t].tbl_src = w(pre + "tsrc"); }
      ea.Z1[t] = b.lay[t].Z1;
      ea.dH1[t] = dh1_buffer(b.lay[t]);
    }
    ea.rp.env_after_mlp = env_after ? 1 : 0;
    ea.species = b.species;
    ea.env = b.env; ea.denv = b.denv; ea.add_denv = 1;
    ea.dlen = b.dlen; ea.ddlen = b.ddlen;
    ea.vec = b.vec; ea.Y = b.Y; ea.dY = b.dY; ea.g = b.g; ea.n_valid = b.rowptr_dst + N; ea.edge_forces = static_cast<T*>(o->edge_forces);
    CKL(launch_edge_fwd(ea, s));
    std::vector<int> all_layers;
    for (int t = 0; t < NL_; ++t) all_layers.push_back(t);
    PH("radial_mlp_fwd");
    if (!chunked) CKS(radial_forward(ea, b, all_layers, 0, E, s));  // all layers at once; chunked passes do it per layer and chunk
    debug.push_back({"Y", b.Y, (long long)D * E});
    debug.push_back({"vec", b.vec, 3 * E});

    // The last layers of the radial MLPs of all interactions but the first run beside the first interaction and its products per atom,
    // which leave most of the chip idle on small systems; the way back (dE/dW of an interaction is not needed before the end of the
    // pass) in the same way.
    if (branches && !chunked && !rt_K && NL_ > 1) {
      cudaStream_t side;
      CKS(branch(s, &side));
      for (int t = 1; t < NL_; ++t) CKS(radial_last(layers[t], b.lay[t], "t" + std::to_string(t) + ".", E, false, side));
    }

    // ---- layers, forward
    bool wigner_done = false, tece_seen = false;
    PH("embed");
    CKL(launch_species_gather(w(folded ? "emb_up" : "emb"), b.species, folded ? b.lay[0].x : b.lay[0].h_in, (int)N, C, s));  // ghosts too
    for (int t = 0; t < NL_; ++t) {
      const LayerPlan& p = layers[t];
      LayerBufs& lb = b.lay[t];
      const std::string pre = "t" + std::to_string(t) + ".";
      const std::string ts = std::to_string(t);
      if (t > 0 || !folded) {  // linear_up (the first layer's is part of the folded embedding)
        PH(("t" + ts + ".fwd.linear_up").c_str());
        std::vector<LinSpec> sp;
        for (int l : p.in_ls)
          sp.push_back({lb.h_in + (long long)l * l * C, (long long)p.Din * C, C, 2 * l + 1, C, pre + "up.l" + std::to_string(l),
                        pre + "upT.l" + std::to_string(l), C, lb.x + (long long)l * l * C, (long long)p.tp.NX * C, C,
                        l == 0 ? w(pre + "up.b") : nullptr});
        CKL(run_linear(sp, t == 0 ? N : NL, s));  // layer 0 embeds every atom; later layers own only local rows
      }
      const T* x_src = lb.x;
      const bool split = overlap && lb.xx && !p.tece;
      if (lb.xx) {
        // Ghost rows of x are copies of rows owned elsewhere: zero them, let the caller's exchange fill
        // them (lmp_data.forward_exchange in the reference, tace/models/lammps.py:82-129).
        CKL(launch_fill_zero(lb.x + NL * p.tp.NX * C, (N - NL) * p.tp.NX * C, s));
        CKS(exchange_begin(0, lb.x, lb.xx, N, p.tp.NX * C, s));
        if (!split) CKS(exchange_join(s));
        x_src = lb.xx;
      }
      std::vector<LinSpec> down = down_specs(p, lb, pre, false);
      unsigned* mtop = p.tece ? nullptr : down_tops(down, lb.mtop, NL, false);
      if (mtop) CK(cudaMemsetAsync(mtop, 0, sizeof(unsigned) * (size_t)NL * (L + 1), s));
      for (int c = 0; c < n_chunks; ++c) {
        const long long e0 = chunk_edge[c], Ec = chunk_edge[c + 1] - e0;
        const int a0 = chunk_atom[c], na = chunk_atom[c + 1] - a0;
        if (chunked) {
          PH("radial_mlp_fwd");
          CKS(radial_forward(ea, b, std::vector<int>{t}, e0, Ec, s));
        }
        PH(("t" + ts + ".fwd.radial_gemm").c_str());
        if (branches && !chunked && t > 0) CKS(merge(s));
        else CKS(radial_last(p, lb, pre, Ec, false, s));
        PH(("t" + ts + ".fwd.tp").c_str());
        if (p.tece) {  // the edge block instead of the tensor product (whole batch only)
          if (chunked) return TACE_ERR_CAPACITY;
          const TeceArgs<T> tc = tece_args(ea, b, lb, pre, x_src, N, NL, E);
          if (!wigner_done) { CKL(launch_tece(tc, TECE_WIGNER, s)); wigner_done = true; }
          CKS(tece_forward(tc, lb, pre, E, s));
          continue;
        }
        TPArgs<T> ta;
        memset(&ta, 0, sizeof(ta));
        ta.L = L; ta.scalar_src = p.scalar_src; ta.Lin = Ln; ta.C = C; ta.n_seg = na; ta.rowptr = b.rowptr_dst + a0;
        ta.e_src = b.e_src; ta.Y = b.Y; ta.W = lb.W; ta.x = x_src; ta.M = lb.M + (long long)a0 * p.tp.NM * C; ta.e_base = e0; ta.n_edges = round_edges(Ec);
        ta.split_sums = lb.xx == nullptr; ta.env = b.env;
        if (mtop) ta.top = mtop + (long long)a0 * (L + 1);
        if (rt_K) { ta.rtab = w(pre + "rtab"); ta.rt_K = rt_K; ta.rt_inv_h = T(rt_K) / T(cfg.cutoff); ta.dlen = b.dlen; }
        if (split) {  // targets that read owned rows only (final in x itself); the others once the ghost rows have arrived
          ta.x = lb.x; ta.row_ids = b.row_ids; ta.row_split = b.row_split + 1; ta.row_part = 0;
          CKL(launch_tp_fwd(ta, s));
          CKS(exchange_join(s));
          ta.x = lb.xx; ta.row_part = 1;
        }
        CKL(launch_tp_fwd(ta, s));
      }
      debug.push_back({"x" + ts, lb.x, N * p.tp.NX * C});
      debug.push_back({"M" + ts, lb.M, NL * p.tp.NM * C});
      PH(("t" + ts + ".fwd.node").c_str());
      CKL(run_linear(down, NL, s));
      if (density) {  // learned normalisation instead of the constant folded into the weights
        const DensityArgs<T> da = density_args(ea, b, lb, pre, NL, E);
        CKL(launch_density_fwd(da, s));
        CKL(launch_scale_rows(lb.Gt, lb.inv_density, NL, (L + m0 + D) * C, (long long)(L + 1 + D) * C, s));
      }
      CKL(launch_gate_fwd(lb.Gt, lb.a, (int)NL, L, C, m0, s));
      {
        std::vector<LinSpec> sp;
        for (int l = 0; l <= L; ++l)
          sp.push_back({lb.a + (long long)l * l * C, (long long)D * C, C, 2 * l + 1, C, pre + "nl.l" + std::to_string(l),
                        pre + "nlT.l" + std::to_string(l), C, lb.As + (long long)l * l * C, (long long)D * C, C,
                        l == 0 ? w(pre + "nl.b") : nullptr});
        // the per-species part works in species-sorted space: this linear writes its rows there, the coefficient linears scatter into `out`
        CKL(run_linear(sp, NL, s, b.species_rank));
      }
      debug.push_back({"A" + ts, lb.As, NL * D * C, b.species_rank, D * C});
      if (bilinear) {
        std::vector<LinSpec> sp;
        for (int l = 0; l <= L; ++l)
          sp.push_back({lb.As + (long long)l * l * C, (long long)D * C, C, 2 * l + 1, C, pre + "pu.l" + std::to_string(l),
                        pre + "puT.l" + std::to_string(l), 2 * C, lb.XY + (long long)l * l * 2 * C, (long long)D * 2 * C, 2 * C,
                        l == 0 ? w(pre + "pu.b") : nullptr});
        CKL(run_linear(sp, NL, s));
        sp.clear();
        sp.push_back({lb.As, (long long)D * C, C, 1, C, pre + "pg", pre + "pgT", p.pb.NP * C, lb.Zg, (long long)p.pb.NP * C, 0,
                      w(pre + "pg.b")});
        CKL(run_linear(sp, NL, s));
        CKL(launch_pbl_fwd(lb.XY, lb.Zg, lb.B2, (int)NL, L, p.pb_lout, C, s));
      }
      {
        std::vector<SpeciesSpec> sp;
        // the products of all correlation orders and the skip connection from the layer input add up in one pass per rank
        const bool res = p.has_res && !res_identity && folded;
        const std::string f = folded ? "f.l" : ".l";
        for (size_t i = 0; i < p.out_ls.size(); ++i) {
          const int l = p.out_ls[i];
          const std::string ls = std::to_string(l);
          T* out = (folded ? lb.h_out : lb.out) + (long long)l * l * C;
          sp.push_back({bilinear ? lb.XY + (long long)l * l * 2 * C : lb.As + (long long)l * l * C, (long long)D * C * (bilinear ? 2 : 1),
                        (long long)C * (bilinear ? 2 : 1), 2 * l + 1, C, pre + "c0" + f + ls, pre + "c0T.l" + ls, C, out,
                        (long long)p.Dout * C, C, l == 0 ? w(pre + (folded ? "cf.b" : "c.b")) : nullptr, true, 0, l});
          if (cfg.correlation >= 2) {
            const int K = p.pb.k[i] * C;
            sp.push_back({lb.B2 + (long long)p.pb.base[i] * C, (long long)p.pb.NB * C, K, 2 * l + 1, K, pre + "c1" + f + ls, pre + "c1T.l" + ls,
                          C, out, (long long)p.Dout * C, C, nullptr, true, kJoin, l, 1});
          }
          if (cfg.correlation >= 3) {
            const int K = p.pb3.k[i] * C;
            sp.push_back({lb.B3 + (long long)p.pb3.base[i] * C, (long long)p.pb3.NB * C, K, 2 * l + 1, K, pre + "c2" + f + ls, pre + "c2T.l" + ls,
                          C, out, (long long)p.Dout * C, C, nullptr, true, kJoin});
          }
          if (res)
            sp.push_back({lb.hs + (long long)l * l * C, (long long)p.Din * C, C, 2 * l + 1, C, pre + "res.l" + ls, pre + "resT.l" + ls, C, out,
                          (long long)p.Dout * C, C, nullptr, true, kJoin, l, 2});
        }
        unsigned* top = species_tops(sp, lb.top, NL, false);
        if (!bilinear && cfg.correlation >= 2) CKL(launch_pb_fwd(lb.As, lb.B2, (int)NL, L, p.pb_lout, C, s, top, 3 * (L + 1)));
        if (cfg.correlation >= 3) CKL(launch_pb3_fwd(lb.As, lb.B2, lb.B3, (int)NL, L, p.last ? -1 : Ln, C, s));
        if (res) CKL(gather_rows(lb.h_in, b.species_perm, lb.hs, NL, p.Din, top ? top + 2 * (L + 1) : nullptr, 3 * (L + 1), s));
        CKL(run_species_linear(sp, b, NL, s));
      }
      if (!folded) {
        std::vector<LinSpec> sp;
        for (int l : p.out_ls)
          sp.push_back({lb.out + (long long)l * l * C, (long long)p.Dout * C, C, 2 * l + 1, C, pre + "lin.l" + std::to_string(l),
                        pre + "linT.l" + std::to_string(l), C, lb.h_out + (long long)l * l * C, (long long)p.Dout * C, C,
                        l == 0 ? w(pre + "lin.b") : nullptr});
        CKL(run_linear(sp, NL, s));
      }
      if (p.has_res && res_identity) {  // tace/models/_e3nn/residual.py:216-250: the ranks the output keeps, copied over
        CKL(launch_add_rows(lb.h_out, (long long)p.Dout * C, lb.h_in, (long long)p.Din * C, NL, p.Dout * C, s));
      } else if (p.has_res && !folded) {  // per-species skip connection from the layer input
        CKL(launch_gather_rows(lb.h_in, b.species_perm, lb.hs, NL, p.Din * C, s));
        std::vector<SpeciesSpec> sp;
        for (int l : p.out_ls)
          sp.push_back({lb.hs + (long long)l * l * C, (long long)p.Din * C, C, 2 * l + 1, C, pre + "res.l" + std::to_string(l),
                        pre + "resT.l" + std::to_string(l), C, lb.h_out + (long long)l * l * C, (long long)p.Dout * C, C,
                        l == 0 ? w(pre + "res.b") : nullptr, true, 1});
        CKL(run_species_linear(sp, b, NL, s));
      }
      debug.push_back({"h" + std::to_string(t + 1), lb.h_out, NL * p.Dout * C});
    }

    // ---- read-out
    PH("readout");
    LayerBufs& top = b.lay[NL_ - 1];
    ReadoutArgs<T> ra;
    memset(&ra, 0, sizeof(ra));
    ra.h = top.h_out; ra.hs = (long long)layers[NL_ - 1].Dout * C; ra.W1 = w("ro.W1"); ra.W2 = w("ro.W2");
    ra.scale = w("scale"); ra.e0 = w("e0"); ra.species = bt->species; ra.atom_graph = b.atom_graph;
    ra.graph_ptr = bt->graph_ptr; ra.rowptr_dst = b.rowptr_dst; ra.node_energy = static_cast<T*>(o->node_energy);
    ra.e_scaled = b.e_scaled; ra.gh = need_grad ? top.gh_out : nullptr; ra.n = (int)NL; ra.C = C; ra.H = H;
    ra.fidelity = bt->fidelity; ra.n_el = n_el;
    ZblArgs<T> za;
    memset(&za, 0, sizeof(za));
    if (zbl) {  // pair repulsion per atom, summed over the incoming edges
      za.rowptr_dst = b.rowptr_dst; za.e_src = b.e_src; za.e_dst = b.e_dst; za.species = b.species; za.dlen = b.dlen;
      za.z = w("zbl.z"); za.rcov = w("zbl.rcov"); za.par = w("zbl.par"); za.p = cfg.envelope_p; za.n = (int)NL; za.E = E;
      za.node = b.zbl_node;
      CKL(launch_zbl_fwd(za, s));
      ra.zbl = b.zbl_node; ra.zbl_after = (zbl == 2);
      ra.factor = b.ro_factor;
    }
    if (cfg.use_alllayer) {  // linear read-outs of the layers below the last
      ra.n_extra = NL_ - 1;
      for (int t = 0; t + 1 < NL_; ++t) {
        ra.extra_h[t] = b.lay[t].h_out; ra.extra_hs[t] = (long long)layers[t].Dout * C; ra.extra_w[t] = w("ro.lin" + std::to_string(t));
      }
      ra.factor = b.ro_factor;
    }
    CKL(launch_readout(ra, s));
    if (o->energy) {
      CKL(launch_graph_energy(b.e_scaled, w("e0"), b.species, bt->graph_ptr, bt->fidelity, n_el, static_cast<T*>(o->energy), B, NL,
                              b.energy_partial, s));
      if (graph_energy_slices(NL, B) > 1) ++launches;  // the slice sums are added by a second kernel
    }
    if (!need_grad) { PH("end"); return TACE_OK; }

    // ---- layers, backward
    backward_pass = true;
    CKS(merge(s));  // a single interaction has not met the branch yet
    for (int t = NL_ - 1; t >= 0; --t) {
      const LayerPlan& p = layers[t];
      LayerBufs& lb = b.lay[t];
      const std::string pre = "t" + std::to_string(t) + ".";
      const std::string ts = std::to_string(t);
      PH(("t" + ts + ".bwd.node").c_str());
      if (cfg.use_alllayer && t + 1 < NL_)  // this layer's own linear read-out, on top of what the layer above sent down
        CKL(launch_readout_linear_bwd(lb.gh_out, (long long)p.Dout * C, b.ro_factor, w("ro.lin" + ts), b.atom_graph, bt->fidelity,
                                      (int)NL, C, s));
      if (!folded) {  // through the final linear; else it is part of the coefficients
        std::vector<LinSpec> sp;
        for (int l : p.out_ls)
          sp.push_back({lb.gh_out + (long long)l * l * C, (long long)p.Dout * C, C, 2 * l + 1, C, pre + "linT.l" + std::to_string(l),
                        pre + "lin.l" + std::to_string(l), C, lb.gout_s + (long long)l * l * C, (long long)p.Dout * C, C, nullptr});
        CKL(run_linear(sp, NL, s, b.species_rank));
      }
      // through the per-species coefficients and the product basis, in species-sorted space
      unsigned* gtop = nullptr;  // largest elements of the rows of gout_s, where they have been taken
      if (!branches) CKS(zero_gradients(p, lb, NL, s));
      {
        std::vector<SpeciesSpec> sp;
        for (int l : p.out_ls)
          sp.push_back({lb.gout_s + (long long)l * l * C, (long long)p.Dout * C, C, 2 * l + 1, C, pre + "c0T.l" + std::to_string(l),
                        pre + "c0.l" + std::to_string(l), C, bilinear ? lb.gXY + (long long)l * l * 2 * C : lb.gAs + (long long)l * l * C,
                        (long long)D * C * (bilinear ? 2 : 1), (long long)C * (bilinear ? 2 : 1), nullptr, false, 0, l});
        if (cfg.correlation < 2) {
          if (folded) CKL(launch_gather_rows(lb.gh_out, b.species_perm, lb.gout_s, NL, p.Dout * C, s));
          CKL(run_species_linear(sp, b, NL, s));
        } else {  // the gradients of every order's basis in the same launch
          // gradient of the second-order basis: written over B2 itself, or into gB2 when the third order still needs B2
          T* g2 = cfg.correlation >= 3 ? lb.gB2 : lb.B2;
          if (cfg.correlation >= 3) {
            for (size_t i = 0; i < p.out_ls.size(); ++i) {
              const int l = p.out_ls[i];
              const int K = p.pb3.k[i] * C;
              sp.push_back({lb.gout_s + (long long)l * l * C, (long long)p.Dout * C, C, 2 * l + 1, C, pre + "c2T.l" + std::to_string(l),
                            pre + "c2.l" + std::to_string(l), K, lb.B3 + (long long)p.pb3.base[i] * C, (long long)p.pb3.NB * C, K,
                            nullptr, false, 0, l});
            }
          }
          for (size_t i = 0; i < p.out_ls.size(); ++i) {
            const int l = p.out_ls[i];
            const int K = p.pb.k[i] * C;
            sp.push_back({lb.gout_s + (long long)l * l * C, (long long)p.Dout * C, C, 2 * l + 1, C, pre + "c1T.l" + std::to_string(l),
                          pre + "c1.l" + std::to_string(l), K, g2 + (long long)p.pb.base[i] * C, (long long)p.pb.NB * C, K, nullptr,
                          false, 0, l});
          }
          gtop = species_tops(sp, lb.gtop, NL, true);
          if (folded) CKL(gather_rows(lb.gh_out, b.species_perm, lb.gout_s, NL, p.Dout, gtop, L + 1, s));
          CKL(run_species_linear(sp, b, NL, s));  // B2 (gB2) and B3 now hold their gradients
          if (cfg.correlation >= 3) {
            CKL(launch_pb3_bwd(lb.As, lb.B2, lb.B3, lb.gB2, lb.gAs, (int)NL, L, p.last ? -1 : Ln, C, s));
            ++launches;
          }
          if (bilinear) {  // back through the gated product, then through the product's own linear_up
            CKL(launch_pbl_bwd(lb.XY, lb.Zg, g2, lb.gXY, lb.gZg, (int)NL, L, p.pb_lout, C, s));
            std::vector<LinSpec> lp;
            for (int l = 0; l <= L; ++l)
              lp.push_back({lb.gXY + (long long)l * l * 2 * C, (long long)D * 2 * C, 2 * C, 2 * l + 1, 2 * C, pre + "puT.l" + std::to_string(l),
                            pre + "pu.l" + std::to_string(l), C, lb.gAs + (long long)l * l * C, (long long)D * C, C, nullptr});
            CKL(run_linear(lp, NL, s));
            lp.clear();
            lp.push_back({lb.gZg, (long long)p.pb.NP * C, 0, 1, p.pb.NP * C, pre + "pgT", pre + "pg", C, lb.gAs, (long long)D * C, 0,
                          nullptr, 1});
            CKL(run_linear(lp, NL, s));
          } else {
            CKL(launch_pb_bwd(lb.As, g2, lb.gAs, (int)NL, L, p.pb_lout, C, s));
          }
        }
      }
      {
        std::vector<LinSpec> sp;
        for (int l = 0; l <= L; ++l)
          sp.push_back({lb.gAs + (long long)l * l * C, (long long)D * C, C, 2 * l + 1, C, pre + "nlT.l" + std::to_string(l),
                        pre + "nl.l" + std::to_string(l), C, lb.ga + (long long)l * l * C, (long long)D * C, C, nullptr});
        CKL(run_linear(sp, NL, s, b.species_perm));  // back to atom order
      }
      std::vector<LinSpec> down = down_specs(p, lb, pre, true);
      CKL(launch_gate_bwd(lb.Gt, lb.ga, lb.gGt, (int)NL, L, C, m0, s, down_tops(down, lb.dtop, NL, true)));
      if (density)  // d / d density_i, and the gradient of the unscaled linear_down output
        CKL(launch_density_node_bwd(lb.gGt, lb.Gt, lb.inv_density, lb.gdens, NL, (L + m0 + D) * C, (long long)(L + 1 + D) * C, s));
      CKL(run_linear(down, NL, s));  // through linear_down
      // edge pass: gradients of the per-edge weights (in place over W), of the angular features and,
      // per edge, of the source features
      if (chunked && !p.scalar_src) CKL(launch_fill_zero(lb.gx, N * p.tp.NX * C, s));  // chunks add their shares
      for (int c = 0; c < n_chunks; ++c) {
        const long long e0 = chunk_edge[c], Ec = chunk_edge[c + 1] - e0;
        const int a0 = chunk_atom[c], na = chunk_atom[c + 1] - a0;
        if (chunked) {  // the per-edge activations and weights of this chunk were not kept: recompute them
          PH("radial_mlp_fwd");
          CKS(radial_forward(ea, b, std::vector<int>{t}, e0, Ec, s));
          PH(("t" + ts + ".fwd.radial_gemm").c_str());
          CKS(radial_last(p, lb, pre, Ec, false, s));
        }
        PH(("t" + ts + ".bwd.tp").c_str());
        if (p.tece) {
          if (t == NL_ - 1) {  // no tensor product above to initialise the accumulators of the layers below
            CKL(launch_fill_zero(b.dY, E * D, s));
            if (b.denv) CKL(launch_fill_zero(b.denv, E, s));
          }
          const TeceArgs<T> tc = tece_args(ea, b, lb, pre, lb.xx ? lb.xx : lb.x, N, NL, E);
          cudaStream_t side = s;
          CKS(merge(s));  // the Wigner gradients of the edge block above
          CKS(tece_backward(tc, b, lb, pre, N, E, !tece_seen, s, &side));
          tece_seen = true;
          PH(("t" + ts + ".bwd.radial_gemm").c_str());
          CKS(radial_last(p, lb, pre, Ec, true, side));
          continue;
        }
        TPArgs<T> ta;
        memset(&ta, 0, sizeof(ta));
        ta.L = L; ta.scalar_src = p.scalar_src; ta.Lin = Ln; ta.C = C; ta.e_src = b.e_src; ta.Y = b.Y;
        ta.W = lb.W; ta.x = lb.xx ? lb.xx : lb.x; ta.gM = lb.M + (long long)a0 * p.tp.NM * C; ta.n_seg = na;
        ta.rowptr = b.rowptr_dst + a0; ta.dW = lb.W; ta.dY = b.dY; ta.e_base = e0; ta.n_edges = round_edges(Ec);
        ta.accumulate_dY = (t != NL_ - 1); ta.dxe = p.scalar_src ? nullptr : b.dxe;
        ta.env = b.env; ta.denv = b.denv; ta.accumulate_denv = (t != NL_ - 1);
        if (rt_K) {
          ta.rtab = w(pre + "rtab"); ta.rt_K = rt_K; ta.rt_inv_h = T(rt_K) / T(cfg.cutoff); ta.dlen = b.dlen;
          ta.dW = nullptr; ta.ddlen = b.ddlen; ta.accumulate_ddlen = (t != NL_ - 1);
        }
        if (overlap && lb.gxx) {
          // Targets with ghost sources first: the per-source sums of the ghost rows are what the owners of those atoms
          // wait for.  While they travel the other targets follow; the sums over owned sources land in the owned rows of
          // xx (x itself still holds those rows, and nothing reads xx any more), to be added to the arrivals after the join.
          const int row = p.tp.NX * C;
          TPArgs<T> tb = ta;
          tb.row_ids = b.row_ids; tb.row_split = b.row_split + 1; tb.row_part = 1;
          CKL(launch_tp_bwd(tb, s));
          PH(("t" + ts + ".bwd.src_sum").c_str());
          CKL(launch_fill_zero(lb.gx, NL * row, s));
          CKL(launch_segment_sum_rows(b.dxe, b.rowptr_src, b.perm_src, lb.gx, (int)NL, (int)(N - NL), row, s));
          CKS(exchange_begin(1, lb.gx, lb.gxx, N, row, s));
          PH(("t" + ts + ".bwd.tp").c_str());
          ta.x = lb.x; ta.row_ids = b.row_ids; ta.row_split = b.row_split + 1; ta.row_part = 0;
          CKL(launch_tp_bwd(ta, s));
          PH(("t" + ts + ".bwd.src_sum").c_str());
          CKL(launch_segment_sum_rows(b.dxe, b.rowptr_src, b.perm_src, lb.xx, 0, (int)NL, row, s));
        } else {
          CKL(launch_tp_bwd(ta, s));
          if (!p.scalar_src) {  // sum the per-edge rows over the edges leaving each source atom
            PH(("t" + ts + ".bwd.src_sum").c_str());
            if (chunked) CKL(launch_chunk_src_sum(b.dxe, b.keys_cs, b.perm_cs, e0, e0 + Ec, (long long)c * N, lb.gx, p.tp.NX * C, s));
            else CKL(launch_segment_sum_rows(b.dxe, b.rowptr_src, b.perm_src, lb.gx, 0, (int)N, p.tp.NX * C, s));
          }
        }
        PH(("t" + ts + ".bwd.radial_gemm").c_str());
        cudaStream_t side = s;
        if (t > 0 && !chunked && !rt_K) CKS(branch(s, &side));
        CKS(radial_last(p, lb, pre, Ec, true, side));  // back through the last radial-MLP layer: H3 <- dE/dh3
        if (chunked) {
          PH("radial_mlp_bwd");
          CKS(radial_backward(ea, b, std::vector<int>{t}, e0, Ec, t != NL_ - 1, s));
        }
      }
      if (lb.gxx) {  // gradients that landed on ghost rows go back to their owners (reverse_exchange)
        if (overlap && !p.tece) {  // already on its way: owned rows of gxx = arrivals + this rank's own sums
          CKS(exchange_join(s));
          CKL(launch_add_inplace(lb.gxx, lb.xx, NL * p.tp.NX * C, s));
        } else {
          CKS(exchange_begin(1, lb.gx, lb.gxx, N, p.tp.NX * C, s));
          CKS(exchange_join(s));
        }
      }
      if (!p.scalar_src) {
        PH(("t" + ts + ".bwd.linear_up").c_str());
        std::vector<LinSpec> sp;
        for (int l : p.in_ls)
          sp.push_back({(lb.gxx ? lb.gxx : lb.gx) + (long long)l * l * C, (long long)p.tp.NX * C, C, 2 * l + 1, C,
                        pre + "upT.l" + std::to_string(l), pre + "up.l" + std::to_string(l), C, lb.gh_in + (long long)l * l * C,
                        (long long)p.Din * C, C, nullptr});
        CKL(run_linear(sp, NL, s));
        if (p.has_res && res_identity) {
          CKL(launch_add_rows(lb.gh_in, (long long)p.Din * C, lb.gh_out, (long long)p.Dout * C, NL, p.Dout * C, s));
        } else if (p.has_res) {
          if (!folded) CKL(launch_gather_rows(lb.gh_out, b.species_perm, lb.gout_s, NL, p.Dout * C, s));
          std::vector<SpeciesSpec> sp2;  // gout_s: the species-sorted gradient of this layer's output
          for (int l : p.out_ls)
            sp2.push_back({lb.gout_s + (long long)l * l * C, (long long)p.Dout * C, C, 2 * l + 1, C, pre + "resT.l" + std::to_string(l),
                           pre + "res.l" + std::to_string(l), C, lb.gh_in + (long long)l * l * C, (long long)p.Din * C, C, nullptr, true, 1, l});
          set_tops(sp2, gtop, 1);
          CKL(run_species_linear(sp2, b, NL, s));
        }
      }
    }

    // ---- back to the edge vectors, then forces and virials
    PH("radial_mlp_bwd");
    CKS(merge(s));
    if (!chunked) CKS(radial_backward(ea, b, all_layers, 0, E, 0, s));  // lay[t].H3 holds dE/dh3 of each layer's radial MLP
    for (int t = 0; t < NL_; ++t)  // the edge blocks' own dependence on the edge lengths (radial projection, cutoff in the softmax)
      if (layers[t].tece) CKL(launch_add_inplace(b.ddlen, b.lay[t].tddlen, E, s));
    if (tece_mask) ea.gvec_extra = b.tgvec;  // and on the edge vectors through the frames
    if (density) {  // the densities' dependence on the edge lengths
      for (int t = 0; t < NL_; ++t) {
        DensityArgs<T> da = density_args(ea, b, b.lay[t], "t" + std::to_string(t) + ".", NL, E);
        da.gdens = b.lay[t].gdens; da.ddlen = b.ddlen;
        CKL(launch_density_bwd(da, s));
      }
    }
    if (zbl) {  // the repulsion's own dependence on the edge lengths
      za.ddlen = b.ddlen; za.factor = (zbl == 1) ? b.ro_factor : nullptr;
      CKL(launch_zbl_bwd(za, s));
    }
    PH("edge_bwd");
    CKL(launch_edge_bwd(ea, s));
    debug.push_back({"g", b.g, 3 * E});
    PH("forces");
    const bool want_virial = (o->virials || o->stress) && !vec_mode;
    ForceArgs<T> fa;
    memset(&fa, 0, sizeof(fa));
    fa.n_atoms = (int)N; fa.n_local = (int)NL; fa.rowptr_dst = b.rowptr_dst; fa.rowptr_src = b.rowptr_src;
    fa.perm_src = b.perm_src; fa.g = b.g; fa.vec = b.vec; fa.forces = static_cast<T*>(o->forces);
    fa.atom_virial = want_virial ? b.atom_virial : nullptr;
    if (fa.forces || fa.atom_virial) CKL(launch_forces(fa, s));
    if (want_virial)
      CKL(launch_graph_virial(b.atom_virial, bt->graph_ptr, static_cast<const T*>(bt->lattice), static_cast<T*>(o->virials),
                             static_cast<T*>(o->stress), B, s));
    PH("end");
    return TACE_OK;
  }

  int64_t debug_read(const char* name, void* dst, int64_t numel, cudaStream_t s) override {
    for (const auto& d : debug) {
      if (d.name == name) {
        const long long n = d.numel < numel ? d.numel : numel;
        if (d.perm) {
          const long long rows = n / d.row;  // whole rows
          if (launch_gather_rows(static_cast<const T*>(d.ptr), d.perm, static_cast<T*>(dst), rows, (int)d.row, s) != cudaSuccess) return TACE_ERR_CUDA;
          return rows * d.row;
        }
        if (cudaMemcpyAsync(dst, d.ptr, sizeof(T) * (size_t)n, cudaMemcpyDeviceToDevice, s) != cudaSuccess) return TACE_ERR_CUDA;
        return n;
      }
    }
    return TACE_ERR_INVALID_ARGUMENT;
  }
};

}  // namespace tace

using tace::ModelBase;

struct TaceModel {
  ModelBase* impl;
};

extern "C" {

const char* tace_status_string(int status) {
  switch (status) {
    case TACE_OK: return "ok";
    case TACE_ERR_INVALID_ARGUMENT: return "invalid argument";
    case TACE_ERR_UNSUPPORTED_CONFIG: return "unsupported model configuration";
    case TACE_ERR_CAPACITY: return "capacity exceeded (workspace too small or index range)";
    case TACE_ERR_CUDA: return "CUDA error";
    case TACE_ERR_NO_DEVICE: return "no sm_100 CUDA device";
    case TACE_ERR_UNKNOWN_WEIGHT: return "unknown weight name";
    case TACE_ERR_WEIGHTS_MISSING: return "weights not fully set";
    default: return "unknown status";
  }
}

int tace_create(const TaceConfig* cfg, TaceModel** out) {
  if (!cfg || !out) return TACE_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  if (cfg->L < 1 || cfg->L > 3 || cfg->num_layers < 1 || cfg->num_layers > tace::kMaxLayers || cfg->num_channel < 32 ||
      cfg->num_channel > 256 || (cfg->num_channel & 31) || cfg->num_elements < 1 || cfg->correlation < 1 ||
      cfg->correlation > 3 || cfg->num_bessel != tace::kNumBessel || cfg->mlp_hidden != tace::kHidden ||
      cfg->readout_hidden < 1 || cfg->readout_hidden > 64 || cfg->envelope_p < 2 || !(cfg->cutoff > 0.0) ||
      !(cfg->avg_num_neighbors > 0.0) || (cfg->dtype != TACE_F32 && cfg->dtype != TACE_F64))
    return TACE_ERR_UNSUPPORTED_CONFIG;
  int dev = 0;
  cudaDeviceProp prop;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaGetDeviceProperties(&prop, dev) != cudaSuccess) return TACE_ERR_NO_DEVICE;
  if (prop.major != 10) return TACE_ERR_NO_DEVICE;
  ModelBase* impl = nullptr;
  int st;
  if (cfg->dtype == TACE_F32) {
    auto* m = new (std::nothrow) tace::Model<float>();
    if (!m) return TACE_ERR_CUDA;
    st = m->init(*cfg); impl = m;
  } else {
    auto* m = new (std::nothrow) tace::Model<double>();
    if (!m) return TACE_ERR_CUDA;
    st = m->init(*cfg); impl = m;
  }
  if (st != TACE_OK) { delete impl; return st; }
  *out = new TaceModel{impl};
  return TACE_OK;
}

void tace_destroy(TaceModel* model) {
  if (!model) return;
  model->impl->release_graphs();
  delete model->impl;
  delete model;
}

int tace_weight_count(const TaceModel* model) { return model ? model->impl->weight_count() : TACE_ERR_INVALID_ARGUMENT; }
int tace_weight_info(const TaceModel* model, int index, const char** name, int64_t* numel) {
  return model ? model->impl->weight_info(index, name, numel) : TACE_ERR_INVALID_ARGUMENT;
}
int tace_set_weight(TaceModel* model, const char* name, const void* host_data, int64_t numel) {
  return model ? model->impl->set_weight(name, host_data, numel) : TACE_ERR_INVALID_ARGUMENT;
}
int tace_workspace_bytes(const TaceModel* model, int64_t n_atoms, int64_t n_local, int64_t n_edges, int32_t n_graphs,
                         size_t* bytes) {
  return model ? const_cast<TaceModel*>(model)->impl->workspace_bytes(n_atoms, n_local, n_edges, n_graphs, bytes)
               : TACE_ERR_INVALID_ARGUMENT;
}
int tace_forward(TaceModel* model, const TaceBatch* batch, const TaceOutputs* out, void* workspace, size_t workspace_bytes,
                 tace_stream_t stream) {
  if (!model) return TACE_ERR_INVALID_ARGUMENT;
  return model->impl->forward_entry(batch, out, workspace, workspace_bytes, static_cast<cudaStream_t>(stream));
}
int tace_set_graph_mode(TaceModel* model, int enable) {
  if (!model) return TACE_ERR_INVALID_ARGUMENT;
  model->impl->graph_mode = enable != 0;
  if (!enable) model->impl->release_graphs();
  return TACE_OK;
}
int tace_set_chunk_edges(TaceModel* model, int64_t max_edges) {
  if (!model || max_edges < 1024) return TACE_ERR_INVALID_ARGUMENT;
  model->impl->max_chunk_edges = max_edges;
  model->impl->release_graphs();
  return TACE_OK;
}
int64_t tace_graph_replays(const TaceModel* model) { return model ? model->impl->graph_replays : TACE_ERR_INVALID_ARGUMENT; }
int tace_set_exchange_sync(TaceModel* model, int host_sync) {
  if (!model || !model->impl) return TACE_ERR_INVALID_ARGUMENT;
  model->impl->exchange_sync = host_sync != 0;
  return TACE_OK;
}

int tace_set_exchange_stream(TaceModel* model, tace_stream_t stream) {
  if (!model || !model->impl) return TACE_ERR_INVALID_ARGUMENT;
  model->impl->exchange_stream = static_cast<cudaStream_t>(stream);
  return TACE_OK;
}

int tace_set_exchange(TaceModel* model, tace_exchange_fn fn, void* user) {
  if (!model) return TACE_ERR_INVALID_ARGUMENT;
  model->impl->exchange_fn = fn;
  model->impl->exchange_user = user;
  return TACE_OK;
}
int tace_device_error(TaceModel* model, int32_t* code) {
  if (!model || !code) return TACE_ERR_INVALID_ARGUMENT;
  int v = 0;
  if (cudaMemcpy(&v, model->impl->dev_error, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return TACE_ERR_CUDA;
  if (v != 0 && cudaMemset(model->impl->dev_error, 0, sizeof(int)) != cudaSuccess) return TACE_ERR_CUDA;
  *code = v;
  return TACE_OK;
}
int64_t tace_launch_count(const TaceModel* model) { return model ? model->impl->launches : TACE_ERR_INVALID_ARGUMENT; }
int tace_profile_enable(TaceModel* model, int enable) {
  if (!model) return TACE_ERR_INVALID_ARGUMENT;
  model->impl->profile = enable != 0;
  model->impl->phase_used = 0;
  return TACE_OK;
}
int tace_profile_count(const TaceModel* model) { return model ? model->impl->phase_count() : TACE_ERR_INVALID_ARGUMENT; }
int tace_profile_read(TaceModel* model, int index, const char** name, float* ms) {
  if (!model || !name || !ms) return TACE_ERR_INVALID_ARGUMENT;
  return model->impl->phase_read(index, name, ms);
}
int64_t tace_debug_read(TaceModel* model, const char* name, void* dst, int64_t numel, tace_stream_t stream) {
  if (!model || !name || !dst) return TACE_ERR_INVALID_ARGUMENT;
  return model->impl->debug_read(name, dst, numel, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
