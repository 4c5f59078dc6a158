// Planner and C ABI of the GB300 Cell step.
//
// bc_plan_create lowers every cell (bc_lower.cpp), decomposes each point tree
// into chains (maximal single-child paths), groups the chains into barrier-
// separated phases by chain level (1 + the highest level of the chains hanging
// below a chain's bottom node), packs each phase's chains into 32-lane warp slots
// (one node per lane; a chain longer than 32 nodes gets a slot of its own with a
// chunk of nodes per lane), packs cells into shared-memory tiles by best-fit-
// decreasing on node count, lays each tile out as one contiguous 16-byte-aligned
// blob and uploads it.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <numeric>
#include <queue>
#include <string>
#include <thread>
#include <vector>

#include "../../include/braincell_gb300_debug.h"
#include "bc_internal.h"
#include "bc_mech.cuh"
#include "bc_ext.cuh"

namespace bc {

static thread_local std::string g_error = "";

void set_error(const std::string& msg) { g_error = msg; }

bc_status fail(bc_status code, const std::string& msg) {
  g_error = msg;
  return code;
}

#define BC_CUDA(call)                                                                     \
  do {                                                                                    \
    cudaError_t e_ = (call);                                                              \
    if (e_ != cudaSuccess)                                                                \
      return fail(BC_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));       \
  } while (0)

static size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

struct CellSched;

}  // namespace bc

// launch classes: 0 packed shared-memory tiles, 1 one big cell per shared-memory
// tile, 2 global-memory tiles, 3 lane tiles (one small cell per thread)
constexpr int kMaxClasses = 4;
// Shared memory that a global-memory tile may take for its separators: two CTAs to an SM.
constexpr size_t kSepSmemLimit = 110 * 1024;
// Longest unbranched run that one lane eliminates in one piece (lane_nodes).
constexpr int kDefaultLaneNodes = 10;

constexpr uint32_t kMarkovBits = BC_M_NAV16 | BC_M_KCA22 | BC_M_KCA11;
constexpr uint32_t kCerebellarBits = BC_M_KV34 | BC_M_KV43 | BC_M_KV11 | BC_M_KIR23 | BC_M_HCN1F | BC_M_HCN1H |
                                     BC_M_CAHVA | BC_M_CAV23 | BC_M_CAV32;
// mechanisms outside the main mix (the extra kernel variants)
constexpr uint32_t kOutOfLineBits = BC_M_NAHH | BC_M_KHH | BC_M_KM | BC_M_KA1 | BC_M_KA2 | BC_M_KK2A | BC_M_KK2B |
                                    BC_M_KNI | kMarkovBits | kCerebellarBits | BC_M_EXT;

namespace bc {

// A region's mechanism bits, with its extension channels' BC_X_* bits (from the
// record) in the high word: the owner masks of state views and current probes.
constexpr uint64_t ext_bits(uint32_t x) { return uint64_t(x) << 32; }
static inline uint64_t region_bits(const bc_batch_spec& s, int64_t k) {
  uint64_t b = s.region_mech[k];
  if (b & BC_M_EXT)
    b |= ext_bits(uint32_t(s.region_params[k * BC_NPARAM + BC_P_EXT_MASK]) |
                  (uint32_t(s.region_params[k * BC_NPARAM + BC_P_EXT_MASK_HI]) << 24));
  return b;
}

// The mechanism bit that owns a BC_STATE_* view and the state slot holding it (V:
// in the tile blob, no slot; V_last: every node; Ci and V_last also have a low word).
static void state_view(int32_t which, uint64_t* bit, int* slot) {
  static const uint32_t kBit[BC_STATE_NAV16_C1] = {
      0,         BC_M_NA,   BC_M_NA,   BC_M_KDR,  BC_M_CAL,  BC_M_CAL,  BC_M_CAT,   BC_M_CAT,  BC_M_HCN,
      BC_M_AHP,  BC_M_CADET, BC_M_NAHH, BC_M_NAHH, BC_M_KHH, BC_M_KM,   BC_M_KA1,   BC_M_KA1,  BC_M_KA2,
      BC_M_KA2,  BC_M_KK2A, BC_M_KK2A, BC_M_KK2B, BC_M_KK2B, BC_M_KNI,  BC_M_ALL};
  static const int kSlot[BC_STATE_NAV16_C1] = {
      -1,         kSlotNaP,   kSlotNaQ,   kSlotKdrP,  kSlotCalP,  kSlotCalQ,  kSlotCatP,  kSlotCatQ,  kSlotHcnP,
      kSlotAhpP,  kSlotCaHi,  kSlotNaHHP, kSlotNaHHQ, kSlotKHHP,  kSlotKMN,   kSlotKA1P,  kSlotKA1Q,  kSlotKA2P,
      kSlotKA2Q,  kSlotKK2AP, kSlotKK2AQ, kSlotKK2BP, kSlotKK2BQ, kSlotKNIP,  kSlotVLastHi};
  if (which < BC_STATE_NAV16_C1) {
    *bit = kBit[which];
    *slot = kSlot[which];
    return;
  }
  // Markov views 25 .. 50 and the cerebellar gates 51 .. 65 sit in slots 26 .. 66
  static const uint32_t kCereb[BC_NSTATE_VIEW - BC_STATE_KV34_M] = {
      BC_M_KV34,  BC_M_KV34,  BC_M_KV43,  BC_M_KV43,  BC_M_KV11,  BC_M_KIR23, BC_M_HCN1F, BC_M_HCN1F,
      BC_M_HCN1H, BC_M_CAHVA, BC_M_CAHVA, BC_M_CAV23, BC_M_CAV23, BC_M_CAV32, BC_M_CAV32};
  // extension channels' states 66 .. 121 in slots 67 .. 122
  static const uint32_t kExt[BC_NSTATE_VIEW - BC_STATE_HCN2_FAST] = {
      BC_X_HCN2, BC_X_HCN2, BC_X_KV33, BC_X_KV22,  BC_X_KV22,  BC_X_KV15,  BC_X_KV15,
      BC_X_KV15, BC_X_NAF,  BC_X_NAF,  BC_X_NAP,   BC_X_NAP,   BC_X_NAIO,  BC_X_NAIO,
      BC_X_FKDR, BC_X_SKDR, BC_X_KDRIO, BC_X_HCNDCN, BC_X_HCNIO, BC_X_CATHP, BC_X_CATHP,
      BC_X_CAHTRE, BC_X_CAHTRE, BC_X_CALDCN, BC_X_CALDCN, BC_X_KCA31, BC_X_SKDCN, BC_X_KKV,
      BC_X_CAN, BC_X_CAIO, BC_X_NAVGRC, BC_X_NAVGRC, BC_X_NAVGRC, BC_X_NAVGRC, BC_X_NAVGRC, BC_X_NAVGRC,
      BC_X_NAVGRC, BC_X_NAVGRC, BC_X_NAVGRC, BC_X_NAVGRC, BC_X_NAVGRC, BC_X_NAVGRC, BC_X_CAV31, BC_X_CAV31,
      BC_X_CAV33, BC_X_CAV33, BC_X_CAV12, BC_X_CAV12, BC_X_CAV12, BC_X_CAV13, BC_X_CAV13, BC_X_CAV13,
      BC_X_CAV21, BC_X_CAHVADCN, BC_X_CALVADCN, BC_X_CALVADCN};
  if (which >= BC_STATE_HCN2_FAST)
    *bit = ext_bits(kExt[which - BC_STATE_HCN2_FAST]);
  else if (which >= BC_STATE_KV34_M)
    *bit = kCereb[which - BC_STATE_KV34_M];
  else
    *bit = which < BC_STATE_KCA22_C2 ? BC_M_NAV16 : (which < BC_STATE_KCA11_C1 ? BC_M_KCA22 : BC_M_KCA11);
  *slot = which + 1;
}

}  // namespace bc

struct LaunchClass {
  int first = 0, count = 0, threads = 256;
  bool smem = true;
  bool lane = false;  // lane tiles: one cell per thread (lane_step_kernel)
  int cluster = 1;  // CTAs per tile (global-memory tiles)
  size_t smem_bytes = 0;
};

struct bc_plan {
  std::vector<LaunchClass> classes;
  int precision = BC_PREC_F32;
  int device = 0;
  int threads = 128;
  int threads_global = 512;
  int tile_nodes = 0;
  int lane_nodes = 1;
  int steps_per_launch = 1000;
  int record_every = 1;
  int max_spikes = 64;
  int use_graph = 0;
  bool extra = false;  // synapses, a network, mechanism probes, or a region using the out-of-line mechanism set
  int state_slots = 1;
  int64_t n_cells = 0, n_cv = 0, n_nodes = 0, n_probes = 0, n_pulses = 0;
  int64_t max_phases = 0, max_chain_nodes = 0;
  size_t real_size = 4;
  std::vector<bc::TileDesc> tiles;  // smem tiles first, then global tiles
  int n_smem_tiles = 0;
  size_t smem_bytes = 0;
  std::vector<int64_t> cell_ncv;
  // (tile, node) of every CV, and room for one view's values; a call holds the mutex until
  // its values have left the device, as several threads may read one plan
  int2* d_cv = nullptr;
  double* d_view = nullptr;
  std::mutex view_mu;
  std::vector<bc::PulseRec> pulses;
  std::vector<int64_t> pulse_src;   // spec pulse id of each record (records are in tile / node order)
  std::vector<double> pulse_scale;  // record amp per nA
  std::vector<double> pulse_amp;    // bc_pulse_set_amp's last amplitudes (nA); the host records follow when next used
  int32_t* d_pulse_src = nullptr;
  double* d_pulse_scale = nullptr;
  double* d_pulse_amp = nullptr;
  double pulses_dt = -1.0;
  std::vector<double> probe_vrest;
  // synapses and connections (host copies; device mirrors below)
  int64_t n_synapses = 0, n_connections = 0;
  std::vector<double> syn_tau, syn_e, syn_scale, conn_delay;
  std::vector<int64_t> out_ptr, out_syn, out_order;  // CSR of connections by presynaptic cell
  std::vector<double> out_w;
  void* d_syn_g = nullptr;
  void* d_syn_tau = nullptr;
  void* d_syn_e = nullptr;
  void* d_syn_scale = nullptr;
  int64_t* d_out_ptr = nullptr;
  int64_t* d_out_syn = nullptr;
  void* d_out_w = nullptr;
  int32_t* d_out_d = nullptr;
  void* d_arrivals = nullptr;
  int64_t arr_slots = 0, net_k = 0;
  double net_dt = 0.0;  // dt the delays were quantised for (0: not yet)
  int32_t* d_rec_cell = nullptr;
  int64_t* d_rec_step = nullptr;
  unsigned long long* d_rec_count = nullptr;  // [0] produced, [1] delivered
  int64_t rec_cap = 0;
  // subtree-surrogate ports: records (tile order), stimulus pulses (nA), GRU
  int64_t n_ports = 0;
  std::vector<bc::PortRec> ports;
  std::vector<bc::PulseRec> port_pulses;
  double port_pulses_dt = -1.0;
  bc::PortRec* d_ports = nullptr;
  bc::PulseRec* d_port_pulses = nullptr;
  float* d_port_h = nullptr;
  int32_t* d_port_flags = nullptr;
  bc::GruWeights* d_gru = nullptr;
  bool gru_set = false;
  // device buffers
  unsigned char* d_blob = nullptr;
  size_t blob_bytes = 0;
  unsigned char* d_scratch = nullptr;
  size_t scratch_bytes = 0;
  unsigned char* d_state = nullptr;
  size_t state_bytes = 0;
  bc::TileDesc* d_tiles = nullptr;
  bc::PulseRec* d_pulses = nullptr;
  double* d_vinit = nullptr;
  int64_t* d_vinit_off = nullptr;
  double* d_traces = nullptr;
  int64_t trace_cap = 0;
  int64_t trace_origin = 0;
  int32_t* d_spike_count = nullptr;
  double* d_spike_times = nullptr;
  int32_t* d_status = nullptr;
  int64_t step = 0;
  size_t device_bytes = 0;
  // launch classes after the first run concurrently on these streams
  cudaStream_t aux[kMaxClasses - 1] = {nullptr, nullptr, nullptr};
  cudaStream_t init_stream = nullptr;  // highest priority: the initial reset
  int aux_prio = 0;                    // priority of the aux streams (that of the last caller's stream)
  bool dry = false;
  unsigned long long* d_timers = nullptr;
  std::vector<std::array<int64_t, 6>> tile_stats;
  cudaEvent_t ev_fork = nullptr, ev_join[kMaxClasses - 1] = {nullptr, nullptr, nullptr};
  // CUDA graph of one run (use_graph): per launch class a chain of kernel nodes,
  // rebuilt when the launch pattern changes, otherwise only re-parameterised.
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t graph_exec = nullptr;
  std::vector<cudaGraphNode_t> graph_nodes;  // [launch][class]
  int64_t graph_launches = -1;
  int32_t graph_k = -1, graph_k_last = -1;
};

namespace bc {

template <typename T>
static bc_status dalloc(bc_plan* p, T** ptr, size_t count) {
  *ptr = nullptr;
  if (count == 0) count = 1;
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(ptr), count * sizeof(T));
  if (e != cudaSuccess) return fail(BC_ERR_CUDA, std::string("cudaMalloc: ") + cudaGetErrorString(e));
  p->device_bytes += count * sizeof(T);
  return BC_OK;
}

static void free_plan(bc_plan* p) {
  cudaFree(p->d_blob);
  cudaFree(p->d_scratch);
  cudaFree(p->d_state);
  cudaFree(p->d_tiles);
  cudaFree(p->d_pulses);
  cudaFree(p->d_pulse_src);
  cudaFree(p->d_pulse_scale);
  cudaFree(p->d_pulse_amp);
  cudaFree(p->d_cv);
  cudaFree(p->d_view);
  cudaFree(p->d_vinit);
  cudaFree(p->d_vinit_off);
  cudaFree(p->d_traces);
  cudaFree(p->d_spike_count);
  cudaFree(p->d_spike_times);
  cudaFree(p->d_status);
  cudaFree(p->d_timers);
  cudaFree(p->d_syn_g);
  cudaFree(p->d_syn_tau);
  cudaFree(p->d_syn_e);
  cudaFree(p->d_syn_scale);
  cudaFree(p->d_out_ptr);
  cudaFree(p->d_out_syn);
  cudaFree(p->d_out_w);
  cudaFree(p->d_out_d);
  cudaFree(p->d_arrivals);
  cudaFree(p->d_rec_cell);
  cudaFree(p->d_rec_step);
  cudaFree(p->d_rec_count);
  cudaFree(p->d_ports);
  cudaFree(p->d_port_pulses);
  cudaFree(p->d_port_h);
  cudaFree(p->d_port_flags);
  cudaFree(p->d_gru);
  for (int k = 0; k < kMaxClasses - 1; ++k) {
    if (p->aux[k]) cudaStreamDestroy(p->aux[k]);
    if (p->ev_join[k]) cudaEventDestroy(p->ev_join[k]);
  }
  if (p->init_stream) cudaStreamDestroy(p->init_stream);
  if (p->ev_fork) cudaEventDestroy(p->ev_fork);
  if (p->graph_exec) cudaGraphExecDestroy(p->graph_exec);
  if (p->graph) cudaGraphDestroy(p->graph);
  delete p;
}

// ------------------------------------------------------------------ chain schedule
// A cell's tree cut into segments at its separators (see SegRec).
struct Seg {
  std::vector<int32_t> nodes;  // bottom -> top (cell-local node ids), may be empty between two separators
  int32_t s = -1, t = -1;      // lower (-1: leaf) / upper separator of the cell
};
struct Sep {
  int32_t node = -1;
  int32_t t = -1;              // upper separator, -1 at the root
  int32_t level = 0;           // 1 + the highest level of the separators below
  std::vector<int32_t> in;     // segments whose upper separator this is
};
struct CellSched {
  std::vector<Seg> segs;
  std::vector<Sep> seps;
  // lowered root .. tree root of the solve; the edges along it are turned around
  std::vector<int32_t> path;
  int32_t n_levels = 0;
  // a cell solved whole (no segments or separators): its nodes in the order of elimination
  std::vector<int32_t> order;
};

// fn(i) for i in [0, n) on up to BC_PLAN_THREADS host threads (default: the
// hardware threads, at most 32), in chunks of 64 items; one thread when n is
// small.  fn must touch only item i's outputs and must not throw.  When a
// worker thread cannot be started, the threads already running (and the
// calling thread) take its share: the items are claimed from one counter.
template <class F>
static void parallel_for(int64_t n, F&& fn) {
  int64_t nt = int64_t(std::thread::hardware_concurrency());
  if (const char* e = std::getenv("BC_PLAN_THREADS")) nt = std::atoll(e);
  nt = std::max<int64_t>(1, std::min<int64_t>({nt, 32, (n + 63) / 64}));
  if (nt <= 1) {
    for (int64_t i = 0; i < n; ++i) fn(i);
    return;
  }
  std::atomic<int64_t> next{0};
  auto work = [&]() {
    for (;;) {
      const int64_t i0 = next.fetch_add(64);
      if (i0 >= n) return;
      for (int64_t i = i0; i < std::min<int64_t>(n, i0 + 64); ++i) fn(i);
    }
  };
  std::vector<std::thread> pool;
  try {
    pool.reserve(size_t(nt - 1));
    for (int64_t t = 1; t < nt; ++t) pool.emplace_back(work);
  } catch (const std::exception&) {
    // std::system_error (no thread) or bad_alloc: carry on with what started
  }
  work();
  for (auto& th : pool) th.join();
}

// Elimination order of a cell solved whole: runs bottom -> top, the runs below a
// branch point before it, in the order of their bottom nodes.
static void order_whole(const LoweredCell& lc, CellSched& cs) {
  const int32_t n = lc.n_node;
  std::vector<std::vector<int32_t>> kids(n);
  int32_t root = 0;
  for (int32_t i = 0; i < n; ++i) {
    if (lc.parent[i] < 0)
      root = i;
    else
      kids[lc.parent[i]].push_back(i);
  }
  auto bottom = [&](int32_t v) {
    while (kids[v].size() == 1) v = kids[v][0];
    return v;
  };
  std::vector<std::pair<int32_t, bool>> todo{{root, false}};  // (top of a run, its branches done)
  while (!todo.empty()) {
    const auto [top, done] = todo.back();
    todo.pop_back();
    const int32_t b = bottom(top);
    if (!done) {
      todo.push_back({top, true});
      std::vector<int32_t> below = kids[b];
      std::sort(below.begin(), below.end(), [&](int32_t x, int32_t y) { return bottom(x) > bottom(y); });
      for (const int32_t k : below) todo.push_back({k, false});
    } else {
      for (int32_t v = b; v != top; v = lc.parent[v]) cs.order.push_back(v);
      cs.order.push_back(top);
    }
  }
}

// Levels of the separators, children before parents.
static void set_levels(CellSched& cs) {
  const int32_t ns = int32_t(cs.seps.size());
  std::vector<int32_t> waits(ns, 0), ready;
  for (Sep& sp : cs.seps) {
    sp.level = 0;
    if (sp.t >= 0) waits[sp.t]++;
  }
  for (int32_t j = 0; j < ns; ++j)
    if (waits[j] == 0) ready.push_back(j);
  cs.n_levels = 0;
  for (size_t k = 0; k < ready.size(); ++k) {
    const Sep& sp = cs.seps[ready[k]];
    cs.n_levels = std::max(cs.n_levels, sp.level + 1);
    if (sp.t < 0) continue;
    cs.seps[sp.t].level = std::max(cs.seps[sp.t].level, sp.level + 1);
    if (--waits[sp.t] == 0) ready.push_back(sp.t);
  }
}

// Segments and separators of one cell.  Runs of more than lane_nodes nodes are cut.  A
// lane's walk costs about 100 cycles a node, all runs at once; a further separator on a
// run costs about 400 on every path through it, so with d branch levels a run of L nodes
// is best cut into sqrt(L / (4 d)) pieces: long unbranched cells are cut, the 50-node
// branches of a 20-level tree are not (256 such cells x 100 steps: 33.3 ms with every run
// cut into sqrt(L / 3.2) pieces).  The cuts depend on the cell alone, so its
// results do not depend on its tile mates or on the launch shape.
static void decompose(const LoweredCell& lc, int lane_nodes, CellSched& cs) {
  const int32_t n = lc.n_node;
  if (n <= kCellLaneNodes) {
    order_whole(lc, cs);
    return;
  }
  std::vector<std::array<int32_t, 2>> kid(n, {-1, -1});
  std::vector<int32_t> nchild(n, 0), parent(lc.parent);
  int32_t root = 0;
  for (int32_t i = 0; i < n; ++i) {
    const int32_t p = lc.parent[i];
    if (p < 0)
      root = i;
    else if (nchild[p]++ == 0)
      kid[p][0] = i;
  }
  // the root of the solve: the first branch point below the lowered root, or the
  // middle of a tree without one
  cs.path.assign(1, root);
  for (int32_t v = root; nchild[v] == 1;) {
    v = kid[v][0];
    cs.path.push_back(v);
  }
  if (nchild[cs.path.back()] == 0) cs.path.resize(cs.path.size() / 2 + 1);
  for (size_t k = 0; k + 1 < cs.path.size(); ++k) {  // turn the edges of the path around
    parent[cs.path[k]] = cs.path[k + 1];
    --nchild[cs.path[k]];
    ++nchild[cs.path[k + 1]];
  }
  root = cs.path.back();
  parent[root] = -1;
  std::vector<int32_t> sep_of(n, -1), start;
  auto add_sep = [&](int32_t v) {
    sep_of[v] = int32_t(cs.seps.size());
    cs.seps.emplace_back();
    cs.seps.back().node = v;
  };
  for (int32_t v = 0; v < n; ++v) {
    if (v == root || nchild[v] >= 2) add_sep(v);
    if (v != root && nchild[v] != 1) start.push_back(v);
  }
  // separators are indexed by 16 bits in a tile: cut less where a cell has very many
  const int64_t room = std::max<int64_t>(0, 60000 - int64_t(cs.seps.size()));
  const int64_t most_per_run = std::max<int64_t>(1, 1 + room / std::max<int64_t>(1, int64_t(start.size())));
  const int64_t whole = std::min(std::max(lane_nodes, 1), 4096);
  // the run from a leaf (itself the bottom node) or above a separator, up to the next separator
  struct Run {
    int32_t lower, upper;
    std::vector<int32_t> nodes;
  };
  std::vector<Run> runs(start.size());
  for (size_t k = 0; k < start.size(); ++k) {
    const int32_t v0 = start[k];
    runs[k].lower = sep_of[v0];
    int32_t v = runs[k].lower >= 0 ? parent[v0] : v0;
    for (; sep_of[v] < 0; v = parent[v]) runs[k].nodes.push_back(v);
    runs[k].upper = sep_of[v];
    if (runs[k].lower >= 0) cs.seps[runs[k].lower].t = runs[k].upper;
  }
  set_levels(cs);
  const double d = std::max(1, cs.n_levels);
  for (const Run& run : runs) {
    int32_t lower = run.lower;
    const int64_t L = int64_t(run.nodes.size());
    int64_t pieces = 1;
    if (L > whole) pieces = std::llround(std::sqrt(double(L) / (4.0 * d)));
    pieces = std::max<int64_t>(1, std::min({pieces, most_per_run, (L + 1) / 2}));
    int64_t k0 = 0;
    for (int64_t q = 0; q < pieces; ++q) {
      // pieces - 1 of the L nodes become separators; the others are shared out evenly
      const int64_t k1 = k0 + (L - (pieces - 1)) * (q + 1) / pieces - (L - (pieces - 1)) * q / pieces;
      Seg sg;
      sg.nodes.assign(run.nodes.begin() + k0, run.nodes.begin() + k1);
      sg.s = lower;
      if (q + 1 < pieces) {
        add_sep(run.nodes[k1]);
        sg.t = sep_of[run.nodes[k1]];
      } else {
        sg.t = run.upper;
      }
      if (sg.s >= 0) cs.seps[sg.s].t = sg.t;
      lower = sg.t;
      cs.segs.push_back(std::move(sg));
      k0 = k1 + 1;
    }
  }
  for (size_t k = 0; k < cs.segs.size(); ++k) cs.seps[cs.segs[k].t].in.push_back(int32_t(k));
  set_levels(cs);
}

// ------------------------------------------------------------------ tile building
struct TileBuild {
  std::vector<int64_t> cells;  // global cell ids
  int cls = 0;                 // launch class
};

struct TileOut {
  TileDesc desc{};
  std::vector<unsigned char> blob;
  std::vector<double> vinit;
  std::vector<PulseRec> pulses;
  std::vector<int64_t> pulse_src;     // spec pulse id of each pulse record
  std::vector<double> pulse_scale;    // record amp per nA of the spec pulse
  std::vector<PortRec> ports;         // stim_begin / stim_end relative to port_pulses
  std::vector<PulseRec> port_pulses;  // amp in nA
  std::vector<std::pair<int64_t, int32_t>> cv_local;  // (global cv id, local node)
  int64_t crit = 0;
};

struct BuildCtx {
  const bc_batch_spec* spec;
  const std::vector<LoweredCell>* cells;
  const std::vector<CellSched>* sched;
  const std::vector<int64_t>* cv_base;  // global cv id of each cell's first CV
  const std::vector<std::vector<int64_t>>* cell_pulses;
  const std::vector<std::vector<int64_t>>* cell_probes;
  const std::vector<std::vector<int32_t>>* pulse_node;  // per cell, node per pulse (parallel to cell_pulses)
  const std::vector<std::vector<int32_t>>* probe_node;
  const std::vector<std::vector<std::pair<int64_t, int32_t>>>* cell_syns;  // per cell: (synapse id, node)
  const std::vector<char>* is_src;                                        // per cell: source of a connection
  // per cell: (port id, endpoint node, attachment CV node); port pulses by port
  const std::vector<std::vector<std::array<int32_t, 3>>>* cell_ports;
  const std::vector<std::vector<int64_t>>* port_pulse_ids;
  int precision;
  int state_slots;
  int param_stride;       // reals per parameter record in the tile blobs
};

template <typename Real>
static void put(std::vector<unsigned char>& b, size_t off, size_t idx, Real v) {
  std::memcpy(b.data() + off + idx * sizeof(Real), &v, sizeof(Real));
}

static bc_status build_tile(const BuildCtx& cx, const TileBuild& tb, int T, TileOut& out) {
  const bc_batch_spec& s = *cx.spec;
  const int R = s.n_regions;
  const size_t rs = cx.precision == BC_PREC_F64 ? 8 : 4;
  const std::vector<int64_t>& cell_list = tb.cells;
  int64_t n_real = 0;
  std::vector<std::vector<int32_t>> node_tile(cell_list.size());
  for (size_t li = 0; li < cell_list.size(); ++li) {
    const LoweredCell& lc = (*cx.cells)[cell_list[li]];
    node_tile[li].assign(lc.n_node, -1);
    n_real += lc.n_node;
  }
  const int W = std::max(1, T / 32);
  const bool lane = tb.cls == 3;  // a lane tile has no segments, separators or warp slots
  auto sched_of = [&](size_t li) -> const CellSched& { return (*cx.sched)[cell_list[li]]; };
  std::vector<SegRec> segs;
  std::vector<SlotRec> slots;
  std::vector<SepRec> seps;
  std::vector<GroupRec> groups;
  std::vector<int32_t> levels;
  std::vector<uint32_t> link;
  std::vector<int32_t> rows;  // row starts of the slots
  int32_t next_node = 0, cell0 = 0, sep0 = 0, n_inbox = 0;
  int n_levels = 0;
  int64_t crit = 0, n_lower = 0;  // nodes of segments with a lower separator (they come first)
  if (!lane) {
    // -------- separators: cells dealt to the warps (longest sweep first, to the warp with the least), then
    // a tile index per separator by warp, level and cell
    struct Cost {
      int64_t cost;
      size_t li;
    };
    std::vector<Cost> by_cost;
    size_t n_sep = 0;
    std::vector<size_t> whole;  // cells of one lane each
    for (size_t li = 0; li < cell_list.size(); ++li) {
      if (!sched_of(li).order.empty()) {
        whole.push_back(li);
        continue;
      }
      by_cost.push_back({int64_t(sched_of(li).n_levels) + int64_t(sched_of(li).seps.size()) / 32, li});
      n_sep += sched_of(li).seps.size();
    }
    if (n_sep >= kLinkCell) return fail(BC_ERR_CAPACITY, "too many branch points in one tile");
    std::stable_sort(by_cost.begin(), by_cost.end(), [](const Cost& a, const Cost& b) { return a.cost > b.cost; });
    const size_t n_groups = std::min(by_cost.size(), size_t(W));
    std::vector<std::vector<size_t>> members(n_groups);
    std::vector<int64_t> group_seps(n_groups, 0);
    for (size_t k = 0; k < by_cost.size(); ++k) {
      const size_t g = k < n_groups ? k
                                    : size_t(std::min_element(group_seps.begin(), group_seps.end()) - group_seps.begin());
      members[g].push_back(by_cost[k].li);
      group_seps[g] += int64_t(sched_of(by_cost[k].li).seps.size());
    }
    std::vector<std::vector<int32_t>> sep_tile(cell_list.size());
    for (size_t li = 0; li < cell_list.size(); ++li) sep_tile[li].resize(sched_of(li).seps.size());
    std::vector<std::pair<size_t, int32_t>> sep_src;  // (cell of the tile, separator of the cell) by tile index
    for (auto& m : members) {
      std::vector<std::vector<std::pair<size_t, int32_t>>> lv;
      for (const size_t li : m) {
        const CellSched& cs = sched_of(li);
        if (lv.size() < size_t(cs.n_levels)) lv.resize(cs.n_levels);
        for (size_t j = 0; j < cs.seps.size(); ++j) lv[cs.seps[j].level].push_back({li, int32_t(j)});
      }
      GroupRec gr{int32_t(levels.size()), 0};
      n_levels = std::max(n_levels, int(lv.size()));
      for (auto& v : lv)
        for (size_t k = 0; k < v.size(); ++k) {
          const auto& x = v[k];
          if (k % 32 == 0) {
            levels.push_back(int32_t(sep_src.size()));
            ++gr.n_chunks;
          }
          if (sched_of(x.first).seps[x.second].in.size() > 4) levels.back() |= int32_t(kChunkMore);
          sep_tile[x.first][x.second] = int32_t(sep_src.size());
          sep_src.push_back(x);
        }
      levels.push_back(int32_t(sep_src.size()));
      groups.push_back(gr);
    }
    // -------- inboxes: one entry per segment, consecutive per upper separator, padded to two or more pairs
    std::vector<std::vector<int32_t>> seg_inbox(cell_list.size());
    for (size_t li = 0; li < cell_list.size(); ++li) seg_inbox[li].resize(sched_of(li).segs.size());
    seps.resize(sep_src.size());
    for (size_t j = 0; j < sep_src.size(); ++j) {
      const auto [li, q] = sep_src[j];
      const Sep& sp = sched_of(li).seps[q];
      const size_t pairs = std::max<size_t>(2, (sp.in.size() + 1) / 2);
      if (pairs > 0xFFFF) return fail(BC_ERR_CAPACITY, "too many branches at one point");
      seps[j] = SepRec{n_inbox / 2, -1, uint16_t(pairs), uint16_t(sp.t >= 0 ? size_t(sep_tile[li][sp.t]) : j), 0};
      for (size_t k = 0; k < sp.in.size(); ++k) seg_inbox[li][sp.in[k]] = n_inbox + int32_t(k);
      n_inbox += int32_t(2 * pairs);
    }
    for (size_t li = 0; li < cell_list.size(); ++li)
      for (size_t k = 0; k < sched_of(li).segs.size(); ++k) {
        const Seg& sg = sched_of(li).segs[k];
        if (sg.s >= 0) seps[sep_tile[li][sg.s]].inbox = seg_inbox[li][k];
      }
    for (SepRec& sp : seps)
      if (sp.inbox < 0) sp.inbox = n_inbox++;
    // the end of a slot's rows, and what the kernel's reads of four rows at a time may touch past it
    auto end_rows = [&]() {
      rows.push_back(next_node);
      while (rows.size() % 4 != 0) rows.push_back(next_node);
      rows.insert(rows.end(), 4, next_node);
    };
    // -------- warp slots: segments with a lower separator first, then the leaves', longest first
    std::vector<std::pair<size_t, int32_t>> seg_src;
    for (int lower = 1; lower >= 0; --lower) {
      std::vector<std::pair<size_t, int32_t>> v;
      for (size_t li = 0; li < cell_list.size(); ++li)
        for (size_t k = 0; k < sched_of(li).segs.size(); ++k)
          if ((sched_of(li).segs[k].s >= 0) == (lower == 1)) v.push_back({li, int32_t(k)});
      // the roots' segments to themselves (k = -1)
      for (const Cost& c : by_cost)
        if (lower == 1) v.push_back({c.li, -1});
      auto len = [&](const std::pair<size_t, int32_t>& x) {
        return x.second < 0 ? size_t(0) : sched_of(x.first).segs[x.second].nodes.size();
      };
      std::stable_sort(v.begin(), v.end(), [&](const auto& x, const auto& y) { return len(x) > len(y); });
      for (size_t q = 0; q < v.size(); q += 32) {
        const size_t n_lanes = std::min<size_t>(32, v.size() - q);
        SlotRec sr{int32_t(rows.size()), int32_t(segs.size()), int16_t(n_lanes), uint16_t(len(v[q])), lower ? kSlotLower : kSlotLeaf};
        for (size_t l = 0; l < n_lanes; ++l) {
          const auto& st = sep_tile[v[q + l].first];
          if (v[q + l].second < 0) {
            const CellSched& cs = sched_of(v[q + l].first);
            const size_t r = size_t(std::find_if(cs.seps.begin(), cs.seps.end(), [](const Sep& x) { return x.t < 0; }) -
                                    cs.seps.begin());
            segs.push_back(SegRec{uint16_t(st[r]), uint16_t(st[r]), 0, 0, 0, 0});
            continue;
          }
          const Seg& sg = sched_of(v[q + l].first).segs[v[q + l].second];
          if (sg.nodes.size() > 0xFFFF) return fail(BC_ERR_CAPACITY, "an unbranched run holds too many nodes");
          segs.push_back(SegRec{uint16_t(st[sg.t]), uint16_t(sg.s >= 0 ? uint32_t(st[sg.s]) : kLinkNone),
                                uint16_t(sg.nodes.size()), 0, seg_inbox[v[q + l].first][v[q + l].second], 0});
        }
        for (size_t k = 0; k < sr.max_len; ++k) {
          rows.push_back(next_node);
          for (size_t l = 0; l < n_lanes && len(v[q + l]) > k; ++l) {
            const Seg& sg = sched_of(v[q + l].first).segs[v[q + l].second];
            node_tile[v[q + l].first][sg.nodes[k]] = next_node++;
            const SegRec& rec = segs[sr.seg0 + l];
            link.push_back(uint32_t(rec.t) | (uint32_t(rec.s) << 16));
          }
        }
        end_rows();
        slots.push_back(sr);
      }
      if (lower == 1) n_lower = next_node;
    }
    // -------- whole cells, largest first
    cell0 = next_node;
    std::stable_sort(whole.begin(), whole.end(),
                     [&](size_t x, size_t y) { return sched_of(x).order.size() > sched_of(y).order.size(); });
    for (size_t q = 0; q < whole.size(); q += 32) {
      const size_t n_lanes = std::min<size_t>(32, whole.size() - q);
      const size_t max_len = sched_of(whole[q]).order.size();
      slots.push_back(SlotRec{int32_t(rows.size()), 0, int16_t(n_lanes), uint16_t(max_len), kSlotCell});
      for (size_t k = 0; k < max_len; ++k) {
        rows.push_back(next_node);
        for (size_t l = 0; l < n_lanes && sched_of(whole[q + l]).order.size() > k; ++l) {
          const LoweredCell& lc = (*cx.cells)[cell_list[whole[q + l]]];
          const std::vector<int32_t>& ord = sched_of(whole[q + l]).order;
          const int32_t p = lc.parent[ord[k]];
          uint32_t lk = kLinkNoParent;
          if (p >= 0) {
            lk = uint32_t(std::find(ord.begin(), ord.end(), p) - ord.begin());
            if (std::count(lc.parent.begin(), lc.parent.end(), p) == 1) lk |= kLinkOnlyChild;
          }
          link.push_back(lk | (kLinkCell << 16));
          node_tile[whole[q + l]][ord[k]] = next_node++;
        }
      }
      end_rows();
    }
    // warp w takes slots w, w + W, ...: the dearest first
    std::stable_sort(slots.begin(), slots.end(), [](const SlotRec& a, const SlotRec& b) {
      return int(a.max_len) + 2 * a.kind > int(b.max_len) + 2 * b.kind;
    });
    sep0 = next_node;
    for (size_t j = 0; j < sep_src.size(); ++j) {
      node_tile[sep_src[j].first][sched_of(sep_src[j].first).seps[sep_src[j].second].node] = next_node++;
      link.push_back(uint32_t(j) | (kLinkSelf << 16));
    }
    // relative length of a step (it orders tiles): the walks of the dearest warp, the sweep, the update
    std::vector<int64_t> warp_cost(W, 0);
    for (size_t k = 0; k < slots.size(); ++k) warp_cost[k % W] += slots[k].max_len;
    crit = *std::max_element(warp_cost.begin(), warp_cost.end()) + 4 * n_levels + n_real / 32;
  }
  out.crit = crit;
  // lane tile: node v of the cell in lane l is tile node v * T + l
  std::vector<int32_t> lane_n;
  int32_t lane_kmax = 0;
  if (lane) {
    if (int64_t(cell_list.size()) > T) return fail(BC_ERR_INVALID, "internal: lane tile with more cells than threads");
    lane_n.assign(size_t(T), 0);
    for (size_t li = 0; li < cell_list.size(); ++li) {
      const LoweredCell& lc = (*cx.cells)[cell_list[li]];
      lane_n[li] = lc.n_node;
      lane_kmax = std::max(lane_kmax, lc.n_node);
      for (int32_t v = 0; v < lc.n_node; ++v) node_tile[li][v] = v * T + int32_t(li);
    }
    if (lane_kmax >= 0xFFFF) return fail(BC_ERR_CAPACITY, "a lane-tile cell has too many nodes");
    n_real = int64_t(lane_kmax) * T;
    out.crit = lane_kmax;
  }
  if (lane) cell0 = sep0 = int32_t(n_real);  // rows in the excess form
  // -------- nodes with heavy mechanisms, ordered by their mechanisms, so that the lanes of a warp share them
  std::vector<int32_t> heavy;
  if (!lane) {
    std::vector<std::pair<uint32_t, int32_t>> v;
    for (size_t li = 0; li < cell_list.size(); ++li) {
      const LoweredCell& lc = (*cx.cells)[cell_list[li]];
      for (int32_t n = 0; n < lc.n_node; ++n) {
        const uint32_t m = lc.region[n] >= 0 ? s.region_mech[cell_list[li] * R + lc.region[n]] : 0u;
        if (m & (BC_M_NA | BC_M_KDR | kOutOfLineBits)) v.push_back({m, node_tile[li][n]});
      }
    }
    std::sort(v.begin(), v.end());
    for (const auto& x : v) heavy.push_back(x.second);
  }
  std::vector<uint16_t> crec;
  if (lane) {  // lane tiles: the parent's node index v within the cell (0xFFFF at the root)
    crec.assign(size_t(n_real), 0);
    for (size_t li = 0; li < cell_list.size(); ++li) {
      const LoweredCell& lc = (*cx.cells)[cell_list[li]];
      for (int32_t v = 0; v < lc.n_node; ++v)
        crec[size_t(node_tile[li][v])] = lc.parent[v] >= 0 ? uint16_t(lc.parent[v]) : uint16_t(0xFFFF);
    }
  }
  // -------- special nodes: clamp pulses (sorted by node) and probes
  std::vector<std::pair<int32_t, int64_t>> tpulse, tprobe;  // (tile node, pulse / probe id)
  for (size_t li = 0; li < cell_list.size(); ++li) {
    const int64_t c = cell_list[li];
    const auto& pl = (*cx.cell_pulses)[c];
    const auto& pn = (*cx.pulse_node)[c];
    for (size_t k = 0; k < pl.size(); ++k) tpulse.push_back({node_tile[li][pn[k]], pl[k]});
    const auto& ql = (*cx.cell_probes)[c];
    const auto& qn = (*cx.probe_node)[c];
    for (size_t k = 0; k < ql.size(); ++k) tprobe.push_back({node_tile[li][qn[k]], ql[k]});
  }
  std::vector<std::pair<int32_t, int64_t>> tsyn;  // (tile node, synapse id)
  bool has_src = false;
  for (size_t li = 0; li < cell_list.size(); ++li) {
    const int64_t c = cell_list[li];
    for (const auto& sv : (*cx.cell_syns)[c]) tsyn.push_back({node_tile[li][sv.second], sv.first});
    has_src = has_src || (*cx.is_src)[c];
  }
  std::stable_sort(tsyn.begin(), tsyn.end(),
                   [](const std::pair<int32_t, int64_t>& x, const std::pair<int32_t, int64_t>& y) { return x.first < y.first; });
  std::stable_sort(tpulse.begin(), tpulse.end(),
                   [](const std::pair<int32_t, int64_t>& x, const std::pair<int32_t, int64_t>& y) { return x.first < y.first; });
  std::sort(tprobe.begin(), tprobe.end());
  std::vector<int32_t> spec_nodes;
  for (auto& x : tpulse) spec_nodes.push_back(x.first);
  for (auto& x : tprobe) spec_nodes.push_back(x.first);
  for (auto& x : tsyn) spec_nodes.push_back(x.first);
  std::sort(spec_nodes.begin(), spec_nodes.end());
  spec_nodes.erase(std::unique(spec_nodes.begin(), spec_nodes.end()), spec_nodes.end());
  if (spec_nodes.size() >= 0xFFFF) return fail(BC_ERR_CAPACITY, "too many clamped / probed / synapse points in one tile");
  if (cell_list.size() >= 0xFFFF) return fail(BC_ERR_CAPACITY, "too many cells in one tile");
  // -------- layout
  const int64_t N = (n_real + 3) & ~int64_t(3);
  const int64_t n_params = int64_t(cell_list.size()) * R;
  if (n_params >= 0xFFFF) return fail(BC_ERR_CAPACITY, "too many parameter records in one tile");
  TileDesc d{};
  d.param_stride = cx.param_stride;
  size_t off = 0;
  d.off_v = int32_t(off);
  off = align16(off + 2 * N * rs);
  d.dyn_bytes = int32_t(off);
  d.off_ab = int32_t(off);
  off = align16(off + 2 * N * rs);
  d.off_pidx = int32_t(off);
  off = align16(off + N * 2);
  d.off_spec = int32_t(off);
  off = align16(off + N * 2);
  d.off_specs = int32_t(off);
  off = align16(off + spec_nodes.size() * sizeof(SpecRec));
  d.off_link = int32_t(off);
  off = align16(off + link.size() * 4);
  d.off_segs = int32_t(off);
  off = align16(off + segs.size() * sizeof(SegRec));
  d.off_slots = int32_t(off);
  off = align16(off + slots.size() * sizeof(SlotRec));
  d.off_seps = int32_t(off);
  off = align16(off + seps.size() * sizeof(SepRec));
  d.off_levels = int32_t(off);
  off = align16(off + levels.size() * 4);
  d.off_groups = int32_t(off);
  off = align16(off + groups.size() * sizeof(GroupRec));
  d.off_rows = int32_t(off);
  off = align16(off + rows.size() * 4);
  d.off_diag0 = int32_t(off);
  off = align16(off + size_t(sep0 - cell0) * rs);
  d.off_heavy = int32_t(off);
  off = align16(off + heavy.size() * 4);
  d.off_crec = int32_t(off);
  off = align16(off + crec.size() * 2);
  d.off_params = int32_t(off);
  off = align16(off + size_t(n_params) * cx.param_stride * rs);
  d.off_mech = int32_t(off);
  off = align16(off + size_t(n_params) * 4);
  d.off_syn = int32_t(off);
  off = align16(off + tsyn.size() * 4);
  d.off_plist = int32_t(off);
  off = align16(off + tprobe.size() * sizeof(ProbeRef));
  d.off_lane_n = -1;
  d.lane_kmax = lane_kmax;
  if (lane) {
    d.off_lane_n = int32_t(off);
    off = align16(off + size_t(T) * 4);
  }
  d.n_cells = int32_t(cell_list.size());
  d.off_ncell = -1;
  d.off_srccell = -1;
  if (has_src) {
    d.off_ncell = int32_t(off);
    off = align16(off + size_t(N) * 2);
    d.off_srccell = int32_t(off);
    off = align16(off + cell_list.size() * 4);
  }
  if (off > size_t(0x7fffffff)) return fail(BC_ERR_CAPACITY, "tile blob exceeds 2 GiB");
  d.blob_bytes = int32_t(off);
  size_t so = 0;
  d.off_dr = int32_t(so);
  so = align16(so + 2 * N * rs);
  d.off_q = int32_t(so);
  so = align16(so + size_t(n_lower) * rs);
  d.off_wparams = int32_t(so);
  if (tb.cls == 2) so = align16(so + size_t(n_params) * cx.param_stride * rs);
  d.off_stamp = -1;
  if (has_src) {
    d.off_stamp = int32_t(so);
    so = align16(so + cell_list.size() * 4);
  }
  size_t n_tile_ports = 0;
  for (size_t li = 0; li < cell_list.size(); ++li) n_tile_ports += (*cx.cell_ports)[cell_list[li]].size();
  d.off_pstage = -1;
  if (n_tile_ports > 0) {
    d.off_pstage = int32_t(so);
    so = align16(so + size_t(kGruSmemBytes) + n_tile_ports * (sizeof(PortStage) + sizeof(PortLocal)));
  }
  // the separators' work area
  d.off_sep = int32_t(so);
  size_t sw = 0;
  d.off_inbox = int32_t(sw);
  sw = align16(sw + 2 * size_t(n_inbox) * rs);
  d.off_srow = int32_t(sw);
  sw = align16(sw + 4 * seps.size() * rs);
  d.off_own = int32_t(sw);
  sw = align16(sw + 2 * seps.size() * rs);
  d.off_xsep = int32_t(sw);
  sw = align16(sw + (seps.size() + kSepPad) * rs);
  d.sep_bytes = int32_t(sw);
  so += sw;
  // in shared memory for a global-memory tile whose CTAs still fit twice on an SM that way
  d.sep_in_smem = tb.cls == 2 && n_tile_ports == 0 && sw + size_t(d.off_rows - d.off_seps) <= kSepSmemLimit;
  d.scratch_bytes = int32_t(so);
  d.n_nodes = int32_t(N);
  d.n_real_nodes = int32_t(n_real);
  d.n_segs = int32_t(segs.size());
  d.n_phases = lane ? 0 : 1 + n_levels;
  d.n_slots = int32_t(slots.size());
  d.n_seps = int32_t(seps.size());
  d.n_inbox = n_inbox;
  d.n_groups = int32_t(groups.size());
  d.n_heavy = int32_t(heavy.size());
  d.n_lower = int32_t(n_lower);
  d.cell0 = cell0;
  d.sep0 = sep0;
  d.n_params = int32_t(n_params);
  // -------- fill
  std::vector<unsigned char>& b = out.blob;
  b.assign(d.blob_bytes, 0);
  out.vinit.assign(n_real, 0.0);
  // the holes of a lane grid and the padding of a tile are boundary rows
  std::memset(b.data() + d.off_pidx, 0xFF, size_t(N) * 2);
  if (lane) {
    std::memcpy(b.data() + d.off_lane_n, lane_n.data(), lane_n.size() * 4);
  }
  auto putr = [&](size_t base_off, size_t idx, double v) {
    if (rs == 8)
      put<double>(b, base_off, idx, v);
    else
      put<float>(b, base_off, idx, float(v));
  };
  for (size_t li = 0; li < cell_list.size(); ++li) {
    const int64_t c = cell_list[li];
    const LoweredCell& lc = (*cx.cells)[c];
    for (int32_t v = 0; v < lc.n_node; ++v) {
      const int32_t j = node_tile[li][v];
      putr(d.off_v, 2 * size_t(j), lc.node_vrest[v]);
      putr(d.off_ab, 2 * size_t(j), lc.alpha[v]);
      putr(d.off_ab, 2 * size_t(j) + 1, lc.beta[v]);
      const uint16_t pi = lc.region[v] >= 0 ? uint16_t(li * R + lc.region[v]) : uint16_t(0xFFFF);
      std::memcpy(b.data() + d.off_pidx + size_t(j) * 2, &pi, 2);
      out.vinit[j] = lc.node_vrest[v];
    }
    if (!lane && !sched_of(li).order.empty()) {
      for (int32_t v = 0; v < lc.n_node; ++v) putr(d.off_diag0, size_t(node_tile[li][v] - cell0), lc.diag[v]);
    } else if (!lane) {
      // the solve's root is path.back(): along the path the old parent is the child
      const std::vector<int32_t>& path = sched_of(li).path;
      for (size_t k = 0; k < path.size(); ++k) {
        const size_t j = size_t(node_tile[li][path[k]]);
        const bool top = k + 1 == path.size();
        putr(d.off_ab, 2 * j, top ? 0.0 : lc.beta[path[k + 1]]);
        putr(d.off_ab, 2 * j + 1, top ? 0.0 : lc.alpha[path[k + 1]]);
      }
    }
    for (int r = 0; r < R; ++r) {
      const int64_t rc = c * R + r;
      for (int k = 0; k < std::min(BC_NPARAM, cx.param_stride - 1); ++k)
        putr(d.off_params, (li * R + r) * cx.param_stride + k, s.region_params[rc * BC_NPARAM + k]);
      const uint32_t m = s.region_mech[rc];
      std::memcpy(b.data() + d.off_mech + (li * R + r) * 4, &m, 4);
    }
    // CV view map
    const int64_t base = (*cx.cv_base)[c];
    for (int32_t k = 0; k < lc.n_cv; ++k) {
      const int32_t v = lc.cv_node[k];
      out.cv_local.push_back({base + k, node_tile[li][v]});
    }
  }
  // special records: pulses in node order, probe ids
  {
    std::vector<uint16_t> spec(N, 0xFFFF);
    std::vector<SpecRec> specs(spec_nodes.size());
    std::vector<int32_t> node_cell(n_real, -1), node_local(n_real, -1);
    for (size_t li = 0; li < cell_list.size(); ++li) {
      const LoweredCell& lc = (*cx.cells)[cell_list[li]];
      for (int32_t v = 0; v < lc.n_node; ++v) {
        node_cell[node_tile[li][v]] = int32_t(li);
        node_local[node_tile[li][v]] = v;
      }
    }
    for (size_t q = 0; q < spec_nodes.size(); ++q) {
      spec[spec_nodes[q]] = uint16_t(q);
      specs[q] = SpecRec{0, 0, -1, 0, 0, {0, 0, 0}};
    }
    size_t kp = 0;
    for (size_t q = 0; q < spec_nodes.size(); ++q) {
      const int32_t node = spec_nodes[q];
      specs[q].pulse_begin = int32_t(out.pulses.size());
      while (kp < tpulse.size() && tpulse[kp].first == node) {
        const int64_t pid = tpulse[kp].second;
        const size_t li = size_t(node_cell[node]);
        const LoweredCell& lc = (*cx.cells)[cell_list[li]];
        const int32_t v = node_local[node];
        PulseRec pr{};
        pr.node = node;
        pr.is_mid = lc.region[v] >= 0 ? 1 : 0;
        if (pr.is_mid) {
          double area = 0.0;
          for (int32_t k = 0; k < lc.n_cv; ++k)
            if (lc.cv_node[k] == v) {
              area = lc.cv_area[k];
              break;
            }
          out.pulse_scale.push_back(1e5 / area);  // nA -> uA/cm^2
        } else {
          out.pulse_scale.push_back(1e-3);  // nA -> mV/ms on a row with the 1 uF dummy capacitance
        }
        pr.amp = s.pulse_amp[pid] * out.pulse_scale.back();
        pr.t_on = s.pulse_t_on[pid];
        pr.t_off = s.pulse_t_off[pid];
        out.pulses.push_back(pr);
        out.pulse_src.push_back(pid);
        ++kp;
      }
      specs[q].pulse_end = int32_t(out.pulses.size());
    }
    size_t ks = 0;
    for (size_t q = 0; q < spec_nodes.size(); ++q) {
      specs[q].syn_begin = int32_t(ks);
      while (ks < tsyn.size() && tsyn[ks].first == spec_nodes[q]) ++ks;
      specs[q].syn_end = int32_t(ks);
    }
    std::vector<int32_t> syn_ids(tsyn.size());
    for (size_t k = 0; k < tsyn.size(); ++k) syn_ids[k] = int32_t(tsyn[k].second);
    if (!syn_ids.empty()) std::memcpy(b.data() + d.off_syn, syn_ids.data(), syn_ids.size() * 4);
    if (has_src) {
      std::vector<uint16_t> ncell(N, 0xFFFF);
      std::vector<int32_t> src(cell_list.size(), -1);
      for (int64_t j = 0; j < n_real; ++j) ncell[j] = uint16_t(node_cell[j]);
      for (size_t li = 0; li < cell_list.size(); ++li)
        if ((*cx.is_src)[cell_list[li]]) src[li] = int32_t(cell_list[li]);
      std::memcpy(b.data() + d.off_ncell, ncell.data(), ncell.size() * 2);
      std::memcpy(b.data() + d.off_srccell, src.data(), src.size() * 4);
    }
    {
      // probes in node order (tprobe is sorted): each special node owns a range
      std::vector<ProbeRef> plist;
      for (const auto& x : tprobe) {
        const int64_t pid = x.second;
        const int32_t field = s.probe_field ? s.probe_field[pid] : BC_STATE_V;
        if (field != BC_STATE_V) {
          plist.push_back(ProbeRef{x.first, int32_t(pid), field, 0});
        } else {
          SpecRec& sr = specs[spec[x.first]];
          if (sr.probe >= 0) return fail(BC_ERR_INVALID, "two voltage probes at the same point of a cell are not supported");
          sr.probe = int32_t(pid);
        }
      }
      d.n_xprobes = int32_t(plist.size());
      if (!plist.empty()) std::memcpy(b.data() + d.off_plist, plist.data(), plist.size() * sizeof(ProbeRef));
    }
    std::memcpy(b.data() + d.off_spec, spec.data(), spec.size() * 2);
    if (!specs.empty()) std::memcpy(b.data() + d.off_specs, specs.data(), specs.size() * sizeof(SpecRec));
  }
  // surrogate ports of the tile's cells (the plan assigns port_offset)
  for (size_t li = 0; li < cell_list.size(); ++li) {
    const int64_t c = cell_list[li];
    for (const auto& pt : (*cx.cell_ports)[c]) {
      PortRec r{};
      r.node = node_tile[li][pt[1]];
      r.att = node_tile[li][pt[2]];
      r.cell = int32_t(c);
      r.id = pt[0];
      r.g = s.port_g[pt[0]];
      r.e = s.port_e[pt[0]];
      r.feat[0] = float(s.port_feat[2 * size_t(pt[0])]);
      r.feat[1] = float(s.port_feat[2 * size_t(pt[0]) + 1]);
      r.stim_begin = int32_t(out.port_pulses.size());
      for (int64_t q : (*cx.port_pulse_ids)[pt[0]]) {
        PulseRec pr{};
        pr.node = r.node;
        pr.amp = s.port_pulse_amp[q];
        pr.t_on = s.port_pulse_t_on[q];
        pr.t_off = s.port_pulse_t_off[q];
        out.port_pulses.push_back(pr);
      }
      r.stim_end = int32_t(out.port_pulses.size());
      out.ports.push_back(r);
    }
  }
  d.n_ports = int32_t(out.ports.size());
  auto put_all = [&](int32_t at, const void* src, size_t bytes) {
    if (bytes) std::memcpy(b.data() + at, src, bytes);
  };
  put_all(d.off_link, link.data(), link.size() * 4);
  put_all(d.off_segs, segs.data(), segs.size() * sizeof(SegRec));
  put_all(d.off_slots, slots.data(), slots.size() * sizeof(SlotRec));
  put_all(d.off_seps, seps.data(), seps.size() * sizeof(SepRec));
  put_all(d.off_levels, levels.data(), levels.size() * 4);
  put_all(d.off_groups, groups.data(), groups.size() * sizeof(GroupRec));
  put_all(d.off_rows, rows.data(), rows.size() * 4);
  put_all(d.off_heavy, heavy.data(), heavy.size() * 4);
  put_all(d.off_crec, crec.data(), crec.size() * 2);
  out.desc = d;
  return BC_OK;
}

static size_t max_optin_smem(int device) {
  int v = 0;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) return 0;
  return size_t(v);
}

static size_t sm_smem(int device) {
  int v = 0;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device) != cudaSuccess) return 0;
  return size_t(v);
}

// First step index s with s * dt >= t (float64), for clamp windows.
static int64_t first_step_at(double t, double dt) {
  if (t <= 0.0) return 0;
  int64_t s = int64_t(std::floor(t / dt));
  if (s < 0) s = 0;
  while (s > 0 && double(s - 1) * dt >= t) --s;
  while (double(s) * dt < t) ++s;
  return s;
}

static bc_status update_pulses(bc_plan* p, double dt, void* stream) {
  if (!p->port_pulses.empty() && p->port_pulses_dt != dt) {
    for (auto& pr : p->port_pulses) {
      pr.on_step = first_step_at(pr.t_on, dt);
      pr.off_step = first_step_at(pr.t_off, dt);
    }
    BC_CUDA(cudaMemcpyAsync(p->d_port_pulses, p->port_pulses.data(), p->port_pulses.size() * sizeof(PulseRec),
                            cudaMemcpyHostToDevice, static_cast<cudaStream_t>(stream)));
    BC_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
    p->port_pulses_dt = dt;
  }
  if (p->pulses.empty() || p->pulses_dt == dt) return BC_OK;
  if (!p->pulse_amp.empty())
    for (size_t k = 0; k < p->pulses.size(); ++k) p->pulses[k].amp = p->pulse_amp[p->pulse_src[k]] * p->pulse_scale[k];
  for (auto& pr : p->pulses) {
    pr.on_step = first_step_at(pr.t_on, dt);
    pr.off_step = first_step_at(pr.t_off, dt);
  }
  BC_CUDA(cudaMemcpyAsync(p->d_pulses, p->pulses.data(), p->pulses.size() * sizeof(PulseRec), cudaMemcpyHostToDevice,
                          static_cast<cudaStream_t>(stream)));
  BC_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
  p->pulses_dt = dt;
  return BC_OK;
}

static bc_status ensure_traces(bc_plan* p, int64_t records, void* stream) {
  if (p->n_probes == 0 || records <= p->trace_cap) return BC_OK;
  int64_t cap = std::max<int64_t>(records, p->trace_cap * 2);
  double* nb = nullptr;
  BC_CUDA(cudaMalloc(reinterpret_cast<void**>(&nb), size_t(cap) * p->n_probes * sizeof(double)));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (p->d_traces && p->trace_cap > 0) {
    BC_CUDA(cudaMemcpyAsync(nb, p->d_traces, size_t(p->trace_cap) * p->n_probes * sizeof(double),
                            cudaMemcpyDeviceToDevice, st));
    BC_CUDA(cudaStreamSynchronize(st));
  }
  cudaFree(p->d_traces);
  p->device_bytes += size_t(cap - p->trace_cap) * p->n_probes * sizeof(double);
  p->d_traces = nb;
  p->trace_cap = cap;
  return BC_OK;
}

// Kernel variant of a plan (see launch_tiles).
static int kernel_variant(const bc_plan* p) {
  if (p->n_ports > 0) return p->extra ? BC_VARIANT_PORTS : BC_VARIANT_PORTS_LEAN;
  return p->extra ? BC_VARIANT_EXTRA : BC_VARIANT_LEAN;
}

static LaunchArgs base_args(bc_plan* p) {
  LaunchArgs a{};
  a.blob = p->d_blob;
  a.scratch = p->d_scratch;
  a.state = p->d_state;
  a.pulses = p->d_pulses;
  a.traces = p->d_traces;
  a.trace_cap = p->trace_cap;
  a.trace_base = p->trace_origin;
  a.n_probes_total = p->n_probes;
  a.record_every = p->record_every;
  a.max_spikes = p->max_spikes;
  a.spike_count = p->d_spike_count;
  a.spike_times = p->d_spike_times;
  a.status = p->d_status;
  a.state_slots = p->state_slots;
  a.cluster = 1;
  a.timers = p->d_timers;
  a.syn_g = p->d_syn_g;
  a.syn_tau = p->d_syn_tau;
  a.syn_e = p->d_syn_e;
  a.syn_scale = p->d_syn_scale;
  a.arrivals = p->n_connections > 0 ? p->d_arrivals : nullptr;
  a.arr_slots = std::max<int64_t>(p->arr_slots, 1);
  a.n_syn = p->n_synapses;
  a.rec_cell = p->d_rec_cell;
  a.rec_step = p->d_rec_step;
  a.rec_count = p->d_rec_count;
  a.rec_cap = p->rec_cap;
  a.ports = p->d_ports;
  a.port_pulses = p->d_port_pulses;
  a.port_h = p->d_port_h;
  a.port_flags = p->d_port_flags;
  a.gru = p->d_gru;
  return a;
}

// Delays in whole steps for dt (network/lowering.py:185-226, "ceil": delays within
// 1e-7 of a whole number of steps count as that number), and the arrival ring:
// launches of at most the shortest delay (so a launch never receives an event its
// own spikes cause) and room for the longest delay past the current launch.
static bc_status prepare_network(bc_plan* p, double dt, void* stream) {
  if (p->n_connections == 0 || p->net_dt == dt) return BC_OK;
  if (p->net_dt != 0.0 && p->step != 0)
    return fail(BC_ERR_INVALID, "a network plan keeps its dt between resets; call bc_reset before changing dt");
  std::vector<int32_t> d(p->n_connections);
  int64_t dmin = INT64_MAX, dmax = 1;
  for (int64_t q = 0; q < p->n_connections; ++q) {
    double raw = p->conn_delay[p->out_order[q]] / dt;
    const double near = std::nearbyint(raw);
    if (std::fabs(raw - near) <= 1e-7 + 1e-7 * std::fabs(near)) raw = near;
    const double st = std::ceil(raw - 1e-12);
    if (st > 1e9) return fail(BC_ERR_INVALID, "connection delay too long for this dt");
    d[q] = int32_t(st);
    const int64_t eff = std::max<int64_t>(d[q], 1);
    dmin = std::min(dmin, eff);
    dmax = std::max(dmax, eff);
  }
  const int64_t k = std::min<int64_t>(p->steps_per_launch, dmin);
  const int64_t slots = k + dmax + 1;
  const size_t rs = p->real_size;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  BC_CUDA(cudaStreamSynchronize(s));
  cudaFree(p->d_arrivals);
  p->d_arrivals = nullptr;
  const size_t bytes = size_t(slots) * size_t(std::max<int64_t>(p->n_synapses, 1)) * rs;
  BC_CUDA(cudaMalloc(&p->d_arrivals, bytes));
  BC_CUDA(cudaMemsetAsync(p->d_arrivals, 0, bytes, s));
  BC_CUDA(cudaMemcpyAsync(p->d_out_d, d.data(), d.size() * 4, cudaMemcpyHostToDevice, s));
  BC_CUDA(cudaStreamSynchronize(s));
  p->arr_slots = slots;
  p->net_k = k;
  p->net_dt = dt;
  return BC_OK;
}

// The launches of one run as a CUDA graph: each launch class is a chain of
// kernel nodes (the classes hold independent cells, so the chains run side by
// side).  The graph is built when the number of launches or their step counts
// change; otherwise only the kernel arguments (first step, trace buffer, ...)
// of its nodes are updated before the replay.
static bc_status enqueue_run_graph(bc_plan* p, int64_t n_steps, double dt, void* stream) {
  const int32_t K = p->steps_per_launch;
  const int64_t L = (n_steps + K - 1) / K;
  const int32_t k_last = int32_t(n_steps - (L - 1) * K);
  const int nc = int(p->classes.size());
  std::vector<LaunchArgs> args(size_t(L) * nc);
  for (int64_t j = 0; j < L; ++j)
    for (int ci = 0; ci < nc; ++ci) {
      LaunchArgs a = base_args(p);
      a.step0 = p->step + j * K;
      a.n_steps = j + 1 == L ? k_last : K;
      a.dt = dt;
      a.tiles = p->d_tiles + p->classes[ci].first;
      a.n_tiles = p->classes[ci].count;
      args[size_t(j) * nc + ci] = a;
    }
  const bool rebuild = !p->graph_exec || p->graph_launches != L || p->graph_k != K || p->graph_k_last != k_last;
  if (rebuild) {
    if (p->graph_exec) cudaGraphExecDestroy(p->graph_exec);
    if (p->graph) cudaGraphDestroy(p->graph);
    p->graph_exec = nullptr;
    p->graph = nullptr;
    p->graph_launches = -1;
    BC_CUDA(cudaGraphCreate(&p->graph, 0));
    p->graph_nodes.assign(size_t(L) * nc, nullptr);
    for (int64_t j = 0; j < L; ++j)
      for (int ci = 0; ci < nc; ++ci) {
        const LaunchClass& lcz = p->classes[ci];
        cudaKernelNodeParams np{};
        const LaunchArgs* hold = nullptr;
        int e = lcz.lane ? lane_node_params(&args[size_t(j) * nc + ci], p->precision, lcz.threads, p->extra, &np, &hold)
                         : tile_node_params(&args[size_t(j) * nc + ci], p->precision, lcz.smem, lcz.threads, lcz.smem_bytes,
                                            kernel_variant(p), &np, &hold);
        if (e) return fail(BC_ERR_CUDA, std::string("graph node: ") + cudaGetErrorString(cudaError_t(e)));
        cudaGraphNode_t dep = j > 0 ? p->graph_nodes[size_t(j - 1) * nc + ci] : nullptr;
        BC_CUDA(cudaGraphAddKernelNode(&p->graph_nodes[size_t(j) * nc + ci], p->graph, dep ? &dep : nullptr,
                                       dep ? 1 : 0, &np));
      }
    BC_CUDA(cudaGraphInstantiate(&p->graph_exec, p->graph, 0));
    p->graph_launches = L;
    p->graph_k = K;
    p->graph_k_last = k_last;
  } else {
    for (int64_t j = 0; j < L; ++j)
      for (int ci = 0; ci < nc; ++ci) {
        const LaunchClass& lcz = p->classes[ci];
        cudaKernelNodeParams np{};
        const LaunchArgs* hold = nullptr;
        int e = lcz.lane ? lane_node_params(&args[size_t(j) * nc + ci], p->precision, lcz.threads, p->extra, &np, &hold)
                         : tile_node_params(&args[size_t(j) * nc + ci], p->precision, lcz.smem, lcz.threads, lcz.smem_bytes,
                                            kernel_variant(p), &np, &hold);
        if (e) return fail(BC_ERR_CUDA, std::string("graph node: ") + cudaGetErrorString(cudaError_t(e)));
        BC_CUDA(cudaGraphExecKernelNodeSetParams(p->graph_exec, p->graph_nodes[size_t(j) * nc + ci], &np));
      }
  }
  BC_CUDA(cudaGraphLaunch(p->graph_exec, static_cast<cudaStream_t>(stream)));
  return BC_OK;
}

static bc_status enqueue_run(bc_plan* p, int64_t n_steps, double dt, void* stream) {
  if (n_steps < 0) return fail(BC_ERR_INVALID, "n_steps must be >= 0");
  if (!(dt > 0.0) || !std::isfinite(dt)) return fail(BC_ERR_INVALID, "dt must be a positive finite number (ms)");
  if (p->n_ports > 0 && !p->gru_set) return fail(BC_ERR_INVALID, "the plan has surrogate ports: call bc_surrogate_set first");
  bc_status st = update_pulses(p, dt, stream);
  if (st != BC_OK) return st;
  const int64_t recs = p->record_every > 0 ? (p->step + n_steps - p->trace_origin) / p->record_every : 0;
  st = ensure_traces(p, recs, stream);
  if (st != BC_OK) return st;
  st = prepare_network(p, dt, stream);
  if (st != BC_OK) return st;
  const bool net = p->n_connections > 0;
  if (p->use_graph && n_steps > 0 && !net) {
    st = enqueue_run_graph(p, n_steps, dt, stream);
    if (st == BC_OK) p->step += n_steps;
    return st;
  }
  const int64_t per_launch = net ? std::min<int64_t>(p->steps_per_launch, p->net_k) : p->steps_per_launch;
  if (p->classes.size() > 1) {
    // the forked class streams take the priority of the caller's stream; work still
    // queued on the streams they replace completes, and this run's forks are ordered
    // after it through the caller's stream (the last run joined into it)
    int prio = 0;
    BC_CUDA(cudaStreamGetPriority(static_cast<cudaStream_t>(stream), &prio));
    if (prio != p->aux_prio) {
      for (int k = 0; k < kMaxClasses - 1; ++k) {
        cudaStream_t ns = nullptr;
        BC_CUDA(cudaStreamCreateWithPriority(&ns, cudaStreamNonBlocking, prio));
        if (p->aux[k]) cudaStreamDestroy(p->aux[k]);
        p->aux[k] = ns;
      }
      p->aux_prio = prio;
    }
  }
  int64_t done = 0;
  while (done < n_steps) {
    const int32_t k = int32_t(std::min<int64_t>(per_launch, n_steps - done));
    LaunchArgs a = base_args(p);
    a.step0 = p->step + done;
    a.n_steps = k;
    a.dt = dt;
    // Classes are independent cells: the first runs on the caller's stream, the
    // others on forked streams so their CTAs can share SMs.
    cudaStream_t main_st = static_cast<cudaStream_t>(stream);
    const int nc = int(p->classes.size());
    if (nc > 1) BC_CUDA(cudaEventRecord(p->ev_fork, main_st));
    for (int ci = 0; ci < nc; ++ci) {
      const LaunchClass& lcz = p->classes[ci];
      cudaStream_t st = main_st;
      if (ci > 0) {
        st = p->aux[ci - 1];
        BC_CUDA(cudaStreamWaitEvent(st, p->ev_fork, 0));
      }
      a.tiles = p->d_tiles + lcz.first;
      a.n_tiles = lcz.count;
      a.cluster = lcz.cluster;
      int e = lcz.lane ? launch_lanes(a, p->precision, lcz.threads, p->extra, st)
                       : launch_tiles(a, p->precision, lcz.smem, lcz.threads, lcz.smem_bytes, kernel_variant(p), st);
      if (e) return fail(BC_ERR_CUDA, std::string("tile kernel launch: ") + cudaGetErrorString(cudaError_t(e)));
      if (ci > 0) {
        BC_CUDA(cudaEventRecord(p->ev_join[ci - 1], st));
        BC_CUDA(cudaStreamWaitEvent(main_st, p->ev_join[ci - 1], 0));
      }
    }
    if (net) {
      // deliver this launch's spikes into the arrival ring, then mark them delivered
      int e = launch_deliver_impl(p->precision, p->d_rec_cell, p->d_rec_step, p->d_rec_count, p->d_rec_count + 1,
                                  p->rec_cap, p->d_out_ptr, p->d_out_syn, p->d_out_w, p->d_out_d, p->d_arrivals,
                                  p->arr_slots, p->n_synapses, stream);
      if (e) return fail(BC_ERR_CUDA, std::string("delivery kernel: ") + cudaGetErrorString(cudaError_t(e)));
      BC_CUDA(cudaMemcpyAsync(p->d_rec_count + 1, p->d_rec_count, sizeof(unsigned long long),
                              cudaMemcpyDeviceToDevice, main_st));
    }
    done += k;
  }
  p->step += n_steps;
  return BC_OK;
}

}  // namespace bc

using namespace bc;

extern "C" {

const char* bc_last_error(void) { return g_error.c_str(); }

int32_t bc_version(void) { return BC_ABI_VERSION; }

void bc_default_options(bc_plan_options* o) {
  std::memset(o, 0, sizeof(*o));
  o->precision = BC_PREC_F32;
  o->threads_per_tile = 0;
  o->tile_nodes = 0;
  o->lane_nodes = kDefaultLaneNodes;
  o->steps_per_launch = 0;
  o->record_every = 1;
  o->max_spikes = 64;
  o->use_graph = 0;
  o->device = 0;
}

bc_status bc_plan_create(const bc_batch_spec* spec, const bc_plan_options* opts_in, bc_plan_t* out) {
  if (!spec || !out) return fail(BC_ERR_INVALID, "null argument");
  *out = nullptr;
  bc_plan_options opts;
  if (opts_in)
    opts = *opts_in;
  else
    bc_default_options(&opts);
  const bc_batch_spec& s = *spec;
  if (s.n_cells <= 0) return fail(BC_ERR_INVALID, "n_cells must be > 0");
  if (s.n_regions <= 0) return fail(BC_ERR_INVALID, "n_regions must be > 0");
  if (opts.precision != BC_PREC_F32 && opts.precision != BC_PREC_F64)
    return fail(BC_ERR_INVALID, "precision must be BC_PREC_F32 or BC_PREC_F64");
  if (opts.tile_order < 0 || opts.tile_order > 1) return fail(BC_ERR_INVALID, "tile_order must be 0 or 1");
  if (opts.threads_per_tile < 0 || opts.threads_per_tile > 1024 || opts.threads_per_tile % 32)
    return fail(BC_ERR_INVALID, "threads_per_tile must be 0 or a multiple of 32 up to 1024");
  if (opts.record_every < 0 || opts.max_spikes < 0) return fail(BC_ERR_INVALID, "record_every/max_spikes must be >= 0");
  if (s.cell_branch_offsets[0] != 0 || s.cell_branch_offsets[s.n_cells] != s.n_branches)
    return fail(BC_ERR_INVALID, "cell_branch_offsets must span [0, n_branches]");
  const bool dry = opts.dry_run != 0;
  if (!dry) BC_CUDA(cudaSetDevice(opts.device));
  bc_plan* p = new bc_plan();
  p->dry = dry;
  p->precision = opts.precision;
  p->device = opts.device;
  p->real_size = opts.precision == BC_PREC_F64 ? 8 : 4;
  p->record_every = opts.record_every;
  p->max_spikes = opts.max_spikes;
  p->use_graph = opts.use_graph;
  p->steps_per_launch = opts.steps_per_launch > 0 ? opts.steps_per_launch : 1000;
  p->lane_nodes = opts.lane_nodes > 0 ? opts.lane_nodes : kDefaultLaneNodes;
  p->n_cells = s.n_cells;
  // ---------------------------------------------------- lower
  std::vector<LoweredCell> cells(s.n_cells);
  std::vector<int64_t> cv_base(s.n_cells + 1, 0);
  {
    // cells lower independently; the failure reported is that of the first failing
    // cell in cell order, as a sequential pass would report it
    std::vector<bc_status> lst(s.n_cells, BC_OK);
    std::vector<std::string> lmsg(s.n_cells);
    parallel_for(s.n_cells, [&](int64_t c) {
      try {
        lst[c] = lower_cell(s, c, cells[c]);
        if (lst[c] != BC_OK) lmsg[c] = bc_last_error();
      } catch (const std::exception& ex) {
        lst[c] = BC_ERR_CAPACITY;
        lmsg[c] = std::string("lowering cell ") + std::to_string(c) + ": " + ex.what();
      }
    });
    for (int64_t c = 0; c < s.n_cells; ++c) {
      if (lst[c] != BC_OK) {
        delete p;
        return fail(lst[c], lmsg[c]);
      }
      cv_base[c + 1] = cv_base[c] + cells[c].n_cv;
      p->n_nodes += cells[c].n_node;
    }
  }
  p->n_cv = cv_base[s.n_cells];
  p->cell_ncv.resize(s.n_cells);
  for (int64_t c = 0; c < s.n_cells; ++c) p->cell_ncv[c] = cells[c].n_cv;
  for (int64_t k = 0; k < s.n_cells * s.n_regions; ++k)
    p->extra = p->extra || (s.region_mech[k] & kOutOfLineBits) != 0;
  for (int64_t k = 0; k < s.n_cells * s.n_regions; ++k) {
    if (s.region_mech[k] & ~BC_M_ALL) {
      delete p;
      return fail(BC_ERR_INVALID, "unknown mechanism bits in region_mech");
    }
    if (s.region_mech[k] & BC_M_EXT) {
      // the record lists its extension channels: integers of known BC_X_* bits (low 24 and
      // the rest), not all 0
      const double lo = s.region_params[k * BC_NPARAM + BC_P_EXT_MASK];
      const double hi = s.region_params[k * BC_NPARAM + BC_P_EXT_MASK_HI];
      const bool ints = lo >= 0.0 && lo < 16777216.0 && lo == std::floor(lo) && hi >= 0.0 && hi < 256.0 &&
                        hi == std::floor(hi);
      const uint32_t x = ints ? uint32_t(lo) | (uint32_t(hi) << 24) : 0u;
      if (!ints || x == 0u || (x & ~BC_X_ALL)) {
        delete p;
        return fail(BC_ERR_INVALID, "a region with BC_M_EXT needs BC_X_* bits in its record's BC_P_EXT_MASK");
      }
    }
  }
  uint32_t all_bits = 0;
  for (int64_t k = 0; k < s.n_cells * s.n_regions; ++k) all_bits |= s.region_mech[k];
  // the Markov, cerebellar and extension states only where a plan has them
  const int S = (all_bits & BC_M_EXT) ? kNumSlotsExt
                                      : ((all_bits & kCerebellarBits) ? kNumSlotsCerebellar
                                                                      : ((all_bits & kMarkovBits) ? kNumSlotsMarkov : kNumSlots));
  p->state_slots = S;
  // ---------------------------------------------------- pulses / probes -> nodes
  std::vector<std::vector<int64_t>> cell_pulses(s.n_cells), cell_probes(s.n_cells);
  std::vector<std::vector<int32_t>> pulse_node(s.n_cells), probe_node(s.n_cells);
  for (int64_t k = 0; k < s.n_pulses; ++k) {
    const int64_t c = s.pulse_cell[k];
    if (c < 0 || c >= s.n_cells) {
      delete p;
      return fail(BC_ERR_INVALID, "pulse_cell out of range");
    }
    const int32_t v = locate_node(s, c, cells[c], s.pulse_branch[k], s.pulse_x[k]);
    if (v < 0) {
      delete p;
      return fail(BC_ERR_INVALID, "pulse location not found");
    }
    if (!(s.pulse_t_off[k] >= s.pulse_t_on[k])) {
      delete p;
      return fail(BC_ERR_INVALID, "pulse_t_off must be >= pulse_t_on");
    }
    cell_pulses[c].push_back(k);
    pulse_node[c].push_back(v);
  }
  p->probe_vrest.assign(s.n_probes, 0.0);
  for (int64_t k = 0; k < s.n_probes; ++k) {
    const int64_t c = s.probe_cell[k];
    if (c < 0 || c >= s.n_cells) {
      delete p;
      return fail(BC_ERR_INVALID, "probe_cell out of range");
    }
    const int32_t v = locate_node(s, c, cells[c], s.probe_branch[k], s.probe_x[k]);
    if (v < 0) {
      delete p;
      return fail(BC_ERR_INVALID, "probe location not found");
    }
    const int32_t field = s.probe_field ? s.probe_field[k] : BC_STATE_V;
    const bool is_current = field >= BC_PROBE_CURRENT && field < BC_PROBE_CURRENT + BC_NCUR;
    if (!is_current && (field < 0 || field >= BC_NSTATE_VIEW || field == BC_STATE_V_LAST)) {
      delete p;
      return fail(BC_ERR_INVALID, "probe_field is not a recordable BC_STATE_* view or a BC_PROBE_CURRENT code");
    }
    if (is_current) {
      static const uint64_t cur_owner[BC_NCUR] = {
          BC_M_IL,  BC_M_KLEAK, BC_M_NA,   BC_M_KDR, BC_M_CAL,           BC_M_CAT,
          BC_M_HCN, BC_M_AHP,   BC_M_NAHH, BC_M_KHH, BC_M_KM,
          BC_M_NA | BC_M_NAHH | BC_M_NAV16 | ext_bits(BC_X_NAF | BC_X_NAP | BC_X_NAIO | BC_X_NAVGRC),
          BC_M_KDR | BC_M_KLEAK | BC_M_AHP | BC_M_KHH | BC_M_KM | BC_M_KA1 | BC_M_KA2 | BC_M_KK2A | BC_M_KK2B | BC_M_KNI |
              BC_M_KCA22 | BC_M_KCA11 | BC_M_KV34 | BC_M_KV43 | BC_M_KV11 | BC_M_KIR23 |
              ext_bits(BC_X_KV33 | BC_X_KV22 | BC_X_KV15 | BC_X_FKDR | BC_X_SKDR | BC_X_KDRIO | BC_X_KCA31 |
                       BC_X_SKDCN | BC_X_KKV),
          BC_M_CAL | BC_M_CAT | BC_M_CAHVA | BC_M_CAV23 | BC_M_CAV32 | ext_bits(BC_X_CATHP | BC_X_CAHTRE | BC_X_CAN | BC_X_CAV31 | BC_X_CAV33 |
                                                                  BC_X_CAV12 | BC_X_CAV13 | BC_X_CAV21 |
                                                                  BC_X_CAHVADCN | BC_X_CALVADCN),
          BC_M_KA1,  BC_M_KA2, BC_M_KK2A, BC_M_KK2B, BC_M_KNI,
          BC_M_NAV16, BC_M_KCA22, BC_M_KCA11, BC_M_KV34, BC_M_KV43, BC_M_KV11, BC_M_KIR23, BC_M_HCN1F, BC_M_HCN1H,
          BC_M_CAHVA, BC_M_CAV23, BC_M_CAV32,
          ext_bits(BC_X_HCN2), ext_bits(BC_X_KV33), ext_bits(BC_X_KV22), ext_bits(BC_X_KV15), ext_bits(BC_X_NAF),
          ext_bits(BC_X_NAP), ext_bits(BC_X_NAIO), ext_bits(BC_X_FKDR), ext_bits(BC_X_SKDR), ext_bits(BC_X_KDRIO),
          ext_bits(BC_X_HCNDCN), ext_bits(BC_X_HCNIO), ext_bits(BC_X_CATHP), ext_bits(BC_X_CAHTRE),
          ext_bits(BC_X_CALDCN), ext_bits(BC_X_KCA31), ext_bits(BC_X_SKDCN), ext_bits(BC_X_KKV), ext_bits(BC_X_CAN),
          ext_bits(BC_X_CAIO), ext_bits(BC_X_NAVGRC), ext_bits(BC_X_CAV31), ext_bits(BC_X_CAV33), ext_bits(BC_X_CAV12),
          ext_bits(BC_X_CAV13), ext_bits(BC_X_CAV21), ext_bits(BC_X_CAHVADCN), ext_bits(BC_X_CALVADCN)};
      const int32_t rg = cells[c].region[v];
      if (rg < 0 || !(region_bits(s, c * s.n_regions + rg) & cur_owner[field - BC_PROBE_CURRENT])) {
        delete p;
        return fail(BC_ERR_INVALID, "probe current: no such mechanism at the probed location");
      }
    } else if (field != BC_STATE_V) {
      // the mechanism that owns the state must be present at the probed CV
      uint64_t owner = 0;
      int slot = -1;
      state_view(field, &owner, &slot);
      const int32_t rg = cells[c].region[v];
      if (rg < 0 || !(region_bits(s, c * s.n_regions + rg) & owner)) {
        delete p;
        return fail(BC_ERR_INVALID, "probe field: no such mechanism at the probed location");
      }
    }
    cell_probes[c].push_back(k);
    probe_node[c].push_back(v);
    p->probe_vrest[k] = cells[c].node_vrest[v];
  }
  p->n_probes = s.n_probes;
  p->n_pulses = s.n_pulses;
  // mechanism probes are recorded by the extra kernel variant only
  bool mech_probes = false;
  for (int64_t k = 0; s.probe_field && k < s.n_probes; ++k) mech_probes = mech_probes || s.probe_field[k] != BC_STATE_V;
  p->extra = p->extra || mech_probes;
  // ---------------------------------------------------- synapses / connections
  std::vector<std::vector<std::pair<int64_t, int32_t>>> cell_syns(s.n_cells);
  std::vector<char> is_src(s.n_cells, 0);
  if (s.n_synapses < 0 || s.n_connections < 0) {
    delete p;
    return fail(BC_ERR_INVALID, "n_synapses and n_connections must be >= 0");
  }
  std::vector<double> syn_scale(s.n_synapses, 0.0);
  for (int64_t k = 0; k < s.n_synapses; ++k) {
    const int64_t c = s.syn_cell[k];
    if (c < 0 || c >= s.n_cells) {
      delete p;
      return fail(BC_ERR_INVALID, "syn_cell out of range");
    }
    if (!(s.syn_tau[k] > 0.0) || !std::isfinite(s.syn_e[k])) {
      delete p;
      return fail(BC_ERR_INVALID, "synapse tau must be > 0 ms and e finite");
    }
    if (!(s.syn_x[k] > 0.0 && s.syn_x[k] < 1.0)) {
      delete p;
      return fail(BC_ERR_INVALID, "a synapse must sit inside a CV (0 < syn_x < 1)");
    }
    const int32_t v = locate_node(s, c, cells[c], s.syn_branch[k], s.syn_x[k]);
    int32_t cv = -1;
    for (int32_t q = 0; q < cells[c].n_cv && v >= 0; ++q)
      if (cells[c].cv_node[q] == v) cv = q;
    if (v < 0 || cv < 0) {
      delete p;
      return fail(BC_ERR_INVALID, "synapse location not found");
    }
    cell_syns[c].push_back({k, v});
    syn_scale[k] = 1e5 / cells[c].cv_area[cv];
  }
  for (int64_t j = 0; j < s.n_connections; ++j) {
    if (s.conn_pre[j] < 0 || s.conn_pre[j] >= s.n_cells || s.conn_post[j] < 0 || s.conn_post[j] >= s.n_synapses) {
      delete p;
      return fail(BC_ERR_INVALID, "connection pre cell or post synapse out of range");
    }
    if (!(s.conn_delay[j] >= 0.0) || !std::isfinite(s.conn_weight[j])) {
      delete p;
      return fail(BC_ERR_INVALID, "connection delay must be >= 0 ms and weight finite");
    }
  }
  // ---------------------------------------------------- surrogate ports
  std::vector<std::vector<std::array<int32_t, 3>>> cell_ports(s.n_cells);
  std::vector<std::vector<int64_t>> port_pulse_ids(std::max<int64_t>(s.n_ports, 0));
  if (s.n_ports < 0 || s.n_port_pulses < 0 || s.n_ports >= (int64_t(1) << 31)) {
    delete p;
    return fail(BC_ERR_INVALID, "n_ports and n_port_pulses must be >= 0");
  }
  for (int64_t k = 0; k < s.n_ports; ++k) {
    const int64_t c = s.port_cell[k];
    if (c < 0 || c >= s.n_cells) {
      delete p;
      return fail(BC_ERR_INVALID, "port_cell out of range");
    }
    if (!(s.port_g[k] > 0.0) || !std::isfinite(s.port_g[k]) || !std::isfinite(s.port_e[k]) ||
        !std::isfinite(s.port_feat[2 * k]) || !std::isfinite(s.port_feat[2 * k + 1])) {
      delete p;
      return fail(BC_ERR_INVALID, "port g must be > 0 and e, features finite");
    }
    const int32_t br = s.port_branch[k];
    const int32_t nb = int32_t(s.cell_branch_offsets[c + 1] - s.cell_branch_offsets[c]);
    if (br < 0 || br >= nb) {
      delete p;
      return fail(BC_ERR_INVALID, "port_branch out of range");
    }
    const int32_t ncv = s.branch_ncv[s.cell_branch_offsets[c] + br];
    const int32_t end = locate_node(s, c, cells[c], br, 1.0);
    const int32_t att = locate_node(s, c, cells[c], br, 1.0 - 0.5 / double(ncv));
    if (end < 0 || att < 0 || cells[c].region[att] < 0) {
      delete p;
      return fail(BC_ERR_INVALID, "port location not found");
    }
    for (const auto& q : cell_ports[c])
      if (q[1] == end) {
        delete p;
        return fail(BC_ERR_INVALID, "two ports at the same branch end are not supported");
      }
    cell_ports[c].push_back({int32_t(k), end, att});
  }
  for (int64_t q = 0; q < s.n_port_pulses; ++q) {
    const int64_t k = s.port_pulse_port[q];
    if (k < 0 || k >= s.n_ports) {
      delete p;
      return fail(BC_ERR_INVALID, "port_pulse_port out of range");
    }
    if (!(s.port_pulse_t_off[q] >= s.port_pulse_t_on[q]) || !std::isfinite(s.port_pulse_amp[q])) {
      delete p;
      return fail(BC_ERR_INVALID, "port pulse needs t_off >= t_on and a finite amplitude");
    }
    port_pulse_ids[k].push_back(q);
  }
  p->n_ports = s.n_ports;
  // every cell of a network records its spikes (the output of a network run);
  // only cells with connections have events to deliver
  if (s.n_connections > 0) std::fill(is_src.begin(), is_src.end(), char(1));
  p->n_synapses = s.n_synapses;
  p->n_connections = s.n_connections;
  p->extra = p->extra || s.n_synapses > 0 || s.n_connections > 0;
  p->syn_tau.assign(s.syn_tau, s.syn_tau + s.n_synapses);
  p->syn_e.assign(s.syn_e, s.syn_e + s.n_synapses);
  p->syn_scale = syn_scale;
  p->conn_delay.assign(s.conn_delay, s.conn_delay + s.n_connections);
  {
    // connections in CSR by presynaptic cell
    std::vector<int64_t> order(s.n_connections);
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](int64_t a, int64_t b) { return s.conn_pre[a] < s.conn_pre[b]; });
    p->out_ptr.assign(s.n_cells + 1, 0);
    for (int64_t j = 0; j < s.n_connections; ++j) p->out_ptr[s.conn_pre[j] + 1]++;
    for (int64_t c = 0; c < s.n_cells; ++c) p->out_ptr[c + 1] += p->out_ptr[c];
    p->out_order = order;
    p->out_syn.resize(s.n_connections);
    p->out_w.resize(s.n_connections);
    for (int64_t q = 0; q < s.n_connections; ++q) {
      p->out_syn[q] = s.conn_post[order[q]];
      p->out_w[q] = s.conn_weight[order[q]];
    }
  }
  // ---------------------------------------------------- schedules
  std::vector<CellSched> sched(s.n_cells);
  {
    // as for the lowering: per-cell outcomes, the first failing cell reported
    std::vector<std::string> dmsg(s.n_cells);
    std::vector<char> dbad(s.n_cells, 0);
    parallel_for(s.n_cells, [&](int64_t c) {
      try {
        decompose(cells[c], p->lane_nodes, sched[c]);
      } catch (const std::exception& ex) {
        dbad[c] = 1;
        dmsg[c] = std::string("scheduling cell ") + std::to_string(c) + ": " + ex.what();
      }
    });
    for (int64_t c = 0; c < s.n_cells; ++c)
      if (dbad[c]) {
        delete p;
        return fail(BC_ERR_CAPACITY, dmsg[c]);
      }
  }
  // ---------------------------------------------------- tile packing
  const size_t rs = p->real_size;
  const size_t smem_cap = dry ? size_t(232448) : max_optin_smem(opts.device);
  if (smem_cap == 0) {
    delete p;
    return fail(BC_ERR_CUDA, "could not query the shared-memory limit of the device");
  }
  const size_t smem_budget = smem_cap - kStaticSmem;
  // shared bytes per node, for packing: V, (alpha, beta) and row pairs, link and region / special indices, and
  // per 6.4 nodes a segment (record, inbox), per 16 a separator, a third of the nodes with a q entry
  const double bpn = 6.0 * double(rs) + 8.0 + (16.0 + 2.0 * double(rs)) / 6.4 + (20.0 + 9.0 * double(rs)) / 16.0 +
                     double(rs) / 3.0;
  int tile_nodes = opts.tile_nodes;
  int n_sm = 152;
  if (!dry && cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, opts.device) != cudaSuccess) n_sm = 152;
  // 0 = auto: two tiles to an SM, so that a small population is spread over the whole GPU, up to the size that
  // ran best on large ones (FP32; FP64 tiles take twice the shared memory).  A step's time is its tile's latency:
  // 300 uneven cells ran 16.2 us a step in 900-node tiles; 16 cells of 129 nodes 6.6 us in three tiles.
  const bool auto_shape = tile_nodes <= 0 && s.n_ports == 0;
  if (auto_shape)
    tile_nodes = int(std::min<int64_t>(std::max<int64_t>((p->n_nodes + 2 * n_sm - 1) / (2 * n_sm), 128),
                                       opts.precision == BC_PREC_F64 ? 1250 : 2500));
  if (tile_nodes <= 0) tile_nodes = 900;
  tile_nodes = std::max(tile_nodes, 16);
  p->tile_nodes = tile_nodes;
  // A tile is never packed with more nodes than the arrays of (V), (alpha, beta) and row pairs and of indices leave
  // room for in shared memory: it would only be split again, and before that it might hold more separators than 16
  // bits count, or go to one cluster as a whole.
  tile_nodes = int(std::min<size_t>(tile_nodes, smem_budget / (6 * rs + 8)));
  // Launch classes: 0 = packed shared-memory tiles (cells <= tile_nodes), 1 = one big
  // cell per shared-memory tile, 2 = global-memory tiles (too big for shared memory).
  // (a thread for every pair of nodes and a warp for the heavy ones, up to 512: two such tiles fill an SM's registers)
  const int T_auto = auto_shape ? std::min(512, (tile_nodes / 2 + 31) / 32 * 32 + 32) : 128;
  const int T_packed = opts.threads_per_tile > 0 ? opts.threads_per_tile : T_auto;
  const int T_big = opts.threads_big > 0 ? opts.threads_big : (auto_shape ? 512 : 256);
  const int T_glob = opts.threads_global > 0 ? opts.threads_global : (s.n_ports > 0 ? BC_PORT_MAX_THREADS : 512);
  if (T_big % 32 || T_big > 1024 || T_glob % 32 || T_glob > 1024) {
    delete p;
    return fail(BC_ERR_INVALID, "thread counts must be multiples of 32 up to 1024");
  }
  if (s.n_ports > 0 && (T_packed > BC_PORT_MAX_THREADS || T_big > BC_PORT_MAX_THREADS || T_glob > BC_PORT_MAX_THREADS)) {
    delete p;
    return fail(BC_ERR_INVALID, "plans with surrogate ports run at most " + std::to_string(BC_PORT_MAX_THREADS) +
                                    " threads per tile");
  }
  int class_threads[kMaxClasses] = {T_packed, T_big, T_glob, kLaneThreads};
  std::vector<int64_t> order(s.n_cells);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(),
                   [&](int64_t a, int64_t b) { return cells[a].n_node > cells[b].n_node; });
  std::vector<TileBuild> builds;
  std::vector<int64_t> fill;
  // Lane tiles: cells of at most lane_cell_nodes tree nodes, kLaneThreads per tile
  // in decreasing size (a tile's threads then walk near-equal trees).  The lane
  // kernel runs the channels (out-of-line ones included when the plan has them) and
  // voltage probes, but no synapses, network, mechanism probes or ports.
  std::vector<char> in_lane(s.n_cells, 0);
  const bool lane_ok = !mech_probes && s.n_synapses == 0 && s.n_connections == 0 && s.n_ports == 0;
  if (opts.lane_cell_nodes > 0 && lane_ok) {
    std::vector<int64_t> lane_cells;
    for (int64_t c : order)
      if (cells[c].n_node <= opts.lane_cell_nodes) lane_cells.push_back(c);
    for (size_t q = 0; q < lane_cells.size(); q += kLaneThreads) {
      TileBuild tb;
      tb.cls = 3;
      for (size_t r = q; r < std::min(lane_cells.size(), q + kLaneThreads); ++r) {
        tb.cells.push_back(lane_cells[r]);
        in_lane[lane_cells[r]] = 1;
      }
      builds.push_back(tb);
      fill.push_back(0);
    }
  }
  // best-fit decreasing: each cell goes to the open packed tile with the least room
  // that still holds it (free room -> tile index), else opens a new tile
  std::multimap<int64_t, size_t> room;
  for (int64_t c : order) {
    if (in_lane[c]) continue;
    const int64_t nn = cells[c].n_node;
    if (nn > tile_nodes) {
      TileBuild tb;
      tb.cells.push_back(c);
      tb.cls = 1;
      builds.push_back(tb);
      fill.push_back(nn);
      continue;
    }
    auto it = room.lower_bound(nn);
    if (it != room.end()) {
      const size_t t = it->second;
      room.erase(it);
      builds[t].cells.push_back(c);
      fill[t] += nn;
      if (tile_nodes - fill[t] > 0 && builds[t].cells.size() < 4096) room.emplace(tile_nodes - fill[t], t);
      continue;
    }
    TileBuild tb;
    tb.cells.push_back(c);
    tb.cls = 0;
    builds.push_back(tb);
    fill.push_back(nn);
    if (tile_nodes - nn > 0) room.emplace(tile_nodes - nn, builds.size() - 1);
  }
  BuildCtx cx{&s, &cells, &sched, &cv_base, &cell_pulses, &cell_probes, &pulse_node, &probe_node, &cell_syns, &is_src,
              &cell_ports, &port_pulse_ids, p->precision, S,
              p->extra ? ((all_bits & BC_M_EXT) ? kParamStride : kParamStrideExtra) : kParamStrideCore};
  std::vector<TileOut> outs;
  outs.reserve(builds.size());
  // Packed tiles: tile_nodes sets how many CTAs share an SM (by the per-node
  // estimate); the shared-memory budget of one tile is then that SM's share, so
  // tiles fill up to tile_nodes without lowering the occupancy.
  const size_t per_sm = dry ? size_t(233472) : sm_smem(opts.device);
  const size_t cta_reserve = 2 * kStaticSmem;  // static shared memory + the system's per-CTA reserve
  // a tile with ports also holds the weight fragments of the GRU
  const size_t est = size_t(double(tile_nodes) * bpn) + 2048 + (s.n_ports > 0 ? size_t(kGruSmemBytes) : 0);
  const size_t ctas_per_sm = std::max<size_t>(1, per_sm / (est + cta_reserve));
  const size_t packed_budget =
      std::min(smem_budget, std::max(est, per_sm / ctas_per_sm > cta_reserve ? per_sm / ctas_per_sm - cta_reserve : est));
  // FP64 tiles that leave half of the SMs idle run as global-memory tiles, each on a cluster of CTAs: a step is bound
  // by the FP64 pipes of the SMs in use, not by where the tile lives (63 tiles of 2500 nodes: 197 us a step on one CTA
  // each, 159 on two; 20 cells of up to 2000: 154 on one, 103 on four).  FP32 tiles are bound by latency and stay.
  // The cluster grows while that takes a fifth off the largest load of an SM, in nodes: the largest tile's share, or
  // that of the CTAs an SM gets (clusters above two CTAs leave about an eighth of the SMs without one; the 63 tiles on
  // four CTAs each: 177 us).  A CTA of 128 nodes already has a warp for each of its four FP64 pipes, so
  // every CTA gets at least twice that.
  std::vector<int> cls_was;
  int want_cluster = 16;
  if (p->precision == BC_PREC_F64 && s.n_ports == 0 && !p->use_graph) {
    size_t n_tiles = 0;
    int64_t largest = 0, total = 0;
    for (size_t t = 0; t < builds.size(); ++t)
      if (builds[t].cls != 3) {
        ++n_tiles;
        largest = std::max(largest, fill[t]);
        total += fill[t];
      }
    const auto load = [&](int c) {
      const int64_t ctas = int64_t(n_tiles) * c, sms = c > 2 ? n_sm * 7 / 8 : n_sm;
      return std::max(double(largest) / c, double((ctas + sms - 1) / sms) * double(total) / double(ctas));
    };
    want_cluster = 1;
    for (int c = 2; c <= 16 && n_tiles > 0 && largest >= 256 * c && load(c) < 0.8 * load(c / 2); c *= 2) want_cluster = c;
    if (want_cluster > 1 && 2 * n_tiles <= size_t(n_sm)) {
      int asked = 0;  // CTA size that the caller gave for the tiles that move
      for (TileBuild& tb : builds) {
        cls_was.push_back(tb.cls);
        if (tb.cls < 2) asked = std::max(asked, tb.cls == 0 ? opts.threads_per_tile : opts.threads_big);
        if (tb.cls < 2) tb.cls = 2;
      }
      if (opts.threads_global <= 0 && asked > 0) class_threads[2] = asked;
    }
  }
  const auto global_cluster = [&]() {
    int count = 0;
    size_t bytes = 0;
    for (size_t t = 0; t < builds.size(); ++t) {
      if (builds[t].cls != 2) continue;
      const TileDesc& d = outs[t].desc;
      if (!d.sep_in_smem) return 1;
      ++count;
      bytes = std::max(bytes, size_t(d.sep_bytes) + size_t(d.off_rows - d.off_seps));
    }
    if (count == 0 || count > n_sm || s.n_ports > 0 || p->use_graph) return 1;
    if (dry) return 2;
    return tile_cluster(p->precision, p->extra ? BC_VARIANT_EXTRA : BC_VARIANT_LEAN, want_cluster, count,
                        class_threads[2], bytes);
  };
build_again:
  for (size_t t = 0; t < builds.size(); ++t) {
    TileOut to;
    bc_status st = build_tile(cx, builds[t], class_threads[builds[t].cls], to);
    if (st != BC_OK) {
      delete p;
      return st;
    }
    const size_t need = size_t(to.desc.blob_bytes) + size_t(to.desc.scratch_bytes);
    const size_t limit = builds[t].cls == 0 ? packed_budget : smem_budget;
    if (builds[t].cls < 2 && need > limit) {
      if (builds[t].cells.size() > 1) {
        // split: move the last cells into the best-fitting packed tiles not built yet
        // (or new ones) and rebuild this one.  As many cells move at once as the
        // overflow's share of the tile (at least one), so a tile of many small cells
        // whose per-cell records outgrow the node estimate is rebuilt a few times,
        // not once per cell.
        const size_t n_in = builds[t].cells.size();
        size_t n_move = size_t(std::ceil(double(n_in) * double(need - limit) / double(need)));
        n_move = std::max<size_t>(1, std::min(n_move, n_in - 1));
        for (size_t q = 0; q < n_move; ++q) {
          const int64_t c = builds[t].cells.back();
          const int64_t nn = cells[c].n_node;
          builds[t].cells.pop_back();
          fill[t] -= nn;
          size_t dest = builds.size();
          for (auto it = room.lower_bound(nn); it != room.end(); ++it)
            if (it->second > t) {
              dest = it->second;
              room.erase(it);
              break;
            }
          if (dest == builds.size()) {
            TileBuild nb;
            nb.cls = 0;
            builds.push_back(nb);
            fill.push_back(0);
          }
          builds[dest].cells.push_back(c);
          fill[dest] += nn;
          if (tile_nodes - fill[dest] > 0 && builds[dest].cells.size() < 4096) room.emplace(tile_nodes - fill[dest], dest);
        }
        --t;
        continue;
      }
      builds[t].cls = need > smem_budget ? 2 : 1;
      st = build_tile(cx, builds[t], class_threads[builds[t].cls], to);
      if (st != BC_OK) {
        delete p;
        return st;
      }
    }
    outs.push_back(std::move(to));
  }
  if (!cls_was.empty() && global_cluster() == 1) {  // no clusters after all: back to shared memory
    for (size_t t = 0; t < builds.size(); ++t) builds[t].cls = cls_was[t];
    cls_was.clear();
    class_threads[2] = T_glob;
    outs.clear();
    goto build_again;
  }
  p->threads = cls_was.empty() ? T_packed : class_threads[2];
  p->threads_global = class_threads[2];
  // tiles ordered by class; one launch per class
  std::vector<size_t> tord;
  for (int cl = 0; cl < kMaxClasses; ++cl) {
    LaunchClass lcz;
    lcz.first = int(tord.size());
    lcz.threads = class_threads[cl];
    lcz.smem = cl < 2;
    lcz.lane = cl == 3;
    for (size_t t = 0; t < builds.size(); ++t)
      if (builds[t].cls == cl) {
        tord.push_back(t);
        const size_t need = size_t(outs[t].desc.blob_bytes) + size_t(outs[t].desc.scratch_bytes);
        if (lcz.smem) lcz.smem_bytes = std::max(lcz.smem_bytes, need);
        const TileDesc& d = outs[t].desc;
        if (cl == 2 && d.sep_in_smem)
          lcz.smem_bytes = std::max(lcz.smem_bytes, size_t(d.sep_bytes) + size_t(d.off_rows - d.off_seps));
      }
    if (opts.tile_order == 1) {
      // longest estimated step first: the block scheduler hands out CTAs in index
      // order, so the tiles left for the last, partly filled wave are the short ones
      std::stable_sort(tord.begin() + lcz.first, tord.end(), [&](size_t x, size_t y) {
        if (outs[x].crit != outs[y].crit) return outs[x].crit > outs[y].crit;
        return outs[x].desc.n_real_nodes > outs[y].desc.n_real_nodes;
      });
    }
    lcz.count = int(tord.size()) - lcz.first;
    // few global-memory tiles: on each the largest cluster of CTAs at which they all run at once (one cell of 18,700
    // nodes: 127 us a step on one CTA, 41 on 16; 16 cells on clusters of 16, more than fit: 81)
    if (cl == 2) lcz.cluster = global_cluster();
    if (lcz.count > 0) p->classes.push_back(lcz);
  }
  p->n_smem_tiles = 0;
  for (auto& lcz : p->classes)
    if (lcz.smem) p->n_smem_tiles += lcz.count;
  // ---------------------------------------------------- concatenate + upload
  size_t blob_total = 0, scratch_total = 0, vinit_total = 0;
  int64_t state_total = 0;
  std::vector<int64_t> vinit_off;
  p->tiles.clear();
  std::vector<int2> cv_map(p->n_cv);
  for (size_t k = 0; k < tord.size(); ++k) {
    TileOut& to = outs[tord[k]];
    TileDesc d = to.desc;
    d.blob_offset = int64_t(blob_total);
    blob_total = align16(blob_total + d.blob_bytes);
    d.state_offset = state_total;
    state_total += int64_t(S) * d.n_nodes;
    if (builds[tord[k]].cls >= 2) {  // global-memory and lane tiles: solver scratch in HBM
      d.scratch_offset = int64_t(scratch_total);
      scratch_total = align16(scratch_total + d.scratch_bytes);
    } else {
      p->smem_bytes = std::max(p->smem_bytes, size_t(d.blob_bytes) + size_t(d.scratch_bytes));
    }
    d.pulse_offset = int64_t(p->pulses.size());
    d.n_pulses = int32_t(to.pulses.size());
    p->pulses.insert(p->pulses.end(), to.pulses.begin(), to.pulses.end());
    p->pulse_src.insert(p->pulse_src.end(), to.pulse_src.begin(), to.pulse_src.end());
    p->pulse_scale.insert(p->pulse_scale.end(), to.pulse_scale.begin(), to.pulse_scale.end());
    d.port_offset = int64_t(p->ports.size());
    d.n_ports = int32_t(to.ports.size());
    for (PortRec r : to.ports) {
      r.stim_begin += int32_t(p->port_pulses.size());
      r.stim_end += int32_t(p->port_pulses.size());
      p->ports.push_back(r);
    }
    p->port_pulses.insert(p->port_pulses.end(), to.port_pulses.begin(), to.port_pulses.end());
    vinit_off.push_back(int64_t(vinit_total));
    vinit_total += to.vinit.size();
    for (size_t q = 0; q < to.cv_local.size(); ++q) {
      cv_map[to.cv_local[q].first] = make_int2(int(k), to.cv_local[q].second);
    }
    p->max_phases = std::max<int64_t>(p->max_phases, d.n_phases);
    p->max_chain_nodes = std::max<int64_t>(p->max_chain_nodes, to.crit);
    p->tiles.push_back(d);
  }
  std::vector<unsigned char> blob(blob_total, 0);
  std::vector<double> vinit(vinit_total);
  for (size_t k = 0; k < tord.size(); ++k) {
    const TileOut& to = outs[tord[k]];
    std::memcpy(blob.data() + p->tiles[k].blob_offset, to.blob.data(), to.blob.size());
    std::copy(to.vinit.begin(), to.vinit.end(), vinit.begin() + vinit_off[k]);
  }
  std::vector<int64_t> outs_crit(outs.size());
  for (size_t q = 0; q < outs.size(); ++q) outs_crit[q] = outs[q].crit;
  outs.clear();
  bc_status st = BC_OK;
#define BC_TRY(x)          \
  do {                     \
    st = (x);              \
    if (st != BC_OK) {     \
      free_plan(p);        \
      return st;           \
    }                      \
  } while (0)
#define BC_TRYC(call)                                                                                \
  do {                                                                                               \
    cudaError_t e_ = (call);                                                                         \
    if (e_ != cudaSuccess) {                                                                         \
      free_plan(p);                                                                                  \
      return fail(BC_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_));                   \
    }                                                                                                \
  } while (0)
  p->tile_stats.clear();
  for (size_t k = 0; k < tord.size(); ++k) {
    const TileDesc& d = p->tiles[k];
    p->tile_stats.push_back({int64_t(d.n_real_nodes), int64_t(d.n_segs), int64_t(d.n_phases),
                             int64_t(outs_crit[tord[k]]), int64_t(builds[tord[k]].cls),
                             int64_t(d.blob_bytes) + int64_t(d.scratch_bytes)});
  }
  if (dry) {
    *out = p;
    return BC_OK;
  }
  p->blob_bytes = blob_total;
  p->scratch_bytes = scratch_total;
  for (const LaunchClass& lcz : p->classes)
    if (!lcz.lane) BC_TRYC(cudaError_t(prepare_tiles(p->precision, lcz.smem, kernel_variant(p))));
  BC_TRY(dalloc(p, &p->d_blob, blob_total));
  BC_TRY(dalloc(p, &p->d_scratch, scratch_total));
  p->state_bytes = size_t(state_total) * rs;
  BC_TRY(dalloc(p, &p->d_state, p->state_bytes));
  BC_TRY(dalloc(p, &p->d_tiles, p->tiles.size()));
  BC_TRY(dalloc(p, &p->d_pulses, p->pulses.size()));
  BC_TRY(dalloc(p, &p->d_vinit, vinit.size()));
  BC_TRY(dalloc(p, &p->d_vinit_off, vinit_off.size()));
  BC_TRY(dalloc(p, &p->d_spike_count, size_t(p->n_probes)));
  BC_TRY(dalloc(p, &p->d_spike_times, size_t(p->n_probes) * std::max(1, p->max_spikes)));
  BC_TRY(dalloc(p, &p->d_status, 1));
  BC_TRY(dalloc(p, &p->d_timers, 4));
  BC_TRYC(cudaMemset(p->d_timers, 0, 4 * sizeof(unsigned long long)));
  BC_TRYC(cudaMemcpy(p->d_blob, blob.data(), blob_total, cudaMemcpyHostToDevice));
  BC_TRY(dalloc(p, &p->d_cv, size_t(p->n_cv)));
  BC_TRY(dalloc(p, &p->d_view, size_t(p->n_cv)));
  BC_TRYC(cudaMemcpy(p->d_cv, cv_map.data(), cv_map.size() * sizeof(int2), cudaMemcpyHostToDevice));
  if (!p->pulses.empty()) {
    const std::vector<int32_t> src(p->pulse_src.begin(), p->pulse_src.end());
    BC_TRY(dalloc(p, &p->d_pulse_src, src.size()));
    BC_TRY(dalloc(p, &p->d_pulse_scale, src.size()));
    BC_TRY(dalloc(p, &p->d_pulse_amp, size_t(p->n_pulses)));
    BC_TRYC(cudaMemcpy(p->d_pulse_src, src.data(), src.size() * 4, cudaMemcpyHostToDevice));
    BC_TRYC(cudaMemcpy(p->d_pulse_scale, p->pulse_scale.data(), src.size() * 8, cudaMemcpyHostToDevice));
  }
  BC_TRYC(cudaMemcpy(p->d_tiles, p->tiles.data(), p->tiles.size() * sizeof(TileDesc), cudaMemcpyHostToDevice));
  BC_TRYC(cudaMemcpy(p->d_vinit, vinit.data(), vinit.size() * sizeof(double), cudaMemcpyHostToDevice));
  BC_TRYC(cudaMemcpy(p->d_vinit_off, vinit_off.data(), vinit_off.size() * sizeof(int64_t), cudaMemcpyHostToDevice));
  BC_TRYC(cudaMemset(p->d_status, 0, sizeof(int32_t)));
  {
    // synapse parameters and the connection CSR, in the plan's precision
    auto up_real = [&](void** dst, const std::vector<double>& src) -> bc_status {
      const size_t n = std::max<size_t>(src.size(), 1);
      cudaError_t e = cudaMalloc(dst, n * rs);
      if (e != cudaSuccess) return fail(BC_ERR_CUDA, std::string("cudaMalloc: ") + cudaGetErrorString(e));
      p->device_bytes += n * rs;
      std::vector<unsigned char> tmp(n * rs, 0);
      for (size_t k = 0; k < src.size(); ++k) {
        if (rs == 8)
          std::memcpy(tmp.data() + k * 8, &src[k], 8);
        else {
          const float f = float(src[k]);
          std::memcpy(tmp.data() + k * 4, &f, 4);
        }
      }
      e = cudaMemcpy(*dst, tmp.data(), n * rs, cudaMemcpyHostToDevice);
      if (e != cudaSuccess) return fail(BC_ERR_CUDA, std::string("cudaMemcpy: ") + cudaGetErrorString(e));
      return BC_OK;
    };
    BC_TRY(up_real(&p->d_syn_g, std::vector<double>(p->n_synapses, 0.0)));
    BC_TRY(up_real(&p->d_syn_tau, p->syn_tau));
    BC_TRY(up_real(&p->d_syn_e, p->syn_e));
    BC_TRY(up_real(&p->d_syn_scale, p->syn_scale));
    BC_TRY(up_real(&p->d_out_w, p->out_w));
    BC_TRY(dalloc(p, &p->d_out_ptr, p->out_ptr.size()));
    BC_TRY(dalloc(p, &p->d_out_syn, p->out_syn.size()));
    BC_TRY(dalloc(p, &p->d_out_d, size_t(p->n_connections)));
    BC_TRYC(cudaMemcpy(p->d_out_ptr, p->out_ptr.data(), p->out_ptr.size() * 8, cudaMemcpyHostToDevice));
    if (p->n_connections > 0)
      BC_TRYC(cudaMemcpy(p->d_out_syn, p->out_syn.data(), p->out_syn.size() * 8, cudaMemcpyHostToDevice));
    int64_t n_src = 0;
    for (int64_t c = 0; c + 1 < int64_t(p->out_ptr.size()); ++c) n_src += p->out_ptr[c + 1] > p->out_ptr[c];
    p->rec_cap = p->n_connections > 0 ? std::max<int64_t>(int64_t(1) << 16, 256 * n_src) : 1;
    BC_TRY(dalloc(p, &p->d_rec_cell, size_t(p->rec_cap)));
    BC_TRY(dalloc(p, &p->d_rec_step, size_t(p->rec_cap)));
    BC_TRY(dalloc(p, &p->d_rec_count, 2));
    BC_TRYC(cudaMemset(p->d_rec_count, 0, 2 * sizeof(unsigned long long)));
  }
  if (p->n_ports > 0) {
    BC_TRY(dalloc(p, &p->d_ports, p->ports.size()));
    BC_TRY(dalloc(p, &p->d_port_pulses, std::max<size_t>(p->port_pulses.size(), 1)));
    BC_TRY(dalloc(p, &p->d_port_h, size_t(p->n_ports) * kPortStride));
    BC_TRY(dalloc(p, &p->d_port_flags, size_t(p->n_cells)));
    BC_TRY(dalloc(p, &p->d_gru, 1));
    BC_TRYC(cudaMemcpy(p->d_ports, p->ports.data(), p->ports.size() * sizeof(PortRec), cudaMemcpyHostToDevice));
  }
  if (p->n_smem_tiles > 0 && p->smem_bytes + kStaticSmem > smem_cap) {
    free_plan(p);
    return fail(BC_ERR_CAPACITY, "tile shared memory exceeds the device limit");
  }
  for (int k = 0; k < kMaxClasses - 1; ++k) {
    BC_TRYC(cudaStreamCreateWithFlags(&p->aux[k], cudaStreamNonBlocking));
    BC_TRYC(cudaEventCreateWithFlags(&p->ev_join[k], cudaEventDisableTiming));
  }
  BC_TRYC(cudaEventCreateWithFlags(&p->ev_fork, cudaEventDisableTiming));
  int prio_least = 0, prio_greatest = 0;
  BC_TRYC(cudaDeviceGetStreamPriorityRange(&prio_least, &prio_greatest));
  BC_TRYC(cudaStreamCreateWithPriority(&p->init_stream, cudaStreamNonBlocking, prio_greatest));
  *out = p;
  // The initial reset runs on the plan's own non-blocking stream of the highest
  // priority: creating a plan waits neither for work other plans have queued on
  // the legacy stream nor, behind their pending blocks, for free SM slots.
  return bc_reset(p, p->init_stream);
}

bc_status bc_lower_cell(const bc_batch_spec* spec, int64_t cell, int32_t* n_cv, int32_t* n_node, double* cv_area,
                        int32_t* cv_node, int32_t* parent, double* alpha, double* beta, double* diag,
                        int32_t* region) {
  if (!spec || !n_cv || !n_node) return fail(BC_ERR_INVALID, "null argument");
  if (cell < 0 || cell >= spec->n_cells) return fail(BC_ERR_INVALID, "cell out of range");
  LoweredCell lc;
  bc_status st = lower_cell(*spec, cell, lc);
  if (st != BC_OK) return st;
  *n_cv = lc.n_cv;
  *n_node = lc.n_node;
  if (cv_area) std::copy(lc.cv_area.begin(), lc.cv_area.end(), cv_area);
  if (cv_node) std::copy(lc.cv_node.begin(), lc.cv_node.end(), cv_node);
  if (parent) std::copy(lc.parent.begin(), lc.parent.end(), parent);
  if (alpha) std::copy(lc.alpha.begin(), lc.alpha.end(), alpha);
  if (beta) std::copy(lc.beta.begin(), lc.beta.end(), beta);
  if (diag) std::copy(lc.diag.begin(), lc.diag.end(), diag);
  if (region) std::copy(lc.region.begin(), lc.region.end(), region);
  return BC_OK;
}

bc_status bc_plan_destroy(bc_plan_t p) {
  if (!p) return fail(BC_ERR_INVALID, "null plan");
  free_plan(p);
  return BC_OK;
}

bc_status bc_plan_info(bc_plan_t p, bc_plan_info_t* info) {
  if (!p || !info) return fail(BC_ERR_INVALID, "null argument");
  std::memset(info, 0, sizeof(*info));
  info->n_cells = p->n_cells;
  info->n_cv = p->n_cv;
  info->n_nodes = p->n_nodes;
  info->n_tiles = int64_t(p->tiles.size());
  info->n_probes = p->n_probes;
  info->n_pulses = p->n_pulses;
  info->threads_per_tile = p->threads;
  info->tile_nodes = p->tile_nodes;
  info->steps_per_launch = p->steps_per_launch;
  info->precision = p->precision;
  info->smem_bytes_per_tile = int64_t(p->smem_bytes);
  info->device_bytes = int64_t(p->device_bytes);
  info->max_phases = p->max_phases;
  info->max_chain_nodes = p->max_chain_nodes;
  info->state_slots = p->state_slots;
  info->n_smem_tiles = int32_t(p->n_smem_tiles);
  info->n_launch_classes = int32_t(p->classes.size());
  info->kernel_variant = kernel_variant(p);
  return BC_OK;
}

bc_status bc_plan_cell_ncv(bc_plan_t p, int64_t* ncv) {
  if (!p || !ncv) return fail(BC_ERR_INVALID, "null argument");
  std::copy(p->cell_ncv.begin(), p->cell_ncv.end(), ncv);
  return BC_OK;
}

#define BC_NEED_DEVICE(p) \
  if ((p)->dry) return fail(BC_ERR_INVALID, "plan was created with dry_run; it has no device state")

bc_status bc_reset(bc_plan_t p, void* stream) {
  if (!p) return fail(BC_ERR_INVALID, "null plan");
  BC_NEED_DEVICE(p);
  BC_CUDA(cudaSetDevice(p->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  LaunchArgs a = base_args(p);
  a.tiles = p->d_tiles;
  a.n_tiles = int32_t(p->tiles.size());
  int e = launch_reset_impl(a, p->precision, 256, p->d_vinit, p->d_vinit_off, stream);
  if (e) return fail(BC_ERR_CUDA, std::string("reset kernel: ") + cudaGetErrorString(cudaError_t(e)));
  if (p->n_probes > 0) {
    BC_CUDA(cudaMemsetAsync(p->d_spike_count, 0, size_t(p->n_probes) * sizeof(int32_t), st));
  }
  BC_CUDA(cudaMemsetAsync(p->d_status, 0, sizeof(int32_t), st));
  if (p->n_synapses > 0) BC_CUDA(cudaMemsetAsync(p->d_syn_g, 0, size_t(p->n_synapses) * p->real_size, st));
  if (p->d_arrivals)
    BC_CUDA(cudaMemsetAsync(p->d_arrivals, 0,
                            size_t(p->arr_slots) * size_t(std::max<int64_t>(p->n_synapses, 1)) * p->real_size, st));
  BC_CUDA(cudaMemsetAsync(p->d_rec_count, 0, 2 * sizeof(unsigned long long), st));
  if (p->n_ports > 0) {
    BC_CUDA(cudaMemsetAsync(p->d_port_h, 0, size_t(p->n_ports) * kPortStride * sizeof(float), st));
    BC_CUDA(cudaMemsetAsync(p->d_port_flags, 0, size_t(p->n_cells) * sizeof(int32_t), st));
  }
  BC_CUDA(cudaStreamSynchronize(st));
  p->step = 0;
  p->trace_origin = 0;
  return BC_OK;
}

bc_status bc_network_spikes(bc_plan_t p, int32_t* cells, int64_t* steps, int64_t cap, int64_t* n_out,
                            void* stream) {
  if (!p || !n_out || (cap > 0 && (!cells || !steps))) return fail(BC_ERR_INVALID, "null argument");
  BC_NEED_DEVICE(p);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  unsigned long long n = 0;
  BC_CUDA(cudaMemcpyAsync(&n, p->d_rec_count, sizeof(n), cudaMemcpyDeviceToHost, s));
  BC_CUDA(cudaStreamSynchronize(s));
  *n_out = int64_t(n);
  const int64_t m = std::min<int64_t>(std::min<int64_t>(int64_t(n), cap), p->rec_cap);
  if (m > 0) {
    BC_CUDA(cudaMemcpyAsync(cells, p->d_rec_cell, size_t(m) * 4, cudaMemcpyDeviceToHost, s));
    BC_CUDA(cudaMemcpyAsync(steps, p->d_rec_step, size_t(m) * 8, cudaMemcpyDeviceToHost, s));
    BC_CUDA(cudaStreamSynchronize(s));
  }
  return BC_OK;
}

// BF16 of a finite float, round to nearest even (as the device conversion).
static uint16_t bf16_rne(float f) {
  uint32_t u;
  std::memcpy(&u, &f, 4);
  u += 0x7fffu + ((u >> 16) & 1u);
  return uint16_t(u >> 16);
}

bc_status bc_surrogate_set(bc_plan_t p, const float* params, const float* norm, void* stream) {
  if (!p || !params || !norm) return fail(BC_ERR_INVALID, "null argument");
  if (p->n_ports == 0) return fail(BC_ERR_INVALID, "the plan has no surrogate ports");
  BC_NEED_DEVICE(p);
  BC_CUDA(cudaSetDevice(p->device));
  for (int k = 0; k < kGruNParam; ++k)
    if (!std::isfinite(params[k])) return fail(BC_ERR_INVALID, "non-finite GRU parameter");
  const float v_scale = norm[0], y_scale = norm[1], lo = norm[2], hi = norm[3], dvdt = norm[4];
  if (!(v_scale > 0.f) || !std::isfinite(v_scale) || !std::isfinite(y_scale) || !(hi >= lo) || !(dvdt > 0.f))
    return fail(BC_ERR_INVALID, "surrogate norm: v_scale > 0, finite y_scale, env_v_hi >= env_v_lo, env_dvdt > 0");
  // the extended weight matrix, as gru_pack_kernel builds it for training
  auto bf = [](float f) {
    const uint32_t u = uint32_t(bf16_rne(f)) << 16;
    float r;
    std::memcpy(&r, &u, 4);
    return r;
  };
  auto value = [&](int n, int k) -> float {
    const int q = n / kGruH, u = n % kGruH;
    if (k < kGruH) return q < 3 ? params[kGruOffWh + (q * kGruH + u) * kGruH + k] : 0.0f;
    const int c = k - kGruH;
    const int xrow = q == 0 ? u : q == 1 ? kGruH + u : 2 * kGruH + u;
    if (c < 2 * kGruX) return q == 2 ? 0.0f : bf(params[kGruOffWx + xrow * kGruX + (c % kGruX)]);
    if (c < 2 * kGruX + 2) {
      const float bsum = q == 0   ? params[kGruOffBx + u] + params[kGruOffBh + u]
                         : q == 1 ? params[kGruOffBx + kGruH + u] + params[kGruOffBh + kGruH + u]
                         : q == 2 ? params[kGruOffBh + 2 * kGruH + u]
                                  : params[kGruOffBx + 2 * kGruH + u];
      const float hi = bf(bsum);
      return c == 2 * kGruX ? hi : bsum - hi;
    }
    return 0.0f;
  };
  GruWeights w{};
  for (int n = 0; n < kGruRows; ++n)
    for (int k = 0; k < kGruK; k += 2)
      w.wext[(n * kGruK + k) / 2] = uint32_t(bf16_rne(value(n, k))) | (uint32_t(bf16_rne(value(n, k + 1))) << 16);
  std::memcpy(w.wo, params + kGruOffWo, sizeof(w.wo));
  w.bo = params[kGruOffBo];
  w.v_scale = v_scale;
  w.y_scale = y_scale;
  w.env_v_lo = lo;
  w.env_v_hi = hi;
  w.env_dvdt = dvdt;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  BC_CUDA(cudaMemcpyAsync(p->d_gru, &w, sizeof(w), cudaMemcpyHostToDevice, st));
  BC_CUDA(cudaStreamSynchronize(st));
  p->gru_set = true;
  return BC_OK;
}

bc_status bc_surrogate_flags(bc_plan_t p, int32_t* flags, void* stream) {
  if (!p || !flags) return fail(BC_ERR_INVALID, "null argument");
  if (p->n_ports == 0) {
    std::fill(flags, flags + p->n_cells, 0);
    return BC_OK;
  }
  BC_NEED_DEVICE(p);
  BC_CUDA(cudaSetDevice(p->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  BC_CUDA(cudaMemcpyAsync(flags, p->d_port_flags, size_t(p->n_cells) * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  BC_CUDA(cudaStreamSynchronize(st));
  return BC_OK;
}

bc_status bc_synapse_download(bc_plan_t p, double* g, void* stream) {
  if (!p || (!g && p->n_synapses > 0)) return fail(BC_ERR_INVALID, "null argument");
  BC_NEED_DEVICE(p);
  if (p->n_synapses == 0) return BC_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  std::vector<unsigned char> tmp(size_t(p->n_synapses) * p->real_size);
  BC_CUDA(cudaMemcpyAsync(tmp.data(), p->d_syn_g, tmp.size(), cudaMemcpyDeviceToHost, s));
  BC_CUDA(cudaStreamSynchronize(s));
  for (int64_t k = 0; k < p->n_synapses; ++k) {
    if (p->real_size == 8) {
      std::memcpy(&g[k], tmp.data() + k * 8, 8);
    } else {
      float f;
      std::memcpy(&f, tmp.data() + k * 4, 4);
      g[k] = double(f);
    }
  }
  return BC_OK;
}

bc_status bc_check(bc_plan_t p, void* stream) {
  if (!p) return fail(BC_ERR_INVALID, "null plan");
  BC_NEED_DEVICE(p);
  int32_t status = 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  BC_CUDA(cudaMemcpyAsync(&status, p->d_status, sizeof(int32_t), cudaMemcpyDeviceToHost, st));
  BC_CUDA(cudaStreamSynchronize(st));
  if (status & 2) return fail(BC_ERR_TIMEOUT, "a bounded device wait gave up (bulk copy did not complete)");
  if (status & 4) return fail(BC_ERR_CAPACITY, "the spike record buffer of the network run overflowed");
  if (status & 1) return fail(BC_ERR_NONFINITE, "non-finite membrane voltage");
  return BC_OK;
}

bc_status bc_run_async(bc_plan_t p, int64_t n_steps, double dt, void* stream) {
  if (!p) return fail(BC_ERR_INVALID, "null plan");
  BC_NEED_DEVICE(p);
  BC_CUDA(cudaSetDevice(p->device));
  return enqueue_run(p, n_steps, dt, stream);
}

bc_status bc_run(bc_plan_t p, int64_t n_steps, double dt, void* stream) {
  bc_status st = bc_run_async(p, n_steps, dt, stream);
  if (st != BC_OK) return st;
  return bc_check(p, stream);
}

bc_status bc_run_timed(bc_plan_t p, int64_t n_steps, double dt, void* stream, double* ms_out) {
  if (!p || !ms_out) return fail(BC_ERR_INVALID, "null argument");
  BC_NEED_DEVICE(p);
  BC_CUDA(cudaSetDevice(p->device));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // prepare tables outside the timed region
  bc_status s0 = update_pulses(p, dt, stream);
  if (s0 != BC_OK) return s0;
  const int64_t recs = p->record_every > 0 ? (p->step + n_steps - p->trace_origin) / p->record_every : 0;
  s0 = ensure_traces(p, recs, stream);
  if (s0 != BC_OK) return s0;
  cudaEvent_t e0, e1;
  BC_CUDA(cudaEventCreate(&e0));
  BC_CUDA(cudaEventCreate(&e1));
  BC_CUDA(cudaEventRecord(e0, st));
  bc_status s1 = enqueue_run(p, n_steps, dt, stream);
  BC_CUDA(cudaEventRecord(e1, st));
  BC_CUDA(cudaEventSynchronize(e1));
  float ms = 0.f;
  BC_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  *ms_out = ms;
  if (s1 != BC_OK) return s1;
  return bc_check(p, stream);
}

static bc_status view_args(int32_t which, int32_t mode, ViewArgs* va) {
  if (which < 0 || which >= BC_NSTATE_VIEW) return fail(BC_ERR_INVALID, "unknown state view");
  *va = ViewArgs{mode, -1, -1, 0, 0.0};
  if (which == BC_STATE_V) return BC_OK;
  uint64_t bit = 0;
  int slot = -1;
  state_view(which, &bit, &slot);
  va->slot = slot;
  if (which == BC_STATE_V_LAST) {
    va->slot_lo = kSlotVLastLo;
  } else {
    va->owner = bit;
    if (which == BC_STATE_CA_CI) va->slot_lo = kSlotCaLo;
  }
  return BC_OK;
}

static bc_status view_io(bc_plan* p, const ViewArgs& va, double* host, void* stream) {
  BC_CUDA(cudaSetDevice(p->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t bytes = size_t(p->n_cv) * 8;
  std::lock_guard<std::mutex> lock(p->view_mu);
  cudaError_t e = cudaSuccess;
  if (va.mode == kViewWrite) e = cudaMemcpyAsync(p->d_view, host, bytes, cudaMemcpyHostToDevice, s);
  int ke = 0;
  if (e == cudaSuccess)
    ke = launch_view_impl(p->d_tiles, p->d_blob, p->d_state, p->precision, p->d_cv, va, p->d_view, p->n_cv, stream);
  if (e == cudaSuccess && !ke && va.mode != kViewWrite)
    e = cudaMemcpyAsync(host, p->d_view, bytes, cudaMemcpyDeviceToHost, s);
  const cudaError_t es = cudaStreamSynchronize(s);  // also after a failure: nothing of this call outlives the lock
  if (ke) return fail(BC_ERR_CUDA, std::string("view kernel: ") + cudaGetErrorString(cudaError_t(ke)));
  if (e == cudaSuccess) e = es;
  if (e != cudaSuccess) return fail(BC_ERR_CUDA, std::string("state view: ") + cudaGetErrorString(e));
  return BC_OK;
}

static bc_status view_call(bc_plan* p, int32_t which, int32_t mode, double* host, void* stream) {
  if (!p || !host) return fail(BC_ERR_INVALID, "null argument");
  BC_NEED_DEVICE(p);
  ViewArgs va;
  const bc_status st = view_args(which, mode, &va);
  return st == BC_OK ? view_io(p, va, host, stream) : st;
}

bc_status bc_state_download(bc_plan_t p, int32_t which, double* out, void* stream) {
  return view_call(p, which, kViewRead, out, stream);
}

bc_status bc_state_upload(bc_plan_t p, int32_t which, const double* in, void* stream) {
  return view_call(p, which, kViewWrite, const_cast<double*>(in), stream);
}

bc_status bc_pulse_set_amp(bc_plan_t p, const double* amp_nA, void* stream) {
  if (!p || (!amp_nA && p->n_pulses > 0)) return fail(BC_ERR_INVALID, "null argument");
  BC_NEED_DEVICE(p);
  if (p->pulses.empty()) return BC_OK;
  BC_CUDA(cudaSetDevice(p->device));
  for (int64_t q = 0; q < p->n_pulses; ++q)
    if (!std::isfinite(amp_nA[q])) return fail(BC_ERR_INVALID, "bc_pulse_set_amp: non-finite amplitude");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  p->pulse_amp.assign(amp_nA, amp_nA + p->n_pulses);
  BC_CUDA(cudaMemcpyAsync(p->d_pulse_amp, p->pulse_amp.data(), p->pulse_amp.size() * 8, cudaMemcpyHostToDevice, st));
  const int ke = launch_pulse_amp_impl(p->d_pulses, p->d_pulse_src, p->d_pulse_scale, p->d_pulse_amp,
                                       int64_t(p->pulses.size()), stream);
  if (ke) return fail(BC_ERR_CUDA, std::string("pulse amplitude kernel: ") + cudaGetErrorString(cudaError_t(ke)));
  BC_CUDA(cudaStreamSynchronize(st));
  return BC_OK;
}

bc_status bc_spike_state_download(bc_plan_t p, double v_th, double* out, void* stream) {
  if (!p || !out) return fail(BC_ERR_INVALID, "null argument");
  BC_NEED_DEVICE(p);
  return view_io(p, ViewArgs{kViewSpike, -1, -1, 0, v_th}, out, stream);
}

// ------------------------------------------------------------------ no-allocation download
constexpr int kNoAllocDevices = 64;
static unsigned char* g_noalloc_scratch[kNoAllocDevices];
static std::mutex g_noalloc_setup_mu;

// One-time (per device) lookup of the scratch address; the caller has set the device.
static bc_status noalloc_scratch(int device, unsigned char** out) {
  if (device < 0 || device >= kNoAllocDevices) return fail(BC_ERR_INVALID, "device ordinal out of range");
  std::lock_guard<std::mutex> lock(g_noalloc_setup_mu);
  if (!g_noalloc_scratch[device]) {
    void* addr = nullptr;
    const int e = noalloc_view_scratch_address(&addr);
    if (e != 0 || !addr)
      return fail(BC_ERR_CUDA, std::string("cudaGetSymbolAddress(no-allocation scratch): ") +
                                   cudaGetErrorString(cudaError_t(e)));
    g_noalloc_scratch[device] = static_cast<unsigned char*>(addr);
  }
  *out = g_noalloc_scratch[device];
  return BC_OK;
}

bc_status bc_state_download_noalloc(bc_plan_t p, int32_t which, double* out, void* stream) {
  if (!p || !out) return fail(BC_ERR_INVALID, "null argument");
  if (which < 0 || which >= BC_NSTATE_VIEW) return fail(BC_ERR_INVALID, "unknown state view");
  if (p->n_cv > BC_NOALLOC_MAX_CV)
    return fail(BC_ERR_INVALID, "bc_state_download_noalloc: plan has " + std::to_string(p->n_cv) +
                                    " CVs, above the fixed scratch capacity of " +
                                    std::to_string(BC_NOALLOC_MAX_CV) +
                                    " (BC_NOALLOC_MAX_CV); use bc_state_download");
  BC_NEED_DEVICE(p);
  BC_CUDA(cudaSetDevice(p->device));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // The call copies to pageable host memory and synchronises the stream, and
  // neither is allowed while the stream is being captured into a graph.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  BC_CUDA(cudaStreamIsCapturing(s, &cap));
  if (cap != cudaStreamCaptureStatusNone)
    return fail(BC_ERR_INVALID, "bc_state_download_noalloc: the stream is being captured; call it outside capture");
  unsigned char* scratch = nullptr;
  bc_status st = noalloc_scratch(p->device, &scratch);
  if (st != BC_OK) return st;
  const int64_t n = p->n_cv;
  if (n == 0) return BC_OK;
  ViewArgs va;
  st = view_args(which, kViewRead, &va);
  if (st != BC_OK) return st;
  // entries [0, n) are written by the view kernel (NaN for absent states) before they are read
  double* d_val = reinterpret_cast<double*>(scratch);
  // Once something is enqueued, every return waits for the stream first, so that
  // no copy or kernel of this call still uses the shared scratch when the next,
  // serialised call (perhaps on another stream) writes it.
  auto failed = [&](const std::string& what, cudaError_t e) {
    (void)cudaStreamSynchronize(s);
    return fail(BC_ERR_CUDA, what + ": " + cudaGetErrorString(e));
  };
  const int ke = launch_view_impl(p->d_tiles, p->d_blob, p->d_state, p->precision, p->d_cv, va, d_val, n, stream);
  if (ke) return failed("view kernel", cudaError_t(ke));
  cudaError_t e = cudaMemcpyAsync(out, d_val, size_t(n) * 8, cudaMemcpyDeviceToHost, s);
  if (e != cudaSuccess) return failed("value download", e);
  e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail(BC_ERR_CUDA, std::string("cudaStreamSynchronize: ") + cudaGetErrorString(e));
  return BC_OK;
}

bc_status bc_probe_count(bc_plan_t p, int64_t* n) {
  if (!p || !n) return fail(BC_ERR_INVALID, "null argument");
  *n = p->record_every > 0 ? (p->step - p->trace_origin) / p->record_every : 0;
  if (*n > p->trace_cap) *n = p->trace_cap;
  return BC_OK;
}

bc_status bc_probe_download(bc_plan_t p, double* traces, int64_t max_records, void* stream) {
  if (!p || (!traces && max_records > 0)) return fail(BC_ERR_INVALID, "null argument");
  int64_t n = 0;
  bc_probe_count(p, &n);
  n = std::min(n, max_records);
  if (n <= 0 || p->n_probes == 0) return BC_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  BC_CUDA(cudaMemcpyAsync(traces, p->d_traces, size_t(n) * p->n_probes * sizeof(double), cudaMemcpyDeviceToHost, s));
  BC_CUDA(cudaStreamSynchronize(s));
  return BC_OK;
}

bc_status bc_spike_download(bc_plan_t p, int32_t* counts, double* times, void* stream) {
  if (!p) return fail(BC_ERR_INVALID, "null plan");
  if (p->n_probes == 0) return BC_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (counts)
    BC_CUDA(cudaMemcpyAsync(counts, p->d_spike_count, size_t(p->n_probes) * 4, cudaMemcpyDeviceToHost, s));
  if (times && p->max_spikes > 0)
    BC_CUDA(cudaMemcpyAsync(times, p->d_spike_times, size_t(p->n_probes) * p->max_spikes * 8, cudaMemcpyDeviceToHost, s));
  BC_CUDA(cudaStreamSynchronize(s));
  return BC_OK;
}

bc_status bc_probe_clear(bc_plan_t p, void* stream) {
  if (!p) return fail(BC_ERR_INVALID, "null plan");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (p->n_probes > 0) BC_CUDA(cudaMemsetAsync(p->d_spike_count, 0, size_t(p->n_probes) * 4, s));
  BC_CUDA(cudaStreamSynchronize(s));
  p->trace_origin = p->step;
  return BC_OK;
}

bc_status bc_plan_tile_stats(bc_plan_t p, int64_t* out) {
  if (!p || !out) return fail(BC_ERR_INVALID, "null argument");
  for (size_t k = 0; k < p->tile_stats.size(); ++k)
    for (int j = 0; j < 6; ++j) out[k * 6 + j] = p->tile_stats[k][j];
  return BC_OK;
}

bc_status bc_debug_phase_cycles(bc_plan_t p, uint64_t* out4, int32_t reset) {
  if (!p || !out4) return fail(BC_ERR_INVALID, "null argument");
  BC_NEED_DEVICE(p);
  BC_CUDA(cudaMemcpy(out4, p->d_timers, 4 * sizeof(uint64_t), cudaMemcpyDeviceToHost));
  if (reset) BC_CUDA(cudaMemset(p->d_timers, 0, 4 * sizeof(uint64_t)));
  return BC_OK;
}

bc_status bc_step_count(bc_plan_t p, int64_t* steps) {
  if (!p || !steps) return fail(BC_ERR_INVALID, "null argument");
  *steps = p->step;
  return BC_OK;
}

}  // extern "C"
