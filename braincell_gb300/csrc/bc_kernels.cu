// sm_103a kernels of the multi-compartment Cell time step.
//
// One CTA owns one tile (one or more whole cells).  For shared-memory tiles the
// tile's blob (voltages, axial coefficients, segment schedule, parameter records)
// is staged into shared memory with TMA bulk copies (cp.async.bulk + mbarrier),
// stays resident for `n_steps` fused time steps, and only the voltages are
// written back with a bulk store.  Mechanism states (gates, calcium) stream from
// a global [slot][node] array, read and written once per node per step.  Tiles
// too large for shared memory run the same code on their global-memory blob.
//
// Per time step (reference: quad/_staggered.py:54-154):
//   segment elimination   -- every unbranched run of nodes between two separators
//                            (branch points, the root, cuts of long runs) is
//                            eliminated by one lane, all runs of the tile at once;
//   separator sweep       -- the small tree of separators, leaf -> root and back
//                            (comp_triang_raw, :641-657; comp_backsub_raw, :742-760),
//                            a warp per group of cells;
//   per-node update       -- V += delta (float-float), CalciumDetailed Ci from the
//                            step-start current (cell.py:2261-2280, ion/calcium.py:
//                            499-505), gates by exp-Euler at the new V (cell.py:
//                            2157-2217), the next step's linearised row
//                            (_staggered.py:449-513, cell.py:1907-1963), clamp
//                            pulses (_compute/layouts.py:960-982) and probes.
// The voltage system is solved for the increment x = V_{n+1} - V_n; with the same
// matrix this gives the same V_{n+1} as the reference's direct form, and in FP32
// it keeps V to ~1e-5 mV over thousands of steps.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "bc_gru.cuh"
#include "bc_internal.h"
#include "bc_mech.cuh"
#include "bc_ext.cuh"

namespace bc {

constexpr int kStatusNonfinite = 1;
constexpr int kStatusTimeout = 2;
constexpr int kStatusRecordOverflow = 4;
constexpr uint16_t kBoundary = 0xFFFF;
constexpr uint16_t kNoSpecial = 0xFFFF;

// ------------------------------------------------------------------ TMA helpers
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

// Bounded wait on phase `parity`; returns false if it gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint32_t max_iter) {
  for (uint32_t it = 0; it < max_iter; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void bulk_s2g(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(src)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void bulk_commit_and_wait() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

constexpr uint32_t kBulkChunk = 32768;  // bytes per bulk copy instruction (multiple of 16)

// A separator's row after the elimination of the segment above it: excess e, rhs r,
// the coupling a to the upper separator and the coupling b of this separator in the
// upper separator's row (a = b = 0 at a root).
template <typename Real>
struct alignas(16) SepRow {
  Real e, r, a, b;
};
// Two inbox entries, read together.
template <typename Real>
struct alignas(16) InPair {
  Real e0, r0, e1, r1;
};

// ------------------------------------------------------------------ tile view
// Per-node pairs, loaded and stored as one vector access.
template <typename Real>
struct PairOf;
template <>
struct PairOf<float> {
  using type = float2;
};
template <>
struct PairOf<double> {
  using type = double2;
};
template <typename Real>
using Pair = typename PairOf<Real>::type;

template <typename Real>
__device__ __forceinline__ Pair<Real> make_pair(Real a, Real b) {
  Pair<Real> p;
  p.x = a;
  p.y = b;
  return p;
}

template <typename Real>
struct TileView {
  Pair<Real>* v;   // (V_hi, V_lo)
  Pair<Real>* ab;  // (alpha, beta); (alpha dt, beta dt) once pre-scaled
  Pair<Real>* dr;  // (row excess, rhs); segment nodes: (p, u) after the elimination
  Real* state;
  const Real* params;
  const SlotRec* slots;        // warp slots of the segment elimination
  const SegRec* segs;
  const SepRec* seps;
  const int32_t* levels;       // chunks of the separator sweeps (see GroupRec)
  const GroupRec* groups;
  const int32_t* rows;         // row starts of the slots
  const Real* diag0;           // axial diagonal of the whole cells' nodes
  const int32_t* heavy;        // nodes with heavy mechanisms
  const uint32_t* link;        // per node: upper separator | lower separator << 16 (kLinkNone, kLinkSelf)
  const uint16_t *pidx, *spec, *crec;  // crec: lane tiles only
  const SpecRec* specs;
  const uint32_t* mech;
  Real* q;                     // nodes of segments with a lower separator
  Pair<Real>* inbox;           // per segment: (excess, rhs) it adds to its upper separator
  SepRow<Real>* srow;          // per separator
  Pair<Real>* own;             // per separator: what the segment above it adds to its upper separator by itself
  Real* xsep;                  // per separator: its solved increment
  const int32_t* syn;       // tile synapse list (global synapse ids)
  const uint16_t* ncell;    // per node: tile-local cell (spike-source tiles only)
  const int32_t* srccell;   // per tile cell: global id of a spike source, -1 otherwise
  int32_t* stamp;           // per tile cell: last step with a crossing
  int N, n_real, n_cells, n_slots, n_groups, n_lower, cell0, sep0, n_seps, n_inbox, n_heavy;
  int pstride;  // reals per parameter record
  bool has_src;

  __device__ __forceinline__ void bind_seps(const TileDesc& td, unsigned char* sepw) {
    inbox = reinterpret_cast<Pair<Real>*>(sepw + td.off_inbox);
    srow = reinterpret_cast<SepRow<Real>*>(sepw + td.off_srow);
    own = reinterpret_cast<Pair<Real>*>(sepw + td.off_own);
  }

  // sepw, sepr: the separators' work area and records (in the scratch and the blob, or
  // both in shared memory for a global-memory tile)
  __device__ __forceinline__ void bind(const TileDesc& td, unsigned char* base, unsigned char* scratch,
                                       unsigned char* sepw, const unsigned char* sepr, void* gstate) {
    v = reinterpret_cast<Pair<Real>*>(base + td.off_v);
    ab = reinterpret_cast<Pair<Real>*>(base + td.off_ab);
    dr = reinterpret_cast<Pair<Real>*>(scratch + td.off_dr);
    state = reinterpret_cast<Real*>(gstate) + td.state_offset;
    params = reinterpret_cast<const Real*>(base + td.off_params);
    slots = reinterpret_cast<const SlotRec*>(base + td.off_slots);
    segs = reinterpret_cast<const SegRec*>(base + td.off_segs);
    seps = reinterpret_cast<const SepRec*>(sepr);
    levels = reinterpret_cast<const int32_t*>(sepr + (td.off_levels - td.off_seps));
    groups = reinterpret_cast<const GroupRec*>(sepr + (td.off_groups - td.off_seps));
    link = reinterpret_cast<const uint32_t*>(base + td.off_link);
    rows = reinterpret_cast<const int32_t*>(base + td.off_rows);
    diag0 = reinterpret_cast<const Real*>(base + td.off_diag0);
    heavy = reinterpret_cast<const int32_t*>(base + td.off_heavy);
    n_heavy = td.n_heavy;
    crec = reinterpret_cast<const uint16_t*>(base + td.off_crec);
    pidx = reinterpret_cast<const uint16_t*>(base + td.off_pidx);
    spec = reinterpret_cast<const uint16_t*>(base + td.off_spec);
    specs = reinterpret_cast<const SpecRec*>(base + td.off_specs);
    mech = reinterpret_cast<const uint32_t*>(base + td.off_mech);
    q = reinterpret_cast<Real*>(scratch + td.off_q);
    bind_seps(td, sepw);
    xsep = reinterpret_cast<Real*>(sepw + td.off_xsep);
    syn = reinterpret_cast<const int32_t*>(base + td.off_syn);
    has_src = td.off_ncell >= 0;
    ncell = has_src ? reinterpret_cast<const uint16_t*>(base + td.off_ncell) : nullptr;
    srccell = has_src ? reinterpret_cast<const int32_t*>(base + td.off_srccell) : nullptr;
    stamp = has_src ? reinterpret_cast<int32_t*>(scratch + td.off_stamp) : nullptr;
    n_cells = td.n_cells;
    pstride = td.param_stride;
    N = td.n_nodes;
    n_real = td.n_real_nodes;
    n_slots = td.n_slots;
    n_groups = td.n_groups;
    n_lower = td.n_lower;
    cell0 = td.cell0;
    sep0 = td.sep0;
    n_seps = td.n_seps;
    n_inbox = td.n_inbox;
  }
};

// Address of `p`, in this CTA's shared memory, in that of CTA `rank` of its cluster.
__device__ __forceinline__ unsigned char* cluster_map(unsigned char* p, uint32_t rank) {
  uint64_t out;
  asm("mapa.u64 %0, %1, %2;" : "=l"(out) : "l"(reinterpret_cast<uint64_t>(p)), "r"(rank));
  return reinterpret_cast<unsigned char*>(out);
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Reciprocal of a pivot, to about 1 ulp in both precisions (pivots are >= 1 on membrane
// rows and O(dt * g / C) on boundary rows, far from the denormal range).
template <typename Real>
__device__ __forceinline__ Real pivot_rcp(Real d) {
  return srcp(d);
}

// a * b and a + b rounded (never parts of a fused multiply-add), and a * b + c fused:
// where the same sum stands in several copies of the code (the two nodes of a lane, the
// forms of a warp, tiles in shared and in global memory), so that a node's result does not
// depend on which copy it met.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }

// float-float accumulation: (hi, lo) += d
template <typename Real>
__device__ __forceinline__ void ff_add(Real& hi, Real& lo, Real d) {
  const Real s = hi + d;
  const Real bb = s - hi;
  const Real err = (hi - (s - bb)) + (d - bb);
  const Real t = lo + err;
  hi = s + t;
  lo = t - (hi - s);
}

// ------------------------------------------------------------------ mechanisms
// The mechanism states of W consecutive nodes, in registers (absent ones are undefined).
template <typename Real, int W>
struct NodeStates {
  Real nap[W], naq[W], kdrp[W], calp[W], calq[W], catp[W], catq[W], hcnp[W], ahpp[W], cahi[W], calo[W];
};

// Loaded by group: a state that is absent but in a present group is read and not used.
constexpr uint32_t kSpikeGroup = BC_M_NA | BC_M_KDR;
constexpr uint32_t kShellGroup = BC_M_CAT | BC_M_AHP | BC_M_CADET;

// W consecutive values of a per-node array (W = 2: one vector access; the arrays keep
// an even node on an 8-byte boundary).
template <int W, typename Real>
__device__ __forceinline__ void load_w(const Real* p, Real (&x)[W]) {
  if constexpr (W == 2) {
    const Pair<Real> t = *reinterpret_cast<const Pair<Real>*>(p);
    x[0] = t.x;
    x[1] = t.y;
  } else {
    x[0] = p[0];
  }
}
template <int W, typename Real>
__device__ __forceinline__ void store_w(Real* p, const Real (&x)[W]) {
  if constexpr (W == 2)
    *reinterpret_cast<Pair<Real>*>(p) = make_pair<Real>(x[0], x[1]);
  else
    p[0] = x[0];
}

template <int W, typename Real>
__device__ __forceinline__ void load_states(const Real* st, int N, uint32_t m, NodeStates<Real, W>& s) {
  if (m & BC_M_CAL) {
    load_w<W>(st + kSlotCalP * N, s.calp);
    load_w<W>(st + kSlotCalQ * N, s.calq);
  }
  if (m & BC_M_HCN) load_w<W>(st + kSlotHcnP * N, s.hcnp);
  if (m & kSpikeGroup) {
    load_w<W>(st + kSlotNaP * N, s.nap);
    load_w<W>(st + kSlotNaQ * N, s.naq);
    load_w<W>(st + kSlotKdrP * N, s.kdrp);
  }
  if (m & kShellGroup) {
    load_w<W>(st + kSlotCatP * N, s.catp);
    load_w<W>(st + kSlotCatQ * N, s.catq);
    load_w<W>(st + kSlotAhpP * N, s.ahpp);
    load_w<W>(st + kSlotCaHi * N, s.cahi);
    load_w<W>(st + kSlotCaLo * N, s.calo);
  }
}

// The cerebellar calcium channels' current density at v from the states in st and
// the calcium reversal potential eca: the step-start current the calcium shell
// integrates (with CaL and CaT), and the ohmic terms of the row.
template <typename Real>
__device__ __forceinline__ Real cerebellar_ca_current(const Real* st, int N, const Real* P, uint32_t m, Real v, Real eca,
                                                      Real* g_out) {
  Real g = Real(0);
  if (m & BC_M_CAHVA) {
    const Real s = st[kSlotCaHvaS * N];
    g += P[BC_P_CAHVA_G] * s * s * st[kSlotCaHvaU * N];
  }
  if (m & BC_M_CAV23) {
    const Real a = st[kSlotCav23M * N];
    g += P[BC_P_CAV23_G] * a * a * a * st[kSlotCav23H * N];
  }
  if (m & BC_M_CAV32) {
    const Real a = st[kSlotCav32M * N];
    g += P[BC_P_CAV32_G] * a * a * st[kSlotCav32H * N];
  }
  if (g_out) *g_out = g;
  return g * (eca - v);
}

// The value a mechanism probe records: state view `field` (a BC_STATE_* other
// than V) of the node whose states start at st, after the node's update.
template <typename Real>
__device__ __forceinline__ double probe_state(const Real* st, int N, int field) {
  if (field == BC_STATE_CA_CI) return double(st[kSlotCaHi * N]) + double(st[kSlotCaLo * N]);
  // slots 9, 10 hold Ci; the Markov views 25.. sit one above their slots 26..
  const int slot = field <= BC_STATE_AHP_P ? field - 1 : (field >= BC_STATE_NAV16_C1 ? field + 1 : field);
  return double(st[slot * N]);
}

// The value a current probe records: current density `code` (BC_CUR_*, uA/cm^2)
// of the node whose states start at st, at voltage v after the node's update,
// with the same terms as the step's currents.
template <typename Real>
__device__ __forceinline__ double probe_current(const Real* st, int N, const Real* P, uint32_t m, Real v, int code) {
  auto eca = [&]() -> Real {
    if (m & BC_M_CADET)
      return Real(kNernstCa) * P[BC_P_CA_TEMP] * dlog(P[BC_P_CA_CO] / (st[kSlotCaHi * N] + st[kSlotCaLo * N]));
    return P[BC_P_ECA];
  };
  auto cur = [&](int c) -> Real {
    switch (c) {
      case BC_CUR_IL:
        return (m & BC_M_IL) ? P[BC_P_IL_G] * (P[BC_P_IL_E] - v) : Real(0);
      case BC_CUR_KLEAK:
        return (m & BC_M_KLEAK) ? P[BC_P_KLEAK_G] * (P[BC_P_EK] - v) : Real(0);
      case BC_CUR_NA: {
        if (!(m & BC_M_NA)) return Real(0);
        const Real p = st[kSlotNaP * N];
        return P[BC_P_NA_G] * p * p * p * st[kSlotNaQ * N] * (P[BC_P_ENA] - v);
      }
      case BC_CUR_KDR: {
        if (!(m & BC_M_KDR)) return Real(0);
        const Real p2 = st[kSlotKdrP * N] * st[kSlotKdrP * N];
        return P[BC_P_KDR_G] * p2 * p2 * (P[BC_P_EK] - v);
      }
      case BC_CUR_CAL: {
        if (!(m & BC_M_CAL)) return Real(0);
        const Real p = st[kSlotCalP * N];
        return P[BC_P_CAL_G] * p * p * st[kSlotCalQ * N] * (eca() - v);
      }
      case BC_CUR_CAT: {
        if (!(m & BC_M_CAT)) return Real(0);
        const Real p = st[kSlotCatP * N];
        return P[BC_P_CAT_G] * p * p * st[kSlotCatQ * N] * (eca() - v);
      }
      case BC_CUR_HCN:
        return (m & BC_M_HCN) ? P[BC_P_HCN_G] * st[kSlotHcnP * N] * (P[BC_P_HCN_E] - v) : Real(0);
      case BC_CUR_AHP: {
        if (!(m & BC_M_AHP)) return Real(0);
        const Real p = st[kSlotAhpP * N];
        return P[BC_P_AHP_G] * p * p * (P[BC_P_EK] - v);
      }
      case BC_CUR_NAHH: {
        if (!(m & BC_M_NAHH)) return Real(0);
        const Real p = st[kSlotNaHHP * N];
        return P[BC_P_NAHH_G] * p * p * p * st[kSlotNaHHQ * N] * (P[BC_P_ENA] - v);
      }
      case BC_CUR_KHH: {
        if (!(m & BC_M_KHH)) return Real(0);
        const Real p2 = st[kSlotKHHP * N] * st[kSlotKHHP * N];
        return P[BC_P_KHH_G] * p2 * p2 * (P[BC_P_EK] - v);
      }
      case BC_CUR_KM:
        return (m & BC_M_KM) ? P[BC_P_KM_G] * st[kSlotKMN * N] * (P[BC_P_EK] - v) : Real(0);
      case BC_CUR_KA1: {
        if (!(m & BC_M_KA1)) return Real(0);
        const Real p2 = st[kSlotKA1P * N] * st[kSlotKA1P * N];
        return P[BC_P_KA1_G] * p2 * p2 * st[kSlotKA1Q * N] * (P[BC_P_EK] - v);
      }
      case BC_CUR_KA2: {
        if (!(m & BC_M_KA2)) return Real(0);
        const Real p2 = st[kSlotKA2P * N] * st[kSlotKA2P * N];
        return P[BC_P_KA2_G] * p2 * p2 * st[kSlotKA2Q * N] * (P[BC_P_EK] - v);
      }
      case BC_CUR_KK2A:
        return (m & BC_M_KK2A) ? P[BC_P_KK2A_G] * st[kSlotKK2AP * N] * st[kSlotKK2AQ * N] * (P[BC_P_EK] - v) : Real(0);
      case BC_CUR_KK2B:
        return (m & BC_M_KK2B) ? P[BC_P_KK2B_G] * st[kSlotKK2BP * N] * st[kSlotKK2BQ * N] * (P[BC_P_EK] - v) : Real(0);
      case BC_CUR_KNI:
        return (m & BC_M_KNI) ? P[BC_P_KNI_G] * st[kSlotKNIP * N] * (P[BC_P_EK] - v) : Real(0);
      case BC_CUR_NAV16:
        return (m & BC_M_NAV16) ? P[BC_P_NAV16_G] * st[(kSlotNav16 + 10) * N] * (P[BC_P_ENA] - v) : Real(0);
      case BC_CUR_KCA22:
        return (m & BC_M_KCA22)
                   ? P[BC_P_KCA22_G] * (st[(kSlotKca22 + 3) * N] + st[(kSlotKca22 + 4) * N]) * (P[BC_P_EK] - v)
                   : Real(0);
      case BC_CUR_KCA11: {
        if (!(m & BC_M_KCA11)) return Real(0);
        Real o = Real(0);
        for (int k = 4; k < 9; ++k) o += st[(kSlotKca11 + k) * N];
        return P[BC_P_KCA11_G] * o * (P[BC_P_EK] - v);
      }
      case BC_CUR_KV34: {
        if (!(m & BC_M_KV34)) return Real(0);
        const Real a = st[kSlotKv34M * N];
        return P[BC_P_KV34_G] * a * a * a * st[kSlotKv34H * N] * (P[BC_P_EK] - v);
      }
      case BC_CUR_KV43: {
        if (!(m & BC_M_KV43)) return Real(0);
        const Real a = st[kSlotKv43A * N];
        return P[BC_P_KV43_G] * a * a * a * st[kSlotKv43B * N] * (P[BC_P_EK] - v);
      }
      case BC_CUR_KV11: {
        if (!(m & BC_M_KV11)) return Real(0);
        const Real n2 = st[kSlotKv11N * N] * st[kSlotKv11N * N];
        return P[BC_P_KV11_G] * n2 * n2 * (P[BC_P_EK] - v);
      }
      case BC_CUR_KIR23:
        return (m & BC_M_KIR23) ? P[BC_P_KIR23_G] * st[kSlotKir23D * N] * (P[BC_P_EK] - v) : Real(0);
      case BC_CUR_HCN1F:
        return (m & BC_M_HCN1F)
                   ? P[BC_P_HCN1F_G] * (st[kSlotHcn1Fast * N] + st[kSlotHcn1Slow * N]) * (P[BC_P_HCN1F_E] - v)
                   : Real(0);
      case BC_CUR_HCN1H:
        return (m & BC_M_HCN1H) ? P[BC_P_HCN1H_G] * st[kSlotHcn1H * N] * (P[BC_P_HCN1H_E] - v) : Real(0);
      case BC_CUR_CAHVA:
        return cerebellar_ca_current(st, N, P, m & BC_M_CAHVA, v, eca(), (Real*)nullptr);
      case BC_CUR_CAV23:
        return cerebellar_ca_current(st, N, P, m & BC_M_CAV23, v, eca(), (Real*)nullptr);
      case BC_CUR_CAV32:
        return cerebellar_ca_current(st, N, P, m & BC_M_CAV32, v, eca(), (Real*)nullptr);
      default:
        // extension channels: the record's list exists only where BC_M_EXT is set
        if (c >= BC_CUR_HCN2 && c <= BC_CUR_CALVADCN && (m & BC_M_EXT)) {
          const Real ci = (m & BC_M_CADET) ? st[kSlotCaHi * N] + st[kSlotCaLo * N] : P[BC_P_CA_CI0];
          const bool ohmic_ca = c == BC_CUR_CATHP || c == BC_CUR_CAHTRE || c == BC_CUR_CAV12 || c == BC_CUR_CAV13;
          return ext_current(st, N, P, ext_mask(P), v, ci, ohmic_ca ? eca() : Real(0),
                             c, (Real*)nullptr);
        }
    }
    return Real(0);
  };
  switch (code) {
    case BC_CUR_ION_NA:
      return double(cur(BC_CUR_NA)) + double(cur(BC_CUR_NAHH)) + double(cur(BC_CUR_NAV16)) + double(cur(BC_CUR_NAF)) +
             double(cur(BC_CUR_NAP)) + double(cur(BC_CUR_NAIO)) + double(cur(BC_CUR_NAVGRC));
    case BC_CUR_ION_K:
      return double(cur(BC_CUR_KDR)) + double(cur(BC_CUR_KLEAK)) + double(cur(BC_CUR_AHP)) + double(cur(BC_CUR_KHH)) +
             double(cur(BC_CUR_KM)) + double(cur(BC_CUR_KA1)) + double(cur(BC_CUR_KA2)) + double(cur(BC_CUR_KK2A)) +
             double(cur(BC_CUR_KK2B)) + double(cur(BC_CUR_KNI)) + double(cur(BC_CUR_KCA22)) + double(cur(BC_CUR_KCA11)) +
             double(cur(BC_CUR_KV34)) + double(cur(BC_CUR_KV43)) + double(cur(BC_CUR_KV11)) + double(cur(BC_CUR_KIR23)) +
             double(cur(BC_CUR_KV33)) + double(cur(BC_CUR_KV22)) + double(cur(BC_CUR_KV15)) + double(cur(BC_CUR_FKDR)) +
             double(cur(BC_CUR_SKDR)) + double(cur(BC_CUR_KDRIO)) + double(cur(BC_CUR_KCA31)) + double(cur(BC_CUR_SKDCN)) +
             double(cur(BC_CUR_KKV));
    case BC_CUR_ION_CA:
      return double(cur(BC_CUR_CAL)) + double(cur(BC_CUR_CAT)) + double(cur(BC_CUR_CAHVA)) + double(cur(BC_CUR_CAV23)) +
             double(cur(BC_CUR_CAV32)) + double(cur(BC_CUR_CATHP)) + double(cur(BC_CUR_CAHTRE)) + double(cur(BC_CUR_CAN)) +
             double(cur(BC_CUR_CAV31)) + double(cur(BC_CUR_CAV33)) + double(cur(BC_CUR_CAV12)) + double(cur(BC_CUR_CAV13)) +
             double(cur(BC_CUR_CAV21)) + double(cur(BC_CUR_CAHVADCN)) + double(cur(BC_CUR_CALVADCN));
    default:
      return double(cur(code));
  }
}

// Channels outside the main workloads' mix (classic Hodgkin-Huxley Na / K, the
// M current, the A current, the slow K2 current, the slow non-inactivating K
// current): kept out of line so that their registers do not weigh on the common
// path; same exp-Euler steps and ohmic currents as the others.
constexpr uint32_t kCerebellarCaChannels = BC_M_CAHVA | BC_M_CAV23 | BC_M_CAV32;
constexpr uint32_t kCerebellarChannels =
    BC_M_KV34 | BC_M_KV43 | BC_M_KV11 | BC_M_KIR23 | BC_M_HCN1F | BC_M_HCN1H | kCerebellarCaChannels;
constexpr uint32_t kExtraChannels = BC_M_NAHH | BC_M_KHH | BC_M_KM | BC_M_KA1 | BC_M_KA2 | BC_M_KK2A | BC_M_KK2B |
                                   BC_M_KNI | BC_M_NAV16 | BC_M_KCA22 | BC_M_KCA11 | kCerebellarChannels | BC_M_EXT;

__device__ __forceinline__ MarkovGraph nav16_graph() { return MarkovGraph{13, 17, 12, kSlotNav16, kNav16Src, kNav16Dst}; }
__device__ __forceinline__ MarkovGraph kca22_graph() { return MarkovGraph{6, 5, 0, kSlotKca22, kKca22Src, kKca22Dst}; }
__device__ __forceinline__ MarkovGraph kca11_graph() { return MarkovGraph{10, 13, 0, kSlotKca11, kKca11Src, kKca11Dst}; }

// One A-current mechanism (p^4 q, E_K) in slots (sp, sq) with parameters from pg.
template <typename Real>
__device__ __forceinline__ void a_current(Real* st, int N, const Real* P, int sp, int sq, int pg, Real mid,
                                          Real inv_slope, Real v, Real dt, bool advance, Real& G, Real& I) {
  Real p = st[sp * N], q = st[sq * N];
  if (advance) {
    const KARates<Real> r(v, P[pg + 1], mid, inv_slope);
    p = gate_it(p, r.pinf, r.ptau, P[pg + 2], dt);
    q = gate_it(q, r.qinf, r.qtau, P[pg + 3], dt);
    st[sp * N] = p;
    st[sq * N] = q;
  }
  const Real p2 = p * p;
  const Real g = P[pg] * p2 * p2 * q;
  G += g;
  I += g * (P[BC_P_EK] - v);
}

// One slow K2 mechanism (p q, E_K) in slots (sp, sq) with parameters from pg.
template <typename Real>
__device__ __forceinline__ void k2_current(Real* st, int N, const Real* P, int sp, int sq, int pg, bool b_form, Real v,
                                           Real dt, bool advance, Real& G, Real& I) {
  Real p = st[sp * N], q = st[sq * N];
  if (advance) {
    const K2Rates<Real> r(v, P[pg + 1], b_form);
    p = gate_it(p, r.pinf, r.ptau, P[pg + 2], dt);
    q = gate_it(q, r.qinf, r.qtau, P[pg + 3], dt);
    st[sp * N] = p;
    st[sq * N] = q;
  }
  const Real g = P[pg] * p * q;
  G += g;
  I += g * (P[BC_P_EK] - v);
}

// The cerebellar HH channels: exp-Euler gates at v, ohmic currents (HCN1 with its
// own reversal potential; HCN1_MA2020_GoC's g carries its Q10 factor already; the
// calcium channels in E_Ca of the calcium ci after this step's shell update).
template <typename Real>
__device__ __forceinline__ void cerebellar_channels(Real* st, int N, const Real* P, uint32_t m, Real v, Real ci,
                                                    Real dt, bool advance, Real& G, Real& I) {
  if (m & BC_M_KV34) {
    Real a = st[kSlotKv34M * N], b = st[kSlotKv34H * N];
    if (advance) {
      const Kv34Rates<Real> r(v);
      a = gate_it(a, r.minf, r.mtau, P[BC_P_KV34_PHI], dt);
      b = gate_it(b, r.hinf, r.htau, P[BC_P_KV34_PHI], dt);
      st[kSlotKv34M * N] = a;
      st[kSlotKv34H * N] = b;
    }
    const Real g = P[BC_P_KV34_G] * a * a * a * b;
    G += g;
    I += g * (P[BC_P_EK] - v);
  }
  if (m & BC_M_KV43) {
    Real a = st[kSlotKv43A * N], b = st[kSlotKv43B * N];
    if (advance) {
      const Kv43Rates<Real> r(v);
      a = gate_it(a, r.ainf, r.atau, P[BC_P_KV43_PHI], dt);
      b = gate_it(b, r.binf, r.btau, P[BC_P_KV43_PHI], dt);
      st[kSlotKv43A * N] = a;
      st[kSlotKv43B * N] = b;
    }
    const Real g = P[BC_P_KV43_G] * a * a * a * b;
    G += g;
    I += g * (P[BC_P_EK] - v);
  }
  if (m & BC_M_KV11) {
    Real n = st[kSlotKv11N * N];
    if (advance) {
      const Kv11Rates<Real> r(v);
      n = gate_ab<Real, true>(n, r.a, r.b, P[BC_P_KV11_PHI], dt);
      st[kSlotKv11N * N] = n;
    }
    const Real n2 = n * n;
    const Real g = P[BC_P_KV11_G] * n2 * n2;
    G += g;
    I += g * (P[BC_P_EK] - v);
  }
  if (m & BC_M_KIR23) {
    Real d = st[kSlotKir23D * N];
    if (advance) {
      const Kir23Rates<Real> r(v);
      d = gate_ab<Real, true>(d, r.a, r.b, P[BC_P_KIR23_PHI], dt);
      st[kSlotKir23D * N] = d;
    }
    const Real g = P[BC_P_KIR23_G] * d;
    G += g;
    I += g * (P[BC_P_EK] - v);
  }
  if (m & BC_M_HCN1F) {
    Real f = st[kSlotHcn1Fast * N], sl = st[kSlotHcn1Slow * N];
    if (advance) {
      const Hcn1fRates<Real> r(v);
      f = gate_it(f, r.finf, r.ftau, P[BC_P_HCN1F_PHI], dt);
      sl = gate_it(sl, r.sinf, r.stau, P[BC_P_HCN1F_PHI], dt);
      st[kSlotHcn1Fast * N] = f;
      st[kSlotHcn1Slow * N] = sl;
    }
    const Real g = P[BC_P_HCN1F_G] * (f + sl);
    G += g;
    I += g * (P[BC_P_HCN1F_E] - v);
  }
  if (m & BC_M_HCN1H) {
    Real h = st[kSlotHcn1H * N];
    if (advance) {
      const Hcn1hRates<Real> r(v);
      h = gate_it(h, r.hinf, r.htau, P[BC_P_HCN1H_PHI], dt);
      st[kSlotHcn1H * N] = h;
    }
    const Real g = P[BC_P_HCN1H_G] * h;
    G += g;
    I += g * (P[BC_P_HCN1H_E] - v);
  }
  if (m & kCerebellarCaChannels) {
    if (advance) {
      if (m & BC_M_CAHVA) {
        const CaHvaRates<Real> r(v);
        st[kSlotCaHvaS * N] = gate_ab<Real, true>(st[kSlotCaHvaS * N], r.sa, r.sb, P[BC_P_CAHVA_PHI], dt);
        st[kSlotCaHvaU * N] = gate_ab<Real, true>(st[kSlotCaHvaU * N], r.ua, r.ub, P[BC_P_CAHVA_PHI], dt);
      }
      if (m & BC_M_CAV23) {
        const Cav23Rates<Real> r(v);
        st[kSlotCav23M * N] = gate_it(st[kSlotCav23M * N], r.minf, r.mtau, Real(1), dt);
        st[kSlotCav23H * N] = gate_it(st[kSlotCav23H * N], r.hinf, r.htau, Real(1), dt);
      }
      if (m & BC_M_CAV32) {
        const Cav32Rates<Real> r(v, P[BC_P_CAV32_VSH]);
        st[kSlotCav32M * N] = gate_it(st[kSlotCav32M * N], r.minf, r.mtau, Real(kCav32PhiM), dt);
        st[kSlotCav32H * N] = gate_it(st[kSlotCav32H * N], r.hinf, r.htau, Real(1), dt);
      }
    }
    const Real eca =
        (m & BC_M_CADET) ? Real(kNernstCa) * P[BC_P_CA_TEMP] * dlog(P[BC_P_CA_CO] / ci) : P[BC_P_ECA];
    Real g = Real(0);
    I += cerebellar_ca_current(st, N, P, m, v, eca, &g);
    G += g;
  }
}

template <typename Real>
__device__ __noinline__ void extra_channels(Real* st, int N, const Real* P, uint32_t m, Real v, Real ci, Real dt,
                                            bool advance,
                                            Real& G, Real& I) {
  if (m & BC_M_NAHH) {
    Real p = st[kSlotNaHHP * N], q = st[kSlotNaHHQ * N];
    if (advance) {
      const NaHHRates<Real> r(v, P[BC_P_NAHH_VSH]);
      const Real phi = P[BC_P_NAHH_PHI];
      p = gate_ab<Real, true>(p, r.ap, r.bp, phi, dt);
      q = gate_ab<Real, true>(q, r.aq, r.bq, phi, dt);
      st[kSlotNaHHP * N] = p;
      st[kSlotNaHHQ * N] = q;
    }
    const Real g = P[BC_P_NAHH_G] * p * p * p * q;
    G += g;
    I += g * (P[BC_P_ENA] - v);
  }
  if (m & BC_M_KHH) {
    Real p = st[kSlotKHHP * N];
    if (advance) {
      const KHHRates<Real> r(v, P[BC_P_KHH_VSH]);
      p = gate_ab<Real, true>(p, r.a, r.b, P[BC_P_KHH_PHI], dt);
      st[kSlotKHHP * N] = p;
    }
    const Real p2 = p * p;
    const Real g = P[BC_P_KHH_G] * p2 * p2;
    G += g;
    I += g * (P[BC_P_EK] - v);
  }
  if (m & BC_M_KM) {
    Real n = st[kSlotKMN * N];
    if (advance) {
      const KMRates<Real> r(v);
      n = gate_it(n, r.ninf, r.ntau, P[BC_P_KM_PHI], dt);
      st[kSlotKMN * N] = n;
    }
    const Real g = P[BC_P_KM_G] * n;
    G += g;
    I += g * (P[BC_P_EK] - v);
  }
  if (m & BC_M_KA1)
    a_current(st, N, P, kSlotKA1P, kSlotKA1Q, BC_P_KA1_G, Real(kKA1Mid), Real(kKA1InvSlope), v, dt, advance, G, I);
  if (m & BC_M_KA2)
    a_current(st, N, P, kSlotKA2P, kSlotKA2Q, BC_P_KA2_G, Real(kKA2Mid), Real(kKA2InvSlope), v, dt, advance, G, I);
  if (m & BC_M_KK2A) k2_current(st, N, P, kSlotKK2AP, kSlotKK2AQ, BC_P_KK2A_G, false, v, dt, advance, G, I);
  if (m & BC_M_KK2B) k2_current(st, N, P, kSlotKK2BP, kSlotKK2BQ, BC_P_KK2B_G, true, v, dt, advance, G, I);
  if (m & BC_M_KNI) {
    Real p = st[kSlotKNIP * N];
    if (advance) {
      const KNIRates<Real> r(v, P[BC_P_KNI_VSH], P[BC_P_KNI_TAUMAX]);
      p = gate_it(p, r.pinf, r.ptau, P[BC_P_KNI_PHI], dt);
      st[kSlotKNIP * N] = p;
    }
    const Real g = P[BC_P_KNI_G] * p;
    G += g;
    I += g * (P[BC_P_EK] - v);
  }
  if (m & kCerebellarChannels) cerebellar_channels(st, N, P, m, v, ci, dt, advance, G, I);
  // Markov channels: the reference's independent-integration family, advanced
  // after the gates (cell.py:2204-2217), each at the new V and Ci
  if (m & (BC_M_NAV16 | BC_M_KCA22 | BC_M_KCA11)) {
    Real kf[17], kb[17];
    if (m & BC_M_NAV16) {
      if (advance) {
        nav16_rates(v, P[BC_P_NAV16_PHI], P[BC_P_NAV16_OON], P[BC_P_NAV16_ALFAC], P[BC_P_NAV16_EPS], kf, kb);
        markov_advance(st, N, nav16_graph(), kf, kb, dt);
      }
      const Real g = P[BC_P_NAV16_G] * st[(kSlotNav16 + 10) * N];  // O
      G += g;
      I += g * (P[BC_P_ENA] - v);
    }
    if (m & BC_M_KCA22) {
      if (advance) {
        kca22_rates(ci, P[BC_P_KCA22_PHI], P[BC_P_KCA22_DIFF], kf, kb);
        markov_advance(st, N, kca22_graph(), kf, kb, dt);
      }
      const Real g = P[BC_P_KCA22_G] * (st[(kSlotKca22 + 3) * N] + st[(kSlotKca22 + 4) * N]);  // O1 + O2
      G += g;
      I += g * (P[BC_P_EK] - v);
    }
    if (m & BC_M_KCA11) {
      if (advance) {
        kca11_rates(v, ci, P[BC_P_KCA11_PHI], P[BC_P_KCA11_QO], P[BC_P_KCA11_QC], kf, kb);
        markov_advance(st, N, kca11_graph(), kf, kb, dt);
      }
      Real o = Real(0);
      for (int k = 4; k < 9; ++k) o += st[(kSlotKca11 + k) * N];  // O0 .. O4
      const Real g = P[BC_P_KCA11_G] * o;
      G += g;
      I += g * (P[BC_P_EK] - v);
    }
  }
  // the extension channels listed in the record (gates independent of the above),
  // the calcium ones in E_Ca of the calcium after this step's shell update
  if (m & BC_M_EXT) {
    const Real eca =
        (m & BC_M_CADET) ? Real(kNernstCa) * P[BC_P_CA_TEMP] * dlog(P[BC_P_CA_CO] / ci) : P[BC_P_ECA];
    ext_channels(st, N, P, v, ci, eca, dt, advance, G, I);
  }
}

// Parameter records of a launch: the main mix's entries that only ever appear with dt
// are replaced by what the step needs (kDer), once per launch, in the records' shared-
// memory copy or in a copy in the tile's scratch:
//   PHI entries -> -dt phi;  CA_TAU -> c = 1 - exp(-dt / tau);  CA_D -> the shell's gain
//   c tau 10 / (2 F d) (c tau = dt where tau is infinite: shell_gain), so that the calcium
//   step is Ci += max(gain ICa, 0) + c (C_rest - Ci);
//   E_Ca of a dynamic ion, which nothing reads -> slope ln C_out, so that its Nernst
//   potential is that minus slope ln Ci: no division beside the logarithm.
template <typename Real>
__device__ __forceinline__ Real launch_param(const Real* P, uint32_t m, int k, Real dt) {
  switch (k) {
    case BC_P_NA_PHI:
    case BC_P_KDR_PHI:
    case BC_P_CAL_PHIP:
    case BC_P_CAL_PHIQ:
    case BC_P_CAT_PHIP:
    case BC_P_CAT_PHIQ:
    case BC_P_HCN_PHI:
    case BC_P_AHP_PHI:
      return -dt * P[k];
    case BC_P_CA_TAU:
      return (m & BC_M_CADET) ? -dexpm1(-dt / P[k]) : P[k];
    case BC_P_CA_D:
      return (m & BC_M_CADET) ? shell_gain(dt, P[BC_P_CA_TAU]) * Real(kCaDrive) / P[k] : P[k];
    case BC_P_ECA:
      return (m & BC_M_CADET) ? Real(kNernstCa) * P[BC_P_CA_TEMP] * dlog(P[BC_P_CA_CO]) : P[k];
    default:
      return P[k];
  }
}
template <typename Real, bool kDer>
__device__ __forceinline__ Real step_param(const Real* P, uint32_t m, int k, Real dt) {
  return kDer ? P[k] : launch_param(P, m, k, dt);
}

// The mechanisms of W consecutive nodes.  `st` points at the first node's slot-0 state
// (stride N).  With kAdv the states move from (v_old) to (v) first: calcium from the
// step-start current (old gates, old V, old Ci), then every gate at v (and the new Ci).
// Returns the membrane conductance G (mS/cm^2) and ionic current I (uA/cm^2) at v with
// the resulting states.  kDer: P are a launch's records (see launch_param).
//
// kHeavy: nodes may have heavy mechanisms (kHeavyMech) too.
// mu is the union of m over the warp (or the node's m): a mechanism's block is entered
// by the whole warp, a uniform branch.  Nodes without the mechanism keep its terms to
// themselves; a pair's states are stored together (pair) when either node has the
// mechanism (a state that a node does not have is never read), unless one of the two is
// another lane's.
template <typename Real, int W, bool kHeavy, bool kExtra, bool kAdv, bool kDer>
__device__ __forceinline__ void node_mechanisms(const NodeStates<Real, W>& s0, Real* st, int N,
                                                const Real* const (&P)[W], const uint32_t (&m)[W], uint32_t mu, bool pair,
                                                const Real (&v_old)[W], const Real (&v)[W], Real dt, Real (&G)[W],
                                                Real (&I)[W]) {
  uint32_t m_any = m[0];
  if constexpr (W == 2) m_any |= m[1];
  auto keep = [&](int slot, uint32_t bit, const Real(&x)[W]) {
    if (W == 1 || pair) {
      if (m_any & bit) store_w<W>(st + slot * N, x);
    } else {
      for (int j = 0; j < W; ++j)
        if (m[j] & bit) st[slot * N + j] = x[j];
    }
  };
  auto k_of = [&](int j, int k) { return step_param<Real, kDer>(P[j], m[j], k, dt); };
  // selects instead of branches: the two nodes' chains interleave
  auto add = [&](int j, uint32_t bit, Real g, Real e) {
    const bool on = (m[j] & bit) != 0;
    const Real i = mul_rn(g, e - v[j]);
    G[j] = add_rn(G[j], on ? g : Real(0));
    I[j] = add_rn(I[j], on ? i : Real(0));
  };
#pragma unroll
  for (int j = 0; j < W; ++j) {
    G[j] = I[j] = Real(0);
    add(j, BC_M_IL, P[j][BC_P_IL_G], P[j][BC_P_IL_E]);
    add(j, BC_M_KLEAK, P[j][BC_P_KLEAK_G], P[j][BC_P_EK]);
  }
  Real ci[W];
#pragma unroll
  for (int j = 0; j < W; ++j) ci[j] = Real(0);
  if ((kHeavy && kExtra) || (mu & (BC_M_CAL | kShellGroup))) {
    Real eca[W];
#pragma unroll
    for (int j = 0; j < W; ++j) {
      ci[j] = P[j][BC_P_CA_CI0];
      eca[j] = P[j][BC_P_ECA];
    }
    if (mu & BC_M_CADET) {
      Real cahi[W], calo[W];
#pragma unroll
      for (int j = 0; j < W; ++j) {
        const bool on = (m[j] & BC_M_CADET) != 0;
        cahi[j] = s0.cahi[j];
        calo[j] = s0.calo[j];
        const Real slope = Real(kNernstCa) * P[j][BC_P_CA_TEMP], e_out = on ? k_of(j, BC_P_ECA) : Real(0);
        Real c = cahi[j] + calo[j], E = fma_rn(-slope, ln_pos(c), e_out);
        if (kAdv) {
          Real ica = Real(0);
          if (mu & BC_M_CAL) {
            const Real i = P[j][BC_P_CAL_G] * s0.calp[j] * s0.calp[j] * s0.calq[j] * (E - v_old[j]);
            ica = add_rn(ica, (m[j] & BC_M_CAL) ? i : Real(0));
          }
          if (mu & BC_M_CAT) {
            const Real i = P[j][BC_P_CAT_G] * s0.catp[j] * s0.catp[j] * s0.catq[j] * (E - v_old[j]);
            ica = add_rn(ica, (m[j] & BC_M_CAT) ? i : Real(0));
          }
          if (kHeavy && kExtra && (m[j] & kCerebellarCaChannels))
            ica += cerebellar_ca_current(st + j, N, P[j], m[j], v_old[j], E, (Real*)nullptr);
          if (kHeavy && kExtra && (m[j] & BC_M_EXT)) ica += ext_ca_current(st + j, N, P[j], v_old[j], c, E);
          const Real drive = ica * k_of(j, BC_P_CA_D);
          ff_add(cahi[j], calo[j],
                 (drive > Real(0) ? drive : Real(0)) + k_of(j, BC_P_CA_TAU) * (P[j][BC_P_CA_CREST] - c));
          c = cahi[j] + calo[j];
          E = fma_rn(-slope, ln_pos(c), e_out);
        }
        ci[j] = on ? c : ci[j];
        eca[j] = on ? E : eca[j];
      }
      if (kAdv) keep(kSlotCaHi, BC_M_CADET, cahi);
      if (kAdv) keep(kSlotCaLo, BC_M_CADET, calo);
    }
    if (mu & BC_M_CAL) {
      Real p[W], q[W];
#pragma unroll
      for (int j = 0; j < W; ++j) {
        p[j] = s0.calp[j];
        q[j] = s0.calq[j];
        if (kAdv) {
          const Real vs = v[j] - P[j][BC_P_CAL_VSH];
          p[j] = cal_p_step(vs, k_of(j, BC_P_CAL_PHIP)).step(p[j]);
          q[j] = cal_q_step(vs, k_of(j, BC_P_CAL_PHIQ)).step(q[j]);
        }
        add(j, BC_M_CAL, P[j][BC_P_CAL_G] * p[j] * p[j] * q[j], eca[j]);
      }
      if (kAdv) keep(kSlotCalP, BC_M_CAL, p);
      if (kAdv) keep(kSlotCalQ, BC_M_CAL, q);
    }
    if (mu & (BC_M_CAT | BC_M_AHP)) {
      if (mu & BC_M_CAT) {
        Real p[W], q[W];
#pragma unroll
        for (int j = 0; j < W; ++j) {
          p[j] = s0.catp[j];
          q[j] = s0.catq[j];
          if (kAdv) {
            const Real vs = v[j] - P[j][BC_P_CAT_VSH];
            p[j] = cat_p_step(vs, k_of(j, BC_P_CAT_PHIP)).step(p[j]);
            q[j] = cat_q_step(vs, k_of(j, BC_P_CAT_PHIQ)).step(q[j]);
          }
          add(j, BC_M_CAT, P[j][BC_P_CAT_G] * p[j] * p[j] * q[j], eca[j]);
        }
        if (kAdv) keep(kSlotCatP, BC_M_CAT, p);
        if (kAdv) keep(kSlotCatQ, BC_M_CAT, q);
      }
      if (mu & BC_M_AHP) {
        Real p[W];
#pragma unroll
        for (int j = 0; j < W; ++j) {
          p[j] = s0.ahpp[j];
          const bool on = (m[j] & BC_M_AHP) != 0;
          if (kAdv) {
            const Real n = P[j][BC_P_AHP_N];
            const Real a = P[j][BC_P_AHP_ALPHA] * (n == Real(2) || !on ? ci[j] * ci[j] : dpow(ci[j], n));
            const Real s = a + P[j][BC_P_AHP_BETA];
            p[j] = p[j] - decay_em1(k_of(j, BC_P_AHP_PHI) * s) * (a * srcp(s) - p[j]);
          }
          add(j, BC_M_AHP, P[j][BC_P_AHP_G] * p[j] * p[j], P[j][BC_P_EK]);
        }
        if (kAdv) keep(kSlotAhpP, BC_M_AHP, p);
      }
    }
  }
  if (mu & BC_M_HCN) {
    Real p[W];
#pragma unroll
    for (int j = 0; j < W; ++j) {
      p[j] = s0.hcnp[j];
      if (kAdv) p[j] = hcn_step(v[j], k_of(j, BC_P_HCN_PHI)).step(p[j]);
      add(j, BC_M_HCN, P[j][BC_P_HCN_G] * p[j], P[j][BC_P_HCN_E]);
    }
    if (kAdv) keep(kSlotHcnP, BC_M_HCN, p);
  }
  // the spike-generating gates: accurate forms, and few nodes, so per node
  if (kHeavy && (mu & kSpikeGroup)) {
#pragma unroll
    for (int j = 0; j < W; ++j) {
      if (m[j] & BC_M_NA) {
        Real p = s0.nap[j], q = s0.naq[j];
        if (kAdv) {
          const NaRates<Real> r(v[j], P[j][BC_P_NA_VSH]);
          const Real k = k_of(j, BC_P_NA_PHI), sp = r.ap + r.bp, sq = r.aq + r.bq;
          p = p - dexpm1(k * sp) * (adiv(r.ap, sp) - p);
          q = q - dexpm1(k * sq) * (adiv(r.aq, sq) - q);
          st[kSlotNaP * N + j] = p;
          st[kSlotNaQ * N + j] = q;
        }
        add(j, BC_M_NA, P[j][BC_P_NA_G] * p * p * p * q, P[j][BC_P_ENA]);
      }
      if (m[j] & BC_M_KDR) {
        Real p = s0.kdrp[j];
        if (kAdv) {
          const KdrRates<Real> r(v[j], P[j][BC_P_KDR_VSH]);
          const Real s = r.a + r.b;
          p = p - dexpm1(k_of(j, BC_P_KDR_PHI) * s) * (adiv_sum(r.a, s) - p);
          st[kSlotKdrP * N + j] = p;
        }
        const Real p2 = p * p;
        add(j, BC_M_KDR, P[j][BC_P_KDR_G] * p2 * p2, P[j][BC_P_EK]);
      }
    }
  }
  // the Markov Kca channels bind the new Ci of a dynamic ion, else the fixed one
  if constexpr (kHeavy && kExtra) {
#pragma unroll
    for (int j = 0; j < W; ++j)
      if (m[j] & kExtraChannels) extra_channels(st + j, N, P[j], m[j], v[j], ci[j], dt, kAdv, G[j], I[j]);
  }
}

// Mechanisms whose nodes are updated in a list of their own, one to a lane: the spike-
// generating gates with their accurate functions, and all out-of-line channels.
constexpr uint32_t kHeavyMech = kSpikeGroup | kExtraChannels;

// The same for one node by itself: its currents as they are, or one step on.
template <typename Real, bool kExtra, bool kAdv>
__device__ __forceinline__ void one_node(const NodeStates<Real, 1>& s, Real* st, int N, const Real* P, uint32_t m,
                                         Real v_old, Real v, Real dt, Real& G, Real& I) {
  const Real* const Pa[1] = {P};
  const uint32_t ma[1] = {m};
  const Real vo[1] = {v_old}, va[1] = {v};
  Real g[1], i[1];
  node_mechanisms<Real, 1, true, kExtra, kAdv, false>(s, st, N, Pa, ma, m, true, vo, va, dt, g, i);
  G = g[0];
  I = i[0];
}

template <typename Real, bool kExtra>
__device__ __forceinline__ void node_currents(Real* st, int N, const Real* P, uint32_t m, Real v, Real dt, Real& G,
                                              Real& I) {
  NodeStates<Real, 1> s;
  load_states(st, N, m, s);
  one_node<Real, kExtra, false>(s, st, N, P, m, v, v, dt, G, I);
}

// Steady state of every gate at v (HH.reset_state), Ci = Ci0.
template <typename Real>
__device__ __forceinline__ void steady_states(const Real* P, uint32_t m, Real* st, int N, Real v) {
  if (m & BC_M_CADET) {
    st[kSlotCaHi * N] = P[BC_P_CA_CI0];
    st[kSlotCaLo * N] = Real(0);
  }
  if (m & BC_M_NA) {
    const NaRates<Real> r(v, P[BC_P_NA_VSH]);
    st[kSlotNaP * N] = r.ap / (r.ap + r.bp);
    st[kSlotNaQ * N] = r.aq / (r.aq + r.bq);
  }
  if (m & BC_M_KDR) {
    const KdrRates<Real> r(v, P[BC_P_KDR_VSH]);
    st[kSlotKdrP * N] = r.a / (r.a + r.b);
  }
  if (m & BC_M_CAL) {
    const CaLRates<Real> r(v, P[BC_P_CAL_VSH]);
    st[kSlotCalP * N] = r.pinf;
    st[kSlotCalQ * N] = r.qinf;
  }
  if (m & BC_M_CAT) {
    const CaTRates<Real> r(v, P[BC_P_CAT_VSH]);
    st[kSlotCatP * N] = r.pinf;
    st[kSlotCatQ * N] = r.qinf;
  }
  if (m & BC_M_HCN) {
    const HcnRates<Real> r(v);
    st[kSlotHcnP * N] = r.pinf;
  }
  if (m & BC_M_AHP) {
    const Real ci = P[BC_P_CA_CI0];
    const Real n = P[BC_P_AHP_N];
    const Real a = P[BC_P_AHP_ALPHA] * (n == Real(2) ? ci * ci : dpow(ci, n));
    st[kSlotAhpP * N] = a / (a + P[BC_P_AHP_BETA]);
  }
  if (m & BC_M_NAHH) {
    const NaHHRates<Real> r(v, P[BC_P_NAHH_VSH]);
    st[kSlotNaHHP * N] = r.ap / (r.ap + r.bp);
    st[kSlotNaHHQ * N] = r.aq / (r.aq + r.bq);
  }
  if (m & BC_M_KHH) {
    const KHHRates<Real> r(v, P[BC_P_KHH_VSH]);
    st[kSlotKHHP * N] = r.a / (r.a + r.b);
  }
  if (m & BC_M_KM) st[kSlotKMN * N] = KMRates<Real>(v).ninf;
  if (m & BC_M_KA1) {
    const KARates<Real> r(v, P[BC_P_KA1_VSH], Real(kKA1Mid), Real(kKA1InvSlope));
    st[kSlotKA1P * N] = r.pinf;
    st[kSlotKA1Q * N] = r.qinf;
  }
  if (m & BC_M_KA2) {
    const KARates<Real> r(v, P[BC_P_KA2_VSH], Real(kKA2Mid), Real(kKA2InvSlope));
    st[kSlotKA2P * N] = r.pinf;
    st[kSlotKA2Q * N] = r.qinf;
  }
  if (m & BC_M_KK2A) {
    const K2Rates<Real> r(v, P[BC_P_KK2A_VSH], false);
    st[kSlotKK2AP * N] = r.pinf;
    st[kSlotKK2AQ * N] = r.qinf;
  }
  if (m & BC_M_KK2B) {
    const K2Rates<Real> r(v, P[BC_P_KK2B_VSH], true);
    st[kSlotKK2BP * N] = r.pinf;
    st[kSlotKK2BQ * N] = r.qinf;
  }
  if (m & BC_M_KNI) st[kSlotKNIP * N] = KNIRates<Real>(v, P[BC_P_KNI_VSH], P[BC_P_KNI_TAUMAX]).pinf;
  if (m & BC_M_KV34) {
    const Kv34Rates<Real> r(v);
    st[kSlotKv34M * N] = r.minf;
    st[kSlotKv34H * N] = r.hinf;
  }
  if (m & BC_M_KV43) {
    const Kv43Rates<Real> r(v);
    st[kSlotKv43A * N] = r.ainf;
    st[kSlotKv43B * N] = r.binf;
  }
  if (m & BC_M_KV11) {
    const Kv11Rates<Real> r(v);
    st[kSlotKv11N * N] = r.a / (r.a + r.b);
  }
  if (m & BC_M_KIR23) {
    const Kir23Rates<Real> r(v);
    st[kSlotKir23D * N] = r.a / (r.a + r.b);
  }
  if (m & BC_M_HCN1F) {
    const Hcn1fRates<Real> r(v);
    st[kSlotHcn1Fast * N] = r.finf;
    st[kSlotHcn1Slow * N] = r.sinf;
  }
  if (m & BC_M_HCN1H) st[kSlotHcn1H * N] = Hcn1hRates<Real>(v).hinf;
  if (m & BC_M_CAHVA) {
    const CaHvaRates<Real> r(v);
    st[kSlotCaHvaS * N] = r.sa / (r.sa + r.sb);
    st[kSlotCaHvaU * N] = r.ua / (r.ua + r.ub);
  }
  if (m & BC_M_CAV23) {
    const Cav23Rates<Real> r(v);
    st[kSlotCav23M * N] = r.minf;
    st[kSlotCav23H * N] = r.hinf;
  }
  if (m & BC_M_CAV32) {
    const Cav32Rates<Real> r(v, P[BC_P_CAV32_VSH]);
    st[kSlotCav32M * N] = r.minf;
    st[kSlotCav32H * N] = r.hinf;
  }
  if (m & BC_M_EXT) ext_steady(P, st, N, v);
  if (m & (BC_M_NAV16 | BC_M_KCA22 | BC_M_KCA11)) {
    // Markov channels start at their stationary distribution (reset_steady_state)
    Real kf[17], kb[17];
    const Real ci = P[BC_P_CA_CI0];
    if (m & BC_M_NAV16) {
      nav16_rates(v, P[BC_P_NAV16_PHI], P[BC_P_NAV16_OON], P[BC_P_NAV16_ALFAC], P[BC_P_NAV16_EPS], kf, kb);
      markov_steady(st, N, nav16_graph(), kf, kb);
    }
    if (m & BC_M_KCA22) {
      kca22_rates(ci, P[BC_P_KCA22_PHI], P[BC_P_KCA22_DIFF], kf, kb);
      markov_steady(st, N, kca22_graph(), kf, kb);
    }
    if (m & BC_M_KCA11) {
      kca11_rates(v, ci, P[BC_P_KCA11_PHI], P[BC_P_KCA11_QO], P[BC_P_KCA11_QC], kf, kb);
      markov_steady(st, N, kca11_graph(), kf, kb);
    }
  }
}

// Row i of the next linear system without its axial part: excess = diagonal minus
// the row's axial coefficients = 1 + dt G / cm, rhs = dt I / cm on membrane rows;
// 0, 0 on boundary rows.  Cells solved whole take the diagonal, 1 + dt (D + G / cm).
// pr: the node's parameter record, negative on boundary rows.
template <typename Real>
__device__ __forceinline__ Pair<Real> node_row(const TileView<Real>& tv, int i, int pr, Real dt, Real G, Real I) {
  const Real invcm = tv.params[size_t(max(pr, 0)) * tv.pstride + BC_P_INVCM];
  Real e = fma_rn(dt, mul_rn(invcm, G), Real(1)), r = mul_rn(mul_rn(dt, invcm), I);
  if (pr < 0) e = r = Real(0);
  if (i >= tv.cell0 && i < tv.sep0) {
    const Real d0 = tv.diag0[i - tv.cell0];
    e = pr < 0 ? mul_rn(dt, d0) : fma_rn(dt, fma_rn(invcm, G, d0), Real(1));
  }
  return make_pair(e, r);
}

// ExpSyn synapses of a node (synapse/markov.py:65-117).  `g` is stored as the
// conductance at the start of a step including that step's events.  advance:
// one dt of decay (exp-Euler of g' = -g / tau, exact); then, unless `last`, the
// events due at `next_step` are added (their ring slot is cleared) and the
// synapse current g (e - V) at v (a total current spread over the CV) is added
// to the node's conductance G and current I for the next row.
template <typename Real>
__device__ __forceinline__ void node_synapses(const LaunchArgs& a, const TileView<Real>& tv, const SpecRec& sr,
                                              Real v, Real dt, bool advance, bool last, int64_t next_step, Real& G,
                                              Real& I) {
  Real* g_all = static_cast<Real*>(a.syn_g);
  const Real* tau = static_cast<const Real*>(a.syn_tau);
  const Real* e = static_cast<const Real*>(a.syn_e);
  const Real* scale = static_cast<const Real*>(a.syn_scale);
  Real* arr = static_cast<Real*>(a.arrivals);
  for (int k = sr.syn_begin; k < sr.syn_end; ++k) {
    const int32_t id = tv.syn[k];
    Real g = g_all[id];
    if (advance) g += decay_em1(-dt / tau[id]) * g;
    if (!last) {
      if (arr) {
        Real* slot = arr + (next_step % a.arr_slots) * a.n_syn + id;
        g += *slot;
        *slot = Real(0);
      }
      const Real gd = g * scale[id];
      G += gd;
      I += gd * (e[id] - v);
    }
    g_all[id] = g;
  }
}

// Clamp pulses active at `step` on node i (the thread that wrote row i adds them).
template <typename Real>
__device__ __forceinline__ void add_node_pulses(const TileView<Real>& tv, const PulseRec* pulses, const SpecRec& sr,
                                                int i, int pr, int64_t step, Real dt) {
  for (int k = sr.pulse_begin; k < sr.pulse_end; ++k) {
    const PulseRec p = pulses[k];
    if (step < p.on_step || step >= p.off_step) continue;
    if (pr < 0)
      tv.dr[i].y += dt * Real(p.amp);
    else
      tv.dr[i].y += dt * tv.params[size_t(pr) * tv.pstride + BC_P_INVCM] * Real(p.amp);
  }
}

// ---------------------------------------------------------------- tree solve
// Row k of the increment system (V_{n+1} = V_n + x), with a = alpha dt of the node,
// b = beta dt of a child (its coefficient in this row) and Delta = V - V_parent in
// float-float:
//   (e + a + sum b) x - a x_parent - sum b x_child = r - a Delta + sum b Delta_child
// where e is the excess of the diagonal over the axial coefficients.
//
// 1. Segments (eliminate_segments): one lane eliminates the nodes of a segment
//    between its lower separator s and upper separator t,
//      E_k = e_k + wE,  F_k = wF,  R_k = r_k + wR - a_k Delta_k,  inv_k = 1 / (E_k + a_k),
//      (wE, wF) = b_k inv_k (E_k, F_k),  wR = b_k (inv_k R_k + Delta_k),
//    starting from wE = wF = b_s, wR = b_s Delta_s (0 at a leaf), then walks back down
//    to leave x_k = p_k + q_k x_s + u_k x_t in every node and to hand both separators
//    their rows' share.  The excess form has no subtraction in a segment's pivots (the
//    separators' own excess, a_s (1 - q - u), has: it cancels where a_s is large).
// 2. Separators (sweep_separators): the same elimination on the tree of separators,
//    one warp per group of cells, level by level, then back down to x.
// 3. Every other node's x is one or two multiply-adds on its separators' x, taken by
//    the update pass (node_increment).
//
// Why this split.  The time of a tile's step is latency: the walks down the tree
// levels with a block barrier at each (18 per step for the 10,000-cell uneven
// population, whose runs have 6.4 nodes on average) took 37 of 54 thousand cycles per
// step of a 2,500-node tile, most of them waiting.  Runs do not depend on one another,
// so one pass covers 94 % of the nodes, and what stays serial is the separator tree
// (one row per branch point), which a warp sweeps without block barriers: three
// barriers per step.

constexpr unsigned kFullMask = 0xffffffffu;

// (alpha dt, beta dt) of node i: pre-scaled in shared-memory tiles, scaled here otherwise
// (rounded as there).
template <typename Real, bool kPre>
__device__ __forceinline__ Pair<Real> coef(const TileView<Real>& tv, int i, Real dt) {
  Pair<Real> c = tv.ab[i];
  if (!kPre) {
    c.x = mul_rn(c.x, dt);
    c.y = mul_rn(c.y, dt);
  }
  return c;
}

template <typename Real>
__device__ __forceinline__ Real vdelta(const Pair<Real>& v, const Pair<Real>& up) {
  return (v.x - up.x) + (v.y - up.y);
}

// One warp slot: lane l eliminates segment seg0 + l.  kLower: the slot's segments
// have a lower separator.  Nodes are taken four at a time: one read of their row
// starts, all loads of the batch issued together, and no branch inside it (a lane past
// its segment's end reads its upper separator's node and keeps what it had).  Node by
// node, each took about 250 cycles a walk, most of it exposed shared-memory latency and
// divergent branches; the dependent arithmetic of a node is about 45.
template <typename Real, bool kPre, bool kLower>
__device__ __forceinline__ void eliminate_slot(const TileView<Real>& tv, const SlotRec& sr, int lane, Real dt) {
  const bool valid = lane < sr.n_lanes;
  const SegRec sg = tv.segs[sr.seg0 + (valid ? lane : 0)];
  const int4* rq = reinterpret_cast<const int4*>(tv.rows + sr.rows0);
  int4 r = rq[0];
  const int len = valid ? int(sg.len) : 0;
  const int max_len = sr.max_len;
  const int nt = tv.sep0 + sg.t;
  int id0 = len > 0 ? r.x + lane : nt;
  Pair<Real> v0 = tv.v[id0];
  Real wE = Real(0), wF = Real(0), wR = Real(0), as = Real(0), ds = Real(0);
  Pair<Real> row_s = make_pair(Real(0), Real(0));
  if (kLower) {
    const int ns = tv.sep0 + sg.s;
    const Pair<Real> cs = coef<Real, kPre>(tv, ns, dt);
    row_s = tv.dr[ns];
    ds = vdelta<Real>(tv.v[ns], v0);
    as = cs.x;
    wE = wF = cs.y;
    wR = mul_rn(cs.y, ds);
  }
  for (int k = 0; k < max_len; k += 4) {
    const int4 rn = rq[k / 4 + 1];
    const int id[5] = {id0, len > k + 1 ? r.y + lane : nt, len > k + 2 ? r.z + lane : nt, len > k + 3 ? r.w + lane : nt,
                       len > k + 4 ? rn.x + lane : nt};
    Pair<Real> row[4], c[4], v[5];
    v[0] = v0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      row[j] = tv.dr[id[j]];
      c[j] = coef<Real, kPre>(tv, id[j], dt);
      v[j + 1] = tv.v[id[j + 1]];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool act = len > k + j;
      const Real delta = vdelta<Real>(v[j], v[j + 1]);
      const Real E = row[j].x + wE;
      const Real R = fma_rn(-c[j].x, delta, row[j].y + wR);
      const Real inv = pivot_rcp(E + c[j].x);
      const Real g = mul_rn(c[j].y, inv);
      if (act) tv.dr[id[j]] = make_pair(mul_rn(inv, R), mul_rn(c[j].x, inv));
      if (kLower) {
        if (act) tv.q[id[j]] = mul_rn(inv, wF);
        wF = act ? mul_rn(g, wF) : wF;
      }
      wE = act ? mul_rn(mul_rn(c[j].y, E), inv) : wE;
      wR = act ? fma_rn(g, R, mul_rn(c[j].y, delta)) : wR;
    }
    id0 = id[4];
    v0 = v[4];
    r = rn;
  }
  if (!kLower && valid) tv.inbox[sg.inbox] = make_pair(wE, wR);
  // back down: x_k = p + q x_s + u x_t
  Real p = Real(0), q = Real(0), u = Real(1);
  for (int k = (max_len - 1) & ~3; k >= 0; k -= 4) {
    r = rq[k / 4];
    const int id[4] = {r.x + lane, r.y + lane, r.z + lane, r.w + lane};
    Pair<Real> d[4];
    Real f[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int i = len > k + j ? id[j] : nt;
      d[j] = tv.dr[i];
      f[j] = kLower ? tv.q[len > k + j ? id[j] : 0] : Real(0);
    }
#pragma unroll
    for (int j = 3; j >= 0; --j) {
      const bool act = len > k + j;
      p = act ? fma_rn(d[j].y, p, d[j].x) : p;
      u = act ? mul_rn(d[j].y, u) : u;
      if (act) tv.dr[id[j]] = make_pair(p, u);
      if (kLower) {
        q = act ? fma_rn(d[j].y, q, f[j]) : q;
        if (act) tv.q[id[j]] = q;
      }
    }
  }
  if (kLower && valid) {
    SepRow<Real> o;
    o.e = fma_rn(as, Real(1) - q - u, row_s.x);
    o.r = fma_rn(as, p - ds, row_s.y);
    o.a = mul_rn(as, u);
    o.b = wF;
    tv.srow[sg.s] = o;
    tv.own[sg.s] = make_pair(wE - wF, wR);
  }
}

// One slot of whole cells: lane l eliminates and back-substitutes its cell, in the
// diagonal form.  A parent with one child is the next row and takes its child's terms
// from registers; other parents collect them in their rows, child by child.  (See
// kCellLaneNodes for which cells, and both sides measured.)
template <typename Real, bool kPre>
__device__ __forceinline__ void solve_cells(const TileView<Real>& tv, const SlotRec& sr, int lane, Real dt) {
  const int32_t* rows = tv.rows + sr.rows0;
  bool carry = false;
  Pair<Real> pc = make_pair(Real(0), Real(0));
  Real pw = Real(0), pR = Real(0), pd = Real(0);
  for (int k = 0; k < sr.max_len; ++k) {
    const int i = rows[k] + lane;
    if (i >= rows[k + 1]) break;  // the lanes with more nodes come first
    const uint32_t lk = tv.link[i];
    const uint32_t par = lk & 0xFF;
    const Pair<Real> q = tv.dr[i], c = coef<Real, kPre>(tv, i, dt), v = tv.v[i];
    const int ip = par == kLinkNoParent ? i : rows[par] + lane;
    Real D = q.x, R = q.y;
    if (carry) {
      D = q.x - pc.x * pw;
      R = q.y + pw * pR + pc.y * pd;
    }
    const Real inv = pivot_rcp(D);
    const Real delta = vdelta<Real>(v, tv.v[ip]);
    R -= c.x * delta;
    tv.dr[i] = make_pair(inv, R);
    const Real w = c.y * inv;
    carry = (lk & kLinkOnlyChild) != 0;
    if (!carry && par != kLinkNoParent) {
      Pair<Real> pp = tv.dr[ip];
      pp.x -= mul_rn(c.x, w);
      pp.y += w * R + c.y * delta;
      tv.dr[ip] = pp;
    }
    pc = c;
    pw = w;
    pR = R;
    pd = delta;
  }
  for (int k = sr.max_len - 1; k >= 0; --k) {
    const int i = rows[k] + lane;
    if (i >= rows[k + 1]) continue;
    const uint32_t par = tv.link[i] & 0xFF;
    const Pair<Real> q = tv.dr[i];
    const Real xp = par == kLinkNoParent ? Real(0) : tv.dr[rows[par] + lane].y;
    tv.dr[i].y = (q.y + coef<Real, kPre>(tv, i, dt).x * xp) * q.x;
  }
}

template <typename Real, bool kPre>
__device__ __forceinline__ void eliminate_segments(const TileView<Real>& tv, int warp, int n_warps, int lane, Real dt) {
  for (int s = warp; s < tv.n_slots; s += n_warps) {
    const SlotRec sr = tv.slots[s];
    if (sr.kind == kSlotLower)
      eliminate_slot<Real, kPre, true>(tv, sr, lane, dt);
    else if (sr.kind == kSlotLeaf)
      eliminate_slot<Real, kPre, false>(tv, sr, lane, dt);
    else
      solve_cells<Real, kPre>(tv, sr, lane, dt);
  }
}

// What the level below does not change about a separator: loaded one level ahead.
template <typename Real>
struct SepItem {
  SepRec rec;
  SepRow<Real> row;
  Pair<Real> own;
};

template <typename Real>
__device__ __forceinline__ SepItem<Real> load_sep(const TileView<Real>& tv, int j) {
  SepItem<Real> it;
  it.rec = tv.seps[j];
  it.row = tv.srow[j];
  it.own = tv.own[j];
  return it;
}

// The separator tree: a warp per group of cells, up to 32 separators of a level at a
// time.  A chunk's own data are loaded while the chunk before is eliminated, inboxes of
// up to four entries are read unconditionally, and the only branches are the loops':
// this is one warp's chain of dependent instructions, where a branch costs 15 to 25
// cycles and a chunk's arithmetic about 100.
template <typename Real>
__device__ __forceinline__ void sweep_separators(const TileView<Real>& tv, int warp, int n_warps, int lane) {
  const InPair<Real>* inbox = reinterpret_cast<const InPair<Real>*>(tv.inbox);
  const int j_last = tv.n_seps - 1;
  for (int g = warp; g < tv.n_groups; g += n_warps) {
    const GroupRec gr = tv.groups[g];
    const int32_t* lv = tv.levels + gr.lv0;
    uint32_t cb = uint32_t(lv[0]), ce = uint32_t(lv[1]);
    int b = int(cb & ~kChunkMore);
    SepItem<Real> it = load_sep(tv, min(b + lane, j_last));
    for (int l = 0; l < gr.n_chunks; ++l) {
      const uint32_t cn = uint32_t(lv[min(l + 2, gr.n_chunks)]);
      const int e = int(ce & ~kChunkMore);
      const SepItem<Real> nx = load_sep(tv, min(e + lane, j_last));
      const InPair<Real> c0 = inbox[it.rec.in0], c1 = inbox[it.rec.in0 + 1];
      Real E = it.row.e + ((c0.e0 + c0.e1) + (c1.e0 + c1.e1));
      Real R = it.row.r + ((c0.r0 + c0.r1) + (c1.r0 + c1.r1));
      if (cb & kChunkMore) {
        for (int k = 2; k < it.rec.n_in; ++k) {
          const InPair<Real> c = inbox[it.rec.in0 + k];
          E += c.e0 + c.e1;
          R += c.r0 + c.r1;
        }
      }
      const Real inv = pivot_rcp(E + it.row.a);
      const Real w = mul_rn(it.row.b, inv);
      const bool valid = b + lane < e;
      if (valid) tv.inbox[it.rec.inbox] = make_pair(fma_rn(w, E, it.own.x), fma_rn(w, R, it.own.y));
      if (valid) *reinterpret_cast<Pair<Real>*>(tv.srow + b + lane) = make_pair(mul_rn(it.row.a, inv), mul_rn(R, inv));
      __syncwarp();
      b = e;
      cb = ce;
      ce = cn;
      it = nx;
    }
    // back down: x = R / D + A / D x_t (A = 0 and t = itself at a root)
    int e = b;
    b = lv[gr.n_chunks - 1] & int(~kChunkMore);
    int j = min(b + lane, j_last);
    uint32_t t = tv.seps[j].t;
    Pair<Real> d = *reinterpret_cast<const Pair<Real>*>(tv.srow + j);
    for (int l = gr.n_chunks - 1; l >= 0; --l) {
      const int b1 = lv[max(l - 1, 0)] & int(~kChunkMore);
      const int j1 = min(b1 + lane, j_last);
      const uint32_t t1 = tv.seps[j1].t;
      const Pair<Real> d1 = *reinterpret_cast<const Pair<Real>*>(tv.srow + j1);
      const Real x = fma_rn(d.x, tv.xsep[t], d.y);
      if (b + lane < e) tv.xsep[b + lane] = x;
      __syncwarp();
      e = b;
      b = b1;
      t = t1;
      d = d1;
    }
  }
}

// The solved increments of nodes i .. i + W - 1; i0: the warp's first node.
template <typename Real, int W>
__device__ __forceinline__ void node_increments(const TileView<Real>& tv, int i, int i0, Real (&x)[W]) {
  if (i0 + 32 * W <= tv.cell0) {  // segment nodes
#pragma unroll
    for (int j = 0; j < W; ++j) {
      const Pair<Real> d = tv.dr[i + j];
      const uint32_t lk = tv.link[i + j];
      x[j] = fma_rn(d.y, tv.xsep[lk & 0xFFFF], d.x);
      if (i + j < tv.n_lower) x[j] = fma_rn(tv.q[i + j], tv.xsep[lk >> 16], x[j]);
    }
  } else {
#pragma unroll
    for (int j = 0; j < W; ++j) {
      const int k = i + j;
      const Pair<Real> d = tv.dr[k];
      if (k >= tv.sep0) {
        x[j] = tv.xsep[k - tv.sep0];  // (0 in the padding)
      } else if (k >= tv.cell0) {
        x[j] = d.y;
      } else {
        const uint32_t lk = tv.link[k];
        x[j] = fma_rn(d.y, tv.xsep[lk & 0xFFFF], d.x);
        if (k < tv.n_lower) x[j] = fma_rn(tv.q[k], tv.xsep[lk >> 16], x[j]);
      }
    }
  }
}

// ------------------------------------------------------------ surrogate ports
// One GRU step per port of the tile and the port's terms in the row of step m
// (the port variant only).  The port injects I = g (e + y_scale y - V_end) into
// its endpoint row: the -g V_end part implicitly (diagonal), the rest at V^m.
// Inputs: ((V_att - e) / v_scale, S / 0.1 nA, feat0, feat1) with V_att the
// attachment CV's voltage at the start of step m and S the port's stimulus
// pulses active at step m (nA).
//
// Pass A (a thread per port) stages the inputs, checks the envelope (an input
// outside it flags the port's cell for the full solve) and adds the row terms
// that do not depend on y.  Pass B, after a barrier, deals work items (M tile of
// 16 ports, group jb of 8 hidden units) round-robin over the warps; lane
// (g, tq) holds ports g and g + 8 of the tile and units 8 jb + 2 tq, +1.  The
// hidden state is read from the half (m & 1) and written to the other half, so
// items do not race; each item adds its part of y's current atomically.
constexpr float kPortStimScale = 0.1f;  // nA

// Launch start / end: the tile's port records and envelope state between global
// memory and the tile scratch.
__device__ __forceinline__ void port_local_load(const PortRec* ports, int n_ports, const float* port_h,
                                                PortLocal* pl, int tid, int T) {
  for (int q = tid; q < n_ports; q += T) {
    const PortRec r = ports[q];
    PortLocal l;
    l.node = r.node;
    l.att = r.att;
    l.cell = r.cell;
    l.id = r.id;
    l.stim_begin = r.stim_begin;
    l.stim_end = r.stim_end;
    l.g = r.g;
    l.e = r.e;
    l.feat[0] = r.feat[0];
    l.feat[1] = r.feat[1];
    const float2 pv = *reinterpret_cast<const float2*>(port_h + size_t(r.id) * kPortStride + kPortVPrev);
    l.v_prev = pv.x;
    l.seen = pv.y;
    l.pad[0] = l.pad[1] = 0;
    pl[q] = l;
  }
}

__device__ __forceinline__ void port_local_store(int n_ports, float* port_h, const PortLocal* pl, int tid, int T) {
  for (int q = tid; q < n_ports; q += T)
    *reinterpret_cast<float2*>(port_h + size_t(pl[q].id) * kPortStride + kPortVPrev) =
        make_float2(pl[q].v_prev, pl[q].seen);
}

template <typename Real>
__device__ __forceinline__ void port_stage(PortLocal* pl, int n_ports, const PulseRec* stim, int32_t* flags,
                                          const GruWeights* __restrict__ W, const Pair<Real>* v, Pair<Real>* dr,
                                          PortStage* stage, int64_t m, Real dt, int tid, int T) {
  for (int q = tid; q < n_ports; q += T) {
    PortLocal& r = pl[q];
    const Pair<Real> va = v[r.att], ve = v[r.node];
    float S = 0.f;
    for (int k = r.stim_begin; k < r.stim_end; ++k) {
      const PulseRec pr = stim[k];
      if (m >= pr.on_step && m < pr.off_step) S += float(pr.amp);
    }
    const float vatt = float(va.x + va.y);
    const float dv = vatt - float(r.e);
    const float rate = r.seen != 0.f ? fabsf(vatt - r.v_prev) / float(dt) : 0.f;
    if (dv < W->env_v_lo || dv > W->env_v_hi || rate > W->env_dvdt) flags[r.cell] = 1;
    r.v_prev = vatt;
    r.seen = 1.f;
    const Real gg = Real(r.g) * Real(1e-3) * dt;  // uS -> row units (1 uF dummy capacitance)
    Pair<Real> row = dr[r.node];
    row.x += gg;
    row.y += gg * (Real(r.e) + Real(W->y_scale) * Real(W->bo) - (ve.x + ve.y));
    dr[r.node] = row;
    PortStage st;
    st.x[0] = dv / W->v_scale;
    st.x[1] = S * (1.0f / kPortStimScale);
    st.x[2] = r.feat[0];
    st.x[3] = r.feat[1];
    st.node = r.node;
    st.coef = float(gg) * W->y_scale;
    st.id = r.id;
    st.pad = 0;
    stage[q] = st;
  }
}

template <typename Real>
__device__ __forceinline__ void port_gru(const PortStage* stage, int n_ports, float* port_h, const uint2* wfrag,
                                        const float* wo_s, Pair<Real>* dr, int64_t m, int warp, int n_warps, int lane,
                                        unsigned long long* ptimers) {
#ifdef BC_PORT_TIMERS
  long long pt0 = clock64();
#define BC_PTICK(slot)                                                                                  \
  do {                                                                                                  \
    const long long pt1 = clock64();                                                                    \
    if (warp == 0 && lane == 0 && ptimers) atomicAdd(ptimers + (slot), (unsigned long long)(pt1 - pt0)); \
    pt0 = pt1;                                                                                          \
  } while (0)
#else
#define BC_PTICK(slot) \
  do {                 \
  } while (0)
#endif
  const int g = lane >> 2, tq = lane & 3;
  const int rd = int(m & 1), wr = rd ^ 1;
  // Work items: (M tile of 16 ports, range of N groups).  Each M tile is split
  // into as many ranges as there are warps for it (1..8), so every warp is busy;
  // the A operand is loaded once per item and reused across its N groups.
  const int n_mt = (n_ports + 15) >> 4;
  const int n_split = max(1, min(8, n_warps / max(n_mt, 1)));
  const int n_items = n_mt * n_split;
  for (int it = warp; it < n_items; it += n_warps) {
    const int mt = it / n_split, sp = it - mt * n_split;
    const int jb_begin = (sp * 8) / n_split, jb_end = ((sp + 1) * 8) / n_split;
    const int qa = mt * 16 + g, qb = qa + 8;
    const bool oka = qa < n_ports, okb = qb < n_ports;
    float* ha = oka ? port_h + size_t(stage[qa].id) * kPortStride : nullptr;
    float* hb = okb ? port_h + size_t(stage[qb].id) * kPortStride : nullptr;
    // A operand straight from the BF16 halves
    uint32_t ah[4][4];
    const uint32_t* ba = oka ? reinterpret_cast<const uint32_t*>(ha + kPortHBf) + rd * (kGruH / 2) : nullptr;
    const uint32_t* bb = okb ? reinterpret_cast<const uint32_t*>(hb + kPortHBf) + rd * (kGruH / 2) : nullptr;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      ah[kk][0] = oka ? ba[kk * 8 + tq] : 0u;
      ah[kk][1] = okb ? bb[kk * 8 + tq] : 0u;
      ah[kk][2] = oka ? ba[kk * 8 + 4 + tq] : 0u;
      ah[kk][3] = okb ? bb[kk * 8 + 4 + tq] : 0u;
    }
    uint32_t ax[4];
    {
      const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 xa = oka ? *reinterpret_cast<const float4*>(stage[qa].x) : z4;
      const float4 xb = okb ? *reinterpret_cast<const float4*>(stage[qb].x) : z4;
      const float fa[4] = {xa.x, xa.y, xa.z, xa.w}, fb[4] = {xb.x, xb.y, xb.z, xb.w};
      xblock_frag(fa, fb, tq, ax);
    }
    BC_PTICK(0);
    float ysa = 0.0f, ysb = 0.0f;
#pragma unroll 1
    for (int jb = jb_begin; jb < jb_end; ++jb) {
      const int j0 = jb * 8 + 2 * tq;
      // FP32 values of this lane's two units (issued ahead of the products)
      const float2 z2 = make_float2(0.f, 0.f);
      const float2 hoa = oka ? *reinterpret_cast<const float2*>(ha + rd * kGruH + j0) : z2;
      const float2 hob = okb ? *reinterpret_cast<const float2*>(hb + rd * kGruH + j0) : z2;
      float acc[4][4];
      gru_preact_frag(wfrag + jb * (kGruFragSlots * 32), lane, ah, ax, acc);
      BC_PTICK(1);
      const float2 wo = *reinterpret_cast<const float2*>(wo_s + j0);
      const GruGate G0 = gru_gate(acc[0][0], acc[1][0], acc[2][0], acc[3][0], hoa.x);
      const GruGate G1 = gru_gate(acc[0][1], acc[1][1], acc[2][1], acc[3][1], hoa.y);
      const GruGate G2 = gru_gate(acc[0][2], acc[1][2], acc[2][2], acc[3][2], hob.x);
      const GruGate G3 = gru_gate(acc[0][3], acc[1][3], acc[2][3], acc[3][3], hob.y);
      if (oka) {
        *reinterpret_cast<float2*>(ha + wr * kGruH + j0) = make_float2(G0.h_new, G1.h_new);
        reinterpret_cast<uint32_t*>(ha + kPortHBf)[wr * (kGruH / 2) + j0 / 2] = pack_bf16(G0.h_new, G1.h_new);
      }
      if (okb) {
        *reinterpret_cast<float2*>(hb + wr * kGruH + j0) = make_float2(G2.h_new, G3.h_new);
        reinterpret_cast<uint32_t*>(hb + kPortHBf)[wr * (kGruH / 2) + j0 / 2] = pack_bf16(G2.h_new, G3.h_new);
      }
      ysa += wo.x * G0.h_new + wo.y * G1.h_new;
      ysb += wo.x * G2.h_new + wo.y * G3.h_new;
      BC_PTICK(2);
    }
    ysa += __shfl_xor_sync(kFullMask, ysa, 1);
    ysa += __shfl_xor_sync(kFullMask, ysa, 2);
    ysb += __shfl_xor_sync(kFullMask, ysb, 1);
    ysb += __shfl_xor_sync(kFullMask, ysb, 2);
    if (tq == 0) {
      if (oka) atomicAdd(&dr[stage[qa].node].y, Real(stage[qa].coef) * Real(ysa));
      if (okb) atomicAdd(&dr[stage[qb].node].y, Real(stage[qb].coef) * Real(ysb));
    }
    BC_PTICK(3);
  }
#undef BC_PTICK
}

template <typename Real>
__device__ __forceinline__ bool is_finite_real(Real x) {
  return isfinite(x);
}

// ------------------------------------------------------------------ the update pass
struct StepCtx {
  int64_t step, rec_slot;
  bool last, record;
};

// One warp's turn of the update: the lane's nodes i .. i + W - 1 (ok: it has any; a lane
// without works on another's and stores nothing), i0 the warp's first node.  V += x, the
// mechanisms, the next step's row, probes, spikes and the pulses of the next step.
// Returns whether a voltage is not finite.
//
// Light nodes go two to a lane in FP32 (kHeavy = false, W = 2): half the loads, stores,
// branches and address arithmetic a node, and two independent chains.  The tile's node
// count is a multiple of 4 and its padding is boundary nodes that move nothing.  Heavy
// nodes (a few somas, or every node of a cell) have a list of their own, one to a lane:
// spread over the light nodes' warps, each made its warp the last at the barrier, with
// about 3 thousand cycles of dependent accurate functions on top of its share.
template <typename Real, int W, bool kHeavy, bool kExtra>
__device__ __forceinline__ bool update_nodes(const LaunchArgs& a, const TileView<Real>& tv, const PulseRec* pulses,
                                             const StepCtx& c, int i, bool ok, int i0, Real dt) {
  int pr[W];
  uint32_t m[W], m_any = 0;
  const Real* P[W];
  bool mine[W], all_mine = ok, any_mine = false;
#pragma unroll
  for (int j = 0; j < W; ++j) {
    const uint16_t rec = tv.pidx[i + j];
    pr[j] = rec == kBoundary ? -1 : int(rec);
    m[j] = pr[j] >= 0 ? tv.mech[pr[j]] : 0u;
    mine[j] = ok && (kHeavy || !(m[j] & kHeavyMech));
    all_mine = all_mine && mine[j];
    any_mine = any_mine || mine[j];
    if (!mine[j]) m[j] = 0u;
    m_any |= m[j];
    P[j] = tv.params + size_t(max(pr[j], 0)) * tv.pstride;
  }
  const uint32_t mu = __reduce_or_sync(kFullMask, m_any);
  // the states live in global memory (L2): read first, needed after the voltage
  NodeStates<Real, W> st;
  load_states(tv.state + i, tv.N, mu, st);
  Real hi[W], lo[W], v_old[W], lo_old[W], x[W], G[W], I[W];
  node_increments<Real, W>(tv, i, i0, x);
  bool bad = false;
#pragma unroll
  for (int j = 0; j < W; ++j) {
    const Pair<Real> vv = tv.v[i + j];
    hi[j] = v_old[j] = vv.x;
    lo[j] = lo_old[j] = vv.y;
    ff_add(hi[j], lo[j], x[j]);
    bad = bad || (mine[j] && !is_finite_real(hi[j]));
  }
  if (all_mine) {
#pragma unroll
    for (int j = 0; j < W; ++j) tv.v[i + j] = make_pair(hi[j], lo[j]);
  } else if (any_mine) {
    for (int j = 0; j < W; ++j)
      if (mine[j]) tv.v[i + j] = make_pair(hi[j], lo[j]);
  }
  if (c.last) {  // last_V of the per-CV spike indicator (cell.py:2384-2386)
#pragma unroll
    for (int j = 0; j < W; ++j)
      if (mine[j]) {
        tv.state[size_t(kSlotVLastHi) * tv.N + i + j] = v_old[j];
        tv.state[size_t(kSlotVLastLo) * tv.N + i + j] = lo_old[j];
      }
  }
  node_mechanisms<Real, W, kHeavy, kExtra, true, true>(st, tv.state + i, tv.N, P, m, mu, all_mine, v_old, hi, dt, G, I);
  Pair<Real> row[W];
  uint16_t spec[W];
  bool special = false;
#pragma unroll
  for (int j = 0; j < W; ++j) {
    row[j] = node_row(tv, i + j, pr[j], dt, G[j], I[j]);
    spec[j] = mine[j] ? tv.spec[i + j] : kNoSpecial;
    special = special || spec[j] != kNoSpecial;
  }
  if (!c.last) {
    if (all_mine) {
#pragma unroll
      for (int j = 0; j < W; ++j) tv.dr[i + j] = row[j];
    } else if (any_mine) {
      for (int j = 0; j < W; ++j)
        if (mine[j]) tv.dr[i + j] = row[j];
    }
  }
  if (special) {
    for (int j = 0; j < W; ++j) {
      if (spec[j] == kNoSpecial) continue;
      const SpecRec sr = tv.specs[spec[j]];
      if (kExtra && sr.syn_begin < sr.syn_end) {
        node_synapses(a, tv, sr, hi[j], dt, true, c.last, c.step + 1, G[j], I[j]);
        if (!c.last) tv.dr[i + j] = node_row(tv, i + j, pr[j], dt, G[j], I[j]);
      }
      if (sr.probe >= 0) {
        const double v1 = double(hi[j]) + double(lo[j]), v0 = double(v_old[j]) + double(lo_old[j]);
        if (v0 < 0.0 && v1 >= 0.0) {
          const int n = a.spike_count[sr.probe];
          if (n < a.max_spikes)
            a.spike_times[int64_t(sr.probe) * a.max_spikes + n] =
                double(c.step) * a.dt + a.dt * (0.0 - v0) / (v1 - v0);
          a.spike_count[sr.probe] = n + 1;
        }
        if (c.record && c.rec_slot < a.trace_cap) a.traces[c.rec_slot * a.n_probes_total + sr.probe] = v1;
      }
      if (!c.last) add_node_pulses(tv, pulses, sr, i + j, pr[j], c.step + 1, dt);
    }
  }
  if (kExtra && tv.has_src) {
    // a spike of the cell: any of its CVs crossing 0 mV upward in this step
    for (int j = 0; j < W; ++j) {
      const uint16_t lc = tv.ncell[i + j];
      if (mine[j] && pr[j] >= 0 && lc != 0xFFFF && Real(v_old[j] + lo_old[j]) < Real(0) && Real(hi[j] + lo[j]) >= Real(0))
        tv.stamp[lc] = int32_t(c.step & 0x7fffffff);
    }
  }
  return bad;
}

// ------------------------------------------------------------------ the step kernel
// kVar: 0 = lean (no optional mechanism), 1 = extra (synapses, network,
// out-of-line channels), 2 = extra + subtree-surrogate ports, 3 = lean + ports
// (plans whose only optional feature is the ports).
// The port variants run at most BC_PORT_MAX_THREADS threads per CTA and ask for
// BC_PORT_MIN_CTAS resident CTAs per SM (their register budget).
template <typename Real, bool kSmem, int kVar>
__global__ void __launch_bounds__(kVar >= 2 ? BC_PORT_MAX_THREADS : 1024, kVar >= 2 ? BC_PORT_MIN_CTAS : 1)
    tile_step_kernel(LaunchArgs a) {
  constexpr bool kExtra = kVar == 1 || kVar == 2;
  constexpr bool kPorts = kVar >= 2;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ int s_status;
  // A global-memory tile runs on a cluster of a.cluster CTAs: warps and threads are
  // counted through the cluster, and the barriers between phases are the cluster's.
  const int csize = kSmem || kPorts ? 1 : a.cluster;
  const int rank = csize == 1 ? 0 : int(blockIdx.x) % csize;
  auto tile_sync = [&]() {
    if (csize == 1)
      __syncthreads();
    else
      cluster_sync();
  };
  const TileDesc td = a.tiles[csize == 1 ? int(blockIdx.x) : int(blockIdx.x) / csize];
  unsigned char* gblob = a.blob + td.blob_offset;
  unsigned char* base;
  unsigned char* scratch;
  if (threadIdx.x == 0) s_status = 0;
  if constexpr (kSmem) {
    base = smem;
    scratch = smem + td.blob_bytes;
    if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      mbar_expect_tx(&bar, uint32_t(td.blob_bytes));
      for (uint32_t off = 0; off < uint32_t(td.blob_bytes); off += kBulkChunk) {
        const uint32_t n = min(kBulkChunk, uint32_t(td.blob_bytes) - off);
        bulk_g2s(smem + off, gblob + off, n, &bar);
      }
    }
    // Bounded wait; the give-up decision is made block-wide so that no thread is
    // left at a barrier that others skip.
    const int ok = __syncthreads_and(mbar_wait(&bar, 0, 1u << 22) ? 1 : 0);
    if (!ok) {
      // The copy never completed: record, wait once more (bounded) and leave.
      if (threadIdx.x == 0) {
        atomicOr(a.status, kStatusTimeout);
        mbar_wait(&bar, 0, 1u << 22);
      }
      return;
    }
  } else {
    base = gblob;
    scratch = a.scratch + td.scratch_offset;
    __syncthreads();
  }
  const Real dt = Real(a.dt);
  const int T = blockDim.x * csize, tid = rank * blockDim.x + threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5, n_warps = T >> 5;
  TileView<Real> tv;
  if constexpr (kSmem) {
    tv.bind(td, base, scratch, scratch + td.off_sep, base + td.off_seps, a.state);
  } else if (td.sep_in_smem) {
    // the separators of a global-memory tile are swept in shared memory (by CTA 0 of a
    // cluster, whose copy the segments of all CTAs fill; xsep is every CTA's own)
    unsigned char* rec = smem + td.sep_bytes;
    for (int k = threadIdx.x; k < (td.off_rows - td.off_seps) / 4; k += blockDim.x)
      reinterpret_cast<int32_t*>(rec)[k] = reinterpret_cast<const int32_t*>(base + td.off_seps)[k];
    tv.bind(td, base, scratch, smem, rec, a.state);
    if (rank > 0) tv.bind_seps(td, cluster_map(smem, 0));
    __syncthreads();
  } else {
    tv.bind(td, base, scratch, scratch + td.off_sep, base + td.off_seps, a.state);
  }
  const PulseRec* pulses = a.pulses + td.pulse_offset;
  if constexpr (kSmem) {
    // the staged axial coefficients become (alpha dt, beta dt) for this launch
    for (int i = tid; i < tv.N; i += T) {
      Pair<Real> c = tv.ab[i];
      c.x *= dt;
      c.y *= dt;
      tv.ab[i] = c;
    }
  }

  // Prologue: the linear system of the first step from the current state.
  for (int i = tid; i < tv.n_real; i += T) {
    const uint16_t pr = tv.pidx[i];
    Real G = Real(0), I = Real(0);
    if (pr != kBoundary) {
      const Real v = tv.v[i].x;
      node_currents<Real, kExtra>(tv.state + i, tv.N, tv.params + size_t(pr) * tv.pstride, tv.mech[pr], v, dt, G, I);
    }
    const uint16_t sp = tv.spec[i];
    if (sp != kNoSpecial) {
      const SpecRec sr = tv.specs[sp];
      if (kExtra && sr.syn_begin < sr.syn_end) node_synapses(a, tv, sr, tv.v[i].x, dt, false, false, a.step0, G, I);
    }
    const int rec = pr == kBoundary ? -1 : int(pr);
    tv.dr[i] = node_row(tv, i, rec, dt, G, I);
    if (sp != kNoSpecial) add_node_pulses(tv, pulses, tv.specs[sp], i, rec, a.step0, dt);
  }
  {
    // the launch's parameter records: in place in shared memory, in the scratch otherwise
    Real* rec = kSmem ? const_cast<Real*>(tv.params) : reinterpret_cast<Real*>(scratch + td.off_wparams);
    if (!kSmem)
      for (int k = tid; k < td.n_params * tv.pstride; k += T) rec[k] = tv.params[k];
    tile_sync();  // the rows above read the records as they were
    for (int r = tid; r < td.n_params; r += T) {
      const Real* P = tv.params + size_t(r) * tv.pstride;
      Real* L = rec + size_t(r) * tv.pstride;
      const uint32_t m = tv.mech[r];
      constexpr int keys[] = {BC_P_CA_D,    BC_P_CA_TAU,  BC_P_NA_PHI,  BC_P_KDR_PHI, BC_P_CAL_PHIP,
                              BC_P_CAL_PHIQ, BC_P_CAT_PHIP, BC_P_CAT_PHIQ, BC_P_HCN_PHI, BC_P_AHP_PHI, BC_P_ECA};
#pragma unroll
      for (int k : keys) L[k] = launch_param(P, m, k, dt);  // CA_D first: it reads CA_TAU
    }
    tv.params = rec;
  }
  // inbox entries that no segment fills stay 0; a root reads its own xsep times 0
  if (rank == 0)
    for (int i = threadIdx.x; i < tv.n_inbox; i += blockDim.x) tv.inbox[i] = make_pair(Real(0), Real(0));
  for (int i = threadIdx.x; i < tv.n_seps + kSepPad; i += blockDim.x) tv.xsep[i] = Real(0);
  for (int i = tv.n_real + tid; i < tv.N; i += T) tv.dr[i] = make_pair(Real(0), Real(0));
  if (tv.has_src)
    for (int c = tid; c < tv.n_cells; c += T) tv.stamp[c] = -1;
  tile_sync();
  PortStage* pstage = nullptr;
  PortLocal* plocal = nullptr;
  uint2* wfrag = nullptr;
  float* wo_s = nullptr;
  if constexpr (kPorts) {
    if (td.n_ports > 0) {
      wfrag = reinterpret_cast<uint2*>(scratch + td.off_pstage);
      wo_s = reinterpret_cast<float*>(scratch + td.off_pstage + kGruFragBytes);
      pstage = reinterpret_cast<PortStage*>(scratch + td.off_pstage + kGruSmemBytes);
      plocal = reinterpret_cast<PortLocal*>(pstage + td.n_ports);
      gru_frag_fill(a.gru->wext, wfrag, tid, T);
      for (int j = tid; j < kGruH; j += T) wo_s[j] = a.gru->wo[j];
      port_local_load(a.ports + td.port_offset, td.n_ports, a.port_h, plocal, tid, T);
      __syncthreads();
      port_stage<Real>(plocal, td.n_ports, a.port_pulses, a.port_flags, a.gru, tv.v, tv.dr, pstage, a.step0, dt,
                       tid, T);
      __syncthreads();
      port_gru<Real>(pstage, td.n_ports, a.port_h, wfrag, wo_s, tv.dr, a.step0, warp, n_warps, lane, a.timers);
      __syncthreads();
    }
  }

#ifdef BC_PHASE_TIMERS
  unsigned long long tm[4] = {0, 0, 0, 0};
  long long t_prev = clock64();
#define BC_TICK(slot)                                 \
  do {                                                \
    const long long t_now = clock64();                \
    tm[slot] += (unsigned long long)(t_now - t_prev); \
    t_prev = t_now;                                   \
  } while (0)
#else
#define BC_TICK(slot) \
  do {                \
  } while (0)
#endif
  // steps to the next trace record, and its index
  int rec_in = 0;
  int64_t rec_slot = 0;
  if (a.record_every > 0) {
    const int64_t since = a.step0 - a.trace_base;
    rec_in = a.record_every - 1 - int(since % a.record_every);
    rec_slot = since / a.record_every;
  }
  for (int s = 0; s < a.n_steps; ++s) {
    const int64_t step = a.step0 + s;
    eliminate_segments<Real, kSmem>(tv, warp, n_warps, lane, dt);
    tile_sync();
    BC_TICK(0);
    if (rank == 0) sweep_separators<Real>(tv, threadIdx.x >> 5, blockDim.x >> 5, lane);
    if (csize > 1) {
      if (rank == 0) {
        __syncthreads();
        for (int r = 1; r < csize; ++r) {
          Real* xr = reinterpret_cast<Real*>(cluster_map(reinterpret_cast<unsigned char*>(tv.xsep), r));
          for (int j = threadIdx.x; j < tv.n_seps; j += blockDim.x) xr[j] = tv.xsep[j];
        }
      }
    }
    tile_sync();
    BC_TICK(1);
    // V update, mechanism states, next row, probes and next pulses
    const bool last = s + 1 == a.n_steps;
    const bool record = a.record_every > 0 && rec_in == 0;
    const StepCtx ctx{step, rec_slot, last, record};
    constexpr int W = sizeof(Real) == 4 ? 2 : 1;
    bool bad = false;
    for (int h0 = (n_warps - 1 - warp) * 32; h0 < tv.n_heavy; h0 += T)
      bad |= update_nodes<Real, 1, true, kExtra>(a, tv, pulses, ctx, tv.heavy[min(h0 + lane, tv.n_heavy - 1)],
                                                 h0 + lane < tv.n_heavy, tv.N, dt);
    if (tv.n_heavy < tv.n_real)
      for (int i0 = warp * (32 * W); i0 < tv.N; i0 += W * T)
        bad |= update_nodes<Real, W, false, kExtra>(a, tv, pulses, ctx, min(i0 + W * lane, tv.N - W),
                                                    i0 + W * lane < tv.N, i0, dt);
    if (bad) s_status = kStatusNonfinite;
    tile_sync();
    if (kExtra && record && td.n_xprobes > 0) {
      // mechanism probes (plans with them run the extra variant): state views after the update
      const ProbeRef* pl = reinterpret_cast<const ProbeRef*>(reinterpret_cast<const unsigned char*>(tv.specs) +
                                                             (td.off_plist - td.off_specs));
      for (int q = tid; q < td.n_xprobes; q += T) {
        const ProbeRef r = pl[q];
        if (rec_slot >= a.trace_cap) continue;
        double val;
        if (r.field >= BC_PROBE_CURRENT) {
          const uint16_t pr = tv.pidx[r.node];
          const Pair<Real> vv = tv.v[r.node];
          val = probe_current(tv.state + r.node, tv.N, tv.params + size_t(pr) * tv.pstride, tv.mech[pr], vv.x + vv.y,
                              r.field - BC_PROBE_CURRENT);
        } else {
          val = probe_state(tv.state + r.node, tv.N, r.field);
        }
        a.traces[rec_slot * a.n_probes_total + r.id] = val;
      }
    }
    if (kExtra && tv.has_src)
      for (int c = tid; c < tv.n_cells; c += T)
        if (tv.stamp[c] == int32_t(step & 0x7fffffff) && tv.srccell[c] >= 0) {
          const unsigned long long r = atomicAdd(a.rec_count, 1ull);
          if (int64_t(r) < a.rec_cap) {
            a.rec_cell[r] = tv.srccell[c];
            a.rec_step[r] = step;
          } else {
            s_status = kStatusRecordOverflow;
          }
        }
    if (--rec_in < 0) {
      rec_in = a.record_every - 1;
      ++rec_slot;
    }
    BC_TICK(2);
    if constexpr (kPorts) {
      if (td.n_ports > 0 && !last) {
        port_stage<Real>(plocal, td.n_ports, a.port_pulses, a.port_flags, a.gru, tv.v, tv.dr, pstage, step + 1, dt,
                         tid, T);
        __syncthreads();
        BC_TICK(2);
        port_gru<Real>(pstage, td.n_ports, a.port_h, wfrag, wo_s, tv.dr, step + 1, warp, n_warps, lane, a.timers);
        __syncthreads();
      }
    }
    BC_TICK(3);
  }
#ifdef BC_PHASE_TIMERS
  if (threadIdx.x == 0 && a.timers)
    for (int q = 0; q < 4; ++q) atomicAdd(a.timers + q, tm[q]);
#endif
  if constexpr (kPorts) {
    if (td.n_ports > 0) port_local_store(td.n_ports, a.port_h, plocal, tid, T);
  }
  if (s_status) atomicOr(a.status, s_status);

  if constexpr (kSmem) {
    fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
      for (uint32_t off = 0; off < uint32_t(td.dyn_bytes); off += kBulkChunk) {
        const uint32_t n = min(kBulkChunk, uint32_t(td.dyn_bytes) - off);
        bulk_s2g(gblob + off, smem + off, n);
      }
      bulk_commit_and_wait();
    }
  }
}

// ------------------------------------------------------------------ lane tiles
// One small cell per thread: node v of the thread's cell is tile node v * L + lane
// (L = blockDim.x), so the threads of a warp touching "their" node v touch
// consecutive addresses of every per-node array (blob, solver scratch, states).
// Parents precede their children in the node order (v_parent < v), so elimination
// runs v = n-1 .. 1 folding each node into its parent, and back-substitution runs
// v = 0 .. n-1.  The rows are those of the tile kernel (increment form,
// float-float V); a thread touches only its own cell, so a step needs no barrier.
// Plans with lane tiles have no synapses, network, mechanism probes or ports;
// kExtra adds the channels outside the main mix.
template <typename Real, bool kExtra>
__global__ void __launch_bounds__(kLaneThreads, sizeof(Real) == 4 ? 8 : 4) lane_step_kernel(LaunchArgs a) {
  __shared__ int s_status;
  const TileDesc td = a.tiles[blockIdx.x];
  unsigned char* base = a.blob + td.blob_offset;
  TileView<Real> tv;
  tv.bind(td, base, a.scratch + td.scratch_offset, a.scratch + td.scratch_offset, base, a.state);
  const int L = blockDim.x, lane = threadIdx.x;
  const int n = reinterpret_cast<const int32_t*>(base + td.off_lane_n)[lane];
  const uint16_t* par = tv.crec;  // parent v of each node
  const Real dt = Real(a.dt);
  const PulseRec* pulses = a.pulses + td.pulse_offset;
  if (lane == 0) s_status = 0;
  __syncthreads();
  // the rows of the first step from the current state
  for (int k = 0; k < n; ++k) {
    const int i = k * L + lane;
    const uint16_t pr = tv.pidx[i];
    Real G = Real(0), I = Real(0);
    if (pr != kBoundary) {
      node_currents<Real, kExtra>(tv.state + i, tv.N, tv.params + size_t(pr) * tv.pstride, tv.mech[pr], tv.v[i].x, dt,
                                  G, I);
    }
    const int rec = pr == kBoundary ? -1 : int(pr);
    tv.dr[i] = node_row(tv, i, rec, dt, G, I);
    const uint16_t sp = tv.spec[i];
    if (sp != kNoSpecial) add_node_pulses(tv, pulses, tv.specs[sp], i, rec, a.step0, dt);
  }
  for (int s = 0; s < a.n_steps; ++s) {
    const int64_t step = a.step0 + s;
    // Elimination, deepest node first.  Node k's contribution to its parent stays
    // in registers (cE, cR) when the parent is node k - 1, the next one visited
    // (the common case along a branch); otherwise it is added to the parent's
    // row in memory, which only a later iteration reads.  Node k - 1's inputs are
    // loaded one iteration ahead: iteration k writes no row but its own and one of
    // a node below k - 1.
    Real cE = Real(0), cR = Real(0);
    if (n > 1) {
      int i = (n - 1) * L + lane;
      int pv = par[i];
      Pair<Real> q = tv.dr[i], c = coef<Real, false>(tv, i, dt), vi = tv.v[i], vp = tv.v[pv * L + lane];
      for (int k = n - 1; k >= 1; --k) {
        const int i1 = i - L;
        int pv1 = 0;
        Pair<Real> q1 = q, c1 = c, vi1 = vi, vp1 = vp;
        if (k > 1) {
          pv1 = par[i1];
          q1 = tv.dr[i1];
          c1 = coef<Real, false>(tv, i1, dt);
          vi1 = tv.v[i1];
          vp1 = tv.v[pv1 * L + lane];
        }
        const Real delta = vdelta<Real>(vi, vp);
        const Real E = q.x + cE;  // excess form, as in the segment elimination: no subtraction in the pivots
        const Real inv = pivot_rcp(E + c.x);
        const Real Rp = (q.y + cR) - c.x * delta;
        tv.dr[i] = make_pair(inv, Rp);
        const Real w = c.y * inv;
        const Real oE = w * E, oR = w * Rp + c.y * delta;
        if (pv == k - 1) {
          cE = oE;
          cR = oR;
        } else {
          const int ip = pv * L + lane;
          Pair<Real> pp = tv.dr[ip];
          pp.x += oE;
          pp.y += oR;
          tv.dr[ip] = pp;
          cE = Real(0);
          cR = Real(0);
        }
        i = i1;
        pv = pv1;
        q = q1;
        c = c1;
        vi = vi1;
        vp = vp1;
      }
    }
    // the root, then back-substitution root first; x of node k - 1 stays in a
    // register for a child that follows its parent
    Real x_prev = Real(0);
    if (n > 0) {
      const Pair<Real> q = tv.dr[lane];
      const Real inv = pivot_rcp(q.x + cE);
      x_prev = (q.y + cR) * inv;
      tv.dr[lane] = make_pair(inv, x_prev);
    }
    if (n > 1) {
      int i = L + lane;
      int pv = par[i];
      Pair<Real> q = tv.dr[i];
      Real al = coef<Real, false>(tv, i, dt).x;
      for (int k = 1; k < n; ++k) {
        const int i1 = i + L;
        int pv1 = 0;
        Pair<Real> q1 = q;
        Real al1 = al;
        if (k + 1 < n) {
          pv1 = par[i1];
          q1 = tv.dr[i1];
          al1 = coef<Real, false>(tv, i1, dt).x;
        }
        const Real xp = pv == k - 1 ? x_prev : tv.dr[pv * L + lane].y;
        const Real x = (q.y + al * xp) * q.x;
        tv.dr[i].y = x;
        x_prev = x;
        i = i1;
        pv = pv1;
        q = q1;
        al = al1;
      }
    }
    // update: V += x, mechanisms, the next row, probes and next pulses; the next
    // node's region and states are loaded one iteration ahead
    const bool last = s + 1 == a.n_steps;
    const int64_t k_since = step + 1 - a.trace_base;
    const bool record = a.record_every > 0 && k_since % a.record_every == 0;
    NodeStates<Real, 1> cur;
    uint16_t pr_cur = kBoundary;
    if (n > 0) {
      pr_cur = tv.pidx[lane];
      if (pr_cur != kBoundary) load_states(tv.state + lane, tv.N, tv.mech[pr_cur], cur);
    }
    for (int k = 0; k < n; ++k) {
      const int i = k * L + lane;
      NodeStates<Real, 1> nxt;
      uint16_t pr_nxt = kBoundary;
      if (k + 1 < n) {
        pr_nxt = tv.pidx[i + L];
        if (pr_nxt != kBoundary) load_states(tv.state + i + L, tv.N, tv.mech[pr_nxt], nxt);
      }
      const Pair<Real> vv = tv.v[i];
      Real hi = vv.x, lo = vv.y;
      const Real v_old = hi, lo_old = lo;
      ff_add(hi, lo, tv.dr[i].y);
      tv.v[i] = make_pair(hi, lo);
      if (last) {  // last_V of the per-CV spike indicator
        tv.state[size_t(kSlotVLastHi) * tv.N + i] = v_old;
        tv.state[size_t(kSlotVLastLo) * tv.N + i] = lo_old;
      }
      if (!is_finite_real(hi)) s_status = kStatusNonfinite;
      const uint16_t pr = pr_cur;
      Real G = Real(0), I = Real(0);
      if (pr != kBoundary)
        one_node<Real, kExtra, true>(cur, tv.state + i, tv.N, tv.params + size_t(pr) * tv.pstride, tv.mech[pr], v_old,
                                     hi, dt, G, I);
      cur = nxt;
      pr_cur = pr_nxt;
      const int rec = pr == kBoundary ? -1 : int(pr);
      if (!last) tv.dr[i] = node_row(tv, i, rec, dt, G, I);
      const uint16_t sp = tv.spec[i];
      if (sp != kNoSpecial) {
        const SpecRec sr = tv.specs[sp];
        if (sr.probe >= 0) {
          const double v1 = double(hi) + double(lo), v0 = double(v_old) + double(lo_old);
          if (v0 < 0.0 && v1 >= 0.0) {
            const int cnt = a.spike_count[sr.probe];
            if (cnt < a.max_spikes)
              a.spike_times[int64_t(sr.probe) * a.max_spikes + cnt] =
                  double(step) * a.dt + a.dt * (0.0 - v0) / (v1 - v0);
            a.spike_count[sr.probe] = cnt + 1;
          }
          if (record) {
            const int64_t slot = k_since / a.record_every - 1;
            if (slot >= 0 && slot < a.trace_cap) a.traces[slot * a.n_probes_total + sr.probe] = v1;
          }
        }
        if (!last) add_node_pulses(tv, pulses, sr, i, rec, step + 1, dt);
      }
    }
  }
  __syncthreads();
  if (lane == 0 && s_status) atomicOr(a.status, s_status);
}

static void* lane_kernel(int precision, bool extra) {
  if (precision == BC_PREC_F64)
    return extra ? reinterpret_cast<void*>(lane_step_kernel<double, true>)
                 : reinterpret_cast<void*>(lane_step_kernel<double, false>);
  return extra ? reinterpret_cast<void*>(lane_step_kernel<float, true>)
               : reinterpret_cast<void*>(lane_step_kernel<float, false>);
}

int launch_lanes(const LaunchArgs& a, int precision, int threads, bool extra, void* stream) {
  if (a.n_tiles <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (threads != kLaneThreads) return int(cudaErrorInvalidConfiguration);
  if (precision == BC_PREC_F64) {
    if (extra)
      lane_step_kernel<double, true><<<a.n_tiles, threads, 0, st>>>(a);
    else
      lane_step_kernel<double, false><<<a.n_tiles, threads, 0, st>>>(a);
  } else {
    if (extra)
      lane_step_kernel<float, true><<<a.n_tiles, threads, 0, st>>>(a);
    else
      lane_step_kernel<float, false><<<a.n_tiles, threads, 0, st>>>(a);
  }
  return int(cudaGetLastError());
}

int lane_node_params(const LaunchArgs* a, int precision, int threads, bool extra, cudaKernelNodeParams* np,
                     const LaunchArgs** hold) {
  if (threads != kLaneThreads) return int(cudaErrorInvalidConfiguration);
  *hold = a;
  np->func = lane_kernel(precision, extra);
  np->gridDim = dim3(a->n_tiles, 1, 1);
  np->blockDim = dim3(threads, 1, 1);
  np->sharedMemBytes = 0u;
  np->extra = nullptr;
  np->kernelParams = reinterpret_cast<void**>(const_cast<LaunchArgs**>(hold));
  return 0;
}

// Reset: V from the initial image, gates at steady state, Ci = Ci0.
template <typename Real>
__global__ void reset_kernel(LaunchArgs a, const double* vinit, const int64_t* vinit_off) {
  const TileDesc td = a.tiles[blockIdx.x];
  unsigned char* base = a.blob + td.blob_offset;
  TileView<Real> tv;
  tv.bind(td, base, base, base, base, a.state);  // scratch unused
  const double* vi = vinit + vinit_off[blockIdx.x];
  for (int i = threadIdx.x; i < tv.n_real; i += blockDim.x) {
    const Real v = Real(vi[i]);
    tv.v[i] = make_pair(v, Real(0));
    tv.state[size_t(kSlotVLastHi) * tv.N + i] = v;  // no step taken: no crossing
    tv.state[size_t(kSlotVLastLo) * tv.N + i] = Real(0);
    const uint16_t pr = tv.pidx[i];
    if (pr == kBoundary) continue;
    const Real* P = tv.params + size_t(pr) * tv.pstride;
    steady_states(P, tv.mech[pr], tv.state + i, tv.N, v);
  }
}

// Reads, writes or tests one named view of every CV, in the reference's CV order
// (view_args): the addresses come from the plan's CV map and tile descriptors, so that a
// call uploads nothing and allocates nothing (tables of byte offsets, built on the host
// and copied on every call, took 24 ms for 5.8 million CVs).
template <typename Real>
__global__ void view_kernel(const TileDesc* tiles, unsigned char* blob, Real* state, const int2* cv, ViewArgs va,
                            double* view, int64_t n) {
  for (int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; k < n; k += int64_t(gridDim.x) * blockDim.x) {
    const int2 c = cv[k];
    const TileDesc& d = tiles[c.x];
    const unsigned char* base = blob + d.blob_offset;
    Pair<Real>& v = reinterpret_cast<Pair<Real>*>(blob + d.blob_offset + d.off_v)[c.y];
    Real* st = state + d.state_offset + c.y;
    const int64_t N = d.n_nodes;
    if (va.mode == kViewSpike) {
      const double last = double(st[kSlotVLastHi * N]) + double(st[kSlotVLastLo * N]), now = double(v.x) + double(v.y);
      view[k] = last < va.v_th && now >= va.v_th ? 1.0 : 0.0;
      continue;
    }
    bool present = true;
    if (va.owner != 0) {
      const uint16_t pr = reinterpret_cast<const uint16_t*>(base + d.off_pidx)[c.y];
      present = pr != kBoundary;
      if (present) {
        const uint32_t m = reinterpret_cast<const uint32_t*>(base + d.off_mech)[pr];
        uint64_t bits = m;
        if (m & BC_M_EXT)
          bits |= uint64_t(ext_mask(reinterpret_cast<const Real*>(base + d.off_params) + size_t(pr) * d.param_stride))
                  << 32;
        present = (bits & va.owner) != 0;
      }
    }
    if (!present) {
      if (va.mode == kViewRead) view[k] = __longlong_as_double(0x7ff8000000000000LL);
      continue;
    }
    Real* hi = va.slot < 0 ? &v.x : st + va.slot * N;
    Real* lo = va.slot < 0 ? &v.y : (va.slot_lo >= 0 ? st + va.slot_lo * N : nullptr);
    if (va.mode == kViewWrite) {
      const double x = view[k];
      *hi = Real(x);
      if (lo) *lo = Real(x - double(*hi));
      if (va.slot < 0) {  // a new voltage starts a fresh history: no step has crossed anything since
        st[kSlotVLastHi * N] = *hi;
        st[kSlotVLastLo * N] = *lo;
      }
    } else {
      view[k] = double(*hi) + (lo ? double(*lo) : 0.0);
    }
  }
}

// New amplitudes (nA, batch order) into the pulse records.
__global__ void pulse_amp_kernel(PulseRec* pulses, const int32_t* src, const double* scale, const double* amp,
                                 int64_t n) {
  for (int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; k < n; k += int64_t(gridDim.x) * blockDim.x)
    pulses[k].amp = amp[src[k]] * scale[k];
}

// ------------------------------------------------------------------ launchers
static void cluster_config(const LaunchArgs& a, int threads, size_t smem_bytes, cudaStream_t st, cudaLaunchConfig_t& cfg,
                           cudaLaunchAttribute& attr) {
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = unsigned(a.cluster);
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3(unsigned(a.n_tiles) * unsigned(a.cluster), 1, 1);
  cfg.blockDim = dim3(unsigned(threads), 1, 1);
  cfg.dynamicSmemBytes = smem_bytes;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
}

// Lets a tile kernel take as much dynamic shared memory as any plan may need, and clusters
// of 16, once for each plan that runs it.  Both limits belong to the kernel, not to the
// launch: set to each launch's own size, the first could be lowered by another thread's plan
// just before the launch, which then failed.
template <typename Kernel>
static cudaError_t raise_limits(Kernel k, bool clusters) {
  int device = 0, cap = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&cap, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, cap - kStaticSmem);
  if (e == cudaSuccess && clusters) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

template <int kVar>
static int prepare_x(int precision, bool smem) {
  if (precision == BC_PREC_F64)
    return int(smem ? raise_limits(tile_step_kernel<double, true, kVar>, false)
                    : raise_limits(tile_step_kernel<double, false, kVar>, kVar < 2));
  return int(smem ? raise_limits(tile_step_kernel<float, true, kVar>, false)
                  : raise_limits(tile_step_kernel<float, false, kVar>, kVar < 2));
}

int prepare_tiles(int precision, bool smem, int variant) {
  switch (variant) {
    case 0:
      return prepare_x<0>(precision, smem);
    case 1:
      return prepare_x<1>(precision, smem);
    case 2:
      return prepare_x<2>(precision, smem);
    default:
      return prepare_x<3>(precision, smem);
  }
}

template <typename Real, bool kSmem, int kVar>
static int launch_impl(const LaunchArgs& a, int threads, size_t smem_bytes, cudaStream_t st) {
  auto k = tile_step_kernel<Real, kSmem, kVar>;
  if (!kSmem && a.cluster > 1) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    cluster_config(a, threads, smem_bytes, st, cfg, attr);
    return int(cudaLaunchKernelEx(&cfg, k, a));
  }
  k<<<a.n_tiles, threads, smem_bytes, st>>>(a);
  return int(cudaGetLastError());
}

// The largest power of two up to `want` at which `count` clusters are resident at once.
template <typename Real, int kVar>
static int usable_cluster(int want, int count, int threads, size_t smem_bytes) {
  auto k = tile_step_kernel<Real, false, kVar>;
  if (raise_limits(k, true) != cudaSuccess) return 1;
  for (int c = want; c > 1; c /= 2) {
    LaunchArgs a{};
    a.n_tiles = 1;
    a.cluster = c;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    cluster_config(a, threads, smem_bytes, nullptr, cfg, attr);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) == cudaSuccess && n >= count) return c;
    (void)cudaGetLastError();
  }
  return 1;
}

int tile_cluster(int precision, int variant, int want, int count, int threads, size_t smem_bytes) {
  if (variant > 1) return 1;
  if (precision == BC_PREC_F64)
    return variant ? usable_cluster<double, 1>(want, count, threads, smem_bytes)
                   : usable_cluster<double, 0>(want, count, threads, smem_bytes);
  return variant ? usable_cluster<float, 1>(want, count, threads, smem_bytes)
                 : usable_cluster<float, 0>(want, count, threads, smem_bytes);
}

template <int kVar>
static int launch_tiles_x(const LaunchArgs& a, int precision, bool smem, int threads, size_t smem_bytes,
                          cudaStream_t st) {
  if (precision == BC_PREC_F64)
    return smem ? launch_impl<double, true, kVar>(a, threads, smem_bytes, st)
                : launch_impl<double, false, kVar>(a, threads, smem_bytes, st);
  return smem ? launch_impl<float, true, kVar>(a, threads, smem_bytes, st)
              : launch_impl<float, false, kVar>(a, threads, smem_bytes, st);
}

int launch_tiles(const LaunchArgs& a, int precision, bool smem, int threads, size_t smem_bytes, int variant,
                 void* stream) {
  if (a.n_tiles <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (variant) {
    case 0:
      return launch_tiles_x<0>(a, precision, smem, threads, smem_bytes, st);
    case 1:
      return launch_tiles_x<1>(a, precision, smem, threads, smem_bytes, st);
    case 2:
      return launch_tiles_x<2>(a, precision, smem, threads, smem_bytes, st);
    default:
      return launch_tiles_x<3>(a, precision, smem, threads, smem_bytes, st);
  }
}

// Kernel-node parameters of one tile launch for a CUDA graph: the same kernel,
// grid, block and shared memory as launch_tiles; `*a` is copied by the graph call
// that consumes the parameters.
template <typename Real, bool kSmem, int kVar>
static int node_impl(const LaunchArgs* a, int threads, size_t smem_bytes, cudaKernelNodeParams* np) {
  np->func = reinterpret_cast<void*>(tile_step_kernel<Real, kSmem, kVar>);
  np->gridDim = dim3(a->n_tiles, 1, 1);
  np->blockDim = dim3(threads, 1, 1);
  np->sharedMemBytes = unsigned(smem_bytes);
  np->extra = nullptr;
  return 0;
}

template <int kVar>
static int node_x(const LaunchArgs* a, int precision, bool smem, int threads, size_t smem_bytes,
                  cudaKernelNodeParams* np) {
  if (precision == BC_PREC_F64)
    return smem ? node_impl<double, true, kVar>(a, threads, smem_bytes, np)
                : node_impl<double, false, kVar>(a, threads, smem_bytes, np);
  return smem ? node_impl<float, true, kVar>(a, threads, smem_bytes, np)
              : node_impl<float, false, kVar>(a, threads, smem_bytes, np);
}

int tile_node_params(const LaunchArgs* a, int precision, bool smem, int threads, size_t smem_bytes, int variant,
                     cudaKernelNodeParams* np, const LaunchArgs** hold) {
  *hold = a;
  int e;
  switch (variant) {
    case 0:
      e = node_x<0>(a, precision, smem, threads, smem_bytes, np);
      break;
    case 1:
      e = node_x<1>(a, precision, smem, threads, smem_bytes, np);
      break;
    case 2:
      e = node_x<2>(a, precision, smem, threads, smem_bytes, np);
      break;
    default:
      e = node_x<3>(a, precision, smem, threads, smem_bytes, np);
      break;
  }
  np->kernelParams = reinterpret_cast<void**>(const_cast<LaunchArgs**>(hold));
  return e;
}

// Event delivery (network/delivery.py:361-394): each spike record (cell, step)
// of the last launch adds, for every connection of its cell, the weight into the
// ring slot of the arrival step step + max(delay, 1).  Several records can hit one
// slot: the additions are atomic, so their order (and the last bits of a sum of
// three or more weights) may vary between runs.
template <typename Real>
__global__ void deliver_kernel(const int32_t* rec_cell, const int64_t* rec_step, const unsigned long long* rec_count,
                               const unsigned long long* rec_done, int64_t rec_cap, const int64_t* out_ptr,
                               const int64_t* out_syn, const Real* out_w, const int32_t* out_d, Real* arrivals,
                               int64_t arr_slots, int64_t n_syn) {
  const int64_t r0 = int64_t(*rec_done);
  const int64_t r1 = min(int64_t(*rec_count), rec_cap);
  for (int64_t r = r0 + blockIdx.x * int64_t(blockDim.x) + threadIdx.x; r < r1; r += int64_t(gridDim.x) * blockDim.x) {
    const int32_t c = rec_cell[r];
    const int64_t s = rec_step[r];
    for (int64_t j = out_ptr[c]; j < out_ptr[c + 1]; ++j) {
      const int64_t arrive = s + max(out_d[j], 1);
      atomicAdd(arrivals + (arrive % arr_slots) * n_syn + out_syn[j], out_w[j]);
    }
  }
}

int launch_deliver_impl(int precision, const int32_t* rec_cell, const int64_t* rec_step,
                        const unsigned long long* rec_count, const unsigned long long* rec_done, int64_t rec_cap,
                        const int64_t* out_ptr, const int64_t* out_syn, const void* out_w, const int32_t* out_d,
                        void* arrivals, int64_t arr_slots, int64_t n_syn, void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (precision == BC_PREC_F64)
    deliver_kernel<double><<<152, 256, 0, st>>>(rec_cell, rec_step, rec_count, rec_done, rec_cap, out_ptr, out_syn,
                                                static_cast<const double*>(out_w), out_d,
                                                static_cast<double*>(arrivals), arr_slots, n_syn);
  else
    deliver_kernel<float><<<152, 256, 0, st>>>(rec_cell, rec_step, rec_count, rec_done, rec_cap, out_ptr, out_syn,
                                               static_cast<const float*>(out_w), out_d, static_cast<float*>(arrivals),
                                               arr_slots, n_syn);
  return int(cudaGetLastError());
}

int launch_reset_impl(const LaunchArgs& a, int precision, int threads, const double* vinit, const int64_t* voff,
                      void* stream) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (a.n_tiles <= 0) return 0;
  if (precision == BC_PREC_F64)
    reset_kernel<double><<<a.n_tiles, threads, 0, st>>>(a, vinit, voff);
  else
    reset_kernel<float><<<a.n_tiles, threads, 0, st>>>(a, vinit, voff);
  return int(cudaGetLastError());
}

static int grid_for(int64_t n, int threads) { return int(std::min<int64_t>((n + threads - 1) / threads, 65535)); }

int launch_view_impl(const TileDesc* tiles, unsigned char* blob, unsigned char* state, int precision, const int2* cv,
                     const ViewArgs& va, double* view, int64_t n, void* stream) {
  if (n <= 0) return 0;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int threads = 256;
  if (precision == BC_PREC_F64)
    view_kernel<double><<<grid_for(n, threads), threads, 0, st>>>(tiles, blob, reinterpret_cast<double*>(state), cv, va,
                                                                  view, n);
  else
    view_kernel<float><<<grid_for(n, threads), threads, 0, st>>>(tiles, blob, reinterpret_cast<float*>(state), cv, va,
                                                                 view, n);
  return int(cudaGetLastError());
}

int launch_pulse_amp_impl(PulseRec* pulses, const int32_t* src, const double* scale, const double* amp, int64_t n,
                          void* stream) {
  if (n <= 0) return 0;
  pulse_amp_kernel<<<grid_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(pulses, src, scale, amp, n);
  return int(cudaGetLastError());
}

// Scratch of bc_state_download_noalloc, part of the module image (no allocation
// call): BC_NOALLOC_MAX_CV values.
static __device__ __align__(256) unsigned char g_noalloc_view_scratch[8 * size_t(BC_NOALLOC_MAX_CV)];

int noalloc_view_scratch_address(void** out) {
  return int(cudaGetSymbolAddress(out, g_noalloc_view_scratch));
}

}  // namespace bc
