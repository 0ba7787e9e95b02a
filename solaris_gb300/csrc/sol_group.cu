// RungeKuttaFehlberg78 / RungeKutta4 driver for systems whose sinks see few
// sources, whole sequences of driver calls in one cooperative launch.
//
// Such a system is a chain of small dependent steps, so its time is the
// number of instructions on the longest chain of a stage: a warp's FP64
// instructions follow each other at 64 cycles whatever the lanes in use, its
// other instructions at ~5.  A stage is two phases with a block barrier after
// each:
//   A. worker warps: a lane per item -- a (sink, source) pair or a body and
//      the origin (rm3 is that "pair") -- forms d, |d|, |d|^-3 and d |d|^-3;
//      drag (in five roles) and migration in worker warps of their own;
//   B. state warps, one lane per state element, which holds its y0, its stage
//      sums and its error terms in registers for the whole launch: a velocity
//      lane adds the GravityAC sum of its (sink, component) in the reference's
//      order, the Kepler term and the gas term; then the next stage input.
// Every stage sum takes its terms in ascending stage order, so a lane adds
// f_r to the sums of all later stages as soon as it has it: only the next
// stage's is on the chain, the others are added during the next phase A, when
// the state warps have nothing else to do (a gather over the stage history
// from shared memory put up to nine multiplications and additions there).
// The sources (the first nm + n_spl bodies: star, planets, super-
// planetesimals) are integrated redundantly by every CTA, so no data crosses
// CTAs during an attempt, and one group barrier per attempt carries the error
// norm.  Each CTA also owns a contiguous range of the other bodies.  The
// arithmetic, operation by operation, is that of the persistent and
// host-driven drivers (and so of the reference,
// RungeKuttaFehlberg78.cpp:66-262, Acceleration.cpp:166-329): the results are
// bit-identical.
//
// The group barrier spins on a generation counter with an iteration limit; a
// CTA that runs out raises SOL_DEV_TIMEOUT and an abort flag that makes every
// other CTA leave at its next barrier; the resident state is then that before
// the launch.  (sol_set_wait_test lowers the limit and can keep one CTA from
// arriving, so that tests reach this path.)
#include <atomic>
#include <mutex>
#include <algorithm>
#include <cmath>
#include <cstring>

#include "sol_crmath.cuh"

namespace {

#define RET(x)                   \
  do {                           \
    int r_ = (x);                \
    if (r_ != SOL_OK) return r_; \
  } while (0)

constexpr int kMaxSources = 32;   // nm + n_spl
constexpr int kMinLocal = 4;      // other bodies per CTA
constexpr int kMaxLocal = 128;
constexpr int kMaxThreads = 1024;
constexpr int kMaxCtas = 256;     // one per SM
constexpr int kWorkersMin = 2;
constexpr int kSpreadSmem = 116 * 1024;  // > half of the 228 KB of an SM: one CTA per SM

struct GroupArgs {
  ForceCtx fc;
  double* y0;           // resident state [6N]
  double* accel;        // f0 of the last driver call
  double* yscale;
  double* ynew;
  double* err;
  unsigned long long* words;  // [2][2][kMaxCtas]: the CTAs' words of exchange()
  int* abort_flag;
  unsigned spin;        // polls of an exchange before it gives up
  int skip_cta;         // failure-path tests: this CTA never arrives (-1: none)
  sol_ctrl* ctrl;
  int n;
  int ns;               // sources: nm + n_spl
  int local;            // other bodies per CTA
  int n_steps;
  int rk4;              // RungeKutta4 driver calls instead of RungeKuttaFehlberg78
  int sim;              // the Simulator's step loop (sol_run_until)
  double e3, h3, cf;    // its event thresholds (0: off)
  sol_sim_line* line;
  int* reason;
  double* yprev;        // the state at the start of a step that stops with an event (or null)
  int vw;               // velocity warps (and as many position warps); the other warps are workers
  int icap;             // items a CTA has room for
  // shared-memory layout (offsets in doubles)
  int o_yt, o_p, o_x, o_gm, o_gbuf, o_dv, o_int;
};

// Exchange k of the launch among the CTAs, by the first warp of each: the
// largest of all CTAs' `mine` (bits of a double that is not negative) and
// whether any has `flag`; false when the wait ran out or another CTA gave up.
// Every CTA stores its word and polls everyone's, so a word's arrival is the
// barrier (~4,000 cycles among 64 CTAs, most of it two or three trips to L2,
// and ~6,000 among 127).  The sign bit is the phase: a word is new when it has this
// exchange's.  Two sets of words alternate; a CTA stores to a set again two
// exchanges later, when every CTA has stored to the other and so has read
// this one.  The words start at zero, the first phase is 1.
struct Exchanged {
  long long worst;
  int any, ok;
};
__device__ __noinline__ Exchanged exchange(const GroupArgs& P, unsigned k, long long mine, int flag) {
  const int lane = threadIdx.x & 31, grid = gridDim.x;
  const int sets = P.sim ? 2 : 1;
  unsigned long long* set = P.words + (size_t)(k & 1) * 2 * kMaxCtas;
  const unsigned long long phase = (unsigned long long)(((k >> 1) & 1) ^ 1) << 63;
  auto store = [](unsigned long long* at, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(at), "l"(v) : "memory");
  };
  if (lane == 0 && (int)blockIdx.x != P.skip_cta) {
    if (P.sim) store(set + kMaxCtas + blockIdx.x, phase | (unsigned long long)(flag != 0));
    store(set + blockIdx.x, phase | (unsigned long long)mine);
  }
  unsigned long long got[2] = {0, 0};
  for (uint32_t q = 0;; ++q) {
    bool all = true;
    for (int t = 0; t < sets; ++t) {
      unsigned long long v[kMaxCtas / 32];  // every load in flight at once
#pragma unroll
      for (int u = 0; u < kMaxCtas / 32; ++u) {
        v[u] = phase;
        if (lane + 32 * u < grid)
          asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[u]) : "l"(set + t * kMaxCtas + lane + 32 * u) : "memory");
      }
      unsigned long long w = 0;
#pragma unroll
      for (int u = 0; u < kMaxCtas / 32; ++u) {
        all = all && (v[u] & (1ull << 63)) == phase;
        const unsigned long long m = v[u] & ~(1ull << 63);
        w = m > w ? m : w;
      }
      got[t] = w;
    }
    if (__all_sync(0xFFFFFFFFu, all)) break;
    // a limit reached, or (looked at now and then) another CTA that gave up
    const bool over = q >= P.spin;
    if (over || (q & 15) == 15) {
      const bool gone = *(volatile int*)P.abort_flag != 0;
      if (over && !gone && lane == 0) {
        atomicOr(&P.ctrl->dev_status, SOL_DEV_TIMEOUT);
        atomicExch(P.abort_flag, 1);
      }
      if (__any_sync(0xFFFFFFFFu, over || gone)) return Exchanged{0, 0, 0};
    }
    if (q >= 256) __nanosleep(32);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long v = __shfl_xor_sync(0xFFFFFFFFu, got[0], o);
    got[0] = v > got[0] ? v : got[0];
  }
  return Exchanged{(long long)got[0], (int)__reduce_or_sync(0xFFFFFFFFu, (unsigned)got[1]), 1};
}

// barrier of a CTA's worker warps (1) or state warps (2) alone
__device__ __forceinline__ void part_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

struct Ctl {
  double t, h, h_next, h_did, error_max, eps;
  long long n_acc, n_rej;
  int status, accepted, abort, nitem, ndrag, nmig;
  double m0pt;
  int event, stop, reason, flush;
  sol_sim_line L;
  long long red[32];  // bits of the state warps' largest |error / yscale|
  // the next evaluation, for the worker warps
  double factor;
  uint32_t flags;
  int cur, last, leave;
};

// Per-CTA view of the shared memory.  Sink slot s < ns is source (body) s,
// slot s >= ns is body l0 + s - ns; slot `zero` of a stage input is the origin.
// The items of a sink follow each other: the origin, then its sources in
// ascending order.
struct View {
  double* yt;    // [2][6 (cap + 1)] stage inputs, double-buffered
  double* p;     // [5][icap] d |d|^-3, then the item's term of GravityAC (3); |d|^-3, |d|
  double* x;     // [3][kMaxSources] r_j rm3_j of the sources
  double* gm;    // [icap]: G m of the item's source; of the origin, -G (m_0 + m_i)
  double* gbuf;  // [3 cap]: drag or migration buffer of each sink
  double* dv;    // [kRoleValues][cap]: the drag's partial results of each planetesimal
  int* ends;     // [icap]: slot subtracted | slot << 16
  int* base;     // [cap + 1]: first item of each sink
  int* mig;      // [cap]: migType of each sink
  int* kind;     // [cap]: gas buffer kind
  int* dlist;    // [ndrag]: slots of the planetesimals (drag)
  int* mlist;    // [nmig]: slots of the migrating bodies
  int stride;    // doubles of one stage input
  int icap, cap, l0, nsink;
};

// Which gas buffer a body uses (Acceleration::ComputeAstroCentric :176-243):
// 1 drag, 2 type-I migration, 3 type-II migration, 0 none.
__device__ __forceinline__ int gas_kind(const ForceCtx& fc, int i) {
  if (!fc.gas.present) return 0;
  const Classes& c = fc.cls;
  if (i >= c.nm && i < c.nm + c.n_spl + c.n_pl) return 1;
  if (fc.has_mig1 && i >= c.n_central + c.n_giant && i < c.nm) return 2;
  if (fc.has_mig2 && i >= c.n_central && i < c.n_central + c.n_giant) return 3;
  return 0;
}

__device__ __forceinline__ double* global_gas_buf(const ForceCtx& fc, int i, int kind) {
  const Classes& c = fc.cls;
  if (kind == 1) return fc.drag + 3 * (i - c.nm);
  if (kind == 2) return fc.mig1 + 3 * (i - (c.n_central + c.n_giant));
  return fc.mig2 + 3 * (i - c.n_central);
}

// Migration of one massive body (the migration part of add_gas_terms): only
// with its flag and while migType allows it (a migration that reaches its
// stop sets migType to No).  Out of line, like the drag: thousands of
// instructions inlined into the stage loop evict the hot path from the
// instruction cache (measured: 3x slower stages).
__device__ __noinline__ void mig_compute(const ForceCtx& fc, int i, int kind, const double* yi, double factor,
                                         uint32_t flags, double* buf, int* mig) {
  const GasDev& g = fc.gas;
  const double m0 = fc.mass[0];
  double d[3];
  if (kind == 2) {
    if (!((flags & SOL_EVAL_TYPE_I) && *mig == SOL_MIGRATION_TYPE_I)) return;
    if (!sol_migration_type1(g, factor, m0, fc.mass[i], fc.mig_stop_at[i], yi, d)) *mig = SOL_MIGRATION_NO;
  } else {
    if (!((flags & SOL_EVAL_TYPE_II) && *mig == SOL_MIGRATION_TYPE_II)) return;
    if (!sol_migration_type2(g, factor, m0, fc.mass[i], fc.mig_stop_at[i], yi, d)) *mig = SOL_MIGRATION_NO;
  }
  buf[0] = d[0];
  buf[1] = d[1];
  buf[2] = d[2];
}

// The rest of GasDragAC (Acceleration.cpp:364-401) from the roles' values: the
// gas velocity (GasComponent.cpp:97-138) and the regime.
__device__ __forceinline__ void drag_finish(const GasDev& g, double factor, double m0pt, const double* yi,
                                           double radius, double density, double cd, double gs, double ge,
                                           const double* dv, int cap, double out[3]) {
  const double lambda = dv[0], r = dv[cap], p = dv[2 * cap], w = dv[3 * cap], ex = dv[4 * cap], rp = dv[5 * cap],
               vc = dv[6 * cap], v = dv[7 * cap];
  double vgx = 0.0, vgy = 0.0;
  {
    const double x = yi[0], y = yi[1];
    if (x == 0.0 && y == 0.0) {
    } else if (y == 0.0) {
      vgy = x > 0.0 ? vc : -vc;
    } else if (x == 0.0) {
      vgx = y > 0.0 ? -vc : vc;
    } else if (x >= y) {
      vgy = x >= 0 ? vc / w : -vc / w;
      vgx = -vgy * p;
    } else {
      vgx = y >= 0 ? -vc / w : vc / w;
      vgy = -vgx * p;
    }
    vgx *= v;
    vgy *= v;
  }
  const double ux = yi[3] - vgx, uy = yi[4] - vgy, uz = yi[5] - 0.0;
  const double rho = rp * ex;
  const double rhoGas = factor * rho;
  double C;
  if (radius <= 0.1 * lambda) {
    // MeanThermalSpeed_CMU(m0, r) -> Temperature_CMU(r, m0) (arguments swapped, :241)
    const double cT = g.sh_c * g.sh_c * r * g.mmw * g.ctp;
    const double vth = g.cvth * sqrt(cT * m0pt);
    C = ge * vth * rhoGas;
  } else if (radius >= 10.0 * lambda) {
    const double ul = sqrt(ux * ux + uy * uy + uz * uz);
    C = gs * ul * rhoGas;
  } else {
    const double l1 = 0.1 * lambda, l2 = 10.0 * lambda;
    const double gE = 1.0 / (density * l1);
    const double gS = 3.0 / 8.0 * cd / (density * l2);
    const double cT = g.sh_c * g.sh_c * r * g.mmw * g.ctp;
    const double vth = g.cvth * sqrt(cT * m0pt);
    const double ul = sqrt(ux * ux + uy * uy + uz * uz);
    const double K = gS * ul / (gE * vth);
    const double eta = l2 / l1;
    const double kappa = log10(K) / log10(eta);
    const double gamma = gE * vth * pow(l1, -kappa);
    C = gamma * pow(radius, kappa) * rhoGas;
  }
  out[0] = -C * ux;
  out[1] = -C * uy;
  out[2] = -C * uz;
}

// One of the five independent parts of GasDragAC (Acceleration.cpp:342-363,
// gas_velocity and gas_density_at of GasComponent.cpp:97-157) for the
// planetesimal of this lane, in the operations of sol_gas_drag:
//   role 0: r, the mean free path lambda(r), and the ratio p of the circular
//           velocity's components with sqrt(1 + p^2);
//   role 1: the density's vertical exponential exp(-(z / h(rc))^2);
//   role 2: the density's power law (or the inner-edge form);
//   role 3: the circular velocity;
//   role 4: its eta(rc) correction.
// A warp takes one role for 32 planetesimals, so its lanes share the
// exponent of their power and run the same instructions; the roles run in
// warps side by side and drag_finish combines them.  Into dv, at stride cap:
// lambda, r, p, sqrt(1 + p^2), the exponential, the power law, the circular
// velocity, the correction.
constexpr int kRoles = 5, kRoleValues = 8;
__device__ __noinline__ void drag_role(const GasDev& g, int role, double m0, const double* yi, double* dv, int cap) {
  const double x = yi[0], y = yi[1], z = yi[2];
  if (role == 0) {
    const double r = sqrt(x * x + y * y + z * z);
    dv[0] = sol_pl(g.mfp_c, g.mfp_i, r);
    dv[cap] = r;
    const double p = x >= y ? y / x : x / y;
    dv[2 * cap] = p;
    dv[3 * cap] = sqrt(1.0 + p * p);
    return;
  }
  const double rc = sqrt(x * x + y * y);
  if (role == 1) {
    const double hh = sol_pl(g.sh_c, g.sh_i, rc);
    const double qq = z / hh;
    dv[4 * cap] = sol_exp_neg(qq * qq);
  } else if (role == 2) {
    if (g.inner_edge < rc) {
      dv[5 * cap] = sol_pl(g.rho_c, g.rho_i, rc);
    } else {
      const double r2c = rc * rc;
      dv[5 * cap] = (g.rho_c * sol_pow(g.inner_edge, g.rho_i - 4.0)) * (r2c * r2c);
    }
  } else if (role == 3) {
    dv[6 * cap] = sqrt((SOL_GAUSS2 * m0) / rc);
  } else {
    dv[7 * cap] = sqrt(1.0 - 2.0 * sol_pl(g.eta_c, g.eta_i, rc));
  }
}

__device__ __forceinline__ int body_of(const GroupArgs& P, const View& V, int s) {
  return s < P.ns ? s : V.l0 + s - P.ns;
}

// What the host reads of an attempt's last evaluation, by the worker warps
// after it: rm3, the nearest neighbour (the smallest |d_ij|, the first in
// source order) and CheckEvent's predicates.  The block barrier at the end
// orders it before the step decision and before the next evaluation.
__device__ __noinline__ void last_evaluation(const GroupArgs& P, const View& V, int* event, int thread, int threads) {
  const ForceCtx& fc = P.fc;
  const bool home = blockIdx.x == 0;
  for (int s = thread; s < V.nsink; s += threads) {
    const int i = body_of(P, V, s);
    if (!(s >= P.ns || home)) continue;
    if (i == 0) {
      fc.nn_idx[0] = -1;
      fc.nn_dist[0] = 0.0;
      continue;
    }
    const int first = V.base[s], end = V.base[s + 1];
    long long rminb = __double_as_longlong(1.0e10);
    int nn = -1;
    for (int it = first + 1; it < end; ++it) {
      const long long rb = __double_as_longlong(V.p[4 * V.icap + it]);
      if (rb < rminb) {
        rminb = rb;
        nn = V.ends[it] >> 16;  // source j is slot j
      }
    }
    const double rm3 = V.p[3 * V.icap + first];
    fc.rm3[i] = rm3;
    fc.nn_idx[i] = nn;
    fc.nn_dist[i] = nn >= 0 ? __longlong_as_double(rminb) : 0.0;
    if (P.sim) {
      const bool ev = (P.e3 > 0.0 && rm3 < P.e3) || (P.h3 > 0.0 && rm3 > P.h3) ||
                      (P.cf > 0.0 && nn >= 0 && P.cf * (fc.radius[i] + fc.radius[nn]) > __longlong_as_double(rminb));
      if (ev) atomicOr(event, 1);
    }
  }
  __syncthreads();
}

// An item in two passes.  The first: rm3 of a body or d |d|^-3 and |d| of a
// pair (GravityAC, Acceleration.cpp:259-261, :294-308), the root and the
// reciprocal by sol_ref_rinv3: latency counts here, and its one FP64
// instruction among FP32 and integer ones is a shorter chain than IEEE square
// root and reciprocal (40 driver calls of 256 bodies: 1.56 ms for 1.86; four
// of 8,193 in gas: 0.608 for 0.634).  The second, once every first pass is
// done: the Kepler term -mu rm3 r of a body (:281-283), G m_j (d |d|^-3 -
// r_j rm3_j) of a pair, both as a fused multiply-add and a multiplication
// (x * 1 - y and x * y - 0 round once, as x - y and x * y do).
__device__ __forceinline__ void first_pass(const View& V, const double* yt, int it, int ends) {
  const double* yi = yt + 6 * (ends & 0xFFFF);
  const double* yj = yt + 6 * (ends >> 16);
  const double xij = yj[0] - yi[0];
  const double yij = yj[1] - yi[1];
  const double zij = yj[2] - yi[2];
  const double rij2 = xij * xij + yij * yij + zij * zij;
  double rij, rijm3;
  sol_ref_rinv3(rij2, rij, rijm3);
  double* p = V.p + it;
  p[0] = xij * rijm3;
  p[V.icap] = yij * rijm3;
  p[2 * V.icap] = zij * rijm3;
  p[3 * V.icap] = rijm3;
  p[4 * V.icap] = rij;
  const int j = ends >> 16;
  if ((ends & 0xFFFF) == V.cap && j < kMaxSources) {  // slot j < ns is a source (a slot beyond them is not read)
    V.x[j] = xij * rijm3;
    V.x[kMaxSources + j] = yij * rijm3;
    V.x[2 * kMaxSources + j] = zij * rijm3;
  }
}
__device__ __forceinline__ double second_pass(bool body, double r, double rm3, double pp, double pj, double gm) {
  const double u = __fma_rn(body ? gm : pp, body ? rm3 : 1.0, body ? -0.0 : -pj);
  return u * (body ? r : gm);
}

// The worker warps of a system without gas whose items, four lanes each, fit
// its workers at once: a lane per component (8 FP64 instructions on the chain
// of a first pass besides the root and the reciprocal's instead of 13), its
// addresses kept in registers.
__device__ __forceinline__ void work_by_component(const GroupArgs& P, const View& V, const Ctl& S, int w, int lane,
                                                  int nwork) {
  const int c = lane & 3, it = (w * 32 + lane) >> 2;
  const bool live = it < S.nitem;
  const int ends = live ? V.ends[it] : 0;
  const bool body = (ends & 0xFFFF) == V.cap;
  const int ca = c < 3 ? c : 0;
  const double* bi = V.yt + 6 * (ends & 0xFFFF) + ca;
  const double* bj = V.yt + 6 * (ends >> 16) + ca;
  double* p = V.p + (size_t)c * V.icap + it;  // c = 3: |d|^-3
  const int j = ends >> 16;
  const bool source = live && body && c < 3 && j < kMaxSources;
  double* xj = V.x + ca * kMaxSources + (j < kMaxSources ? j : 0);
  const double gm = live ? V.gm[it] : 0.0;
  for (;;) {
    __syncthreads();
    if (S.leave) return;
    const int o = S.cur * V.stride, last = S.last;  // (all of Ctl's between the two barriers: submit() writes the next)
    const double x = bj[o] - bi[o];
    const double sq = x * x;
    const double qx = __shfl_sync(0xFFFFFFFFu, sq, 0, 4), qy = __shfl_sync(0xFFFFFFFFu, sq, 1, 4),
                 qz = __shfl_sync(0xFFFFFFFFu, sq, 2, 4);
    const double rij2 = qx + qy + qz;
    double rij = 0.0, rijm3 = 0.0;
    if (live) sol_ref_rinv3(rij2, rij, rijm3);
    const double pp = x * rijm3;
    if (live) {
      if (source) *xj = pp;
      if (c == 3) {
        p[0] = rijm3;
        p[V.icap] = rij;
      }
    }
    part_sync(1, nwork * 32);
    const double t = second_pass(body, x, rijm3, pp, *xj, gm);
    if (live && c < 3) p[0] = t;
    __syncthreads();
    if (last) last_evaluation(P, V, const_cast<int*>(&S.event), w * 32 + lane, nwork * 32);
  }
}

// The worker warps: for every evaluation between the two block barriers the
// items, and drag and migration of systems with gas, in units of a warp.
__device__ __noinline__ void work(const GroupArgs& P, const View& V, const Ctl& S) {
  const ForceCtx& fc = P.fc;
  const bool home = blockIdx.x == 0;
  const int lane = threadIdx.x & 31;
  const int nwork = (int)(blockDim.x >> 5) - 2 * P.vw;
  const int w = (int)(threadIdx.x >> 5) - 2 * P.vw;
  const int nitem = S.nitem, ndrag = S.ndrag, nmig = S.nmig;
  if (ndrag == 0 && nmig == 0 && 4 * nitem <= 32 * nwork) {
    work_by_component(P, V, S, w, lane, nwork);
    return;
  }
  const int w_role = (ndrag + 31) >> 5;
  for (;;) {
    __syncthreads();
    if (S.leave) return;
    const double* yt = V.yt + S.cur * V.stride;
    const uint32_t flags = S.flags;
    const int last = S.last;  // (as above)
    const bool drag = ndrag > 0 && (flags & SOL_EVAL_GAS_DRAG);
    const bool mig = nmig > 0 && (flags & (SOL_EVAL_TYPE_I | SOL_EVAL_TYPE_II));
    const int u_drag = drag ? kRoles * w_role : 0;
    const int u_mig = u_drag + (mig ? (nmig + 31) >> 5 : 0);
    const int units = u_mig + ((nitem + 31) >> 5);
    for (int u = w; u < units; u += nwork) {  // the longest first
      if (u >= u_mig) {
        const int it = (u - u_mig) * 32 + lane;
        if (it < nitem) first_pass(V, yt, it, V.ends[it]);
      } else if (u < u_drag) {  // one role for 32 planetesimals
        const int role = u / w_role;
        const int d = (u - role * w_role) * 32 + lane;
        if (d < ndrag) {
          drag_role(fc.gas, role, fc.mass[0], yt + 6 * V.dlist[d], V.dv + d, V.cap);
        }
      } else {  // migration: a lane per massive body
        const int m = (u - u_drag) * 32 + lane;
        if (m < nmig) {
          const int s = V.mlist[m], i = body_of(P, V, s), kind = V.kind[s];
          mig_compute(fc, i, kind, yt + 6 * s, S.factor, flags, V.gbuf + 3 * s, V.mig + s);
        }
      }
    }
    part_sync(1, nwork * 32);
    for (int x = w * 32 + lane; x < 3 * nitem; x += nwork * 32) {
      const int c = x / nitem, it = x - c * nitem, e = V.ends[it];
      double* p = V.p + (size_t)c * V.icap + it;
      const bool body = (e & 0xFFFF) == V.cap;
      *p = second_pass(body, yt[6 * (e >> 16) + c], V.p[3 * V.icap + it], *p,
                       body ? 0.0 : V.x[c * kMaxSources + (e >> 16)], V.gm[it]);
    }
    if (drag) {  // the drag's regime part from the roles, a lane per planetesimal
      for (int d = w * 32 + lane; d < ndrag; d += nwork * 32) {
        const int sd = V.dlist[d], i = body_of(P, V, sd);
        double out[3];
        drag_finish(fc.gas, S.factor, S.m0pt, yt + 6 * sd, fc.radius[i], fc.density[i], fc.cd[i], fc.gamma_stokes[i],
                    fc.gamma_epstein[i], V.dv + d, V.cap, out);
        for (int k = 0; k < 3; ++k) V.gbuf[3 * sd + k] = out[k];
        if (last && (sd >= P.ns || home)) {  // the buffers hold the last evaluation's drag
          double* gb = global_gas_buf(fc, i, 1);
          for (int k = 0; k < 3; ++k) gb[k] = out[k];
        }
      }
    }
    __syncthreads();
    if (last) last_evaluation(P, V, const_cast<int*>(&S.event), w * 32 + lane, nwork * 32);
  }
}

// A state lane: element `e` (6 slot + component) of sink slot s.
struct Lane {
  int s, k, i, e;  // k: component of position or velocity
  bool vel, live, write;
  int items, gas;   // the sink's items and its gas buffer's kind
  const double* q;  // its items' terms of component k
};

// Phase B: dy/dt of this element at the stage input yt.
__device__ __forceinline__ double derivative(const View& V, const Lane& L, const double* yt) {
  if (L.i == 0) return 0.0;  // Acceleration.cpp:253-254, :266
  if (!L.vel) return yt[L.e + 3];
  const double* q = L.q;
  double acc = 0.0;
#pragma unroll 4
  for (int n = 1; n < L.items; ++n) acc += q[n];
  double a = q[0];  // Kepler term first (Acceleration.cpp:281-283)
  a += acc;
  if (L.gas == 1 || (L.gas >= 2 && V.mig[L.s] != SOL_MIGRATION_NO)) a += V.gbuf[3 * L.s + L.k];
  return a;
}

// The RKF78 tableau (RungeKuttaFehlberg78.cpp:41-56): coefficient of f_q in stage j
__device__ constexpr double rk_a(int j, int q) {
  constexpr double A[13][12] = {
      {0},
      {2.0 / 27.0},
      {1.0 / 36.0, 1.0 / 12.0},
      {1.0 / 24.0, 0, 1.0 / 8.0},
      {5.0 / 12.0, 0, -25.0 / 16.0, 25.0 / 16.0},
      {1.0 / 20.0, 0, 0, 1.0 / 4.0, 1.0 / 5.0},
      {-25.0 / 108.0, 0, 0, 125.0 / 108.0, -65.0 / 27.0, 125.0 / 54.0},
      {31.0 / 300.0, 0, 0, 0, 61.0 / 225.0, -2.0 / 9.0, 13.0 / 900.0},
      {2.0, 0, 0, -53.0 / 6.0, 704.0 / 45.0, -107.0 / 9.0, 67.0 / 90.0, 3.0},
      {-91.0 / 108.0, 0, 0, 23.0 / 108.0, -976.0 / 135.0, 311.0 / 54.0, -19.0 / 60.0, 17.0 / 6.0, -1.0 / 12.0},
      {2383.0 / 4100.0, 0, 0, -341.0 / 164.0, 4496.0 / 1025.0, -301.0 / 82.0, 2133.0 / 4100.0, 45.0 / 82.0,
       45.0 / 164.0, 18.0 / 41.0},
      {3.0 / 205.0, 0, 0, 0, 0, -6.0 / 41.0, -3.0 / 205.0, -3.0 / 41.0, 3.0 / 41.0, 6.0 / 41.0},
      {-1777.0 / 4100.0, 0, 0, -341.0 / 164.0, 4496.0 / 1025.0, -289.0 / 82.0, 2193.0 / 4100.0, 51.0 / 82.0,
       33.0 / 164.0, 12.0 / 41.0, 0, 1.0}};
  return A[j][q];
}

// Running sums of one element over an attempt, every one in ascending stage
// order as the reference adds it (:169-242): the stage sums, the 7th-order
// sum and the error combination.
template <int N>
struct Int {
  static constexpr int value = N;
};
struct Sums {
  double s[13];
  double t, hold, e;
};
template <int Q, int J>
__device__ __forceinline__ void add_stage(Sums& S, double f) {
  constexpr double a = rk_a(J, Q);
  if constexpr (Q == 0) S.s[J] = a * f;
  else if constexpr (a != 0.0) S.s[J] = S.s[J] + a * f;
}
template <int Q, int J>
__device__ __forceinline__ void add_stages(Sums& S, double f) {
  if constexpr (J <= 12) {
    add_stage<Q, J>(S, f);
    add_stages<Q, J + 1>(S, f);
  }
}
// f_Q into everything but stage Q + 1's sum
template <int Q>
__device__ __forceinline__ void add_later(Sums& S, double f) {
  constexpr double D0 = 41.0 / 840.0, D5 = 34.0 / 105.0, D6 = 9.0 / 35.0, D8 = 9.0 / 280.0, D10 = 41.0 / 840.0;
  add_stages<Q, Q + 2>(S, f);
  if constexpr (Q == 0) {
    S.t = D0 * f;
    S.e = f;
  }
  if constexpr (Q == 5) S.t = S.t + D5 * f;
  if constexpr (Q == 6 || Q == 8) S.hold = f;
  if constexpr (Q == 7) S.t = S.t + D6 * (S.hold + f);
  if constexpr (Q == 9) S.t = S.t + D8 * (S.hold + f);
  if constexpr (Q == 10) {
    S.t = S.t + D10 * f;
    S.e = S.e + f;
  }
  if constexpr (Q == 11) S.e = S.e - f;
}

// The next step size after an accepted step (RungeKuttaFehlberg78.cpp:113-118); thread 0.
__device__ __forceinline__ void grow(Ctl& S) {
  const double em = S.error_max, h = S.h_did;
  S.h_next = em > 1.89e-4 ? (0.9 * h * sol_inv_root<5>(em)) : (5.0 * h);
  S.h = S.h_next;
}

// Simulator::DecisionMaking up to where the host has work
// (Simulator.cpp:181-250), after an accepted step of S.h_did; thread 0.
__device__ __forceinline__ void sim_decision(Ctl& S, int any) {
  sol_sim_line& L = S.L;
  L.steps += 1;
  L.elapsed += S.h_did;
  L.last_save += S.h_did;
  S.flush = 0;
  if (any) {
    S.reason = SOL_STOP_EVENT;
    S.stop = 1;
  } else {
    const double clock = L.relative_end ? L.elapsed : S.t;
    if (fabs(clock) >= fabs(L.length)) {
      S.reason = SOL_STOP_LENGTH;
      S.stop = 1;
    } else {
      if (fabs(clock + S.h_next) > fabs(L.length)) S.h_next = L.length - clock;
      if (fabs(L.last_save) >= fabs(L.output)) {
        S.reason = SOL_STOP_OUTPUT;
        S.stop = 1;
      } else {
        if (fabs(L.last_save + S.h_next) > fabs(L.output)) S.h_next = L.output - L.last_save;
        S.flush = (L.steps % 100) == 0;  // Tools::CheckAgainstSmallestNumber every CheckForSM steps
      }
    }
  }
  S.h = S.h_next;
}

template <int MAXT>
__global__ void __launch_bounds__(MAXT) k_group_rkf78(GroupArgs P) {
  extern __shared__ __align__(16) double smem[];
  __shared__ Ctl S;
  const ForceCtx& fc = P.fc;
  const int ns = P.ns;
  const bool home = blockIdx.x == 0;
  View V;
  V.cap = ns + P.local;
  V.icap = P.icap;
  V.l0 = ns + blockIdx.x * P.local;
  const int nsink = ns + max(min(V.l0 + P.local, P.n) - V.l0, 0);
  V.nsink = nsink;
  V.stride = 6 * (V.cap + 1);
  V.yt = smem + P.o_yt;
  V.p = smem + P.o_p;
  V.x = smem + P.o_x;
  V.gm = smem + P.o_gm;
  V.gbuf = smem + P.o_gbuf;
  V.dv = smem + P.o_dv;
  V.ends = reinterpret_cast<int*>(smem + P.o_int);
  V.base = V.ends + V.icap;
  V.mig = V.base + V.cap + 1;
  V.kind = V.mig + V.cap;
  V.dlist = V.kind + V.cap;
  V.mlist = V.dlist + V.cap;
  for (int s = threadIdx.x; s < nsink; s += blockDim.x) {
    const int i = body_of(P, V, s);
    V.mig[s] = fc.mig_type[i];
    const int kind = gas_kind(fc, i);
    V.kind[s] = kind;
    // (the drag's is formed anew by the first evaluation)
    for (int k = 0; k < 3; ++k) V.gbuf[3 * s + k] = kind >= 2 ? global_gas_buf(fc, i, kind)[k] : 0.0;
    const int nsrc = (fc.type[i] <= SOL_PROTO_PLANET) ? ns : fc.cls.nm;
    // items of sinks i >= 1: the origin, sources 1 <= j < nsrc, j != i
    V.base[s] = i == 0 ? 0 : nsrc - ((i < nsrc) ? 1 : 0);
  }
  for (int e = threadIdx.x; e < 2 * V.stride; e += blockDim.x) V.yt[e] = 0.0;
  __syncthreads();
  if (threadIdx.x == 0) {
    int at = 0, nd = 0, nmg = 0;
    for (int s = 0; s < nsink; ++s) {
      const int cnt = V.base[s];
      V.base[s] = at;
      at += cnt;
      if (V.kind[s] == 1) V.dlist[nd++] = s;
      else if (V.kind[s] >= 2) V.mlist[nmg++] = s;
    }
    V.base[nsink] = at;
    S.nitem = at;
    S.ndrag = nd;
    S.nmig = nmg;
    S.m0pt = fc.gas.present ? pow(fc.mass[0], fc.gas.pt) : 0.0;
    const sol_ctrl c = *P.ctrl;
    S.t = c.t;
    S.h = c.h_next;  // Driver: bodyData->h = timeLine->hNext (:74-75)
    S.h_next = c.h_next;
    S.h_did = c.h_did;
    S.error_max = c.error_max;
    S.eps = c.eps;
    S.n_acc = c.n_accepted;
    S.n_rej = c.n_rejected;
    S.status = c.dev_status;
    S.accepted = 0;
    S.leave = 0;
    S.abort = 0;
    S.event = 0;
    S.stop = 0;
    S.reason = SOL_STOP_STEPS;
    S.flush = 0;
    if (P.sim) S.L = *P.line;
  }
  __syncthreads();
  for (int s = threadIdx.x; s < nsink; s += blockDim.x) {
    const int i = body_of(P, V, s);
    if (i == 0) continue;
    const int nsrc = (fc.type[i] <= SOL_PROTO_PLANET) ? ns : fc.cls.nm;
    int it = V.base[s];
    V.ends[it] = V.cap | (s << 16);  // (zero slot, s): the body's own position
    V.gm[it] = -(SOL_GAUSS2 * (fc.mass[0] + fc.mass[i]));
    ++it;
    for (int j = 1; j < nsrc; ++j) {
      if (j == i) continue;
      V.ends[it] = s | (j << 16);
      V.gm[it] = SOL_GAUSS2 * fc.mass[j];
      ++it;
    }
  }
  // a state lane's element: velocity warps first, then position warps, then workers
  const int warp = threadIdx.x >> 5;
  const bool worker = warp >= 2 * P.vw;
  Lane L;
  L.vel = warp < P.vw;
  const int x = threadIdx.x - (L.vel ? 0 : 32 * P.vw);
  L.live = !worker && x < 3 * nsink;
  L.s = L.live ? x / 3 : 0;
  L.k = L.live ? x - 3 * L.s : 0;
  L.i = body_of(P, V, L.s);
  L.e = 6 * L.s + L.k + (L.vel ? 3 : 0);
  L.write = L.live && (L.s >= ns || home);
  L.items = V.base[L.s + 1] - V.base[L.s];
  L.gas = V.kind[L.s];
  L.q = V.p + (size_t)L.k * V.icap + V.base[L.s];
  const size_t ge = 6 * (size_t)L.i + (L.e - 6 * L.s);  // the element in the context's arrays
  __syncthreads();
  if (worker) {
    const View Vw = V;  // (a copy: what is passed by reference lives in local memory)
    work(P, Vw, S);
    return;
  }
  // ---- the state warps ----
  const int nstate = 64 * P.vw;
  double y0 = L.live ? P.y0[ge] : 0.0;
  double f0 = 0.0, ys = 1.0, yn = 0.0, err = 0.0;
  bool ran = false, pending = false;
  unsigned k = 0;  // group barriers passed
  int cur = 0;     // stage-input buffer
  // hand the stage input x to the workers; the caller's own work until
  // collect() overlaps phase A
  auto submit = [&](double x, double factor, uint32_t flags, int last) {
    cur ^= 1;
    if (L.live) V.yt[cur * V.stride + L.e] = x;
    if (threadIdx.x == 0) {
      S.cur = cur;
      S.factor = factor;
      S.flags = flags;
      S.last = last;
    }
    __syncthreads();
  };
  auto collect = [&]() -> double {
    __syncthreads();
    return L.live ? derivative(V, L, V.yt + cur * V.stride) : 0.0;
  };
  for (int step = 0; step < P.n_steps && S.status == 0 && !S.stop; ++step) {
    ran = true;
    const double t0 = S.t;
    // RKF78 evaluates every stage at the step's start time; RK4 at t + c h
    // (RungeKutta4.cpp:101-116)
    auto factor_at = [&](double t) { return fc.gas.present ? sol_reduction_factor(fc.gas, t) : 1.0; };
    const double fac = factor_at(t0);
    // first evaluation with every term on (:77-82)
    submit(y0, fac, SOL_EVAL_ALL, 0);
    if (pending && threadIdx.x == 0) grow(S);  // the accepted step's growth, which this evaluation does not need
    pending = false;
    f0 = collect();
    const double h1 = S.h;
    double h = h1;
    if (P.rk4) {  // RungeKutta4::Driver and Step (RungeKutta4.cpp:20-129)
      const double b1 = 1.0 / 6.0, b2 = 1.0 / 3.0, b3 = 1.0 / 3.0, b4 = 1.0 / 6.0;
      double f = f0, t = b1 * f0;
      for (int r = 1; r <= 3; ++r) {
        const double c = r < 3 ? 1.0 / 2.0 : 1.0;  // a21, a32, a43 and the stage times
        submit(y0 + h * (c * f), threadIdx.x == 0 ? factor_at(t0 + c * h) : 1.0, SOL_EVAL_GAS_DRAG, r == 3);
        f = collect();
        t = t + (r == 1 ? b2 : r == 2 ? b3 : b4) * f;
      }
      yn = y0 + h * t;
      __syncthreads();  // the workers' last_evaluation
      int any = S.event;
      if (warp == 0 && P.sim && gridDim.x > 1) {  // the event flags of every CTA
        const Exchanged x = exchange(P, k++, 0, any);
        any = x.any;
        if (!x.ok) S.abort = 1;
      }
      if (threadIdx.x == 0) {
        S.h_did = h;
        S.t += S.h_did;
        S.h_next = h;  // RK4 keeps its step size (and a clamp of it)
        S.h = h;
        S.accepted = 1;
        S.n_acc++;
        if (P.sim) sim_decision(S, any);
        S.event = 0;
      }
      part_sync(2, nstate);
    } else {
      ys = fabs(y0) + fabs(h * f0) + 1.0e-30;  // yscale (:87-89)
      for (;;) {
        Sums A;
        double f = f0;
        // stage R from f_(R-1): unrolled, each R its own coefficients
        auto stage = [&](auto R) {
          constexpr int r = decltype(R)::value;
          add_stage<r - 1, r>(A, f);
          // migration only at the first evaluation of a driver call (:94-95)
          submit(y0 + h * A.s[r], fac, SOL_EVAL_GAS_DRAG, r == 12);
          add_later<r - 1>(A, f);
          f = collect();
        };
        stage(Int<1>());
        stage(Int<2>());
        stage(Int<3>());
        stage(Int<4>());
        stage(Int<5>());
        stage(Int<6>());
        stage(Int<7>());
        stage(Int<8>());
        stage(Int<9>());
        stage(Int<10>());
        stage(Int<11>());
        stage(Int<12>());
        // the error estimate and the scaled norm (:236-242, :252-262)
        err = h * fabs(A.e - f) * 41.0 / 840.0;
        long long m = 0;  // bits: these maxima are never negative
        if (L.live) {
          const double q = fabs(err / ys);
          if (q > 0.0) m = __double_as_longlong(q);  // a NaN entry never replaces the maximum
        }
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) {
          const long long o = __shfl_xor_sync(0xFFFFFFFFu, m, w);
          m = o > m ? o : m;
        }
        if ((threadIdx.x & 31) == 0) S.red[warp] = m;
        __syncthreads();  // the workers' last_evaluation, too
        if (warp == 0) {
          for (int w = 1; w < 2 * P.vw; ++w) m = S.red[w] > m ? S.red[w] : m;
          int any = S.event;
          if (gridDim.x > 1) {
            const Exchanged x = exchange(P, k++, m, any);
            m = x.worst;
            any = x.any;
            if (!x.ok) S.abort = 1;
          }
          if (threadIdx.x == 0) {
            // every CTA takes the same decision (:98-133)
            const double em = __longlong_as_double(m) / S.eps;
            S.error_max = em;
            if (em < 1.0) {
              S.h_did = h;
              S.t += S.h_did;
              S.accepted = 1;
              S.n_acc++;
              if (P.sim) {  // whether to go on depends on the next step size
                grow(S);
                sim_decision(S, any);
              }
            } else {
              S.accepted = 0;
              S.n_rej++;
              const double hTemp = 0.9 * h * sol_inv_root<4>(em);
              const double hn = fabs(hTemp) > fabs(0.1 * h) ? hTemp : 0.1 * h;
              S.h = hn;
              if (S.t + hn == S.t) S.status |= SOL_DEV_UNDERFLOW;
            }
            S.event = 0;
          }
        }
        // the 7th-order result (:236-238), while thread 0 waits for the others
        yn = y0 + h * A.t;
        part_sync(2, nstate);
        if (S.accepted || S.status || S.abort) break;
        h = S.h;
      }
    }
    if (S.abort) break;
    pending = !P.rk4 && !P.sim && S.accepted;
    if (S.accepted) {  // y0 <- the new state, flushed below the smallest number when due
      // the step-start state kept when the step stops with an event
      if (P.sim && P.yprev && S.stop && S.reason == SOL_STOP_EVENT && L.write) P.yprev[ge] = y0;
      y0 = S.flush && fabs(yn) < 1.0e-50 ? 0.0 : yn;
    }
  }
  // A block may start late: what it reads at its start (the state, the control
  // record, the migration's state and buffers) is written from here on, when every
  // block has exchanged a word with the others.  (RK4 calls outside the step loop
  // have had no exchange yet.)
  if (ran && P.rk4 && !P.sim && gridDim.x > 1 && !S.abort) {
    if (warp == 0) {
      __threadfence();
      if (!exchange(P, k, 0, 0).ok) S.abort = 1;
    }
  }
  if (threadIdx.x == 0) {
    if (pending) grow(S);
    S.leave = 1;
  }
  __syncthreads();  // the workers leave
  if (S.abort) return;
  // what the driver calls leave in the context: the state, and the last
  // call's f0, yscale, result and error
  if (ran && L.write) {
    P.y0[ge] = y0;
    P.accel[ge] = f0;
    P.ynew[ge] = yn;
    if (!P.rk4) {
      P.yscale[ge] = ys;
      P.err[ge] = err;
    }
  }
  if (ran && home)  // migrating bodies are sources
    for (int q = threadIdx.x; q < S.nmig; q += nstate) {
      const int s = V.mlist[q], i = body_of(P, V, s);
      double* gb = global_gas_buf(fc, i, V.kind[s]);
      for (int c = 0; c < 3; ++c) gb[c] = V.gbuf[3 * s + c];
      fc.mig_type[i] = V.mig[s];
    }
  if (home && threadIdx.x == 0) {
    sol_ctrl* c = P.ctrl;
    c->t = S.t;
    c->h = S.h;
    c->h_next = S.h_next;
    c->h_did = S.h_did;
    c->error_max = S.error_max;
    c->accepted = S.accepted;
    c->n_accepted = S.n_acc;
    c->n_rejected = S.n_rej;
    atomicOr(&c->dev_status, S.status);
    if (P.sim) {
      sol_sim_line T = S.L;
      T.time = S.t;
      T.h_next = S.h_next;
      T.h_did = S.h_did;
      *P.line = T;
      *P.reason = S.stop ? S.reason : SOL_STOP_STEPS;
    }
  }
}

// Shared-memory layout for a capacity of cap sinks and P.icap items (offsets in doubles).
size_t layout(GroupArgs& P, int cap) {
  size_t o = 0;
  auto take = [&](int& field, size_t doubles) {
    field = (int)o;
    o += (doubles + 1) & ~(size_t)1;  // 16-byte alignment
  };
  take(P.o_yt, (size_t)2 * 6 * (cap + 1));
  take(P.o_p, (size_t)5 * P.icap);
  take(P.o_x, (size_t)3 * kMaxSources);
  take(P.o_gm, (size_t)P.icap);
  take(P.o_gbuf, (size_t)3 * cap);
  take(P.o_dv, (size_t)kRoleValues * cap);
  // ints: item ends (icap), first items (cap + 1), migType, gas kind, drag and
  // migration lists (cap each)
  take(P.o_int, ((size_t)P.icap + (size_t)5 * cap + 2) / 2);
  return o * sizeof(double);
}

}  // namespace

// Whether the system can run its RKF78 / RK4 driver calls on the group path.
int sol_group_eligible(const sol_ctx* c) {
  if (c->barycentric) return 0;
  const int ns = c->cls.nm + c->cls.n_spl;
  return ns >= 1 && ns <= kMaxSources && c->n - ns <= 152 * kMaxLocal;
}

// n_steps RKF78 (or, with rk4, RungeKutta4) driver calls in one cooperative
// launch of the group kernel.  Returns SOL_ERR_STATE (nothing launched) when
// the system does not fit.
int sol_group_rkf78(sol_ctx* c, int n_steps, const GroupSim* sim, int rk4) {
  if (!sol_group_eligible(c)) return SOL_ERR_STATE;
  if (!c->d_persist) {
    const size_t doubles = 2 * 7 * 32 + 4096 + 8;
    if (cudaMalloc((void**)&c->d_persist, sizeof(double) * doubles) != cudaSuccess) {
      sol_set_error("cudaMalloc of the persistent-driver scratch failed");
      return SOL_ERR_NOMEM;
    }
    SOL_CUDA(cudaMemset(c->d_persist, 0, sizeof(double) * doubles));
  }
  int n_sm = 0;
  SOL_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, c->device));
  GroupArgs P;
  memset(&P, 0, sizeof(P));
  const int ns = c->cls.nm + c->cls.n_spl;
  // bodies per CTA: the smallest power of two whose grid is co-resident, one
  // CTA per SM (at least half an SM's shared memory each: CTAs packed onto one
  // SM would share its FP64 pipe).
  // Fewer bodies a CTA shorten no chain once a phase's lanes fit one or two
  // warps, and more CTAs make the exchange longer: measured at 253 test
  // particles (cycles a stage, and between two attempts) 3,700 and 11,340 with
  // 2 bodies a CTA, 3,620 and 10,210 with 4, 4,230 and 9,640 with 8, 5,320 and
  // 8,860 with 16.
  const void* kernel = nullptr;
  int local = 0, grid = 0, threads = 0;
  size_t smem = 0;
  const int others = c->n - ns;
  for (int cand = kMinLocal; cand <= kMaxLocal; cand *= 2) {
    const int g = others > 0 ? (others + cand - 1) / cand : 1;
    if (g > n_sm || g > kMaxCtas) continue;
    // a source: the origin and at most ns - 2 others; another body: the origin and nm - 1
    P.icap = ns * ns + cand * c->cls.nm;
    const int cap = ns + cand;
    P.vw = (3 * cap + 31) / 32;
    const int gas = c->has_gas ? kRoles * ((cap + 31) / 32) + (ns + 31) / 32 : 0;
    const int units = gas ? gas + (P.icap + 31) / 32 : (4 * P.icap + 31) / 32;  // four lanes an item, or one
    const int workers = std::min(std::max(units, kWorkersMin), kMaxThreads / 32 - 2 * P.vw);
    const size_t sm = std::max(layout(P, cap), (size_t)kSpreadSmem);
    if (sm > 200 * 1024 || workers < 1) break;
    const int th = 32 * (2 * P.vw + workers);
    kernel = th <= 512 ? (const void*)k_group_rkf78<512> : (const void*)k_group_rkf78<kMaxThreads>;
    SOL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    int per_sm = 0;
    SOL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, th, sm));
    if (g <= per_sm * n_sm) {
      local = cand;
      grid = g;
      smem = sm;
      threads = th;
      break;
    }
  }
  if (!local) return SOL_ERR_STATE;
  P.fc = c->fc;
  P.y0 = c->d_y0;
  P.accel = c->d_accel;
  P.yscale = c->d_yscale;
  P.ynew = c->d_y;
  P.err = c->d_err;
  P.words = reinterpret_cast<unsigned long long*>(c->d_persist + 2 * 7 * 32);
  P.abort_flag = reinterpret_cast<int*>(c->d_persist + 2 * 7 * 32 + 4096);
  P.spin = c->test_spin ? c->test_spin : SOL_SPIN_LIMIT;
  P.skip_cta = c->test_skip_cta;
  P.ctrl = c->d_ctrl;
  P.n = c->n;
  P.ns = ns;
  P.local = local;
  P.n_steps = n_steps;
  P.rk4 = rk4 ? 1 : 0;
  if (sim) {
    P.sim = 1;
    P.e3 = sim->e3;
    P.h3 = sim->h3;
    P.cf = sim->cf;
    P.line = sim->line;
    P.reason = sim->reason;
    P.yprev = sim->yprev;
  }
  SOL_CUDA(cudaMemsetAsync(P.words, 0, (4 * kMaxCtas + 1) * sizeof(*P.words), c->stream));
  SOL_CUDA(cudaMemsetAsync(P.abort_flag, 0, sizeof(int), c->stream));
  void* args[] = {&P};
  SOL_CUDA(cudaLaunchCooperativeKernel(kernel, grid, threads, args, smem, c->stream));
  SOL_LAUNCHED();
  return SOL_OK;
}
