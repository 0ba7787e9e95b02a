// Force evaluation: the GB300 replacement of Acceleration::Compute
// (Solaris/Acceleration.cpp:60-246) and its gravity, gas-drag and migration
// terms.
//
// One evaluation:
//   k_prepass     one thread per body: rm3[j] = 1/|r_j|^3 exactly as
//                 GravityAC computes it (:256-264), and the structure-of-arrays
//                 source table {x, y, z, G m, x rm3, y rm3, z rm3} that the pair
//                 kernel streams; per-block partial sums of the indirect term.
//   k_ind_reduce  one block: the indirect-term totals (split forms; k_split_table
//                 does it where it runs).
//   the pairs     FP64: k_gravity_ac_ref (tiles of 64 sources, the sums in
//                 source order by a warp of their own) or k_gravity_ac (a thread
//                 a sink, few sources); SPLIT_FF: k_split_table, then k_pairs_sym
//                 (unordered pairs of massive bodies) and / or k_pairs_ff, or
//                 k_pairs_few; SPLIT: k_pairs or k_pairs_few.  The 2-D kernels'
//                 source tiles are staged in shared memory by bulk copies
//                 (cp.async.bulk, the TMA engine) completing on an mbarrier,
//                 double buffered; k_combine adds their partials.  The epilogue
//                 adds gas drag and type-I/II migration for the sink.
#include <cstdio>
#include <cstring>
#include <atomic>
#include <mutex>

#include "sol_internal.cuh"
#include "sol_crmath.cuh"
#include "sol_pair.cuh"

int sol_force_uses_chunk_partials(const sol_ctx* c, int precision);

namespace {

constexpr int kSinkBlock = 128;  // sinks per CTA
constexpr int kTile = 256;       // sources per shared-memory tile
constexpr int kPrepassBlock = 256;

enum SrcArray { SX = 0, SY, SZ, SGM, SPX, SPY, SPZ, SGF, SRC_ARRAYS = 8 };  // SGF: G m as (hi, lo) floats
// Float table of the SPLIT_FF 2-D kernel, after the SRC_ARRAYS doubles: each
// coordinate as its grid triple a + b + c (f2_grid_disp in sol_pair.cuh) and
// G m as (hi, lo), one float array each (two sources load as one float2).
enum FTab { FAX = 0, FBX, FCX, FAY, FBY, FCY, FAZ, FBZ, FCZ, FGH, FGL, FTAB_USED = 11, FTAB_ARRAYS = 12 };
constexpr int kSrcDoubles = SRC_ARRAYS + FTAB_ARRAYS / 2;  // doubles per padded body in the source table
// ind_sum slots: [0..5] the indirect sums, [6] the grid G1 of the float table
constexpr int kIndGrid = 6;

constexpr int kChunkTiles = 16;             // sources per work unit of the 2-D pair kernel
constexpr int kChunk = kChunkTiles * kTile;  // 4,096
enum PartSlot { PAX = 0, PAY, PAZ, PR2, PIDX, PART_SLOTS = 5 };

__device__ __forceinline__ double eval_time(const TimeSpec& ts) {
  return ts.base ? (*ts.base + ts.c * (*ts.h)) : ts.t_host;
}

// ---- prepass ----------------------------------------------------------------
__device__ __forceinline__ float* ftab(const ForceCtx& fc) { return reinterpret_cast<float*>(fc.src + (size_t)SRC_ARRAYS * fc.npad); }

// Body j's rm3 and its entries of the source table (zeros for padding bodies)
struct SourceRow {
  double gm, px, py, pz;
};
__device__ __forceinline__ SourceRow source_row(const ForceCtx& fc, int j, double x, double yy, double z) {
  SourceRow r = {0.0, 0.0, 0.0, 0.0};
  if (j < fc.cls.n) {
    double rm3 = 0.0;
    if (j >= 1) {
      if (!fc.barycentric) {
        // Acceleration.cpp:259-261
        double r2 = x * x + yy * yy + z * z;
        double d;
        sol_ref_rinv3(r2, d, rm3);
        fc.rm3[j] = rm3;
      }
      r.gm = SOL_GAUSS2 * fc.mass[j];
    }
    r.px = x * rm3;
    r.py = yy * rm3;
    r.pz = z * rm3;
    if (fc.barycentric) r.gm = fc.mass[j];  // GravityBC uses m_j and scales by G at the end
  }
  double* s = fc.src;
  const int np = fc.npad;
  s[SX * np + j] = x;
  s[SY * np + j] = yy;
  s[SZ * np + j] = z;
  s[SGM * np + j] = r.gm;
  s[SPX * np + j] = r.px;
  s[SPY * np + j] = r.py;
  s[SPZ * np + j] = r.pz;
  return r;
}

// prec: SOL_PRECISION_*.  The split forms also sum the indirect term; SPLIT_FF
// (2-D kernel, ff = 1) also takes the largest |coordinate| and writes G m as
// float (hi, lo) arrays of the float table.  clear: a status word to zero for
// the kernels that follow (or null).
__global__ void k_prepass(ForceCtx fc, const double* __restrict__ y, int split, int ff, int* clear) {
  const int n = fc.cls.n;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (clear && j == 0) *clear = 0;
  double q[6] = {0, 0, 0, 0, 0, 0};  // indirect contributions: massive range, super-planetesimal range
  unsigned mbits = 0;                 // |coordinate| maximum as FP32 bits, rounded up
  if (j < fc.npad) {
    double x = 0, yy = 0, z = 0;
    if (j < n) {
      x = y[6 * j + 0];
      yy = y[6 * j + 1];
      z = y[6 * j + 2];
    }
    const SourceRow r = source_row(fc, j, x, yy, z);
    if (split && j < n && j >= 1) {
      int slot = (j < fc.cls.nm) ? 0 : ((j < fc.cls.nm + fc.cls.n_spl) ? 3 : -1);
      if (slot >= 0) {
        q[slot + 0] = r.gm * r.px;
        q[slot + 1] = r.gm * r.py;
        q[slot + 2] = r.gm * r.pz;
      }
    }
    float gh = __double2float_rn(r.gm);
    float gl = __double2float_rn(r.gm - (double)gh);
    reinterpret_cast<float2*>(fc.src + (size_t)SGF * fc.npad)[j] = make_float2(gh, gl);
    if (ff) {
      float* T = ftab(fc);
      T[(size_t)FGH * fc.npad + j] = gh;
      T[(size_t)FGL * fc.npad + j] = gl;
      const double m = fmax(fabs(x), fmax(fabs(yy), fabs(z)));
      mbits = __float_as_uint(__double2float_ru(m));
    }
  }
  if (!split) return;
  // the block's sums of the indirect contributions, in a fixed order, and its largest |coordinate|
  __shared__ double red[kPrepassBlock / 32][8];
  __shared__ unsigned far[kPrepassBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double v[8] = {q[0], q[1], q[2], q[3], q[4], q[5], 0.0, 0.0};
  const double mine = warp_sum8(v, lane);
  if ((lane & 3) == 0) red[warp][4 * (lane >> 4 & 1) + 2 * (lane >> 3 & 1) + (lane >> 2 & 1)] = mine;
  const unsigned wmax = __reduce_max_sync(0xFFFFFFFFu, mbits);
  if (lane == 0) far[warp] = wmax;
  __syncthreads();
  if (threadIdx.x < 6) {
    double t = red[0][threadIdx.x];
    for (int w = 1; w < kPrepassBlock / 32; ++w) t += red[w][threadIdx.x];
    fc.ind_part[6 * blockIdx.x + threadIdx.x] = t;
  }
  if (ff && threadIdx.x == 6) {
    unsigned m = far[0];
    for (int w = 1; w < kPrepassBlock / 32; ++w) m = max(m, far[w]);
    fc.ind_part[6 * fc.n_ind_blocks + blockIdx.x] = __hiloint2double(0, (int)m);
  }
}

// The indirect-term totals from the blocks' sums, a warp each, by a block of 256
// threads: [0..2] over [1, nm); [3..5] over [1, nm + n_spl).
__device__ __forceinline__ void ind_totals(const ForceCtx& fc) {
  __shared__ double tot[6];
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (k < 6) {
    double t = 0.0;
    for (int b = lane; b < fc.n_ind_blocks; b += 32) t += fc.ind_part[6 * b + k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
    if (lane == 0) tot[k] = t;
  }
  __syncthreads();
  if (threadIdx.x < 6) fc.ind_sum[threadIdx.x] = threadIdx.x < 3 ? tot[threadIdx.x] : tot[threadIdx.x - 3] + tot[threadIdx.x];
}
__global__ void __launch_bounds__(256) k_ind_reduce(ForceCtx fc) { ind_totals(fc); }

// A stage's input y0 + h (a_0 f_0 + ...), summed left to right
// (RungeKuttaFehlberg78.cpp:170-232, RungeKutta4.cpp:413-433), and what k_prepass
// makes of it for the FP64 forms: a thread per element, then one per body.  Both
// are a few dependent instructions, so a launch of its own was most of either
// (a stage with its evaluation, in two launches and in one: 200 bodies 27.3 and
// 23.8 us, 1,033 71.8 and 68.4, 4,000 509 and 505).
constexpr int kStageBodies = 32;
template <int K>
__global__ void __launch_bounds__(6 * kStageBodies) k_stage_prepass(ForceCtx fc, const double* __restrict__ y0,
                                                                    double* __restrict__ out, StageArgs s,
                                                                    const sol_ctrl* ctrl) {
  __shared__ double sv[6 * kStageBodies];
  const double h = ctrl->h;
  const int i = blockIdx.x * (6 * kStageBodies) + threadIdx.x;
  double v = 0.0;
  if (i < 6 * fc.cls.n) {
    double f[K];
#pragma unroll
    for (int k = 0; k < K; ++k) f[k] = s.f[k][i];
    double acc = s.a[0] * f[0];
#pragma unroll
    for (int k = 1; k < K; ++k) acc = acc + s.a[k] * f[k];
    v = y0[i] + h * acc;
    out[i] = v;
  }
  sv[threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.x < kStageBodies) {
    const int b = 6 * threadIdx.x;
    source_row(fc, blockIdx.x * kStageBodies + threadIdx.x, sv[b], sv[b + 1], sv[b + 2]);
  }
}

// Grid triples of every coordinate (f2_grid_disp): a = G1 rint(x / G1),
// b = G2 rint((x - a) / G2), c = float(x - a - b); a and b are exact floats
// (at most 2^23 of their grid), x - a and x - a - b exact doubles.  Padding
// bodies (no mass) are set apart from the others and from each other, so that
// k_pairs_sym, which does not mask them, meets no close pair among them.
// The grid G1 = 2^(E - 23), every |coordinate| < 2^E, each block takes from the
// prepass blocks' maxima; block 0 also does k_ind_reduce's sums (a launch of its
// own cost 5 us).
__global__ void __launch_bounds__(kPrepassBlock) k_split_table(ForceCtx fc, const double* __restrict__ y,
                                                               float* __restrict__ bound) {
  __shared__ unsigned far[kPrepassBlock / 32];
  const int j = blockIdx.x * kPrepassBlock + threadIdx.x;  // < npad, a whole number of blocks
  double x[3] = {0.0, 0.0, 0.0};
  if (j < fc.cls.n)
    for (int k = 0; k < 3; ++k) x[k] = y[6 * j + k];
  unsigned mb = 0;
  for (int b = threadIdx.x; b < fc.n_ind_blocks; b += kPrepassBlock)
    mb = max(mb, (unsigned)__double2loint(fc.ind_part[6 * fc.n_ind_blocks + b]));
  mb = __reduce_max_sync(0xFFFFFFFFu, mb);
  if ((threadIdx.x & 31) == 0) far[threadIdx.x >> 5] = mb;
  __syncthreads();
  for (int w = 0; w < kPrepassBlock / 32; ++w) mb = max(mb, far[w]);
  const int E = max(mb ? (int)(mb >> 23) - 127 + 1 : 0, -90) - 23;
  const double G1 = __hiloint2double((1023 + E) << 20, 0);
  // adding and subtracting 1.5 2^52 G rounds to the grid G
  const double M1 = __hiloint2double(((1023 + E + 52) << 20) | 0x80000, 0);
  const double M2 = __hiloint2double(((1023 + E + 28) << 20) | 0x80000, 0);
  float* T = ftab(fc);
  const int np = fc.npad;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double a = (x[k] + M1) - M1;
    const double r = x[k] - a;
    const double b = (r + M2) - M2;
    T[(size_t)(FAX + 3 * k) * np + j] = (float)a;
    T[(size_t)(FBX + 3 * k) * np + j] = (float)b;
    T[(size_t)(FCX + 3 * k) * np + j] = __double2float_rn(r - b);
  }
  if (bound) bound[j] = 3.0e38f;  // for k_near_bound
  if (j >= fc.cls.n) T[(size_t)FAX * np + j] = (float)((4194304.0 + 1024.0 * (j - fc.cls.n)) * G1);
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) fc.ind_sum[kIndGrid] = G1;
    ind_totals(fc);
  }
}

// ---- tile pipeline -----------------------------------------------------------
template <int NARR>
struct TileSmem {
  double v[2][NARR][kTile];
  uint64_t bar[2];
};

template <int NARR>
__device__ __forceinline__ void issue_tile(TileSmem<NARR>& sm, const double* src, int npad, int tile, int stage) {
  sol_mbar_expect_tx(&sm.bar[stage], NARR * kTile * 8);
  for (int k = 0; k < NARR; ++k)
    sol_bulk_g2s(&sm.v[stage][k][0], src + (size_t)k * npad + (size_t)tile * kTile, kTile * 8, &sm.bar[stage]);
}

// Reference-form pair arithmetic (GravityAC, Acceleration.cpp:294-317): IEEE
// sqrt and division, no contraction, sources in ascending order.
__device__ __forceinline__ void pair_fp64(const TileSmem<7>& sm, int st, int jj, int j, int i, int ns, double xi,
                                          double yi, double zi, double& ax, double& ay, double& az, long long& rminb,
                                          int& nn) {
  if (j >= 1 && j < ns && j != i) {
    double xij = sm.v[st][SX][jj] - xi;
    double yij = sm.v[st][SY][jj] - yi;
    double zij = sm.v[st][SZ][jj] - zi;
    double rij2 = xij * xij + yij * yij + zij * zij;
    double rij, rijm3;
    sol_ref_rinv3(rij2, rij, rijm3);
    long long rb = __double_as_longlong(rij);
    if (rb < rminb) {
      rminb = rb;
      nn = j;
    }
    double gm = sm.v[st][SGM][jj];
    ax += gm * (xij * rijm3 - sm.v[st][SPX][jj]);
    ay += gm * (yij * rijm3 - sm.v[st][SPY][jj]);
    az += gm * (zij * rijm3 - sm.v[st][SPZ][jj]);
  }
}

// Split pair arithmetic: FP64 displacement and r^2; rsqrt seed in FP32 with
// the FP64 <-> FP32 conversions done by integer operations on the bit
// patterns (they stay off the FP64 pipe); one FP64 Newton correction of
// r^-3 carried to second order in the residual e = 1 - r^2 y0^2:
//   r^-3 = y0^3 (1 - e)^(-3/2) = y0^3 (1 + 3/2 e + 15/8 e^2 + O(e^3)),
// |e| < 2^-20, so the truncation is below 1e-18.  The seed's square and cube
// come from the integer pipe (sol_seed_square_cube), and so does t = 3/2 e +
// 15/8 e^2 (sol_split_t), leaving FP64 the residual e, G m y0^3 and
// G m y0^3 + (G m y0^3) t by one DFMA (split_gm_rinv3): with the
// displacement, r^2 and the three accumulations, 12 FP64 operations per pair,
// the floor of this recipe.
__device__ __forceinline__ double split_gm_rinv3(double r2, double gm) {
  // the seed of r2 == 0 (the sink itself) is finite
  double u, y3;
  sol_seed_square_cube(sol_rsqrt_seed(r2), u, y3);
  const double e = __fma_rn(-r2, u, 1.0);
  const double gy = gm * y3;
  return __fma_rn(gy, sol_split_t(e), gy);
}

__device__ __forceinline__ void pair_split(const TileSmem<4>& sm, int st, int jj, int j, int i, int ns, double xi,
                                           double yi, double zi, double& ax, double& ay, double& az,
                                           long long& r2minb, int& nn) {
  double dx = sm.v[st][SX][jj] - xi;
  double dy = sm.v[st][SY][jj] - yi;
  double dz = sm.v[st][SZ][jj] - zi;
  double r2 = __fma_rn(dx, dx, __fma_rn(dy, dy, dz * dz));
  double gm = (j < ns) ? sm.v[st][SGM][jj] : 0.0;  // gm of j == 0 and of padding is 0
  double s = split_gm_rinv3(r2, gm);
  ax = __fma_rn(s, dx, ax);
  ay = __fma_rn(s, dy, ay);
  az = __fma_rn(s, dz, az);
  long long rb = __double_as_longlong(r2);
  bool better = (rb < r2minb) & (j >= 1) & (j < ns) & (j != i);
  r2minb = better ? rb : r2minb;
  nn = better ? j : nn;
}

__device__ __forceinline__ void two_sum(double& s, double& c, double a) {
  double t = s + a;
  double bp = t - s;
  double err = (s - (t - bp)) + (a - bp);
  s = t;
  c += err;
}

// two_sum's result, bit for bit, with three FP64 instructions less: the larger of s
// and a by exponent (compared and selected on the integer pipe), then FastTwoSum.
__device__ __forceinline__ void add_ordered(double& s, double& c, double a) {
  const bool a_less = (__double2hiint(a) & 0x7FF00000) <= (__double2hiint(s) & 0x7FF00000);
  const double big = a_less ? s : a, small = a_less ? a : s;
  s = big + small;
  c += small - (s - big);
}

// spin: the limit of every mbarrier wait; withhold >= 0: that tile is never
// copied, so its wait runs out (failure-path tests only; -1 in production).
template <int PREC>
__global__ void __launch_bounds__(kSinkBlock) k_gravity_ac(ForceCtx fc, const double* __restrict__ y,
                                                           double* __restrict__ dydt, TimeSpec ts, uint32_t flags,
                                                           int* dev_status, uint32_t spin, int withhold) {
  constexpr int NARR = (PREC == SOL_PRECISION_FP64) ? 7 : 4;
  __shared__ __align__(128) TileSmem<NARR> sm;
  const Classes& c = fc.cls;
  const int n = sol_sink_hi(fc);  // sinks [sink_lo, n)
  const int i = fc.sink_lo + blockIdx.x * kSinkBlock + threadIdx.x;
  const int i_first = fc.sink_lo + blockIdx.x * kSinkBlock;
  // NOfMassive of GravityAC (:285-289); types are sorted, so the first sink
  // of the CTA has the largest source range.
  const int ns_cta = (fc.type[min(i_first, n - 1)] <= SOL_PROTO_PLANET) ? c.nm + c.n_spl : c.nm;
  const int ns = (i < n && fc.type[i] <= SOL_PROTO_PLANET) ? c.nm + c.n_spl : c.nm;
  const int ntiles = (ns_cta + kTile - 1) / kTile;

  double xi = 0, yi = 0, zi = 0;
  if (i < n) {
    xi = y[6 * i + 0];
    yi = y[6 * i + 1];
    zi = y[6 * i + 2];
  }
  if (threadIdx.x == 0) {
    sol_mbar_init(&sm.bar[0], 1);
    sol_mbar_init(&sm.bar[1], 1);
    sol_fence_barrier_init();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (ntiles > 0 && withhold != 0) issue_tile<NARR>(sm, fc.src, fc.npad, 0, 0);
    if (ntiles > 1 && withhold != 1) issue_tile<NARR>(sm, fc.src, fc.npad, 1, 1);
  }

  double ax = 0.0, ay = 0.0, az = 0.0;  // FP64: running sums; SPLIT: tile partials
  double sx = 0.0, sy = 0.0, sz = 0.0, cx = 0.0, cy = 0.0, cz = 0.0;  // SPLIT compensated totals
  long long rminb = (PREC == SOL_PRECISION_FP64) ? __double_as_longlong(1.0e10) : __double_as_longlong(1.0e20);
  int nn = -1;
  int issued = ntiles < 2 ? ntiles : 2;
  int t = 0;
  bool timed_out = false;

  for (; t < ntiles; ++t) {
    const int st = t & 1;
    const uint32_t parity = (t >> 1) & 1;
    const bool ok = sol_mbar_wait_n(&sm.bar[st], parity, spin);
    const int j0 = t * kTile;
    const int jmax = min(kTile, ns_cta - j0);  // sources beyond the CTA's range are never read
    if (ok && i < n && i >= 1) {
      if constexpr (PREC == SOL_PRECISION_FP64) {
#pragma unroll 4
        for (int jj = 0; jj < jmax; ++jj)
          pair_fp64(*reinterpret_cast<TileSmem<7>*>(&sm), st, jj, j0 + jj, i, ns, xi, yi, zi, ax, ay, az, rminb,
                    nn);
      } else {
        double tx = 0.0, ty = 0.0, tz = 0.0;
#pragma unroll 4
        for (int jj = 0; jj < jmax; ++jj)
          pair_split(*reinterpret_cast<TileSmem<4>*>(&sm), st, jj, j0 + jj, i, ns, xi, yi, zi, tx, ty, tz, rminb,
                     nn);
        two_sum(sx, cx, tx);
        two_sum(sy, cy, ty);
        two_sum(sz, cz, tz);
      }
    }
    // every thread is done with stage st; a timeout anywhere stops the whole CTA
    if (__syncthreads_or(!ok)) {
      timed_out = true;
      break;
    }
    if (threadIdx.x == 0 && t + 2 < ntiles) {
      sol_fence_proxy_async();
      if (t + 2 != withhold) issue_tile<NARR>(sm, fc.src, fc.npad, t + 2, st);
    }
    if (t + 2 < ntiles) issued = t + 3;
  }
  if (timed_out) {
    if (threadIdx.x == 0) {
      atomicOr(dev_status, SOL_DEV_TIMEOUT);
      // drain the copies still in flight (bounded) before the CTA exits
      for (int u = t; u < issued; ++u) sol_mbar_wait_n(&sm.bar[u & 1], (u >> 1) & 1, spin);
    }
    __syncthreads();
    return;
  }
  if (i >= n) return;
  double* out = dydt + 6 * i;
  if (i == 0) {  // GravityAC :253-254, :266
    for (int k = 0; k < 6; ++k) out[k] = 0.0;
    fc.nn_idx[0] = -1;
    fc.nn_dist[0] = 0.0;
    return;
  }
  const double* yv = y + 6 * i;
  const double mu = SOL_GAUSS2 * (fc.mass[0] + fc.mass[i]);
  const double rm3i = fc.rm3[i];
  double a[3];
  a[0] = -mu * rm3i * xi;  // Kepler term first (:281-283)
  a[1] = -mu * rm3i * yi;
  a[2] = -mu * rm3i * zi;
  if constexpr (PREC == SOL_PRECISION_FP64) {
    a[0] += ax;
    a[1] += ay;
    a[2] += az;
    fc.nn_idx[i] = nn;
    fc.nn_dist[i] = nn >= 0 ? __longlong_as_double(rminb) : 0.0;
  } else {
    const double* S = fc.ind_sum + ((fc.type[i] <= SOL_PROTO_PLANET) ? 3 : 0);
    const bool src_i = i < ns;
    const double* s = fc.src;
    const int np = fc.npad;
    double own[3] = {0.0, 0.0, 0.0};
    if (src_i) {
      double gmi = s[SGM * np + i];
      own[0] = gmi * s[SPX * np + i];
      own[1] = gmi * s[SPY * np + i];
      own[2] = gmi * s[SPZ * np + i];
    }
    a[0] += (sx + cx) - (S[0] - own[0]);
    a[1] += (sy + cy) - (S[1] - own[1]);
    a[2] += (sz + cz) - (S[2] - own[2]);
    // the reference's rij for the chosen neighbour (Acceleration.cpp:301-305), bit for bit
    double rij = 0.0;
    if (nn >= 0) {
      const double xij = y[6 * nn + 0] - xi, yij = y[6 * nn + 1] - yi, zij = y[6 * nn + 2] - zi;
      rij = __dsqrt_rn(xij * xij + yij * yij + zij * zij);
      if (!(rij < 1.0e10)) nn = -1;
    }
    fc.nn_idx[i] = nn;
    fc.nn_dist[i] = nn >= 0 ? rij : 0.0;
  }
  add_gas_terms(fc, i, yv, eval_time(ts), flags, a);
  out[0] = yv[3];
  out[1] = yv[4];
  out[2] = yv[5];
  out[3] = a[0];
  out[4] = a[1];
  out[5] = a[2];
}

// ---- FP64 GravityAC for sinks with many sources -------------------------------
// A CTA takes spc sinks.  Its producing warps compute the pair terms of a
// tile of kRefTile sources for all of them (the reference's arithmetic,
// Acceleration.cpp:294-317; a warp takes one sink and half a tile at a time)
// into one of two shared tiles, while its summing warp -- one lane per
// (sink, component) -- add the previous tile's terms in ascending source
// order: the reference's sequential sums, bit for bit.
//
// What bounds it.  The FP64 pipe is shared by the SM's four sub-partitions
// and takes one warp instruction per 16 cycles (19 for additions and
// multiplications), and one warp's instructions follow each other at 64
// cycles at the earliest, dependent or not.  So a pair costs its warp's FP64
// instructions, and a source costs each summing warp one more however few of
// its lanes have a sink: the sums fill 30 of 32 lanes (10 sinks a summing
// warp) where a warp per component would leave most of them empty, and the
// squares of the displacement join the term multiplications and the
// remainders of the root and the quotient (sol_crmath.cuh) on the integer
// pipe: 9 FP64 instructions a pair beside its three sums, where both pipes are
// about equally loaded.  (With the product r^2 r moved there too: 16,411
// bodies 6.95 ms for 7.02, 2,049 160 us for 156.)  A system of a few sinks per
// SM is bound by the sums' serial chain instead, 64 cycles a source alone and
// ~105 beside the producers, hence warps of their own for them rather than a
// phase in which the producers wait.  (Two half tiles interleaved in a
// producing warp, 108 registers: 1,033 bodies 62.3 us for 64.1, 4,099 646 for
// 509.)
//
// Measured (one evaluation, us; before: the two kernels this one replaces,
// 4 sinks x 224 sources with 12 summing lanes, and 32 sinks alternating
// between producing and summing): 300 bodies 37 -> 25 (prepass included), 1,033
// 94 -> 64, 2,049 305 -> 155, 4,099 900 -> 509, 16,411 10,800 -> 7,040, 65,536
// 150,000 -> 106,400.
constexpr int kRefTile = 64;      // sources per round
constexpr int kRefMaxSinks = 10;  // of a CTA: 30 of its summing warp's 32 lanes
constexpr int kRefProducers = 7;  // its other warps
constexpr int kRefRow = 33;       // doubles per row of terms (odd: conflict-free columns)
constexpr int kMaxDevices = 64;

constexpr size_t ref_smem(int spc) {
  return sizeof(double) * (2 * 7 * kRefTile + 2 * (size_t)kRefTile * kRefRow) +
         (sizeof(long long) + sizeof(int)) * (size_t)kRefTile * spc;
}

// rij and 1 / rij^3 of a displacement, the squares on the integer pipe (a z
// that is zero for every pair, a planar system, stays on the fast path)
__device__ __forceinline__ void ref_pair(double xij, double yij, double zij, bool valid, double& rij, double& rijm3) {
  bool ok = true;
  const double qx = sol_exact_dsqr<false>(xij, ok);
  const double qy = sol_exact_dsqr<false>(yij, ok);
  const double qz = sol_exact_dsqr<true>(zij, ok);
  ok = ok & sol_ref_rinv3_fast(qx + qy + qz, rij, rijm3);
  if (!ok & valid) {
    const double2 v = sol_ref_pair_ieee(xij, yij, zij);
    rij = v.x;
    rijm3 = v.y;
  }
}

// Three CTAs an SM (80 registers).  With four (64 registers, a few spilled):
// 1,033 bodies 66.3 us for 64.1, 4,099 521 for 509, 16,411 7.02 ms for 7.05.
__global__ void __launch_bounds__((1 + kRefProducers) * 32, 3)
    k_gravity_ac_ref(ForceCtx fc, const double* __restrict__ y, double* __restrict__ dydt, TimeSpec ts, uint32_t flags,
                     int spc) {
  extern __shared__ __align__(16) double ref_dyn[];
  __shared__ double sink_pos[kRefMaxSinks][3];
  __shared__ int sink_ns[kRefMaxSinks];
  __shared__ double acc[32];
  __shared__ double nn_d[kRefMaxSinks];
  __shared__ int nn_i[kRefMaxSinks];
  double* srct = ref_dyn;                      // [2][7][kRefTile] source tiles
  double* terms = srct + 2 * 7 * kRefTile;     // [2][kRefTile][kRefRow]
  long long* nn_r = reinterpret_cast<long long*>(terms + 2 * kRefTile * kRefRow);  // [2 spc][32] nearest so far
  int* nn_j = reinterpret_cast<int*>(nn_r + kRefTile * spc);
  const Classes& c = fc.cls;
  const int n = sol_sink_hi(fc);  // sinks [sink_lo, n)
  const int i0 = fc.sink_lo + blockIdx.x * spc;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x < spc) {
    const int i = i0 + threadIdx.x;
    const bool live = i < n && i >= 1;
    sink_ns[threadIdx.x] = live ? ((fc.type[i] <= SOL_PROTO_PLANET) ? c.nm + c.n_spl : c.nm) : 0;
    for (int k = 0; k < 3; ++k) sink_pos[threadIdx.x][k] = i < n ? y[6 * i + k] : 0.0;
  }
  for (int q = threadIdx.x; q < kRefTile * spc; q += blockDim.x) {
    nn_r[q] = __double_as_longlong(1.0e10);
    nn_j[q] = -1;
  }
  const double* src = fc.src;
  const int np = fc.npad;
  constexpr int kLoads = (7 * kRefTile + kRefProducers * 32 - 1) / (kRefProducers * 32);
  const int pt = (warp - 1) * 32 + lane;  // producing thread
  if (warp >= 1)
    for (int q = pt; q < 7 * kRefTile; q += kRefProducers * 32) srct[q] = src[(size_t)(q / kRefTile) * np + (q % kRefTile)];
  __syncthreads();
  int ns_cta = 0;
  for (int s = 0; s < spc; ++s) ns_cta = max(ns_cta, sink_ns[s]);
  const int rounds = (ns_cta + kRefTile - 1) / kRefTile;
  double a_sum = 0.0;
  // round r: the producers fill term tile r & 1 from source tile r & 1 and
  // fetch the next sources; the summing warp adds term tile (r - 1) & 1
  for (int r = 0; r <= rounds; ++r) {
    if (warp >= 1) {
      if (r < rounds) {
        double pre[kLoads];
        const bool more = r + 1 < rounds;
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
          const int q = pt + u * kRefProducers * 32;
          pre[u] = (more && q < 7 * kRefTile)
                       ? src[(size_t)(q / kRefTile) * np + (r + 1) * kRefTile + (q % kRefTile)]
                       : 0.0;
        }
        const double* st = srct + (r & 1) * 7 * kRefTile;
        double* out = terms + (size_t)(r & 1) * kRefTile * kRefRow;
#pragma unroll 1
        for (int item = warp - 1; item < 2 * spc; item += kRefProducers) {  // (sink, half of the tile)
          const int s = item >> 1;
          const int p = (item & 1) * 32 + lane;
          const int j = r * kRefTile + p;
          const bool valid = j >= 1 && j < sink_ns[s] && j != i0 + s;
          const double xij = st[SX * kRefTile + p] - sink_pos[s][0];
          const double yij = st[SY * kRefTile + p] - sink_pos[s][1];
          const double zij = st[SZ * kRefTile + p] - sink_pos[s][2];
          double rij, rijm3;
          ref_pair(xij, yij, zij, valid, rij, rijm3);
          double tx, ty, tz;
          sol_ref_terms(st[SGM * kRefTile + p], rijm3, xij, yij, zij, st[SPX * kRefTile + p], st[SPY * kRefTile + p],
                        st[SPZ * kRefTile + p], tx, ty, tz);
          // a source the sink does not take adds +0, which changes no sum:
          // a sum that starts at +0 is never -0
          double* o = out + (size_t)p * kRefRow + 3 * s;
          o[0] = tx;
          o[1] = ty;
          o[2] = tz;
          if (!valid) o[0] = o[1] = o[2] = 0.0;
          const long long rb = __double_as_longlong(rij);
          if (valid && rb < nn_r[item * 32 + lane]) {
            nn_r[item * 32 + lane] = rb;
            nn_j[item * 32 + lane] = j;
          }
        }
        double* nx = srct + ((r + 1) & 1) * 7 * kRefTile;
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
          const int q = pt + u * kRefProducers * 32;
          if (q < 7 * kRefTile) nx[q] = pre[u];
        }
      }
    } else if (r > 0) {
      if (lane < 3 * spc) {  // 3 sink + component
        const double* col = terms + (size_t)((r - 1) & 1) * kRefTile * kRefRow + lane;
#pragma unroll
        for (int p = 0; p < kRefTile; ++p) a_sum += col[p * kRefRow];
      }
    }
    __syncthreads();
  }
  if (warp == 0) acc[lane] = a_sum;
  // nearest neighbour of a sink: the smallest distance over its 64 columns,
  // ties to the lowest index (each column keeps its first minimum)
  for (int s = warp; s < spc; s += 1 + kRefProducers) {
    long long b = nn_r[(2 * s) * 32 + lane];
    int bj = nn_j[(2 * s) * 32 + lane];
    const long long b2 = nn_r[(2 * s + 1) * 32 + lane];
    const int j2 = nn_j[(2 * s + 1) * 32 + lane];
    if (b2 < b || (b2 == b && (unsigned)j2 < (unsigned)bj)) {
      b = b2;
      bj = j2;
    }
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
      const long long ob = __shfl_xor_sync(0xFFFFFFFFu, b, w);
      const int oj = __shfl_xor_sync(0xFFFFFFFFu, bj, w);
      if (ob < b || (ob == b && (unsigned)oj < (unsigned)bj)) {
        b = ob;
        bj = oj;
      }
    }
    if (lane == 0) {
      nn_d[s] = bj >= 0 ? __longlong_as_double(b) : 0.0;
      nn_i[s] = bj;
    }
  }
  __syncthreads();
  if (threadIdx.x >= spc) return;
  const int s = threadIdx.x;
  const int i = i0 + s;
  if (i >= n) return;
  double* out = dydt + 6 * i;
  if (i == 0) {  // GravityAC :253-254, :266
    for (int k = 0; k < 6; ++k) out[k] = 0.0;
    fc.nn_idx[0] = -1;
    fc.nn_dist[0] = 0.0;
    return;
  }
  const double* yv = y + 6 * i;
  const double xi = sink_pos[s][0], yi = sink_pos[s][1], zi = sink_pos[s][2];
  const double mu = SOL_GAUSS2 * (fc.mass[0] + fc.mass[i]);
  const double rm3i = fc.rm3[i];
  double a[3];
  a[0] = -mu * rm3i * xi;  // Kepler term first (:281-283)
  a[1] = -mu * rm3i * yi;
  a[2] = -mu * rm3i * zi;
  a[0] += acc[3 * s + 0];
  a[1] += acc[3 * s + 1];
  a[2] += acc[3 * s + 2];
  fc.nn_idx[i] = nn_i[s];
  fc.nn_dist[i] = nn_d[s];
  add_gas_terms(fc, i, yv, eval_time(ts), flags, a);
  out[0] = yv[3];
  out[1] = yv[4];
  out[2] = yv[5];
  out[3] = a[0];
  out[4] = a[1];
  out[5] = a[2];
}

// GravityBC_SelfInteracting / _NonSelfInteracting (Acceleration.cpp:541-634):
// massive sinks and non-massive sinks both sum over massive sources in
// descending order, scale by G at the end; no rm3.
__global__ void __launch_bounds__(kSinkBlock) k_gravity_bc(ForceCtx fc, const double* __restrict__ y,
                                                           double* __restrict__ dydt, TimeSpec ts,
                                                           uint32_t flags) {
  const int n = fc.cls.n;
  const int i = blockIdx.x * kSinkBlock + threadIdx.x;
  if (i >= n) return;
  const double* s = fc.src;
  const int np = fc.npad;
  const double* yv = y + 6 * i;
  double xi = yv[0], yi = yv[1], zi = yv[2];
  double a[3] = {0.0, 0.0, 0.0};
  long long rminb = __double_as_longlong(1.0e10);
  int nn = -1;
  for (int j = fc.cls.nm - 1; j >= 0; j--) {
    if (j == i) continue;
    double dx = s[SX * np + j] - xi;
    double dy = s[SY * np + j] - yi;
    double dz = s[SZ * np + j] - zi;
    double rij2 = dx * dx + dy * dy + dz * dz;
    double rij = __dsqrt_rn(rij2);
    long long rb = __double_as_longlong(rij);
    if (rb < rminb) {
      rminb = rb;
      nn = j;
    }
    double cc = __ddiv_rn(s[SGM * np + j] * 1.0, rij2 * rij);
    a[0] += cc * dx;
    a[1] += cc * dy;
    a[2] += cc * dz;
  }
  a[0] *= SOL_GAUSS2;
  a[1] *= SOL_GAUSS2;
  a[2] *= SOL_GAUSS2;
  fc.nn_idx[i] = nn;
  fc.nn_dist[i] = nn >= 0 ? __longlong_as_double(rminb) : 0.0;
  add_gas_terms(fc, i, yv, eval_time(ts), flags, a);
  double* out = dydt + 6 * i;
  out[0] = yv[3];
  out[1] = yv[4];
  out[2] = yv[5];
  out[3] = a[0];
  out[4] = a[1];
  out[5] = a[2];
}


// 2-D pair kernel of the SPLIT form: blockIdx.x = block of kSinkBlock sinks,
// blockIdx.y = chunk of `chunk` sources.  Each CTA writes, per sink, its
// partial acceleration sum and nearest-neighbour candidate for the chunk;
// k_combine adds the chunks in a fixed order.  Many small work units let the
// block scheduler balance the FP64 pipe load across SMs.  (SPLIT_FF has its
// own 2-D kernel, k_pairs_ff.)
template <int MODE>
__global__ void __launch_bounds__(kSinkBlock) k_pairs(ForceCtx fc, const double* __restrict__ y,
                                                      double* __restrict__ part, int* dev_status, int chunk) {
  static_assert(MODE == SOL_PRECISION_SPLIT, "k_pairs serves the SPLIT form");
  constexpr int NARR = 4;  // x, y, z and G m
  __shared__ __align__(128) TileSmem<NARR> sm;
  const Classes& c = fc.cls;
  const int n = sol_sink_hi(fc);  // sinks [sink_lo, n)
  const int np = fc.npad;
  const int i = fc.sink_lo + blockIdx.x * kSinkBlock + threadIdx.x;
  const int i_first = fc.sink_lo + blockIdx.x * kSinkBlock;
  const int ns_cta = (fc.type[min(i_first, n - 1)] <= SOL_PROTO_PLANET) ? c.nm + c.n_spl : c.nm;
  const int ns = (i < n && fc.type[i] <= SOL_PROTO_PLANET) ? c.nm + c.n_spl : c.nm;
  const int j_begin = blockIdx.y * chunk;
  const int j_end = min(j_begin + chunk, ns_cta);
  const int t_begin = j_begin / kTile;
  const int ntiles = j_end > j_begin ? (j_end - j_begin + kTile - 1) / kTile : 0;
  const int arr[NARR] = {SX, SY, SZ, SGM};

  double xi = 0, yi = 0, zi = 0;
  if (i < n) {
    xi = y[6 * i + 0];
    yi = y[6 * i + 1];
    zi = y[6 * i + 2];
  }
  if (threadIdx.x == 0) {
    sol_mbar_init(&sm.bar[0], 1);
    sol_mbar_init(&sm.bar[1], 1);
    sol_fence_barrier_init();
  }
  __syncthreads();
  auto issue = [&](int t, int stage) {
    sol_mbar_expect_tx(&sm.bar[stage], NARR * kTile * 8);
    for (int k = 0; k < NARR; ++k)
      sol_bulk_g2s(&sm.v[stage][k][0], fc.src + (size_t)arr[k] * np + (size_t)(t_begin + t) * kTile, kTile * 8,
                   &sm.bar[stage]);
  };
  if (threadIdx.x == 0) {
    if (ntiles > 0) issue(0, 0);
    if (ntiles > 1) issue(1, 1);
  }
  double ax = 0.0, ay = 0.0, az = 0.0;  // chunk sums of the per-tile partials
  double cx = 0.0, cy = 0.0, cz = 0.0;  // compensation terms
  long long r2minb = __double_as_longlong(1.0e20);
  int nn = -1;
  int issued = ntiles < 2 ? ntiles : 2;
  int t = 0;
  bool timed_out = false;
  for (; t < ntiles; ++t) {
    const int st = t & 1;
    const bool ok = sol_mbar_wait(&sm.bar[st], (t >> 1) & 1);
    const int j0 = (t_begin + t) * kTile;
    const int jmax = min(kTile, j_end - j0);  // sources beyond the chunk's range are never read
    if (ok && i < n && i >= 1) {
      double tx = 0.0, ty = 0.0, tz = 0.0;
#pragma unroll 4
      for (int jj = 0; jj < jmax; ++jj)
        pair_split(*reinterpret_cast<TileSmem<4>*>(&sm), st, jj, j0 + jj, i, ns, xi, yi, zi, tx, ty, tz, r2minb, nn);
      two_sum(ax, cx, tx);
      two_sum(ay, cy, ty);
      two_sum(az, cz, tz);
    }
    if (__syncthreads_or(!ok)) {
      timed_out = true;
      break;
    }
    if (threadIdx.x == 0 && t + 2 < ntiles) {
      sol_fence_proxy_async();
      issue(t + 2, st);
    }
    if (t + 2 < ntiles) issued = t + 3;
  }
  if (timed_out) {
    if (threadIdx.x == 0) {
      atomicOr(dev_status, SOL_DEV_TIMEOUT);
      for (int u = t; u < issued; ++u) sol_mbar_wait(&sm.bar[u & 1], (u >> 1) & 1);
    }
    __syncthreads();
    return;
  }
  if (i >= n) return;
  const size_t base = (size_t)blockIdx.y * PART_SLOTS * np + i;
  part[base + PAX * np] = ax + cx;
  part[base + PAY * np] = ay + cy;
  part[base + PAZ * np] = az + cz;
  part[base + PR2 * np] = nn >= 0 ? __longlong_as_double(r2minb) : 1.0e300;
  part[base + PIDX * np] = __longlong_as_double((long long)nn);
}

// ---- SPLIT_FF 2-D kernel: float-float pairs with no FP64 instruction -------
// Same grid as k_pairs (blockIdx.x: kSinkBlock sinks; blockIdx.y: a chunk of
// sources, 1 to kChunkTiles tiles as ff_chunk chooses so that the grid
// fills the GPU) and the same partial outputs for k_combine.  The sources'
// grid triples and G m (hi, lo) arrive tile by tile in shared memory by bulk
// copies; each thread takes two sources per step in paired FP32
// instructions: the displacement from the grid triples (exact parts, no
// FP64), r^2, G m r^-3 and the accumulation in float-float (sol_pair.cuh).
// Pairs closer than the grid G1 (|d| < G1, where the triple displacement
// would lose relative accuracy) take FP64 arithmetic, as pairs below 1e-12 AU
// do in the other float-float kernels.  Tiles whose sources are all valid
// for every sink of the warp (no sink index, no central body, no source
// beyond a sink's source count or the chunk) run without per-pair tests.
constexpr int kFF = FTAB_USED;

struct FFTile {
  float v[2][kFF][kTile];
  uint64_t bar[2];
};

// One FP64 pair of the close-pair branch: G m r^-3 d into (fx, fy, fz);
// r^2 for the nearest-neighbour comparison as (hi, lo) floats.
__device__ __forceinline__ void ff_close_pair(const ForceCtx& fc, int j, double xi, double yi, double zi, float gh,
                                           float gl, double& fx, double& fy, double& fz, float& r2h, float& r2l) {
  const double* s = fc.src;
  const int np = fc.npad;
  const double dx = s[SX * np + j] - xi, dy = s[SY * np + j] - yi, dz = s[SZ * np + j] - zi;
  const double r2 = __fma_rn(dx, dx, __fma_rn(dy, dy, dz * dz));
  r2h = __double2float_rn(r2);
  r2l = __double2float_rn(r2 - (double)r2h);
  if (r2 > 0.0) {
    const double rinv = __drcp_rn(__dsqrt_rn(r2));
    const double sd = ((double)gh + (double)gl) * (rinv * rinv * rinv);
    fx = __fma_rn(sd, dx, fx);
    fy = __fma_rn(sd, dy, fy);
    fz = __fma_rn(sd, dz, fz);
  }
}

// Nearest-neighbour candidate: the smallest r^2 (hi, then lo), the first in
// ascending source order.
__device__ __forceinline__ void ff_nn(float r2h, float r2l, bool ok, int j, float& mh, float& ml, int& nn) {
  const bool better = ok & ((r2h < mh) | ((r2h == mh) & (r2l < ml)));
  mh = better ? r2h : mh;
  ml = better ? r2l : ml;
  nn = better ? j : nn;
}

// Two sources (j, j + 1) of the tile against the sink, their table rows in
// sv (one float2 per row).  MASKED: per-pair validity (source range, the
// sink itself, the chunk end) is tested.  The accumulators are renormalised
// when renorm is set: after the second pair of every group of four sources,
// as ff_four_sources does, so a sink gets the same bits whether its warp
// takes a tile on the masked path or the fast one.
template <bool MASKED>
__device__ __forceinline__ void ff_two_sources(const float2* sv, int j, int i, int ns, int jend, bool renorm,
                                               const float* ai, const float* bi, const float* ci, float thr,
                                               const ForceCtx& fc, double xi, double yi, double zi, float2* Ah,
                                               float2* Al, double& fx, double& fy, double& fz, float& mh, float& ml,
                                               int& nn) {
  float2 h[3], l[3];
#pragma unroll
  for (int k = 0; k < 3; ++k)
    f2_grid_disp(sv[FAX + 3 * k], sv[FBX + 3 * k], sv[FCX + 3 * k], ai[k], bi[k], ci[k], h[k], l[k]);
  float2 gh = sv[FGH];
  float2 gl = sv[FGL];
  float2 r2h, r2l;
  f2_ff_r2(h, l, r2h, r2l);
  bool ok0 = true, ok1 = true;
  if constexpr (MASKED) {
    ok0 = (j >= 1) & (j < ns) & (j != i) & (j < jend);
    ok1 = (j + 1 >= 1) & (j + 1 < ns) & (j + 1 != i) & (j + 1 < jend);
  }
  float2 qh = r2h, ql = r2l;
  if (!ok0 || r2h.x < thr) {
    if (ok0) ff_close_pair(fc, j, xi, yi, zi, gh.x, gl.x, fx, fy, fz, r2h.x, r2l.x);
    gh.x = gl.x = 0.0f;
    qh.x = 1.0f;
    ql.x = 0.0f;
  }
  if (!ok1 || r2h.y < thr) {
    if (ok1) ff_close_pair(fc, j + 1, xi, yi, zi, gh.y, gl.y, fx, fy, fz, r2h.y, r2l.y);
    gh.y = gl.y = 0.0f;
    qh.y = 1.0f;
    ql.y = 0.0f;
  }
  float2 sh, se;
  f2_ff_gm_rinv3(qh, ql, gh, gl, sh, se);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    f2_ff_accumulate_lazy(Ah[k], Al[k], sh, se, h[k], l[k]);
    if (renorm) f2_fast_two_sum(Ah[k], Al[k], Ah[k], Al[k]);
  }
  ff_nn(r2h.x, r2l.x, ok0, j, mh, ml, nn);
  ff_nn(r2h.y, r2l.y, ok1, j + 1, mh, ml, nn);
}


// Four sources (j .. j + 3) of a fast tile: the displacements and r^2 of both
// pairs of sources first, one test for a close pair among the four, then
// G m r^-3 and the accumulation of both in one basic block, the branch no
// longer splitting the step into short blocks the scheduler cannot
// interleave (16.10 -> 14.96 ms at 65,536 bodies); the accumulators are
// renormalised once per step instead of after each half (14.52 ms); the
// nearest-neighbour update runs only when the four sources' smallest r^2
// reaches the running minimum, which over a sink's sources happens about
// ln(N) times (13.92 ms).  The update itself is exact either way.
__device__ __forceinline__ void ff_close_lane(const ForceCtx& fc, int j, double xi, double yi, double zi, float& gh,
                                              float& gl, double& fx, double& fy, double& fz, float& r2h, float& r2l,
                                              float& qh, float& ql, float thr) {
  if (r2h < thr) {
    ff_close_pair(fc, j, xi, yi, zi, gh, gl, fx, fy, fz, r2h, r2l);
    gh = gl = 0.0f;
    qh = 1.0f;
    ql = 0.0f;
  }
}
__device__ __forceinline__ void ff_four_sources(const float2* va, const float2* vb, int j, const float* ai,
                                                const float* bi, const float* ci, float thr, const ForceCtx& fc,
                                                double xi, double yi, double zi, float2* Ah, float2* Al, double& fx,
                                                double& fy, double& fz, float& mh, float& ml, int& nn) {
  float2 ha[3], la[3], hb[3], lb[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    f2_grid_disp(va[FAX + 3 * k], va[FBX + 3 * k], va[FCX + 3 * k], ai[k], bi[k], ci[k], ha[k], la[k]);
    f2_grid_disp(vb[FAX + 3 * k], vb[FBX + 3 * k], vb[FCX + 3 * k], ai[k], bi[k], ci[k], hb[k], lb[k]);
  }
  float2 gha = va[FGH], gla = va[FGL], ghb = vb[FGH], glb = vb[FGL];
  float2 r2ha, r2la, r2hb, r2lb;
  f2_ff_r2(ha, la, r2ha, r2la);
  f2_ff_r2(hb, lb, r2hb, r2lb);
  float2 qha = r2ha, qla = r2la, qhb = r2hb, qlb = r2lb;
  const float m4 = fminf(fminf(r2ha.x, r2ha.y), fminf(r2hb.x, r2hb.y));
  if (m4 < thr) {
    ff_close_lane(fc, j, xi, yi, zi, gha.x, gla.x, fx, fy, fz, r2ha.x, r2la.x, qha.x, qla.x, thr);
    ff_close_lane(fc, j + 1, xi, yi, zi, gha.y, gla.y, fx, fy, fz, r2ha.y, r2la.y, qha.y, qla.y, thr);
    ff_close_lane(fc, j + 2, xi, yi, zi, ghb.x, glb.x, fx, fy, fz, r2hb.x, r2lb.x, qhb.x, qlb.x, thr);
    ff_close_lane(fc, j + 3, xi, yi, zi, ghb.y, glb.y, fx, fy, fz, r2hb.y, r2lb.y, qhb.y, qlb.y, thr);
  }
  float2 sha, sea, shb, seb;
  f2_ff_gm_rinv3(qha, qla, gha, gla, sha, sea);
  f2_ff_gm_rinv3(qhb, qlb, ghb, glb, shb, seb);
#pragma unroll
  for (int k = 0; k < 3; ++k) {  // both halves, one renormalisation
    f2_ff_accumulate_lazy(Ah[k], Al[k], sha, sea, ha[k], la[k]);
    f2_ff_accumulate_lazy(Ah[k], Al[k], shb, seb, hb[k], lb[k]);
    f2_fast_two_sum(Ah[k], Al[k], Ah[k], Al[k]);
  }
  // a new nearest neighbour is rare: only when the four sources' smallest
  // r^2 reaches the running minimum (or a close pair replaced an r^2)
  if (m4 <= mh || m4 < thr) {
    ff_nn(r2ha.x, r2la.x, true, j, mh, ml, nn);
    ff_nn(r2ha.y, r2la.y, true, j + 1, mh, ml, nn);
    ff_nn(r2hb.x, r2lb.x, true, j + 2, mh, ml, nn);
    ff_nn(r2hb.y, r2lb.y, true, j + 3, mh, ml, nn);
  }
}

// Three CTAs per SM (up to 170 registers): the four-source step keeps both
// halves' temporaries live at once.
__global__ void __launch_bounds__(kSinkBlock, 3) k_pairs_ff(ForceCtx fc, const double* __restrict__ y,
                                                         double* __restrict__ part, int* dev_status, int chunk,
                                                         int j_lo, int j_hi) {
  __shared__ __align__(128) FFTile sm;
  const Classes& c = fc.cls;
  const int n = sol_sink_hi(fc);  // sinks [sink_lo, n)
  const int np = fc.npad;
  const int i = fc.sink_lo + blockIdx.x * kSinkBlock + threadIdx.x;
  const int i_first = fc.sink_lo + blockIdx.x * kSinkBlock;
  const int ns_cta = (fc.type[min(i_first, n - 1)] <= SOL_PROTO_PLANET) ? c.nm + c.n_spl : c.nm;
  const int ns = (i < n && fc.type[i] <= SOL_PROTO_PLANET) ? c.nm + c.n_spl : c.nm;
  const int j_begin = j_lo + blockIdx.y * chunk;  // sources [j_lo, j_hi); j_lo a whole number of tiles
  const int j_end = min(j_begin + chunk, min(ns_cta, j_hi));
  const int t_begin = j_begin / kTile;
  const int ntiles = j_end > j_begin ? (j_end - j_begin + kTile - 1) / kTile : 0;
  const bool live = i < n && i >= 1;

  const float* T = ftab(fc);
  float ai[3], bi[3], ci[3];
  double xi = 0, yi = 0, zi = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    ai[k] = i < n ? T[(size_t)(FAX + 3 * k) * np + i] : 0.0f;
    bi[k] = i < n ? T[(size_t)(FBX + 3 * k) * np + i] : 0.0f;
    ci[k] = i < n ? T[(size_t)(FCX + 3 * k) * np + i] : 0.0f;
  }
  if (i < n) {
    xi = y[6 * i + 0];
    yi = y[6 * i + 1];
    zi = y[6 * i + 2];
  }
  const double G1 = fc.ind_sum[kIndGrid];
  // |d| < max(G1, 2^-50): the FP64 branch (the floor keeps every r^2 the
  // float-float path sees a normal float)
  const float thr = fmaxf((float)(G1 * G1), 7.888609052210118e-31f);

  if (threadIdx.x == 0) {
    sol_mbar_init(&sm.bar[0], 1);
    sol_mbar_init(&sm.bar[1], 1);
    sol_fence_barrier_init();
  }
  __syncthreads();
  auto issue = [&](int t, int stage) {
    sol_mbar_expect_tx(&sm.bar[stage], kFF * kTile * 4);
    for (int k = 0; k < kFF; ++k)
      sol_bulk_g2s(&sm.v[stage][k][0], T + (size_t)k * np + (size_t)(t_begin + t) * kTile, kTile * 4,
                   &sm.bar[stage]);
  };
  if (threadIdx.x == 0) {
    if (ntiles > 0) issue(0, 0);
    if (ntiles > 1) issue(1, 1);
  }
  double ax = 0.0, ay = 0.0, az = 0.0, cx = 0.0, cy = 0.0, cz = 0.0;  // chunk sums, compensated
  double fx = 0.0, fy = 0.0, fz = 0.0;                                  // close pairs, FP64
  float mh = 3.0e38f, ml = 0.0f;
  int nn = -1;
  int issued = ntiles < 2 ? ntiles : 2;
  int t = 0;
  bool timed_out = false;
  for (; t < ntiles; ++t) {
    const int st = t & 1;
    const bool ok = sol_mbar_wait(&sm.bar[st], (t >> 1) & 1);
    const int j0 = (t_begin + t) * kTile;
    const int jend = min(j0 + kTile, j_end);
    // the warp's sinks all see every source of the tile, none of them is in it
    const bool clean = live && j0 >= 1 && jend == j0 + kTile && j0 + kTile <= ns && (i < j0 || i >= j0 + kTile);
    const bool fast = __all_sync(0xFFFFFFFFu, clean);
    if (ok && live) {
      float2 Ah[3], Al[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) Ah[k] = Al[k] = make_float2(0.0f, 0.0f);
      if (fast) {
        // four sources per step: one 16-byte shared load per table row
#pragma unroll 1
        for (int jj = 0; jj < kTile; jj += 4) {
          float2 va[kFF], vb[kFF];
#pragma unroll
          for (int k = 0; k < kFF; ++k) {
            const float4 q = *reinterpret_cast<const float4*>(&sm.v[st][k][jj]);
            va[k] = make_float2(q.x, q.y);
            vb[k] = make_float2(q.z, q.w);
          }
          ff_four_sources(va, vb, j0 + jj, ai, bi, ci, thr, fc, xi, yi, zi, Ah, Al, fx, fy, fz, mh, ml, nn);
        }
      } else {
        for (int jj = 0; jj < jend - j0; jj += 2) {
          float2 va[kFF];
#pragma unroll
          for (int k = 0; k < kFF; ++k) va[k] = *reinterpret_cast<const float2*>(&sm.v[st][k][jj]);
          ff_two_sources<true>(va, j0 + jj, i, ns, jend, (jj & 2) != 0, ai, bi, ci, thr, fc, xi, yi, zi, Ah, Al, fx,
                               fy, fz, mh, ml, nn);
        }
      }
      // the tile's float-float partials (even and odd sources) into the FP64 chunk sums
      two_sum(ax, cx, ((double)Ah[0].x + (double)Al[0].x) + ((double)Ah[0].y + (double)Al[0].y));
      two_sum(ay, cy, ((double)Ah[1].x + (double)Al[1].x) + ((double)Ah[1].y + (double)Al[1].y));
      two_sum(az, cz, ((double)Ah[2].x + (double)Al[2].x) + ((double)Ah[2].y + (double)Al[2].y));
    }
    if (__syncthreads_or(!ok)) {
      timed_out = true;
      break;
    }
    if (threadIdx.x == 0 && t + 2 < ntiles) {
      sol_fence_proxy_async();
      issue(t + 2, st);
    }
    if (t + 2 < ntiles) issued = t + 3;
  }
  if (timed_out) {
    if (threadIdx.x == 0) {
      atomicOr(dev_status, SOL_DEV_TIMEOUT);
      for (int u = t; u < issued; ++u) sol_mbar_wait(&sm.bar[u & 1], (u >> 1) & 1);
    }
    __syncthreads();
    return;
  }
  if (i >= n) return;
  const size_t base = (size_t)blockIdx.y * PART_SLOTS * np + i;
  part[base + PAX * np] = (ax + cx) + fx;
  part[base + PAY * np] = (ay + cy) + fy;
  part[base + PAZ * np] = (az + cz) + fz;
  part[base + PR2 * np] = nn >= 0 ? (double)mh + (double)ml : 1.0e300;
  part[base + PIDX * np] = __longlong_as_double((long long)nn);
}

#include "sol_pairs_sym.cuh"

// Where the partials of an evaluation lie in the context's d_part (offsets in
// doubles): of the block pairs of k_pairs_sym (bodies [0, nb block)), sources'
// and sinks' sides, and of k_pairs_ff on what is left: r1, every sink and the
// sources from `from` on; r2, the sinks from there on and the sources before.
struct FFPlan {
  int block = kTile, nb = 0, per = 1, chunks = 0;  // k_pairs_sym
  int from = 0;                                    // nb block
  int n1 = 0, chunk1 = kTile, n2 = 0, chunk2 = kTile;
  size_t o_j = 0, o_i = 0, o_1 = 0, o_2 = 0, o_bound = 0;
};

// Per sink: the partials in a fixed order, the nearest neighbour (the
// smallest r^2, ties to the lower index as the reference's ascending scan),
// distanceOfNN recomputed in the reference's FP64 arithmetic for the chosen
// neighbour, the Kepler and indirect terms, and the gas terms.
// Bounded by the latency of the partials' loads (a few tens to some hundreds a
// sink, far apart): a CTA's warps share its sinks' partials, four loaded at a
// time, a warp a component adds the warps' sums, and the first warp finishes.
// The sums are 128-bit integers (FixSum), ~75 integer instructions a partial, as
// accurate as compensated ones: those take 12 FP64 instructions a partial (21
// with two_sum) of 16 cycles each.  An evaluation of 10,007 bodies 338 us for
// 372, of 65,536 11.10 ms for 11.29; the kernel 30 and 131 us for 63 and 332
// (27 and 131 with plain FP64 sums; one thread a sink 65 and 213).
constexpr int kCombineSinks = 32, kCombineWarps = 8, kCombineLoads = 4;

// A sum of doubles as a 128-bit integer A 2^(base - 1075), on the integer pipe.
// A value of exponent field e is shifted left by e - base, 0 to 63 places; a
// larger one raises the base so that it lies kFixPlace places up (fix_add_slow),
// what lies below the last place is cut off: 2^-106 of the largest value, as a
// compensated sum's second word.  2^11 values of the window's end fit.
struct FixSum {
  unsigned long long lo;
  long long hi;
  int base;
};
constexpr int kFixPlace = 54, kFixEmpty = -(1 << 20), kFixNan = 1 << 20;

__device__ __forceinline__ void fix_add_shifted(FixSum& a, long long m, int sh) {
  const unsigned r = sh & 31;
  const unsigned w0 = (unsigned)m, w1 = (unsigned)(m >> 32), w2 = (unsigned)((int)w1 >> 31);
  const unsigned s0 = w0 << r, s1 = __funnelshift_l(w0, w1, r), s2 = __funnelshift_l(w1, w2, r);
  const bool word = sh >= 32;
  const unsigned long long lo = word ? (unsigned long long)s0 << 32 : ((unsigned long long)s1 << 32 | s0);
  const unsigned long long hi = word ? ((unsigned long long)s2 << 32 | s1) : ((unsigned long long)w2 << 32 | s2);
  const unsigned long long t = a.lo + lo;
  a.hi += (long long)(hi + (t < lo ? 1u : 0u));
  a.lo = t;
}
static __device__ __noinline__ FixSum fix_add_slow(FixSum a, double v) {
  const long long b = __double_as_longlong(v);
  const int ef = (int)(b >> 52) & 0x7FF;
  if (ef == 0x7FF || a.base == kFixNan) {  // as a compensated sum of an infinity gives
    a.base = kFixNan;
    return a;
  }
  long long m = (b & 0xFFFFFFFFFFFFFll) | (ef ? 1ll << 52 : 0ll);
  if (b < 0) m = -m;
  const int e = max(ef, 1);
  int sh = e - a.base;
  if (sh > 63) {
    const int up = min(sh - kFixPlace, 127);
    if (up >= 64) {
      a.lo = (unsigned long long)(a.hi >> (up - 64));
      a.hi >>= 63;
    } else {
      a.lo = (a.lo >> up) | ((unsigned long long)a.hi << (64 - up));
      a.hi >>= up;
    }
    a.base = e - kFixPlace;
    sh = kFixPlace;
  }
  if (sh < 0) {
    m >>= min(-sh, 63);
    sh = 0;
  }
  fix_add_shifted(a, m, sh);
  return a;
}
__device__ __forceinline__ void fix_add(FixSum& a, double v) {
  const unsigned h = (unsigned)__double2hiint(v), l = (unsigned)__double2loint(v);
  const int ef = (int)(h >> 20) & 0x7FF;
  const int sh = ef - a.base;
  if ((unsigned)sh > 63u || ef == 0) {
    if ((h << 1 | l) != 0u) a = fix_add_slow(a, v);
    return;
  }
  const unsigned sg = (unsigned)((int)h >> 31);
  const unsigned long long m = ((unsigned long long)((h & 0xFFFFFu) | 0x100000u) << 32) | l;
  const unsigned long long sx = (unsigned long long)sg << 32 | sg;
  fix_add_shifted(a, (long long)((m ^ sx) - sx), sh);
}
// The sum as a double and the rest
static __device__ __noinline__ double2 fix_value(FixSum a) {
  if (a.base == kFixNan) return make_double2(__longlong_as_double(0x7FF8000000000000LL), 0.0);
  const bool neg = a.hi < 0;
  unsigned long long hi = (unsigned long long)a.hi, lo = a.lo;
  if (neg) {
    lo = ~lo + 1;
    hi = ~hi + (lo == 0 ? 1 : 0);
  }
  if ((hi | lo) == 0) return make_double2(0.0, 0.0);
  int z = hi ? __clzll((long long)hi) : 64 + __clzll((long long)lo);
  const int ex = 127 - z - 52 + a.base - 1075;  // of the leading 53 bits' last
  if (z >= 64) {
    hi = lo;
    lo = 0;
    z -= 64;
  }
  if (z) {
    hi = hi << z | lo >> (64 - z);
    lo <<= z;
  }
  const double top = ldexp((double)(hi >> 11), ex), rest = ldexp((double)((hi & 0x7FF) << 42 | lo >> 22), ex - 53);
  return make_double2(neg ? -top : top, neg ? -rest : rest);
}

__global__ void __launch_bounds__(kCombineSinks* kCombineWarps, 4)
    k_combine(ForceCtx fc, const double* __restrict__ y, double* __restrict__ dydt, const double* __restrict__ part,
              FFPlan pl, TimeSpec ts, uint32_t flags) {
  static_assert(kCombineSinks == 32, "a warp finishes");
  __shared__ double sh_s[kCombineWarps][6][32];
  __shared__ long long sh_r2[kCombineWarps][32];
  __shared__ int sh_nn[kCombineWarps][32];
  __shared__ double sh_tot[3][32];
  const Classes& c = fc.cls;
  const int n = sol_sink_hi(fc);  // sinks [sink_lo, n)
  const int np = fc.npad;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = fc.sink_lo + blockIdx.x * kCombineSinks + lane;
  FixSum s[3] = {{0, 0, kFixEmpty}, {0, 0, kFixEmpty}, {0, 0, kFixEmpty}};
  long long best = __double_as_longlong(1.0e300);  // r^2 >= 0: the order of doubles is that of their bits
  int nn = -1;
  auto near = [&](long long r2, int j) {
    if (j >= 0 && (r2 < best || (r2 == best && j < nn))) {
      best = r2;
      nn = j;
    }
  };
  // partials [0, count), at(k) the first word of partial k and `stride` its
  // words' distance
  auto add = [&](int count, size_t stride, auto at) {
    for (int g = kCombineLoads * warp; g < count; g += kCombineLoads * kCombineWarps) {
      double v[kCombineLoads][PART_SLOTS];
#pragma unroll
      for (int u = 0; u < kCombineLoads; ++u) {
        const double* p = at(min(g + u, count - 1));
#pragma unroll
        for (int k = 0; k < PART_SLOTS; ++k) v[u][k] = p[k * stride];
      }
#pragma unroll
      for (int u = 0; u < kCombineLoads; ++u) {
        if (g + u >= count) break;
#pragma unroll
        for (int k = 0; k < 3; ++k) fix_add(s[k], v[u][PAX + k]);
        near(__double_as_longlong(v[u][PR2]), (int)__double_as_longlong(v[u][PIDX]));
      }
    }
  };
  if (i < n && i > 0) {
    const int B = i / pl.block;
    if (B < pl.nb) {
      const double* pj = part + pl.o_j + (i - B * pl.block);  // as a source of the blocks below
      add(B, pl.block, [&](int I) { return pj + sym_pair_index(I, B, pl.nb) * PART_SLOTS * pl.block; });
      const int first = B / pl.per;  // as a sink of its own block's chunks
      const double* pi = part + pl.o_i + (size_t)first * PART_SLOTS * np + i;
      add(pl.chunks - first, np, [&](int k) { return pi + (size_t)k * PART_SLOTS * np; });
    } else {
      add(pl.n2, np, [&](int k) { return part + pl.o_2 + (size_t)k * PART_SLOTS * np + i; });
    }
    add(pl.n1, np, [&](int k) { return part + pl.o_1 + (size_t)k * PART_SLOTS * np + i; });
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double2 d = fix_value(s[k]);
    sh_s[warp][k][lane] = d.x;
    sh_s[warp][3 + k][lane] = d.y;
  }
  sh_r2[warp][lane] = best;
  sh_nn[warp][lane] = nn;
  __syncthreads();
  if (warp < 3) {
    double t = sh_s[0][warp][lane], l = sh_s[0][3 + warp][lane];
#pragma unroll
    for (int w = 1; w < kCombineWarps; ++w) {
      add_ordered(t, l, sh_s[w][warp][lane]);
      l += sh_s[w][3 + warp][lane];
    }
    sh_tot[warp][lane] = t + l;
  }
  __syncthreads();
  if (warp > 0 || i >= n) return;
  double* out = dydt + 6 * i;
  if (i == 0) {
    for (int k = 0; k < 6; ++k) out[k] = 0.0;
    fc.nn_idx[0] = -1;
    fc.nn_dist[0] = 0.0;
    return;
  }
#pragma unroll
  for (int w = 1; w < kCombineWarps; ++w) near(sh_r2[w][lane], sh_nn[w][lane]);
  const double* yv = y + 6 * i;
  const int ns = (fc.type[i] <= SOL_PROTO_PLANET) ? c.nm + c.n_spl : c.nm;
  const double mu = SOL_GAUSS2 * (fc.mass[0] + fc.mass[i]);
  const double rm3i = fc.rm3[i];
  const double xi = yv[0], yi = yv[1], zi = yv[2];
  double a[3];
  a[0] = -mu * rm3i * xi;
  a[1] = -mu * rm3i * yi;
  a[2] = -mu * rm3i * zi;
  const double* S = fc.ind_sum + ((fc.type[i] <= SOL_PROTO_PLANET) ? 3 : 0);
  const double* tab = fc.src;
  double own[3] = {0.0, 0.0, 0.0};
  if (i < ns) {
    const double gmi = tab[SGM * np + i];
    own[0] = gmi * tab[SPX * np + i];
    own[1] = gmi * tab[SPY * np + i];
    own[2] = gmi * tab[SPZ * np + i];
  }
  a[0] += sh_tot[0][lane] - (S[0] - own[0]);
  a[1] += sh_tot[1][lane] - (S[1] - own[1]);
  a[2] += sh_tot[2][lane] - (S[2] - own[2]);
  if (nn >= 0) {
    // the reference's rij for this j (Acceleration.cpp:301-305), bit for bit
    const double xij = y[6 * nn + 0] - xi, yij = y[6 * nn + 1] - yi, zij = y[6 * nn + 2] - zi;
    const double rij = __dsqrt_rn(xij * xij + yij * yij + zij * zij);
    if (rij < 1.0e10) {
      fc.nn_idx[i] = nn;
      fc.nn_dist[i] = rij;
    } else {
      fc.nn_idx[i] = -1;
      fc.nn_dist[i] = 0.0;
    }
  } else {
    fc.nn_idx[i] = -1;
    fc.nn_dist[i] = 0.0;
  }
  add_gas_terms(fc, i, yv, eval_time(ts), flags, a);
  out[0] = yv[3];
  out[1] = yv[4];
  out[2] = yv[5];
  out[3] = a[0];
  out[4] = a[1];
  out[5] = a[2];
}

// ---- split forms for systems of up to kFewSplitMax bodies --------------------
// The 2-D split kernel has ceil(N / 128) x ceil(N / 4096) work units, too few
// to fill the GPU below ~16,000 bodies.  Here one warp takes one sink and its
// lanes split the sources (lane l takes l, l + 32, ...): each lane
// accumulates its share in the split arithmetic (SPLIT: FP64 FMA; SPLIT_FF:
// float-float folded into compensated FP64 every kFoldRounds of its
// sources), then the warp adds the 32 partials in a fixed shuffle tree with
// compensation (deterministic) and lane 0 finishes as k_combine does.  Every
// FP64 instruction runs on full warps: on the GB300 the FP64 pipe is scarce
// and is charged per warp instruction.
constexpr int kFewSplitWarps = 8;
constexpr int kFewSplitMax = 16384;  // SPLIT: the warp-per-sink kernel up to here
constexpr int kFfMinBodies = 4096;   // SPLIT_FF: k_pairs_ff from here (below, the warp-per-sink kernel or k_pairs_sym)
constexpr int kFoldRounds = 64;

__device__ __forceinline__ void warp_two_sum(double& s, double& c) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double so = __shfl_down_sync(0xffffffffu, s, off);
    const double co = __shfl_down_sync(0xffffffffu, c, off);
    two_sum(s, c, so);
    c += co;
  }
}

template <int MODE>
__global__ void __launch_bounds__(kFewSplitWarps * 32) k_pairs_few(ForceCtx fc, const double* __restrict__ y,
                                                                   double* __restrict__ dydt, TimeSpec ts,
                                                                   uint32_t flags) {
  const Classes& c = fc.cls;
  const int n = sol_sink_hi(fc);  // sinks [sink_lo, n)
  const int np = fc.npad;
  const int lane = threadIdx.x & 31;
  const int i = fc.sink_lo + blockIdx.x * kFewSplitWarps + (threadIdx.x >> 5);
  if (i >= n) return;  // whole warps leave together
  const int ns = (i >= 1) ? ((fc.type[i] <= SOL_PROTO_PLANET) ? c.nm + c.n_spl : c.nm) : 0;
  const double xi = y[6 * i + 0], yi = y[6 * i + 1], zi = y[6 * i + 2];
  const double* sx = fc.src + (size_t)SX * np;
  const double* sy = fc.src + (size_t)SY * np;
  const double* sz = fc.src + (size_t)SZ * np;
  double ax = 0.0, ay = 0.0, az = 0.0, cx = 0.0, cy = 0.0, cz = 0.0;
  double r2best = 1.0e300;  // this lane's first minimum of r^2 (ascending j)
  int nn = -1;
  if constexpr (MODE == SOL_PRECISION_SPLIT) {
    const double* sg = fc.src + (size_t)SGM * np;
    long long r2b = __double_as_longlong(1.0e20);
#pragma unroll 4
    for (int j = lane; j < ns; j += 32) {
      const double dx = sx[j] - xi, dy = sy[j] - yi, dz = sz[j] - zi;
      const double r2 = __fma_rn(dx, dx, __fma_rn(dy, dy, dz * dz));
      const double gm = (j >= 1 && j != i) ? sg[j] : 0.0;  // the sink itself and the central body: 0
      const double sc = split_gm_rinv3(r2, gm);
      ax = __fma_rn(sc, dx, ax);
      ay = __fma_rn(sc, dy, ay);
      az = __fma_rn(sc, dz, az);
      const long long rb = __double_as_longlong(r2);
      const bool better = (rb < r2b) & (j >= 1) & (j != i);
      r2b = better ? rb : r2b;
      nn = better ? j : nn;
    }
    if (nn >= 0) r2best = __longlong_as_double(r2b);
  } else {
    const float2* sg = reinterpret_cast<const float2*>(fc.src + (size_t)SGF * np);
    FFAcc A;
#pragma unroll
    for (int k = 0; k < 3; ++k) A.h[k] = A.l[k] = 0.0f;
    double fx = 0.0, fy = 0.0, fz = 0.0;  // the FP64 branch of very close pairs
    float mh = 1.0e20f, ml = 0.0f;
    int round = 0;
#pragma unroll 2
    for (int j = lane; j < ns; j += 32) {
      const float2 g = (j >= 1) ? sg[j] : make_float2(0.0f, 0.0f);  // the sink itself contributes 0 * d = 0
      float r2h, r2l;
      ff_pair_accumulate(sx[j] - xi, sy[j] - yi, sz[j] - zi, g, A, fx, fy, fz, r2h, r2l);
      const bool better = ((r2h < mh) | ((r2h == mh) & (r2l < ml))) & (j >= 1) & (j != i);
      mh = better ? r2h : mh;
      ml = better ? r2l : ml;
      nn = better ? j : nn;
      if (++round == kFoldRounds) {
        round = 0;
        two_sum(ax, cx, (double)A.h[0] + (double)A.l[0]);
        two_sum(ay, cy, (double)A.h[1] + (double)A.l[1]);
        two_sum(az, cz, (double)A.h[2] + (double)A.l[2]);
#pragma unroll
        for (int k = 0; k < 3; ++k) A.h[k] = A.l[k] = 0.0f;
      }
    }
    // the float-float remainder and the FP64 close pairs
    two_sum(ax, cx, ((double)A.h[0] + (double)A.l[0]) + fx);
    two_sum(ay, cy, ((double)A.h[1] + (double)A.l[1]) + fy);
    two_sum(az, cz, ((double)A.h[2] + (double)A.l[2]) + fz);
    if (nn >= 0) r2best = (double)mh + (double)ml;
  }
  warp_two_sum(ax, cx);
  warp_two_sum(ay, cy);
  warp_two_sum(az, cz);
  // nearest neighbour: the smallest r^2, ties to the lower index
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const double ro = __shfl_down_sync(0xffffffffu, r2best, off);
    const int jo = __shfl_down_sync(0xffffffffu, nn, off);
    if (jo >= 0 && (nn < 0 || ro < r2best || (ro == r2best && jo < nn))) {
      r2best = ro;
      nn = jo;
    }
  }
  if (lane != 0) return;
  double* out = dydt + 6 * i;
  if (i == 0) {
    for (int k = 0; k < 6; ++k) out[k] = 0.0;
    fc.nn_idx[0] = -1;
    fc.nn_dist[0] = 0.0;
    return;
  }
  const double* yv = y + 6 * i;
  const double mu = SOL_GAUSS2 * (fc.mass[0] + fc.mass[i]);
  const double rm3i = fc.rm3[i];
  double a[3];
  a[0] = -mu * rm3i * xi;
  a[1] = -mu * rm3i * yi;
  a[2] = -mu * rm3i * zi;
  const double* S = fc.ind_sum + ((fc.type[i] <= SOL_PROTO_PLANET) ? 3 : 0);
  const double* src = fc.src;
  double own[3] = {0.0, 0.0, 0.0};
  if (i < ns) {
    const double gmi = src[SGM * np + i];
    own[0] = gmi * src[SPX * np + i];
    own[1] = gmi * src[SPY * np + i];
    own[2] = gmi * src[SPZ * np + i];
  }
  a[0] += (ax + cx) - (S[0] - own[0]);
  a[1] += (ay + cy) - (S[1] - own[1]);
  a[2] += (az + cz) - (S[2] - own[2]);
  double rij = 0.0;
  if (nn >= 0) {
    // the reference's rij for this j (Acceleration.cpp:301-305), bit for bit
    const double xij = y[6 * nn + 0] - xi, yij = y[6 * nn + 1] - yi, zij = y[6 * nn + 2] - zi;
    rij = __dsqrt_rn(xij * xij + yij * yij + zij * zij);
    if (!(rij < 1.0e10)) nn = -1;
  }
  fc.nn_idx[i] = nn;
  fc.nn_dist[i] = nn >= 0 ? rij : 0.0;
  add_gas_terms(fc, i, yv, eval_time(ts), flags, a);
  out[0] = yv[3];
  out[1] = yv[4];
  out[2] = yv[5];
  out[3] = a[0];
  out[4] = a[1];
  out[5] = a[2];
}

}  // namespace

// parts: 1 = prepass (and indirect totals), 2 = pair kernel, 3 = both.
static int device_sms(int device) {
  // per device, filled on first use; contexts of several host threads may
  // race to fill it with the same value, hence the atomic
  static std::atomic<int> sms[kMaxDevices];
  const int dev = (device >= 0 && device < kMaxDevices) ? device : 0;
  int nsm = sms[dev].load(std::memory_order_acquire);
  if (nsm == 0) {
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || nsm < 1) nsm = 152;
    sms[dev].store(nsm, std::memory_order_release);
  }
  return nsm;
}

// Sources per CTA of k_pairs_ff for nsink sinks and nsrc sources: 1 to
// kChunkTiles tiles; among the grids that give every SM at least the three
// CTAs it holds at once, the one whose busiest SM has the least work (its CTAs
// times the tiles of a CTA plus half a tile of per-CTA work), ties to the
// larger chunk; the finest chunk when no grid is that large.  Small systems
// fill the GPU, and sizes just past a whole number of CTAs per SM avoid a
// nearly empty last round.
static int ff_chunk(int device, long nsink, long nsrc) {
  const long nsm = device_sms(device), resident = 3;
  const long nb = (nsink + kSinkBlock - 1) / kSinkBlock;
  int best_ct = 1;
  double best = 1e300;
  for (int ct = kChunkTiles; ct >= 1; ct >>= 1) {
    const long ctas = nb * ((nsrc + ct * kTile - 1) / (ct * kTile));
    if (ctas < resident * nsm) continue;
    const double cost = (double)((ctas + nsm - 1) / nsm) * (ct + 0.5);
    if (cost < best) {
      best = cost;
      best_ct = ct;
    }
  }
  return best_ct * kTile;
}

// How a SPLIT_FF evaluation is divided.  k_pairs_sym takes the massive bodies
// (which attract each other) in whole blocks, the last one padded where every
// body is massive; k_pairs_ff the rest.  From kSymMin bodies on (us an
// evaluation with it and without: 1,025 bodies 65 and 52, 1,250 65 and 71, 2,049
// 67 and 99, 3,100 86 and 145, 4,096 98 and 108, 7,000 188 and 236), kSymMinMixed
// where others are left to k_pairs_ff (two launches more: 100 light bodies beside
// 6,200 massive 204 and 192, beside 8,300 295 and 340), up to kSymMax, beyond
// which the block pairs' partials (10 KB each) would pass 1.4 GB.  Small blocks are many and
// short tasks, large ones have fewer partials (us with 64, 128 and 256 bodies:
// 2,049 65, 90, 141; 10,007 339, 345, 383; 12,288 480, 459, 479; 16,384 808, 772,
// 783; 24,000 1,679, 1,605, 1,583).  One block of sources a CTA up to kSymSingle
// blocks; above, two and then four halve the sinks' partials (336 MB at 65,536
// bodies) for much the same time (24,000 bodies: 1.61 ms with one, 1.65 with
// two; 45,000: 5.36 and 5.41; 65,536: 11.17 and 11.19).
constexpr int kSymMin = 1152, kSymMinMixed = 7168, kSymMax = 131072, kSymSingle = 192;

static int sym_block(int massive) { return massive < 11000 ? 64 : massive < 20000 ? 128 : 256; }
// the bodies k_pairs_sym takes
static int sym_bodies(int n, const Classes& cls) {
  // every body massive: the last block padded; else whole tiles (k_pairs_ff goes on from one)
  const int massive = cls.nm == n ? n : cls.nm / kTile * kTile;
  return massive >= (cls.nm == n ? kSymMin : kSymMinMixed) && massive <= kSymMax ? massive : 0;
}
static void sym_shape(FFPlan& p, int block, int nb) {
  p.block = block;
  p.nb = nb;
  p.per = block < 256 || nb <= kSymSingle ? 1 : (nb <= 256 ? 2 : 4);
  p.chunks = (nb + p.per - 1) / p.per;
}
static size_t sym_doubles(const FFPlan& p, int npad) {
  return ((size_t)p.nb * (p.nb - 1) / 2 * p.block + (size_t)p.chunks * npad) * PART_SLOTS + npad;
}

// room: doubles of the partials' buffer (k_pairs_ff alone where the block pairs' do not fit)
static FFPlan ff_plan(int device, int n, const Classes& cls, int npad, size_t room, bool blocks = true) {
  FFPlan p;
  const int massive = blocks ? sym_bodies(n, cls) : 0;
  if (massive > 0) {
    const int block = sym_block(massive);
    sym_shape(p, block, (massive + block - 1) / block);
    p.from = p.nb * block;
  }
  const int sources = cls.nm + cls.n_spl;
  if (p.nb == 0) {
    p.chunk1 = ff_chunk(device, n, n);
    p.n1 = (n + p.chunk1 - 1) / p.chunk1;
  } else if (p.from < n) {
    if (sources > p.from) {
      p.chunk1 = ff_chunk(device, n, sources - p.from);
      p.n1 = (sources - p.from + p.chunk1 - 1) / p.chunk1;
    }
    p.chunk2 = ff_chunk(device, n - p.from, p.from);
    p.n2 = (p.from + p.chunk2 - 1) / p.chunk2;
  }
  size_t o = 0;
  auto take = [&](size_t doubles) {
    const size_t at = o;
    o += doubles;
    return at;
  };
  p.o_j = take((size_t)p.nb * (p.nb > 0 ? p.nb - 1 : 0) / 2 * p.block * PART_SLOTS);
  p.o_i = take((size_t)p.chunks * PART_SLOTS * npad);
  p.o_1 = take((size_t)p.n1 * PART_SLOTS * npad);
  p.o_2 = take((size_t)p.n2 * PART_SLOTS * npad);
  p.o_bound = take(p.nb > 0 ? npad : 0);
  if (o > room && p.nb > 0) return ff_plan(device, n, cls, npad, room, false);
  return p;
}

template <int BLOCK>
static int launch_sym(sol_ctx* c, const ForceCtx& fc, const double* d_y, const FFPlan& p, const float* bound) {
  static std::atomic<int> ready[kMaxDevices];  // the kernel's shared-memory size is allowed
  const int dev = (c->device >= 0 && c->device < kMaxDevices) ? c->device : 0;
  if (!ready[dev].load(std::memory_order_acquire)) {
    SOL_CUDA(cudaFuncSetAttribute(k_pairs_sym<BLOCK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sizeof(SymShared<BLOCK>)));
    ready[dev].store(1, std::memory_order_release);
  }
  const int tasks = sym_tasks_above(p.chunks, p.per) + p.nb;
  k_pairs_sym<BLOCK><<<tasks, sym_threads(BLOCK), sizeof(SymShared<BLOCK>), c->stream>>>(
      fc, d_y, c->d_part + p.o_i, c->d_part + p.o_j, bound, p.nb, p.per);
  SOL_LAUNCHED();
  return SOL_OK;
}

// Sinks per CTA of k_gravity_ac_ref: the CTAs spread over the SMs, so an SM's
// work is its CTAs (the busiest SM's, k) times what one costs a source: spc
// sinks' pairs and the summing warp's, which cost about 1.9 sinks (16 cycles of
// the FP64 pipe against ~9 a sink).  For each k the fewest sinks that reach it.
// (21 sinks with two summing and 14 producing warps, one such CTA an SM at 80
// registers: 10,007 bodies 3.28 ms for 2.79, 65,536 121 for 106; two at 64: 2.89
// and 106.)
static int ref_sinks(int nsink, int nsm) {
  double best = 1e300;
  int spc = 1;
  const long k0 = ((long)nsink + (long)nsm * kRefMaxSinks - 1) / ((long)nsm * kRefMaxSinks);
  for (long k = k0; k < k0 + 3; ++k) {
    const int sp = (int)(((long)nsink + k * nsm - 1) / (k * nsm));
    const double cost = (double)k * (sp + 1.9);
    if (cost < best) {
      best = cost;
      spc = sp;
    }
  }
  return spc;
}

// Whether k_gravity_ac_ref is the faster one for ns sources (k_gravity_ac: a
// thread a sink).  The thread's chain is 0.92 us a source until the sinks fill
// the FP64 pipe (0.041 ns a pair); the other takes 4.2 us a tile of 64 sources
// and, per sink, 1.7 ns a tile and 1.5 besides, whether the tile is full or not.
// Measured (an evaluation, us, thread / tiles): 12 sources and 1,000 sinks 20 /
// 16, 5,000 sinks 23 / 33; 64 and 20,000 110 / 88; 128 and 200 sinks 126 / 17,
// 100,000 sinks 612 / 425; 3 sources and 256 sinks 11 / 14.
static bool ref_pays(int ns, int nsink) {
  const double tiles = (ns + kRefTile - 1) / kRefTile;
  const double by_thread = 9.0 + ns * std::max(0.92, 0.6 + 4.1e-5 * nsink);
  const double by_tiles = 8.0 + 4.2 * tiles + 1.0e-3 * nsink * (1.5 + 1.7 * tiles);
  return ns >= 224 || by_thread > 1.15 * by_tiles;
}

static int launch_ref(sol_ctx* c, const ForceCtx& fc, const double* d_y, double* d_dydt, TimeSpec ts, uint32_t flags,
                      int nsink) {
  // per device: the SM count, once the kernel's shared-memory size is
  // allowed (contexts of several host threads may race to set it: the same
  // values, hence an atomic published after the attribute calls)
  static std::atomic<int> ref_sms[kMaxDevices];
  const int dev = (c->device >= 0 && c->device < kMaxDevices) ? c->device : 0;
  int nsm = ref_sms[dev].load(std::memory_order_acquire);
  if (nsm == 0) {
    SOL_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device));
    SOL_CUDA(cudaFuncSetAttribute(k_gravity_ac_ref, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)ref_smem(kRefMaxSinks)));
    ref_sms[dev].store(nsm, std::memory_order_release);
  }
  const int spc = ref_sinks(nsink, nsm);
  k_gravity_ac_ref<<<(nsink + spc - 1) / spc, (1 + kRefProducers) * 32, ref_smem(spc), c->stream>>>(fc, d_y, d_dydt, ts,
                                                                                                  flags, spc);
  SOL_LAUNCHED();
  return SOL_OK;
}

// The sinks of fc's range [sink_lo, sol_sink_hi) (every body by default);
// the prepass always covers every body (the sources).
static int force_launch(sol_ctx* c, const ForceCtx& fc, const double* d_y, double* d_dydt, TimeSpec ts,
                        uint32_t flags, int parts, int* d_clear) {
  const int nsink = sol_sink_hi(fc) - fc.sink_lo;
  const int split = (c->precision != SOL_PRECISION_FP64 && !c->barycentric) ? 1 : 0;
  // SPLIT_FF systems beyond the warp-per-sink kernel run on the float table
  const int ff2d = split && c->precision == SOL_PRECISION_SPLIT_FF && sol_force_uses_chunk_partials(c, c->precision);
  FFPlan plan;
  float* bound = nullptr;
  if (split && sol_force_uses_chunk_partials(c, c->precision)) {
    if (!c->d_part) {
      sol_set_error("split precision selected without sol_set_precision");
      return SOL_ERR_STATE;
    }
    if (ff2d) {
      plan = ff_plan(c->device, c->n, c->cls, fc.npad, c->part_doubles);
      if (plan.nb > 0) bound = reinterpret_cast<float*>(c->d_part + plan.o_bound);
    }
  }
  if (parts & 1) {
    const int nb_pre = (fc.npad + kPrepassBlock - 1) / kPrepassBlock;
    k_prepass<<<nb_pre, kPrepassBlock, 0, c->stream>>>(fc, d_y, split, ff2d, d_clear);
    SOL_LAUNCHED();
    if (split && !c->barycentric && !ff2d) {
      k_ind_reduce<<<1, 256, 0, c->stream>>>(fc);
      SOL_LAUNCHED();
    }
    if (ff2d) {
      k_split_table<<<nb_pre, kPrepassBlock, 0, c->stream>>>(fc, d_y, bound);
      SOL_LAUNCHED();
    }
  }
  if (!(parts & 2) || nsink <= 0) return SOL_OK;
  const int nb = (nsink + kSinkBlock - 1) / kSinkBlock;
  if (c->barycentric) {
    k_gravity_bc<<<nb, kSinkBlock, 0, c->stream>>>(fc, d_y, d_dydt, ts, flags);
    SOL_LAUNCHED();
    return SOL_OK;
  }
  if (!split && ref_pays(c->cls.nm + c->cls.n_spl, nsink)) return launch_ref(c, fc, d_y, d_dydt, ts, flags, nsink);
  if (split && !sol_force_uses_chunk_partials(c, c->precision)) {
    const int grid = (nsink + kFewSplitWarps - 1) / kFewSplitWarps;
    if (c->precision == SOL_PRECISION_SPLIT_FF)
      k_pairs_few<SOL_PRECISION_SPLIT_FF><<<grid, kFewSplitWarps * 32, 0, c->stream>>>(fc, d_y, d_dydt, ts, flags);
    else
      k_pairs_few<SOL_PRECISION_SPLIT><<<grid, kFewSplitWarps * 32, 0, c->stream>>>(fc, d_y, d_dydt, ts, flags);
    SOL_LAUNCHED();
    return SOL_OK;
  }
  if (split) {
    int* status = &c->d_ctrl->dev_status;
    if (c->precision == SOL_PRECISION_SPLIT_FF) {
      if (plan.nb > 0) {
        const int tiles = (plan.from + kTile - 1) / kTile;
        const dim3 grid_bound(tiles, (tiles < kBoundBlocks ? tiles : kBoundBlocks) * kBoundParts);
        k_near_bound<<<grid_bound, kTile, 0, c->stream>>>(fc, bound, tiles);
        SOL_LAUNCHED();
        const int r = plan.block == 64    ? launch_sym<64>(c, fc, d_y, plan, bound)
                      : plan.block == 128 ? launch_sym<128>(c, fc, d_y, plan, bound)
                                          : launch_sym<256>(c, fc, d_y, plan, bound);
        if (r != SOL_OK) return r;
      }
      if (plan.n1 > 0) {
        k_pairs_ff<<<dim3(nb, plan.n1), kSinkBlock, 0, c->stream>>>(fc, d_y, c->d_part + plan.o_1, status,
                                                                    plan.chunk1, plan.from, c->n);
        SOL_LAUNCHED();
      }
      if (plan.n2 > 0 && sol_sink_hi(fc) > plan.from) {
        ForceCtx rest = fc;
        rest.sink_lo = fc.sink_lo > plan.from ? fc.sink_lo : plan.from;
        rest.sink_hi = sol_sink_hi(fc);
        const int nb2 = (rest.sink_hi - rest.sink_lo + kSinkBlock - 1) / kSinkBlock;
        k_pairs_ff<<<dim3(nb2, plan.n2), kSinkBlock, 0, c->stream>>>(rest, d_y, c->d_part + plan.o_2, status,
                                                                     plan.chunk2, 0, plan.from);
        SOL_LAUNCHED();
      }
    } else {
      plan.chunk1 = kChunk;
      plan.n1 = (c->n + kChunk - 1) / kChunk;
      k_pairs<SOL_PRECISION_SPLIT><<<dim3(nb, plan.n1), kSinkBlock, 0, c->stream>>>(fc, d_y, c->d_part, status, kChunk);
      SOL_LAUNCHED();
    }
    k_combine<<<(nsink + kCombineSinks - 1) / kCombineSinks, kCombineSinks * kCombineWarps, 0, c->stream>>>(
        fc, d_y, d_dydt, c->d_part, plan, ts, flags);
  } else {
    k_gravity_ac<SOL_PRECISION_FP64><<<nb, kSinkBlock, 0, c->stream>>>(fc, d_y, d_dydt, ts, flags,
                                                                       &c->d_ctrl->dev_status, SOL_SPIN_LIMIT, -1);
  }
  SOL_LAUNCHED();
  return SOL_OK;
}

int sol_force_launch_parts(sol_ctx* c, const double* d_y, double* d_dydt, TimeSpec ts, uint32_t flags, int parts,
                           int* d_clear) {
  return force_launch(c, c->fc, d_y, d_dydt, ts, flags, parts, d_clear);
}

int sol_force_launch(sol_ctx* c, const double* d_y, double* d_dydt, TimeSpec ts, uint32_t flags) {
  return sol_force_launch_parts(c, d_y, d_dydt, ts, flags, 3);
}

// The FP64 forms, while a launch is a part of an evaluation (beyond, k_stage's grid
// of whole warps of elements is as good).
bool sol_force_takes_stage(const sol_ctx* c) {
  return (c->precision == SOL_PRECISION_FP64 || c->barycentric) && c->n <= 16384;
}
int sol_force_launch_stage(sol_ctx* c, int k, const StageArgs& s, const double* y0, double* yt, double* d_dydt,
                           TimeSpec ts, uint32_t flags) {
  const int g = c->fc.npad / kStageBodies, b = 6 * kStageBodies;
  switch (k) {
    case 1: k_stage_prepass<1><<<g, b, 0, c->stream>>>(c->fc, y0, yt, s, c->d_ctrl); break;
    case 2: k_stage_prepass<2><<<g, b, 0, c->stream>>>(c->fc, y0, yt, s, c->d_ctrl); break;
    case 3: k_stage_prepass<3><<<g, b, 0, c->stream>>>(c->fc, y0, yt, s, c->d_ctrl); break;
    case 4: k_stage_prepass<4><<<g, b, 0, c->stream>>>(c->fc, y0, yt, s, c->d_ctrl); break;
    case 6: k_stage_prepass<6><<<g, b, 0, c->stream>>>(c->fc, y0, yt, s, c->d_ctrl); break;
    case 7: k_stage_prepass<7><<<g, b, 0, c->stream>>>(c->fc, y0, yt, s, c->d_ctrl); break;
    case 8: k_stage_prepass<8><<<g, b, 0, c->stream>>>(c->fc, y0, yt, s, c->d_ctrl); break;
    case 9: k_stage_prepass<9><<<g, b, 0, c->stream>>>(c->fc, y0, yt, s, c->d_ctrl); break;
    default: sol_set_error("stage with %d terms", k); return SOL_ERR_ARG;
  }
  SOL_LAUNCHED();
  return sol_force_launch_parts(c, yt, d_dydt, ts, flags, 2);
}

// Sinks [lo, hi) only (heliocentric contexts): a rank's block of a
// sink-partitioned system.
int sol_force_launch_sinks(sol_ctx* c, const double* d_y, double* d_dydt, TimeSpec ts, uint32_t flags, int lo,
                           int hi) {
  ForceCtx fc = c->fc;
  fc.sink_lo = lo;
  fc.sink_hi = hi;
  return force_launch(c, fc, d_y, d_dydt, ts, flags, 3, nullptr);
}

int sol_force_tile() { return kTile; }
int sol_force_src_doubles() { return kSrcDoubles; }
// Partials for either split form's 2-D kernels and, with `blocks`, for the block
// pairs of a SPLIT_FF system that k_pairs_sym serves, of this system and of every
// smaller one it can become (removed bodies): fewer blocks can have more chunks.
static size_t part_doubles(const sol_ctx* c, bool blocks) {
  const size_t np = c->npad;
  size_t most = (size_t)((c->n + kChunk - 1) / kChunk) * PART_SLOTS * np;  // SPLIT
  // k_pairs_ff alone: the number of chunks changes at whole sink blocks only
  for (int n = (c->n + kSinkBlock - 1) / kSinkBlock * kSinkBlock; n >= 1; n -= kSinkBlock) {
    const int ch = ff_chunk(c->device, n, n);
    const size_t d = (size_t)((n + ch - 1) / ch) * PART_SLOTS * np;
    if (d > most) most = d;
  }
  if (!blocks || sym_bodies(c->n, c->cls) == 0) return most;
  size_t sym = 0;
  for (int m = 64; m <= c->cls.nm + 255 && m <= kSymMax + 255; m += 64)
    for (int block = 64; block <= 256; block *= 2)
      if (m % block == 0 && m >= kSymMin && (sym_block(m) == block || sym_block(m - block + 1) == block)) {
        FFPlan p;
        sym_shape(p, block, m / block);
        const size_t d = sym_doubles(p, c->npad);
        if (d > sym) sym = d;
      }
  if (sym > 0 && c->cls.nm < c->n)  // k_pairs_ff on the rest, in chunks of one tile at the least
    sym += ((size_t)(kTile + c->cls.n_spl + kTile - 1) / kTile + (c->cls.nm + kTile - 1) / kTile) * PART_SLOTS * np;
  return sym > most ? sym : most;
}
// The partials' buffer for a split precision (not cleared: what is read has been
// written), kept where it is large enough; without the block pairs' where they do
// not fit.  A larger one may become necessary with another precision, or when the
// last light body is removed; captured graphs hold the old one's address.
int sol_force_alloc_parts(sol_ctx* c, int precision) {
  for (bool blocks : {true, false}) {
    if (blocks && precision != SOL_PRECISION_SPLIT_FF) continue;
    const size_t doubles = part_doubles(c, blocks);
    if (c->d_part && c->part_doubles >= doubles) return SOL_OK;
    double* part = nullptr;
    if (cudaMalloc((void**)&part, sizeof(double) * doubles) != cudaSuccess) {
      cudaGetLastError();
      continue;
    }
    if (c->d_part) {
      for (DriverGraph& G : c->graphs) sol_graph_release(G);
      SOL_CUDA(cudaStreamSynchronize(c->stream));
      cudaFree(c->d_part);
    }
    c->d_part = part;
    c->part_doubles = doubles;
    return SOL_OK;
  }
  sol_set_error("cudaMalloc of the split partials failed");
  return SOL_ERR_NOMEM;
}
// whether the split forms of this system run the 2-D kernel (and need its
// chunk partials); the same test as the dispatch in sol_force_launch_parts
int sol_force_uses_chunk_partials(const sol_ctx* c, int precision) {
  const int few_max = precision == SOL_PRECISION_SPLIT_FF ? kFfMinBodies - 1 : kFewSplitMax;
  if (precision == SOL_PRECISION_SPLIT_FF && sym_bodies(c->n, c->cls) > 0) return 1;
  return !(c->n <= few_max && c->cls.nm + c->cls.n_spl >= kTile);
}
int sol_force_prepass_blocks(int npad) { return (npad + kPrepassBlock - 1) / kPrepassBlock; }

// ---- caller-allocated variant ---------------------------------------------------
// sol_gravity_noalloc serves callers that must not allocate device memory
// themselves: code running under someone else's memory manager (a host
// framework that owns every device byte, a fixed-budget plugin) or in a
// real-time loop where an allocation would stall.  Its scratch -- the
// structure-of-arrays source table, the per-block indirect-term partials and
// a status word -- is this file-scope array, sized for at most
// kNoAllocMaxBodies bodies (about 1 MiB), present on every device that loads
// the library until the process exits.
namespace {
constexpr int kNoAllocMaxBodies = 16384;
constexpr int kNoAllocPrepassBlocks = kNoAllocMaxBodies / kPrepassBlock;
constexpr size_t kNoAllocSrc = (size_t)SRC_ARRAYS * kNoAllocMaxBodies;
constexpr size_t kNoAllocPart = 6 * (size_t)kNoAllocPrepassBlocks;
constexpr size_t kNoAllocDoubles = kNoAllocSrc + kNoAllocPart + 8 /* sums */ + 8 /* status */;
static_assert(kTile == 256 && kTile % kSinkBlock == 0, "tiles are whole blocks of every size, and whole sink blocks");
static_assert(kNoAllocMaxBodies % kTile == 0, "scratch must hold whole tiles");
}  // namespace

static __device__ __align__(256) double g_noalloc_scratch[kNoAllocDoubles];

namespace {
std::mutex g_noalloc_mu;
double* g_noalloc_addr[64];  // device address of g_noalloc_scratch, per device ordinal
// failure-path test hook (sol_set_wait_test with no context): the mbarrier
// spin limit of the next calls (0: SOL_SPIN_LIMIT) and a tile never copied
std::atomic<unsigned> g_noalloc_spin{0};
std::atomic<int> g_noalloc_withhold{-1};

// Host code cannot use g_noalloc_scratch as a device address: resolve it once
// per device, with that device current.  The same first call loads every
// kernel instance this entry point launches (with CUDA's lazy module loading
// a kernel's first launch would otherwise load it then), so later calls --
// of either precision -- do no loading work.
int noalloc_scratch(double** out) {
  int dev = 0;
  SOL_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    sol_set_error("device ordinal %d out of range", dev);
    return SOL_ERR_ARG;
  }
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return sol_cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)", __FILE__, __LINE__);
    cudaFuncAttributes fa;
    SOL_CUDA(cudaFuncGetAttributes(&fa, k_prepass));
    SOL_CUDA(cudaFuncGetAttributes(&fa, k_ind_reduce));
    SOL_CUDA(cudaFuncGetAttributes(&fa, k_gravity_ac<SOL_PRECISION_FP64>));
    SOL_CUDA(cudaFuncGetAttributes(&fa, k_gravity_ac<SOL_PRECISION_SPLIT>));
    g_noalloc_addr[dev] = (double*)p;
  }
  *out = g_noalloc_addr[dev];
  return SOL_OK;
}

int* noalloc_status_word(double* scratch) { return (int*)(scratch + kNoAllocSrc + kNoAllocPart + 8); }
}  // namespace

void sol_noalloc_wait_test(unsigned spin_limit, int withhold_tile) {
  g_noalloc_spin.store(spin_limit);
  g_noalloc_withhold.store(withhold_tile);
}

extern "C" int sol_gravity_noalloc_status(void* stream, int32_t* status) {
  double* scratch = nullptr;
  int rc = noalloc_scratch(&scratch);
  if (rc != SOL_OK) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  int word = 0;
  SOL_CUDA(cudaMemcpyAsync(&word, noalloc_status_word(scratch), sizeof(int), cudaMemcpyDeviceToHost, st));
  SOL_CUDA(cudaStreamSynchronize(st));
  if (status) *status = word;
  if (word & SOL_DEV_TIMEOUT) {
    sol_set_error("sol_gravity_noalloc: a bounded device wait ran out; the outputs of that call are incomplete");
    return SOL_ERR_TIMEOUT;
  }
  return SOL_OK;
}

extern "C" int sol_gravity_noalloc(const sol_nbodies* counts, const int32_t* d_type, const double* d_mass,
                                   const double* d_y, double* d_dydt, double* d_rm3, int32_t* d_nn_idx,
                                   double* d_nn_dist, int32_t precision, void* stream) {
  if (!counts || !d_type || !d_mass || !d_y || !d_dydt || !d_rm3 || !d_nn_idx || !d_nn_dist) {
    sol_set_error("sol_gravity_noalloc: null argument");
    return SOL_ERR_ARG;
  }
  const sol_nbodies& k = *counts;
  const int parts[7] = {k.central_body, k.giant_planet, k.rocky_planet, k.proto_planet, k.super_planetesimal,
                        k.planetesimal, k.test_particle};
  long long n = 0;
  for (int q = 0; q < 7; ++q) {
    if (parts[q] < 0) {
      sol_set_error("sol_gravity_noalloc: negative body count");
      return SOL_ERR_ARG;
    }
    n += parts[q];
  }
  if (k.central_body != 1) {
    sol_set_error("sol_gravity_noalloc: need exactly one central body");
    return SOL_ERR_ARG;
  }
  if (n > kNoAllocMaxBodies) {
    sol_set_error("sol_gravity_noalloc: %lld bodies exceed the fixed scratch capacity of %d bodies", n,
                  kNoAllocMaxBodies);
    return SOL_ERR_ARG;
  }
  if (precision != SOL_PRECISION_FP64 && precision != SOL_PRECISION_SPLIT) {
    sol_set_error("sol_gravity_noalloc: unknown precision %d", precision);
    return SOL_ERR_ARG;
  }
  double* scratch = nullptr;
  int rc = noalloc_scratch(&scratch);
  if (rc != SOL_OK) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  ForceCtx fc;
  memset(&fc, 0, sizeof(fc));
  fc.cls.n = (int)n;
  fc.cls.n_central = k.central_body;
  fc.cls.n_giant = k.giant_planet;
  fc.cls.n_rocky = k.rocky_planet;
  fc.cls.n_proto = k.proto_planet;
  fc.cls.n_spl = k.super_planetesimal;
  fc.cls.n_pl = k.planetesimal;
  fc.cls.nm = k.central_body + k.giant_planet + k.rocky_planet + k.proto_planet;
  fc.npad = (int)(((n + kTile - 1) / kTile) * kTile);
  fc.precision = precision;
  fc.type = d_type;
  fc.mass = d_mass;
  fc.rm3 = d_rm3;
  fc.nn_idx = d_nn_idx;
  fc.nn_dist = d_nn_dist;
  fc.src = scratch;  // SRC_ARRAYS x npad doubles at stride npad
  fc.ind_part = scratch + kNoAllocSrc;
  fc.ind_sum = scratch + kNoAllocSrc + kNoAllocPart;
  fc.n_ind_blocks = (fc.npad + kPrepassBlock - 1) / kPrepassBlock;
  int* status = noalloc_status_word(scratch);
  // The array keeps the previous call's contents: the source table and the
  // partials are rewritten in full below, the status word must start at zero
  // (the prepass clears it).
  // rm3[0] (the central body) is never computed and reads as 0, as in the
  // reference, whose rm3 array starts zeroed (Acceleration.cpp:65-69).
  SOL_CUDA(cudaMemsetAsync(d_rm3, 0, sizeof(double), st));
  const int split = precision == SOL_PRECISION_SPLIT;
  k_prepass<<<fc.n_ind_blocks, kPrepassBlock, 0, st>>>(fc, d_y, split, 0, status);
  SOL_LAUNCHED();
  if (split) {
    k_ind_reduce<<<1, 256, 0, st>>>(fc);
    SOL_LAUNCHED();
  }
  TimeSpec ts{nullptr, nullptr, 0.0, 0.0};
  const int nb = (int)((n + kSinkBlock - 1) / kSinkBlock);
  const unsigned spin_hook = g_noalloc_spin.load();
  const unsigned spin = spin_hook ? spin_hook : SOL_SPIN_LIMIT;
  const int withhold = g_noalloc_withhold.load();
  if (split)
    k_gravity_ac<SOL_PRECISION_SPLIT><<<nb, kSinkBlock, 0, st>>>(fc, d_y, d_dydt, ts, 0u, status, spin, withhold);
  else
    k_gravity_ac<SOL_PRECISION_FP64><<<nb, kSinkBlock, 0, st>>>(fc, d_y, d_dydt, ts, 0u, status, spin, withhold);
  SOL_LAUNCHED();
  return SOL_OK;
}
