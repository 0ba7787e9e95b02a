// Discrete adjoint of the fixed-step RungeKuttaFehlberg78 integration
// (RungeKuttaFehlberg78::Step at constant h, y_{n+1} = the 7th-order result,
// Solaris/RungeKuttaFehlberg78.cpp:147-250) with GravityAC forces
// (Solaris/Acceleration.cpp:248-329).
//
// Forward: n fixed steps on the device, the state stored every K steps, and of
// the last K (or fewer) steps, where the backward pass begins, every stage
// state Y_k (k = 0..10).  Backward, one segment of K steps at a time from the
// last: the segment (but for the last one) is recomputed from its checkpoint
// with its stage states kept; then, step by step from the last, the stage adjoints
//   w_k = h b_k lambda + h sum_{j>k} a_jk nu_j,   nu_k = J(Y_k)^T w_k
// and lambda_n = lambda_{n+1} + sum_k nu_k, with the mass gradient
// accumulated from the same w_k.  Stages 11 and 12 only enter the error
// estimate, so their adjoints are zero.  J^T w is a hand-written
// vector-Jacobian product of the pair force (block pairs, or a CTA per body).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "sol_pair.cuh"

int sol_rkf78_stages(sol_ctx* c, const double* d_y0, double* d_y, double* const* stage_out);

namespace {

constexpr int kBlock = 256;
constexpr int kVjpThreads = 128;  // threads of k_vjp: one body's pairs
constexpr int kVjpWarps = kVjpThreads / 32;
constexpr int kPreBodies = 32;    // bodies per CTA of k_vjp_cotangent, a lane each in its sums: 192 elements
constexpr int kAdjStages = 11;  // stages 0..10 reach y_{n+1}

// RKF78 tableau (RungeKuttaFehlberg78.cpp:41-56): a[j][k] and the weights b
const double kA[13][13] = {
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
    {3.0 / 205.0, 0, 0, 0, 0, -6.0 / 41.0, -3.0 / 205.0, -3.0 / 41.0, 3.0 / 41.0, 6.0 / 41.0, 0},
    {-1777.0 / 4100.0, 0, 0, -341.0 / 164.0, 4496.0 / 1025.0, -289.0 / 82.0, 2193.0 / 4100.0, 51.0 / 82.0,
     33.0 / 164.0, 12.0 / 41.0, 0, 1.0}};
const double kB[13] = {41.0 / 840.0, 0, 0, 0, 0, 34.0 / 105.0, 9.0 / 35.0, 9.0 / 35.0, 9.0 / 280.0, 9.0 / 280.0,
                       41.0 / 840.0, 0, 0};

struct Lin {
  const double* v[kAdjStages + 1];
  double c[kAdjStages + 1];
  int k;
};

// out = base + scale * sum_i c_i v_i (base may be null)
__global__ void k_lincomb(int nv, double* __restrict__ out, const double* __restrict__ base, double scale, Lin L) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nv; e += gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int i = 0; i < L.k; ++i) acc = __fma_rn(L.c[i], L.v[i][e], acc);
    out[e] = base ? __fma_rn(scale, acc, base[e]) : scale * acc;
  }
}

// The stage's cotangent w = h b_k lambda + h sum_j a_jk nu_j (L, scaled by h),
// the structure-of-arrays view of (state, cotangent) that the pair kernels
// stream -- x, y, z, m, wx, wy, wz -- and this CTA's sums of the cotangent's
// velocity part over its bodies: [0..2] those with index >= 1, [3..5] those
// below nm.  One thread per element, kPreBodies bodies per CTA; sw: 6 kPreBodies words.
__device__ __forceinline__ void cotangent(int n, int nm, const double* __restrict__ Y, const double* __restrict__ mass,
                                          double h, const Lin& L, double* __restrict__ w, double* __restrict__ soa,
                                          double* __restrict__ wsum, double* sw) {
  const int i0 = blockIdx.x * kPreBodies;
  const int b = threadIdx.x / 6, k = threadIdx.x - 6 * b;
  const int i = i0 + b;
  if (b < kPreBodies) {
    double acc = 0.0;
    if (i < n) {
      const size_t e = 6 * (size_t)i + k;
      double v[kAdjStages + 1];  // every load in flight before the first product
#pragma unroll
      for (int q = 0; q <= kAdjStages; ++q) v[q] = q < L.k ? L.v[q][e] : 0.0;
#pragma unroll
      for (int q = 0; q <= kAdjStages; ++q)
        if (q < L.k) acc = __fma_rn(L.c[q], v[q], acc);
      acc = h * acc;
      w[e] = acc;
      if (k < 3) {
        soa[(size_t)k * n + i] = Y[e];
        if (k == 0) soa[(size_t)3 * n + i] = mass[i];
      } else {
        soa[(size_t)(k + 1) * n + i] = acc;
      }
    }
    sw[threadIdx.x] = acc;
  }
  __syncthreads();
  const int sum = threadIdx.x >> 5, lane = threadIdx.x & 31;  // a warp per sum
  if (sum < 6) {
    const int j = i0 + lane;
    double t = j >= 1 && j < (sum < 3 ? n : nm) ? sw[6 * lane + 3 + sum % 3] : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) wsum[6 * (size_t)blockIdx.x + sum] = t;
  }
}
__global__ void __launch_bounds__(6 * kPreBodies) k_vjp_cotangent(int n, int nm, const double* __restrict__ Y,
                                                                  const double* __restrict__ mass, double h, Lin L,
                                                                  double* __restrict__ w, double* __restrict__ soa,
                                                                  double* __restrict__ wsum) {
  __shared__ double sw[6 * kPreBodies];
  cotangent(n, nm, Y, mass, h, L, w, soa, wsum, sw);
}

// r^-3 and r^-2 of r^2: the FP32 seed y of 1/r, its square (exact) and cube
// from the integer pipe, and one FP64 residual e = 1 - r^2 y^2 (|e| < 2^-20):
// r^-3 = y^3 (1 + 3/2 e + 15/8 e^2), r^-2 = y^2 (1 + e + e^2), both within
// about an ulp, for four FP64 instructions.  r^2 outside [2^-100, 2^100]
// (coincident bodies, infinities, NaN) takes rsqrt.
static __device__ __noinline__ double2 rinv32_slow(double r2) {
  const double r = rsqrt(r2);
  return make_double2(r * r * r, r * r);
}
__device__ __forceinline__ void rinv32(double r2, double& rm3, double& rm2) {
  double u, y3;
  sol_seed_square_cube(sol_rsqrt_seed(r2), u, y3);
  const double e = __fma_rn(-r2, u, 1.0);
  rm3 = __fma_rn(y3, sol_split_t(e), y3);
  rm2 = __fma_rn(u, __fma_rn(e, e, e), u);
  const unsigned ex = ((unsigned)__double2hiint(r2)) >> 20;
  if (ex - 923u >= 200u) {
    const double2 v = rinv32_slow(r2);
    rm3 = v.x;
    rm2 = v.y;
  }
}

// Body k's part of nu, dm and d/d m_0 from its sums over the other bodies (tot)
// and over the cotangents of its sinks (Wv), r, w_v of the body in x and wk:
// part 0 to 2, a component of nu; 3, the masses.
__device__ __forceinline__ void vjp_finish_body(int part, int k, const double* x, const double* wk, double mk, double m0,
                                                const double* tot, const double* Wv, const double* w, double* nu,
                                                double* __restrict__ dm, double* __restrict__ m0_part) {
  const double G = SOL_GAUSS2;
  const double r2 = __fma_rn(x[0], x[0], __fma_rn(x[1], x[1], x[2] * x[2]));
  double rm3, rm2;
  rinv32(r2, rm3, rm2);
  if (part < 3) {
    const double xc = part == 0 ? x[0] : part == 1 ? x[1] : x[2], wc = part == 0 ? wk[0] : part == 1 ? wk[1] : wk[2];
    const double tc = part == 0 ? tot[0] : part == 1 ? tot[1] : tot[2], sc = part == 0 ? tot[4] : part == 1 ? tot[5] : tot[6];
    const double g = __fma_rn(mk, tc, __fma_rn(-wc, tot[3], -3.0 * sc));
    // Kepler term -G (m0 + m_k) r_k / |r_k|^3 and indirect term -G m_k r_k / |r_k|^3 (for the sinks of k):
    // T(r) v = v / r^3 - 3 r (r . v) / r^5
    const double mu = -(m0 + mk);
    const double vx = __fma_rn(mu, wk[0], -mk * Wv[0]), vy = __fma_rn(mu, wk[1], -mk * Wv[1]),
                 vz = __fma_rn(mu, wk[2], -mk * Wv[2]);
    const double dv = __fma_rn(x[0], vx, __fma_rn(x[1], vy, x[2] * vz));
    const double s = 3.0 * (rm3 * rm2) * dv;
    const double t = __fma_rn(part == 0 ? vx : part == 1 ? vy : vz, rm3, -s * xc);
    nu[6 * (size_t)k + part] = G * (g + t);
    nu[6 * (size_t)k + 3 + part] = w[6 * (size_t)k + part];  // d(position)/dt = velocity
  } else {
    const double rk_w = __fma_rn(x[0], wk[0], __fma_rn(x[1], wk[1], x[2] * wk[2])) * rm3;  // w_k . r_k / |r_k|^3
    const double rk_W = __fma_rn(x[0], Wv[0], __fma_rn(x[1], Wv[1], x[2] * Wv[2])) * rm3;
    dm[k] += G * (tot[7] - rk_w - rk_W);
    m0_part[k] -= G * rk_w;
  }
}

// nu = J(Y)^T w for the heliocentric gravity with Kepler and indirect terms:
// one CTA per body k, its threads split the other bodies j and the CTA sums
// in a fixed order.  Also dm[k] += w . d(dydt)/d m_k, and the per-body terms
// of d/d m_0 into m0_part[k] (added over the calls; summed once at the end).
//
// With d = r_j - r_k, v = [k source of j] m_k w_j - [j source of k] m_j w_k,
// the pair adds T(d) v = v / r^3 - 3 d (d . v) / r^5 to the gradient.  m_k and
// w_k are the CTA's own, so the first part is m_k sum w_j / r^3 -
// w_k sum m_j / r^3 (four FMAs), and d . v = m_k (d . w_j) - m_j (d . w_k)
// shares d . w_j with the mass gradient.  The sum of w_j over the sinks of k,
// which the indirect term wants, is k_vjp_cotangent's total less k's own.
//
// FP64 pipe: 28 FP64 instructions a pair (about 55 with rsqrt, v and T(d) v
// by component), 16 cycles of the SM's pipe each: 55 us at 1,033 bodies with the sums; a
// body per CTA of four warps rather than per warp spreads 1,033 bodies evenly
// over the SMs (7 CTAs each) and keeps 28 warps in flight.  Measured at 1,033
// bodies: 72 us a product (76% of the pipe), from 116 (and three more launches, one now).
__global__ void __launch_bounds__(kVjpThreads) k_vjp(int n, int nm, int nspl, const double* __restrict__ soa,
                                                     const double* __restrict__ wsum, int nwsum,
                                                     const double* __restrict__ w, double* __restrict__ nu,
                                                     double* __restrict__ dm, double* __restrict__ m0_part) {
  __shared__ double red[kVjpWarps][8];
  __shared__ double tot[8];
  __shared__ double W[3];
  const int k = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (k == 0) {  // the central body's state is fixed: its dydt is 0 (Acceleration.cpp:266)
    if (threadIdx.x < 6) nu[threadIdx.x] = 0.0;
    return;
  }
  const double* X = soa;
  const double* Yy = soa + n;
  const double* Z = soa + 2 * (size_t)n;
  const double* M = soa + 3 * (size_t)n;
  const double* WX = soa + 4 * (size_t)n;
  const double* WY = soa + 5 * (size_t)n;
  const double* WZ = soa + 6 * (size_t)n;
  const double xk = X[k], yk = Yy[k], zk = Z[k], mk = M[k];
  const double wkx = WX[k], wky = WY[k], wkz = WZ[k];
  const int ns_k = k < nm ? nm + nspl : nm;   // sources of k: j < ns_k
  // k is a source of the sinks j < jk: every body (k massive), the massive
  // ones (k a super-planetesimal) or none
  const int jk = k < nm ? n : (k < nm + nspl ? nm : 0);
  const int jmax = max(jk, ns_k);
  if (warp < 3) {  // component `warp` of the sum of w_v over the sinks of k
    double t = 0.0;
    if (jk > 0)
      for (int b = lane; b < nwsum; b += 32) t += wsum[6 * (size_t)b + (k < nm ? warp : 3 + warp)];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) W[warp] = k < nm ? t - (warp == 0 ? wkx : (warp == 1 ? wky : wkz)) : t;
  }
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0};  // sum w_j / r^3 (3), m_j / r^3, d (d . v) / r^5 (3), -(d . w_j) / r^3
  for (int j = 1 + threadIdx.x; j < jmax; j += kVjpThreads) {
    const double dx = X[j] - xk, dy = Yy[j] - yk, dz = Z[j] - zk;  // r_j - r_k
    const bool sink = j < jk, source = j < ns_k;
    const double wjx = sink ? WX[j] : 0.0, wjy = sink ? WY[j] : 0.0, wjz = sink ? WZ[j] : 0.0;
    const double mj = source ? M[j] : 0.0;
    if (j == k) continue;
    const double r2 = __fma_rn(dx, dx, __fma_rn(dy, dy, dz * dz));
    double rm3, rm2;
    rinv32(r2, rm3, rm2);
    const double p = __fma_rn(dx, wjx, __fma_rn(dy, wjy, dz * wjz));
    const double q = __fma_rn(dx, wkx, __fma_rn(dy, wky, dz * wkz));
    // d a_j / d m_k = G (r_k - r_j) / |r_k - r_j|^3 (direct part)
    v[7] = __fma_rn(-rm3, p, v[7]);
    const double s = (__fma_rn(mk, p, -mj * q) * rm2) * rm3;
    v[0] = __fma_rn(rm3, wjx, v[0]);
    v[1] = __fma_rn(rm3, wjy, v[1]);
    v[2] = __fma_rn(rm3, wjz, v[2]);
    v[3] = __fma_rn(rm3, mj, v[3]);
    v[4] = __fma_rn(s, dx, v[4]);
    v[5] = __fma_rn(s, dy, v[5]);
    v[6] = __fma_rn(s, dz, v[6]);
  }
  const double mine = warp_sum8(v, lane);
  if ((lane & 3) == 0) red[warp][4 * (lane >> 4 & 1) + 2 * (lane >> 3 & 1) + (lane >> 2 & 1)] = mine;
  __syncthreads();
  if (threadIdx.x < 8) {
    double t = red[0][threadIdx.x];
    for (int u = 1; u < kVjpWarps; ++u) t += red[u][threadIdx.x];
    tot[threadIdx.x] = t;
  }
  __syncwarp();
  if (threadIdx.x >= 4) return;
  const double x[3] = {xk, yk, zk}, wk[3] = {wkx, wky, wkz};
  vjp_finish_body(threadIdx.x, k, x, wk, mk, M[0], tot, W, w, nu, dm, m0_part);
}

// ---- block pairs: every unordered pair once --------------------------------------
// Seen from j, d changes its sign and p = d . w_j and q = d . w_k change places,
// so r^-3, p, q and s = (m_k p - m_j q) / r^5 serve both bodies: 20 FP64
// instructions shared and 8 a side, 36 an unordered pair where k_vjp takes 56.
// Bodies in blocks of 32.  A CTA has one pair of blocks (I, J), I <= J, its four
// warps eight of the 32 steps each: lane l of a warp holds body k = 32 I + l
// with its sums, and at step t takes body 32 J + (l + t) mod 32 from shared
// memory, whose sums pass from lane to lane by shuffles.  (I = J: steps 1 to 16,
// the last by half of the lanes.)  The warps' sums are added in shared memory
// and written, k's and j's sides, to part[pair][side][8][32]; k_vjp_finish adds
// a body's partials.  Blocks that lie beyond the sources attract nothing: only
// pairs with I below nsb = ceil(sources / 32).
//
// FP64 pipe: 18 instructions a pair and body, 16.5 cycles each: 34 us at 1,033
// bodies (561 CTAs, 3.7 an SM).  Measured, the product with its cotangent:
// 1,033 bodies 82 -> 61 us, 4,000 460 -> 285, 16,384 7.1 -> 4.4 ms.
constexpr int kPairBodies = 32;
constexpr int kPairWarps = 4;
constexpr int kPairSteps = 32 / kPairWarps;
constexpr int kFinishWarps = 16;
// Bodies for which it is used: below kPairMin k_vjp's one launch is shorter (a
// product with its cotangent, us: 300 bodies 19 and 26, 500 33 and 29, 700 49 and
// 38), beyond kPairMax the partials, 4 KB a block pair, would pass 0.54 GB.
constexpr int kPairMin = 448, kPairMax = 16384;

__host__ __device__ __forceinline__ size_t vjp_pair(int I, int J, int nb) {
  return (size_t)I * nb - (size_t)I * (I - 1) / 2 + (J - I);
}

__global__ void __launch_bounds__(32 * kPairWarps, 4)
    k_vjp_pairs(int n, int nm, int nspl, int nb, const double* __restrict__ soa, double* __restrict__ part) {
  __shared__ double sj[7][kPairBodies];
  __shared__ double red[2][kPairWarps][8][32];
  int I = 0, J = blockIdx.x;  // row I has nb - I pairs
  {
    const float t = 2.0f * nb + 1.0f;
    I = max(0, min(nb - 1, (int)(0.5f * (t - sqrtf(fmaxf(0.0f, t * t - 8.0f * (float)J))))));
    while (I > 0 && (long long)vjp_pair(I, I, nb) > (long long)blockIdx.x) --I;
    while (I + 1 < nb && (long long)vjp_pair(I + 1, I + 1, nb) <= (long long)blockIdx.x) ++I;
    J = I + (int)(blockIdx.x - vjp_pair(I, I, nb));
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // a body beyond the system: apart from all others, no pair of it counts
  for (int q = threadIdx.x; q < 7 * kPairBodies; q += 32 * kPairWarps) {
    const int row = q / kPairBodies, j = J * kPairBodies + q % kPairBodies;
    sj[row][q % kPairBodies] = j < n ? soa[(size_t)row * n + j] : (row == 0 ? 1.0e6 * (1 + q % kPairBodies) : 0.0);
  }
  const int k = I * kPairBodies + lane;
  const bool livek = k >= 1 && k < n;
  const double xk = k < n ? soa[k] : -1.0e6, yk = k < n ? soa[n + k] : 0.0, zk = k < n ? soa[2 * (size_t)n + k] : 0.0;
  const double mk = livek ? soa[3 * (size_t)n + k] : 0.0;
  const double wkx = livek ? soa[4 * (size_t)n + k] : 0.0, wky = livek ? soa[5 * (size_t)n + k] : 0.0,
               wkz = livek ? soa[6 * (size_t)n + k] : 0.0;
  const bool diag = I == J;
  const int steps = diag ? kPairSteps / 2 : kPairSteps;
  const int t0 = diag ? 1 + warp * steps : warp * steps;
  double v[8] = {0, 0, 0, 0, 0, 0, 0, 0}, u[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  __syncthreads();
#pragma unroll 1
  for (int t = t0;; ++t) {
    const int q = (lane + t) & 31, j = J * kPairBodies + q;
    const bool live = livek && j >= 1 && j < n && !(diag && t == 16 && lane >= 16);
    const bool ks = live && (k < nm || (k < nm + nspl && j < nm));  // k attracts j
    const bool js = live && (j < nm || (j < nm + nspl && k < nm));  // j attracts k
    const double dx = sj[0][q] - xk, dy = sj[1][q] - yk, dz = sj[2][q] - zk;
    const double wjx = ks ? sj[4][q] : 0.0, wjy = ks ? sj[5][q] : 0.0, wjz = ks ? sj[6][q] : 0.0;
    const double vkx = js ? wkx : 0.0, vky = js ? wky : 0.0, vkz = js ? wkz : 0.0;
    const double mj = js ? sj[3][q] : 0.0, mi = ks ? mk : 0.0;
    if (ks | js) {
      const double r2 = __fma_rn(dx, dx, __fma_rn(dy, dy, dz * dz));
      double rm3, rm2;
      rinv32(r2, rm3, rm2);
      const double p = __fma_rn(dx, wjx, __fma_rn(dy, wjy, dz * wjz));
      const double g = __fma_rn(dx, vkx, __fma_rn(dy, vky, dz * vkz));
      const double s = (__fma_rn(mi, p, -mj * g) * rm2) * rm3;
      v[0] = __fma_rn(rm3, wjx, v[0]);
      v[1] = __fma_rn(rm3, wjy, v[1]);
      v[2] = __fma_rn(rm3, wjz, v[2]);
      v[3] = __fma_rn(rm3, mj, v[3]);
      v[4] = __fma_rn(s, dx, v[4]);
      v[5] = __fma_rn(s, dy, v[5]);
      v[6] = __fma_rn(s, dz, v[6]);
      v[7] = __fma_rn(-rm3, p, v[7]);
      u[0] = __fma_rn(rm3, vkx, u[0]);
      u[1] = __fma_rn(rm3, vky, u[1]);
      u[2] = __fma_rn(rm3, vkz, u[2]);
      u[3] = __fma_rn(rm3, mi, u[3]);
      u[4] = __fma_rn(-s, dx, u[4]);
      u[5] = __fma_rn(-s, dy, u[5]);
      u[6] = __fma_rn(-s, dz, u[6]);
      u[7] = __fma_rn(rm3, g, u[7]);
    }
    if (t == t0 + steps - 1) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        red[0][warp][c][lane] = v[c];
        red[1][warp][c][q] = u[c];
      }
      break;
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) u[c] = __shfl_sync(0xffffffffu, u[c], (lane + 1) & 31);
  }
  __syncthreads();
  double* out = part + (size_t)blockIdx.x * 16 * 32;
  for (int x = threadIdx.x; x < 8 * 32; x += 32 * kPairWarps) {
    const int c = x >> 5, l = x & 31;
    const double a = (red[0][0][c][l] + red[0][1][c][l]) + (red[0][2][c][l] + red[0][3][c][l]);
    const double b = (red[1][0][c][l] + red[1][1][c][l]) + (red[1][2][c][l] + red[1][3][c][l]);
    out[x] = diag ? a + b : a;
    out[8 * 32 + x] = diag ? 0.0 : b;
  }
}

// A block's bodies: the partials in block order, the body's own terms (nu, dm,
// m0_part), at a step's last stage (lam_out not null) lambda + sum nu (S), and
// the cotangent of the next stage (L.k > 0; wsum_next is not wsum, which other
// CTAs may still read).  Bounded by the latency of the partials' loads.
__global__ void __launch_bounds__(32 * kFinishWarps) k_vjp_finish(
    int n, int nm, int nspl, int nb, int nsb, double* __restrict__ soa, const double* __restrict__ part,
    const double* __restrict__ wsum, double* __restrict__ w, double* nu, double* __restrict__ dm,
    double* __restrict__ m0_part, const double* __restrict__ lam, double* lam_out, Lin S,
    const double* __restrict__ Ynext, const double* __restrict__ mass, double h, Lin L,
    double* __restrict__ wsum_next) {
  __shared__ double tot[kFinishWarps / 8][8][32];
  __shared__ double W[6];
  __shared__ double sw[6 * kPreBodies];
  static_assert(kPreBodies == kPairBodies, "a CTA finishes a block and prepares it");
  const int B = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  {
    // partial q of the block, q < nq: from row q as the column B, then the row's own
    const int c = warp & 7, nq = B < nsb ? nb : nsb;
    double t = 0.0;
    constexpr int kStep = kFinishWarps / 8;
#pragma unroll 4
    for (int q = warp >> 3; q < nq; q += kStep) {
      const size_t at = q < B ? vjp_pair(q, B, nb) * 2 + 1 : vjp_pair(B, q, nb) * 2;
      t += part[at * 256 + 32 * c + lane];
    }
    tot[warp >> 3][c][lane] = t;
  }
  if (warp < 6) {
    double t = 0.0;
    for (int b = lane; b < nb; b += 32) t += wsum[6 * (size_t)b + warp];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) W[warp] = t;
  }
  __syncthreads();
  const int k = B * kPairBodies + lane;
  if (warp < 4 && k < n) {
    if (k == 0) {
      if (warp < 3) nu[warp] = nu[3 + warp] = 0.0;
    } else {
      const double x[3] = {soa[k], soa[n + k], soa[2 * (size_t)n + k]};
      const double wk[3] = {soa[4 * (size_t)n + k], soa[5 * (size_t)n + k], soa[6 * (size_t)n + k]};
      // the sum of w over the sinks of k: every other body, the massive ones, none
      const bool massive = k < nm, source = k < nm + nspl;
      double mine[8], Wv[3];
#pragma unroll
      for (int q = 0; q < 3; ++q) Wv[q] = massive ? W[q] - wk[q] : source ? W[3 + q] : 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        mine[q] = tot[0][q][lane];
#pragma unroll
        for (int u = 1; u < kFinishWarps / 8; ++u) mine[q] += tot[u][q][lane];
      }
      vjp_finish_body(warp, k, x, wk, soa[3 * (size_t)n + k], mass[0], mine, Wv, w, nu, dm, m0_part);
    }
  }
  __syncthreads();
  if (lam_out) {
    const size_t e = 6 * (size_t)B * kPairBodies + threadIdx.x;
    if (threadIdx.x < 6 * kPairBodies && e < 6 * (size_t)n) {
      double acc = 0.0;
      for (int q = 0; q < S.k; ++q) acc = __fma_rn(S.c[q], S.v[q][e], acc);
      lam_out[e] = __fma_rn(1.0, acc, lam[e]);
    }
    __syncthreads();
  }
  if (L.k > 0) cotangent(n, nm, Ynext, mass, h, L, w, soa, wsum_next, sw);
}

// dm[0] += sum of the per-body parts, one block, fixed order
__global__ void k_sum_m0(int n, const double* __restrict__ part, double* __restrict__ dm) {
  __shared__ double red[kBlock];
  double a = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) a += part[i];
  red[threadIdx.x] = a;
  __syncthreads();
  for (int s = kBlock / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) dm[0] += red[0];
}

inline int grid_for(int n) {
  int g = (n + kBlock - 1) / kBlock;
  return g < 1 ? 1 : (g > 152 * 16 ? 152 * 16 : g);
}

#define RET(x)                   \
  do {                           \
    int r_ = (x);                \
    if (r_ != SOL_OK) return r_; \
  } while (0)

}  // namespace

// Adjoint state kept in the context between forward and backward.
struct sol_adjoint_state {
  int n_steps = 0, every = 0, n_cp = 0;
  double h = 0.0;
  double* d_cp = nullptr;     // checkpoints, (n_cp) x 6N
  double* d_stages = nullptr; // every x 11 x 6N stage states of one segment
  int stages_of = -1;         // which segment's they are (-1: none that still holds)
  double* d_nu = nullptr;     // 11 x 6N stage adjoints
  double* d_lam = nullptr;    // 6N, and the next step's
  double* d_lam2 = nullptr;
  double* d_w = nullptr;      // 6N
  double* d_soa = nullptr;    // 7N
  double* d_wsum = nullptr;   // two of 6 per CTA of k_vjp_cotangent
  double* d_part = nullptr;   // partials of k_vjp_pairs, or null: k_vjp
  double* d_dm = nullptr;     // N
  double* d_m0p = nullptr;    // N
  double* d_tmp = nullptr;    // 6N
};

void sol_adjoint_free(sol_adjoint_state* a) {
  if (!a) return;
  double* p[] = {a->d_cp, a->d_stages, a->d_nu, a->d_lam, a->d_lam2, a->d_w, a->d_soa, a->d_wsum, a->d_part, a->d_dm, a->d_m0p,
                a->d_tmp};
  for (double* q : p)
    if (q) cudaFree(q);
  delete a;
}

// The masses or the precision changed: stage states of the forward pass no
// longer are what recomputing their segment gives.
void sol_adjoint_model_changed(sol_ctx* c) {
  if (c->adj) c->adj->stages_of = -1;
}

namespace {
int set_fixed_h(sol_ctx* c, double h) {
  sol_ctrl hc;
  memset(&hc, 0, sizeof(hc));
  hc.h = h;
  hc.h_next = h;
  hc.eps = c->eps;
  SOL_CUDA(cudaMemcpyAsync(c->d_ctrl, &hc, sizeof(hc), cudaMemcpyHostToDevice, c->stream));
  return SOL_OK;
}

size_t stage_doubles(const sol_adjoint_state* a, size_t nv) {
  return (size_t)std::min(a->every, a->n_steps) * kAdjStages * nv;
}

// One step from `from` to `to` (which may be the same), its stage states to
// step `slot` of the segment's
int step_keeping_stages(sol_ctx* c, sol_adjoint_state* a, int slot, const double* from, double* to) {
  const size_t nv = c->nv;
  double* base = a->d_stages + (size_t)slot * kAdjStages * nv;
  double* outs[13];
  for (int k = 0; k < 13; ++k) outs[k] = k < kAdjStages ? base + (size_t)k * nv : nullptr;
  SOL_CUDA(cudaMemcpyAsync(outs[0], from, sizeof(double) * nv, cudaMemcpyDeviceToDevice, c->stream));
  RET(sol_rkf78_stages(c, outs[0], to, outs));
  return SOL_OK;
}

// w_k / h: kB[k] lambda + sum_{j > k} a_jk nu_j
Lin stage_cotangent(const sol_adjoint_state* a, const double* lam, int k, size_t nv) {
  Lin L;
  memset(&L, 0, sizeof(L));
  L.v[L.k] = lam;
  L.c[L.k++] = kB[k];
  for (int j = k + 1; j < kAdjStages; ++j)
    if (kA[j][k] != 0.0) {
      L.v[L.k] = a->d_nu + (size_t)j * nv;
      L.c[L.k++] = kA[j][k];
    }
  return L;
}

// nu = J(Y)^T w of the cotangent w = h sum_i L.c[i] L.v[i]
int vjp(sol_ctx* c, sol_adjoint_state* a, const double* Y, double h, const Lin& L, double* nu) {
  const int n = c->n;
  const int nb = (n + kPreBodies - 1) / kPreBodies;
  k_vjp_cotangent<<<nb, 6 * kPreBodies, 0, c->stream>>>(n, c->cls.nm, Y, c->d_mass, h, L, a->d_w, a->d_soa,
                                                        a->d_wsum);
  SOL_LAUNCHED();
  k_vjp<<<n, kVjpThreads, 0, c->stream>>>(n, c->cls.nm, c->cls.n_spl, a->d_soa, a->d_wsum, nb, a->d_w, nu, a->d_dm,
                                          a->d_m0p);
  SOL_LAUNCHED();
  return SOL_OK;
}
}  // namespace

extern "C" int sol_adjoint_forward(sol_ctx* c, double h, int32_t n_steps, int32_t every, const double* y0,
                                   double* y_final) {
  if (!c || !y0 || n_steps < 1 || every < 1 || !(h != 0.0)) {
    sol_set_error("sol_adjoint_forward: bad arguments");
    return SOL_ERR_ARG;
  }
  if (c->barycentric || c->has_gas) {
    sol_set_error("the adjoint covers heliocentric gravity without a nebula");
    return SOL_ERR_ARG;
  }
  SOL_CUDA(cudaSetDevice(c->device));
  sol_adjoint_free(c->adj);
  c->adj = new sol_adjoint_state();
  sol_adjoint_state* a = c->adj;
  a->n_steps = n_steps;
  a->every = every;
  a->h = h;
  a->n_cp = (n_steps + every - 1) / every;
  const size_t nv = c->nv;
  auto alloc = [&](double** p, size_t cnt) -> int {
    if (cudaMalloc((void**)p, sizeof(double) * (cnt ? cnt : 1)) != cudaSuccess) {
      sol_set_error("adjoint allocation of %zu doubles failed", cnt);
      return SOL_ERR_NOMEM;
    }
    return SOL_OK;
  };
  RET(alloc(&a->d_cp, (size_t)a->n_cp * nv));
  // the last segment's stage states, if there is room for them now
  const int last = a->n_cp - 1;
  if (cudaMalloc((void**)&a->d_stages, sizeof(double) * stage_doubles(a, nv)) != cudaSuccess) {
    cudaGetLastError();
    a->d_stages = nullptr;
  }
  SOL_CUDA(cudaMemcpyAsync(c->d_y0, y0, sizeof(double) * nv, cudaMemcpyHostToDevice, c->stream));
  RET(set_fixed_h(c, h));
  for (int s = 0; s < n_steps; ++s) {
    if (s % every == 0)
      SOL_CUDA(cudaMemcpyAsync(a->d_cp + (size_t)(s / every) * nv, c->d_y0, sizeof(double) * nv,
                               cudaMemcpyDeviceToDevice, c->stream));
    if (a->d_stages && s >= last * every)
      RET(step_keeping_stages(c, a, s - last * every, c->d_y0, c->d_y));
    else
      RET(sol_rkf78_stages(c, c->d_y0, c->d_y, nullptr));
    SOL_CUDA(cudaMemcpyAsync(c->d_y0, c->d_y, sizeof(double) * nv, cudaMemcpyDeviceToDevice, c->stream));
  }
  if (a->d_stages) a->stages_of = last;
  c->state_valid = 1;
  if (y_final) SOL_CUDA(cudaMemcpyAsync(y_final, c->d_y0, sizeof(double) * nv, cudaMemcpyDeviceToHost, c->stream));
  SOL_CUDA(cudaStreamSynchronize(c->stream));
  return SOL_OK;
}

extern "C" int sol_adjoint_backward(sol_ctx* c, const double* dl_dy_final, double* dl_dy0, double* dl_dmass) {
  if (!c || !dl_dy_final || !c->adj || !c->adj->d_cp) {
    sol_set_error("sol_adjoint_backward: run sol_adjoint_forward first");
    return SOL_ERR_STATE;
  }
  SOL_CUDA(cudaSetDevice(c->device));
  sol_adjoint_state* a = c->adj;
  const size_t nv = c->nv;
  const int n = c->n;
  auto alloc = [&](double** p, size_t cnt) -> int {
    if (*p) return SOL_OK;
    if (cudaMalloc((void**)p, sizeof(double) * (cnt ? cnt : 1)) != cudaSuccess) {
      sol_set_error("adjoint allocation of %zu doubles failed", cnt);
      return SOL_ERR_NOMEM;
    }
    return SOL_OK;
  };
  RET(alloc(&a->d_stages, stage_doubles(a, nv)));
  RET(alloc(&a->d_nu, (size_t)kAdjStages * nv));
  RET(alloc(&a->d_lam, nv));
  RET(alloc(&a->d_lam2, nv));
  RET(alloc(&a->d_w, nv));
  RET(alloc(&a->d_soa, 7 * (size_t)n));
  const int nb = (n + kPairBodies - 1) / kPairBodies;
  const int ns = c->cls.nm + c->cls.n_spl, nsb = (ns + kPairBodies - 1) / kPairBodies;
  const size_t npairs = vjp_pair(nsb, nsb, nb);
  RET(alloc(&a->d_wsum, 12 * (size_t)nb));
  if (n >= kPairMin && n <= kPairMax && !a->d_part &&
      cudaMalloc((void**)&a->d_part, sizeof(double) * npairs * 16 * 32) != cudaSuccess) {
    cudaGetLastError();  // no room for the partials: k_vjp needs none
    a->d_part = nullptr;
  }
  RET(alloc(&a->d_dm, n));
  RET(alloc(&a->d_m0p, n));
  RET(alloc(&a->d_tmp, nv));
  SOL_CUDA(cudaMemcpyAsync(a->d_lam, dl_dy_final, sizeof(double) * nv, cudaMemcpyHostToDevice, c->stream));
  SOL_CUDA(cudaMemsetAsync(a->d_dm, 0, sizeof(double) * n, c->stream));
  SOL_CUDA(cudaMemsetAsync(a->d_m0p, 0, sizeof(double) * n, c->stream));
  RET(set_fixed_h(c, a->h));
  const double h = a->h;
  const int g = grid_for((int)nv);
  for (int seg = a->n_cp - 1; seg >= 0; --seg) {
    const int s0 = seg * a->every;
    const int s1 = std::min(a->n_steps, s0 + a->every);
    // recompute the segment, keeping the stage states Y_0..Y_10 of every step
    if (a->stages_of != seg) {
      a->stages_of = -1;
      SOL_CUDA(cudaMemcpyAsync(a->d_tmp, a->d_cp + (size_t)seg * nv, sizeof(double) * nv, cudaMemcpyDeviceToDevice,
                               c->stream));
      for (int s = s0; s < s1; ++s) RET(step_keeping_stages(c, a, s - s0, a->d_tmp, a->d_tmp));
      a->stages_of = seg;
    }
    // backward through the segment's steps
    int buf = 0;
    for (int s = s1 - 1; s >= s0; --s) {
      const double* Ys = a->d_stages + (size_t)(s - s0) * kAdjStages * nv;
      // lambda + sum nu, once the step's stages are done
      Lin S;
      memset(&S, 0, sizeof(S));
      for (int k = 0; k < kAdjStages; ++k) {
        S.v[S.k] = a->d_nu + (size_t)k * nv;
        S.c[S.k++] = 1.0;
      }
      for (int k = kAdjStages - 1; k >= 0; --k) {
        double* nu = a->d_nu + (size_t)k * nv;
        const bool first = s == s1 - 1 && k == kAdjStages - 1;
        if (!a->d_part) {
          RET(vjp(c, a, Ys + (size_t)k * nv, h, stage_cotangent(a, a->d_lam, k, nv), nu));
          continue;
        }
        double* wsum = a->d_wsum + (size_t)buf * 6 * nb;
        if (first) {
          k_vjp_cotangent<<<nb, 6 * kPreBodies, 0, c->stream>>>(n, c->cls.nm, Ys + (size_t)k * nv, c->d_mass, h,
                                                                stage_cotangent(a, a->d_lam, k, nv), a->d_w, a->d_soa,
                                                                wsum);
          SOL_LAUNCHED();
        }
        k_vjp_pairs<<<(unsigned)npairs, 32 * kPairWarps, 0, c->stream>>>(n, c->cls.nm, c->cls.n_spl, nb, a->d_soa,
                                                                         a->d_part);
        SOL_LAUNCHED();
        // the next stage: this step's, or the last one of the step before (none at the segment's start)
        const bool end = k == 0;
        Lin next;
        memset(&next, 0, sizeof(next));
        const double* Yn = nullptr;
        if (!end) {
          next = stage_cotangent(a, a->d_lam, k - 1, nv);
          Yn = Ys + (size_t)(k - 1) * nv;
        } else if (s > s0) {
          next = stage_cotangent(a, a->d_lam2, kAdjStages - 1, nv);
          Yn = Ys - nv;  // stage 10 of the step before
        }
        k_vjp_finish<<<nb, 32 * kFinishWarps, 0, c->stream>>>(n, c->cls.nm, c->cls.n_spl, nb, nsb, a->d_soa, a->d_part, wsum, a->d_w,
                                                nu, a->d_dm, a->d_m0p, a->d_lam, end ? a->d_lam2 : nullptr, S, Yn,
                                                c->d_mass, h, next, a->d_wsum + (size_t)(1 - buf) * 6 * nb);
        SOL_LAUNCHED();
        buf = 1 - buf;
      }
      if (!a->d_part) {
        k_lincomb<<<g, kBlock, 0, c->stream>>>((int)nv, a->d_lam2, a->d_lam, 1.0, S);
        SOL_LAUNCHED();
      }
      std::swap(a->d_lam2, a->d_lam);
    }
  }
  k_sum_m0<<<1, kBlock, 0, c->stream>>>(n, a->d_m0p, a->d_dm);
  SOL_LAUNCHED();
  if (dl_dy0) SOL_CUDA(cudaMemcpyAsync(dl_dy0, a->d_lam, sizeof(double) * nv, cudaMemcpyDeviceToHost, c->stream));
  if (dl_dmass) SOL_CUDA(cudaMemcpyAsync(dl_dmass, a->d_dm, sizeof(double) * n, cudaMemcpyDeviceToHost, c->stream));
  SOL_CUDA(cudaStreamSynchronize(c->stream));
  return SOL_OK;
}

extern "C" int sol_set_masses(sol_ctx* c, const double* mass) {
  if (!c || !mass) return SOL_ERR_ARG;
  SOL_CUDA(cudaSetDevice(c->device));
  SOL_CUDA(cudaMemcpyAsync(c->d_mass, mass, sizeof(double) * c->n, cudaMemcpyHostToDevice, c->stream));
  SOL_CUDA(cudaStreamSynchronize(c->stream));
  sol_adjoint_model_changed(c);
  // captured driver graphs read masses from device memory: nothing to rebuild
  return SOL_OK;
}
