// Discrete adjoint of the fixed-step RungeKuttaFehlberg78 integration
// (RungeKuttaFehlberg78::Step at constant h, y_{n+1} = the 7th-order result,
// Solaris/RungeKuttaFehlberg78.cpp:147-250) with GravityAC forces
// (Solaris/Acceleration.cpp:248-329).
//
// Forward: n fixed steps on the device, the state stored every K steps.
// Backward, one segment of K steps at a time from the last: the segment is
// recomputed from its checkpoint with every stage state Y_k (k = 0..10) of
// every step kept; then, step by step from the last, the stage adjoints
//   w_k = h b_k lambda + h sum_{j>k} a_jk nu_j,   nu_k = J(Y_k)^T w_k
// and lambda_n = lambda_{n+1} + sum_k nu_k, with the mass gradient
// accumulated from the same w_k.  Stages 11 and 12 only enter the error
// estimate, so their adjoints are zero.  J^T w is a hand-written
// vector-Jacobian product of the pair force (one warp per body).
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
constexpr int kPreBodies = 42;    // bodies per CTA of k_vjp_cotangent: 252 elements
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
// the structure-of-arrays view of (state, cotangent) that k_vjp streams -- x,
// y, z, m, wx, wy, wz -- and this CTA's sums of the cotangent's velocity part
// over its bodies: [0..2] those with index >= 1, [3..5] those below nm.  One
// thread per element, kPreBodies bodies per CTA.
__global__ void __launch_bounds__(6 * kPreBodies) k_vjp_cotangent(int n, int nm, const double* __restrict__ Y,
                                                                  const double* __restrict__ mass, double h, Lin L,
                                                                  double* __restrict__ w, double* __restrict__ soa,
                                                                  double* __restrict__ wsum) {
  __shared__ double sw[6 * kPreBodies];
  const int i0 = blockIdx.x * kPreBodies;
  const int b = threadIdx.x / 6, k = threadIdx.x - 6 * b;
  const int i = i0 + b;
  double acc = 0.0;
  if (i < n) {
    const size_t e = 6 * (size_t)i + k;
    for (int q = 0; q < L.k; ++q) acc = __fma_rn(L.c[q], L.v[q][e], acc);
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
  __syncthreads();
  if (threadIdx.x < 6) {
    const int c = 3 + threadIdx.x % 3;
    const int hi = min(i0 + kPreBodies, threadIdx.x < 3 ? n : nm);
    double t = 0.0;
    for (int j = max(i0, 1); j < hi; ++j) t += sw[6 * (j - i0) + c];
    wsum[6 * (size_t)blockIdx.x + threadIdx.x] = t;
  }
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

// Eight sums over the warp in 9 additions a lane (40 for eight shuffle
// trees): at the first three steps a lane hands half of its sums to its
// partner and takes the other half.  Lane l ends with sum
// 4 (l >> 4 & 1) + 2 (l >> 3 & 1) + (l >> 2 & 1).
__device__ __forceinline__ double warp_sum8(double (&v)[8], int lane) {
#pragma unroll
  for (int half = 4, off = 16; half >= 1; half >>= 1, off >>= 1) {
    const bool up = (lane & off) != 0;
#pragma unroll
    for (int q = 0; q < half; ++q) {
      const double send = up ? v[q] : v[q + half];
      const double keep = up ? v[q + half] : v[q];
      v[q] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  return v[0];
}

__device__ __forceinline__ void tensor_apply(double dx, double dy, double dz, double rm3, double rm5, double vx,
                                             double vy, double vz, double& ox, double& oy, double& oz) {
  // T(d) v = v / r^3 - 3 d (d . v) / r^5
  const double dv = __fma_rn(dx, vx, __fma_rn(dy, vy, dz * vz));
  const double s = 3.0 * rm5 * dv;
  ox = __fma_rn(vx, rm3, -s * dx);
  oy = __fma_rn(vy, rm3, -s * dy);
  oz = __fma_rn(vz, rm3, -s * dz);
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
  if (threadIdx.x != 0) return;
  const double G = SOL_GAUSS2;
  const double gx = __fma_rn(mk, tot[0], __fma_rn(-wkx, tot[3], -3.0 * tot[4]));
  const double gy = __fma_rn(mk, tot[1], __fma_rn(-wky, tot[3], -3.0 * tot[5]));
  const double gz = __fma_rn(mk, tot[2], __fma_rn(-wkz, tot[3], -3.0 * tot[6]));
  // Kepler term -G (m0 + m_k) r_k / |r_k|^3 and indirect term -G m_k r_k / |r_k|^3 (for the sinks of k)
  const double r2 = __fma_rn(xk, xk, __fma_rn(yk, yk, zk * zk));
  double rm3, rm2;
  rinv32(r2, rm3, rm2);
  const double mu = -(M[0] + mk);
  const double Wx = W[0], Wy = W[1], Wz = W[2];  // 0 when k is no source
  double kx, ky, kz;
  tensor_apply(xk, yk, zk, rm3, rm3 * rm2, __fma_rn(mu, wkx, -mk * Wx), __fma_rn(mu, wky, -mk * Wy),
               __fma_rn(mu, wkz, -mk * Wz), kx, ky, kz);
  nu[6 * (size_t)k + 0] = G * (gx + kx);
  nu[6 * (size_t)k + 1] = G * (gy + ky);
  nu[6 * (size_t)k + 2] = G * (gz + kz);
  nu[6 * (size_t)k + 3] = w[6 * (size_t)k + 0];  // d(position)/dt = velocity
  nu[6 * (size_t)k + 4] = w[6 * (size_t)k + 1];
  nu[6 * (size_t)k + 5] = w[6 * (size_t)k + 2];
  const double rk_w = __fma_rn(xk, wkx, __fma_rn(yk, wky, zk * wkz)) * rm3;  // w_k . r_k / |r_k|^3
  const double rk_W = __fma_rn(xk, Wx, __fma_rn(yk, Wy, zk * Wz)) * rm3;
  dm[k] += G * (tot[7] - rk_w - rk_W);
  m0_part[k] -= G * rk_w;
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
  double* d_nu = nullptr;     // 11 x 6N stage adjoints
  double* d_lam = nullptr;    // 6N
  double* d_w = nullptr;      // 6N
  double* d_soa = nullptr;    // 7N
  double* d_wsum = nullptr;   // 6 per CTA of k_vjp_cotangent
  double* d_dm = nullptr;     // N
  double* d_m0p = nullptr;    // N
  double* d_tmp = nullptr;    // 6N
};

void sol_adjoint_free(sol_adjoint_state* a) {
  if (!a) return;
  double* p[] = {a->d_cp, a->d_stages, a->d_nu, a->d_lam, a->d_w, a->d_soa, a->d_wsum, a->d_dm, a->d_m0p, a->d_tmp};
  for (double* q : p)
    if (q) cudaFree(q);
  delete a;
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
  SOL_CUDA(cudaMemcpyAsync(c->d_y0, y0, sizeof(double) * nv, cudaMemcpyHostToDevice, c->stream));
  RET(set_fixed_h(c, h));
  for (int s = 0; s < n_steps; ++s) {
    if (s % every == 0)
      SOL_CUDA(cudaMemcpyAsync(a->d_cp + (size_t)(s / every) * nv, c->d_y0, sizeof(double) * nv,
                               cudaMemcpyDeviceToDevice, c->stream));
    RET(sol_rkf78_stages(c, c->d_y0, c->d_y, nullptr));
    SOL_CUDA(cudaMemcpyAsync(c->d_y0, c->d_y, sizeof(double) * nv, cudaMemcpyDeviceToDevice, c->stream));
  }
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
  RET(alloc(&a->d_stages, (size_t)a->every * kAdjStages * nv));
  RET(alloc(&a->d_nu, (size_t)kAdjStages * nv));
  RET(alloc(&a->d_lam, nv));
  RET(alloc(&a->d_w, nv));
  RET(alloc(&a->d_soa, 7 * (size_t)n));
  RET(alloc(&a->d_wsum, 6 * (size_t)((n + kPreBodies - 1) / kPreBodies)));
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
    SOL_CUDA(cudaMemcpyAsync(a->d_tmp, a->d_cp + (size_t)seg * nv, sizeof(double) * nv, cudaMemcpyDeviceToDevice,
                             c->stream));
    for (int s = s0; s < s1; ++s) {
      double* base = a->d_stages + (size_t)(s - s0) * kAdjStages * nv;
      double* outs[13];
      for (int k = 0; k < 13; ++k) outs[k] = k < kAdjStages ? base + (size_t)k * nv : nullptr;
      SOL_CUDA(cudaMemcpyAsync(outs[0], a->d_tmp, sizeof(double) * nv, cudaMemcpyDeviceToDevice, c->stream));
      RET(sol_rkf78_stages(c, outs[0], a->d_tmp, outs));
    }
    // backward through the segment's steps
    for (int s = s1 - 1; s >= s0; --s) {
      const double* Ys = a->d_stages + (size_t)(s - s0) * kAdjStages * nv;
      for (int k = kAdjStages - 1; k >= 0; --k) {
        Lin L;
        memset(&L, 0, sizeof(L));
        L.v[L.k] = a->d_lam;
        L.c[L.k++] = kB[k];
        for (int j = k + 1; j < kAdjStages; ++j)
          if (kA[j][k] != 0.0) {
            L.v[L.k] = a->d_nu + (size_t)j * nv;
            L.c[L.k++] = kA[j][k];
          }
        RET(vjp(c, a, Ys + (size_t)k * nv, h, L, a->d_nu + (size_t)k * nv));
      }
      Lin L;
      memset(&L, 0, sizeof(L));
      for (int k = 0; k < kAdjStages; ++k) {
        L.v[L.k] = a->d_nu + (size_t)k * nv;
        L.c[L.k++] = 1.0;
      }
      k_lincomb<<<g, kBlock, 0, c->stream>>>((int)nv, a->d_w, a->d_lam, 1.0, L);
      SOL_LAUNCHED();
      std::swap(a->d_w, a->d_lam);
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
  // captured driver graphs read masses from device memory: nothing to rebuild
  return SOL_OK;
}
