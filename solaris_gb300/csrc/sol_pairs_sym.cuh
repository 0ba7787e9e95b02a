// SPLIT_FF pairs of massive bodies, each unordered pair once (included by
// sol_force.cu inside its namespace).
//
// A pair's displacement, r^2 and r^-3 are the same numbers seen from either
// body (d changes its sign, exactly), and both bodies take a term from it:
// G m_j r^-3 d on i, -G m_i r^-3 d on j.  k_pairs_ff forms them twice; here a
// pair costs 59 FP32 operations shared by its two terms and 42 for each term,
// 71.5 a term instead of 103.5.
//
// Bodies are taken in blocks of 64, 128 or 256.  A CTA has a block I of sinks, two a
// thread (the two lanes of its paired FP32 instructions: a warp's 64 sinks),
// and runs over the source blocks J >= I of a chunk.  Within a warp the 32
// lanes work on 32 different sources at a time; a source's sums travel from
// lane to lane by shuffles, past all 64 sinks in 32 steps, while its position
// comes from shared memory.  The sinks' sums stay in registers.  After 32
// steps the source's sums are added in FP64 to the CTA's partial of block J:
// the warps work on different 32-source parts of J between two barriers, so
// every sum has a fixed order.  k_combine adds a body's partials, as source
// of the blocks below its own and as sink of its own block's chunks.  The block
// itself (J = I) is evaluated as sinks alone, every source.
//
// The arithmetic of a term is k_pairs_ff's (sol_pair.cuh), with a sum folded
// into FP64 every 128 (sink) or 32 (source) terms a lane instead of 128.
// Either side of a block pair can be left out (a block of sinks alone,
// sol_accel_sinks_device): what is computed keeps its order and so its bits.
//
// Bounded by the FP32 pipe: 71.5 operations a term are 7.6 ms at 65,536 bodies;
// the kernel takes 10.8 (70 %), an evaluation 11.06 for 13.9 before, of 16,384
// bodies 0.77 ms for 0.99, of 10,007 335 us for 455, of 2,049 66 for 99.  Its
// error is no larger: bodies of comparable pull on each other as from the centre,
// 24 systems of 8,000 to 16,384, median of the largest against the reference form
// 1.5e-13 for 2.0e-13; rms against long double (2,049 to 50,000 bodies) 9.2e-15
// for 9.7e-15.  The FP64 sums are compensated as k_pairs_ff's are; without that
// (and the two lanes' low words added in FP32) an evaluation takes 10.87 ms and
// 331 us, and what a later sum cancels down to is lost.
//
// Pairs closer than the grid (ff_close_pair) leave their FP32 terms zero: the
// sink takes the FP64 term at once, the source's side is marked and evaluated
// after the block pair by a pass over it in source order (sym_close_pass).

// Bodies per block (and sources per tile): BLOCK, 64 to 256; a thread has two sinks.
__host__ __device__ constexpr int sym_threads(int block) { return block / 2; }
// Four CTAs an SM (128 registers): measured at 65,536 bodies 10.7 ms against
// 11.3 with three (144 registers), and 11.3 against 12.1 before the bounds of
// k_near_bound; one source at a time a warp -- two interleaved take 160
// registers and three CTAs -- 12.0.
__host__ __device__ constexpr int sym_ctas(int block) { return 1024 / block; }

// A source's table entries, each twice (both lanes of a paired operand), two
// to a 16-byte load.
constexpr int kSymRows = (kFF + 1) / 2;
template <int BLOCK>
struct SymTile {
  float4 v[kSymRows][BLOCK];
};
struct SymSource {
  float2 v[2 * kSymRows];
};
template <int BLOCK>
__device__ __forceinline__ SymSource sym_load(const SymTile<BLOCK>& T, int q) {
  SymSource s;
#pragma unroll
  for (int k = 0; k < kSymRows; ++k) {
    const float4 w = T.v[k][q];
    s.v[2 * k] = make_float2(w.x, w.y);
    s.v[2 * k + 1] = make_float2(w.z, w.w);
  }
  return s;
}
template <int BLOCK>
struct SymShared {
  SymTile<BLOCK> tile;
  // FP64 sums of the sources of J: totals and, where more than one warp adds to
  // one, compensation
  double js[BLOCK > 64 ? 2 : 1][3][BLOCK];
  float jmh[BLOCK], jml[BLOCK];  // their nearest sink of I
  int jnn[BLOCK];
  int close;
  // a thread's FP64 sums of its two sinks (here, not in registers: they change
  // every 128 sources only): totals and compensation; with blocks below 256, whose
  // CTAs have one block of sources and one total of it, that total and the close pairs
  double sums[2][6][sym_threads(BLOCK)];
};

// Nearest neighbour of one body: the smallest r^2 (hi, then lo), ties to the lower index.
struct SymNear {
  float h, l;
  int j;
};
__device__ __forceinline__ void sym_near(SymNear& m, float h, float l, bool ok, int j) {
  const bool better = ok & ((h < m.h) | ((h == m.h) & ((l < m.l) | ((l == m.l) & ((unsigned)j < (unsigned)m.j)))));
  m.h = better ? h : m.h;
  m.l = better ? l : m.l;
  m.j = better ? j : m.j;
}

// r^2 below which a pair is close (ff_close_pair), as in k_pairs_ff: |d| < max(G1, 2^-50)
__device__ __forceinline__ float sym_close_r2(const ForceCtx& fc) {
  const double G1 = fc.ind_sum[kIndGrid];
  return fmaxf((float)(G1 * G1), 7.888609052210118e-31f);
}

// The sum of two float-float numbers of one source (its two lanes'), to 2^-70 and
// better, before its one rounding: the FP32 parts added exactly, so that two of
// seven FP64 instructions (a conversion is one) go.
__device__ __forceinline__ double sym_lanes(float2 h, float2 l) {
  float u, e, v, w, f, g;
  ff_two_sum(h.x, h.y, u, e);
  ff_two_sum(l.x, l.y, v, w);
  ff_two_sum(e, v, f, g);
  return (double)u + ((double)f + (double)(g + w));
}

// v into component k of source q's sums; first: the first value of a block pair.
// (With blocks of 64 bodies there is one, its only warp's, and the close pairs'.)
template <int BLOCK>
__device__ __forceinline__ void sym_add_source(SymShared<BLOCK>& sm, int k, int q, double v, bool first) {
  if (BLOCK == 64 || first) {
    sm.js[0][k][q] = v;
    if constexpr (BLOCK > 64) sm.js[1][k][q] = 0.0;
  } else if constexpr (BLOCK > 64) {
    add_ordered(sm.js[0][k][q], sm.js[1][k][q], v);
  }
}

// Component k's total of up to 128 sources, and a close pair, into the thread's sums
template <int BLOCK>
__device__ __forceinline__ void sym_add_sink(SymShared<BLOCK>& sm, int k, double v) {
  if constexpr (BLOCK > 128)
    add_ordered(sm.sums[0][k][threadIdx.x], sm.sums[1][k][threadIdx.x], v);
  else
    sm.sums[0][k][threadIdx.x] = v;
}
template <int BLOCK>
__device__ __forceinline__ void sym_add_close(SymShared<BLOCK>& sm, int k, double v) {
  if constexpr (BLOCK > 128)
    add_ordered(sm.sums[0][k][threadIdx.x], sm.sums[1][k][threadIdx.x], v);
  else
    sm.sums[1][k][threadIdx.x] += v;
}

struct SymSinks {  // the thread's two sinks
  float2 a[3], b[3], c[3];  // grid triples
  float2 gh, gl;            // -G m
  int i0, i1;
};
struct SymSums {
  float2 h[3], l[3];
};

__device__ __forceinline__ float2 sym_shift(float2 v, int from) {
  return make_float2(__shfl_sync(0xFFFFFFFFu, v.x, from), __shfl_sync(0xFFFFFFFFu, v.y, from));
}

// d, r^2 of one source and both sinks
__device__ __forceinline__ void sym_displacement(const SymSource& J, const SymSinks& S, float2* h, float2* l,
                                                 float2& r2h, float2& r2l) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float2 s1 = f2_sub(J.v[FAX + 3 * k], S.a[k]);
    const float2 s2 = f2_sub(J.v[FBX + 3 * k], S.b[k]);
    const float2 s3 = f2_sub(J.v[FCX + 3 * k], S.c[k]);
    float2 l0;
    f2_fast_two_sum(s1, s2, h[k], l0);
    l[k] = f2_add(l0, s3);
  }
  f2_ff_r2(h, l, r2h, r2l);
}

// A source's nearest sink in the CTA's shared arrays: read always, written
// when a sink is nearer (about ln N times)
template <int BLOCK>
__device__ __forceinline__ void sym_near_source(SymShared<BLOCK>& sm, int q, const SymSinks& S, int ns, float2 r2h,
                                                float2 r2l) {
  SymNear m = {sm.jmh[q], sm.jml[q], sm.jnn[q]};
  sym_near(m, r2h.x, r2l.x, (S.i0 >= 1) & (S.i0 < ns), S.i0);
  sym_near(m, r2h.y, r2l.y, (S.i1 >= 1) & (S.i1 < ns), S.i1);
  sm.jmh[q] = m.h;
  sm.jml[q] = m.l;
  sm.jnn[q] = m.j;
}

// A step of a warp once d and r^2 are known: the terms into the sinks' sums A
// and the source's travelling sums B.  The float-float sums are renormalised at
// every second step (second).
template <bool DI, bool DJ, bool SECOND>
__device__ __forceinline__ void sym_terms(const float2* h, const float2* l, float2 qh, float2 ql, float2 gh, float2 gl,
                                          float2 mh, float2 ml, int from, SymSums& A, SymSums& B) {
  float2 Rh, Rl, sh, se;
  f2_ff_rinv3(qh, ql, Rh, Rl);
  if (DJ) {
    f2_ff_scale(mh, ml, Rh, Rl, sh, se);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      f2_ff_accumulate_lazy(B.h[k], B.l[k], sh, se, h[k], l[k]);
      if (SECOND) f2_fast_two_sum(B.h[k], B.l[k], B.h[k], B.l[k]);
      // the source's sums move on with it
      B.h[k] = sym_shift(B.h[k], from);
      B.l[k] = sym_shift(B.l[k], from);
    }
  }
  if (DI) {
    f2_ff_scale(gh, gl, Rh, Rl, sh, se);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      f2_ff_accumulate_lazy(A.h[k], A.l[k], sh, se, h[k], l[k]);
      if (SECOND) f2_fast_two_sum(A.h[k], A.l[k], A.h[k], A.l[k]);
    }
  }
}

template <bool DI, bool DJ, bool SECOND, int BLOCK>
__device__ __forceinline__ void sym_step(SymShared<BLOCK>& sm, const ForceCtx& fc, const double* __restrict__ y, int q,
                                         int from, int j0, int ns, float thr, const SymSinks& S, SymSums& A,
                                         SymNear& n0, SymNear& n1, SymSums& B) {
  float2 h[3], l[3], r2h, r2l;
  const SymSource J = sym_load(sm.tile, q);
  sym_displacement(J, S, h, l, r2h, r2l);
  // (the whole warp takes one way: the sources' sums pass through shuffles)
  if (__builtin_expect(!__any_sync(0xFFFFFFFFu, fminf(r2h.x, r2h.y) < thr), 1)) {
    sym_terms<DI, DJ, SECOND>(h, l, r2h, r2l, J.v[FGH], J.v[FGL], S.gh, S.gl, from, A, B);
  } else {
    float2 qh = r2h, ql = r2l, gh = J.v[FGH], gl = J.v[FGL], mh = S.gh, ml = S.gl;
    const int j = j0 + q;
    if (r2h.x < thr) {
      const double* p = y + 6 * (size_t)S.i0;
      double f[3] = {0.0, 0.0, 0.0};
      if (S.i0 < ns && j < ns) ff_close_pair(fc, j, p[0], p[1], p[2], gh.x, gl.x, f[0], f[1], f[2], r2h.x, r2l.x);
      if (DI)
        for (int k = 0; k < 3; ++k) sym_add_close(sm, k, f[k]);
      gh.x = gl.x = mh.x = ml.x = ql.x = 0.0f;
      qh.x = 1.0f;
      sm.close = 1;
    }
    if (r2h.y < thr) {
      const double* p = y + 6 * (size_t)S.i1;
      double f[3] = {0.0, 0.0, 0.0};
      if (S.i1 < ns && j < ns) ff_close_pair(fc, j, p[0], p[1], p[2], gh.y, gl.y, f[0], f[1], f[2], r2h.y, r2l.y);
      if (DI)
        for (int k = 0; k < 3; ++k) sym_add_close(sm, 3 + k, f[k]);
      gh.y = gl.y = mh.y = ml.y = ql.y = 0.0f;
      qh.y = 1.0f;
      sm.close = 1;
    }
    __syncwarp();
    sym_terms<DI, DJ, SECOND>(h, l, qh, ql, gh, gl, mh, ml, from, A, B);
  }
  const bool near_i = DI && (r2h.x <= n0.h || r2h.y <= n1.h);
  const bool near_j = DJ && fminf(r2h.x, r2h.y) <= sm.jmh[q];
  if (near_i | near_j) {
    if (DI) {
      const int j = j0 + q;
      const bool src = (j >= 1) & (j < ns);
      sym_near(n0, r2h.x, r2l.x, src & (j != S.i0), j);
      sym_near(n1, r2h.y, r2l.y, src & (j != S.i1), j);
    }
    if (DJ) sym_near_source(sm, q, S, ns, r2h, r2l);
  }
}

// 32 steps of a warp: its 64 sinks past the 32 sources of part `sub` of the
// tile.  DI / DJ: the sinks' / the sources' sums.
template <bool DI, bool DJ, int BLOCK>
__device__ __forceinline__ void sym_part(SymShared<BLOCK>& sm, const ForceCtx& fc, const double* __restrict__ y, int sub,
                                         int lane, int j0, int ns, float thr, const SymSinks& S, SymSums& A,
                                         SymNear& n0, SymNear& n1, SymSums& B) {
  const int from = (lane + 1) & 31;
#pragma unroll 1
  for (int t = 0; t < 32; t += 2) {
    sym_step<DI, DJ, false>(sm, fc, y, sub * 32 + ((lane + t) & 31), from, j0, ns, thr, S, A, n0, n1, B);
    __syncwarp();  // the next lane's source, whose nearest sink this one may just have written
    sym_step<DI, DJ, true>(sm, fc, y, sub * 32 + ((lane + t + 1) & 31), from, j0, ns, thr, S, A, n0, n1, B);
    __syncwarp();
  }
}

// The source side of the close pairs of a block pair, in sink order.
template <int BLOCK>
__device__ __noinline__ void sym_close_pass(SymShared<BLOCK>& sm, const ForceCtx& fc, const double* __restrict__ y, int i0,
                                            int j0, int ns, float thr) {
  const float* T = ftab(fc);
  const int np = fc.npad;
  for (int q = threadIdx.x; q < BLOCK; q += sym_threads(BLOCK)) {
    const int j = j0 + q;
    if (j >= ns) continue;
    const double* p = y + 6 * (size_t)j;
    const SymSource J = sym_load(sm.tile, q);
    double f[3] = {0.0, 0.0, 0.0};
    for (int i = i0; i < min(i0 + BLOCK, ns); ++i) {
      float2 h[3], l[3], r2h, r2l;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const float2 s1 = f2_sub(J.v[FAX + 3 * k], f2_splat(T[(size_t)(FAX + 3 * k) * np + i]));
        const float2 s2 = f2_sub(J.v[FBX + 3 * k], f2_splat(T[(size_t)(FBX + 3 * k) * np + i]));
        const float2 s3 = f2_sub(J.v[FCX + 3 * k], f2_splat(T[(size_t)(FCX + 3 * k) * np + i]));
        float2 l0;
        f2_fast_two_sum(s1, s2, h[k], l0);
        l[k] = f2_add(l0, s3);
      }
      f2_ff_r2(h, l, r2h, r2l);
      if (!(r2h.x < thr)) continue;
      float a, b;
      ff_close_pair(fc, i, p[0], p[1], p[2], T[(size_t)FGH * np + i], T[(size_t)FGL * np + i], f[0], f[1], f[2], a, b);
    }
    for (int k = 0; k < 3; ++k) {
      if constexpr (BLOCK > 64)
        add_ordered(sm.js[0][k][q], sm.js[1][k][q], f[k]);
      else
        sm.js[0][k][q] += f[k];
    }
  }
}

// An upper bound of every body's squared distance to its nearest neighbour:
// the smallest among the sources of its own block and the next ones
// (kBoundBlocks in all), in FP32 from the grid triples' two leading parts.  What
// they leave out, up to 2^-24 G1 a component, is ~2^-23 of a distance of G1 or
// more, which the factor covers, but of any size for a closer pair: such a
// pair's r^2 is below sym_close_r2, and the bound is not.  A sink starts its
// search there, so that a new minimum is rare (without it every block pair begins
// with ~5 updates a body, and hardly a step of a warp has none).
constexpr int kBoundBlocks = 4;
constexpr int kBoundParts = 4, kBoundSources = kTile / kBoundParts;  // a block in quarters: a shorter chain
__global__ void __launch_bounds__(kTile) k_near_bound(ForceCtx fc, float* __restrict__ bound, int nb) {
  __shared__ float2 sx[kBoundSources], sy[kBoundSources], sz[kBoundSources];
  const float* T = ftab(fc);
  const int np = fc.npad, ns = fc.cls.nm;
  const int i = blockIdx.x * kTile + threadIdx.x;
  const int j0 = ((blockIdx.x + blockIdx.y / kBoundParts) % nb) * kTile + blockIdx.y % kBoundParts * kBoundSources;
  auto at = [&](int k, int j) {
    return make_float2(T[(size_t)(FAX + 3 * k) * np + j], T[(size_t)(FBX + 3 * k) * np + j]);
  };
  const float2 x = at(0, i), yy = at(1, i), z = at(2, i);
  if (threadIdx.x < kBoundSources) {
    sx[threadIdx.x] = at(0, j0 + threadIdx.x);
    sy[threadIdx.x] = at(1, j0 + threadIdx.x);
    sz[threadIdx.x] = at(2, j0 + threadIdx.x);
  }
  __syncthreads();
  float m = 3.0e38f;
  const int q1 = min(kBoundSources, ns - j0);
#pragma unroll 8
  for (int q = j0 == 0 ? 1 : 0; q < q1; ++q) {
    const float dx = (sx[q].x - x.x) + (sx[q].y - x.y), dy = (sy[q].x - yy.x) + (sy[q].y - yy.y),
                dz = (sz[q].x - z.x) + (sz[q].y - z.y);
    const float r2 = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz));
    m = (j0 + q != i && r2 < m) ? r2 : m;
  }
  // k_split_table set 3e38; the order of floats that are not negative is that of their bits
  m = fmaxf(m, sym_close_r2(fc));
  atomicMin(reinterpret_cast<int*>(bound) + i, __float_as_int(fminf(m * 1.0001f, 3.0e38f)));
}

// part_i: [chunk][PART_SLOTS][npad] as k_pairs_ff's; part_j: per block pair
// I < J, packed by I, [PART_SLOTS][BLOCK].
__device__ __forceinline__ size_t sym_pair_index(int I, int J, int nb) {
  return (size_t)I * (nb - 1) - (size_t)I * (I - 1) / 2 + (J - I - 1);
}

// CTAs of chunks 0 .. C - 1 whose sinks lie in blocks below the chunk's: chunk c
// has per c of them.
__host__ __device__ __forceinline__ int sym_tasks_above(int C, int per) { return per * (C * (C - 1) / 2); }

template <int BLOCK>
__global__ void __launch_bounds__(sym_threads(BLOCK), sym_ctas(BLOCK))
    k_pairs_sym(ForceCtx fc, const double* __restrict__ y, double* __restrict__ part_i, double* __restrict__ part_j,
                const float* __restrict__ bound, int nb, int per) {
  extern __shared__ __align__(16) unsigned char sym_dyn[];
  SymShared<BLOCK>& sm = *reinterpret_cast<SymShared<BLOCK>*>(sym_dyn);
  constexpr int kThreads = sym_threads(BLOCK), kParts = BLOCK / 32;
  // The CTA's block of sinks I and its chunk C of `per` blocks of sources: first
  // the chunks above I's own, by chunk, then the nb of I's own, whose diagonal
  // block takes less, so that the last to start are short.  No CTA is launched
  // for nothing: on a grid of I x C whose lower half returned at once the CTAs
  // left gathered on some of the SMs (10,007 bodies: 529 us an evaluation, 424
  // on this one).
  const int task = blockIdx.x;
  const int above = sym_tasks_above((nb + per - 1) / per, per);
  int I, C;
  if (task < above) {
    C = (int)((1.0f + sqrtf(1.0f + 8.0f * (float)(task / per))) * 0.5f);
    while (sym_tasks_above(C, per) > task) --C;
    while (sym_tasks_above(C + 1, per) <= task) ++C;
    I = task - sym_tasks_above(C, per);
  } else {
    I = task - above;
    C = I / per;
  }
  const int Jlo = max(I, C * per), Jhi = min(nb, (C + 1) * per);
  const int np = fc.npad, ns = fc.cls.nm;
  const int lo = fc.sink_lo, hi = sol_sink_hi(fc);
  auto wanted = [&](int B) { return B * BLOCK < hi && (B + 1) * BLOCK > lo; };
  const bool want_i = wanted(I);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float* T = ftab(fc);
  SymSinks S;
  S.i0 = I * BLOCK + warp * 64 + lane;
  S.i1 = S.i0 + 32;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    S.a[k] = make_float2(T[(size_t)(FAX + 3 * k) * np + S.i0], T[(size_t)(FAX + 3 * k) * np + S.i1]);
    S.b[k] = make_float2(T[(size_t)(FBX + 3 * k) * np + S.i0], T[(size_t)(FBX + 3 * k) * np + S.i1]);
    S.c[k] = make_float2(T[(size_t)(FCX + 3 * k) * np + S.i0], T[(size_t)(FCX + 3 * k) * np + S.i1]);
  }
  S.gh = make_float2(-T[(size_t)FGH * np + S.i0], -T[(size_t)FGH * np + S.i1]);
  S.gl = make_float2(-T[(size_t)FGL * np + S.i0], -T[(size_t)FGL * np + S.i1]);
  const float thr = sym_close_r2(fc);
  for (int k = 0; k < 12; ++k) sm.sums[k / 6][k % 6][threadIdx.x] = 0.0;
  SymNear n0 = {bound[S.i0], 3.0e38f, -1}, n1 = {bound[S.i1], 3.0e38f, -1};
  for (int J = Jlo; J < Jhi; ++J) {
    const bool want_j = J != I && wanted(J);
    if (!want_i && !want_j) continue;
    const int j0 = J * BLOCK;
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < kSymRows; ++k)
      for (int q = threadIdx.x; q < BLOCK; q += kThreads) {
        const float v = T[(size_t)(2 * k) * np + j0 + q];
        const float w = 2 * k + 1 < kFF ? T[(size_t)(2 * k + 1) * np + j0 + q] : 0.0f;
        sm.tile.v[k][q] = make_float4(v, v, w, w);
      }
    for (int q = threadIdx.x; q < BLOCK; q += kThreads) {
      sm.jmh[q] = bound[j0 + q];
      sm.jml[q] = 3.0e38f;
      sm.jnn[q] = -1;
    }
    if (threadIdx.x == 0) sm.close = 0;
    __syncthreads();
    SymSums A;
#pragma unroll
    for (int k = 0; k < 3; ++k) A.h[k] = A.l[k] = make_float2(0.0f, 0.0f);
#pragma unroll 1
    for (int p = 0; p < kParts; ++p) {
      const int sub = (p + 2 * warp) & (kParts - 1);  // a part of its own for every warp, its first for p = 0 and 1
      const int q = sub * 32 + lane;
      SymSums B;
#pragma unroll
      for (int k = 0; k < 3; ++k) B.h[k] = B.l[k] = make_float2(0.0f, 0.0f);
      if (want_i && want_j)
        sym_part<true, true>(sm, fc, y, sub, lane, j0, ns, thr, S, A, n0, n1, B);
      else if (want_i)
        sym_part<true, false>(sm, fc, y, sub, lane, j0, ns, thr, S, A, n0, n1, B);
      else
        sym_part<false, true>(sm, fc, y, sub, lane, j0, ns, thr, S, A, n0, n1, B);
      if (want_j) {
#pragma unroll
        for (int k = 0; k < 3; ++k)
          sym_add_source(sm, k, q, sym_lanes(B.h[k], B.l[k]), p < 2);
      }
      if (want_i && ((p & 3) == 3 || p == kParts - 1)) {  // the sinks' float-float sums of 128 sources into FP64
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          sym_add_sink(sm, k, (double)A.h[k].x + (double)A.l[k].x);
          sym_add_sink(sm, 3 + k, (double)A.h[k].y + (double)A.l[k].y);
          A.h[k] = A.l[k] = make_float2(0.0f, 0.0f);
        }
      }
      __syncthreads();
    }
    if (want_j) {
      if (sm.close) {
        sym_close_pass(sm, fc, y, I * BLOCK, j0, ns, thr);
        __syncthreads();
      }
      double* out = part_j + sym_pair_index(I, J, nb) * PART_SLOTS * BLOCK;
      for (int q = threadIdx.x; q < BLOCK; q += kThreads) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          double v = sm.js[0][k][q];
          if constexpr (BLOCK > 64) v += sm.js[1][k][q];
          out[(PAX + k) * BLOCK + q] = v;
        }
        out[PR2 * BLOCK + q] = sm.jnn[q] >= 0 ? (double)sm.jmh[q] + (double)sm.jml[q] : 1.0e300;
        out[PIDX * BLOCK + q] = __longlong_as_double((long long)sm.jnn[q]);
      }
    }
  }
  if (!want_i) return;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const SymNear& m = u ? n1 : n0;
    double* out = part_i + (size_t)C * PART_SLOTS * np + (u ? S.i1 : S.i0);
#pragma unroll
    for (int k = 0; k < 3; ++k)
      out[(size_t)(PAX + k) * np] = sm.sums[0][3 * u + k][threadIdx.x] + sm.sums[1][3 * u + k][threadIdx.x];
    out[(size_t)PR2 * np] = m.j >= 0 ? (double)m.h + (double)m.l : 1.0e300;
    out[(size_t)PIDX * np] = __longlong_as_double((long long)m.j);
  }
}
