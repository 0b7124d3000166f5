// Converging multigrid: solves the reference's discrete pressure operator
// (5-point Laplacian with edge ghosts, outlet row pinned at 0; the operator of
// pressure_solvers/multigrid_solver.py:173-183) to ||b - A p||_2 <= rtol ||b||_2.
//
// Structure of one refinement iteration (one body of the graph's while node):
//   levels 0 .. lc-1   k_cv_down: 2 red-black sweeps from e = 0 in a shared-
//                      memory tile, residual, 2x2 restriction
//   levels lc .. D     k_cv_block: one 1024-thread block holding the smallest
//                      levels (<= 16384 cells) in shared memory: sweeps,
//                      restriction, the FP64 dense solve of the coarsest grid,
//                      prolongation, sweeps
//   levels lc-1 .. 1   k_cv_up: e += P(e_coarse), 2 red-black sweeps
//   level 0            k_cv_up0: e += P(e_coarse), 1 red-black sweep (a
//                      V(2,1) cycle on the fine grid: from the warm starts of
//                      a developed flow it ends in as many cycles as V(2,2)
//                      with a halo of 3 instead of 5), then p += e, the
//                      residual r = b - A p for the next iteration, its FP64
//                      norm, and (k_cv_check, or the last block beside
//                      other instances) the convergence test that sets
//                      the while node's condition with cudaGraphSetConditional
//
// Precision.  The V-cycle runs in FP32.  The refinement state p and the
// refinement residual are kept in double-FP32 ("double-single") arithmetic:
// p = hi + lo with |lo| <= ulp(hi)/2, updated and applied with the error-free
// transformations TwoSum (Knuth) and TwoProd (Dekker, via fma), which carry a
// ~48-bit significand on the FP32 pipes.  GB300 executes FP64 at 1/64 of the
// FP32 rate, and a plain-FP64 residual cost ~25 us per cycle at 2048x512.
// FP64 proper is kept where it is cheap: the coarsest-grid dense solve and the
// global norms that decide termination.
// The pressure state ping-pongs between two buffers (a tile's halo must see the
// old values while neighbouring tiles write the new ones).
// Coarse operators are rediscretised at spacing 2^l h; the outlet Dirichlet
// point stays where the fine grid has it (ghost g * e_last with
// g = (theta - 1) / theta, theta = (1 - 2^-l) / 2).  The oracle is
// oracle/ref_np.py mg_converge (FP64 throughout).
#include "aj_internal.cuh"
#include <algorithm>
#include <math.h>
#include <string.h>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

namespace aj {

constexpr int CV_NS = 2;                         // red-black sweeps per smoothing phase
constexpr int CV_BLOCK_THREADS = 1024;
constexpr int CV_BLOCK_MAX_CELLS = 16384;        // levels handled by the one-block kernel

struct CvLvl {
  int n, m, level;
  float ax, ay, g;   // g: outlet ghost factor of this level (level >= 1)
};

static double ghost_factor(int level) {
  double th = 0.5 * (1.0 - pow(2.0, -level));
  return (th - 1.0) / th;
}

static CvLvl cv_level(const AjStepParams& p, const Layout& L, int l) {
  CvLvl c;
  c.n = L.ln[l];
  c.m = L.lm[l];
  c.level = l;
  double hx = p.dx * (double)(1 << l), hy = p.dy * (double)(1 << l);
  c.ax = (float)(1.0 / (hx * hx));
  c.ay = (float)(1.0 / (hy * hy));
  c.g = l > 0 ? (float)ghost_factor(l) : 0.f;
  return c;
}

// ---------------------------------------------------------------- double-FP32
// (df, two_sum, quick_two_sum, two_prod, df_add: aj_internal.cuh)
__device__ __forceinline__ df df_neg(df a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ df df_mul(df a, df b) {
  df p = two_prod(a.hi, b.hi);
  p.lo += a.hi * b.lo + a.lo * b.hi;
  return quick_two_sum(p.hi, p.lo);
}

// ---------------------------------------------------------------- paired double-FP32
// Two double-FP32 values side by side (a thread's two columns of a tile row)
// through the same error-free transformations on the paired FP32
// instructions (f2, add2, sub2: aj_internal.cuh).
struct df2 {
  float2 hi, lo;
};
__device__ __forceinline__ df2 two_sum2(float2 a, float2 b) {
  const float2 s = add2(a, b);
  const float2 bb = sub2(s, a);
  return {s, add2(sub2(a, sub2(s, bb)), sub2(b, bb))};
}
__device__ __forceinline__ df2 quick_two_sum2(float2 a, float2 b) {
  const float2 s = add2(a, b);
  return {s, sub2(b, sub2(s, a))};
}
// Dekker's addition with one TwoSum: error <= ~2^-47 max(|a|, |b|), which in
// the residual below stays ~1e-14 |p| ax, far under the 1e-6 |b| targets
__device__ __forceinline__ df2 df2_add_s(df2 a, df2 b) {
  df2 s = two_sum2(a.hi, b.hi);
  s.lo = add2(s.lo, add2(a.lo, b.lo));
  return quick_two_sum2(s.hi, s.lo);
}
__device__ __forceinline__ df2 df2_add_f(df2 a, float2 b) {
  df2 s = two_sum2(a.hi, b);
  s.lo = add2(s.lo, a.lo);
  return quick_two_sum2(s.hi, s.lo);
}
// a * b for one double-FP32 a: TwoProd by fma, whose error term is formed
// negated (fma(-a, b, p) = -(a b - p) exactly) and subtracted
__device__ __forceinline__ df2 df2_mul_u(df a, df2 b) {
  const float2 ah = f2(a.hi);
  const float2 p = __fmul2_rn(ah, b.hi);
  const float2 en = __ffma2_rn(f2(-a.hi), b.hi, p);
  const float2 cross = __ffma2_rn(ah, b.lo, __fmul2_rn(f2(a.lo), b.hi));
  return quick_two_sum2(p, sub2(cross, en));
}
// b - a: TwoSum of b and -a.hi with the signs carried through
__device__ __forceinline__ df2 df2_rsub_f(float2 b, df2 a) {
  const float2 s = sub2(b, a.hi);
  const float2 bb = add2(s, a.hi);
  const float2 e = sub2(sub2(b, bb), add2(a.hi, sub2(s, bb)));
  return quick_two_sum2(s, sub2(e, a.lo));
}
// r = b - (ax ((xp + xm) - 2c) + ay ((yp + ym) - 2c)), all double-FP32 (-2c is
// exact, so each second difference costs two additions, not three)
__device__ __forceinline__ df2 df2_residual(float2 b, df2 c, df2 xp, df2 xm, df2 yp, df2 ym,
                                            df ax, df ay) {
  const df2 c2{__fmul2_rn(c.hi, f2(-2.f)), __fmul2_rn(c.lo, f2(-2.f))};
  const df2 sx = df2_add_s(df2_add_s(xp, xm), c2);
  const df2 sy = df2_add_s(df2_add_s(yp, ym), c2);
  return df2_rsub_f(b, df2_add_s(df2_mul_u(ax, sx), df2_mul_u(ay, sy)));
}

struct DfCoef {
  float axh, axl, ayh, ayl;   // 1/dx^2 and 1/dy^2 split into hi + lo
};
static DfCoef df_coef(double ax, double ay) {
  DfCoef c;
  c.axh = (float)ax;
  c.axl = (float)(ax - (double)c.axh);
  c.ayh = (float)ay;
  c.ayl = (float)(ay - (double)c.ayh);
  return c;
}

// ---------------------------------------------------------------- tiles
// A smoothing block covers a region of 4 G rows by 64 columns - its output
// cells and a halo - in one round trip of 8-byte reads.  A thread owns a column
// pair over four rows: those cells' e, right-hand side and inverse diagonal
// live in registers for the whole kernel, and shared memory carries only what
// neighbouring threads read, the even columns in one plane and the odd ones in
// another (unit stride for every access).  A red-black half-sweep updates one
// cell of each row: its vertical neighbours but the run's two ends are the
// thread's own, of the horizontal ones one is, so four updates cost six
// shared reads and four writes, and a half-sweep reads only the other colour,
// so one barrier separates two of them.
// Cells outside the level, and level 0's pinned outlet row, hold 0 and an
// inverse diagonal of 0, so every cell is updated alike (the diagonal carries
// the ghost rule).  The region's border is bordered by zeros: after half-sweep
// h the cells at distance h + 1 or more from it hold exact red-black values,
// and the output cells lie far enough inside (CP_H_DOWN, CP_H_UP; even, so that
// a column pair or a 2x2 block is never cut, and regions start at even
// coordinates: a cell's colour is (row + column) & 1 in the region too).
// Level-0 down and up kernels together in a stream, against tiles with every
// cell in shared memory: 1024x256 10.9 -> 7.0 us, 2048x512 25.0 -> 16.1 us,
// 4096x2048 143 -> 84 us (down 51 -> 24, up 89 -> 59: 4.7 TB/s).
constexpr int CP_RUN = 4, CP_COLS = 64, CP_PAIRS = CP_COLS / 2;
constexpr int CP_H_DOWN = 6;   // four half-sweeps and the residual need 5
constexpr int CP_H_UP = 4;     // four half-sweeps (level 0: two, and p + e one cell further)
// Threads an SM holds at once (the kernels' register bound: 56).  1152 against
// 768 for level 0's up kernel: 4096x2048 64.5 -> 58.9 us; 1536 spill.
constexpr int CP_THREADS_SM = 1152;
constexpr int CP_LD = CP_PAIRS + 1;   // plane row: one zero beside the first (odd columns) or last pair

__device__ __forceinline__ float2 cp_ldg2(const float* p) {
  return __ldg(reinterpret_cast<const float2*>(p));
}
__device__ __forceinline__ void cp_st2(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }

template <int G, int H>
struct CpTile {
  static constexpr int ROWS = CP_RUN * G, OUT_I = ROWS - 2 * H, OUT_J = CP_COLS - 2 * H;
  static constexpr int PLANE = (ROWS + 2) * CP_LD;   // a zero row above and below
  int tx, ty, gi, gj;   // the thread's first cell in the level (possibly outside)
  int n, m;
  long k;               // its index
  float* X;             // this thread's place in the planes of even and odd columns
  float* Y;
  __device__ __forceinline__ CpTile(const CvLvl& L, float* planes)
      : tx(threadIdx.x), ty(threadIdx.y), n(L.n), m(L.m) {
    gi = blockIdx.y * OUT_I - H + CP_RUN * ty;
    gj = blockIdx.x * OUT_J - H + 2 * tx;
    k = (long)gi * m + gj;
    X = planes + (CP_RUN * ty + 1) * CP_LD + tx;
    Y = planes + PLANE + (CP_RUN * ty + 1) * CP_LD + 1 + tx;
  }
  // row r of the thread lies in the level (m is even: a pair is never cut)
  __device__ __forceinline__ bool in(int r) const {
    return (unsigned)(gi + r) < (unsigned)n && (unsigned)gj < (unsigned)m;
  }
  // row r belongs to the block's output
  __device__ __forceinline__ bool mine(int r) const {
    const int i = CP_RUN * ty + r;
    return i >= H && i < ROWS - H && tx >= H / 2 && tx < CP_PAIRS - H / 2 && in(r);
  }
  __device__ __forceinline__ void zero_planes(float* planes) const {
    for (int t = ty * CP_PAIRS + tx; t < 2 * PLANE; t += CP_PAIRS * G) planes[t] = 0.f;
  }
  __device__ __forceinline__ void load(const float* src, float2* v) const {
#pragma unroll
    for (int r = 0; r < CP_RUN; ++r)
      v[r] = in(r) ? cp_ldg2(src + k + (long)r * m) : make_float2(0.f, 0.f);
  }
  __device__ __forceinline__ void put(const float2* x) const {
#pragma unroll
    for (int r = 0; r < CP_RUN; ++r) {
      X[r * CP_LD] = x[r].x;
      Y[r * CP_LD] = x[r].y;
    }
  }
  // the cells of one colour: even rows' even columns and odd rows' odd ones are red (0)
  template <int COLOR>
  __device__ __forceinline__ void put_color(const float2* x) const {
#pragma unroll
    for (int r = 0; r < CP_RUN; ++r) {
      if ((r + COLOR) & 1) Y[r * CP_LD] = x[r].y;
      else X[r * CP_LD] = x[r].x;
    }
  }
  // ax (up + down) + ay (left + right) of the cell of row r that has colour COLOR
  template <int COLOR>
  __device__ __forceinline__ float nb(const CvLvl& L, const float2* x, int r) const {
    float up, dn, sides;
    if ((r + COLOR) & 1) {
      up = r > 0 ? x[r > 0 ? r - 1 : 0].y : Y[-CP_LD];
      dn = r + 1 < CP_RUN ? x[r + 1 < CP_RUN ? r + 1 : r].y : Y[CP_RUN * CP_LD];
      sides = X[r * CP_LD + 1] + x[r].x;
    } else {
      up = r > 0 ? x[r > 0 ? r - 1 : 0].x : X[-CP_LD];
      dn = r + 1 < CP_RUN ? x[r + 1 < CP_RUN ? r + 1 : r].x : X[CP_RUN * CP_LD];
      sides = x[r].y + Y[r * CP_LD - 1];
    }
    return fmaf(L.ax, dn + up, L.ay * sides);
  }
  template <int COLOR>
  __device__ __forceinline__ void half_sweep(const CvLvl& L, const float2* b, const float2* inv,
                                             float2* x) const {
    float v[CP_RUN];
#pragma unroll
    for (int r = 0; r < CP_RUN; ++r) v[r] = nb<COLOR>(L, x, r);
#pragma unroll
    for (int r = 0; r < CP_RUN; ++r) {
      if ((r + COLOR) & 1) x[r].y = (b[r].y - v[r]) * inv[r].y;
      else x[r].x = (b[r].x - v[r]) * inv[r].x;
    }
  }
  // the diagonals of row r's pair
  __device__ __forceinline__ float2 diag(const CvLvl& L, int r) const {
    float d = -2.f * (L.ax + L.ay);
    if (gi + r == 0) d += L.ax;
    if (gi + r == n - 1) d += L.level == 0 ? L.ax : L.ax * L.g;
    return make_float2(gj == 0 ? d + L.ay : d, gj + 1 == m - 1 ? d + L.ay : d);
  }
  // their inverses, 0 for cells that stay 0
  __device__ __forceinline__ void inverse(const CvLvl& L, float2* inv) const {
    const float c = 1.f / (-2.f * (L.ax + L.ay));
    if (gi >= 1 && gi + CP_RUN <= n - 1 && gj >= 1 && gj + 2 <= m - 1) {
#pragma unroll
      for (int r = 0; r < CP_RUN; ++r) inv[r] = f2(c);
    } else {
#pragma unroll
      for (int r = 0; r < CP_RUN; ++r) {
        const float2 d = diag(L, r);
        const bool live = in(r) && !(L.level == 0 && gi + r == n - 1);
        inv[r] = live ? make_float2(1.f / d.x, 1.f / d.y) : f2(0.f);
      }
    }
  }
  // x += P(e_coarse) inside the level: the cell-centred bilinear prolongation
  // (weights 9/16, 3/16, 3/16, 1/16), first along the rows.  Ghosts: row -1
  // copies row 0 (inlet Neumann), row nc is g times row nc - 1 (outlet ghost),
  // columns clamp (wall Neumann).
  __device__ __forceinline__ void prolong(const CvLvl& L, const float* __restrict__ ec, int nc,
                                          int mc, float g, float2* x) const {
    const int I0 = (gi >> 1) - 1, J = gj >> 1;
    const int Jl = min(max(J - 1, 0), mc - 1), Jc = min(max(J, 0), mc - 1),
              Jr = min(max(J + 1, 0), mc - 1);
    float2 h[CP_RUN / 2 + 2];
#pragma unroll
    for (int i = 0; i < CP_RUN / 2 + 2; ++i) {
      const int I = min(max(I0 + i, 0), nc - 1);
      const float* e = ec + (long)I * mc;
      const float c = 3.f * ldg(e + Jc), f = I0 + i >= nc ? g : 1.f;
      h[i] = make_float2(f * (c + ldg(e + Jl)), f * (c + ldg(e + Jr)));
    }
#pragma unroll
    for (int r = 0; r < CP_RUN; ++r) {
      const float2 a = h[r / 2 + 1], o = (r & 1) ? h[r / 2 + 2] : h[r / 2];
      if (in(r) && !(L.level == 0 && gi + r == n - 1))
        x[r] = fma2(fma2(a, f2(3.f), o), f2(1.f / 16.f), x[r]);
    }
  }
};

// pre-smoothing from e = 0, residual, 2x2 average onto the coarse rhs.  On
// level 0 the residual alternates between two buffers (r0, r1) with the
// pressure state: *cur selects the one the last iteration wrote.  The first
// half-sweep from zero needs no neighbours, and after the last one the black
// cells' residuals are 0 by construction, so only the red cells' are formed.
template <int G>
__global__ void __launch_bounds__(32 * G, CP_THREADS_SM / (32 * G)) k_cv_down(
    CvLvl L, const float* r0, const float* r1, const int* cur, float* __restrict__ e_out,
    float* __restrict__ rc, const int* done) {
  pdl_wait();
  using T = CpTile<G, CP_H_DOWN>;
  __shared__ float planes[2 * T::PLANE];
  // both flags in one round trip, the first tested while the tile is loaded
  const int skip = *done, second = r1 ? *cur : 0;
  const T t(L, planes);
  float2 b[CP_RUN], x[CP_RUN], inv[CP_RUN];
  t.load(second ? r1 : r0, b);
  t.zero_planes(planes);
  t.inverse(L, inv);
  if (skip) return;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < CP_RUN; ++r)
    x[r] = (r & 1) ? make_float2(0.f, b[r].y * inv[r].y) : make_float2(b[r].x * inv[r].x, 0.f);
  t.template put_color<0>(x);
  __syncthreads();
  t.template half_sweep<1>(L, b, inv, x);
  t.template put_color<1>(x);
  __syncthreads();
  t.template half_sweep<0>(L, b, inv, x);
  t.template put_color<0>(x);
  __syncthreads();
  t.template half_sweep<1>(L, b, inv, x);
  t.template put_color<1>(x);
  __syncthreads();
  float res[CP_RUN];
#pragma unroll
  for (int r = 0; r < CP_RUN; ++r) {
    const float2 d = t.diag(L, r);
    const float nb = t.template nb<0>(L, x, r);
    const float v = (r & 1) ? b[r].y - fmaf(d.y, x[r].y, nb) : b[r].x - fmaf(d.x, x[r].x, nb);
    res[r] = L.level == 0 && t.gi + r == t.n - 1 ? 0.f : v;
  }
#pragma unroll
  for (int r = 0; r < CP_RUN; r += 2) {
    if (!t.mine(r)) continue;
    cp_st2(e_out + t.k + (long)r * t.m, x[r]);
    cp_st2(e_out + t.k + (long)(r + 1) * t.m, x[r + 1]);
    rc[(long)((t.gi + r) >> 1) * (t.m >> 1) + (t.gj >> 1)] = 0.25f * (res[r] + res[r + 1]);
  }
}

// e + P(e_coarse), post-smoothing, store (levels >= 1)
template <int G>
__global__ void __launch_bounds__(32 * G, CP_THREADS_SM / (32 * G)) k_cv_up(
    CvLvl L, const float* __restrict__ r, const float* __restrict__ e_in,
    const float* __restrict__ ec, int nc, int mc, float gc, float* __restrict__ e_out,
    const int* done) {
  pdl_wait();
  using T = CpTile<G, CP_H_UP>;
  __shared__ float planes[2 * T::PLANE];
  const int skip = *done;
  const T t(L, planes);
  float2 b[CP_RUN], x[CP_RUN], inv[CP_RUN];
  t.load(r, b);
  t.load(e_in, x);
  t.zero_planes(planes);
  t.prolong(L, ec, nc, mc, gc, x);
  t.inverse(L, inv);
  if (skip) return;
  __syncthreads();
  t.put(x);
  __syncthreads();
#pragma unroll
  for (int s = 0; s < CV_NS; ++s) {
    t.template half_sweep<0>(L, b, inv, x);
    t.template put_color<0>(x);
    __syncthreads();
    t.template half_sweep<1>(L, b, inv, x);
    if (s + 1 == CV_NS) break;
    t.template put_color<1>(x);
    __syncthreads();
  }
#pragma unroll
  for (int q = 0; q < CP_RUN; ++q)
    if (t.mine(q)) cp_st2(e_out + t.k + (long)q * t.m, x[q]);
}

// asynchronous 8-byte global-to-shared copy; zeros when !in (the source is
// then not read)
__device__ __forceinline__ void cv_cp8(float* dst, const float* src, bool in) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src),
               "r"(in ? 8 : 0));
}

struct CvCheck {
  int max_cycles;
  int use_handle;
  cudaGraphConditionalHandle h;
  int apart = 0;   // the test runs in a kernel of its own (k_cv_check)
};

// convergence bookkeeping after a V-cycle (device scalars; one thread).  All
// fields are loaded before any is stored: interleaved, every load waited for
// the store before it (a chain of dependent round trips at the end of the
// cycle's last kernel).  The test compares squares - sum r^2 against the
// solve's target rtol^2 sum b^2 - so that no FP64 root or quotient (1/64 of
// the FP32 rate) stands between two cycles; k_cv_out forms the norms.
__device__ void cv_check_body(DevScalars* sc, const CvCheck& ck) {
  int done = sc->mg_done, cycles = sc->mg_cycles, err = sc->err, loops = sc->loops;
  const double target = sc->target, a0 = sc->acc[0];
  const int was_done = done;
  if (!was_done) {
    cycles += 1;
    sc->abs_sq = a0;
    if (!isfinite(a0)) {
      err = AJ_ERR_NONFINITE;
      done = 1;
    } else if (a0 <= target) {
      done = 1;
    } else if (cycles >= ck.max_cycles) {
      err = AJ_ERR_NOT_CONVERGED;
      done = 1;
    }
  }
  sc->acc[0] = 0.0;
  if (ck.use_handle) {
    // independent bound on the while node: never more bodies than max_cycles + 1
    loops += 1;
    if (loops > ck.max_cycles + 1 && !done) {
      err = AJ_ERR_NOT_CONVERGED;
      done = 1;
    }
    sc->loops = loops;
  }
  sc->mg_cycles = cycles;
  sc->err = err;
  sc->mg_done = done;
  if (ck.use_handle) cudaGraphSetConditional(ck.h, done ? 0u : 1u);
}

// a ping-pong pair: the pressure state (each buffer N hi values followed by N
// lo values) or the level-0 residual (N floats each)
struct PState {
  float* a;   // buffer 0
  float* b;   // buffer 1
};

// level 0: e + P(e_coarse), post-smoothing, p += e (double-FP32, ping-pong), the
// residual of the reference operator for the next iteration (double-FP32), its
// FP64 norm, and the convergence test (k_cv_check, or the last block).  The
// residual ping-pongs with the pressure (rs.a pairs with ps.a): a block reads
// the current residual over its region while its neighbours write the next
// one, so the two must never share a buffer.  The pressure of the region goes
// to shared memory beside the other reads (8-byte asynchronous copies of the
// thread's own pairs, zero outside the level and on the pinned outlet row).
template <int G>
__global__ void __launch_bounds__(32 * G, CP_THREADS_SM / (32 * G)) k_cv_up0(
    CvLvl L, PState rs, const float* __restrict__ e_in, const float* __restrict__ ec, int nc,
    int mc, float gc, PState ps, const float* __restrict__ b0, DevScalars* sc, DfCoef co,
    CvCheck ck, int profile) {
  pdl_wait();
  using T = CpTile<G, CP_H_UP>;
  const int met = sc->mg_done, cur = sc->pcur;   // one round trip
  if (!profile && met) {
    // met before this body ran (the initial guess already satisfied the
    // tolerance, or the rhs is zero): every kernel of the body skipped its
    // work and no block reaches the convergence test, so end the loop here
    // (a body after a converged one never runs: the test set the condition)
    if (ck.use_handle && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 &&
        threadIdx.y == 0)
      cudaGraphSetConditional(ck.h, 0u);
    return;
  }
  __shared__ float planes[2 * T::PLANE];
  __shared__ __align__(8) float PH[T::ROWS * CP_COLS];
  __shared__ __align__(8) float PL[T::ROWS * CP_COLS];
  const T t(L, planes);
  const long N = (long)L.n * L.m;
  const float* __restrict__ pin = cur ? ps.b : ps.a;
  float* __restrict__ pout = cur ? ps.a : ps.b;
  float* __restrict__ r_next = cur ? rs.a : rs.b;
  const int q0 = CP_RUN * t.ty * CP_COLS + 2 * t.tx;   // the thread's place in PH and PL
  float2 b[CP_RUN], x[CP_RUN], inv[CP_RUN];
  t.load(cur ? rs.b : rs.a, b);
  t.load(e_in, x);
#pragma unroll
  for (int r = 0; r < CP_RUN; ++r) {
    const bool in = t.in(r) && t.gi + r != L.n - 1;
    const long k = in ? t.k + (long)r * L.m : 0;
    cv_cp8(PH + q0 + r * CP_COLS, pin + k, in);
    cv_cp8(PL + q0 + r * CP_COLS, pin + N + k, in);
    if (t.gi + r == L.n - 1) x[r] = f2(0.f);   // the outlet row's error is 0
  }
  asm volatile("cp.async.commit_group;\n" ::);
  t.zero_planes(planes);
  t.prolong(L, ec, nc, mc, gc, x);
  t.inverse(L, inv);
  __syncthreads();
  t.put(x);
  __syncthreads();
  t.template half_sweep<0>(L, b, inv, x);
  t.template put_color<0>(x);
  __syncthreads();
  t.template half_sweep<1>(L, b, inv, x);
  // p + e on the region's cells; what the residual reads of them is exact
  t.load(b0, b);
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
  for (int r = 0; r < CP_RUN; ++r) {
    float* ph = PH + q0 + r * CP_COLS;
    float* pl = PL + q0 + r * CP_COLS;
    const df2 v = df2_add_f(df2{*reinterpret_cast<float2*>(ph), *reinterpret_cast<float2*>(pl)}, x[r]);
    cp_st2(ph, v.hi);
    cp_st2(pl, v.lo);
  }
  __syncthreads();
  float acc = 0.f;
  if (t.mine(0)) {
    const df ax{co.axh, co.axl}, ay{co.ayh, co.ayl};
    auto row = [&](int r) {
      const int q = q0 + r * CP_COLS;
      return df2{*reinterpret_cast<const float2*>(PH + q), *reinterpret_cast<const float2*>(PL + q)};
    };
    df2 c = row(0), xm = t.gi > 0 ? row(-1) : c;   // Neumann ghost at the inlet
#pragma unroll
    for (int r = 0; r < CP_RUN; ++r) {
      if (!t.mine(r)) break;
      const int q = q0 + r * CP_COLS;
      const df2 xp = row(r + 1);   // row n - 1 holds the pinned 0
      // the pair's left and right neighbours, the cell itself at the walls
      const bool lw = t.gj == 0, rw = t.gj + 2 >= L.m;
      const df2 yp{make_float2(c.hi.y, rw ? c.hi.y : PH[q + 2]),
                   make_float2(c.lo.y, rw ? c.lo.y : PL[q + 2])};
      const df2 ym{make_float2(lw ? c.hi.x : PH[q - 1], c.hi.x),
                   make_float2(lw ? c.lo.x : PL[q - 1], c.lo.x)};
      const long k = t.k + (long)r * L.m;
      cp_st2(pout + k, c.hi);
      cp_st2(pout + N + k, c.lo);
      float2 rr{0.f, 0.f};
      if (t.gi + r != L.n - 1) {
        const df2 res = df2_residual(b[r], c, xp, xm, yp, ym, ax, ay);
        rr = add2(res.hi, res.lo);
      }
      if (!profile) cp_st2(r_next + k, rr);
      acc = fmaf(rr.x, rr.x, acc);
      acc = fmaf(rr.y, rr.y, acc);
      xm = c;
      c = xp;
    }
  }
  if (profile) return;
  __shared__ df ws[G];
  const df s = warp_sum_df(acc);
  if (t.tx == 0) ws[t.ty] = s;
  __syncthreads();
  if (t.ty > 0) return;
  static_assert(G <= 16, "half a warp adds the warps");
  const double total = warp_sum<16>(t.tx < G ? df_double(ws[t.tx]) : 0.0);
  if (t.tx == 0) {
    atomicAdd(&sc->acc[0], total);
    if (ck.apart) return;
    __threadfence();
    if (atomicAdd(&sc->red_count, 1u) == gridDim.x * gridDim.y - 1) {
      __threadfence();
      sc->red_count = 0u;
      sc->pcur = 1 - cur;
      cv_check_body(sc, ck);
    }
  }
}

// the convergence test of a cycle whose k_cv_up0 left it out; nothing to do
// where the target was met before the cycle (k_cv_up0 ended the loop itself)
__global__ void k_cv_check(DevScalars* sc, CvCheck ck) {
  pdl_wait();
  if (sc->mg_done) return;
  sc->pcur = 1 - sc->pcur;
  cv_check_body(sc, ck);
}

struct CvBlock {
  int lc, D, ncoarse, pre;
  int n[AJ_MAX_LEVELS + 1], m[AJ_MAX_LEVELS + 1];
  int eoff[AJ_MAX_LEVELS + 1], roff[AJ_MAX_LEVELS + 1], voff;   // shared-memory float offsets
  float ax[AJ_MAX_LEVELS + 1], ay[AJ_MAX_LEVELS + 1], g[AJ_MAX_LEVELS + 1];
  const float* r_in;      // rhs of level lc (global)
  float* e_out;           // correction of level lc (global)
  const double* Ainv;     // coarsest inverse, row-major ncoarse^2
  const int* done;
};

// shared-memory footprint of levels lc..D: e with a one-cell zero border and
// r, per level, plus the FP64 vector of the dense coarsest solve
static size_t block_levels_smem(const Layout& L, int lc) {
  size_t s = 0;
  for (int k = lc; k <= L.nlev; ++k)
    s += ((size_t)(L.ln[k] + 2) * (L.lm[k] + 2) + (size_t)L.ln[k] * L.lm[k]) * 4;
  s = (s + 15) & ~(size_t)15;
  const size_t N = (size_t)L.ln[L.nlev] * L.lm[L.nlev];
  return s + N * 8;
}
// whether the coarsest inverse is copied to shared memory (when it fits)
static bool block_prefetch(const Layout& L, int lc) {
  const size_t N = (size_t)L.ln[L.nlev] * L.lm[L.nlev];
  return N <= AJ_MAX_COARSE && block_levels_smem(L, lc) + N * N * 8 <= kBlockSmemMax;
}
size_t converge_block_smem(const Layout& L, int lc) {
  const size_t N = (size_t)L.ln[L.nlev] * L.lm[L.nlev];
  return block_levels_smem(L, lc) + (block_prefetch(L, lc) ? N * N * 8 : 0);
}

// A thread's place in a (rows x w) sweep of the block: column tx, first row
// ty, row stride rs (threads beyond rs * w rows idle).
struct Lane2 {
  int tx, ty, rs;
};
__device__ __forceinline__ Lane2 lane2(int w) {
  Lane2 l;
  l.tx = threadIdx.x % w;
  l.ty = threadIdx.x / w;
  l.rs = blockDim.x / w;
  return l;
}

__device__ __forceinline__ float blk_inv_diag(int i, int j, int n, int m, float ax, float ay,
                                              float g, float inv_int) {
  if (i > 0 && i < n - 1 && j > 0 && j < m - 1) return inv_int;
  float dd = -2.f * (ax + ay);
  if (i == 0) dd += ax;
  if (j == 0) dd += ay;
  if (j == m - 1) dd += ay;
  if (i == n - 1) dd += ax * g;
  return __frcp_rn(dd);
}

// red-black sweeps of one level held in shared memory (E bordered, R not)
__device__ __forceinline__ void blk_sweeps(float* E, const float* R, int n, int m, float ax,
                                           float ay, float g) {
  const int W = m + 2, hw = (m + 1) >> 1;
  const Lane2 q = lane2(hw);
  const float inv_int = 1.f / (-2.f * (ax + ay));
  for (int h = 0; h < 2 * CV_NS; ++h) {
    const int color = h & 1;
    if (q.ty < q.rs) {
      for (int i = q.ty; i < n; i += q.rs) {
        const int j = ((color + i) & 1) + 2 * q.tx;
        if (j >= m) continue;
        const int c = (i + 1) * W + (j + 1);
        const float nb = ax * (E[c + W] + E[c - W]) + ay * (E[c + 1] + E[c - 1]);
        E[c] = (R[i * m + j] - nb) * blk_inv_diag(i, j, n, m, ax, ay, g, inv_int);
      }
    }
    __syncthreads();
  }
}

// Levels lc..D in one block of CV_BLOCK_THREADS threads, every level resident
// in shared memory: pre-smoothing, residual and restriction down to the
// coarsest grid, its FP64 dense solve, prolongation and post-smoothing back
// to level lc.  Replaces 2 (D - lc) launches of the tile kernels by one.
__global__ void __launch_bounds__(CV_BLOCK_THREADS) k_cv_block(CvBlock a) {
  pdl_wait();
  if (*a.done) return;
  extern __shared__ __align__(16) float smf[];
  // level arrays are addressed from smf directly so that every access is a
  // shared-memory access
  auto E = [&](int k) { return smf + a.eoff[k]; };
  auto R = [&](int k) { return smf + a.roff[k]; };
  double* V = reinterpret_cast<double*>(smf + a.voff);
  double* Ainv_s = V + a.ncoarse;
  // start loading the coarsest inverse now, so its latency hides behind the
  // smoothing of the finer levels
  if (a.pre)
    for (int t = threadIdx.x; t < a.ncoarse * a.ncoarse; t += blockDim.x) Ainv_s[t] = a.Ainv[t];
  for (int k = a.lc; k <= a.D; ++k) {
    float* e = E(k);
    const int cnt = (a.n[k] + 2) * (a.m[k] + 2);
    for (int t = threadIdx.x; t < cnt; t += blockDim.x) e[t] = 0.f;
  }
  {
    const int cnt = a.n[a.lc] * a.m[a.lc];
    float* r0 = R(a.lc);
    for (int t = threadIdx.x; t < cnt; t += blockDim.x) r0[t] = ldg(a.r_in + t);
  }
  __syncthreads();
  // down: smooth, residual, restrict (coarse cell = average of 4 fine residuals)
  for (int k = a.lc; k < a.D; ++k) {
    const int n = a.n[k], m = a.m[k], W = m + 2;
    const float ax = a.ax[k], ay = a.ay[k], g = a.g[k];
    blk_sweeps(E(k), R(k), n, m, ax, ay, g);
    const int nc = n >> 1, mc = m >> 1;
    const Lane2 q = lane2(mc);
    const float* e = E(k);
    const float* rk = R(k);
    float* rk1 = R(k + 1);
    if (q.ty < q.rs) {
      for (int I = q.ty; I < nc; I += q.rs) {
        const int J = q.tx;
        float s = 0.f;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int i = 2 * I + (u & 1), j = 2 * J + (u >> 1);
          const int c = (i + 1) * W + (j + 1);
          float dd = -2.f * (ax + ay);
          if (i == 0) dd += ax;
          if (j == 0) dd += ay;
          if (j == m - 1) dd += ay;
          if (i == n - 1) dd += ax * g;
          const float Ae = ax * (e[c + W] + e[c - W]) + ay * (e[c + 1] + e[c - 1]) + dd * e[c];
          s += rk[i * m + j] - Ae;
        }
        rk1[I * mc + J] = 0.25f * s;
      }
    }
    __syncthreads();
  }
  // coarsest: e = A^-1 r in FP64 (one warp per row)
  {
    const int m = a.m[a.D], W = m + 2, N = a.ncoarse;
    const float* rD = R(a.D);
    float* eD = E(a.D);
    for (int t = threadIdx.x; t < N; t += blockDim.x) V[t] = (double)rD[t];
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int row = warp; row < N; row += nw) {
      const double* arow = (a.pre ? Ainv_s : a.Ainv) + (long)row * N;
      double s = 0.0;
      for (int c = lane; c < N; c += 32) s += arow[c] * V[c];
      s = warp_sum(s);
      if (lane == 0) {
        const int i = row / m, j = row - i * m;
        eD[(i + 1) * W + (j + 1)] = (float)s;
      }
    }
    __syncthreads();
  }
  // up: prolong, smooth
  for (int k = a.D - 1; k >= a.lc; --k) {
    const int n = a.n[k], m = a.m[k], W = m + 2;
    const int nc = a.n[k + 1], mc = a.m[k + 1], Wc = mc + 2;
    const float gc = a.g[k + 1];
    const float* Ec = E(k + 1);
    float* Ek = E(k);
    const Lane2 q = lane2(m);
    if (q.ty < q.rs) {
      for (int gi = q.ty; gi < n; gi += q.rs) {
        const int gj = q.tx;
        const int I = gi >> 1, J = gj >> 1;
        const int Ii = (gi & 1) ? I + 1 : I - 1;
        int Jj = (gj & 1) ? J + 1 : J - 1;
        Jj = Jj < 0 ? 0 : (Jj >= mc ? mc - 1 : Jj);
        const float c0 = Ec[(I + 1) * Wc + (J + 1)], cy = Ec[(I + 1) * Wc + (Jj + 1)];
        float cx, cxy;
        if (Ii < 0) {
          cx = c0;
          cxy = cy;
        } else if (Ii >= nc) {
          cx = gc * c0;
          cxy = gc * cy;
        } else {
          cx = Ec[(Ii + 1) * Wc + (J + 1)];
          cxy = Ec[(Ii + 1) * Wc + (Jj + 1)];
        }
        Ek[(gi + 1) * W + (gj + 1)] += (9.f * c0 + 3.f * cx + 3.f * cy + cxy) * (1.f / 16.f);
      }
    }
    __syncthreads();
    blk_sweeps(Ek, R(k), n, m, a.ax[k], a.ay[k], a.g[k]);
  }
  {
    const int n = a.n[a.lc], m = a.m[a.lc], W = m + 2;
    const Lane2 q = lane2(m);
    const float* e0 = E(a.lc);
    if (q.ty < q.rs)
      for (int i = q.ty; i < n; i += q.rs) a.e_out[(long)i * m + q.tx] = e0[(i + 1) * W + q.tx + 1];
  }
}

// ---------------------------------------------------------------- direct coarse solve
// The rediscretised operator of level ld is separable: A = ax Tx (x) I +
// ay I (x) Ty, with Ty the 1-D Neumann-Neumann Laplacian (edge ghosts at both
// walls) and Tx the 1-D operator with an edge ghost at the inlet and the
// outlet ghost g * e_last.  The orthonormal DCT-II basis diagonalises Ty
// (eigenvalues -4 sin^2(pi k / 2m)), so A e = r splits into m independent
// tridiagonal systems (ax Tx + ay lambda_k) e_k = r_k in x, one per cosine
// mode, solved here by parallel cyclic reduction.  The whole coarse part of
// the V-cycle below level ld is replaced by this exact solve: a cosine
// transform (k_cv_dct<true>), the m tridiagonal solves (k_cv_dpcr) and the
// inverse transform (k_cv_dct<false>).
constexpr int CV_DIRECT_MAX_CELLS = 65536;
constexpr int CV_DIRECT_MAX_M = 128;
constexpr int CV_DIRECT_MAX_N = 1024;

struct CvDirect {
  int n, m;
  float ax, g;
  const float* r;      // level-ld rhs [n][m]
  const float* cy;     // cosine basis Cy[k][j] (orthonormal DCT-II), then its transpose
  const float* ly;     // ay * lambda_k
  float2* kk;          // cyclic reduction's multipliers [m][steps][n] (k_cv_dfactor)
  float* dd;           // and its final diagonals [m][n]
  int steps;
  float* rhat;         // mode coefficients of r, transposed [m][n]
  float* ehat;         // mode coefficients of e, transposed [m][n]
  float* e;            // level-ld correction [n][m]
  const int* done;
};

int converge_direct_level(const Layout& L) {
  for (int l = 1; l <= L.nlev; ++l) {
    const long cells = (long)L.ln[l] * L.lm[l];
    if (cells <= CV_DIRECT_MAX_CELLS && L.lm[l] <= CV_DIRECT_MAX_M && L.ln[l] <= CV_DIRECT_MAX_N &&
        L.ln[l] >= 2)
      return l;
  }
  return 0;
}

// The cosine transforms: FWD rhat[k][i] = sum_j Cy[k][j] r[i][j], else
// e[i][j] = sum_k ehat[k][i] Cy[k][j] (with the transposed basis both are row
// by row products).  16 x 32 output tiles, 2 outputs a thread: at 512 x 128
// that is 128 blocks, and since the three kernels of this solve are bound by
// their own latency (one block's staging round, its product and a launch),
// more and lighter blocks win: 32 x 32 tiles with 4-byte reads took 8.0 and 8.3
// us cold, these with 16-byte reads of both panels and of the shared rows 6.6
// and 6.9.
// The basis is staged before the wait for the previous kernel.
constexpr int CV_DI = 16, CV_DC = 32;
constexpr int CV_DK = CV_DIRECT_MAX_M + 4;   // row stride: 16-byte rows, free of bank conflicts
template <bool FWD>
__global__ void __launch_bounds__(256) k_cv_dct(CvDirect a) {
  __shared__ __align__(16) float As[CV_DI][CV_DK];   // a row of r, or a column of ehat
  __shared__ __align__(16) float Cs[CV_DC][CV_DK];   // rows of the basis
  const int n = a.n, m = a.m, m4 = (m + 3) & ~3;
  const int i0 = blockIdx.x * CV_DI, c0 = blockIdx.y * CV_DC;
  const int t = threadIdx.x;
  const float* __restrict__ basis = a.cy + (FWD ? 0 : (long)m * m);
  const bool vec = (m & 3) == 0;   // 16-byte rows (the buffers are 256-byte aligned)
  if (vec) {
    for (int q = t; q < CV_DC * (m >> 2); q += 256) {
      const int row = q / (m >> 2), c = (q - row * (m >> 2)) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c0 + row < m) v = __ldg(reinterpret_cast<const float4*>(basis + (long)(c0 + row) * m + c));
      *reinterpret_cast<float4*>(&Cs[row][c]) = v;
    }
  } else {
    for (int q = t; q < CV_DC * m4; q += 256) {
      const int row = q / m4, c = q - row * m4;
      Cs[row][c] = c0 + row < m && c < m ? ldg(basis + (long)(c0 + row) * m + c) : 0.f;
    }
  }
  pdl_wait();
  if (*a.done) return;
  if (FWD && vec) {
    for (int q = t; q < CV_DI * (m >> 2); q += 256) {
      const int row = q / (m >> 2), c = (q - row * (m >> 2)) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (i0 + row < n) v = __ldg(reinterpret_cast<const float4*>(a.r + (long)(i0 + row) * m + c));
      *reinterpret_cast<float4*>(&As[row][c]) = v;
    }
  } else if (FWD) {
    for (int q = t; q < CV_DI * m4; q += 256) {
      const int row = q / m4, c = q - row * m4;
      As[row][c] = i0 + row < n && c < m ? ldg(a.r + (long)(i0 + row) * m + c) : 0.f;
    }
  } else {   // [mode][row] in global memory: transposed on the way
#pragma unroll 4
    for (int q = t; q < CV_DI * m4; q += 256) {
      const int row = q & (CV_DI - 1), c = q / CV_DI;
      As[row][c] = i0 + row < n && c < m ? ldg(a.ehat + (long)c * n + i0 + row) : 0.f;
    }
  }
  __syncthreads();
  // thread: row t & 15 and columns t >> 4 and 16 + (t >> 4) forward (rhat is
  // stored row by row), else column t & 31 and rows t >> 5 and 8 + (t >> 5)
  const int ri = FWD ? (t & 15) : (t >> 5), rc = FWD ? (t >> 4) : (t & 31);
  const float* pa0 = As[ri];
  const float* pa1 = As[FWD ? ri : ri + 8];
  const float* pc0 = Cs[rc];
  const float* pc1 = Cs[FWD ? rc + 16 : rc];
  float s0 = 0.f, s1 = 0.f;
#pragma unroll 8
  for (int j = 0; j < m4; j += 4) {
    const float4 x0 = *reinterpret_cast<const float4*>(pa0 + j);
    const float4 y0 = *reinterpret_cast<const float4*>(pc0 + j);
    const float4 x1 = FWD ? x0 : *reinterpret_cast<const float4*>(pa1 + j);
    const float4 y1 = FWD ? *reinterpret_cast<const float4*>(pc1 + j) : y0;
    s0 = fmaf(x0.x, y0.x, s0);
    s1 = fmaf(x1.x, y1.x, s1);
    s0 = fmaf(x0.y, y0.y, s0);
    s1 = fmaf(x1.y, y1.y, s1);
    s0 = fmaf(x0.z, y0.z, s0);
    s1 = fmaf(x1.z, y1.z, s1);
    s0 = fmaf(x0.w, y0.w, s0);
    s1 = fmaf(x1.w, y1.w, s1);
  }
  if (FWD) {
    const int i = i0 + ri, k = c0 + rc;
    if (i < n && k < m) a.rhat[(long)k * n + i] = s0;
    if (i < n && k + 16 < m) a.rhat[(long)(k + 16) * n + i] = s1;
  } else {
    const int i = i0 + ri, j = c0 + rc;
    if (i < n && j < m) a.e[(long)i * m + j] = s0;
    if (i + 8 < n && j < m) a.e[(long)(i + 8) * m + j] = s1;
  }
}

// Parallel cyclic reduction of (ax Tx + ay lambda_k) ehat_k = rhat_k, n
// unknowns along x, one block per cosine mode k.  Everything but the
// right-hand side depends on the grid alone, so aj_prepare runs the
// reduction of the matrix once and keeps each step's two multipliers and the
// final diagonals (k_cv_dfactor): a solve then reads them in one round trip,
// before the wait for the transform, and a step is two products where it was
// two divisions and eight shared reads.
__global__ void __launch_bounds__(1024) k_cv_dfactor(CvDirect a) {
  extern __shared__ __align__(16) float sh[];
  const int n = a.n, k = blockIdx.x, i = threadIdx.x;
  float *Ac = sh, *Bc = Ac + n, *Cc = Bc + n, *An = Cc + n, *Bn = An + n, *Cn = Bn + n;
  if (i < n) {
    float dx = -2.f;
    if (i == 0) dx += 1.f;
    if (i == n - 1) dx += a.g;
    Ac[i] = i > 0 ? a.ax : 0.f;
    Cc[i] = i < n - 1 ? a.ax : 0.f;
    Bc[i] = fmaf(a.ax, dx, ldg(a.ly + k));
  }
  __syncthreads();
  for (int st = 1, s = 0; st < n; st <<= 1, ++s) {
    if (i < n) {
      float an = 0.f, bn = Bc[i], cn = 0.f, k1 = 0.f, k2 = 0.f;
      if (i - st >= 0) {
        k1 = Ac[i] / Bc[i - st];
        an = -Ac[i - st] * k1;
        bn -= Cc[i - st] * k1;
      }
      if (i + st < n) {
        k2 = Cc[i] / Bc[i + st];
        cn = -Cc[i + st] * k2;
        bn -= Ac[i + st] * k2;
      }
      An[i] = an;
      Bn[i] = bn;
      Cn[i] = cn;
      a.kk[((long)k * a.steps + s) * n + i] = make_float2(k1, k2);
    }
    __syncthreads();
    float* t;
    t = Ac; Ac = An; An = t;
    t = Bc; Bc = Bn; Bn = t;
    t = Cc; Cc = Cn; Cn = t;
  }
  if (i < n) a.dd[(long)k * n + i] = Bc[i];
}

template <int STEPS>
__global__ void __launch_bounds__(1024) k_cv_dpcr(CvDirect a) {
  __shared__ float D[2][CV_DIRECT_MAX_N];
  const int n = a.n, k = blockIdx.x, i = threadIdx.x;
  const bool in = i < n;
  float2 kk[STEPS];
  float dd = 1.f;
#pragma unroll
  for (int s = 0; s < STEPS; ++s)
    kk[s] = in ? __ldg(a.kk + ((long)k * STEPS + s) * n + i) : make_float2(0.f, 0.f);
  if (in) dd = ldg(a.dd + (long)k * n + i);
  pdl_wait();
  if (*a.done) return;
  float d = in ? ldg(a.rhat + (long)k * n + i) : 0.f;
#pragma unroll
  for (int s = 0; s < STEPS; ++s) {
    const int st = 1 << s;
    float* b = D[s & 1];
    if (in) b[i] = d;
    __syncthreads();
    if (in && i - st >= 0) d -= b[i - st] * kk[s].x;
    if (in && i + st < n) d -= b[i + st] * kk[s].y;
  }
  if (in) a.ehat[(long)k * n + i] = d / dd;
}

static int direct_steps(int n) {
  int s = 0;
  for (int st = 1; st < n; st <<= 1) ++s;
  return s;
}
size_t converge_direct_floats(int n, int m) {   // the multipliers, then the diagonals
  return (size_t)n * m * (2 * direct_steps(n) + 1);
}

template <int STEPS>
static void dpcr_launch(const CvDirect& d, cudaStream_t st) {
  if (d.steps == STEPS)
    launch_pdl(true, k_cv_dpcr<STEPS>, dim3(d.m), dim3(cdiv(d.n, 32) * 32), 0, st, d);
  else if constexpr (STEPS > 1)
    dpcr_launch<STEPS - 1>(d, st);
}

static void direct_launch(const CvDirect& d, cudaStream_t st) {
  const dim3 g(cdiv(d.n, CV_DI), cdiv(d.m, CV_DC));
  launch_pdl(true, k_cv_dct<true>, dim3(g), dim3(256), 0, st, d);
  dpcr_launch<10>(d, st);   // n <= CV_DIRECT_MAX_N = 2^10
  launch_pdl(true, k_cv_dct<false>, dim3(g), dim3(256), 0, st, d);
}

static CvDirect direct_args(const AjStepParams& p, const Layout& L, void* ws, const int* done);

// ---------------------------------------------------------------- set-up / solve
// The initial double-FP32 state, outlet row pinned; a block per 8 rows.
// With a history (warm start AJ_WARM_EXTRAPOLATE) of two solutions
// p = p1 + (dt / dt1) (p1 - p2), of one solution p = p1; else p0 (or 0).
struct CvHist {
  const float* h;   // two slots of N hi values followed by N lo values; null: none
  long N;
};
constexpr int CV_ROWS = 8;   // rows per block of the whole-grid kernels (unrolled)

// The extrapolation history as this solve sees it: a solve that finished
// since the last commit (hist_pending) has filed its solution in the other
// slot.  The last block of k_cv_resid commits the rotation.
struct HistView {
  int cur, n;
  float dtp;
};
__device__ __forceinline__ HistView hist_view(const DevScalars* sc) {
  // all five fields loaded unconditionally (one round trip), then selected
  const int pend = sc->hist_pending, cur = sc->hist_cur, n = sc->hist_n;
  const float dtl = sc->dt_last, dtp = sc->dt_prev;
  HistView h;
  if (pend) {
    h.cur = 1 - cur;
    h.n = n < 2 ? n + 1 : 2;
    h.dtp = dtl;
  } else {
    h.cur = cur;
    h.n = n;
    h.dtp = dtp;
  }
  return h;
}
__global__ void __launch_bounds__(256) k_cv_init(const float* __restrict__ p0,
                                                 float* __restrict__ ps, int n, int m, CvHist hs,
                                                 const DevScalars* sc) {
  pdl_wait();
  const long N = (long)n * m;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const HistView hv = hist_view(sc);
  const int hn = hs.h ? hv.n : 0;
  const float* __restrict__ h1 = hs.h ? hs.h + (long)hv.cur * 2 * N : nullptr;
  const float* __restrict__ h2 = hs.h ? hs.h + (long)(1 - hv.cur) * 2 * N : nullptr;
  float ratio = 1.f;
  if (hn >= 2 && sc->dt > 0.f && hv.dtp > 0.f) ratio = sc->dt / hv.dtp;
  const int i0 = blockIdx.y * CV_ROWS;
  // every row's loads first (the stores below would otherwise hold each
  // row's loads back behind the previous row's stores)
  float a_hi[CV_ROWS], a_lo[CV_ROWS], b_hi[CV_ROWS], b_lo[CV_ROWS];
#pragma unroll
  for (int r = 0; r < CV_ROWS; ++r) {
    const int i = i0 + r;
    const long k = (long)i * m + j;
    a_hi[r] = a_lo[r] = b_hi[r] = b_lo[r] = 0.f;
    if (i < n - 1) {
      if (hn >= 1) {
        a_hi[r] = h1[k];
        a_lo[r] = h1[N + k];
      } else if (p0) {
        a_hi[r] = p0[k];
      }
      if (hn >= 2) {
        b_hi[r] = h2[k];
        b_lo[r] = h2[N + k];
      }
    }
  }
#pragma unroll
  for (int r = 0; r < CV_ROWS; ++r) {
    const int i = i0 + r;
    if (i < n) {
      const long k = (long)i * m + j;
      df v{a_hi[r], a_lo[r]};
      if (hn >= 2 && i != n - 1) {
        const df a = v, b{b_hi[r], b_lo[r]};
        v = df_add(a, df_mul(df{ratio, 0.f}, df_add(a, df_neg(b))));
      }
      ps[k] = v.hi;
      ps[N + k] = v.lo;
    }
  }
}

// Residual of the reference operator before the first cycle (double-FP32)
// and the FP64 norms of r and b; a thread a column pair over four rows with
// 8-byte reads and paired arithmetic, a block bands of 32 rows by 64 columns.
// What bounds it: a band's chain of reads and double-FP32 arithmetic at 24 warps
// an SM.  Cold, a thread one column over eight rows -> this: 2048x512 13.4 -> 12
// us, 4096x2048 60 -> 43 (51 with a block for every band).
constexpr int CVR_ROWS = 4;
constexpr unsigned CVR_BLOCKS = 456;   // three an SM
__global__ void __launch_bounds__(256) k_cv_resid(const float* __restrict__ ps,
                                                  const float* __restrict__ b,
                                                  float* __restrict__ r, int n, int m, DfCoef co,
                                                  DevScalars* sc, double rtol) {
  pdl_wait();
  const long N = (long)n * m;
  const df ax{co.axh, co.axl}, ay{co.ayh, co.ayl};
  df sum{0.f, 0.f}, sumb{0.f, 0.f};
  const int j = 2 * (blockIdx.x * 32 + (threadIdx.x & 31));
  // a block walks bands of 32 rows: its three atomics on the scalars, and not
  // its loads, set the time when every band had a block of its own
  for (int i0 = (blockIdx.y * 8 + (threadIdx.x >> 5)) * CVR_ROWS; j < m && i0 < n;
       i0 += gridDim.y * 8 * CVR_ROWS) {
    float acc = 0.f, accb = 0.f;
    auto pair = [&](const float* f, long k) { return *reinterpret_cast<const float2*>(f + k); };
    // all loads first: the state at rows i0 - 1 .. i0 + 4, the pair's column
    // neighbours and b
    df2 c[CVR_ROWS + 2];
    df lf[CVR_ROWS], rt[CVR_ROWS];
    float2 bv[CVR_ROWS];
#pragma unroll
    for (int q = 0; q < CVR_ROWS + 2; ++q) {
      const int i = i0 - 1 + q;
      c[q].hi = c[q].lo = f2(0.f);
      if (i >= 0 && i < n) {
        const long k = (long)i * m + j;
        c[q].hi = pair(ps, k);
        c[q].lo = pair(ps, N + k);
      }
    }
#pragma unroll
    for (int q = 0; q < CVR_ROWS; ++q) {
      const long k = (long)(i0 + q) * m + j;
      bv[q] = f2(0.f);
      lf[q] = rt[q] = df{0.f, 0.f};
      if (i0 + q < n - 1) {
        bv[q] = pair(b, k);
        if (j > 0) lf[q] = df{ps[k - 1], ps[N + k - 1]};
        if (j + 2 < m) rt[q] = df{ps[k + 2], ps[N + k + 2]};
      }
    }
#pragma unroll
    for (int q = 0; q < CVR_ROWS; ++q) {
      const int i = i0 + q;
      if (i >= n) break;
      float2 rr = f2(0.f);
      if (i != n - 1) {
        const df2 x = c[q + 1], xm = i > 0 ? c[q] : x;
        // the neighbours' edge ghosts are the cell itself
        const df2 yp{make_float2(x.hi.y, j + 2 < m ? rt[q].hi : x.hi.y),
                     make_float2(x.lo.y, j + 2 < m ? rt[q].lo : x.lo.y)};
        const df2 ym{make_float2(j > 0 ? lf[q].hi : x.hi.x, x.hi.x),
                     make_float2(j > 0 ? lf[q].lo : x.lo.x, x.lo.x)};
        const df2 res = df2_residual(bv[q], x, c[q + 2], xm, yp, ym, ax, ay);
        rr = add2(res.hi, res.lo);
        accb = fmaf(bv[q].x, bv[q].x, accb);
        accb = fmaf(bv[q].y, bv[q].y, accb);
      }
      cp_st2(r + (long)i * m + j, rr);
      acc = fmaf(rr.x, rr.x, acc);
      acc = fmaf(rr.y, rr.y, acc);
    }
    sum = df_add(sum, df{acc, 0.f});
    sumb = df_add(sumb, df{accb, 0.f});
  }
  const double t = block_sum_df(sum), tb = block_sum_df(sumb);
  if (threadIdx.x == 0) {
    atomicAdd(&sc->acc[0], t);
    atomicAdd(&sc->acc[1], tb);
  }
  // the last block: commit the history rotation, reset the solve's counters
  // and run the test before the first cycle (the guess may already satisfy rtol)
  __shared__ int am_last;
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned int ticket = atomicAdd(&sc->red_count, 1u);
    am_last = ticket == gridDim.x * gridDim.y - 1;
  }
  __syncthreads();
  if (am_last && threadIdx.x == 0) {
    __threadfence();
    // every field first, then the stores (see cv_check_body)
    const HistView hv = hist_view(sc);
    const double a0 = sc->acc[0], a1 = sc->acc[1];
    // ||r|| <= rtol ||b|| (rtol alone for b = 0), in squares
    const double target = rtol * rtol * (a1 > 0.0 ? a1 : 1.0);
    int err = AJ_OK, done = 0;
    if (!isfinite(a0) || !isfinite(target)) {
      err = AJ_ERR_NONFINITE;
      done = 1;
    } else if (a0 <= target) {
      done = 1;
    }
    sc->hist_cur = hv.cur;
    sc->hist_n = hv.n;
    sc->dt_prev = hv.dtp;
    sc->hist_pending = 0;
    sc->red_count = 0u;
    sc->mg_cycles = 0;
    sc->loops = 0;
    sc->pcur = 0;
    sc->bsq = a1;
    sc->target = target;
    sc->abs_sq = a0;
    sc->acc[0] = 0.0;
    sc->acc[1] = 0.0;
    sc->err = err;
    sc->mg_done = done;
  }
}

// p = hi + lo; with a history, the state also goes to the free slot (the
// next solve's k_cv_resid makes it the latest); thread 0 files the statistics.
// V: floats a thread, 4 where p is 16-byte aligned (N is a multiple of 4).
template <int V>
__global__ void __launch_bounds__(256) k_cv_out(PState ps, DevScalars* sc, float* __restrict__ p,
                                                long N, float* hist, AjStats* stats) {
  pdl_wait();
  const long k = (blockIdx.x * (long)blockDim.x + threadIdx.x) * V;
  const float* src = sc->pcur ? ps.b : ps.a;
  if (k < N) {
    alignas(16) float hi[V], lo[V], out[V];
    auto get = [](float* v, const float* f) {
      if constexpr (V == 4) *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(f);
      else v[0] = f[0];
    };
    auto put = [](float* f, const float* v) {
      if constexpr (V == 4) *reinterpret_cast<float4*>(f) = *reinterpret_cast<const float4*>(v);
      else f[0] = v[0];
    };
    get(hi, src + k);
    get(lo, src + N + k);
#pragma unroll
    for (int q = 0; q < V; ++q) out[q] = hi[q] + lo[q];
    put(p + k, out);
    if (hist) {
      float* dst = hist + (long)(1 - sc->hist_cur) * 2 * N;
      put(dst + k, hi);
      put(dst + N + k, lo);
    }
  }
  if (k == 0) {
    // every field first, then the stores (stats may alias nothing the
    // compiler can prove, so interleaved each load waited for a store)
    const int cycles = sc->mg_cycles, done = sc->mg_done, err = sc->err;
    const double bsq = sc->bsq, abs_sq = sc->abs_sq;
    const double bnorm = sqrt(bsq), rel = sqrt(abs_sq) / (bnorm > 0.0 ? bnorm : 1.0);
    const float dt = sc->dt;
    if (hist) {
      sc->hist_pending = 1;
      sc->dt_last = dt;
    }
    if (stats) {
      stats->cycles = cycles;
      stats->converged = done && err == AJ_OK;   // the tolerance met, not just the loop ended
      stats->err = err;
      stats->pad = 0;
      stats->rel_residual = rel;
      stats->rhs_norm = bnorm;
      stats->dt = dt;
      stats->abs_residual_sq = abs_sq;
    }
  }
}

static CvBlock block_args(const AjStepParams& p, const Layout& L, void* ws, const int* done) {
  CvBlock a;
  memset(&a, 0, sizeof(a));
  a.lc = L.lc;
  a.D = L.nlev;
  a.ncoarse = L.ncoarse;
  a.pre = block_prefetch(L, L.lc) ? 1 : 0;
  size_t off = 0;   // floats; the same order as block_levels_smem
  for (int k = L.lc; k <= L.nlev; ++k) {
    a.eoff[k] = (int)off;
    off += (size_t)(L.ln[k] + 2) * (L.lm[k] + 2);
    a.roff[k] = (int)off;
    off += (size_t)L.ln[k] * L.lm[k];
  }
  a.voff = (int)((off + 3) & ~(size_t)3);
  for (int k = 0; k <= L.nlev; ++k) {
    CvLvl c = cv_level(p, L, k);
    a.n[k] = c.n;
    a.m[k] = c.m;
    a.ax[k] = c.ax;
    a.ay[k] = c.ay;
    a.g[k] = c.g;
  }
  a.r_in = at<float>(ws, L.B[L.lc]);
  a.e_out = at<float>(ws, L.T[L.lc]);
  a.Ainv = at<double>(ws, L.cinv);
  a.done = done;
  return a;
}

static CvDirect direct_args(const AjStepParams& p, const Layout& L, void* ws, const int* done) {
  CvDirect d;
  const CvLvl c = cv_level(p, L, L.ld);
  d.n = c.n;
  d.m = c.m;
  d.ax = c.ax;
  d.g = c.g;
  d.r = at<float>(ws, L.B[L.ld]);
  d.cy = at<float>(ws, L.dcy);
  d.ly = at<float>(ws, L.dly);
  d.steps = direct_steps(d.n);
  d.kk = at<float2>(ws, L.dpf);
  d.dd = at<float>(ws, L.dpf) + 2 * (size_t)d.n * d.m * d.steps;
  d.rhat = at<float>(ws, L.X[L.ld]);
  d.ehat = at<float>(ws, L.dtmp);
  d.e = at<float>(ws, L.T[L.ld]);
  d.done = done;
  return d;
}

static PState pstate(const Layout& L, void* ws) {
  return PState{at<float>(ws, L.p64), at<float>(ws, L.p64b)};
}

// The shape of an n x m level: regions of 48 rows (0), of 32 rows (1: more and
// shorter blocks, where those are no more than the SMs) or of 64 rows (2, for
// the autotuner; level 0's up kernel has 48).  Level-0 down and up kernels
// together in a stream, us, 48 / 32 / 64 rows: 256x64 6.7 / 6.0 / 6.9, 512x96
// 6.8 / 6.0 / 7.1, 1024x256 7.0 / 7.7 / 7.2, 2048x512 16.1 / 16.1 / 16.4,
// 4096x2048 84 / 88 / 87.  crowd: how many such levels run side by side (an
// ensemble's instances by their cells): all their blocks share the SMs.
constexpr int CV_TILE_VARIANTS = 3, CV_SMALL_BLOCKS = 152;
static int cv_shape(int n, int m, float crowd = 1.f) {
  using T = CpTile<8, CP_H_DOWN>;
  return crowd * cdiv(n, T::OUT_I) * cdiv(m, T::OUT_J) <= CV_SMALL_BLOCKS ? 1 : 0;
}

template <int G, int H>
static dim3 tiles(const CvLvl& c) {
  return dim3(cdiv(c.m, CpTile<G, H>::OUT_J), cdiv(c.n, CpTile<G, H>::OUT_I));
}

// level-0 kernels with G row groups
template <int G>
static void level0_down(const CvLvl& c, const Layout& L, void* ws, const int* done,
                        cudaStream_t st) {
  const DevScalars* sc = at<DevScalars>(ws, 0);
  launch_pdl(true, k_cv_down<G>, tiles<G, CP_H_DOWN>(c), dim3(CP_PAIRS, G), 0, st, c,
             at<float>(ws, L.B[0]), at<float>(ws, L.T[0]), &sc->pcur, at<float>(ws, L.X[0]),
             at<float>(ws, L.B[1]), done);
}
template <int G>
static void level0_up(const AjStepParams& p, const CvLvl& c, const Layout& L, void* ws,
                      DevScalars* sc, const CvCheck& ck, int profile, cudaStream_t st) {
  launch_pdl(true, k_cv_up0<G>, tiles<G, CP_H_UP>(c), dim3(CP_PAIRS, G), 0, st, c,
             PState{at<float>(ws, L.B[0]), at<float>(ws, L.T[0])}, at<float>(ws, L.X[0]),
             at<float>(ws, L.T[1]), L.ln[1], L.lm[1], (float)ghost_factor(1), pstate(L, ws),
             at<float>(ws, L.b0), sc, df_coef(1.0 / (p.dx * p.dx), 1.0 / (p.dy * p.dy)), ck,
             profile);
}
// variant v of a level: 0 the shape that its size gives, the others the
// autotuner's alternatives
static int variant_shape(int v, const CvLvl& c) { return (cv_shape(c.n, c.m) + v) % CV_TILE_VARIANTS; }
static void level0_down_s(int sh, const CvLvl& c, const Layout& L, void* ws, const int* done,
                          cudaStream_t st) {
  if (sh == 2) level0_down<16>(c, L, ws, done, st);
  else if (sh == 1) level0_down<8>(c, L, ws, done, st);
  else level0_down<12>(c, L, ws, done, st);
}
static void level0_up_s(int sh, const AjStepParams& p, const CvLvl& c, const Layout& L, void* ws,
                        DevScalars* sc, const CvCheck& ck, int profile, cudaStream_t st) {
  if (sh == 1) level0_up<8>(p, c, L, ws, sc, ck, profile, st);
  else level0_up<12>(p, c, L, ws, sc, ck, profile, st);
}

// the kernels of a level >= 1 in its size's shape
template <int G>
static void level_down(const CvLvl& c, const Layout& L, void* ws, int l, const int* done,
                       cudaStream_t st) {
  launch_pdl(true, k_cv_down<G>, tiles<G, CP_H_DOWN>(c), dim3(CP_PAIRS, G), 0, st, c,
             at<float>(ws, L.B[l]), nullptr, done, at<float>(ws, L.X[l]),
             at<float>(ws, L.B[l + 1]), done);
}
template <int G>
static void level_up(const CvLvl& c, const Layout& L, void* ws, int l, const int* done,
                     cudaStream_t st) {
  launch_pdl(true, k_cv_up<G>, tiles<G, CP_H_UP>(c), dim3(CP_PAIRS, G), 0, st, c,
             at<float>(ws, L.B[l]), at<float>(ws, L.X[l]), at<float>(ws, L.T[l + 1]), L.ln[l + 1],
             L.lm[l + 1], (float)ghost_factor(l + 1), at<float>(ws, L.T[l]), done);
}

// one refinement iteration
// Whether a cycle's test has a kernel of its own.  In the last block of
// k_cv_up0 it makes every block wait at its end for a fence and a counter, and
// the next cycle for that block's chain.  Four cycles in line, us, in the last
// block -> apart: 256x64 80.7 -> 80.3, 512x128 86.7 -> 82.4, 1024x256 99.0 ->
// 94.9, 2048x512 163 -> 160, 4096x1024 386 -> 377, 4096x2048 641 -> 632.  Beside
// other instances (crowd) the extra launch costs what it saves.  (The sums on
// 64 addresses instead of one: slower, 1024x256 103, 4096x2048 638 - the FP64
// sum of the 64 outweighs the atomics.)
int converge_check_apart(const Layout& L) { return L.crowd <= 1.f; }

static void cv_body(const AjStepParams& p, const Layout& L, void* ws,
                    cudaGraphConditionalHandle h, int use_handle, cudaStream_t st) {
  DevScalars* sc = at<DevScalars>(ws, 0);
  const int* done = &sc->mg_done;
  const int lc = L.lc;
  // level 0: the shape that the autotuner took instead of the rule's, or the rule's
  const CvLvl c0 = cv_level(p, L, 0);
  const int tuned = tile_variant(p.nx, p.ny);
  const int sh0 = tuned ? variant_shape(tuned, c0) : cv_shape(c0.n, c0.m, L.crowd);
  for (int l = 0; l < lc; ++l) {
    CvLvl c = cv_level(p, L, l);
    const int sh = cv_shape(c.n, c.m, L.crowd);
    if (l == 0) level0_down_s(sh0, c, L, ws, done, st);
    else if (sh == 1) level_down<8>(c, L, ws, l, done, st);
    else level_down<12>(c, L, ws, l, done, st);
  }
  if (L.ld > 0) {
    direct_launch(direct_args(p, L, ws, done), st);
  } else {
    k_cv_block<<<1, CV_BLOCK_THREADS, converge_block_smem(L, lc), st>>>(block_args(p, L, ws, done));
  }
  for (int l = lc - 1; l >= 1; --l) {
    CvLvl c = cv_level(p, L, l);
    const int sh = cv_shape(c.n, c.m, L.crowd);
    if (sh == 1) level_up<8>(c, L, ws, l, done, st);
    else level_up<12>(c, L, ws, l, done, st);
  }
  const CvCheck ck{p.max_cycles, use_handle, h, converge_check_apart(L)};
  level0_up_s(sh0, p, c0, L, ws, sc, ck, 0, st);
  if (ck.apart) launch_pdl(true, k_cv_check, dim3(1), dim3(1), 0, st, sc, ck);
}

// Cycles recorded in line before the while node.  An iteration of the node
// costs ~4 us beyond its kernels (a cycle at 2048x512 49 us in line, 53 us in
// the node), a cycle skipped in line ~1 us a kernel, so as many are unrolled as
// nearly every solve runs: two from a warm start (two or three run), four
// from zero (four or five).  A solve that its guess already meets pays for it,
// us, in the node -> in line: from zero with no right-hand side 256x64 42 -> 56,
// 2048x512 54 -> 88, warm 41 -> 44, 53 -> 66; one with one cycle to run gains
// (warm, 60 -> 50, 102 -> 84).
constexpr int CV_INLINE_WARM = 2, CV_INLINE_ZERO = 4;
int converge_inline_cycles(const AjStepParams& p) {
  return std::min(p.warm_start == AJ_WARM_ZERO ? CV_INLINE_ZERO : CV_INLINE_WARM, p.max_cycles);
}

static cudaStream_t side_stream() {
  static cudaStream_t s = nullptr;
  if (!s) cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  return s;
}

// the initial double-FP32 state (needs the step's dt and the history, not
// the rhs: the step runs it beside the predictor)
int converge_init(const AjStepParams& p, const Layout& L, void* ws, const float* p0,
                  cudaStream_t st) {
  DevScalars* sc = at<DevScalars>(ws, 0);
  const long N = (long)p.nx * p.ny;
  const PState ps = pstate(L, ws);
  const dim3 rgrid(cdiv(p.ny, 256), cdiv(p.nx, CV_ROWS));
  const bool extrap = p.warm_start == AJ_WARM_EXTRAPOLATE && L.hist;
  CvHist hs{extrap ? at<float>(ws, L.hist) : nullptr, N};
  launch_pdl(true, k_cv_init, dim3(rgrid), dim3(256), 0, st, p.warm_start ? p0 : nullptr, ps.a,
             p.nx, p.ny, hs, (const DevScalars*)sc);
  return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

int converge_solve(const AjStepParams& p, const Layout& L, void* ws, const float* p0,
                   float* pout, cudaStream_t st, const NnWarm* nn, AjStats* stats,
                   bool init_done) {
  DevScalars* sc = at<DevScalars>(ws, 0);
  const long N = (long)p.nx * p.ny;
  const PState ps = pstate(L, ws);
  const dim3 rgrid(cdiv(p.ny, 256), cdiv(p.nx, CV_ROWS));
  const bool extrap = p.warm_start == AJ_WARM_EXTRAPOLATE && L.hist;
  if (!init_done) {
    const int rc = converge_init(p, L, ws, p0, st);
    if (rc != AJ_OK) return rc;
  }
  if (nn && nn->packed) {
    const int rc = nn_correct_state(p, L, ws, at<float>(ws, L.b0), *nn, ps.a, st);
    if (rc != AJ_OK) return rc;
  }
  launch_pdl(true, k_cv_resid, dim3(cdiv(p.ny, 64), std::min<unsigned>(cdiv(p.nx, 8 * CVR_ROWS),
                                                             std::max(1u, CVR_BLOCKS / (unsigned)cdiv(p.ny, 64)))),
             dim3(256), 0, st, ps.a, at<float>(ws, L.b0),
             at<float>(ws, L.B[0]), p.nx, p.ny, df_coef(1.0 / (p.dx * p.dx), 1.0 / (p.dy * p.dy)),
             sc, p.mg_rtol);

  cudaStreamCaptureStatus cs;
  unsigned long long id;
  cudaGraph_t g;
  const cudaGraphNode_t* deps;
  const cudaGraphEdgeData* ed;
  size_t nd;
  if (cudaStreamGetCaptureInfo(st, &cs, &id, &g, &deps, &ed, &nd) != cudaSuccess)
    return AJ_ERR_CUDA;
  if (cs != cudaStreamCaptureStatusActive) {
    // eager launches (profiling mode): a fixed number of loop bodies, each
    // skipping its work once the target is met
    int unroll = eager_unroll(p.max_cycles);
    for (int k = 0; k < unroll; ++k) cv_body(p, L, ws, 0, 0, st);
  } else {
    // the refinement loop: the first cycles in line (each of a cycle's
    // kernels skips its work once the target is met), the others in a while
    // node appended to the graph being captured
    cudaGraphConditionalHandle h;
    if (cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault) != cudaSuccess)
      return AJ_ERR_CUDA;
    for (int k = 0; k < converge_inline_cycles(p); ++k) cv_body(p, L, ws, h, 1, st);
    if (cudaStreamGetCaptureInfo(st, &cs, &id, &g, &deps, &ed, &nd) != cudaSuccess)
      return AJ_ERR_CUDA;
    // the params union has no default constructor: zero-initialised storage
    alignas(cudaGraphNodeParams) unsigned char npbuf[sizeof(cudaGraphNodeParams)];
    memset(npbuf, 0, sizeof(npbuf));
    cudaGraphNodeParams& np = *reinterpret_cast<cudaGraphNodeParams*>(npbuf);
    np.type = cudaGraphNodeTypeConditional;
    np.conditional.handle = h;
    np.conditional.type = cudaGraphCondTypeWhile;
    np.conditional.size = 1;
    cudaGraphNode_t node;
    if (cudaGraphAddNode(&node, g, deps, ed, nd, &np) != cudaSuccess) return AJ_ERR_CUDA;
    if (cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1,
                                            cudaStreamSetCaptureDependencies) != cudaSuccess)
      return AJ_ERR_CUDA;
    cudaGraph_t body = np.conditional.phGraph_out[0];
    cudaStream_t side = side_stream();
    if (cudaStreamBeginCaptureToGraph(side, body, nullptr, nullptr, 0,
                                      cudaStreamCaptureModeRelaxed) != cudaSuccess)
      return AJ_ERR_CUDA;
    cv_body(p, L, ws, h, 1, side);
    cudaGraph_t out;
    if (cudaStreamEndCapture(side, &out) != cudaSuccess) return AJ_ERR_CUDA;
  }
  float* hist = extrap ? at<float>(ws, L.hist) : nullptr;
  if (N % 4 == 0 && (reinterpret_cast<uintptr_t>(pout) & 15) == 0)
    launch_pdl(true, k_cv_out<4>, dim3(cdiv(N, 1024)), dim3(256), 0, st, ps, sc, pout, N, hist, stats);
  else
    launch_pdl(true, k_cv_out<1>, dim3(cdiv(N, 256)), dim3(256), 0, st, ps, sc, pout, N, hist, stats);
  return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

// dense matrix of the coarsest converging-mode operator, inverted on the host
static bool coarse_inverse(const AjStepParams& p, const Layout& L, std::vector<double>& inv) {
  const int l = L.nlev, n = L.ln[l], m = L.lm[l], N = n * m;
  double hx = p.dx * (double)(1 << l), hy = p.dy * (double)(1 << l);
  double ax = 1.0 / (hx * hx), ay = 1.0 / (hy * hy), g = ghost_factor(l);
  std::vector<double> A((size_t)N * N, 0.0);
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < m; ++j) {
      int r = i * m + j;
      double d = -2.0 * (ax + ay);
      if (i == 0) d += ax; else A[(size_t)r * N + (i - 1) * m + j] += ax;
      if (i == n - 1) d += ax * g; else A[(size_t)r * N + (i + 1) * m + j] += ax;
      if (j == 0) d += ay; else A[(size_t)r * N + i * m + j - 1] += ay;
      if (j == m - 1) d += ay; else A[(size_t)r * N + i * m + j + 1] += ay;
      A[(size_t)r * N + r] += d;
    }
  inv.assign((size_t)N * N, 0.0);
  for (int i = 0; i < N; ++i) inv[(size_t)i * N + i] = 1.0;
  for (int c = 0; c < N; ++c) {          // Gauss-Jordan with partial pivoting
    int piv = c;
    for (int r = c + 1; r < N; ++r)
      if (fabs(A[(size_t)r * N + c]) > fabs(A[(size_t)piv * N + c])) piv = r;
    if (fabs(A[(size_t)piv * N + c]) < 1e-300) return false;
    if (piv != c)
      for (int k = 0; k < N; ++k) {
        std::swap(A[(size_t)c * N + k], A[(size_t)piv * N + k]);
        std::swap(inv[(size_t)c * N + k], inv[(size_t)piv * N + k]);
      }
    double s = 1.0 / A[(size_t)c * N + c];
    for (int k = 0; k < N; ++k) {
      A[(size_t)c * N + k] *= s;
      inv[(size_t)c * N + k] *= s;
    }
    for (int r = 0; r < N; ++r) {
      if (r == c) continue;
      double f = A[(size_t)r * N + c];
      if (f == 0.0) continue;
      for (int k = 0; k < N; ++k) {
        A[(size_t)r * N + k] -= f * A[(size_t)c * N + k];
        inv[(size_t)r * N + k] -= f * inv[(size_t)c * N + k];
      }
    }
  }
  return true;
}

int converge_first_block_level(const Layout& L) {
  // the coarsest level always; finer ones while they are small enough and fit
  int lc = L.nlev;
  for (int l = L.nlev - 1; l >= 1; --l) {
    if ((long)L.ln[l] * L.lm[l] > CV_BLOCK_MAX_CELLS) break;
    if (L.lm[l] > CV_BLOCK_THREADS) break;      // one row per pass of the block
    if (converge_block_smem(L, l) > kBlockSmemMax) break;
    lc = l;
  }
  return lc;
}

int converge_prepare(const AjStepParams& p, const Layout& L, void* ws, cudaStream_t st) {
  std::vector<double> inv;
  if (!coarse_inverse(p, L, inv)) return AJ_ERR_PARAM;
  std::vector<float> cy, ly;
  if (L.ld > 0) {
    // orthonormal DCT-II basis of the level-ld Neumann-Neumann y operator and
    // its eigenvalues times 1/hy^2
    const int m = L.lm[L.ld];
    const double hy = p.dy * (double)(1 << L.ld), ay = 1.0 / (hy * hy);
    const double pi = 3.14159265358979323846;
    cy.resize(2 * (size_t)m * m);
    ly.resize(m);
    for (int k = 0; k < m; ++k) {
      const double sk = k == 0 ? sqrt(1.0 / m) : sqrt(2.0 / m);
      for (int j = 0; j < m; ++j) cy[(size_t)k * m + j] = (float)(sk * cos(pi * k * (2 * j + 1) / (2.0 * m)));
      for (int j = 0; j < m; ++j) cy[(size_t)m * m + (size_t)j * m + k] = cy[(size_t)k * m + j];
      const double sn = sin(pi * k / (2.0 * m));
      ly[k] = (float)(-4.0 * ay * sn * sn);
    }
    if (cudaMemcpyAsync(at<float>(ws, L.dcy), cy.data(), cy.size() * 4, cudaMemcpyHostToDevice,
                        st) != cudaSuccess ||
        cudaMemcpyAsync(at<float>(ws, L.dly), ly.data(), ly.size() * 4, cudaMemcpyHostToDevice,
                        st) != cudaSuccess)
      return AJ_ERR_CUDA;
    const CvDirect d = direct_args(p, L, ws, nullptr);
    k_cv_dfactor<<<d.m, cdiv(d.n, 32) * 32, 6 * d.n * sizeof(float), st>>>(d);
    if (cudaGetLastError() != cudaSuccess) return AJ_ERR_CUDA;
  }
  if (cudaFuncSetAttribute(k_cv_block, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kBlockSmemMax + 1024) != cudaSuccess)
    return AJ_ERR_CUDA;
  if (cudaMemcpyAsync(at<double>(ws, L.cinv), inv.data(), inv.size() * sizeof(double),
                      cudaMemcpyHostToDevice, st) != cudaSuccess)
    return AJ_ERR_CUDA;
  return cudaStreamSynchronize(st) == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

// One launch of a converging-mode kernel on the workspace's current contents
// (instrumentation: lets a caller time the kernel on its own).  which:
// 0 = level-0 smoothing + residual + restriction, 1 = level-0 prolongation +
// smoothing + pressure update + residual (the solver state is left untouched),
// 2 = the coarse solve (the separable direct solve, or the one-block kernel).
int profile_pressure_kernel(const AjStepParams& p, const Layout& L, void* ws, int which,
                            cudaStream_t st) {
  if (p.mg_mode != AJ_MG_CONVERGE) return AJ_ERR_PARAM;
  DevScalars* sc = at<DevScalars>(ws, 0);
  const int* never = reinterpret_cast<const int*>(&sc->zero);
  CvLvl c = cv_level(p, L, 0);
  const int sh = variant_shape(tile_variant(p.nx, p.ny), c);
  if (which == 0) {
    level0_down_s(sh, c, L, ws, never, st);
  } else if (which == 1) {
    CvCheck ck{p.max_cycles, 0, 0};
    // profile mode reads the current state buffer and writes only the other one
    level0_up_s(sh, p, c, L, ws, sc, ck, 1, st);
  } else if (which == 2) {
    if (L.ld > 0) {
      direct_launch(direct_args(p, L, ws, never), st);
    } else {
      k_cv_block<<<1, CV_BLOCK_THREADS, converge_block_smem(L, L.lc), st>>>(
          block_args(p, L, ws, never));
    }
  } else {
    return AJ_ERR_PARAM;
  }
  return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

// ---------------------------------------------------------------- autotuner
// The level-0 tile shape per grid shape.  converge_autotune times every
// candidate (level-0 pre-smoothing + post-smoothing kernels, profile mode, on
// a prepared workspace) and keeps the fastest (the default unless another is
// 5 % faster); the choice is cached per
// (nx, ny, SM count) for the life of the process and is part of every graph
// key, so graphs captured before and after a tuning never mix.
namespace {
std::mutex g_tune_mu;
std::map<std::tuple<int, int, int>, int> g_tune;
int sm_count() {
  static int n = -1;
  if (n < 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 0;
  }
  return n;
}
}  // namespace

int tile_variant(int nx, int ny) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  auto it = g_tune.find({nx, ny, sm_count()});
  return it == g_tune.end() ? 0 : it->second;
}

int converge_autotune(const AjStepParams& p, const Layout& L, void* ws, int reps, float* times_ms,
                      int* chosen, cudaStream_t st) {
  if (p.mg_mode != AJ_MG_CONVERGE) return AJ_ERR_PARAM;
  DevScalars* sc = at<DevScalars>(ws, 0);
  const int* never = reinterpret_cast<const int*>(&sc->zero);
  const CvLvl c = cv_level(p, L, 0);
  const CvCheck ck{p.max_cycles, 0, 0};
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)
    return AJ_ERR_CUDA;
  int best = 0;
  float best_ms = 1e30f;
  for (int v = 0; v < CV_TILE_VARIANTS; ++v) {
    for (int w = 0; w < 2; ++w) {   // warm-up
      level0_down_s(variant_shape(v, c), c, L, ws, never, st);
      level0_up_s(variant_shape(v, c), p, c, L, ws, sc, ck, 1, st);
    }
    cudaEventRecord(e0, st);
    for (int r = 0; r < reps; ++r) {
      level0_down_s(variant_shape(v, c), c, L, ws, never, st);
      level0_up_s(variant_shape(v, c), p, c, L, ws, sc, ck, 1, st);
    }
    cudaEventRecord(e1, st);
    if (cudaEventSynchronize(e1) != cudaSuccess) {
      cudaEventDestroy(e0);
      cudaEventDestroy(e1);
      return AJ_ERR_CUDA;
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    ms /= (float)(reps > 0 ? reps : 1);
    if (times_ms) times_ms[v] = ms;
    // another shape must beat the default by 5 % to be taken (the candidates
    // are often within run-to-run noise of each other)
    if (v == 0 || ms < 0.95f * best_ms) {
      best_ms = ms;
      best = v;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune[{p.nx, p.ny, sm_count()}] = best;
  }
  if (chosen) *chosen = best;
  return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

}  // namespace aj

