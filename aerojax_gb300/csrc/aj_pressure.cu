// Pressure Poisson solve.
//
// Parity mode reproduces poisson_multigrid (pressure_solvers/multigrid_solver.py:55-241)
// and poisson_multigrid_mac (pressure_solvers/multigrid_solver_mac.py:59-246):
// undamped Jacobi with edge ghosts, coarse levels that keep the fine dx/dy,
// unscaled 2x2-average restriction, a prolongation that leaves the last fine
// row and column zero, 10 coarsest sweeps, outlet row reset after each smoothing
// phase, and the absolute early exit sum(r^2) dx dy < tol^2 after each cycle.
// A tiled kernel per direction on the finest levels; the levels below (every
// level and every cycle on small grids) on one cluster (aj_parity_cluster.cu).
//
// The converging mode lives in aj_converge.cu; this file dispatches to it.
#include "aj_parity_pair.cuh"

#include <cooperative_groups.h>
#include <math.h>

namespace aj {

// b = rhs (* mask for MAC), b[-1, :] = 0 for the von Karman outlet
// (multigrid_solver.py:75-77, multigrid_solver_mac.py:78-83)
__global__ void k_mg_rhs(const float* __restrict__ rhs, const float* __restrict__ mask,
                         float* __restrict__ b, int nx, int ny, int mac, int outlet) {
  long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= (long)nx * ny) return;
  int i = (int)(k / ny);
  float v = mac ? rhs[k] * mask[k] : rhs[k];
  b[k] = (outlet && i == nx - 1) ? 0.f : v;
}

int launch_mg_rhs(const AjStepParams& p, const Layout& L, void* ws, const float* rhs,
                  const float* mask, cudaStream_t st) {
  long n = (long)p.nx * p.ny;
  k_mg_rhs<<<cdiv(n, 256), 256, 0, st>>>(rhs, mask, at<float>(ws, L.b0), p.nx, p.ny,
                                         p.grid_type == AJ_GRID_MAC,
                                         p.flow_type == AJ_FLOW_VON_KARMAN);
  return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

// ---------------------------------------------------------- other flow types
// Lid-driven cavity: b -= mean(b) before the cycles (multigrid_solver.py:78-80)
// and p -= p[nx/2, ny/2] after them.  The mean: FP64 block partials, summed
// in block order by the last block (reproducible), kept in sc->acc[2].
constexpr int kMeanBlocks = 256;
__global__ void __launch_bounds__(256) k_mean_partials(const float* __restrict__ b, long n,
                                                       DevScalars* sc, double* part) {
  double s = 0.0;
  for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < n;
       k += (long)gridDim.x * blockDim.x)
    s += (double)b[k];
  const double bs = block_sum(s);
  __shared__ int am_last;
  if (threadIdx.x == 0) {
    part[blockIdx.x] = bs;
    __threadfence();
    am_last = atomicAdd(&sc->red_count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!am_last || threadIdx.x != 0) return;
  __threadfence();
  double t = 0.0;
  for (unsigned q = 0; q < gridDim.x; ++q) t += __ldcg(part + q);
  sc->acc[2] = t / (double)n;
  sc->red_count = 0u;
}
__global__ void k_sub_mean(float* __restrict__ b, long n, const DevScalars* sc) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k < n) b[k] = b[k] - (float)sc->acc[2];
}
__global__ void k_store_center(const float* __restrict__ p, long c, DevScalars* sc) {
  sc->acc[3] = (double)p[c];
}
__global__ void k_sub_center(float* __restrict__ p, long n, const DevScalars* sc) {
  const long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k < n) p[k] = p[k] - (float)sc->acc[3];
}

// ====================================================================== parity
// restriction of a mask level followed by the > 0.5 threshold
// (multigrid_solver_mac.py:213-214)
__global__ void k_mask_restrict(const float* __restrict__ mf, float* __restrict__ mc, int n,
                                int m) {
  int J = blockIdx.x * blockDim.x + threadIdx.x;
  int I = blockIdx.y * blockDim.y + threadIdx.y;
  int nc = n / 2, mc_ = m / 2;
  if (I >= nc || J >= mc_) return;
  const float* f = mf + (long)(2 * I) * m + 2 * J;
  float r = 0.25f * (f[0] + f[m] + f[1] + f[m + 1]);
  mc[(long)I * mc_ + J] = r > 0.5f ? 1.f : 0.f;
}

// value of the reference prolongation at fine (a, b) from coarse c (nc x mc)
__device__ __forceinline__ float prolong_ref(const float* __restrict__ c, int nc, int mc, int a,
                                             int b) {
  int I = a >> 1, J = b >> 1, ao = a & 1, bo = b & 1;
  if (!ao && !bo) return ldg(c + (long)I * mc + J);
  if (ao && !bo) return I <= nc - 2 ? 0.5f * (ldg(c + (long)I * mc + J) + ldg(c + (long)(I + 1) * mc + J)) : 0.f;
  if (!ao && bo) return J <= mc - 2 ? 0.5f * (ldg(c + (long)I * mc + J) + ldg(c + (long)I * mc + J + 1)) : 0.f;
  if (I <= nc - 2 && J <= mc - 2)
    return 0.25f * (ldg(c + (long)I * mc + J) + ldg(c + (long)(I + 1) * mc + J) +
                    ldg(c + (long)I * mc + J + 1) + ldg(c + (long)(I + 1) * mc + J + 1));
  return 0.f;
}

struct ParJac {
  const float* pin;    // null = zero guess
  const float* b;
  const float* mask;   // MAC: p_new *= mask
  float* pout;
  const int* skip;
  int n, m, zero_last;
  float ax, ay, den;
};

// one undamped Jacobi sweep with edge ghosts (multigrid_solver.py:158-171):
// the coarsest level's sweeps when its bands do not fit the cluster's blocks
__global__ void __launch_bounds__(256) k_par_jacobi(ParJac a) {
  if (a.skip && *a.skip) return;
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= a.n || j >= a.m) return;
  auto pv = [&](int ii, int jj) -> float {
    return a.pin ? ldg(a.pin + (long)ii * a.m + jj) : 0.f;
  };
  int ip = i + 1 < a.n ? i + 1 : a.n - 1, im = i > 0 ? i - 1 : 0;
  int jp = j + 1 < a.m ? j + 1 : a.m - 1, jm = j > 0 ? j - 1 : 0;
  long k = (long)i * a.m + j;
  float pn = (a.ax * (pv(ip, j) + pv(im, j)) + a.ay * (pv(i, jp) + pv(i, jm)) - ldg(a.b + k)) / a.den;
  if (a.mask) pn = pn * ldg(a.mask + k);
  if (a.zero_last && i == a.n - 1) pn = 0.f;
  a.pout[k] = pn;
}

__global__ void k_par_begin(DevScalars* sc) {
  sc->red_count = 0u;
  sc->mg_skip = 0;
  sc->mg_cycles = 0;
  sc->acc[0] = 0.0;
  sc->acc[1] = 0.0;
  sc->err = AJ_OK;
}

// converged = sum r^2 dx dy < tol^2 (multigrid_solver.py:222-232), run by the
// last block of the level-0 up kernel once every block's norm is in
__device__ void par_check_body(DevScalars* sc, double dxdy, double tol2, int first) {
  if (first) sc->bnorm = sqrt(sc->acc[1]);
  double s = sc->acc[0];
  sc->mg_cycles += 1;
  sc->abs_sq = s * dxdy;
  sc->rel = sc->bnorm > 0.0 ? sqrt(s) / sc->bnorm : sqrt(s);
  if (!isfinite(s)) sc->err = AJ_ERR_NONFINITE;
  sc->mg_skip = (s * dxdy < tol2) ? 1 : 0;
  sc->acc[0] = 0.0;
  sc->acc[1] = 0.0;
}

// the coarsest level's 10 Jacobi sweeps from a zero guess
// (multigrid_solver.py:186-187) on a cluster of kCoarseCtas blocks: block k
// holds rows [k R, k R + R) of the iterate (ping-pong) and of b in shared
// memory and reads the rows next to its band from its neighbours' shared
// memory.  One cluster barrier per sweep: a sweep reads one buffer and writes
// the other, so after the barrier nobody still reads what the next sweep
// overwrites.  The skip test comes before any barrier and is the same for
// every block; after the last barrier a block reads only its own memory.
// Same arithmetic as k_par_jacobi.
__global__ void __cluster_dims__(kCoarseCtas, 1, 1) __launch_bounds__(kCoarseThreads)
    k_par_coarsest(const float* __restrict__ b, const float* __restrict__ mask,
                   float* __restrict__ x, int n, int m, float ax, float ay, float den,
                   const int* skip) {
  if (skip && *skip) return;
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int R = coarse_band_rows(n);
  const int r0 = rank * R, nr = max(0, min(n, r0 + R) - r0);
  extern __shared__ float psm[];
  float* P = psm;
  float* Q = psm + R * m;
  float* Bs = psm + 2 * R * m;
  for (int q = threadIdx.x; q < nr * m; q += blockDim.x) Bs[q] = b[(long)r0 * m + q];
  __syncthreads();
  for (int s = 0; s < 10; ++s) {
    for (int q = threadIdx.x; q < nr * m; q += blockDim.x) {
      const int li = q / m, j = q - li * m, i = r0 + li;
      const int ip = i + 1 < n ? i + 1 : n - 1, im = i > 0 ? i - 1 : 0;
      const int jp = j + 1 < m ? j + 1 : m - 1, jm = j > 0 ? j - 1 : 0;
      auto pv = [&](int ii, int jj) -> float {
        if (s == 0) return 0.f;
        const int owner = ii / R;
        const float* base = owner == rank ? P : cl.map_shared_rank(P, owner);
        return base[(ii - owner * R) * m + jj];
      };
      float pn = (ax * (pv(ip, j) + pv(im, j)) + ay * (pv(i, jp) + pv(i, jm)) - Bs[q]) / den;
      if (mask) pn = pn * mask[(long)i * m + j];
      Q[q] = pn;
    }
    cl.sync();
    float* t = P;
    P = Q;
    Q = t;
  }
  for (int q = threadIdx.x; q < nr * m; q += blockDim.x) x[(long)r0 * m + q] = P[q];
}

// whether the coarsest level's sweeps run as one k_par_coarsest block
bool parity_coarsest_fused(const Layout& L) {
  return (size_t)coarse_band_rows(L.ln[L.nlev]) * L.lm[L.nlev] * 12 <= kBlockSmemMax;
}

// ---- one level of the V-cycle per launch, on tiles
// (multigrid_solver.py:173-211).  A block stages a region of 4 G rows by 64
// columns - its 4 (G - 2) x 56 output cells and a halo of four - in one round
// trip, a thread holding a column pair over four rows in registers
// (aj_parity_pair.cuh), and shared memory carries only what neighbouring
// threads read.  Each block writes only its own cells, and no output aliases
// an input another block reads.  What bounds it: on the coarser grids a
// block's own chain (the staging round and four barriers), on the finest one
// issue (1.3 region cells per output cell).  A whole MAC cycle at 2048x512
// 77.8 -> 38.7 us, at 4096x2048 407 -> 143 us (before: a division and two global
// reads a cell and sweep, and every level on its own launches).
struct ParTile {
  const float* xin;   // down: the cycle's input state (null: zero); up: the level's down result
  const float* xc;    // up: the coarser level's result (prolonged on the fly)
  const float* b;
  const float* mask;  // MAC level mask (null: collocated)
  float* xout;        // down: the state after the two pre-sweeps; up: after the post-sweeps
  float* bc;          // down: the restricted residual (the coarser level's b)
  DevScalars* sc;     // up on level 0: the residual norm (multigrid_solver.py:229-231)
  const int* skip;
  int n, m, nc, mc, zero_last, mac_outlet, also_b;
  int pairs;          // every level array is 8-byte aligned (rows are even)
  PairCoef co;
  double dxdy, tol2;  // up on level 0: the early-exit test
};
constexpr unsigned PT_BIG_BLOCKS = 304;   // two of 512 threads on each of 152 SMs
constexpr int PT_RUN = 4, PT_W = 64, PT_H = 4, PT_OUT = PT_W - 2 * PT_H;

// two adjacent cells of a global array
__device__ __forceinline__ float2 pt_ld(const ParTile& a, const float* p) {
  return a.pairs ? __ldg(reinterpret_cast<const float2*>(p)) : make_float2(ldg(p), ldg(p + 1));
}
__device__ __forceinline__ void pt_st(const ParTile& a, float* p, float2 v) {
  if (a.pairs) {
    pair_st(p, v);
  } else {
    p[0] = v.x;
    p[1] = v.y;
  }
}

// this thread's cells of its block's region, clipped to the domain; mine:
// whether they are output cells; k0: the global index of the first
struct PtOwn : PairOwn {
  bool mine, left, right;
  int gj;
  long k0;
};
struct PtGeo {
  static constexpr int m = PT_W;
};
__device__ __forceinline__ bool pair_lf(const PtGeo&, const PtOwn& o) { return o.left; }
__device__ __forceinline__ bool pair_rt(const PtGeo&, const PtOwn& o) { return o.right; }
template <int G>
__device__ __forceinline__ PtOwn pt_own(const ParTile& a) {
  PtOwn o;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int gi0 = blockIdx.y * (PT_RUN * (G - 2)) - PT_H, gj0 = blockIdx.x * PT_OUT - PT_H;
  o.gj = gj0 + 2 * tx;
  o.ga = gi0 + PT_RUN * ty;
  o.glo = max(gi0, 0);
  o.ghi = min(gi0 + PT_RUN * G, a.n);
  // tiles start at multiples of 4 rows and even columns: a run or a pair is
  // never cut by the domain's first row or column, nor a pair by its last
  const bool in = o.ga >= 0 && o.gj >= 0 && o.gj < a.m;
  o.cnt = in ? max(min(PT_RUN, a.n - o.ga), 0) : 0;
  o.left = o.gj > max(gj0, 0);
  o.right = o.gj + 2 < min(gj0 + PT_W, a.m);
  o.q = PT_RUN * ty * PT_W + 2 * tx;
  o.mine = o.cnt > 0 && tx >= PT_H / 2 && tx < (PT_H + PT_OUT) / 2 && ty >= 1 && ty < G - 1;
  o.k0 = (long)o.ga * a.m + o.gj;
  return o;
}
__device__ __forceinline__ void pt_load(const ParTile& a, const PtOwn& o, const float* src,
                                        float2* v) {
#pragma unroll
  for (int r = 0; r < PT_RUN; ++r)
    v[r] = r < o.cnt ? pt_ld(a, src + o.k0 + (long)r * a.m) : make_float2(0.f, 0.f);
}

// down: two pre-sweeps (the second resets the outlet row), the residual and
// its 2x2 average onto the coarser level (multigrid_solver.py:182-201)
template <int G, bool MAC>
__global__ void __launch_bounds__(32 * G, 1024 / (32 * G)) k_par_down(ParTile a) {
  pdl_wait();
  if (a.skip && *a.skip) return;
  __shared__ __align__(8) float A[PT_RUN * G * PT_W], D[PT_RUN * G * PT_W];
  const PtOwn o = pt_own<G>(a);
  constexpr PtGeo geo{};
  float2 x[PT_RUN], b[PT_RUN], k[PT_RUN];
  pt_load(a, o, a.b, b);
  if (MAC) pt_load(a, o, a.mask, k);
  auto mask = [&](int r) { return k[r]; };
  auto none = [](int) { return false; };
  auto last = [&](int r) { return a.zero_last && o.ga + r == a.n - 1; };
  auto outlet = [&](int r) { return a.mac_outlet && o.ga + r == a.n - 1; };
  if (a.xin) {
    pt_load(a, o, a.xin, x);
    pair_store<PT_RUN>(geo, o, A, x);
    __syncthreads();
    pair_sweep<MAC, PT_RUN>(a.co, geo, o, A, b, mask, none, x);
  } else {
    pair_sweep0<MAC, PT_RUN>(a.co, o, b, mask, x);
  }
  pair_store<PT_RUN>(geo, o, D, x);
  __syncthreads();
  pair_sweep<MAC, PT_RUN>(a.co, geo, o, D, b, mask, last, x);
  pair_store<PT_RUN>(geo, o, A, x);
  __syncthreads();
  if (!o.mine) return;
#pragma unroll
  for (int r = 0; r < PT_RUN; ++r)
    if (r < o.cnt) pt_st(a, a.xout + o.k0 + (long)r * a.m, x[r]);
  float2 ra{0.f, 0.f};
  float* bc = a.bc + (long)(o.ga >> 1) * a.mc + (o.gj >> 1);
  pair_resid<PT_RUN>(a.co, geo, o, A, b, outlet, x, [&](int r, float2 v) {
    // summed in the order (0,0), (1,0), (0,1), (1,1)
    if (r & 1) bc[(long)(r / 2) * a.mc] = 0.25f * (ra.x + v.x + ra.y + v.y);
    ra = v;
  });
}

// up: p + P(e) and two post-sweeps (the second resets the outlet row,
// multigrid_solver.py:203-211); with NORM (level 0) also sum (b - A p)^2 and,
// on the first cycle, b^2 (exact squares, compensated sums, FP64 across
// blocks)
template <int G, bool MAC, bool NORM>
__global__ void __launch_bounds__(32 * G, 1024 / (32 * G)) k_par_up(ParTile a) {
  pdl_wait();
  if (a.skip && *a.skip) return;
  __shared__ __align__(8) float A[PT_RUN * G * PT_W], D[PT_RUN * G * PT_W];
  const PtOwn o = pt_own<G>(a);
  constexpr PtGeo geo{};
  float2 x[PT_RUN], b[PT_RUN], k[PT_RUN];
  pt_load(a, o, a.xin, x);
  pt_load(a, o, a.b, b);
  if (MAC) pt_load(a, o, a.mask, k);
  auto mask = [&](int r) { return k[r]; };
  auto none = [](int) { return false; };
  auto last = [&](int r) { return a.zero_last && o.ga + r == a.n - 1; };
  auto outlet = [&](int r) { return a.mac_outlet && o.ga + r == a.n - 1; };
  const int I0 = o.ga >> 1, J = o.gj >> 1;
  const float* e = a.xc + (long)I0 * a.mc + J;
  pair_prolong<PT_RUN>(
      o, a.nc, J <= a.mc - 2,
      [&](int i, int d) { return I0 + i < a.nc ? ldg(e + (long)i * a.mc + d) : 0.f; }, x);
  pair_store<PT_RUN>(geo, o, A, x);
  __syncthreads();
  pair_sweep<MAC, PT_RUN>(a.co, geo, o, A, b, mask, none, x);
  pair_store<PT_RUN>(geo, o, D, x);
  __syncthreads();
  pair_sweep<MAC, PT_RUN>(a.co, geo, o, D, b, mask, last, x);
  if (o.mine) {
#pragma unroll
    for (int r = 0; r < PT_RUN; ++r)
      if (r < o.cnt) pt_st(a, a.xout + o.k0 + (long)r * a.m, x[r]);
  }
  if constexpr (NORM) {
    pair_store<PT_RUN>(geo, o, A, x);
    __syncthreads();
    __shared__ df ws[2 * G];
    df s{0.f, 0.f};
    if (o.mine)
      pair_resid<PT_RUN>(a.co, geo, o, A, b, outlet, x, [&](int, float2 v) {
        // (b - A p) in FP32 as the reference evaluates it; its square exactly
        s = pair_add_sq(s, v);
      });
    s = warp_sum_df(s);
    if (threadIdx.x == 0) ws[threadIdx.y] = s;
    if (a.also_b) {
      s = df{0.f, 0.f};
#pragma unroll
      for (int r = 0; r < PT_RUN; ++r)
        if (o.mine && r < o.cnt) s = pair_add_sq(s, b[r]);
      s = warp_sum_df(s);
      if (threadIdx.x == 0) ws[G + threadIdx.y] = s;
    }
    __syncthreads();
    if (threadIdx.y > 0) return;
    const int l = threadIdx.x;
    const double tr = warp_sum<G>(df_double(ws[l % G])),
                 tb = a.also_b ? warp_sum<G>(df_double(ws[G + l % G])) : 0.0;
    if (l == 0) {
      atomicAdd(&a.sc->acc[0], tr);
      if (a.also_b) atomicAdd(&a.sc->acc[1], tb);
      __threadfence();
      // every block's sums are in: the early-exit test
      if (atomicAdd(&a.sc->red_count, 1u) == gridDim.x * gridDim.y - 1) {
        __threadfence();
        a.sc->red_count = 0u;
        par_check_body(a.sc, a.dxdy, a.tol2, a.also_b);
      }
    }
  }
}

__global__ void k_copy(const float* __restrict__ s, float* __restrict__ d, long n) {
  long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k < n) d[k] = s[k];
}

__global__ void k_stats(const DevScalars* sc, AjStats* st, int converge_mode) {
  pdl_wait();
  // all loads before the stores (interleaved, each load waits for a store)
  const int cycles = sc->mg_cycles, conv = converge_mode ? sc->mg_done : sc->mg_skip;
  const int err = sc->err;
  const double rel = sc->rel, bnorm = sc->bnorm, abs_sq = sc->abs_sq;
  const float dt = sc->dt;
  st->cycles = cycles;
  st->converged = conv;
  st->err = err;
  st->pad = 0;
  st->rel_residual = rel;
  st->rhs_norm = bnorm;
  st->dt = dt;
  st->abs_residual_sq = abs_sq;
}

// Taylor-Green: the reference's residual wraps periodically while its
// smoother keeps edge ghosts (multigrid_solver.py:158-183), so the residual
// at a boundary cell needs the smoothed iterate on the far side of the
// domain.  Its V-cycle therefore runs unfused: Jacobi sweeps (k_par_jacobi),
// then these kernels.
// r = b - A x with wrapped neighbours, 2x2 average onto the coarser b
__global__ void __launch_bounds__(256) k_tg_resid_restrict(const float* __restrict__ x,
                                                           const float* __restrict__ b,
                                                           float* __restrict__ bc, int n, int m,
                                                           float ax, float ay, const int* skip) {
  if (skip && *skip) return;
  const int J = blockIdx.x * blockDim.x + threadIdx.x;
  const int I = blockIdx.y * blockDim.y + threadIdx.y;
  const int nc = n / 2, mc = m / 2;
  if (I >= nc || J >= mc) return;
  float r[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = 2 * I + (q & 1), j = 2 * J + (q >> 1);
    const int ip = i + 1 < n ? i + 1 : 0, im = i > 0 ? i - 1 : n - 1;
    const int jp = j + 1 < m ? j + 1 : 0, jm = j > 0 ? j - 1 : m - 1;
    const float c = ldg(x + (long)i * m + j);
    const float lap = ax * (ldg(x + (long)ip * m + j) + ldg(x + (long)im * m + j) - 2.f * c) +
                      ay * (ldg(x + (long)i * m + jp) + ldg(x + (long)i * m + jm) - 2.f * c);
    r[q] = ldg(b + (long)i * m + j) - lap;
  }
  // summed in the order (0,0), (1,0), (0,1), (1,1) like the tiled kernels
  bc[(long)I * mc + J] = 0.25f * (r[0] + r[1] + r[2] + r[3]);
}
// x += P(xc) in place (the reference prolongation, last row and column 0)
__global__ void __launch_bounds__(256) k_tg_prolong_add(float* __restrict__ x,
                                                        const float* __restrict__ xc, int n,
                                                        int m, const int* skip) {
  if (skip && *skip) return;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= n || j >= m) return;
  const long k = (long)i * m + j;
  x[k] = x[k] + prolong_ref(xc, n / 2, m / 2, i, j);
}
// level 0 after the cycle: sum (b - A x)^2 with wrapped neighbours (and, on
// the first cycle, b^2) in double-FP32 per block, FP64 across blocks; the
// last block runs the early-exit test
__global__ void __launch_bounds__(256) k_tg_norm(const float* __restrict__ x,
                                                 const float* __restrict__ b, int n, int m,
                                                 float ax, float ay, DevScalars* sc, double dxdy,
                                                 double tol2, int also_b, const int* skip) {
  if (skip && *skip) return;
  df rr{0.f, 0.f}, bb{0.f, 0.f};
  const long N = (long)n * m;
  for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < N;
       k += (long)gridDim.x * blockDim.x) {
    const int i = (int)(k / m), j = (int)(k - (long)i * m);
    const int ip = i + 1 < n ? i + 1 : 0, im = i > 0 ? i - 1 : n - 1;
    const int jp = j + 1 < m ? j + 1 : 0, jm = j > 0 ? j - 1 : m - 1;
    const float c = ldg(x + k);
    const float lap = ax * (ldg(x + (long)ip * m + j) + ldg(x + (long)im * m + j) - 2.f * c) +
                      ay * (ldg(x + (long)i * m + jp) + ldg(x + (long)i * m + jm) - 2.f * c);
    const float bv = ldg(b + k);
    const float res = bv - lap;
    rr = df_add(rr, two_prod(res, res));
    bb = df_add(bb, two_prod(bv, bv));
  }
  const double s = block_sum_df(rr);
  const double sb = also_b ? block_sum_df(bb) : 0.0;
  __shared__ int am_last;
  if (threadIdx.x == 0) {
    atomicAdd(&sc->acc[0], s);
    if (also_b) atomicAdd(&sc->acc[1], sb);
    __threadfence();
    am_last = atomicAdd(&sc->red_count, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (am_last && threadIdx.x == 0) {
    __threadfence();
    sc->red_count = 0u;
    par_check_body(sc, dxdy, tol2, also_b);
  }
}

static int parity_solve(const AjStepParams& p, const Layout& L, void* ws, const float* mask,
                        const float* p0, float* pout, AjStats* stats, cudaStream_t st) {
  DevScalars* sc = at<DevScalars>(ws, 0);
  const int mac = p.grid_type == AJ_GRID_MAC;
  const float ax = (float)(1.0 / (p.dx * p.dx)), ay = (float)(1.0 / (p.dy * p.dy));
  const float den = (float)(2.0 * (1.0 / (p.dx * p.dx) + 1.0 / (p.dy * p.dy)));
  const double tol = p.mg_tolerance > 0 ? p.mg_tolerance : AJ_PARITY_TOL_DEFAULT;
  const int nl = L.nlev;
  float* b0 = at<float>(ws, L.b0);
  float* T0 = at<float>(ws, L.T0);
  const int* skip = &sc->mg_skip;
  dim3 blk(32, 8);
  const long N0 = (long)p.nx * p.ny;
  const int lt = parity_cluster_level(p, L);   // levels lt.. run on a cluster
  if (lt > 0) k_par_begin<<<1, 1, 0, st>>>(sc);
  if (lt > 0 && p0) k_copy<<<cdiv(N0, 256), 256, 0, st>>>(p0, pout, N0);
  if (p.flow_type == AJ_FLOW_LID_DRIVEN_CAVITY) {   // b -= mean(b) (multigrid_solver.py:78-80)
    k_mean_partials<<<kMeanBlocks, 256, 0, st>>>(b0, N0, sc, at<double>(ws, L.part));
    k_sub_mean<<<cdiv(N0, 256), 256, 0, st>>>(b0, N0, sc);
  }

  auto X = [&](int l) { return l == 0 ? pout : at<float>(ws, L.X[l]); };
  auto T = [&](int l) { return l == 0 ? T0 : at<float>(ws, L.T[l]); };
  auto B = [&](int l) { return l == 0 ? b0 : at<float>(ws, L.B[l]); };
  auto M = [&](int l) -> const float* {
    if (!mac) return nullptr;
    return l == 0 ? mask : at<float>(ws, L.M[l]);
  };
  const int vk = p.flow_type == AJ_FLOW_VON_KARMAN;
  const float* masks[AJ_MAX_LEVELS + 1];
  for (int l = 0; l <= nl; ++l) masks[l] = M(l);
  int rc = AJ_OK;
  // levels lt.. of one cycle on the cluster (with lt = 0 the whole solve)
  auto cluster = [&](const int* sk) {
    rc |= launch_parity_cluster(p, L, ws, lt, masks, B(lt), p0, X(lt), sk, stats, st);
  };
  // the coarsest level's 10 sweeps from zero, ending in X(nl)
  auto coarsest = [&](const int* sk) {
    if (lt == nl) {
      cluster(sk);
    } else if (parity_coarsest_fused(L)) {
      const int n = L.ln[nl], m = L.lm[nl];
      const size_t csm = (size_t)coarse_band_rows(n) * m * 12;
      cudaFuncSetAttribute(k_par_coarsest, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)kBlockSmemMax);
      k_par_coarsest<<<kCoarseCtas, kCoarseThreads, csm, st>>>(B(nl), M(nl), X(nl), n, m, ax, ay,
                                                               den, sk);
    } else {
      int n = L.ln[nl], m = L.lm[nl];
      dim3 g(cdiv(m, 32), cdiv(n, 8));
      ParJac a{};
      a.b = B(nl);
      a.mask = M(nl);
      a.skip = sk;
      a.n = n;
      a.m = m;
      a.ax = ax;
      a.ay = ay;
      a.den = den;
      for (int s = 0; s < 10; ++s) {
        a.pin = s == 0 ? nullptr : (s % 2 == 1 ? T(nl) : X(nl));
        a.pout = s % 2 == 0 ? T(nl) : X(nl);
        k_par_jacobi<<<g, blk, 0, st>>>(a);
      }
    }
  };
  if (p.flow_type == AJ_FLOW_TAYLOR_GREEN) {
    // unfused V-cycle (the wrapped residual needs the other side of the domain):
    // every level's iterate lives in X(l), T(l) is the sweeps' other buffer
    for (int cyc = 0; cyc < p.v_cycles; ++cyc) {
      const int* sk = cyc == 0 ? nullptr : skip;
      auto sweeps = [&](int l, const float* first_in) {
        ParJac a{};
        a.b = B(l);
        a.mask = M(l);
        a.skip = sk;
        a.n = L.ln[l];
        a.m = L.lm[l];
        a.ax = ax;
        a.ay = ay;
        a.den = den;
        dim3 g(cdiv(a.m, 32), cdiv(a.n, 8));
        a.pin = first_in;
        a.pout = T(l);
        k_par_jacobi<<<g, blk, 0, st>>>(a);
        a.pin = T(l);
        a.pout = X(l);
        k_par_jacobi<<<g, blk, 0, st>>>(a);
      };
      for (int l = 0; l < nl; ++l) {
        sweeps(l, (l == 0 && !(cyc == 0 && !p0)) ? X(0) : nullptr);
        dim3 g(cdiv(L.lm[l + 1], 32), cdiv(L.ln[l + 1], 8));
        k_tg_resid_restrict<<<g, blk, 0, st>>>(X(l), B(l), B(l + 1), L.ln[l], L.lm[l], ax, ay, sk);
      }
      coarsest(sk);
      for (int l = nl - 1; l >= 0; --l) {
        dim3 g(cdiv(L.lm[l], 32), cdiv(L.ln[l], 8));
        k_tg_prolong_add<<<g, blk, 0, st>>>(X(l), X(l + 1), L.ln[l], L.lm[l], sk);
        sweeps(l, X(l));
      }
      k_tg_norm<<<kMeanBlocks, 256, 0, st>>>(X(0), B(0), p.nx, p.ny, ax, ay, sc, p.dx * p.dy,
                                             tol * tol, cyc == 0, sk);
    }
    if (stats) k_stats<<<1, 1, 0, st>>>(sc, stats, 0);
    return rc == AJ_OK && cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
  }
  const int nt = lt < nl ? lt : nl;   // levels 0 .. nt-1 by the tiled kernels
  if (lt == 0) cluster(nullptr);
  auto aligned = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 7) == 0; };
  const int pairs = aligned(pout) && (!mac || aligned(mask));   // the workspace's arrays are
  // a level's kernel on regions of 64 rows where those fill the GPU twice over
  // (less of their work is halo), else of 32 rows (more and shorter blocks)
  auto launch = [&](int l, auto big, auto small, const ParTile& a) {
    const unsigned gx = cdiv(L.lm[l], PT_OUT), g16 = cdiv(L.ln[l], PT_RUN * 14);
    if (gx * g16 >= PT_BIG_BLOCKS)
      launch_pdl(true, big, dim3(gx, g16), dim3(32, 16), 0, st, a);
    else
      launch_pdl(true, small, dim3(gx, cdiv(L.ln[l], PT_RUN * 6)), dim3(32, 8), 0, st, a);
  };
  for (int cyc = 0; cyc < p.v_cycles && lt > 0; ++cyc) {
    const int* sk = cyc == 0 ? nullptr : skip;   // the first cycle always runs
    // down the V: levels 0..nt-1; each level's pre-smoothed state goes to T,
    // its restricted residual to the next level's b
    for (int l = 0; l < nt; ++l) {
      ParTile a{};
      a.xin = (l == 0 && !(cyc == 0 && !p0)) ? X(0) : nullptr;
      a.b = B(l);
      a.mask = M(l);
      a.xout = T(l);
      a.bc = B(l + 1);
      a.skip = sk;
      a.n = L.ln[l];
      a.m = L.lm[l];
      a.nc = L.ln[l + 1];
      a.mc = L.lm[l + 1];
      a.zero_last = vk;
      a.mac_outlet = mac && vk;
      a.pairs = pairs;
      a.co = parity_coef(p);
      if (mac) launch(l, k_par_down<16, true>, k_par_down<8, true>, a);
      else launch(l, k_par_down<16, false>, k_par_down<8, false>, a);
    }
    // below: the cluster, or the coarsest level's 10 sweeps from zero, into X(nt)
    if (lt < nl) cluster(sk);
    else coarsest(sk);
    // up the V: T + P(coarser X), two post-sweeps, into X; level 0 also
    // forms the residual norm and its last block runs the early-exit test
    // (multigrid_solver.py:222-232)
    for (int l = nt - 1; l >= 0; --l) {
      ParTile a{};
      a.xin = T(l);
      a.xc = X(l + 1);
      a.b = B(l);
      a.mask = M(l);
      a.xout = X(l);
      a.sc = sc;
      a.skip = sk;
      a.n = L.ln[l];
      a.m = L.lm[l];
      a.nc = L.ln[l + 1];
      a.mc = L.lm[l + 1];
      a.zero_last = vk;
      a.mac_outlet = mac && vk;
      a.also_b = cyc == 0;
      a.pairs = pairs;
      a.co = parity_coef(p);
      a.dxdy = p.dx * p.dy;
      a.tol2 = tol * tol;
      if (l == 0 && mac) launch(l, k_par_up<16, true, true>, k_par_up<8, true, true>, a);
      else if (l == 0) launch(l, k_par_up<16, false, true>, k_par_up<8, false, true>, a);
      else if (mac) launch(l, k_par_up<16, true, false>, k_par_up<8, true, false>, a);
      else launch(l, k_par_up<16, false, false>, k_par_up<8, false, false>, a);
    }
  }
  if (p.flow_type == AJ_FLOW_LID_DRIVEN_CAVITY) {   // p -= p[nx/2, ny/2]
    k_store_center<<<1, 1, 0, st>>>(pout, (long)(p.nx / 2) * p.ny + p.ny / 2, sc);
    k_sub_center<<<cdiv(N0, 256), 256, 0, st>>>(pout, N0, sc);
  }
  if (stats && lt > 0) k_stats<<<1, 1, 0, st>>>(sc, stats, 0);   // the whole solve files its own
  return rc == AJ_OK && cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

int parity_kernel_count(const AjStepParams& p, const Layout& L) {
  const int lt = parity_cluster_level(p, L), nt = lt < L.nlev ? lt : L.nlev;
  const int below = lt <= L.nlev || parity_coarsest_fused(L) ? 1 : 10;
  int n = p.flow_type == AJ_FLOW_LID_DRIVEN_CAVITY ? 4 : 0;     // mean and centre pin
  if (p.flow_type == AJ_FLOW_TAYLOR_GREEN) return 2 + p.v_cycles * (6 * L.nlev + below + 1);
  if (lt == 0) return n + 1;                                    // the whole solve
  return n + 2 + p.v_cycles * (2 * nt + below);                 // begin, cycles, statistics
}

int prepare_pressure(const AjStepParams& p, const Layout& L, void* ws, const float* mask,
                     cudaStream_t st) {
  if (p.mg_mode == AJ_MG_PARITY) {
    if (p.grid_type == AJ_GRID_MAC) {
      dim3 blk(32, 8);
      for (int l = 0; l < L.nlev; ++l) {
        const float* mf = l == 0 ? mask : at<float>(ws, L.M[l]);
        int n = L.ln[l], m = L.lm[l];
        dim3 g(cdiv(m / 2, 32), cdiv(n / 2, 8));
        k_mask_restrict<<<g, blk, 0, st>>>(mf, at<float>(ws, L.M[l + 1]), n, m);
      }
    }
  } else if (p.mg_mode == AJ_MG_CONVERGE) {
    int rc = converge_prepare(p, L, ws, st);
    if (rc != AJ_OK) return rc;
  }
  return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

int launch_pressure(const AjStepParams& p, const Layout& L, void* ws, const float* mask,
                    const float* p0, float* pout, AjStats* stats, cudaStream_t st,
                    const NnWarm* nn, bool init_done) {
  int rc;
  if (p.mg_mode == AJ_MG_PARITY) {
    rc = parity_solve(p, L, ws, mask, p0, pout, stats, st);
    if (rc != AJ_OK) return rc;
  } else {
    rc = converge_solve(p, L, ws, p0, pout, st, nn, stats, init_done);   // k_cv_out: stats
    if (rc != AJ_OK) return rc;
  }
  return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

}  // namespace aj
