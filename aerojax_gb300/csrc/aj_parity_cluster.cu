// The lower levels of the parity V-cycle - or, on small grids, every level
// and every cycle - in one launch of one thread-block cluster.
//
// The reference's V-cycle (pressure_solvers/multigrid_solver.py:173-232,
// multigrid_solver_mac.py:59-246) as a chain of one kernel per level and
// direction costs 4-8 us a launch on its coarse levels whatever their size:
// each launch waits for the one before it, reads its operands from global
// memory and fills a fraction of the SMs.  Here block k of the cluster keeps
// a band of rows of every level in shared memory for the whole cycle:
//   - bands nest: R rows of the coarsest level, 2R of the next finer, ...;
//   - a level's band carries a halo deep enough that its two sweeps and the
//     residual (3 rows) are computed redundantly without any exchange, and the
//     coarsest level's covers its nine sweeps after the first, which starts from
//     zero, and the two rows that the finer level's prolongation reads (11);
//     both are kept one row deeper (PC_HALO, PC_HALO_COARSE), even, so that a
//     2x2 block stays in one thread;
//   - a block stores what its neighbours' halos need (the restricted residual
//     going down, the corrected iterate going up) straight into their shared
//     memory, and one cluster barrier per level and direction publishes it.
// So a cycle over levels lt .. nl costs 2 (nl - lt) - 1 cluster barriers (two
// more for the residual norm when level 0 is inside) instead of 2 (nl - lt) +
// 1 launches.  Within a level a thread owns a pair of columns over a run of
// rows whose iterate and right-hand side stay in registers from sweep to
// sweep; shared memory carries only what the neighbouring threads read.
// Every pass covers the band with its whole halo, the ends of the array taken
// as edges: the halo rows this spoils are, sweep by sweep, the ones no longer
// needed.
// What bounds it: the chain of short passes (a block barrier each) and the
// cluster barriers (~0.3 us) on 16 SMs - hence the limit on a thread's run:
// above it the tiled kernels, which use all SMs, are the faster ones.
// Measured: a step_pure step at 512x96 with 3 cycles 130 -> 70 us (the solve
// in one launch instead of 28); a cycle at 256x64 38.7 -> 16.8 us, at 512x128
// 39.0 -> 19.5 us.
#include "aj_parity_pair.cuh"

#include <cooperative_groups.h>
#include <math.h>

namespace aj {

namespace cg = cooperative_groups;

constexpr int PC_THREADS = 1024, PC_WARPS = PC_THREADS / 32;
static_assert(PC_WARPS == 32, "one warp adds the warp sums");
constexpr int PC_MAX_CTAS = 16;
constexpr int PC_RUN = 4;            // rows of a thread's column pair (2 on small bands)
constexpr int PC_RUN_COARSE = 6;     // rows of a thread's column, coarsest level
constexpr int PC_HALO = 4, PC_HALO_COARSE = 12;   // even: 2x2 blocks stay in one thread

struct PcLvl {
  int n, m;            // the level's size
  int R, H;            // band rows and halo rows of a block
  int run;             // rows of a thread (pc_own)
  int active;          // threads that own cells, whole warps
  float inv_cols;      // 1 / (column pairs; columns on the coarsest level)
  int off;             // floats: B, A, D (, F above the coarsest), then the mask
  const float* mask;   // MAC level mask
};

struct ParCluster {
  PcLvl lv[AJ_MAX_LEVELS + 1];
  int lt, nl;          // levels lt .. nl
  int cycles;          // whole solve (lt = 0): cycles to run; else 1
  int whole, have_x0, zero_last, mac_outlet;
  const float* b;      // level lt's right-hand side
  const float* x0;     // whole solve: the initial state (have_x0)
  float* x;            // level lt's result
  const int* skip;     // not whole: cycles after convergence are skipped
  DevScalars* sc;
  AjStats* stats;      // whole solve: nullable
  PairCoef co;
  double dxdy, tol2;
};

// a barrier of a level's active warps (the others wait at the level's end)
__device__ __forceinline__ void pc_sync(const PcLvl& L) {
  asm volatile("bar.sync 1, %0;\n" ::"r"(L.active) : "memory");
}

// A thread's cells of a level: W columns from c
struct PcOwn : PairOwn {
  int c;
};
__device__ __forceinline__ bool pair_lf(const PcLvl&, const PcOwn& o) { return o.c > 0; }
__device__ __forceinline__ bool pair_rt(const PcLvl& L, const PcOwn& o) { return o.c + 2 < L.m; }
template <int W>
__device__ __forceinline__ PcOwn pc_own(const PcLvl& L, int rank) {
  PcOwn o;
  const int r0 = rank * L.R;
  o.glo = max(r0 - L.H, 0);
  o.ghi = min(r0 + L.R + L.H, L.n);
  const int cols = W == 2 ? L.m >> 1 : L.m;
  // t / cols by a float product, exact for these sizes
  const int g = (int)(((float)(int)threadIdx.x + 0.5f) * L.inv_cols);
  o.c = W * ((int)threadIdx.x - g * cols);
  o.ga = o.glo + g * L.run;
  o.cnt = max(min(L.run, o.ghi - o.ga), 0);
  o.q = (o.ga - (r0 - L.H)) * L.m + o.c;
  return o;
}

// Stores a thread's values of own rows in the halos of the blocks that reach
// them within h rows: f(peer's array, offset to add to an index here, first
// row, end row).  Every block's array has the same layout R rows further on,
// so a peer d blocks away holds the same cell d R m places off.
template <typename F>
__device__ __forceinline__ void pc_push(cg::cluster_group& cl, float* arr, const PcLvl& L, int h,
                                        int rank, F&& f) {
  const int C = (int)cl.num_blocks(), r0 = rank * L.R;
  for (int d = 1; (d - 1) * L.R < h; ++d) {
    const int off = d * L.R * L.m;
    if (rank + d < C) f(cl.map_shared_rank(arr, rank + d), -off, r0 + d * L.R - h, L.n);
    if (rank >= d) f(cl.map_shared_rank(arr, rank - d), off, 0, r0 - (d - 1) * L.R + h);
  }
}

template <bool MAC>
__global__ void __launch_bounds__(PC_THREADS, 1) k_par_cluster(const __grid_constant__ ParCluster a) {
  pdl_wait();
  if (a.skip && *a.skip) return;   // the same for every block
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), C = (int)cl.num_blocks();
  cl.barrier_arrive();             // no remote store before every block has started
  extern __shared__ __align__(16) float pcs[];
  __shared__ double nrm[2 * PC_MAX_CTAS];
  __shared__ df wsum[2 * PC_WARPS];
  __shared__ double sq[2];   // sum r^2 and sum b^2
  __shared__ int stop;
  const int lt = a.lt, nl = a.nl, tid = threadIdx.x;
  auto r0 = [&](int l) { return rank * a.lv[l].R; };
  auto base = [&](int l) { return r0(l) - a.lv[l].H; };
  auto lo = [&](int l, int h) { return max(r0(l) - h, 0); };
  auto hi = [&](int l, int h) { return min(r0(l) + a.lv[l].R + h, a.lv[l].n); };
  auto size = [&](int l) { return (a.lv[l].R + 2 * a.lv[l].H) * a.lv[l].m; };
  auto arr = [&](int l, int k) { return pcs + a.lv[l].off + k * size(l); };   // 0 B, 1 A, 2 D, 3 F
  auto msk = [&](int l) { return arr(l, l == nl ? 3 : 4); };
  // a contiguous run of rows from global memory, four loads in flight
  auto stage = [&](float* dst, const float* src, int l, int h) {
    const int m = a.lv[l].m, g0 = lo(l, h), cnt = (hi(l, h) - g0) * m;
    float* d = dst + (g0 - base(l)) * m;
    const float* s = src + (long)g0 * m;
#pragma unroll 4
    for (int q = tid; q < cnt; q += PC_THREADS) d[q] = ldg(s + q);
  };
  stage(arr(lt, 0), a.b, lt, a.lv[lt].H);
  if (a.whole && a.have_x0) stage(arr(0, 3), a.x0, 0, PC_HALO);
  if (MAC)
    for (int l = lt; l <= nl; ++l) stage(msk(l), a.lv[l].mask, l, a.lv[l].H);
  __syncthreads();
  cl.barrier_wait();
  int cycles = 0;
  for (int cyc = 0; cyc < a.cycles; ++cyc) {
    // down: two pre-sweeps (the second resets the outlet row), the residual
    // and its 2x2 average onto the coarser level
    for (int l = lt; l < nl; ++l) {
      const PcLvl& L = a.lv[l];
      const PcLvl& Lc = a.lv[l + 1];
      float *A = arr(l, 1), *D = arr(l, 2), *Bc = arr(l + 1, 0);
      auto none = [](int) { return false; };
      if (tid < L.active) {
        const PcOwn o = pc_own<2>(L, rank);
        const float* M = msk(l);
        auto mask = [&](int r) { return pair_ld(M + o.q + r * L.m); };
        auto last = [&](int r) { return a.zero_last && o.ga + r == L.n - 1; };
        float2 x[PC_RUN], b[PC_RUN];
        pair_load<PC_RUN>(L, o, arr(l, 0), b);
        if (l == 0 && (cyc > 0 || a.have_x0)) {
          pair_load<PC_RUN>(L, o, arr(0, 3), x);
          pair_sweep<MAC, PC_RUN>(a.co, L, o, arr(0, 3), b, mask, none, x);
        } else {   // from zero
          pair_sweep0<MAC, PC_RUN>(a.co, o, b, mask, x);
        }
        pair_store<PC_RUN>(L, o, A, x);
        pc_sync(L);
        pair_sweep<MAC, PC_RUN>(a.co, L, o, A, b, mask, last, x);
        pair_store<PC_RUN>(L, o, D, x);
        pc_sync(L);
        const int I0 = lo(l + 1, 0), I1 = hi(l + 1, 0), bc = base(l + 1), mc = Lc.m, J = o.c >> 1;
        auto outlet = [&](int r) { return a.mac_outlet && o.ga + r == L.n - 1; };
        float2 ra{0.f, 0.f};
        float w[PC_RUN / 2];   // the coarse rows of the run
        pair_resid<PC_RUN>(a.co, L, o, D, b, outlet, x, [&](int r, float2 v) {
          // runs start at even rows: rows r - 1 and r of a 2x2 block; summed in
          // the order (0,0), (1,0), (0,1), (1,1)
          if (r & 1) w[r / 2] = 0.25f * (ra.x + v.x + ra.y + v.y);
          ra = v;
        });
        const int Ia = o.ga >> 1, qc = (Ia - bc) * mc + J;
        auto put = [&](float* dst, int off, int from, int to) {
#pragma unroll
          for (int i = 0; i < PC_RUN / 2; ++i)
            if (2 * i < o.cnt && Ia + i >= max(I0, from) && Ia + i < min(I1, to))
              dst[qc + off + i * mc] = w[i];
        };
        put(Bc, 0, I0, I1);
        pc_push(cl, Bc, Lc, Lc.H, rank, put);
      }
      cl.sync();
    }
    if (tid < a.lv[nl].active) {   // coarsest: ten sweeps from zero
      const PcLvl& L = a.lv[nl];
      const int m = L.m;
      const PcOwn o = pc_own<1>(L, rank);
      float x[PC_RUN_COARSE], b[PC_RUN_COARSE], k[PC_RUN_COARSE];
#pragma unroll
      for (int r = 0; r < PC_RUN_COARSE; ++r) {
        const bool in = r < o.cnt;
        b[r] = in ? arr(nl, 0)[o.q + r * m] : 0.f;
        k[r] = MAC && in ? msk(nl)[o.q + r * m] : 1.f;
        x[r] = pair_div(0.f - b[r], a.co);
        if (MAC) x[r] = x[r] * k[r];
      }
      const bool last = o.ga + o.cnt >= o.ghi;
      float *S = arr(nl, 1), *T = arr(nl, 2);   // A and D in turn: the tenth iterate in D
      for (int s = 0; s < 10; ++s) {
#pragma unroll
        for (int r = 0; r < PC_RUN_COARSE; ++r)
          if (r < o.cnt) S[o.q + r * m] = x[r];
        pc_sync(L);
        if (s == 9) break;
        float prev = o.cnt > 0 && o.ga > o.glo ? S[o.q - m] : x[0];
        const float below = o.cnt > 0 && !last ? S[o.q + o.cnt * m] : 0.f;
#pragma unroll
        for (int r = 0; r < PC_RUN_COARSE; ++r) {
          if (r >= o.cnt) break;
          const int q = o.q + r * m;
          const float cur = x[r], end = last ? cur : below;
          const float next =
              r + 1 < PC_RUN_COARSE && r + 1 < o.cnt ? x[r + 1 < PC_RUN_COARSE ? r + 1 : r] : end;
          const float yp = o.c + 1 < m ? S[q + 1] : cur, ym = o.c > 0 ? S[q - 1] : cur;
          const float p = pair_div(fmaf(a.co.ay, yp + ym, a.co.ax * (next + prev)) - b[r], a.co);
          x[r] = MAC ? p * k[r] : p;
          prev = cur;
        }
        float* t = S;
        S = T;
        T = t;
      }
    }
    __syncthreads();
    // up: D + P(e), two post-sweeps (the second resets the outlet row); the
    // last visit is level lt's
    df rr{0.f, 0.f}, bb{0.f, 0.f};
    for (int l = nl - 1; l >= lt; --l) {
      const PcLvl& L = a.lv[l];
      const int nc = a.lv[l + 1].n, mc = a.lv[l + 1].m, bc = base(l + 1);
      const float* E = arr(l + 1, l + 1 == nl ? 2 : 3);
      float *A = arr(l, 1), *D = arr(l, 2), *F = arr(l, 3);
      const int ga = lo(l, 0), gb = hi(l, 0);
      auto none = [](int) { return false; };
      float2 x[PC_RUN], b[PC_RUN];
      PcOwn o;
      if (tid < L.active) {
        o = pc_own<2>(L, rank);
        const float* M = msk(l);
        auto mask = [&](int r) { return pair_ld(M + o.q + r * L.m); };
        auto last = [&](int r) { return a.zero_last && o.ga + r == L.n - 1; };
        pair_load<PC_RUN>(L, o, arr(l, 0), b);
        pair_load<PC_RUN>(L, o, D, x);
        // (the coarse array holds every row this reads; those past its valid
        // halo go into fine halo rows that no sweep needs)
        const int J = o.c >> 1;
        const float* e = E + ((o.ga >> 1) - bc) * mc + J;
        pair_prolong<PC_RUN>(o, nc, J <= mc - 2, [&](int i, int d) { return e[i * mc + d]; }, x);
        pair_store<PC_RUN>(L, o, A, x);
        pc_sync(L);
        pair_sweep<MAC, PC_RUN>(a.co, L, o, A, b, mask, none, x);
        pair_store<PC_RUN>(L, o, D, x);
        pc_sync(L);
        pair_sweep<MAC, PC_RUN>(a.co, L, o, D, b, mask, last, x);
        if (l == lt && !a.whole) {   // straight to global memory (m is even)
#pragma unroll
          for (int r = 0; r < PC_RUN; ++r) {
            const int gi = o.ga + r;
            if (r < o.cnt && gi >= ga && gi < gb) pair_st(a.x + (long)gi * L.m + o.c, x[r]);
          }
        } else {
          // own rows, and what the neighbours' halos need of them: two rows for
          // the finer level's prolongation, four as the next cycle's start
          auto put = [&](float* dst, int off, int from, int to) {
#pragma unroll
            for (int r = 0; r < PC_RUN; ++r) {
              const int gi = o.ga + r;
              if (r < o.cnt && gi >= max(ga, from) && gi < min(gb, to))
                pair_st(dst + o.q + off + r * L.m, x[r]);
            }
          };
          put(F, 0, ga, gb);
          pc_push(cl, F, L, l == 0 ? PC_HALO : 2, rank, put);
        }
      }
      if (l == lt && !a.whole) return;
      cl.sync();
      // level 0: the residual norm (multigrid_solver.py:222-232): exact
      // squares, their sums compensated (TwoSum), one FP64 value per block
      if (l > 0 || tid >= L.active) continue;
      auto outlet = [&](int r) { return a.mac_outlet && o.ga + r == L.n - 1; };
      pair_load<PC_RUN>(L, o, F, x);   // the halo rows too, as the neighbours stored them
      pair_resid<PC_RUN>(a.co, L, o, F, b, outlet, x, [&](int r, float2 v) {
        const int gi = o.ga + r;
        if (gi < ga || gi >= gb) return;
        rr = pair_add_sq(rr, v);
        if (cyc == 0) bb = pair_add_sq(bb, b[r]);
      });
    }
    if (!a.whole) break;   // the coarsest level alone
    // the early-exit test, the blocks' sums added by every block alike (FP64
    // in one warp only: it runs at 1/64 of the FP32 rate)
#pragma unroll 1
    for (int q = 0; q < (cyc == 0 ? 2 : 1); ++q) {
      const df s = warp_sum_df(q ? bb : rr);
      if ((tid & 31) == 0) wsum[q * PC_WARPS + (tid >> 5)] = s;
    }
    __syncthreads();
    // the residual's by warp 0, b's by warp 1 (first cycle)
    const int which = tid >> 5, lane = tid & 31;
    const bool adds = tid < (cyc == 0 ? 64 : 32);
    if (adds) {   // the warps' sums; lane q files the block's in block q
      const double t = warp_sum(df_double(wsum[tid]));
      if (lane < C) cl.map_shared_rank(nrm, lane)[which * PC_MAX_CTAS + rank] = t;
    }
    cl.sync();
    if (adds) {
      const double t = warp_sum<PC_MAX_CTAS>(lane < C ? nrm[which * PC_MAX_CTAS + lane] : 0.0);
      if (lane == 0) sq[which] = t;
      if (tid == 0) stop = t * a.dxdy < a.tol2;
    }
    cycles = cyc + 1;
    __syncthreads();
    if (stop) break;
  }
  // the result: level lt's own rows
  const PcLvl& L = a.lv[lt];
  const int m = L.m, bl = base(lt), g0 = lo(lt, 0), cnt = (hi(lt, 0) - g0) * m;
  const float* F = arr(lt, a.whole ? 3 : 2) + (g0 - bl) * m;
  for (int q = tid; q < cnt; q += PC_THREADS) a.x[(long)g0 * m + q] = F[q];
  if (a.whole && rank == 0 && tid == 0) {
    DevScalars* sc = a.sc;
    const float dt = sc->dt;
    const double rsq = sq[0], bsq = sq[1];
    const int conv = stop, err = isfinite(rsq) ? AJ_OK : AJ_ERR_NONFINITE;
    const double bnorm = sqrt(bsq), abs_sq = rsq * a.dxdy;
    const double rel = bnorm > 0.0 ? sqrt(rsq) / bnorm : sqrt(rsq);
    sc->red_count = 0u;
    sc->mg_skip = conv;
    sc->mg_cycles = cycles;
    sc->acc[0] = sc->acc[1] = 0.0;
    sc->err = err;
    sc->bnorm = bnorm;
    sc->rel = rel;
    sc->abs_sq = abs_sq;
    if (a.stats) {
      a.stats->cycles = cycles;
      a.stats->converged = conv;
      a.stats->err = err;
      a.stats->pad = 0;
      a.stats->rel_residual = rel;
      a.stats->rhs_norm = bnorm;
      a.stats->dt = dt;
      a.stats->abs_residual_sq = abs_sq;
    }
  }
}

// ------------------------------------------------------------------ launch
// the attributes of both instances on the current device
static bool pc_attrs() {
  bool ok = true;
  for (auto f : {k_par_cluster<false>, k_par_cluster<true>})
    ok = ok &&
         cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kBlockSmemMax) == cudaSuccess &&
         cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess;
  return ok;
}

// blocks per cluster: 16 (beyond the portable 8) where the device takes it
static int pc_max_ctas() {
  static const int n = [] {
    pc_attrs();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(PC_MAX_CTAS);
    cfg.blockDim = dim3(PC_THREADS);
    cfg.dynamicSmemBytes = kBlockSmemMax;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = PC_MAX_CTAS;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int k = 0;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&k, k_par_cluster<true>, &cfg);
    cudaGetLastError();
    return e == cudaSuccess && k > 0 ? PC_MAX_CTAS : 8;
  }();
  return n;
}

// the bands of levels lt .. nl over C blocks; returns the dynamic shared
// memory in bytes, 0 where a thread's run of rows would be too long
static size_t pc_levels(const Layout& L, int lt, int C, bool mac, PcLvl* lv) {
  const int nl = L.nlev;
  const int Rc = (L.ln[nl] + C - 1) / C;
  size_t off = 0;
  for (int l = lt; l <= nl; ++l) {
    PcLvl& v = lv[l];
    v.n = L.ln[l];
    v.m = L.lm[l];
    v.R = Rc << (nl - l);
    v.H = l == nl ? PC_HALO_COARSE : PC_HALO;
    const int cols = l == nl ? v.m : v.m / 2, rows = v.R + 2 * v.H;
    if (cols > PC_THREADS) return 0;
    const int groups = PC_THREADS / cols;
    // two rows a thread while half the threads suffice, else four
    if (l == nl) v.run = (int)cdiv(rows, groups);
    else v.run = (rows / 2) * cols <= PC_THREADS / 2 ? 2 : PC_RUN;
    if (v.run > PC_RUN_COARSE || (int)cdiv(rows, v.run) > groups) return 0;
    v.active = (int)cdiv((long)cdiv(rows, v.run) * cols, 32) * 32;
    v.inv_cols = 1.f / cols;
    v.off = (int)off;
    off += (size_t)((l == nl ? 3 : 4) + (mac ? 1 : 0)) * rows * v.m;
  }
  return off * sizeof(float);
}

static int pc_ctas(const Layout& L) {
  int C = pc_max_ctas();
  while (C > 1 && C > L.ln[L.nlev]) C /= 2;   // a band of at least one coarsest row
  return C;
}

// The first level the cluster takes; nl + 1 if not even the coarsest one's
// bands fit in shared memory and in the threads' runs.  The whole solve where
// level 0 fits (a cycle, collocated: 384x96 18.4 us against 20.5 us with tiled
// level-0 kernels, 512x128 19.5 against 20.4); else the levels whose bands,
// halo included, are at most PC_TAIL_CELLS cells: below that a level's two
// launches cost more than its share of the cluster's time.  Limits of 1000 /
// 1800 / 3600 / none, us a cycle, collocated: 96x2048 25.4 / 25.4 / 24.6 / 27.5,
// 640x256 21.8 / 21.1 / 21.1 / 20.8, 1008x368 24.2 / 24.2 / 24.0 / 26.7, 1024x512
// 27.9 / 26.2 / 26.2 / 26.2, 768x768 28.2 / 27.0 / 27.1 / 27.3, 2048x512 36.9 /
// 35.6 / 35.6 / 36.5, 4096x1024 72.6 / 72.3 / 72.3 / 71.4 (MAC alike).
constexpr int PC_TAIL_CELLS = 1800;
int parity_cluster_level(const AjStepParams& p, const Layout& L) {
  const int C = pc_ctas(L), nl = L.nlev;
  PcLvl lv[AJ_MAX_LEVELS + 1];
  for (int lt = p.flow_type == AJ_FLOW_TAYLOR_GREEN ? nl : 0; lt <= nl; ++lt) {
    const size_t bytes = pc_levels(L, lt, C, p.grid_type == AJ_GRID_MAC, lv);
    if (bytes == 0 || bytes > kBlockSmemMax) continue;
    if (lt == 0 || lt == nl || (lv[lt].R + 2 * lv[lt].H) * lv[lt].m <= PC_TAIL_CELLS) return lt;
  }
  return nl + 1;
}

// Levels lt .. nl of one cycle (b: level lt's right-hand side, x: its result,
// masks: the MAC level masks from level lt on), or with lt = 0 the whole solve.
int launch_parity_cluster(const AjStepParams& p, const Layout& L, void* ws, int lt,
                          const float* const* masks, const float* b, const float* x0, float* x,
                          const int* skip, AjStats* stats, cudaStream_t st) {
  const bool mac = p.grid_type == AJ_GRID_MAC;
  const int vk = p.flow_type == AJ_FLOW_VON_KARMAN;
  ParCluster a{};
  const int C = pc_ctas(L);
  if (!pc_attrs()) return AJ_ERR_CUDA;
  const size_t bytes = pc_levels(L, lt, C, mac, a.lv);
  if (mac)
    for (int l = lt; l <= L.nlev; ++l) a.lv[l].mask = masks[l];
  a.lt = lt;
  a.nl = L.nlev;
  a.whole = lt == 0;
  a.cycles = a.whole ? p.v_cycles : 1;
  a.have_x0 = a.whole && x0;
  a.zero_last = vk;
  a.mac_outlet = mac && vk;
  a.b = b;
  a.x0 = x0;
  a.x = x;
  a.skip = skip;
  a.sc = at<DevScalars>(ws, 0);
  a.stats = stats;
  a.co = parity_coef(p);
  a.dxdy = p.dx * p.dy;
  const double tol = p.mg_tolerance > 0 ? p.mg_tolerance : AJ_PARITY_TOL_DEFAULT;
  a.tol2 = tol * tol;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(PC_THREADS);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  const cudaError_t e = mac ? cudaLaunchKernelEx(&cfg, k_par_cluster<true>, a)
                            : cudaLaunchKernelEx(&cfg, k_par_cluster<false>, a);
  return e == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

}  // namespace aj
