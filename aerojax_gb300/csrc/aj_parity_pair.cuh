// The parity V-cycle's cell arithmetic, shared by the tiled kernels
// (aj_pressure.cu) and the cluster kernel (aj_parity_cluster.cu): a thread owns
// a pair of adjacent columns over a run of rows, the iterate and the
// right-hand side of those cells in registers (two columns to a paired FP32
// instruction), and reads only its neighbours' cells from a shared array.
// The array's ends count as edges (ghost = the cell itself): where they are
// not the domain's, each sweep spoils one more row or column of the halo.
#pragma once
#include "aj_internal.cuh"

namespace aj {

struct PairCoef {
  float ax, ay, den, rden;   // rden = 1 / den
};

inline PairCoef parity_coef(const AjStepParams& p) {
  const double ax = 1.0 / (p.dx * p.dx), ay = 1.0 / (p.dy * p.dy);
  const float den = (float)(2.0 * (ax + ay));
  return PairCoef{(float)ax, (float)ay, den, 1.f / den};
}

// s / den for the sweeps' constant divisor: s rden and one Newton correction
// of the quotient by its exact residual (Markstein 1990), three operations
// instead of a division per cell, and the division's quotient short of under-
// and overflow (an infinite s gives NaN: the norm ends as non-finite either way)
__device__ __forceinline__ float pair_div(float s, const PairCoef& a) {
  const float q = s * a.rden;
  return fmaf(fmaf(-q, a.den, s), a.rden, q);
}
__device__ __forceinline__ float2 pair_div(float2 s, const PairCoef& a) {
  const float2 q = mul2(s, f2(a.rden));
  return fma2(fma2(q, f2(-a.den), s), f2(a.rden), q);
}

__device__ __forceinline__ float2 pair_ld(const float* p) {
  return *reinterpret_cast<const float2*>(p);
}
__device__ __forceinline__ void pair_st(float* p, float2 v) { *reinterpret_cast<float2*>(p) = v; }

// A thread's cells: rows [ga, ga + cnt) of its columns at index q of an array;
// [glo, ghi): the array's rows inside the domain.  The functions below also
// take the kernel's own description L of the array: L.m is its row length, and
// pair_lf, pair_rt say whether a column lies to the left and right.  (Kept in
// the thread's registers, the row length cost the cluster kernel 7 %.)
struct PairOwn {
  int ga, cnt, q, glo, ghi;
};

// What a sweep or residual needs of the neighbours, read from S: the rows
// above and below the run and each row's sides.  All reads are issued before
// any is used; rows past cnt hold anything.
template <int RUN>
struct PairNb {
  float2 above, below;
  float lf[RUN], rt[RUN];
  bool last;   // no row below the run
};
template <int RUN, class G, class O>
__device__ __forceinline__ PairNb<RUN> pair_nb(const G& L, const O& o, const float* S, const float2* x) {
  const int m = L.m;
  PairNb<RUN> t;
  t.last = o.ga + o.cnt >= o.ghi;
  t.above = o.cnt > 0 && o.ga > o.glo ? pair_ld(S + o.q - m) : x[0];
  t.below = o.cnt > 0 && !t.last ? pair_ld(S + o.q + o.cnt * m) : x[0];
#pragma unroll
  for (int r = 0; r < RUN; ++r) {
    t.lf[r] = r < o.cnt && pair_lf(L, o) ? S[o.q + r * m - 1] : x[r].x;
    t.rt[r] = r < o.cnt && pair_rt(L, o) ? S[o.q + r * m + 2] : x[r].y;
  }
  return t;
}
template <int RUN>
__device__ __forceinline__ float2 pair_next(const PairOwn& o, const PairNb<RUN>& t, const float2* x,
                                            int r) {
  const float2 end = t.last ? x[r] : t.below;
  return r + 1 < RUN && r + 1 < o.cnt ? x[r + 1 < RUN ? r + 1 : r] : end;
}

// one undamped Jacobi sweep with edge ghosts (multigrid_solver.py:158-171);
// MAC: times the mask pair k(r); rows where zero(r) are reset to 0
template <bool MAC, int RUN, class G, class O, typename K, typename Z>
__device__ __forceinline__ void pair_sweep(const PairCoef& a, const G& L, const O& o, const float* S,
                                           const float2* b, K&& k, Z&& zero, float2* x) {
  const PairNb<RUN> t = pair_nb<RUN>(L, o, S, x);
  float2 prev = t.above;
#pragma unroll
  for (int r = 0; r < RUN; ++r) {
    const float2 cur = x[r], next = pair_next<RUN>(o, t, x, r);
    const float2 sx = mul2(f2(a.ax), add2(next, prev));
    const float2 sy = add2(make_float2(cur.y, t.rt[r]), make_float2(t.lf[r], cur.x));
    float2 p = pair_div(sub2(fma2(f2(a.ay), sy, sx), b[r]), a);
    if (MAC && r < o.cnt) p = mul2(p, k(r));
    if (zero(r)) p = make_float2(0.f, 0.f);
    x[r] = p;
    prev = cur;
  }
}
// the same from a zero iterate
template <bool MAC, int RUN, typename K>
__device__ __forceinline__ void pair_sweep0(const PairCoef& a, const PairOwn& o, const float2* b,
                                            K&& k, float2* x) {
#pragma unroll
  for (int r = 0; r < RUN; ++r) {
    x[r] = pair_div(sub2(f2(0.f), b[r]), a);
    if (MAC && r < o.cnt) x[r] = mul2(x[r], k(r));
  }
}

// b - A x of the thread's cells (the MAC variant zeroes A x where zero(r)):
// f(r, value pair) for the rows it owns
template <int RUN, class G, class O, typename Z, typename F>
__device__ __forceinline__ void pair_resid(const PairCoef& a, const G& L, const O& o, const float* S,
                                           const float2* b, Z&& zero, const float2* x, F&& f) {
  const PairNb<RUN> t = pair_nb<RUN>(L, o, S, x);
  float2 prev = t.above;
#pragma unroll
  for (int r = 0; r < RUN; ++r) {
    const float2 cur = x[r], next = pair_next<RUN>(o, t, x, r), two = mul2(cur, f2(2.f));
    const float2 sx = mul2(f2(a.ax), sub2(add2(next, prev), two));
    const float2 sy = sub2(add2(make_float2(cur.y, t.rt[r]), make_float2(t.lf[r], cur.x)), two);
    float2 lap = fma2(f2(a.ay), sy, sx);
    if (zero(r)) lap = make_float2(0.f, 0.f);
    if (r < o.cnt) f(r, sub2(b[r], lap));
    prev = cur;
  }
}

// x += the reference prolongation (multigrid_solver.py:134-156) of the coarse
// rows from I0 = ga / 2 (ga even): e(i, d) the coarse cell of row I0 + i and
// column J + d, 0 where there is none; in: column J + 1 exists.  Even columns
// are a coarse column, odd ones its mean with the next (0 past the last); odd
// rows the mean of their two coarse rows, the last one 0.
template <int RUN, typename E>
__device__ __forceinline__ void pair_prolong(const PairOwn& o, int nc, bool in, E&& e, float2* x) {
  const int I0 = o.ga >> 1;
  float2 w[RUN / 2 + 1];
#pragma unroll
  for (int i = 0; i <= RUN / 2; ++i) {
    const bool ok = 2 * i <= o.cnt && o.cnt > 0;
    w[i].x = ok ? e(i, 0) : 0.f;
    w[i].y = ok && in ? e(i, 1) : 0.f;
  }
#pragma unroll
  for (int r = 0; r < RUN; ++r) {
    const float2 u = w[r / 2], v = w[r / 2 + 1];
    float2 p;
    if (r & 1) {
      const bool mid = I0 + r / 2 <= nc - 2;
      p.x = mid ? 0.5f * (u.x + v.x) : 0.f;
      p.y = mid && in ? 0.25f * (u.x + v.x + u.y + v.y) : 0.f;
    } else {
      p.x = u.x;
      p.y = in ? 0.5f * (u.x + u.y) : 0.f;
    }
    x[r] = add2(x[r], p);
  }
}

template <int RUN, class G, class O>
__device__ __forceinline__ void pair_load(const G& L, const O& o, const float* S, float2* v) {
#pragma unroll
  for (int r = 0; r < RUN; ++r)
    v[r] = r < o.cnt ? pair_ld(S + o.q + r * L.m) : make_float2(0.f, 0.f);
}
template <int RUN, class G, class O>
__device__ __forceinline__ void pair_store(const G& L, const O& o, float* S, const float2* v) {
#pragma unroll
  for (int r = 0; r < RUN; ++r)
    if (r < o.cnt) pair_st(S + o.q + r * L.m, v[r]);
}

// s + v.x^2 + v.y^2, the squares exact (TwoProd).  Against df_add of one square
// after the other the norms' mean error is 2 % smaller (four pairs a thread,
// random fields), a cycle at 512x96 0.2 us shorter.
__device__ __forceinline__ df pair_add_sq(df s, float2 v) {
  const df p = two_prod(v.x, v.x), q = two_prod(v.y, v.y), t = two_sum(p.hi, q.hi);
  return df_add(s, df{t.hi, t.lo + (p.lo + q.lo)});
}

}  // namespace aj
