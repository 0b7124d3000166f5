// Momentum predictor: RK3 / Heun RK2 stages with implicit Brinkman
// penalisation, upwind or WENO5 advection, Laplacian (+ biharmonic) diffusion,
// Smagorinsky eddy viscosity and the CFL time step.
//
// Collocated stages follow advection_schemes/rk3_simple_new.py:175-358; the
// MAC stages follow advection_schemes/rk3_mac.py:220-504.  Each stage is one
// kernel that reads the stage input with its halo straight from global memory
// (L1/L2 serve the neighbour re-reads) and writes the stage output.  The last
// stage also applies the hard mask and the boundary conditions, by evaluating
// the stage formula at the cell the boundary condition copies from.
#include "aj_internal.cuh"
#include <algorithm>
#include <math.h>

namespace aj {

// ============================================================ set-up: chi
// chi = sigmoid(-sdf / (0.1 dx)) when an SDF is given, else 1 - mask
// (rk3_simple_new.py:194-200).  MAC uses chi = 1 - mask interpolated to
// faces on the fly (rk3_mac.py:462-463), so only the collocated array exists.
__global__ void k_chi(const float* __restrict__ mask, const float* __restrict__ sdf,
                      float* __restrict__ chi, long n, float inv_w) {
  long k = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  if (sdf) {
    float x = -sdf[k] * inv_w;
    // logistic function, evaluated on the branch that cannot overflow
    float c = x >= 0.f ? 1.f / (1.f + expf(-x)) : expf(x) / (1.f + expf(x));
    chi[k] = c;
  } else {
    chi[k] = 1.f - mask[k];
  }
}

int launch_chi(const AjStepParams& p, const Layout& L, void* ws, const float* mask,
               const float* sdf, cudaStream_t st) {
  if (p.grid_type != AJ_GRID_COLLOCATED) return AJ_OK;
  long n = (long)p.nx * p.ny;
  k_chi<<<cdiv(n, 256), 256, 0, st>>>(mask, p.has_sdf ? sdf : nullptr, at<float>(ws, L.chi), n,
                                      (float)(1.0 / (0.1 * p.dx)));
  return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

// ============================================================ dt
__global__ void k_set_dt(DevScalars* sc, float dt, float dtc) {
  pdl_wait();
  sc->dt = dt;
  sc->dt_corr = dtc > 0.f ? dtc : dt;
}

int launch_set_dt(const AjStepParams& p, void* ws, cudaStream_t st) {
  launch_pdl(true, k_set_dt, dim3(1), dim3(1), 0, st, at<DevScalars>(ws, 0), (float)p.dt,
             (float)p.dt_correction);
  return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

// A stage's dt: read from the device, or known to the host.  A step with a
// fixed dt needs no launch of its own to put it on the device: its first
// stage writes it for the kernels after it.
struct StageDt {
  DevScalars* write = nullptr;   // first stage of a fixed-dt step
  const float* src = nullptr;    // the device's dt; when known, a word that nothing writes
  float dt = 0.f, dtc = 0.f;
  int known = 0;
};
__device__ __forceinline__ float stage_dt(const StageDt& d) { return d.known ? d.dt : *d.src; }
// (the large kernels do it on their edge blocks' branch: before the loads it
// cost the staggered upwind stages at 4096x2048 223 -> 281 us)
__device__ __forceinline__ void stage_dt_write(const StageDt& d) {
  if (d.write && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0) {
    d.write->dt = d.dt;
    d.write->dt_corr = d.dtc > 0.f ? d.dtc : d.dt;
  }
}

// compute_cfl_timestep (timestepping/cfl_adaptive_dt.py:6-71): block maxima,
// atomicMax, and the last block to finish turns the maximum into dt.
__global__ void k_cfl(const float* __restrict__ u, const float* __restrict__ v, long nu_,
                      long nv_, int mac, DevScalars* sc, float* dt_out, double h, double nu,
                      double cfl, double dt_min, double dt_max, float dtc_host) {
  pdl_wait();
  float m = 0.f;
  const long stride = (long)gridDim.x * blockDim.x;
  const long n = nu_ > nv_ ? nu_ : nv_;
  // grid-stride in batches of CFL_BATCH: a batch's loads are all issued
  // before its maxima
  constexpr int CFL_BATCH = 8;
  for (long k0 = blockIdx.x * (long)blockDim.x + threadIdx.x; k0 < n;
       k0 += CFL_BATCH * stride) {
    float a[CFL_BATCH], b[CFL_BATCH];
#pragma unroll
    for (int q = 0; q < CFL_BATCH; ++q) {
      const long k = k0 + q * stride;
      a[q] = k < nu_ ? u[k] : 0.f;
      b[q] = k < nv_ ? v[k] : 0.f;
    }
#pragma unroll
    for (int q = 0; q < CFL_BATCH; ++q) {
      if (mac) {
        m = fmaxf(m, fabsf(a[q]));
        m = fmaxf(m, fabsf(b[q]));
      } else {
        m = fmaxf(m, sqrtf(a[q] * a[q] + b[q] * b[q]));
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ float wm[32];
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) wm[w] = m;
  __syncthreads();
  if (w == 0) {
    m = lane < (int)(blockDim.x >> 5) ? wm[lane] : 0.f;
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) {
      atomic_max_nonneg(&sc->cfl_max_bits, m);
      __threadfence();
      unsigned int done = atomicAdd(&sc->cfl_count, 1u);
      if (done == gridDim.x - 1) {
        __threadfence();
        float mx = __uint_as_float(atomicAdd(&sc->cfl_max_bits, 0u));
        const double EPS = 1e-12;
        double dtc = h / ((double)mx + EPS);
        double dtv = 0.25 * h * h / (nu + EPS);
        double dt = (dtc < dtv ? dtc : dtv) * cfl;
        dt = dt < dt_max ? dt : dt_max;
        dt = dt > dt_min ? dt : dt_min;
        sc->dt = (float)dt;
        sc->dt_corr = dtc_host > 0.f ? dtc_host : (float)dt;
        if (dt_out) *dt_out = (float)dt;
        sc->cfl_max_bits = 0u;
        sc->cfl_count = 0u;
      }
    }
  }
}

int launch_cfl(const AjStepParams& p, void* ws, const float* u, const float* v, float* dt_out,
               cudaStream_t st) {
  int mac = p.grid_type == AJ_GRID_MAC;
  long nu_ = mac ? (long)(p.nx + 1) * p.ny : (long)p.nx * p.ny;
  long nv_ = mac ? (long)p.nx * (p.ny + 1) : (long)p.nx * p.ny;
  long n = nu_ > nv_ ? nu_ : nv_;
  unsigned blocks = cdiv(n, 256 * 8);
  if (blocks > 1216) blocks = 1216;
  if (blocks < 1) blocks = 1;
  launch_pdl(true, k_cfl, dim3(blocks), dim3(256), 0, st, u, v, nu_, nv_, mac,
             at<DevScalars>(ws, 0), dt_out, p.dx < p.dy ? p.dx : p.dy, p.nu, p.cfl_target,
             p.dt_min, p.dt_max, (float)p.dt_correction);
  return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

// ============================================================ LES
// |S| = sqrt(2(Sxx^2 + Syy^2 + 2 Sxy^2) + 1e-10) with periodic central
// gradients (solver/les_models.py:22-54 via solver/operators.py:11-38).
struct Strain {
  float smag, sxx, syy, sxy;
};

__device__ __forceinline__ Strain strain_at(const float* __restrict__ u,
                                            const float* __restrict__ v, int i, int j, int nx,
                                            int ny, float h2x, float h2y) {
  int ip = wrapi(i + 1, nx), im = wrapi(i - 1, nx), jp = wrapi(j + 1, ny), jm = wrapi(j - 1, ny);
  float du_dx = (ldg(u + (long)ip * ny + j) - ldg(u + (long)im * ny + j)) * h2x;
  float du_dy = (ldg(u + (long)i * ny + jp) - ldg(u + (long)i * ny + jm)) * h2y;
  float dv_dx = (ldg(v + (long)ip * ny + j) - ldg(v + (long)im * ny + j)) * h2x;
  float dv_dy = (ldg(v + (long)i * ny + jp) - ldg(v + (long)i * ny + jm)) * h2y;
  Strain s;
  s.sxx = du_dx;
  s.syy = dv_dy;
  s.sxy = 0.5f * (du_dy + dv_dx);
  s.smag = sqrtf(2.0f * (s.sxx * s.sxx + s.syy * s.syy + 2.0f * s.sxy * s.sxy) + 1e-10f);
  return s;
}

// constant_smagorinsky (les_models.py:179-200): nu_sgs = (C_s Delta)^2 |S|
__global__ void k_les_const(const float* __restrict__ u, const float* __restrict__ v,
                            float* __restrict__ nsg, int nx, int ny, float h2x, float h2y,
                            float coef) {
  pdl_wait();
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= nx || j >= ny) return;
  Strain s = strain_at(u, v, i, j, nx, ny, h2x, h2y);
  nsg[(long)i * ny + j] = coef * s.smag;
}

// constant Smagorinsky on the MAC grid: the strain of the cell-centred
// velocities (solver/operators_mac.py:118-127) formed from the faces on the fly,
// the same arithmetic as k_mac_to_center followed by k_les_const
__global__ void k_les_const_mac(const float* __restrict__ u, const float* __restrict__ v,
                                float* __restrict__ nsg, int nx, int ny, float h2x, float h2y,
                                float coef) {
  pdl_wait();
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= nx || j >= ny) return;
  // rounded like the stored centre values (no contraction into the gradients)
  auto uc = [&](int a, int b) {
    return __fmul_rn(0.5f, __fadd_rn(ldg(u + (long)(a + 1) * ny + b), ldg(u + (long)a * ny + b)));
  };
  auto vc = [&](int a, int b) {
    return __fmul_rn(0.5f,
                     __fadd_rn(ldg(v + (long)a * (ny + 1) + b + 1), ldg(v + (long)a * (ny + 1) + b)));
  };
  const int ip = wrapi(i + 1, nx), im = wrapi(i - 1, nx), jp = wrapi(j + 1, ny),
            jm = wrapi(j - 1, ny);
  const float du_dx = (uc(ip, j) - uc(im, j)) * h2x;
  const float du_dy = (uc(i, jp) - uc(i, jm)) * h2y;
  const float dv_dx = (vc(ip, j) - vc(im, j)) * h2x;
  const float dv_dy = (vc(i, jp) - vc(i, jm)) * h2y;
  const float sxx = du_dx, syy = dv_dy, sxy = 0.5f * (du_dy + dv_dx);
  const float smag = sqrtf(2.0f * (sxx * sxx + syy * syy + 2.0f * sxy * sxy) + 1e-10f);
  nsg[(long)i * ny + j] = coef * smag;
}

// MAC faces to cell centres (solver/operators_mac.py:118-127)
__global__ void k_mac_to_center(const float* __restrict__ u, const float* __restrict__ v,
                                float* __restrict__ uc, float* __restrict__ vc, int nx, int ny) {
  pdl_wait();
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= nx || j >= ny) return;
  uc[(long)i * ny + j] = 0.5f * (u[(long)(i + 1) * ny + j] + u[(long)i * ny + j]);
  vc[(long)i * ny + j] = 0.5f * (v[(long)i * (ny + 1) + j + 1] + v[(long)i * (ny + 1) + j]);
}

// dynamic_smagorinsky (les_models.py:79-176) in one pass down the rows: the
// strain |S|, S_ij; the 5x5 periodic box filters (les_models.py:57-76) of u,
// v, uu, uv, vv and |S| S_ij, five columns, then five rows (the summation
// order is not the reference's 25 rolls; in FP32 the separable sums are as
// close to the FP64 result as the reference's own FP32 evaluation, or closer);
// Leonard stress L_ij, model tensor M_ij and the contractions LM and MM; their
// 3x3 interior averages, C_d = <LM>/(<MM>+1e-8) clipped to [0, 0.2] and
// nu_sgs = C_d Delta^2 |S|.
// A block owns a strip of columns, a thread a column, with five more at each
// end (wrapped), and walks a run of rows.  Each stage works one row behind
// the one before it, on rows that earlier steps left in shared memory for the
// neighbouring columns and in registers for its own: one barrier a row.
// What bounds it: instructions issued.  As four kernels (strain, filter, LM and
// MM, average) it moved 33 arrays through memory; this reads two and writes
// one, with the same bits.
constexpr int DY_THREADS = 256, DY_HALO = 5, DY_LEAD = 7;   // rows from load to result
// Rows a block: 12 of a run's rows are lead.  Up to four rows one block an SM
// covers the grid, and the short chain is worth more than a second block;
// longer runs are halved by two.  us at 152 / 304 blocks (four kernels):
// 256x64 5.8 / 5.8 (6.2), 512x128 7.5 / 8.3 (7.3), 1024x256 16.5 / 11.4 (12.6),
// 2048x512 19.5 at 304 (36), 4096x2048 106 at 304, 112 at 608 (294).
static int dyn_rows(int nx, int strips) {
  auto rows = [&](int blocks) { return (int)cdiv(nx, std::max(1, blocks / strips)); };
  const int one = rows(152);
  return one <= 4 ? std::max(one, 2) : rows(304);
}
struct DynRow {
  float2 uv[3][DY_THREADS + 4], pd[2][DY_THREADS + 4], ft[2][DY_THREADS + 4], lm[2][DY_THREADS + 4];
  float po[2][DY_THREADS + 4];
};
__global__ void __launch_bounds__(DY_THREADS, 2) k_dyn(const float* __restrict__ u,
                                                       const float* __restrict__ v, int nx, int ny,
                                                       int width, int run, float h2x, float h2y,
                                                       float a2, float delta2,
                                                       float* __restrict__ nsg,
                                                       float* __restrict__ cd) {
  pdl_wait();
  __shared__ DynRow S;
  const int t = threadIdx.x + 2;                       // two pad columns at each end
  const int j = blockIdx.x * width + (int)threadIdx.x - DY_HALO;
  const int jw = (j % ny + ny) % ny;
  const int r0 = blockIdx.y * run, r1 = min(r0 + run, nx);
  const bool mine = (int)threadIdx.x >= DY_HALO && (int)threadIdx.x < DY_HALO + width && j < ny;
  const bool inside = j > 0 && j < ny - 1;
  const float inv = 1.0f / 25.0f;
  int row = ((r0 - DY_HALO) % nx + nx) % nx;           // the row that the next load takes
  auto next = [&]() {
    const long k = (long)row * ny + jw;
    row = row + 1 < nx ? row + 1 : 0;
    return make_float2(ldg(u + k), ldg(v + k));
  };
  float2 c0 = make_float2(0.f, 0.f), c1 = c0, c2 = next();   // (u, v), rows k-2, k-1, k
  float2 f0 = c0, f1 = c0, f2_ = c0;                   // filtered (u, v), rows k-6, k-5, k-4
  float2 uvv = c0, fd = c0;                            // filtered (uu, vv), (Pxx, Pyy), row k-5
  float uvt = 0.f, fo = 0.f;                           // filtered uv, Pxy, row k-5
  float2 ha[5], hb[5], hc[5];                          // column sums of (u, v), (uu, vv), (Pxx, Pyy)
  float hd[5], he[5];                                  // and of uv, Pxy: rows k-6 .. k-2
  float sm[7];                                         // |S|, rows k-7 .. k-1
  float2 l[3][3];                                      // (LM, MM), rows k-8 .. k-6, columns j-1 .. j+1
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    ha[q] = hb[q] = hc[q] = c0;
    hd[q] = he[q] = 0.f;
  }
#pragma unroll
  for (int q = 0; q < 7; ++q) sm[q] = 0.f;
#pragma unroll
  for (int q = 0; q < 9; ++q) l[q / 3][q % 3] = c0;
  float2 *uv0 = S.uv[0], *uv1 = S.uv[1], *uv2 = S.uv[2];     // rows k-2, k-1, k
  const int steps = r1 - r0 + DY_HALO + DY_LEAD;
#pragma unroll 5
  for (int n = 0; n < steps; ++n) {                    // row k = r0 - 5 + n is in c2
    const int a = n & 1, b = a ^ 1;                    // this step's slot, the last one's
    const float2 ahead = next();
    uv2[t] = c2;
    // strain at row k - 1
    float2 pd;
    float po;
    {
      const float2 yp = uv1[t + 1], ym = uv1[t - 1];
      const float du_dx = (c2.x - c0.x) * h2x, dv_dx = (c2.y - c0.y) * h2x;
      const float du_dy = (yp.x - ym.x) * h2y, dv_dy = (yp.y - ym.y) * h2y;
      const float sxy = 0.5f * (du_dy + dv_dx);
      const float smag =
          sqrtf(2.0f * (du_dx * du_dx + dv_dy * dv_dy + 2.0f * sxy * sxy) + 1e-10f);
#pragma unroll
      for (int q = 0; q < 6; ++q) sm[q] = sm[q + 1];
      sm[6] = smag;
      pd = make_float2(smag * du_dx, smag * dv_dy);
      po = smag * sxy;
    }
    // column sums at row k - 2
    {
      float2 sa = make_float2(0.f, 0.f), sb = sa, sc = sa;
      float sd = 0.f, se = 0.f;
#pragma unroll
      for (int d = -2; d <= 2; ++d) {
        const float2 w = uv0[t + d];
        sa = add2(sa, w);
        sb = fma2(w, w, sb);
        sd = fmaf(w.x, w.y, sd);
        sc = add2(sc, S.pd[b][t + d]);
        se += S.po[b][t + d];
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        ha[q] = ha[q + 1];
        hb[q] = hb[q + 1];
        hc[q] = hc[q + 1];
        hd[q] = hd[q + 1];
        he[q] = he[q + 1];
      }
      ha[4] = sa;
      hb[4] = sb;
      hc[4] = sc;
      hd[4] = sd;
      he[4] = se;
    }
    S.pd[a][t] = pd;
    S.po[a][t] = po;
    // LM and MM at row k - 5, from the filtered rows k - 6 .. k - 4
    f0 = f1;
    f1 = f2_;
    const float2 uvv1 = uvv, fd1 = fd;
    const float uvt1 = uvt, fo1 = fo;
    {
      float2 sa = make_float2(0.f, 0.f), sb = sa, sc = sa;
      float sd = 0.f, se = 0.f;
#pragma unroll
      for (int d = 0; d < 5; ++d) {
        sa = add2(sa, ha[d]);
        sb = add2(sb, hb[d]);
        sc = add2(sc, hc[d]);
        sd += hd[d];
        se += he[d];
      }
      const float2 i2 = f2(inv);
      f2_ = mul2(sa, i2);
      uvv = mul2(sb, i2);
      fd = mul2(sc, i2);
      uvt = __fmul_rn(sd, inv);
      fo = __fmul_rn(se, inv);
    }
    float2 lmv;
    {
      const float2 yp = S.ft[b][t + 1], ym = S.ft[b][t - 1];
      const float du_dx = (f2_.x - f0.x) * h2x, dv_dx = (f2_.y - f0.y) * h2x;
      const float du_dy = (yp.x - ym.x) * h2y, dv_dy = (yp.y - ym.y) * h2y;
      const float sxy = 0.5f * (du_dy + dv_dx);
      const float smag =
          sqrtf(2.0f * (du_dx * du_dx + dv_dy * dv_dy + 2.0f * sxy * sxy) + 1e-10f);
      const float u_ = f1.x, v_ = f1.y;
      const float L11 = u_ * u_ - uvv1.x, L12 = u_ * v_ - uvt1, L22 = v_ * v_ - uvv1.y;
      const float M11 = a2 * smag * du_dx - fd1.x;
      const float M12 = a2 * smag * sxy - fo1;
      const float M22 = a2 * smag * dv_dy - fd1.y;
      lmv.x = L11 * M11 + L12 * M12 + L22 * M22;
      lmv.y = M11 * M11 + M12 * M12 + M22 * M22;
    }
    S.ft[a][t] = f2_;
    // the average at row k - 7, from LM and MM of rows k - 8 .. k - 6
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      l[0][q] = l[1][q];
      l[1][q] = l[2][q];
      l[2][q] = S.lm[b][t - 1 + q];
    }
    S.lm[a][t] = lmv;
    const int g = r0 - DY_HALO + n - DY_LEAD;
    if (mine && g >= r0) {
      float2 m = make_float2(0.f, 0.f);
      if (inside && g > 0 && g < nx - 1) {
#pragma unroll
        for (int q = 0; q < 9; ++q) m = add2(m, l[q / 3][q % 3]);
        m = mul2(m, f2(1.0f / 9.0f));
      }
      float c = m.x / (m.y + 1e-8f);
      c = fminf(fmaxf(c, 0.0f), 0.2f);
      const long k = (long)g * ny + j;
      nsg[k] = c * delta2 * sm[0];
      if (cd) cd[k] = c;
    }
    c0 = c1;
    c1 = c2;
    c2 = ahead;
    float2* w = uv0;
    uv0 = uv1;
    uv1 = uv2;
    uv2 = w;
    __syncthreads();
  }
}

int launch_les(const AjStepParams& p, const Layout& L, void* ws, int model, const float* u,
               const float* v, int mac_input, float* nsg, float* cd, cudaStream_t st) {
  int nx = p.nx, ny = p.ny;
  dim3 blk(32, 8), grd(cdiv(ny, 32), cdiv(nx, 8));
  float h2x = (float)(1.0 / (2.0 * p.dx)), h2y = (float)(1.0 / (2.0 * p.dy));
  double delta = p.les_delta > 0 ? p.les_delta : sqrt(p.dx * p.dy);
  long n = (long)nx * ny;
  float* D = at<float>(ws, L.dyn);
  const float *uu = u, *vv = v;
  if (mac_input && model == AJ_LES_SMAGORINSKY) {
    double c = p.smagorinsky_constant * delta;
    launch_pdl(true, k_les_const_mac, dim3(grd), dim3(blk), 0, st, u, v, nsg, nx, ny, h2x, h2y,
               (float)(c * c));
    return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
  }
  if (mac_input) {
    float* uc = D;
    float* vc = D + n;
    launch_pdl(true, k_mac_to_center, dim3(grd), dim3(blk), 0, st, u, v, uc, vc, nx, ny);
    uu = uc;
    vv = vc;
  }
  if (model == AJ_LES_SMAGORINSKY) {
    double c = p.smagorinsky_constant * delta;
    launch_pdl(true, k_les_const, dim3(grd), dim3(blk), 0, st, uu, vv, nsg, nx, ny, h2x, h2y,
               (float)(c * c));
  } else if (model == AJ_LES_DYNAMIC) {
    const int strips = (int)cdiv(ny, DY_THREADS - 2 * DY_HALO), width = (int)cdiv(ny, strips);
    const int run = dyn_rows(nx, strips);
    launch_pdl(true, k_dyn, dim3(strips, cdiv(nx, run)), dim3((width + 2 * DY_HALO + 31) / 32 * 32), 0,
               st, uu, vv, nx, ny, width, run, h2x, h2y, 4.0f, (float)(delta * delta), nsg, cd);
  } else {
    return AJ_ERR_PARAM;
  }
  return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

// ============================================================ collocated RK
struct RkArgs {
  const float *uin, *vin, *u0, *v0, *chi, *mask, *nsg, *k1u, *k1v;
  float *uout, *vout, *k1u_out, *k1v_out;
  StageDt dt;
  int nx, ny;
  float idx, idy, idx2, idy2, nu, inv_eta, U, nuh_fac;
  int dc, stage, rk2, flow, slip;
};

__device__ __forceinline__ float lap5(float xp, float xm, float yp, float ym, float c, float idx2,
                                      float idy2) {
  return (xp + xm - 2.f * c) * idx2 + (yp + ym - 2.f * c) * idy2;
}
template <bool PER>
__device__ __forceinline__ float lap_at(const float* __restrict__ f, int i, int j, int nx, int ny,
                                        float idx2, float idy2) {
  float c = ldg(f + (long)i * ny + j);
  float xp = ldg(f + (long)pidx<PER>(i + 1, nx) * ny + j);
  float xm = ldg(f + (long)pidx<PER>(i - 1, nx) * ny + j);
  float yp = ldg(f + (long)i * ny + pidx<PER>(j + 1, ny));
  float ym = ldg(f + (long)i * ny + pidx<PER>(j - 1, ny));
  return lap5(xp, xm, yp, ym, c, idx2, idy2);
}

// WENO5 reconstruction of a derivative from five one-sided differences
// (Jiang & Shu 1996 smoothness indicators and linear weights 1/10, 6/10, 3/10;
// Hamilton-Jacobi form of Jiang & Peng 2000).
__device__ __forceinline__ float weno5(float v1, float v2, float v3, float v4, float v5) {
  const float eps = 1e-6f;
  float b1 = (13.f / 12.f) * (v1 - 2.f * v2 + v3) * (v1 - 2.f * v2 + v3) +
             0.25f * (v1 - 4.f * v2 + 3.f * v3) * (v1 - 4.f * v2 + 3.f * v3);
  float b2 = (13.f / 12.f) * (v2 - 2.f * v3 + v4) * (v2 - 2.f * v3 + v4) +
             0.25f * (v2 - v4) * (v2 - v4);
  float b3 = (13.f / 12.f) * (v3 - 2.f * v4 + v5) * (v3 - 2.f * v4 + v5) +
             0.25f * (3.f * v3 - 4.f * v4 + v5) * (3.f * v3 - 4.f * v4 + v5);
  // the weights' divisions with the fast reciprocal (2 ulp; the denominators,
  // (1e-6 + beta)^2 and the weights' sum, stay far below 2^126 for any
  // velocity field a step can hold)
  float a1 = __fdividef(0.1f, (eps + b1) * (eps + b1));
  float a2 = __fdividef(0.6f, (eps + b2) * (eps + b2));
  float a3 = __fdividef(0.3f, (eps + b3) * (eps + b3));
  float q1 = v1 * (1.f / 3.f) - (7.f / 6.f) * v2 + (11.f / 6.f) * v3;
  float q2 = -v2 * (1.f / 6.f) + (5.f / 6.f) * v3 + v4 * (1.f / 3.f);
  float q3 = v3 * (1.f / 3.f) + (5.f / 6.f) * v4 - v5 * (1.f / 6.f);
  return __fdividef(a1 * q1 + a2 * q2 + a3 * q3, a1 + a2 + a3);
}

// upwind-biased WENO5 derivative of f along one axis at (i, j)
template <bool PER, int AXIS>
__device__ __forceinline__ float weno_d(const float* __restrict__ f, int i, int j, int nx,
                                        int ny, float ih, float vel) {
  float g[7];
  const int c = AXIS == 0 ? i : j, n = AXIS == 0 ? nx : ny;
  if (c >= 3 && c <= n - 4) {   // the seven points lie inside the grid: plain offsets
    const float* q = f + (long)i * ny + j;
    const long st = AXIS == 0 ? ny : 1;
#pragma unroll
    for (int o = -3; o <= 3; ++o) g[o + 3] = ldg(q + o * st);
  } else {
#pragma unroll
    for (int o = -3; o <= 3; ++o) {
      long k = AXIS == 0 ? (long)pidx<PER>(i + o, nx) * ny + j : (long)i * ny + pidx<PER>(j + o, ny);
      g[o + 3] = ldg(f + k);
    }
  }
  // D_m = (f[m+1]-f[m])/h for m = i-3 .. i+2  ->  d[0..5]
  float d0 = (g[1] - g[0]) * ih, d1 = (g[2] - g[1]) * ih, d2 = (g[3] - g[2]) * ih;
  float d3 = (g[4] - g[3]) * ih, d4 = (g[5] - g[4]) * ih, d5 = (g[6] - g[5]) * ih;
  // weno5(d0..d4) upwind of a positive velocity, weno5(d5..d1) otherwise: the
  // operands are chosen first and one reconstruction runs (no divergence
  // where the velocity changes sign inside a warp)
  const bool up = vel > 0.f;
  return weno5(up ? d0 : d5, up ? d1 : d4, up ? d2 : d3, up ? d3 : d2, up ? d4 : d1);
}

// weno5 in the two lanes of paired FP32 instructions, every operation in the
// order and with the contractions of the scalar function in the collocated
// kernel: the two kernels give the same bits there.  The weights' reciprocals are single instructions: their
// arguments are at least 1e-12, and 0 beyond 2^126 as in the scalar function.
__device__ __forceinline__ float rcp_norm(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float2 weno5_pair(float2 v1, float2 v2, float2 v3, float2 v4,
                                             float2 v5) {
  const float2 m2 = f2(-2.f), m4 = f2(-4.f), c13 = f2(13.f / 12.f), c4 = f2(0.25f);
  const float2 s1 = add2(fma2(m2, v2, v1), v3), s2 = add2(fma2(m2, v3, v2), v4),
               s3 = add2(fma2(m2, v4, v3), v5), t = mul2(f2(3.f), v3);
  const float2 e1 = add2(fma2(m4, v2, v1), t), e2 = sub2(v2, v4), e3 = add2(fma2(m4, v4, t), v5);
  const float2 b1 = fma2(mul2(c13, s1), s1, mul2(mul2(c4, e1), e1));
  const float2 b2 = fma2(mul2(c4, e2), e2, mul2(mul2(c13, s2), s2));
  const float2 b3 = fma2(mul2(c13, s3), s3, mul2(mul2(c4, e3), e3));
  auto weight = [](float w, float2 b) {
    const float2 d = add2(f2(1e-6f), b), q = mul2(d, d);
    return mul2(f2(w), make_float2(rcp_norm(q.x), rcp_norm(q.y)));
  };
  const float2 a1 = weight(0.1f, b1), a2 = weight(0.6f, b2), a3 = weight(0.3f, b3);
  const float2 third = f2(1.f / 3.f), m6 = f2(-1.f / 6.f), c56 = f2(5.f / 6.f);
  const float2 q1 = fma2(f2(11.f / 6.f), v3, fma2(v1, third, mul2(f2(-7.f / 6.f), v2)));
  const float2 q2 = fma2(v4, third, fma2(c56, v3, mul2(v2, m6)));
  const float2 q3 = fma2(v5, m6, fma2(v3, third, mul2(c56, v4)));
  const float2 num = fma2(a3, q3, fma2(a2, q2, mul2(a1, q1))), den = add2(add2(a1, a2), a3);
  return make_float2(__fdividef(num.x, den.x), __fdividef(num.y, den.y));
}

// weno_d7 in pairs: g[0..6] the samples -3 .. 3 of each lane
__device__ __forceinline__ float2 weno_d7_pair(const float2 (&g)[7], float ih, float2 vel) {
  float2 d[6];
#pragma unroll
  for (int q = 0; q < 6; ++q) d[q] = mul2(sub2(g[q + 1], g[q]), f2(ih));
  const bool ux = vel.x > 0.f, uy = vel.y > 0.f;
  float2 v[5];
#pragma unroll
  for (int q = 0; q < 5; ++q)
    v[q] = make_float2(ux ? d[q].x : d[5 - q].x, uy ? d[q].y : d[5 - q].y);
  return weno5_pair(v[0], v[1], v[2], v[3], v[4]);
}

// the Laplacian's Laplacian at a cell two or more from every edge, from the 13
// values it touches (first letter: row i + 1 (p) or i - 1 (m), second: column)
__device__ __forceinline__ float bih13(const RkArgs& a, float fc, float fxp, float fxm, float fyp,
                                       float fym, float xp2, float xm2, float yp2, float ym2,
                                       float pp, float pm, float mp, float mm, float lap) {
  const float lxp = lap5(xp2, fc, pp, pm, fxp, a.idx2, a.idy2);    // lap_at(i + 1, j)
  const float lxm = lap5(fc, xm2, mp, mm, fxm, a.idx2, a.idy2);    // lap_at(i - 1, j)
  const float lyp = lap5(pp, mp, yp2, fc, fyp, a.idx2, a.idy2);    // lap_at(i, j + 1)
  const float lym = lap5(pm, mm, fc, ym2, fym, a.idx2, a.idy2);    // lap_at(i, j - 1)
  return (lxp + lxm - 2.f * lap) * a.idx2 + (lyp + lym - 2.f * lap) * a.idy2;
}
// first-order upwind advection
__device__ __forceinline__ float upwind5(const RkArgs& a, float fc, float fxp, float fxm,
                                         float fyp, float fym, float uc, float vc) {
  float fx = uc > 0.f ? uc * (fc - fxm) * a.idx : uc * (fxp - fc) * a.idx;
  float fy = vc > 0.f ? vc * (fc - fym) * a.idy : vc * (fyp - fc) * a.idy;
  return fx + fy;
}
// the right-hand side from its terms; s: nu_sgs (0 without)
template <bool HYPER>
__device__ __forceinline__ float rhs_sum(const RkArgs& a, float adv, float lap, float bih, float s) {
  float nu_arg = a.dc ? a.nu + s : a.nu;              // the GUI passes nu + nu_sgs as nu
  float nut = a.nsg ? nu_arg + s : nu_arg;            // rk: nu + nu_sgs
  float r = -adv + nut * lap;
  if (HYPER) r -= nu_arg * a.nuh_fac * bih;
  return r;
}
// the stage's update of x0 with slope r (k1: the first slope, RK2's last stage)
__device__ __forceinline__ float stage_sum(const RkArgs& a, float x0, float r, float chi, float k1,
                                           float dt) {
  float den = 1.f + dt * chi * a.inv_eta;
  if (a.rk2) {
    if (a.stage == 1) return brinkman_div(x0 + dt * r, den);
    return brinkman_div(x0 + 0.5f * dt * (k1 + r), den);
  }
  if (a.stage == 1) return brinkman_div(x0 + dt * r, den);
  float xs = x0 + dt * r;
  if (a.stage == 2) return brinkman_div(0.75f * x0 + 0.25f * xs, den);
  return brinkman_div((1.f / 3.f) * x0 + (2.f / 3.f) * xs, den);
}

// explicit right-hand side for one velocity component f at (i, j)
// (rk3_simple_new.py:284-313)
template <bool PER, bool HYPER, int ADV>
__device__ __forceinline__ float rhs_comp(const RkArgs& a, const float* __restrict__ f, int i,
                                          int j) {
  const int nx = a.nx, ny = a.ny;
  long k = (long)i * ny + j;
  float uc = ldg(a.uin + k), vc = ldg(a.vin + k);
  // Cells two or more from every edge: each value the advection, the
  // Laplacian and the bi-Laplacian touch lies inside the grid unclamped, so
  // the 13 distinct values are loaded once instead of 25 clamped loads; the
  // Laplacians are lap_at's expressions on the same values.
  const bool inner = i >= 2 && i <= nx - 3 && j >= 2 && j <= ny - 3;
  float fc, fxm, fxp, fym, fyp, lap, bih = 0.f;
  if (inner) {
    const float* q = f + k;
    fc = ldg(q);
    fxm = ldg(q - ny);
    fxp = ldg(q + ny);
    fym = ldg(q - 1);
    fyp = ldg(q + 1);
    lap = lap5(fxp, fxm, fyp, fym, fc, a.idx2, a.idy2);
    if (HYPER) {
      const float xp2 = ldg(q + 2 * ny), xm2 = ldg(q - 2 * ny), yp2 = ldg(q + 2), ym2 = ldg(q - 2);
      const float pp = ldg(q + ny + 1), pm = ldg(q + ny - 1), mp = ldg(q - ny + 1),
                  mm = ldg(q - ny - 1);
      bih = bih13(a, fc, fxp, fxm, fyp, fym, xp2, xm2, yp2, ym2, pp, pm, mp, mm, lap);
    }
  } else {
    fc = ldg(f + k);
    fxm = ldg(f + (long)pidx<PER>(i - 1, nx) * ny + j);
    fxp = ldg(f + (long)pidx<PER>(i + 1, nx) * ny + j);
    fym = ldg(f + (long)i * ny + pidx<PER>(j - 1, ny));
    fyp = ldg(f + (long)i * ny + pidx<PER>(j + 1, ny));
    lap = lap_at<PER>(f, i, j, nx, ny, a.idx2, a.idy2);
    if (HYPER) {
      // biharmonic = Laplacian of the edge-padded Laplacian
      int ip = pidx<PER>(i + 1, nx), im = pidx<PER>(i - 1, nx);
      int jp = pidx<PER>(j + 1, ny), jm = pidx<PER>(j - 1, ny);
      float lxp = lap_at<PER>(f, ip, j, nx, ny, a.idx2, a.idy2);
      float lxm = lap_at<PER>(f, im, j, nx, ny, a.idx2, a.idy2);
      float lyp = lap_at<PER>(f, i, jp, nx, ny, a.idx2, a.idy2);
      float lym = lap_at<PER>(f, i, jm, nx, ny, a.idx2, a.idy2);
      bih = (lxp + lxm - 2.f * lap) * a.idx2 + (lyp + lym - 2.f * lap) * a.idy2;
    }
  }
  float adv;
  if (ADV == AJ_ADV_WENO5) {
    adv = uc * weno_d<PER, 0>(f, i, j, nx, ny, a.idx, uc) +
          vc * weno_d<PER, 1>(f, i, j, nx, ny, a.idy, vc);
  } else {
    adv = upwind5(a, fc, fxp, fxm, fyp, fym, uc, vc);
  }
  return rhs_sum<HYPER>(a, adv, lap, bih, a.nsg ? ldg(a.nsg + k) : 0.f);
}

// stage update of one component at (i, j); returns the stage output
template <bool PER, bool HYPER, int ADV>
__device__ __forceinline__ float stage_val(const RkArgs& a, const float* f, const float* f0,
                                           const float* k1, float* k1_out, int i, int j,
                                           float dt) {
  long k = (long)i * a.ny + j;
  // the cell's own reads beside the stencil's: after the store of k1 the
  // compiler leaves them behind it, a round trip of their own (three upwind
  // stages at 3001x1503 157 us, so 123)
  const float x0 = ldg(f0 + k), chi = ldg(a.chi + k);
  const float g = a.rk2 && a.stage == 2 ? ldg(k1 + k) : 0.f;
  const float r = rhs_comp<PER, HYPER, ADV>(a, f, i, j);
  if (a.rk2 && a.stage == 1 && k1_out) k1_out[k] = r;
  return stage_sum(a, x0, r, chi, g, dt);
}

// one stage of component COMP at (i, j).  The last stage applies the hard mask
// (rk3_simple_new.py:334-335), then the boundary conditions (:250-280): a
// value, or the stage at the cell that the boundary copies from.  One
// evaluation for all of them: with one at each branch the kernel waited on
// instruction fetches (WENO5 128x32 three stages 21 us).
template <bool PER, bool HYPER, int ADV, int COMP>
__device__ __forceinline__ void rk_col_one(const RkArgs& a, int i, int j, float dt) {
  const int nx = a.nx, ny = a.ny;
  const bool last = a.rk2 ? a.stage == 2 : a.stage == 3;
  int ii = i, jj = j;
  float o = 0.f;
  bool set = false;
  if (last) {
    const bool wall = j == 0 || j == ny - 1, end = i == 0 || i == nx - 1;
    if (a.flow == AJ_FLOW_VON_KARMAN) {
      ii = i == nx - 1 ? nx - 2 : i;
      if (COMP == 0) {
        set = i == 0 || (!a.slip && wall);
        if (i == 0 && (a.slip || !wall)) o = a.U;
        if (a.slip) jj = j == 0 ? 1 : (j == ny - 1 ? ny - 2 : j);
      } else {
        set = i == 0 || wall;
      }
    } else if (a.flow == AJ_FLOW_LID_DRIVEN_CAVITY) {
      set = end || wall;
      if (COMP == 0 && !end && j == ny - 1 && j != 0) o = a.U;
    }
    if (!set) set = !(ldg(a.mask + (long)ii * ny + jj) > 0.5f);
  }
  if (!set)
    o = COMP == 0 ? stage_val<PER, HYPER, ADV>(a, a.uin, a.u0, a.k1u, last ? nullptr : a.k1u_out, ii, jj, dt)
                  : stage_val<PER, HYPER, ADV>(a, a.vin, a.v0, a.k1v, last ? nullptr : a.k1v_out, ii, jj, dt);
  (COMP == 0 ? a.uout : a.vout)[(long)i * ny + j] = o;
}
template <bool PER, bool HYPER, int ADV>
__device__ __forceinline__ void rk_col_cell(const RkArgs& a, int i, int j, float dt) {
  const bool last = a.rk2 ? a.stage == 2 : a.stage == 3;
  if (!last || PER) {   // no boundary conditions
    // both components in one scope share their loads (a periodic grid's last
    // stage apart, with one component a branch: three stages at 3001x1503,
    // upwind, 142 us, so 135; WENO5 1000x252 28, so 25)
    const long k = (long)i * a.ny + j;
    if (last && !(ldg(a.mask + k) > 0.5f)) {
      a.uout[k] = a.vout[k] = 0.f;
      return;
    }
    a.uout[k] = stage_val<PER, HYPER, ADV>(a, a.uin, a.u0, a.k1u, a.k1u_out, i, j, dt);
    a.vout[k] = stage_val<PER, HYPER, ADV>(a, a.vin, a.v0, a.k1v, a.k1v_out, i, j, dt);
    return;
  }
  rk_col_one<PER, HYPER, ADV, 0>(a, i, j, dt);
  rk_col_one<PER, HYPER, ADV, 1>(a, i, j, dt);
}

template <bool PER, bool HYPER, int ADV>
__global__ void __launch_bounds__(256) k_rk_col(RkArgs a) {
  pdl_wait();
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  int i = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= a.nx || j >= a.ny) return;
  stage_dt_write(a.dt);
  rk_col_cell<PER, HYPER, ADV>(a, i, j, stage_dt(a.dt));
}

// The upwind stage four columns a thread: 16-byte reads of the five rows that
// the Laplacian and the bi-Laplacian touch serve four cells where each cell
// read its 13 values by itself (27 reads for four cells instead of 120; the
// stage waited on them, at half the SM's warps).  Cells that lie within two
// of an edge, and their vectors' others, go cell by cell on the first blocks.
__host__ __device__ inline int rk4_edge_blocks(int nx, int ny) {
  return (4 * ny + 8 * (nx - 4) + 255) / 256;
}
template <bool HYPER>
__global__ void __launch_bounds__(256) k_rk_col4(RkArgs a) {
  pdl_wait();
  const int nx = a.nx, ny = a.ny;
  const float dt = stage_dt(a.dt);
  const int edge = rk4_edge_blocks(nx, ny);
  if ((int)blockIdx.x < edge) {   // a cell each: two rows, four columns at each end
    stage_dt_write(a.dt);
    const int e = blockIdx.x * 256 + threadIdx.y * 32 + threadIdx.x, f = e - 4 * ny;
    if (f < 0) rk_col_cell<false, HYPER, AJ_ADV_UPWIND>(a, e < 2 * ny ? e / ny : nx - 4 + e / ny, e % ny, dt);
    else if (f < 8 * (nx - 4))
      rk_col_cell<false, HYPER, AJ_ADV_UPWIND>(a, 2 + f / 8, f % 8 < 4 ? f % 8 : ny - 8 + f % 8, dt);
    return;
  }
  const int bj = (ny + 127) / 128, b = blockIdx.x - edge;
  const int j = (b % bj * 32 + threadIdx.x) * 4, i = b / bj * 8 + threadIdx.y;
  if (i < 2 || i > nx - 3 || j < 4 || j > ny - 8) return;
  const long k = (long)i * ny + j;
  const bool last = a.rk2 ? a.stage == 2 : a.stage == 3;
  struct F4 {
    float v[4];
  };
  auto ld = [&](const float* p) {
    const float4 t = __ldg(reinterpret_cast<const float4*>(p));
    return F4{t.x, t.y, t.z, t.w};
  };
  const F4 uc = ld(a.uin + k), vc = ld(a.vin + k), chi = ld(a.chi + k);
  const F4 sg = a.nsg ? ld(a.nsg + k) : F4{0.f, 0.f, 0.f, 0.f};
  const F4 mk = last ? ld(a.mask + k) : F4{1.f, 1.f, 1.f, 1.f};
  auto component = [&](const float* f, const F4& fc, const float* f0, const float* k1,
                       float* k1_out, float* out) {
    const float* q = f + k;
    const F4 xm = ld(q - ny), xp = ld(q + ny), x0 = ld(f0 + k);
    const F4 g = a.rk2 && last ? ld(k1 + k) : F4{0.f, 0.f, 0.f, 0.f};
    // columns j - 2 .. j + 5 of row i, j - 1 .. j + 4 of rows i - 1 and i + 1
    float c[8] = {0.f, 0.f, fc.v[0], fc.v[1], fc.v[2], fc.v[3], 0.f, 0.f};
    float m[6] = {0.f, xm.v[0], xm.v[1], xm.v[2], xm.v[3], 0.f};
    float p[6] = {0.f, xp.v[0], xp.v[1], xp.v[2], xp.v[3], 0.f};
    F4 xm2{}, xp2{};
    if (HYPER) {
      const float2 l = __ldg(reinterpret_cast<const float2*>(q - 2));
      const float2 r = __ldg(reinterpret_cast<const float2*>(q + 4));
      c[0] = l.x, c[1] = l.y, c[6] = r.x, c[7] = r.y;
      m[0] = ldg(q - ny - 1), m[5] = ldg(q - ny + 4);
      p[0] = ldg(q + ny - 1), p[5] = ldg(q + ny + 4);
      xm2 = ld(q - 2 * (long)ny);
      xp2 = ld(q + 2 * (long)ny);
    } else {
      c[1] = ldg(q - 1), c[6] = ldg(q + 4);
    }
    float o[4], slope[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float w = c[t + 2], yp = c[t + 3], ym = c[t + 1];
      const float lap = lap5(p[t + 1], m[t + 1], yp, ym, w, a.idx2, a.idy2);
      const float bih = HYPER ? bih13(a, w, p[t + 1], m[t + 1], yp, ym, xp2.v[t], xm2.v[t],
                                      c[t + 4], c[t], p[t + 2], p[t], m[t + 2], m[t], lap)
                              : 0.f;
      const float adv = upwind5(a, w, p[t + 1], m[t + 1], yp, ym, uc.v[t], vc.v[t]);
      slope[t] = rhs_sum<HYPER>(a, adv, lap, bih, sg.v[t]);
      const float x = stage_sum(a, x0.v[t], slope[t], chi.v[t], g.v[t], dt);
      o[t] = mk.v[t] > 0.5f ? x : 0.f;
    }
    if (a.rk2 && !last && k1_out)
      *reinterpret_cast<float4*>(k1_out + k) = make_float4(slope[0], slope[1], slope[2], slope[3]);
    *reinterpret_cast<float4*>(out + k) = make_float4(o[0], o[1], o[2], o[3]);
  };
  component(a.uin, uc, a.u0, a.k1u, a.k1u_out, a.uout);
  component(a.vin, vc, a.v0, a.k1v, a.k1v_out, a.vout);
}
constexpr int RK4_MIN_NY = 64;
constexpr long RK4_MIN_CELLS = 1 << 17;
// whether a stage runs four columns a thread: whole 16-byte rows, every array
// aligned, and a grid large enough that the blocks' number does not set the
// time.  Three stages, plain / with hyperviscosity, us, a cell a thread ->
// four: 512x128 7.5 / 11.2 -> 8.0 / 10.5, 1024x256 12.2 / 19.0 -> 9.4 / 12.1,
// 2048x512 28.1 / 45.7 -> 19.7 / 27.6, 4096x2048 294 / 392 -> 147 / 200.
static bool rk_col4_ok(const RkArgs& a) {
  if (a.ny % 4 || a.ny < RK4_MIN_NY || a.nx < 8 || (long)a.nx * a.ny < RK4_MIN_CELLS) return false;
  for (const void* p : {(const void*)a.uin, (const void*)a.vin, (const void*)a.u0,
                        (const void*)a.v0, (const void*)a.chi, (const void*)a.mask,
                        (const void*)a.nsg, (const void*)a.uout, (const void*)a.vout})
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;
  return true;
}

// WENO5 stages, non-periodic, a run of rows a thread: the thread walks R cells
// in x with its column's seven u and v in registers, and the two components
// are the lanes of paired FP32 instructions, reconstructions included (both
// components share the advecting velocity).  What bounds it: instructions
// issued.  Cells within three of an edge go one component a thread on the
// first blocks.  Three stages, us, a cell a thread -> this: 128x32 10.4 -> 9.9,
// 512x128 12.4 -> 10.6, 1024x256 24.7 -> 17.1, 2048x512 68 -> 47.
struct ColRows {
  static constexpr int HB = 3, R = 2;
  __host__ __device__ static int edge_blocks(int nx, int ny) {
    return (2 * 2 * HB * (ny + nx - 2 * HB) + 255) / 256;
  }
};
__global__ void __launch_bounds__(256, 4) k_rk_col_rows(RkArgs a) {
  pdl_wait();
  constexpr int HB = ColRows::HB, R = ColRows::R, E = 2 * HB;
  const int nx = a.nx, ny = a.ny;
  const float dt = stage_dt(a.dt);
  const int edge = ColRows::edge_blocks(nx, ny);
  if ((int)blockIdx.x < edge) {
    stage_dt_write(a.dt);
    const int cells = E * (ny + nx - 2 * HB);
    int e = blockIdx.x * 256 + threadIdx.y * 32 + threadIdx.x;
    if (e >= 2 * cells) return;
    const bool comp = e >= cells;
    if (comp) e -= cells;
    const int f = e - E * ny, q = f < 0 ? e / ny : f % E;
    const int i = f < 0 ? (q < HB ? q : nx - E + q) : HB + f / E;
    const int j = f < 0 ? e % ny : (q < HB ? q : ny - E + q);
    if (comp) rk_col_one<false, false, AJ_ADV_WENO5, 1>(a, i, j, dt);
    else rk_col_one<false, false, AJ_ADV_WENO5, 0>(a, i, j, dt);
    return;
  }
  const int bj = (ny + 31) / 32, b = blockIdx.x - edge;
  const int j = b % bj * 32 + threadIdx.x, i0 = HB + (b / bj * 8 + threadIdx.y) * R;
  if (j < HB || j > ny - 1 - HB || i0 > nx - 1 - HB) return;
  const bool last = a.rk2 ? a.stage == 2 : a.stage == 3;
  long k = (long)i0 * ny + j;
  auto at = [&](long q) { return make_float2(ldg(a.uin + q), ldg(a.vin + q)); };
  float2 x[7];   // column j, rows i - 3 .. i + 3
#pragma unroll
  for (int q = 1; q < 7; ++q) x[q] = at(k + (long)(q - 4) * ny);
#pragma unroll
  for (int r = 0; r < R; ++r, k += ny) {
    if (i0 + r > nx - 1 - HB) break;
#pragma unroll
    for (int q = 0; q < 6; ++q) x[q] = x[q + 1];
    x[6] = at(k + 3 * (long)ny);
    const float2 c = x[3];
    const float2 y[7] = {at(k - 3), at(k - 2), at(k - 1), c, at(k + 1), at(k + 2), at(k + 3)};
    const float2 adv = fma2(f2(c.y), weno_d7_pair(y, a.idy, f2(c.y)),
                            mul2(f2(c.x), weno_d7_pair(x, a.idx, f2(c.x))));
    const float s = a.nsg ? ldg(a.nsg + k) : 0.f, chi = ldg(a.chi + k);
    const float lu = lap5(x[4].x, x[2].x, y[4].x, y[2].x, c.x, a.idx2, a.idy2);
    const float lv = lap5(x[4].y, x[2].y, y[4].y, y[2].y, c.y, a.idx2, a.idy2);
    const float ru = rhs_sum<false>(a, adv.x, lu, 0.f, s), rv = rhs_sum<false>(a, adv.y, lv, 0.f, s);
    if (a.rk2 && !last && a.k1u_out) {
      a.k1u_out[k] = ru;
      a.k1v_out[k] = rv;
    }
    const bool two = a.rk2 && last;
    float uo = stage_sum(a, ldg(a.u0 + k), ru, chi, two ? ldg(a.k1u + k) : 0.f, dt);
    float vo = stage_sum(a, ldg(a.v0 + k), rv, chi, two ? ldg(a.k1v + k) : 0.f, dt);
    if (last && !(ldg(a.mask + k) > 0.5f)) uo = vo = 0.f;
    a.uout[k] = uo;
    a.vout[k] = vo;
  }
}

template <bool PER>
static void dispatch_rk_col(const RkArgs& a, bool hyper, int adv, dim3 g, dim3 b, cudaStream_t st) {
  if (!PER && adv == AJ_ADV_UPWIND && rk_col4_ok(a)) {
    const dim3 g4(rk4_edge_blocks(a.nx, a.ny) + cdiv(a.ny, 128) * cdiv(a.nx, 8));
    if (hyper) launch_pdl(true, k_rk_col4<true>, dim3(g4), dim3(32, 8), 0, st, a);
    else launch_pdl(true, k_rk_col4<false>, dim3(g4), dim3(32, 8), 0, st, a);
    return;
  }
  if (!PER && !hyper && adv == AJ_ADV_WENO5 && a.nx > 4 * ColRows::HB && a.ny > 4 * ColRows::HB) {
    const unsigned rows = cdiv(a.nx - 2 * ColRows::HB, 8 * ColRows::R);
    launch_pdl(true, k_rk_col_rows,
               dim3(ColRows::edge_blocks(a.nx, a.ny) + rows * cdiv(a.ny, 32)), dim3(32, 8), 0, st,
               a);
    return;
  }
  if (hyper) {
    if (adv == AJ_ADV_WENO5) launch_pdl(true, k_rk_col<PER, true, AJ_ADV_WENO5>, dim3(g), dim3(b),
                                        0, st, a);
    else launch_pdl(true, k_rk_col<PER, true, AJ_ADV_UPWIND>, dim3(g), dim3(b), 0, st, a);
  } else {
    if (adv == AJ_ADV_WENO5) launch_pdl(true, k_rk_col<PER, false, AJ_ADV_WENO5>, dim3(g), dim3(b),
                                        0, st, a);
    else launch_pdl(true, k_rk_col<PER, false, AJ_ADV_UPWIND>, dim3(g), dim3(b), 0, st, a);
  }
}

// ============================================================ MAC RK
// u: (nx+1) x ny faces, v: nx x (ny+1) faces, mask / nu_sgs: nx x ny cells.
struct RkMac {
  const float *uin, *vin, *u0, *v0, *mask, *nsg, *k1u, *k1v;
  float *uout, *vout, *k1u_out, *k1v_out;
  StageDt dt;
  int nx, ny;
  float idx, idy, idx2, idy2, nu, inv_eta, U, nuh;
  int stage, rk2, flow, slip;
};

// velocities after the boundary conditions of rk3_mac.py:292-330, the
// working copy the advection term uses (:381)
__device__ __forceinline__ float uw_at(const RkMac& a, const float* __restrict__ u, int i, int j) {
  const int nx = a.nx, ny = a.ny;
  if (a.flow == AJ_FLOW_VON_KARMAN) {
    if (!a.slip && (j == 0 || j == ny - 1)) return 0.f;
    if (i == 0) return a.U;
    int ii = i == nx ? nx - 1 : i;
    int jj = a.slip ? (j == 0 ? 1 : (j == ny - 1 ? ny - 2 : j)) : j;
    return ldg(u + (long)ii * ny + jj);
  } else if (a.flow == AJ_FLOW_LID_DRIVEN_CAVITY) {
    if (i == 0 || i == nx) return 0.f;
    if (j == 0) return 0.f;
    if (j == ny - 1) return a.U;
    return ldg(u + (long)i * ny + j);
  }
  return ldg(u + (long)i * ny + j);
}

__device__ __forceinline__ float vw_at(const RkMac& a, const float* __restrict__ v, int i, int j) {
  const int nx = a.nx, ny = a.ny;
  const int nyv = ny + 1;
  if (a.flow == AJ_FLOW_VON_KARMAN) {
    if (i == 0 || j == 0 || j == ny) return 0.f;
    int ii = i == nx - 1 ? nx - 2 : i;
    return ldg(v + (long)ii * nyv + j);
  } else if (a.flow == AJ_FLOW_LID_DRIVEN_CAVITY) {
    if (i == 0 || i == nx - 1 || j == 0 || j == ny) return 0.f;
    return ldg(v + (long)i * nyv + j);
  }
  return ldg(v + (long)i * nyv + j);
}

// Laplacian on faces with symmetric (== edge for one cell) ghosts for slip
// walls, or antisymmetric wall ghosts for no-slip (rk3_mac.py:268-290)
template <int COMP>
__device__ __forceinline__ float lap_face(const RkMac& a, const float* __restrict__ f, int i,
                                          int j) {
  const int n = COMP == 0 ? a.nx + 1 : a.nx;
  const int m = COMP == 0 ? a.ny : a.ny + 1;
  float c = ldg(f + (long)i * m + j);
  float xp, xm, yp, ym;
  if (a.slip) {
    xp = ldg(f + (long)clampi(i + 1, n) * m + j);
    xm = ldg(f + (long)clampi(i - 1, n) * m + j);
    yp = ldg(f + (long)i * m + clampi(j + 1, m));
    ym = ldg(f + (long)i * m + clampi(j - 1, m));
  } else if (COMP == 0) {
    // y ghosts are -f at the wall, then x padded by edge
    xp = ldg(f + (long)clampi(i + 1, n) * m + j);
    xm = ldg(f + (long)clampi(i - 1, n) * m + j);
    yp = j + 1 < m ? ldg(f + (long)i * m + j + 1) : -c;
    ym = j - 1 >= 0 ? ldg(f + (long)i * m + j - 1) : -c;
  } else {
    xp = i + 1 < n ? ldg(f + (long)(i + 1) * m + j) : -c;
    xm = i - 1 >= 0 ? ldg(f + (long)(i - 1) * m + j) : -c;
    yp = ldg(f + (long)i * m + clampi(j + 1, m));
    ym = ldg(f + (long)i * m + clampi(j - 1, m));
  }
  return (xp + xm - 2.f * c) * a.idx2 + (yp + ym - 2.f * c) * a.idy2;
}

template <int COMP>
__device__ __forceinline__ float bih_face(const RkMac& a, const float* __restrict__ f, int i,
                                          int j, float lc) {
  // Laplacian of the face Laplacian with the same ghost rule
  const int n = COMP == 0 ? a.nx + 1 : a.nx;
  const int m = COMP == 0 ? a.ny : a.ny + 1;
  float xp, xm, yp, ym;
  if (a.slip) {
    xp = lap_face<COMP>(a, f, clampi(i + 1, n), j);
    xm = lap_face<COMP>(a, f, clampi(i - 1, n), j);
    yp = lap_face<COMP>(a, f, i, clampi(j + 1, m));
    ym = lap_face<COMP>(a, f, i, clampi(j - 1, m));
  } else if (COMP == 0) {
    xp = lap_face<COMP>(a, f, clampi(i + 1, n), j);
    xm = lap_face<COMP>(a, f, clampi(i - 1, n), j);
    yp = j + 1 < m ? lap_face<COMP>(a, f, i, j + 1) : -lc;
    ym = j - 1 >= 0 ? lap_face<COMP>(a, f, i, j - 1) : -lc;
  } else {
    xp = i + 1 < n ? lap_face<COMP>(a, f, i + 1, j) : -lc;
    xm = i - 1 >= 0 ? lap_face<COMP>(a, f, i - 1, j) : -lc;
    yp = lap_face<COMP>(a, f, i, clampi(j + 1, m));
    ym = lap_face<COMP>(a, f, i, clampi(j - 1, m));
  }
  return (xp + xm - 2.f * lc) * a.idx2 + (yp + ym - 2.f * lc) * a.idy2;
}

// x-face interpolation of a cell field (operators_mac.py:130-137)
__device__ __forceinline__ float xface(const float* __restrict__ c, int i, int j, int nx, int ny) {
  return 0.5f * (ldg(c + (long)clampi(i, nx) * ny + j) + ldg(c + (long)clampi(i - 1, nx) * ny + j));
}
__device__ __forceinline__ float yface(const float* __restrict__ c, int i, int j, int nx, int ny) {
  return 0.5f * (ldg(c + (long)i * ny + clampi(j, ny)) + ldg(c + (long)i * ny + clampi(j - 1, ny)));
}

// u-momentum right-hand side at u-face (i, j) (rk3_mac.py:373-400, 425-458)
template <bool HYPER>
__device__ float rhs_mac_u(const RkMac& a, int i, int j) {
  const int nx = a.nx, ny = a.ny;
  float uw = uw_at(a, a.uin, i, j);
  // v at the u-face: centre average of v_work, edge-padded in x, face average
  auto vcen = [&](int ci) {
    ci = clampi(ci, nx);
    return 0.5f * (vw_at(a, a.vin, ci, j + 1) + vw_at(a, a.vin, ci, j));
  };
  float v_at_u = 0.5f * (vcen(i) + vcen(i - 1));
  // the periodic (Taylor-Green) flow wraps both differences (rk3_mac.py's
  // wrap padding and np.roll), every other flow pads by the edge
  const bool per = a.flow == AJ_FLOW_TAYLOR_GREEN;
  float uxm = uw_at(a, a.uin, per ? wrapi(i - 1, nx + 1) : (i > 0 ? i - 1 : 0), j);
  float uxp = uw_at(a, a.uin, per ? wrapi(i + 1, nx + 1) : (i < nx ? i + 1 : nx), j);
  float back = (uw - uxm) * a.idx, fwd = (uxp - uw) * a.idx;
  // upwind blend 0.5 (1 + tanh(u / 0.05)) of rk3_mac.py (upwind_weight)
  float al = upwind_weight(uw);
  float adv_x = uw * (al * back + (1.f - al) * fwd);
  float du_dy;
  if (per)
    du_dy = (uw_at(a, a.uin, i, wrapi(j + 1, ny)) - uw_at(a, a.uin, i, wrapi(j - 1, ny))) *
            (0.5f * a.idy);
  else if (j == 0) du_dy = (uw_at(a, a.uin, i, 1) - uw) * a.idy;
  else if (j == ny - 1) du_dy = (uw - uw_at(a, a.uin, i, ny - 2)) * a.idy;
  else du_dy = (uw_at(a, a.uin, i, j + 1) - uw_at(a, a.uin, i, j - 1)) * (0.5f * a.idy);
  float adv = (adv_x + v_at_u * du_dy) * xface(a.mask, i, j, nx, ny);
  float lap = lap_face<0>(a, a.uin, i, j);
  float nut = a.nsg ? a.nu + xface(a.nsg, i, j, nx, ny) : a.nu;
  float r = -adv + nut * lap;
  if (HYPER) r -= a.nuh * bih_face<0>(a, a.uin, i, j, lap);
  return r;
}

template <bool HYPER>
__device__ float rhs_mac_v(const RkMac& a, int i, int j) {
  const int nx = a.nx, ny = a.ny;
  float vw = vw_at(a, a.vin, i, j);
  auto ucen = [&](int cj) {
    cj = clampi(cj, ny);
    return 0.5f * (uw_at(a, a.uin, i + 1, cj) + uw_at(a, a.uin, i, cj));
  };
  float u_at_v = 0.5f * (ucen(j) + ucen(j - 1));
  const bool per = a.flow == AJ_FLOW_TAYLOR_GREEN;
  float vym = vw_at(a, a.vin, i, per ? wrapi(j - 1, ny + 1) : (j > 0 ? j - 1 : 0));
  float vyp = vw_at(a, a.vin, i, per ? wrapi(j + 1, ny + 1) : (j < ny ? j + 1 : ny));
  float back = (vw - vym) * a.idy, fwd = (vyp - vw) * a.idy;
  float al = upwind_weight(vw);
  float adv_y = vw * (al * back + (1.f - al) * fwd);
  float dv_dx;
  if (per)
    dv_dx = (vw_at(a, a.vin, wrapi(i + 1, nx), j) - vw_at(a, a.vin, wrapi(i - 1, nx), j)) *
            (0.5f * a.idx);
  else if (i == 0) dv_dx = (vw_at(a, a.vin, 1, j) - vw) * a.idx;
  else if (i == nx - 1) dv_dx = (vw - vw_at(a, a.vin, nx - 2, j)) * a.idx;
  else dv_dx = (vw_at(a, a.vin, i + 1, j) - vw_at(a, a.vin, i - 1, j)) * (0.5f * a.idx);
  float adv = (u_at_v * dv_dx + adv_y) * yface(a.mask, i, j, nx, ny);
  float lap = lap_face<1>(a, a.vin, i, j);
  float nut = a.nsg ? a.nu + yface(a.nsg, i, j, nx, ny) : a.nu;
  float r = -adv + nut * lap;
  if (HYPER) r -= a.nuh * bih_face<1>(a, a.vin, i, j, lap);
  return r;
}

// RK stage update of one face from its right-hand side r and face chi
template <int COMP>
__device__ __forceinline__ float finish_mac(const RkMac& a, long k, float r, float chi, float dt,
                                            float* k1o) {
  float x0 = ldg((COMP == 0 ? a.u0 : a.v0) + k);
  float den = 1.f + dt * chi * a.inv_eta;
  if (a.rk2) {
    if (a.stage == 1) {
      if (k1o) k1o[k] = r;
      return brinkman_div(x0 + dt * r, den);
    }
    float out = brinkman_div(x0 + 0.5f * dt * (ldg((COMP == 0 ? a.k1u : a.k1v) + k) + r), den);
    return chi < 0.5f ? out : 0.f;                   // hard mask (rk3_mac.py:498-499)
  }
  if (a.stage == 1) return brinkman_div(x0 + dt * r, den);
  float xs = x0 + dt * r;
  if (a.stage == 2) return brinkman_div(0.75f * x0 + 0.25f * xs, den);
  float out = brinkman_div((1.f / 3.f) * x0 + (2.f / 3.f) * xs, den);
  return chi < 0.5f ? out : 0.f;                     // hard mask (rk3_mac.py:483-484)
}

template <int COMP, bool HYPER>
__device__ __forceinline__ float stage_mac(const RkMac& a, int i, int j, float dt, float* k1o) {
  const int m = COMP == 0 ? a.ny : a.ny + 1;
  long k = (long)i * m + j;
  float r = COMP == 0 ? rhs_mac_u<HYPER>(a, i, j) : rhs_mac_v<HYPER>(a, i, j);
  // chi on faces = face average of (1 - mask)
  float chi;
  if (COMP == 0) {
    chi = 0.5f * ((1.f - ldg(a.mask + (long)clampi(i, a.nx) * a.ny + j)) +
                  (1.f - ldg(a.mask + (long)clampi(i - 1, a.nx) * a.ny + j)));
  } else {
    chi = 0.5f * ((1.f - ldg(a.mask + (long)i * a.ny + clampi(j, a.ny))) +
                  (1.f - ldg(a.mask + (long)i * a.ny + clampi(j - 1, a.ny))));
  }
  return finish_mac<COMP>(a, k, r, chi, dt, k1o);
}

// ------------------------------------------------------------ MAC WENO5
// WENO5-JS on the staggered grid (no reference counterpart; the reference's
// MAC advection is the blended upwind above, rk3_mac.py:373-417).  Both
// derivatives of both components use the upwind WENO5 reconstruction of
// weno5() on the boundary-conditioned working copies, upwinded on the sign of
// the advecting velocity at the face, with ghost values three cells deep by
// edge padding (non-periodic flows) or wrap (Taylor-Green):
//   adv_u = u d_x(u) + v_at_u d_y(u),   adv_v = u_at_v d_x(v) + v d_y(v).
// FAST: the face and every value its stencils read lie in the interior of the
// slip-wall von Karman channel, where the working copy is the input itself.
template <bool FAST>
__device__ __forceinline__ float uw_f(const RkMac& a, int i, int j) {
  return FAST ? ldg(a.uin + (long)i * a.ny + j) : uw_at(a, a.uin, i, j);
}
template <bool FAST>
__device__ __forceinline__ float vw_f(const RkMac& a, int i, int j) {
  return FAST ? ldg(a.vin + (long)i * (a.ny + 1) + j) : vw_at(a, a.vin, i, j);
}

// ghost index of a WENO5 stencil: edge (clamp) or periodic wrap
__device__ __forceinline__ int widx(int i, int n, bool per) {
  return per ? wrapi(i, n) : clampi(i, n);
}

// upwind WENO5 derivative from seven samples g[0..6] = f[i-3 .. i+3]
__device__ __forceinline__ float weno_d7(const float (&g)[7], float ih, float vel) {
  float d0 = (g[1] - g[0]) * ih, d1 = (g[2] - g[1]) * ih, d2 = (g[3] - g[2]) * ih;
  float d3 = (g[4] - g[3]) * ih, d4 = (g[5] - g[4]) * ih, d5 = (g[6] - g[5]) * ih;
  const bool up = vel > 0.f;   // operands first, one reconstruction (as in weno_d)
  return weno5(up ? d0 : d5, up ? d1 : d4, up ? d2 : d3, up ? d3 : d2, up ? d4 : d1);
}

template <bool HYPER, bool FAST>
__device__ float rhs_mac_u_weno(const RkMac& a, int i, int j) {
  const int nx = a.nx, ny = a.ny;
  const bool per = a.flow == AJ_FLOW_TAYLOR_GREEN;
  const float uw = uw_f<FAST>(a, i, j);
  auto vcen = [&](int ci) {
    ci = clampi(ci, nx);
    return 0.5f * (vw_f<FAST>(a, ci, j + 1) + vw_f<FAST>(a, ci, j));
  };
  const float v_at_u = 0.5f * (vcen(i) + vcen(i - 1));
  float g[7];
#pragma unroll
  for (int o = -3; o <= 3; ++o) g[o + 3] = uw_f<FAST>(a, FAST ? i + o : widx(i + o, nx + 1, per), j);
  const float dudx = weno_d7(g, a.idx, uw);
#pragma unroll
  for (int o = -3; o <= 3; ++o) g[o + 3] = uw_f<FAST>(a, i, FAST ? j + o : widx(j + o, ny, per));
  const float dudy = weno_d7(g, a.idy, v_at_u);
  const float adv = (uw * dudx + v_at_u * dudy) * xface(a.mask, i, j, nx, ny);
  const float lap = lap_face<0>(a, a.uin, i, j);
  const float nut = a.nsg ? a.nu + xface(a.nsg, i, j, nx, ny) : a.nu;
  float r = -adv + nut * lap;
  if (HYPER) r -= a.nuh * bih_face<0>(a, a.uin, i, j, lap);
  return r;
}

template <bool HYPER, bool FAST>
__device__ float rhs_mac_v_weno(const RkMac& a, int i, int j) {
  const int nx = a.nx, ny = a.ny;
  const bool per = a.flow == AJ_FLOW_TAYLOR_GREEN;
  const float vw = vw_f<FAST>(a, i, j);
  auto ucen = [&](int cj) {
    cj = clampi(cj, ny);
    return 0.5f * (uw_f<FAST>(a, i + 1, cj) + uw_f<FAST>(a, i, cj));
  };
  const float u_at_v = 0.5f * (ucen(j) + ucen(j - 1));
  float g[7];
#pragma unroll
  for (int o = -3; o <= 3; ++o) g[o + 3] = vw_f<FAST>(a, FAST ? i + o : widx(i + o, nx, per), j);
  const float dvdx = weno_d7(g, a.idx, u_at_v);
#pragma unroll
  for (int o = -3; o <= 3; ++o) g[o + 3] = vw_f<FAST>(a, i, FAST ? j + o : widx(j + o, ny + 1, per));
  const float dvdy = weno_d7(g, a.idy, vw);
  const float adv = (u_at_v * dvdx + vw * dvdy) * yface(a.mask, i, j, nx, ny);
  const float lap = lap_face<1>(a, a.vin, i, j);
  const float nut = a.nsg ? a.nu + yface(a.nsg, i, j, nx, ny) : a.nu;
  float r = -adv + nut * lap;
  if (HYPER) r -= a.nuh * bih_face<1>(a, a.vin, i, j, lap);
  return r;
}

// one stage of one face, upwind (the reference) or WENO5
template <int COMP, bool HYPER, int ADV, bool FAST = false>
__device__ __forceinline__ float stage_mac_any(const RkMac& a, int i, int j, float dt, float* k1o) {
  if (ADV != AJ_ADV_WENO5) return stage_mac<COMP, HYPER>(a, i, j, dt, k1o);
  const int m = COMP == 0 ? a.ny : a.ny + 1;
  const long k = (long)i * m + j;
  const float r = COMP == 0 ? rhs_mac_u_weno<HYPER, FAST>(a, i, j)
                            : rhs_mac_v_weno<HYPER, FAST>(a, i, j);
  float chi;
  if (COMP == 0) {
    chi = 0.5f * ((1.f - ldg(a.mask + (long)clampi(i, a.nx) * a.ny + j)) +
                  (1.f - ldg(a.mask + (long)clampi(i - 1, a.nx) * a.ny + j)));
  } else {
    chi = 0.5f * ((1.f - ldg(a.mask + (long)i * a.ny + clampi(j, a.ny))) +
                  (1.f - ldg(a.mask + (long)i * a.ny + clampi(j - 1, a.ny))));
  }
  return finish_mac<COMP>(a, k, r, chi, dt, k1o);
}

// Interior faces of the von Karman channel with slip walls (u faces
// 2 <= i <= nx-2, 2 <= j <= ny-3; v faces 2 <= i <= nx-3, 2 <= j <= ny-2):
// every neighbour the stencils touch, including the bi-Laplacian's, is an
// unmodified value of the input field, so the boundary-condition index logic
// drops out.  Same operations in the same order as the general path.
template <bool HYPER>
__device__ __forceinline__ float stage_mac_u_int(const RkMac& a, int i, int j, float dt,
                                                 float* k1o) {
  const int ny = a.ny, nyv = ny + 1;
  const long k = (long)i * ny + j;
  const float* u = a.uin + k;
  const float uw = ldg(u), uxm = ldg(u - ny), uxp = ldg(u + ny), uym = ldg(u - 1),
              uyp = ldg(u + 1);
  const float* v = a.vin + (long)i * nyv + j;
  const float vc_i = 0.5f * (ldg(v + 1) + ldg(v));
  const float vc_m = 0.5f * (ldg(v - nyv + 1) + ldg(v - nyv));
  const float v_at_u = 0.5f * (vc_i + vc_m);
  const float back = (uw - uxm) * a.idx, fwd = (uxp - uw) * a.idx;
  const float al = upwind_weight(uw);
  const float adv_x = uw * (al * back + (1.f - al) * fwd);
  const float du_dy = (uyp - uym) * (0.5f * a.idy);
  const float m_i = ldg(a.mask + k), m_im = ldg(a.mask + k - ny);
  const float adv = (adv_x + v_at_u * du_dy) * (0.5f * (m_i + m_im));
  const float lap = (uxp + uxm - 2.f * uw) * a.idx2 + (uyp + uym - 2.f * uw) * a.idy2;
  const float nut = a.nsg ? a.nu + 0.5f * (ldg(a.nsg + k) + ldg(a.nsg + k - ny)) : a.nu;
  float r = -adv + nut * lap;
  if (HYPER) {
    auto lapat = [&](const float* c) {
      const float cc = ldg(c);
      return (ldg(c + ny) + ldg(c - ny) - 2.f * cc) * a.idx2 +
             (ldg(c + 1) + ldg(c - 1) - 2.f * cc) * a.idy2;
    };
    const float xp = lapat(u + ny), xm = lapat(u - ny), yp = lapat(u + 1), ym = lapat(u - 1);
    r -= a.nuh * ((xp + xm - 2.f * lap) * a.idx2 + (yp + ym - 2.f * lap) * a.idy2);
  }
  const float chi = 0.5f * ((1.f - m_i) + (1.f - m_im));
  return finish_mac<0>(a, k, r, chi, dt, k1o);
}

template <bool HYPER>
__device__ __forceinline__ float stage_mac_v_int(const RkMac& a, int i, int j, float dt,
                                                 float* k1o) {
  const int ny = a.ny, nyv = ny + 1;
  const long k = (long)i * nyv + j;
  const float* v = a.vin + k;
  const float vw = ldg(v), vym = ldg(v - 1), vyp = ldg(v + 1), vxm = ldg(v - nyv),
              vxp = ldg(v + nyv);
  const float* u = a.uin + (long)i * ny + j;
  const float uc_j = 0.5f * (ldg(u + ny) + ldg(u));
  const float uc_m = 0.5f * (ldg(u + ny - 1) + ldg(u - 1));
  const float u_at_v = 0.5f * (uc_j + uc_m);
  const float back = (vw - vym) * a.idy, fwd = (vyp - vw) * a.idy;
  const float al = upwind_weight(vw);
  const float adv_y = vw * (al * back + (1.f - al) * fwd);
  const float dv_dx = (vxp - vxm) * (0.5f * a.idx);
  const long c = (long)i * ny + j;
  const float m_j = ldg(a.mask + c), m_jm = ldg(a.mask + c - 1);
  const float adv = (u_at_v * dv_dx + adv_y) * (0.5f * (m_j + m_jm));
  const float lap = (vxp + vxm - 2.f * vw) * a.idx2 + (vyp + vym - 2.f * vw) * a.idy2;
  const float nut = a.nsg ? a.nu + 0.5f * (ldg(a.nsg + c) + ldg(a.nsg + c - 1)) : a.nu;
  float r = -adv + nut * lap;
  if (HYPER) {
    auto lapat = [&](const float* q) {
      const float cc = ldg(q);
      return (ldg(q + nyv) + ldg(q - nyv) - 2.f * cc) * a.idx2 +
             (ldg(q + 1) + ldg(q - 1) - 2.f * cc) * a.idy2;
    };
    const float xp = lapat(v + nyv), xm = lapat(v - nyv), yp = lapat(v + 1), ym = lapat(v - 1);
    r -= a.nuh * ((xp + xm - 2.f * lap) * a.idx2 + (yp + ym - 2.f * lap) * a.idy2);
  }
  const float chi = 0.5f * ((1.f - m_j) + (1.f - m_jm));
  return finish_mac<1>(a, k, r, chi, dt, k1o);
}

// The values that the two faces of one interior cell read, u-face (i, j) in
// lane x and v-face (i, j) in lane y.  "Along" is a face's own direction (x
// for u, y for v), "across" the other.
struct FacePair {
  float2 c, am, ap, cm, cp;   // the face, its neighbours along and across
  float2 q2, q3;              // the cross velocity's far faces: v at (i-1, j+1), (i-1, j); u at
                              // (i+1, j-1), (i, j-1); its near ones are (vyp, vw) and (uxp, uw)
  float2 mc, mo;              // mask of the cell and of its neighbour across each face
  float2 sc, so;              // eddy viscosity, likewise
};

__device__ __forceinline__ float2 pair_cross(const FacePair& f) {
  const float2 half = f2(0.5f);
  const float2 q0 = make_float2(f.ap.y, f.ap.x), q1 = make_float2(f.c.y, f.c.x);
  return mul2(half, add2(mul2(half, add2(q0, q1)), mul2(half, add2(f.q2, f.q3))));
}

// right-hand side of both faces from the advection before its mask; chi out.
// Every lane evaluates its face's expressions in the order of stage_mac_u_int
// and stage_mac_v_int (products added by fma where those contract).
__device__ __forceinline__ float2 pair_rhs(const RkMac& a, const FacePair& f, float2 adv,
                                           float2& chi) {
  const float2 half = f2(0.5f);
  adv = mul2(adv, mul2(half, add2(f.mc, f.mo)));
  // Laplacian: x terms are u's along and v's across sums, y terms the others
  const float2 s_al = add2(f.ap, f.am), s_ac = add2(f.cp, f.cm);
  const float2 two_c = mul2(f2(2.f), f.c);
  const float2 lap = fma2(sub2(make_float2(s_al.x, s_ac.y), two_c), f2(a.idx2),
                          mul2(sub2(make_float2(s_ac.x, s_al.y), two_c), f2(a.idy2)));
  float2 nut = f2(a.nu);
  if (a.nsg) nut = add2(nut, mul2(half, add2(f.sc, f.so)));
  chi = mul2(half, add2(sub2(f2(1.f), f.mc), sub2(f2(1.f), f.mo)));
  return fma2(nut, lap, make_float2(-adv.x, -adv.y));
}

// the blended upwind advection of both faces
__device__ __forceinline__ float2 pair_upwind(const RkMac& a, const FacePair& f) {
  const float2 cross = pair_cross(f);
  const float2 h_al = make_float2(a.idx, a.idy);
  const float2 back = mul2(sub2(f.c, f.am), h_al), fwd = mul2(sub2(f.ap, f.c), h_al);
  const float2 al = make_float2(upwind_weight(f.c.x), upwind_weight(f.c.y));
  const float2 adv_al = mul2(f.c, fma2(al, back, mul2(sub2(f2(1.f), al), fwd)));
  const float2 d_ac = mul2(sub2(f.cp, f.cm), make_float2(0.5f * a.idy, 0.5f * a.idx));
  return fma2(cross, d_ac, adv_al);
}

// both faces of interior cell (i, j), one cell a thread
__device__ __forceinline__ float2 stage_mac_uv_int(const RkMac& a, int i, int j, float dt,
                                                   float* k1u, float* k1v) {
  const int ny = a.ny, nyv = ny + 1;
  const long ku = (long)i * ny + j, kv = (long)i * nyv + j;
  const float* u = a.uin + ku;
  const float* v = a.vin + kv;
  FacePair f;
  f.c = make_float2(ldg(u), ldg(v));
  f.am = make_float2(ldg(u - ny), ldg(v - 1));
  f.ap = make_float2(ldg(u + ny), ldg(v + 1));
  f.cm = make_float2(ldg(u - 1), ldg(v - nyv));
  f.cp = make_float2(ldg(u + 1), ldg(v + nyv));
  f.q2 = make_float2(ldg(v - nyv + 1), ldg(u + ny - 1));
  f.q3 = make_float2(f.cm.y, f.cm.x);
  f.mc = f2(ldg(a.mask + ku));
  f.mo = make_float2(ldg(a.mask + ku - ny), ldg(a.mask + ku - 1));
  f.sc = f.so = f2(0.f);
  if (a.nsg) {
    f.sc = f2(ldg(a.nsg + ku));
    f.so = make_float2(ldg(a.nsg + ku - ny), ldg(a.nsg + ku - 1));
  }
  float2 chi;
  const float2 r = pair_rhs(a, f, pair_upwind(a, f), chi);
  return make_float2(finish_mac<0>(a, ku, r.x, chi.x, dt, k1u),
                     finish_mac<1>(a, kv, r.y, chi.y, dt, k1v));
}

// one stage of face (i, j) of u (COMP 0) or v; the last one rewrites the
// boundary rows: a value, or the stage of the interior face they copy
template <int COMP, bool HYPER, int ADV>
__device__ __forceinline__ void rk_mac_face(const RkMac& a, int i, int j, float dt) {
  const int nx = a.nx, ny = a.ny, m = COMP == 0 ? ny : ny + 1;
  if (i >= (COMP == 0 ? nx + 1 : nx) || j >= m) return;
  const bool last = a.rk2 ? a.stage == 2 : a.stage == 3;
  int ii = i, jj = j;
  float o = 0.f;
  bool fixed = false;
  if (last && a.flow == AJ_FLOW_VON_KARMAN) {
    if (COMP == 0) {
      fixed = (!a.slip && (j == 0 || j == ny - 1)) || i == 0;
      if (i == 0 && (a.slip || (j != 0 && j != ny - 1))) o = a.U;
      ii = i == nx ? nx - 1 : i;
      jj = a.slip ? (j == 0 ? 1 : (j == ny - 1 ? ny - 2 : j)) : j;
    } else {
      fixed = i == 0 || j == 0 || j == ny;
      ii = i == nx - 1 ? nx - 2 : i;
    }
  } else if (last && a.flow == AJ_FLOW_LID_DRIVEN_CAVITY) {
    if (COMP == 0) {
      fixed = i == 0 || i == nx || j == 0 || j == ny - 1;
      if (i != 0 && i != nx && j == ny - 1 && j != 0) o = a.U;
    } else {
      fixed = i == 0 || i == nx - 1 || j == 0 || j == ny;
    }
  }
  if (!fixed)
    o = stage_mac_any<COMP, HYPER, ADV>(a, ii, jj, dt,
                                        last ? nullptr : (COMP == 0 ? a.k1u_out : a.k1v_out));
  (COMP == 0 ? a.uout : a.vout)[(long)i * m + j] = o;
}

// one stage of face (i, j) of one component, 0 <= i <= nx, 0 <= j <= ny: the
// interior faces of the slip-wall channel without the index logic.  WENO5's
// 7-point stencils and the face velocities stay off the rows that the boundary
// conditions rewrite (u 4 <= i <= nx-4, 4 <= j <= ny-5; v 4 <= i <= nx-5,
// 4 <= j <= ny-4)
template <int COMP, bool HYPER, int ADV>
__device__ __forceinline__ void rk_mac_one(const RkMac& a, int i, int j, float dt) {
  constexpr int HB = ADV == AJ_ADV_WENO5 ? 4 : 2;
  const int ei = COMP == 0 ? a.nx - HB : a.nx - 1 - HB, ej = COMP == 0 ? a.ny - 1 - HB : a.ny - HB;
  if (!(a.flow == AJ_FLOW_VON_KARMAN && a.slip && i >= HB && i <= ei && j >= HB && j <= ej))
    return rk_mac_face<COMP, HYPER, ADV>(a, i, j, dt);
  const bool last = a.rk2 ? a.stage == 2 : a.stage == 3;
  float* k1o = last ? nullptr : (COMP == 0 ? a.k1u_out : a.k1v_out);
  const float o = ADV == AJ_ADV_WENO5 ? stage_mac_any<COMP, HYPER, ADV, true>(a, i, j, dt, k1o)
                  : COMP == 0         ? stage_mac_u_int<HYPER>(a, i, j, dt, k1o)
                                      : stage_mac_v_int<HYPER>(a, i, j, dt, k1o);
  (COMP == 0 ? a.uout : a.vout)[(long)i * (COMP == 0 ? a.ny : a.ny + 1) + j] = o;
}

// The same for the kernel of a cell a thread.  Here the evaluation stands at
// each branch: with rk_mac_face's one for all, and the two components' interior
// reads apart, three stages took 66 us with WENO5 and hyperviscosity at
// 1000x252, so 63; upwind with hyperviscosity at 3001x1503 227, so 222; WENO5
// between no-slip walls there 805, so 756.  (Where threads share a block of edge
// cells, as in k_rk_mac_rows, the one call site wins.)
template <int COMP, bool HYPER, int ADV>
__device__ __forceinline__ void rk_mac_branch(const RkMac& a, int i, int j, float dt) {
  const int nx = a.nx, ny = a.ny, m = COMP == 0 ? ny : ny + 1;
  if (i >= (COMP == 0 ? nx + 1 : nx) || j >= m) return;
  const bool last = a.rk2 ? a.stage == 2 : a.stage == 3;
  constexpr int HB = ADV == AJ_ADV_WENO5 ? 4 : 2;
  const int ei = COMP == 0 ? nx - HB : nx - 1 - HB, ej = COMP == 0 ? ny - 1 - HB : ny - HB;
  float* k1o = last ? nullptr : (COMP == 0 ? a.k1u_out : a.k1v_out);
  auto stage = [&](int ii, int jj) {
    return stage_mac_any<COMP, HYPER, ADV>(a, ii, jj, dt, k1o);
  };
  float o = 0.f;
  if (a.flow == AJ_FLOW_VON_KARMAN && a.slip && i >= HB && i <= ei && j >= HB && j <= ej) {
    if constexpr (ADV == AJ_ADV_WENO5) o = stage_mac_any<COMP, HYPER, ADV, true>(a, i, j, dt, k1o);
    else if constexpr (COMP == 0) o = stage_mac_u_int<HYPER>(a, i, j, dt, k1o);
    else o = stage_mac_v_int<HYPER>(a, i, j, dt, k1o);
  } else if (!last) {
    o = stage(i, j);
  } else if (a.flow == AJ_FLOW_VON_KARMAN) {
    if (COMP == 0) {
      if (!a.slip && (j == 0 || j == ny - 1)) o = 0.f;
      else if (i == 0) o = a.U;
      else o = stage(i == nx ? nx - 1 : i, a.slip ? (j == 0 ? 1 : (j == ny - 1 ? ny - 2 : j)) : j);
    } else if (i != 0 && j != 0 && j != ny) {
      o = stage(i == nx - 1 ? nx - 2 : i, j);
    }
  } else if (a.flow == AJ_FLOW_LID_DRIVEN_CAVITY) {
    if (COMP == 0) {
      if (i == 0 || i == nx || j == 0) o = 0.f;
      else o = j == ny - 1 ? a.U : stage(i, j);
    } else if (i != 0 && i != nx - 1 && j != 0 && j != ny) {
      o = stage(i, j);
    }
  } else {
    o = stage(i, j);
  }
  (COMP == 0 ? a.uout : a.vout)[(long)i * m + j] = o;
}

template <bool HYPER, int ADV>
__global__ void __launch_bounds__(256) k_rk_mac(RkMac a) {
  pdl_wait();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i = blockIdx.y * blockDim.y + threadIdx.y;
  const float dt = stage_dt(a.dt);
  stage_dt_write(a.dt);
  if (ADV != AJ_ADV_WENO5 && a.flow == AJ_FLOW_VON_KARMAN && a.slip && i >= 2 && i <= a.nx - 3 &&
      j >= 2 && j <= a.ny - 3) {
    // both faces of an interior cell in one scope: without hyperviscosity they
    // share the paired FP32 instructions, with it their loads
    const bool last = a.rk2 ? a.stage == 2 : a.stage == 3;
    float uo, vo;
    if (HYPER) {
      uo = stage_mac_u_int<HYPER>(a, i, j, dt, last ? nullptr : a.k1u_out);
      vo = stage_mac_v_int<HYPER>(a, i, j, dt, last ? nullptr : a.k1v_out);
    } else {
      const float2 o = stage_mac_uv_int(a, i, j, dt, last ? nullptr : a.k1u_out,
                                        last ? nullptr : a.k1v_out);
      uo = o.x;
      vo = o.y;
    }
    a.uout[(long)i * a.ny + j] = uo;
    a.vout[(long)i * (a.ny + 1) + j] = vo;
    return;
  }
  rk_mac_branch<0, HYPER, ADV>(a, i, j, dt);
  rk_mac_branch<1, HYPER, ADV>(a, i, j, dt);
}

// The stage of the slip-wall von Karman channel a run of rows a thread: the
// thread walks R cells in x with its columns' values in registers, so a cell
// reads 12 values (WENO5: 21) where one by itself read 20 (58), and both
// faces share the paired FP32 instructions, WENO5's reconstructions too.
// Cells within HB of an edge, where the boundary conditions' index logic
// applies, go one face a thread on the first blocks.  What bounds it:
// instructions issued (WENO5), L2 reads (upwind).  Two rows a thread; one was
// 3 to 5 % slower, four and eight ran out of threads below 2048x512.  Three
// stages, us, a cell a thread -> this, upwind / WENO5: 128x32 13.2 / 21.9 ->
// 11.5 / 14.2, 512x128 15.1 / 26.3 -> 11.8 / 16.0, 1021x509 26.7 / 66 ->
// 18.2 / 33, 2048x512 40 / 113 -> 30 / 58, 4096x2048 236 / 699 -> 223 / 441.
template <int ADV>
struct MacRows {
  static constexpr int HB = ADV == AJ_ADV_WENO5 ? 4 : 2;   // edge cells: i < HB, i > nx-1-HB, ...
  static constexpr int R = 2;
  static constexpr int BLOCKS = ADV == AJ_ADV_WENO5 ? 4 : 5;   // blocks an SM (64, 48 registers)
  __host__ __device__ static int edge_blocks(int nx, int ny) {
    return (2 * (2 * HB + 1) * (ny + 1 + nx - 2 * HB) + 255) / 256;   // u and v faces
  }
};
template <int ADV>
__global__ void __launch_bounds__(256, MacRows<ADV>::BLOCKS) k_rk_mac_rows(RkMac a) {
  pdl_wait();
  using M = MacRows<ADV>;
  constexpr int HB = M::HB, R = M::R;
  const int nx = a.nx, ny = a.ny, nyv = ny + 1;
  // upwind reads src even where the host knows dt (src is then not the scalars'
  // dt, which the first stage's edge block writes): without that read the
  // compiler orders the loads after it differently, and three stages at
  // 4096x2048 take 285 us instead of 223
  const float read = ADV == AJ_ADV_WENO5 ? 0.f : *a.dt.src;
  const float dt = ADV == AJ_ADV_WENO5 ? stage_dt(a.dt) : (a.dt.known ? a.dt.dt : read);
  const int edge = M::edge_blocks(nx, ny);
  if ((int)blockIdx.x < edge) {
    stage_dt_write(a.dt);
    constexpr int E = 2 * HB + 1;   // rows (columns) at both ends
    const int cells = E * (nyv + nx - 2 * HB);
    int e = blockIdx.x * 256 + threadIdx.y * 32 + threadIdx.x;
    if (e >= 2 * cells) return;
    const bool comp = e >= cells;
    if (comp) e -= cells;
    const int f = e - E * nyv, q = f < 0 ? e / nyv : f % E;
    const int i = f < 0 ? (q < HB ? q : nx - 2 * HB + q) : HB + f / E;
    const int j = f < 0 ? e % nyv : (q < HB ? q : ny - 2 * HB + q);
    if (comp) rk_mac_one<1, false, ADV>(a, i, j, dt);
    else rk_mac_one<0, false, ADV>(a, i, j, dt);
    return;
  }
  const int bj = (ny + 31) / 32, b = blockIdx.x - edge;
  const int j = b % bj * 32 + threadIdx.x, i0 = HB + (b / bj * 8 + threadIdx.y) * R;
  if (j < HB || j > ny - 1 - HB || i0 > nx - 1 - HB) return;
  const bool last = a.rk2 ? a.stage == 2 : a.stage == 3;
  float* k1u = last ? nullptr : a.k1u_out;
  float* k1v = last ? nullptr : a.k1v_out;
  const float* u = a.uin + (long)i0 * ny + j;
  const float* v = a.vin + (long)i0 * nyv + j;
  const float* m = a.mask + (long)i0 * ny + j;
  const float* sg = a.nsg ? a.nsg + (long)i0 * ny + j : nullptr;
  constexpr int XW = ADV == AJ_ADV_WENO5 ? 7 : 3, XH = XW / 2;
  float2 x[XW];   // column j of u and v, rows i - XH .. i + XH
#pragma unroll
  for (int q = 1; q < XW; ++q)
    x[q] = make_float2(ldg(u + (long)(q - 1 - XH) * ny), ldg(v + (long)(q - 1 - XH) * nyv));
  float um = ldg(u - 1);           // u at (i, j - 1)
  float v_mp = ldg(v - nyv + 1);   // v at (i - 1, j + 1)
  float m_im = ldg(m - ny), s_im = sg ? ldg(sg - ny) : 0.f;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = i0 + r;
    if (i > nx - 1 - HB) break;
#pragma unroll
    for (int q = 0; q + 1 < XW; ++q) x[q] = x[q + 1];
    x[XW - 1] = make_float2(ldg(u + (long)XH * ny), ldg(v + (long)XH * nyv));
    const float u_pm = ldg(u + ny - 1);
    FacePair f;
    f.c = x[XH];
    const float up = ldg(u + 1), vm = ldg(v - 1), vp = ldg(v + 1);
    f.am = make_float2(x[XH - 1].x, vm);
    f.ap = make_float2(x[XH + 1].x, vp);
    f.cm = make_float2(um, x[XH - 1].y);
    f.cp = make_float2(up, x[XH + 1].y);
    f.q2 = make_float2(v_mp, u_pm);
    f.q3 = make_float2(f.cm.y, f.cm.x);
    const float m_c = ldg(m);
    f.mc = f2(m_c);
    f.mo = make_float2(m_im, ldg(m - 1));
    f.sc = f.so = f2(0.f);
    if (sg) {
      const float s_c = ldg(sg);
      f.sc = f2(s_c);
      f.so = make_float2(s_im, ldg(sg - 1));
      s_im = s_c;
      sg += ny;
    }
    float2 adv;
    if constexpr (ADV == AJ_ADV_WENO5) {
      // u in lane x, v in lane y; both derivatives in x, then both in y
      const float2 cross = pair_cross(f);
      const float2 vx = make_float2(f.c.x, cross.y), vy = make_float2(cross.x, f.c.y);
      const float2 y[7] = {make_float2(ldg(u - 3), ldg(v - 3)), make_float2(ldg(u - 2), ldg(v - 2)),
                           make_float2(um, vm), f.c, make_float2(up, vp),
                           make_float2(ldg(u + 2), ldg(v + 2)), make_float2(ldg(u + 3), ldg(v + 3))};
      adv = fma2(vy, weno_d7_pair(y, a.idy, vy), mul2(vx, weno_d7_pair(x, a.idx, vx)));
    } else {
      adv = pair_upwind(a, f);
    }
    float2 chi;
    const float2 rhs = pair_rhs(a, f, adv, chi);
    const long ku = (long)i * ny + j, kv = (long)i * nyv + j;
    a.uout[ku] = finish_mac<0>(a, ku, rhs.x, chi.x, dt, k1u);
    a.vout[kv] = finish_mac<1>(a, kv, rhs.y, chi.y, dt, k1v);
    um = u_pm;
    v_mp = vp;
    m_im = m_c;
    u += ny;
    v += nyv;
    m += ny;
  }
}

template <int ADV>
static bool mac_rows_ok(const RkMac& a, bool hyper) {
  return !hyper && a.flow == AJ_FLOW_VON_KARMAN && a.slip && a.nx > 4 * MacRows<ADV>::HB &&
         a.ny > 4 * MacRows<ADV>::HB;
}
template <int ADV>
static void dispatch_rk_mac(const RkMac& a, bool hyper, cudaStream_t st) {
  if (mac_rows_ok<ADV>(a, hyper)) {
    using M = MacRows<ADV>;
    const unsigned rows = cdiv(a.nx - 2 * M::HB, 8 * M::R);
    launch_pdl(true, k_rk_mac_rows<ADV>, dim3(M::edge_blocks(a.nx, a.ny) + rows * cdiv(a.ny, 32)),
               dim3(32, 8), 0, st, a);
    return;
  }
  // 16 x 16 blocks: measured 4.5 us per step faster than 32 x 8 (and than
  // 64 x 4, 8 x 32) on the 2048x512 workload
  const dim3 blk(16, 16), grd(cdiv(a.ny + 1, 16), cdiv(a.nx + 1, 16));
  if (hyper) launch_pdl(true, k_rk_mac<true, ADV>, dim3(grd), dim3(blk), 0, st, a);
  else launch_pdl(true, k_rk_mac<false, ADV>, dim3(grd), dim3(blk), 0, st, a);
}

// ============================================================ driver
int launch_predictor(const AjStepParams& p, const Layout& L, void* ws, const float* u,
                     const float* v, const float* mask, const float* nsg, int double_count,
                     float* us, float* vs, cudaStream_t st, DtFrom dt) {
  StageDt sdt;
  sdt.known = dt != DtFrom::device;
  DevScalars* sc = at<DevScalars>(ws, 0);
  sdt.src = sdt.known ? reinterpret_cast<const float*>(&sc->zero) : &sc->dt;
  sdt.dt = (float)p.dt;
  sdt.dtc = (float)p.dt_correction;
  const int nx = p.nx, ny = p.ny;
  const bool rk2 = p.fast_mode != 0;
  const int nstage = rk2 ? 2 : 3;
  const bool hyper = p.nu_hyper_ratio > 0.0;
  float* A[2] = {at<float>(ws, L.sA_u), at<float>(ws, L.sA_v)};
  float* B[2] = {at<float>(ws, L.sB_u), at<float>(ws, L.sB_v)};
  float* K[2] = {at<float>(ws, L.k1_u), at<float>(ws, L.k1_v)};
  const double eta = p.grid_type == AJ_GRID_MAC ? (p.brinkman_eta > 1e-10 ? p.brinkman_eta : 1e-10)
                                                : p.brinkman_eta;
  if (p.grid_type == AJ_GRID_COLLOCATED) {
    if (p.advection != AJ_ADV_UPWIND && p.advection != AJ_ADV_WENO5) return AJ_ERR_PARAM;
    RkArgs a{};
    a.u0 = u;
    a.v0 = v;
    a.chi = at<float>(ws, L.chi);
    a.mask = mask;
    a.nsg = nsg;
    a.k1u = K[0];
    a.k1v = K[1];
    a.nx = nx;
    a.ny = ny;
    a.idx = (float)(1.0 / p.dx);
    a.idy = (float)(1.0 / p.dy);
    a.idx2 = (float)(1.0 / (p.dx * p.dx));
    a.idy2 = (float)(1.0 / (p.dy * p.dy));
    a.nu = (float)p.nu;
    a.inv_eta = (float)(1.0 / eta);
    a.U = (float)p.U_inf;
    a.nuh_fac = (float)(p.nu_hyper_ratio * p.dx * p.dy);
    a.dc = double_count;
    a.rk2 = rk2;
    a.flow = p.flow_type;
    a.slip = p.slip_walls;
    dim3 blk(32, 8), grd(cdiv(ny, 32), cdiv(nx, 8));
    const float* in_u = u;
    const float* in_v = v;
    for (int s = 1; s <= nstage; ++s) {
      a.stage = s;
      a.dt = sdt;
      if (s == 1 && dt == DtFrom::host) a.dt.write = sc;
      a.uin = in_u;
      a.vin = in_v;
      bool last = s == nstage;
      float** dst = (s % 2 == 1) ? A : B;
      a.uout = last ? us : dst[0];
      a.vout = last ? vs : dst[1];
      a.k1u_out = (rk2 && s == 1) ? K[0] : nullptr;
      a.k1v_out = (rk2 && s == 1) ? K[1] : nullptr;
      if (p.flow_type == AJ_FLOW_TAYLOR_GREEN) dispatch_rk_col<true>(a, hyper, p.advection, grd, blk, st);
      else dispatch_rk_col<false>(a, hyper, p.advection, grd, blk, st);
      in_u = a.uout;
      in_v = a.vout;
    }
  } else {
    if (p.advection != AJ_ADV_UPWIND && p.advection != AJ_ADV_WENO5) return AJ_ERR_PARAM;
    if (tile_predictor_ok(p, u, mask, nsg)) {
      if (dt != DtFrom::device) launch_set_dt(p, ws, st);
      const float* sb[4] = {A[0], A[1], B[0], B[1]};
      return launch_predictor_tile(p, ws, u, v, mask, nsg, us, vs, nullptr, sb, st);
    }
    RkMac a{};
    a.u0 = u;
    a.v0 = v;
    a.mask = mask;
    a.nsg = nsg;
    a.k1u = K[0];
    a.k1v = K[1];
    a.nx = nx;
    a.ny = ny;
    a.idx = (float)(1.0 / p.dx);
    a.idy = (float)(1.0 / p.dy);
    a.idx2 = (float)(1.0 / (p.dx * p.dx));
    a.idy2 = (float)(1.0 / (p.dy * p.dy));
    a.nu = (float)p.nu;
    a.inv_eta = (float)(1.0 / eta);
    a.U = (float)p.U_inf;
    a.nuh = (float)(p.nu * p.nu_hyper_ratio * p.dx * p.dy);
    a.rk2 = rk2;
    a.flow = p.flow_type;
    a.slip = p.slip_walls;
    const float* in_u = u;
    const float* in_v = v;
    for (int s = 1; s <= nstage; ++s) {
      a.stage = s;
      a.dt = sdt;
      if (s == 1 && dt == DtFrom::host) a.dt.write = sc;
      a.uin = in_u;
      a.vin = in_v;
      bool last = s == nstage;
      float** dst = (s % 2 == 1) ? A : B;
      a.uout = last ? us : dst[0];
      a.vout = last ? vs : dst[1];
      a.k1u_out = (rk2 && s == 1) ? K[0] : nullptr;
      a.k1v_out = (rk2 && s == 1) ? K[1] : nullptr;
      if (p.advection == AJ_ADV_WENO5) dispatch_rk_mac<AJ_ADV_WENO5>(a, hyper, st);
      else dispatch_rk_mac<AJ_ADV_UPWIND>(a, hyper, st);
      in_u = a.uout;
      in_v = a.vout;
    }
  }
  return cudaGetLastError() == cudaSuccess ? AJ_OK : AJ_ERR_CUDA;
}

}  // namespace aj
