// kernels_fp64.cu -- explicit kernels of the FP64 step (compiled with -fmad=false: only the fma
// written out are fused), in the reference's operand order, so with its bits (the exceptions: fp64.cuh).
//
// All are bound by the FP64 pipe (fp64.cuh), so each is written for few of its operations: a
// product that two cells or two interfaces share is formed once (at the face, or carried down the
// column), metrics divide by their stored reciprocals, halves are taken in the exponent, and sums do
// not start with 0 + x.
#include "fp64.cuh"
#include "diffusion.cuh"

#include <algorithm>

namespace lg {

template <> __device__ __forceinline__ F64 dsqrt<F64>(F64 x) { return root(x); }

namespace {

struct CarriedF {
  const F64 *nl_u, *nl_v, *nl_w, *l_u, *l_v, *l_w, *old_u, *old_v, *pgcw, *vsg_x, *vsg_y, *vsg_z, *pvt_x, *pvt_y, *pvt_z,
      *mdt_x, *mdt_y, *mdt_z;
};
// the four sides of a dual point: v, u, v, u points (mo_vorticities.F90:423-538); not in: a non-periodic
// boundary point, where the vorticity is 0
struct RotSides { long long v0, u1, v2, u3; bool in; };
__device__ __forceinline__ RotSides rot_sides(const Dims& D, int ji, int jk, int jl) {
  const bool edge = ji == 1 || jk == 1 || ji == D.ny + 1 || jk == D.nx + 1;
  RotSides s;
  s.in = !edge || D.periodic;
  s.v0 = IX(D, ji, (jk == D.nx + 1) ? 1 : jk, jl);
  s.u1 = IX(D, (ji == 1) ? D.ny : ji - 1, jk, jl);
  s.v2 = IX(D, ji, (jk == 1) ? D.nx : jk - 1, jl);
  s.u3 = IX(D, (ji == D.ny + 1) ? 1 : ji, jk, jl);
  return s;
}
struct PGradF { F64 *nl_u, *nl_v, *nl_w, *l_u, *l_v, *l_w, *old_u, *old_v, *pgcw; };

// marching threads: a chunk of the column's levels each (blockIdx.z), of eight levels (the layer above a
// chunk is formed twice) and of fewer, down to two, where that leaves an SM under 1536 threads
dim3 march_grid(const Dims& D) {
  dim3 g((unsigned)((D.ny + 31) / 32), (unsigned)((D.nx + 3) / 4), 1);
  const long long cells = 128LL * g.x * g.y * D.nl;
  const int len = (int)std::min(8LL, std::max(2LL, cells / (152LL * 1536)));
  g.z = (unsigned)((D.nl + len - 1) / len);
  return g;
}
__device__ __forceinline__ int march_first(const Dims& D, unsigned z) {
  const int len = (D.nl + (int)gridDim.z - 1) / (int)gridDim.z;
  return min((int)z * len, D.nl) + 1;
}
dim3 cell_grid(int rows, int cols, int levs) {
  return dim3((unsigned)((rows + 31) / 32), (unsigned)levs, (unsigned)((cols + 7) / 8));
}
const dim3 kMarchBlock(32, 4), kCellBlock(32, 8);

__global__ void k64_recip(Dims D, Grid<F64> G, F64* rdx, F64* rdy, F64* rdz) {
  LG_IDX3;
  const long long q = IX(D, ji, jk, jl);
  if (ji <= D.ny && jk <= D.nx + 1) rdx[q] = 1.0 / G.dx[q];
  if (ji <= D.ny + 1 && jk <= D.nx) rdy[q] = 1.0 / G.dy[q];
  if (ji <= D.ny && jk <= D.nx) rdz[q] = 1.0 / G.dz[q];
}

// ---- gradient of a scalar, mo_gradient_operators.F90:17-130 -----------------------------------------
// The vertical gradient gz at w levels 2..nl and, in the terrain-following layers, each column's
// two products of the remap to the horizontal faces (mo_averaging.F90:56-136), W5(l)*gz(l) and
// W6(l)*gz(l+1), which the four faces of the column share.  gz_sfc: gz at level nl+1 (never written
// by grad_vert) as the array holds it.
__global__ void __launch_bounds__(128) k64_grad_vert(Dims D, Grid<F64> G, const F64* rdz, const F64* s, F64* gz,
                                                     F64* w5, F64* w6) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1, jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const int l0 = march_first(D, blockIdx.z), l1 = march_first(D, blockIdx.z + 1) - 1;
  if (l0 > l1) return;
  long long q = IX(D, ji, jk, l0);
  F64 cur = s[q];
  F64 g = (l0 >= 2) ? div_rn(s[q - D.plane] - cur, G.dz[q], rdz[q]) : 0.0;
  for (int jl = l0; jl <= l1; ++jl, q += D.plane) {
    F64 gn = 0.0;
    if (jl < D.nl) {
      const F64 nxt = s[q + D.plane];
      gn = div_rn(cur - nxt, G.dz[q + D.plane], rdz[q + D.plane]);
      cur = nxt;
    }
    if (jl >= 2) gz[q] = g;
    if (jl > D.nf) {
      w5[q] = G.ipw[4][q] * g;
      if (jl < D.nl) w6[q] = G.ipw[5][q] * gn;
      else if (D.freeslip) w6[q] = G.ipw[5][q] * gz[q + D.plane];
    }
    g = gn;
  }
}

// the horizontal gradient at u and v points; false where the reference leaves the point untouched
__device__ __forceinline__ bool grad_x64(const Dims& D, const Grid<F64>& G, const F64* rdx, const F64* s,
                                         const F64* w5, const F64* w6, int ji, int jk, int jl, F64* r) {
  const bool inner = jk >= 2 && jk <= D.nx;
  if (!inner && !D.periodic) return false;
  const long long a = IX(D, ji, inner ? jk - 1 : D.nx, jl), b = IX(D, ji, inner ? jk : 1, jl);
  F64 g = div_rn(s[b] - s[a], G.dx[b], rdx[b]);
  if (jl > D.nf) {
    F64 m = w5[a] + w5[b];
    if (jl < D.nl || D.freeslip) m = m + w6[a] + w6[b];
    g = g - G.slope_x[IX(D, ji, jk, jl)] * half(m);
  }
  *r = g;
  return true;
}
__device__ __forceinline__ bool grad_y64(const Dims& D, const Grid<F64>& G, const F64* rdy, const F64* s,
                                         const F64* w5, const F64* w6, int ji, int jk, int jl, F64* r) {
  const bool inner = ji >= 2 && ji <= D.ny;
  if (!inner && !D.periodic) return false;
  const long long a = IX(D, inner ? ji - 1 : D.ny, jk, jl), b = IX(D, inner ? ji : 1, jk, jl);
  F64 g = div_rn(s[a] - s[b], G.dy[b], rdy[b]);
  if (jl > D.nf) {
    F64 m = w5[a] + w5[b];
    if (jl < D.nl || D.freeslip) m = m + w6[a] + w6[b];
    g = g - G.slope_y[IX(D, ji, jk, jl)] * half(m);
  }
  *r = g;
  return true;
}
__global__ void k64_grad_hor(Dims D, Grid<F64> G, Recip R, const F64* s, const F64* w5, const F64* w6,
                             F64* rx, F64* ry) {
  LG_IDX3;
  F64 r;
  if (ji <= D.ny && jk <= D.nx + 1 && grad_x64(D, G, R.dx, s, w5, w6, ji, jk, jl, &r)) rx[IX(D, ji, jk, jl)] = r;
  if (ji <= D.ny + 1 && jk <= D.nx && grad_y64(D, G, R.dy, s, w5, w6, ji, jk, jl, &r)) ry[IX(D, ji, jk, jl)] = r;
}

// ---- divergence of a horizontal vector, mo_divergence_operators.F90:16-68 ---------------------------
// A face hands its two cells the flux f*area and, in the terrain-following layers, the slope term
// 0.5*f*slope of the contravariant vertical velocity (mo_averaging.F90:16-54).  The faces of a
// non-periodic boundary, which the reference leaves untouched at 0, are written as 0: the arrays serve
// several fields in turn.
__device__ __forceinline__ void face_x(const Dims& D, const Grid<F64>& G, F64 f, const Faces& F, int jl, long long q) {
  F.px[q] = f * G.area_x[q];
  if (jl > D.nf) F.hx[q] = half(f) * G.slope_x[q];
}
__device__ __forceinline__ void face_y(const Dims& D, const Grid<F64>& G, F64 f, const Faces& F, int jl, long long q) {
  F.py[q] = f * G.area_y[q];
  if (jl > D.nf) F.hy[q] = half(f) * G.slope_y[q];
}

// the vertical part of a column's divergence, walked down: the reference's sum at an interface runs
// over the four slope terms of the layer above and then of the layer below, so the sum over a layer's
// own terms serves as the start of the interface below it
struct SlopeTerms { F64 a, b, c, d; };
__device__ __forceinline__ SlopeTerms slope_terms(const Dims& D, const Grid<F64>& G, const F64* hx, const F64* hy,
                                                  long long q) {
  return SlopeTerms{hx[q + D.P] * G.ipw[0][q], hy[q] * G.ipw[1][q], hx[q] * G.ipw[2][q], hy[q + 1] * G.ipw[3][q]};
}
__device__ __forceinline__ F64 own_sum(const SlopeTerms& t) { return -t.a - t.b - t.c - t.d; }
__device__ __forceinline__ F64 join(F64 above, const SlopeTerms& t) { return above - t.a - t.b - t.c - t.d; }

// the contravariant correction at interface l = nf+1..nl of the layers above and below it
struct Contra {
  F64 sum;  // own_sum of the current layer
  // at the chunk's first level l0 (> nf): the correction at its upper interface
  __device__ __forceinline__ F64 start(const Dims& D, const Grid<F64>& G, const F64* hx, const F64* hy, long long q,
                                          int l0) {
    const SlopeTerms t = slope_terms(D, G, hx, hy, q);
    sum = own_sum(t);
    if (l0 == D.nf + 1) return sum;
    return join(own_sum(slope_terms(D, G, hx, hy, q - D.plane)), t);
  }
  // the correction at the lower interface of layer jl (jl == nf, or nf < jl < nl); q: layer jl
  __device__ __forceinline__ F64 below(const Dims& D, const Grid<F64>& G, const F64* hx, const F64* hy, long long q,
                                          int jl) {
    const SlopeTerms t = slope_terms(D, G, hx, hy, q + D.plane);
    const F64 r = (jl == D.nf) ? own_sum(t) : join(sum, t);
    sum = own_sum(t);
    return r;
  }
};
struct ColumnDiv {
  Contra c;
  F64 up;  // correction times area at the upper interface
  __device__ __forceinline__ void start(const Dims& D, const Grid<F64>& G, const Faces& F, long long q, int l0) {
    up = 0.0;
    c.sum = 0.0;
    if (l0 > D.nf) up = c.start(D, G, F.hx, F.hy, q, l0) * G.area_z[q];
  }
  // divergence of layer jl
  __device__ __forceinline__ F64 step(const Dims& D, const Grid<F64>& G, const Faces& F, F64 V, F64 rV, long long q,
                                         int jl) {
    F64 s = F.px[q + D.P] + F.py[q] - F.px[q] - F.py[q + 1];
    F64 lo = 0.0;
    if (jl == D.nf || (jl > D.nf && jl < D.nl)) lo = c.below(D, G, F.hx, F.hy, q, jl) * G.area_z[q + D.plane];
    if (jl == D.nf) s = s - lo;
    else if (jl == D.nl) s = s + up;
    else if (jl > D.nf) s = s + (up - lo);
    up = lo;
    return div_rn(s, V, rV);
  }
};

// faces of the gradient of a scalar, and their divergence (theta_v_adv_3rd_order)
__global__ void k64_grad_faces(Dims D, Grid<F64> G, Recip R, const F64* s, const F64* w5, const F64* w6, Faces F) {
  LG_IDX3;
  F64 r;
  if (ji <= D.ny && jk <= D.nx + 1)
    face_x(D, G, grad_x64(D, G, R.dx, s, w5, w6, ji, jk, jl, &r) ? r : 0.0, F, jl, IX(D, ji, jk, jl));
  if (ji <= D.ny + 1 && jk <= D.nx)
    face_y(D, G, grad_y64(D, G, R.dy, s, w5, w6, ji, jk, jl, &r) ? r : 0.0, F, jl, IX(D, ji, jk, jl));
}
__global__ void __launch_bounds__(128) k64_div(Dims D, Grid<F64> G, const F64* rvol, Faces F, F64* out) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1, jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const int l0 = march_first(D, blockIdx.z), l1 = march_first(D, blockIdx.z + 1) - 1;
  if (l0 > l1) return;
  long long q = IX(D, ji, jk, l0);
  ColumnDiv c;
  c.start(D, G, F, q, l0);
  for (int jl = l0; jl <= l1; ++jl, q += D.plane) out[q] = c.step(D, G, F, G.volume[q], rvol[q], q, jl);
}

// theta_v_adv_3rd_order edge values, mo_multiplications.F90:134-202
__global__ void k64_theta_edges(Dims D, const F64* th, const F64* Dv, const F64* u, const F64* v, F64* tvu,
                                F64* tvv) {
  LG_IDX3;
  const F64 c = D.theta_edge_c;
  if (ji <= D.ny && jk <= D.nx + 1) {
    const bool inner = jk >= 2 && jk <= D.nx;
    if (inner || D.periodic) {
      const long long a = IX(D, ji, inner ? jk - 1 : D.nx, jl), b = IX(D, ji, inner ? jk : 1, jl);
      tvu[IX(D, ji, jk, jl)] = half(th[a] + th[b]) - c * Dv[upwind(u[b]) ? a : b];
    }
  }
  if (ji <= D.ny + 1 && jk <= D.nx) {
    const bool inner = ji >= 2 && ji <= D.ny;
    if (inner || D.periodic) {
      const long long a = IX(D, inner ? ji : 1, jk, jl), b = IX(D, inner ? ji - 1 : D.ny, jk, jl);
      tvv[IX(D, ji, jk, jl)] = half(th[a] + th[b]) - c * Dv[upwind(v[a]) ? a : b];
    }
  }
}

// ---- scalar tendencies, mo_scalar_tend_expl.F90:106-177 ---------------------------------------------
// faces of the gas mass flux and of the theta_v flux (theta_order 3: edge values tvu, tvv; 2: the
// mean of the two cells)
__global__ void k64_gas_faces(Dims D, Grid<F64> G, StateT<F64> Ss, const F64* u_new, const F64* v_new,
                              const F64* tvu, const F64* tvv, Faces M, Faces T) {
  LG_IDX3;
  const F64* rg = Ss.rho + (long long)(D.g - 1) * D.fstride;
  auto th = [&](long long p) { return G.theta_v_bg[p] + Ss.tp[p]; };
  if (ji <= D.ny && jk <= D.nx + 1) {
    const bool inner = jk >= 2 && jk <= D.nx;
    const long long q = IX(D, ji, jk, jl);
    F64 f = 0.0, g = 0.0;  // (a non-periodic boundary's faces carry no flux)
    if (inner || D.periodic) {
      const long long a = IX(D, ji, inner ? jk - 1 : D.nx, jl), b = IX(D, ji, inner ? jk : 1, jl);
      f = half(rg[a] + rg[b]) * u_new[b];
      g = D.theta_order == 2 ? half(th(a) + th(b)) * f : tvu[q] * f;
    }
    face_x(D, G, f, M, jl, q);
    face_x(D, G, g, T, jl, q);
  }
  if (ji <= D.ny + 1 && jk <= D.nx) {
    const bool inner = ji >= 2 && ji <= D.ny;
    const long long q = IX(D, ji, jk, jl);
    F64 f = 0.0, g = 0.0;
    if (inner || D.periodic) {
      const long long a = IX(D, inner ? ji - 1 : D.ny, jk, jl), b = IX(D, inner ? ji : 1, jk, jl);
      f = half(rg[a] + rg[b]) * v_new[b];
      g = D.theta_order == 2 ? half(th(a) + th(b)) * f : tvv[q] * f;
    }
    face_y(D, G, f, M, jl, q);
    face_y(D, G, g, T, jl, q);
  }
}

// their divergences and the diabatic term: the gas and rho*theta_v tendencies (k_gas_theta<F64>
// formed every face two to five times and c_p of every condensate anew: 2084 us a launch at
// 192x192x80)
__global__ void __launch_bounds__(128) k64_gas_theta(Dims D, Grid<F64> G, StateT<F64> Ss, const F64* rvol, Faces M,
                                                     Faces T, const F64* cpi, const F64* cpw, const F64* hd,
                                                     const F64* rad, const F64* csh, F64* t_rho, F64* t_rt,
                                                     const F64* mdt, const F64* tdh, const F64* ptr,
                                                     const F64* pth) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1, jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const int l0 = march_first(D, blockIdx.z), l1 = march_first(D, blockIdx.z + 1) - 1;
  if (l0 > l1) return;
  const long long goff = (long long)(D.g - 1) * D.fstride;
  long long q = IX(D, ji, jk, l0);
  ColumnDiv cm, ct;
  cm.start(D, G, M, q, l0);
  ct.start(D, G, T, q, l0);
  for (int jl = l0; jl <= l1; ++jl, q += D.plane) {
    const F64 V = G.volume[q], rV = rvol[q];
    const F64 div_m = cm.step(D, G, M, V, rV, q, jl), div_t = ct.step(D, G, T, V, rV, q, jl);
    F64 heat = hd[q] + rad[q];
    if (pth) heat = heat + pth[q];
    heat = heat + csh[q];
    if (tdh) heat = heat + tdh[q];
    F64 r = -div_t;
    if (nonzero(heat)) {
      const F64 rg = Ss.rho[q + goff];
      F64 cv;  // c_v_mass_weighted_air, mo_derived.F90:157-187 (odd constituents are ice)
      if (D.lmoist) {
        const F64 ci = cpi[q], cw = cpw[q];
        cv = Ss.rho[q] * ci;
        for (int jc = 2; jc <= D.nc; ++jc) cv = cv + Ss.rho[q + (long long)(jc - 1) * D.fstride] * ((jc & 1) ? ci : cw);
        const F64 rv = Ss.rho[q + goff + D.fstride];
        cv = cv + (rg - rv) * kC_D_V;
        cv = cv + rv * kC_V_V;
      } else {
        cv = rg * kC_D_V;
      }
      r = r + kC_D_V * rg / cv * heat / (kC_D_P * (G.exner_bg[q] + Ss.ep[q]));
    }
    F64 tg = -div_m;
    if (mdt) tg = tg + mdt[q + goff];
    if (ptr) {
      const F64 ptg = ptr[q + goff];
      tg = tg + ptg;
      r = r + (mdt ? ptg + mdt[q + goff] : ptg) * (G.theta_v_bg[q] + Ss.tp[q]);
    } else if (mdt) {
      r = r + mdt[q + goff] * (G.theta_v_bg[q] + Ss.tp[q]);
    }
    t_rho[q + goff] = tg;
    t_rt[q] = r;
  }
}

// the contravariant correction of the new wind at the interfaces nf+1..nl, for the tracers
__global__ void __launch_bounds__(128) k64_contra(Dims D, Grid<F64> G, const F64* hx, const F64* hy, F64* cw) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1, jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const int l0 = max(march_first(D, blockIdx.z), D.nf + 1), l1 = march_first(D, blockIdx.z + 1) - 1;
  if (l0 > l1) return;
  long long q = IX(D, ji, jk, l0);
  Contra c;
  cw[q] = c.start(D, G, hx, hy, q, l0);
  for (int jl = l0 + 1; jl <= l1; ++jl) {
    cw[q + D.plane] = c.below(D, G, hx, hy, q, jl - 1);
    q += D.plane;
  }
}
__global__ void k64_wind_slopes(Dims D, Grid<F64> G, const F64* u, const F64* v, F64* hx, F64* hy) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int jk = blockIdx.z * blockDim.y + threadIdx.y + 1;
  const int jl = blockIdx.y + D.nf + 1;
  const long long q = IX(D, ji, jk, jl);
  if (ji <= D.ny && jk <= D.nx + 1) hx[q] = half(u[q]) * G.slope_x[q];
  if (ji <= D.ny + 1 && jk <= D.nx) hy[q] = half(v[q]) * G.slope_y[q];
}

// scalar_tend_expl for the tracers, mo_scalar_tend_expl.F90:24-104, with
// scalar_times_vector_h_upstream (mo_multiplications.F90:206-287) and div_h_tracers
// (mo_divergence_operators.F90:70-147): velocity, area and upwind cell of each of a cell's six faces
// are found once for all tracers.  At the first substep the old tendency has weight 0 and is not read.
__global__ void __launch_bounds__(256) k64_tracers(Dims D, Grid<F64> G, const F64* rvol, StateT<F64> Ss,
                                                   const F64* u_new, const F64* v_new, const F64* cw, F64* t_rho,
                                                   int rk_step, const F64* mdt, const F64* ptr) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl);
  struct F { F64 v, a; long long i; };
  auto fx = [&](int kf) {
    const bool inner = kf >= 2 && kf <= D.nx;
    F f{0.0, 0.0, q};
    if (!inner && !D.periodic) return f;
    f.v = u_new[IX(D, ji, inner ? kf : 1, jl)];
    f.a = G.area_x[IX(D, ji, kf, jl)];
    f.i = IX(D, ji, upwind(f.v) ? (inner ? kf - 1 : D.nx) : (inner ? kf : 1), jl);
    return f;
  };
  auto fy = [&](int i_f) {
    const bool inner = i_f >= 2 && i_f <= D.ny;
    F f{0.0, 0.0, q};
    if (!inner && !D.periodic) return f;
    f.v = v_new[IX(D, inner ? i_f : 1, jk, jl)];
    f.a = G.area_y[IX(D, i_f, jk, jl)];
    f.i = IX(D, upwind(f.v) ? (inner ? i_f : 1) : (inner ? i_f - 1 : D.ny), jk, jl);
    return f;
  };
  const F e = fx(jk + 1), n = fy(ji), w = fx(jk), s = fy(ji + 1);
  const bool has_up = jl > D.nf, has_lo = jl == D.nf || (jl > D.nf && jl < D.nl);
  F64 cu = 0.0, cl = 0.0, au = 0.0, al = 0.0;
  long long iu = q, il = q;
  if (has_up) {
    cu = cw[q];
    au = G.area_z[q];
    if (!positive(cu)) iu = q - D.plane;
  }
  if (has_lo) {
    cl = cw[q + D.plane];
    al = G.area_z[q + D.plane];
    if (positive(cl)) il = q + D.plane;
  }
  const F64 V = G.volume[q], rV = rvol[q];
  for (int jc = 1; jc <= D.ncons; ++jc) {
    if (jc == D.g) continue;
    const F64* r = Ss.rho + (long long)(jc - 1) * D.fstride;
    F64 c = r[e.i] * e.v * e.a + r[n.i] * n.v * n.a - r[w.i] * w.v * w.a - r[s.i] * s.v * s.a;
    if (has_up && has_lo && jl != D.nf) c = c + (r[iu] * cu * au - r[il] * cl * al);
    else if (has_lo) c = c - r[il] * cl * al;
    else if (has_up) c = c + r[iu] * cu * au;
    F64 f = -div_rn(c, V, rV);
    if (mdt) f = f + mdt[q + (long long)(jc - 1) * D.fstride];
    if (ptr) f = f + ptr[q + (long long)((jc < D.g ? jc : D.g) - 1) * D.fstride];
    F64* t = t_rho + (long long)(jc - 1) * D.fstride;
    t[q] = (rk_step == 1) ? f : half(t[q]) + half(f);
  }
}

// what the pressure gradient reads of a cell: theta_v, c_d_p*rho_g/sum(rho) and rho_g/sum(rho) - 1
__global__ void k64_pgrad_cells(Dims D, Grid<F64> G, StateT<F64> S, F64* th, F64* decel, F64* cond) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl);
  th[q] = G.theta_v_bg[q] + S.tp[q];
  F64 sum = S.rho[q];
  for (int jc = 1; jc <= D.nc; ++jc) sum = sum + S.rho[q + (long long)jc * D.fstride];
  const F64 rg = S.rho[q + (long long)(D.g - 1) * D.fstride], y = rcp_near(sum);
  decel[q] = div_rn(kC_D_P * rg, sum, y);
  cond[q] = div_rn(rg, sum, y) - 1.0;
}
// manage_p_grad, mo_p_grad.F90:20-104, after the gradients of exner_pert (gx,gy,gz) and, for
// theta_adv_order 3, the edge values of theta (tvu,tvv) and theta' (tpu,tpv) are known; also
// calc_p_grad_condensates_v, mo_p_grad.F90:106-120 (identical at both substeps because it always
// reads state_old).  (With theta and both quotients formed at each of a cell's six faces: 902 us
// at 192x192x80.)
__global__ void k64_pgrad(Dims D, Grid<F64> G, StateT<F64> S, const F64* gx, const F64* gy, const F64* gz,
                          const F64* th, const F64* decel, const F64* cond, const F64* tvu, const F64* tvv,
                          const F64* tpu, const F64* tpv, PGradF P, int lfirst) {
  LG_IDX3;
  auto negsum = [&](F64 nl, F64 l) { return D.luse_bg ? -nl - l : -nl; };
  // one face between cells a and b: point q, evaluated at qr
  auto face = [&](long long q, long long qr, long long a, long long b, const F64* g, const F64* tv, const F64* tp,
                  const F64* eg, F64* nl, F64* l, F64* old) {
    if (!lfirst) old[q] = negsum(nl[q], D.luse_bg ? l[q] : 0.0);
    const F64 de = half(decel[a] + decel[b]);
    const F64 nlv = de * ((D.theta_order == 2 ? half(th[a] + th[b]) : tv[qr]) * g[qr]);
    F64 lv = 0.0;
    nl[q] = nlv;
    if (D.luse_bg) {
      lv = de * ((D.theta_order == 2 ? half(S.tp[a] + S.tp[b]) : tp[qr]) * eg[qr]);
      l[q] = lv;
    }
    if (lfirst) old[q] = negsum(nlv, lv);
  };
  // u points.  Periodic jk = nx+1 ends as a copy of jk = 1 (scalar_times_vector_h2
  // copies it last), so it is evaluated from column 1.  Non-periodic boundary edges stay
  // at their initial zero in every array of the reference (no operator writes them and
  // whole-array products multiply zeros), so only p_grad_acc_old is refreshed there.
  if (jl <= D.nl && ji <= D.ny && jk <= D.nx + 1) {
    const long long q = IX(D, ji, jk, jl);
    const bool inner = jk >= 2 && jk <= D.nx;
    if (inner || D.periodic)
      face(q, IX(D, ji, inner ? jk : 1, jl), IX(D, ji, inner ? jk - 1 : D.nx, jl), IX(D, ji, inner ? jk : 1, jl), gx, tvu, tpu,
           G.egu, P.nl_u, P.l_u, P.old_u);
    else
      P.old_u[q] = negsum(P.nl_u[q], P.l_u[q]);
  }
  // v points (periodic ji = ny+1 from row 1)
  if (jl <= D.nl && ji <= D.ny + 1 && jk <= D.nx) {
    const long long q = IX(D, ji, jk, jl);
    const bool inner = ji >= 2 && ji <= D.ny;
    if (inner || D.periodic)
      face(q, IX(D, inner ? ji : 1, jk, jl), IX(D, inner ? ji - 1 : 1, jk, jl), IX(D, inner ? ji : D.ny, jk, jl), gy, tvv, tpv,
           G.egv, P.nl_v, P.l_v, P.old_v);
    else
      P.old_v[q] = negsum(P.nl_v[q], P.l_v[q]);
  }
  // w points, levels 2..nl
  if (jl >= 2 && jl <= D.nl && ji <= D.ny && jk <= D.nx) {
    const long long q = IX(D, ji, jk, jl), qa = q - D.plane;
    const F64 de = half(decel[qa] + decel[q]);
    P.nl_w[q] = de * (half(th[qa] + th[q]) * gz[q]);
    if (D.luse_bg) P.l_w[q] = de * (half(S.tp[qa] + S.tp[q]) * G.egw[q]);
    P.pgcw[q] = half(cond[qa] + cond[q]) * G.gm[q];  // p_grad_condensates_w
  }
}

// ---- potential vorticity and its flux, mo_vorticities.F90, mo_vorticity_flux.F90 -------------------
// grid-only factors (RotGrid)
__global__ void k64_rot_grid(Dims D, Grid<F64> G, F64* m0, F64* m1, F64* m2, F64* m3) {
  LG_IDX3;
  if (ji > D.ny + 1 || jk > D.nx + 1 || jl <= D.nf) return;
  const long long q = IX(D, ji, jk, jl);
  const RotSides n = rot_sides(D, ji, jk, jl);
  if (!n.in) return;
  const F64 up = F64(kR_E) + G.z_area_dual_z[q];
  m0[q] = up / (F64(kR_E) + G.z_v[n.v0]) * G.dy[n.v0];
  m1[q] = -(up / (F64(kR_E) + G.z_u[n.u1])) * G.dx[n.u1];
  m2[q] = -(up / (F64(kR_E) + G.z_v[n.v2])) * G.dy[n.v2];
  m3[q] = up / (F64(kR_E) + G.z_u[n.u3]) * G.dx[n.u3];
}
// rel_vort_z_local, mo_vorticities.F90:423-538, over the dual area: the wind of each of the four sides
// extrapolated to the dual point's height
__device__ __forceinline__ F64 zeta_z64(const Dims& D, const Grid<F64>& G, const RotGrid& X, const F64* u, const F64* v, int ji,
                                        int jk, int jl) {
  const long long q = IX(D, ji, jk, jl), pl = D.plane;
  const RotSides n = rot_sides(D, ji, jk, jl);
  F64 r = 0.0;
  if (!n.in) return r;
  if (jl <= D.nf) {
    r = G.dy[n.v0] * v[n.v0] - G.dx[n.u1] * u[n.u1] - G.dy[n.v2] * v[n.v2] + G.dx[n.u3] * u[n.u3];
  } else {
    const F64 zd = G.z_area_dual_z[q];
    auto side = [&](const F64* x, const F64* z, const F64* m, long long i) {
      const F64 z0 = z[i], x0 = x[i], dz = zd - z0;
      const bool above = (positive(dz) || jl == D.nl) && jl != 1;
      const long long o = above ? i - pl : i + pl;
      return m[q] * (x0 + dz * ((x0 - x[o]) / (z0 - z[o])));
    };
    r = side(v, G.z_v, X.m0, n.v0) + side(u, G.z_u, X.m1, n.u1) + side(v, G.z_v, X.m2, n.v2) + side(u, G.z_u, X.m3, n.u3);
  }
  return r / G.area_dual_z[q];
}
__global__ void k64_zeta_z(Dims D, Grid<F64> G, RotGrid X, StateT<F64> S, F64* zz) {
  LG_IDX3;
  if (ji <= D.ny + 1 && jk <= D.nx + 1) zz[IX(D, ji, jk, jl)] = zeta_z64(D, G, X, S.u, S.v, ji, jk, jl);
}
// eta_z at (ny+1, nx+1, nl)
__global__ void k64_eta_z(Dims D, Grid<F64> G, RotGrid X, StateT<F64> S, F64* ez) {
  LG_IDX3;
  if (ji > D.ny + 1 || jk > D.nx + 1) return;
  const int i = (D.periodic && ji == D.ny + 1) ? 1 : ji, k = (D.periodic && jk == D.nx + 1) ? 1 : jk;
  F64 e = 0.0;
  if (!D.llinear) e = zeta_z64(D, G, X, S.u, S.v, i, k, jl);
  if (D.lcorio) e = e + G.fvec_z[IX(D, i, k, 1)];
  if (D.periodic || (i >= 2 && i <= D.ny && k >= 2 && k <= D.nx)) {
    const F64* rg = S.rho + (long long)(D.g - 1) * D.fstride;
    const int km = (k == 1) ? D.nx : k - 1, im = (i == 1) ? D.ny : i - 1;
    e = e / quarter_of(rg[IX(D, i, km, jl)] + rg[IX(D, i, k, jl)] + rg[IX(D, im, k, jl)] + rg[IX(D, im, km, jl)]);
  }
  ez[IX(D, ji, jk, jl)] = e;
}
// dx times the covariant wind (horizontal_covariant_x/y, mo_averaging.F90:138-176) at u and v points,
// which the two interfaces of the layer share
__global__ void k64_covariant(Dims D, Grid<F64> G, StateT<F64> S, F64* cx, F64* cy) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl);
  const F64* w = S.w;
  const bool lower = jl < D.nl || D.freeslip;
  auto remap = [&](long long a, long long b) {
    F64 m = G.ipw[4][a] * w[a] + G.ipw[4][b] * w[b];
    if (lower) m = m + G.ipw[5][a] * w[a + D.plane] + G.ipw[5][b] * w[b + D.plane];
    return half(m);
  };
  F64 x = S.u[q], y = S.v[q];
  if (jl > D.nf) {
    if (jk >= 2 || D.periodic) x = x + G.slope_x[q] * remap(jk >= 2 ? q - D.P : IX(D, ji, D.nx, jl), q);
    if (ji >= 2 || D.periodic) y = y + G.slope_y[q] * remap(ji >= 2 ? q - 1 : IX(D, D.ny, jk, jl), q);
  }
  cx[q] = G.dx[q] * x;
  cy[q] = G.dy[q] * y;
}
// eta_x (ny+1, nx, nl+1) and eta_y (ny, nx+1, nl+1); level 1 takes the vorticity of level 2, and the
// surface level the general form
__global__ void k64_eta_xy(Dims D, Grid<F64> G, StateT<F64> S, const F64* cx, const F64* cy, F64* ex, F64* ey) {
  LG_IDX3;
  const int lev = max(jl, 2);
  const F64* rg = S.rho + (long long)(D.g - 1) * D.fstride;
  if (ji <= D.ny + 1 && jk <= D.nx) {
    const int i = (D.periodic && ji == D.ny + 1) ? 1 : ji;
    const bool inner = i >= 2 && i <= D.ny;
    F64 e = 0.0;
    if (jl == D.NL) {
      e = eta_x_at<F64>(D, G, S, i, jk, jl);
    } else {
      const long long b = IX(D, inner ? i : 1, jk, lev), a = IX(D, inner ? i - 1 : D.ny, jk, lev), q = IX(D, i, jk, lev);
      if (!D.llinear && (inner || D.periodic))
        e = (G.dz[a] * S.w[a] - cy[b - D.plane] - G.dz[b] * S.w[b] + cy[b]) / G.area_dual_x[q];
      if (D.lcorio) e = e + G.fvec_x[IX(D, i, jk, 1)];
      if (inner || D.periodic) e = e / rho_avg_h<F64>(D, G, rg, inner ? i - 1 : D.ny, jk, inner ? i : 1, jk, jl);
    }
    ex[IX(D, ji, jk, jl)] = e;
  }
  if (ji <= D.ny && jk <= D.nx + 1) {
    const int k = (D.periodic && jk == D.nx + 1) ? 1 : jk;
    const bool inner = k >= 2 && k <= D.nx;
    F64 e = 0.0;
    if (jl == D.NL) {
      e = eta_y_at<F64>(D, G, S, ji, k, jl);
    } else {
      const long long b = IX(D, ji, inner ? k : 1, lev), a = IX(D, ji, inner ? k - 1 : D.nx, lev), q = IX(D, ji, k, lev);
      if (!D.llinear && (inner || D.periodic))
        e = (-(G.dz[b] * S.w[b]) - cx[b] + G.dz[a] * S.w[a] + cx[b - D.plane]) / G.area_dual_y[q];
      if (D.lcorio) e = e + G.fvec_y[IX(D, ji, k, 1)];
      if (inner || D.periodic) e = e / rho_avg_h<F64>(D, G, rg, ji, inner ? k - 1 : D.nx, ji, inner ? k : 1, jl);
    }
    ey[IX(D, ji, jk, jl)] = e;
  }
}
// mass flux densities, mo_vector_tend_expl.F90:64-80: at u and v points, and of the vertical one its
// two products with half the inner-product weights of a layer, which the layer's four faces share:
// q5 = 0.5*W5*(rho*w)(l), q6 = 0.5*W6*(rho*w)(l+1) (free-slip value at the surface, 0 at the top)
__global__ void k64_mass_flux(Dims D, Grid<F64> G, StateT<F64> S, F64* uph, F64* vph, F64* q5, F64* q6) {
  LG_IDX3;
  const F64* rg = S.rho + (long long)(D.g - 1) * D.fstride;
  const long long q = IX(D, ji, jk, jl);
  F64 f;  // (0 at a non-periodic boundary, which the reference leaves untouched: the arrays serve others in turn)
  if (ji <= D.ny && jk <= D.nx + 1) uph[q] = stv_h_x<F64>(D, rg, S.u, ji, jk, jl, &f) ? f : F64(0.0);
  if (ji <= D.ny + 1 && jk <= D.nx) vph[q] = stv_h_y<F64>(D, rg, S.v, ji, jk, jl, &f) ? f : F64(0.0);
  if (ji > D.ny || jk > D.nx) return;
  const long long b = q + D.plane;
  F64 up = 0.0, lo = 0.0;
  if (jl >= 2) up = half(rg[q - D.plane] + rg[q]) * S.w[q];
  if (jl < D.nl) {
    lo = half(rg[q] + rg[b]) * S.w[b];
  } else if (D.freeslip) {
    const long long a = q - D.plane;
    lo = (rg[q] + (rg[a] - rg[q]) / (G.z_scalar[a] - G.z_scalar[q]) * (G.z_w[b] - G.z_scalar[q])) * S.w[b];
  }
  q5[q] = half(G.ipw[4][q]) * up;
  q6[q] = half(G.ipw[5][q]) * lo;
}
// calc_vorticity_flux_term, mo_vorticity_flux.F90:16-171
__global__ void k64_vort_flux(Dims D, Grid<F64> G, const F64* ex, const F64* ey, const F64* ez, const F64* uph, const F64* vph,
                              const F64* q5, const F64* q6, F64* px, F64* py, F64* pz) {
  LG_IDX3;
  const long long q = IX(D, ji, jk, jl), pl = D.plane;
  if (ji <= D.ny && jk <= D.nx + 1) {
    const bool inner = jk >= 2 && jk <= D.nx;
    if (inner || D.periodic) {
      const int kk = inner ? jk : 1, km = inner ? jk - 1 : D.nx;
      const long long a = IX(D, ji, km, jl), b = IX(D, ji, kk, jl);
      const F64 e0 = ey[b], e1 = ey[b + pl];
      px[q] = trsk_u<F64>(D, G, vph, uph, ez, ji, km, kk, kk + 1, jl) - q5[a] * e0 - q6[a] * e1 - q5[b] * e0 - q6[b] * e1;
    }
  }
  if (ji <= D.ny + 1 && jk <= D.nx) {
    const bool inner = ji >= 2 && ji <= D.ny;
    if (inner || D.periodic) {
      const int ii = inner ? ji : 1, im = inner ? ji - 1 : D.ny;
      const long long a = IX(D, im, jk, jl), b = IX(D, ii, jk, jl);
      const F64 e0 = ex[b], e1 = ex[b + pl];
      py[q] = trsk_v<F64>(D, G, uph, ez, im, ii, jk, jl) + q5[a] * e0 + q6[a] * e1 + q5[b] * e0 + q6[b] * e1;
    }
  }
  if (jl >= 2 && ji <= D.ny && jk <= D.nx) {
    const long long a = q - pl, e = q + D.P, s = q + 1;
    pz[q] = half(G.ipw[0][a] * uph[e - pl] * ey[e] - G.ipw[1][a] * vph[a] * ex[q] + G.ipw[2][a] * uph[a] * ey[q]
                 - G.ipw[3][a] * vph[s - pl] * ex[s] + G.ipw[0][q] * uph[e] * ey[e] - G.ipw[1][q] * vph[q] * ex[q]
                 + G.ipw[2][q] * uph[q] * ey[q] - G.ipw[3][q] * vph[s] * ex[s]);
  }
}

// combination of the explicit wind tendencies, mo_vector_tend_expl.F90:258-310, and the forward step
// of the horizontal wind, mo_manage_pchevi.F90:86-89; at the first substep the old tendency has
// weight 0 and is not read
__global__ void k64_tend_wind(Dims D, StateT<F64> So, StateT<F64> Sn, Tend<F64> Tn, CarriedF C, int rk_step) {
  LG_IDX3;
  const F64 chw = 0.5 + kIMPL_THERMO_WEIGHT, ohw = 1.0 - (0.5 + kIMPL_THERMO_WEIGHT), cvw = 1.0 - kIMPL_THERMO_WEIGHT;
  const long long q = IX(D, ji, jk, jl);
  auto weigh = [&](F64 f, F64* t) {
    if (rk_step == 2) f = half(*t) + half(f);
    *t = f;
    return f;
  };
  if (jl <= D.nl && ji <= D.ny && jk <= D.nx + 1) {
    F64 f = ohw * C.old_u[q] - chw * (C.nl_u[q] + C.l_u[q]) - half(C.vsg_x[q]) + C.pvt_x[q];
    if (C.mdt_x) f = f + C.mdt_x[q];
    Sn.u[q] = So.u[q] + F64(D.dtime) * weigh(f, Tn.u + q);
  }
  if (jl <= D.nl && ji <= D.ny + 1 && jk <= D.nx) {
    F64 f = ohw * C.old_v[q] - chw * (C.nl_v[q] + C.l_v[q]) - half(C.vsg_y[q]) + C.pvt_y[q];
    if (C.mdt_y) f = f + C.mdt_y[q];
    Sn.v[q] = So.v[q] + F64(D.dtime) * weigh(f, Tn.v + q);
  }
  if (ji <= D.ny && jk <= D.nx) {
    const F64 l = C.l_w[q];
    F64 f = -(cvw * (C.nl_w[q] + l));
    if (!D.luse_bg) f = f - (1.0 - (1.0 - kIMPL_THERMO_WEIGHT)) * l;
    f = f - half(C.vsg_z[q]) + C.pvt_z[q] + C.pgcw[q];
    if (C.mdt_z) f = f + C.mdt_z[q];
    weigh(f, Tn.w + q);
  }
}

// ---- diffusion closure (diffusion.cuh) --------------------------------------------------------------
// update_n_squared and tke_update, mo_eff_diff_coeffs.F90:620-669, mo_tke.F90:19-66, marching down the
// levels (theta_v, its reciprocal and the interface's n_squared are carried); gx, gy, gz: the gradient
// of the TKE (0 at non-periodic boundary edges and at the first and last level); decay_c =
// 8*pi^2/mean_velocity_area
__global__ void __launch_bounds__(128) k64_diff_tke(Dims D, Grid<F64> G, const F64* rdz, StateT<F64> S, DiffBuf<F64> B,
                                                    const F64* gx, const F64* gy, const F64* gz, double decay_c) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1, jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const int l0 = march_first(D, blockIdx.z), l1 = march_first(D, blockIdx.z + 1) - 1;
  if (l0 > l1) return;
  long long q = IX(D, ji, jk, l0);
  auto theta = [&](long long p) { return G.theta_v_bg[p] + S.tp[p]; };
  // g * 0.5*(1/theta(l-1) + 1/theta(l)) * dtheta/dz at the interface above layer p
  auto nz = [&](F64 tha, F64 ra, F64 thb, F64 rb, long long p) {
    return G.gm[p] * (half(ra + rb) * div_rn(tha - thb, G.dz[p], rdz[p]));
  };
  F64 th = theta(q), rth = rcp(th), n_up = 0.0;
  if (l0 >= 2) {
    const F64 ta = theta(q - D.plane);
    n_up = nz(ta, rcp(ta), th, rth, q);
  }
  for (int jl = l0; jl <= l1; ++jl, q += D.plane) {
    const long long b = q + D.plane, e = q + D.P, s = q + 1;
    F64 n_lo = 0.0;
    if (jl < D.nl) {
      const F64 tb = theta(b), rb = rcp(tb);
      n_lo = nz(th, rth, tb, rb, b);
      th = tb;
      rth = rb;
    }
    F64 nsq = 0.0;
    if (jl > 1 && jl < D.nl) nsq = G.ipw[4][q] * n_up + G.ipw[5][q] * n_lo;
    B.nsq[q] = nsq;
    n_up = n_lo;
    const F64 adv = G.ipw[0][q] * S.u[e] * gx[e] + G.ipw[1][q] * S.v[q] * gy[q] + G.ipw[2][q] * S.u[q] * gx[q]
                  + G.ipw[3][q] * S.v[s] * gy[s] + G.ipw[4][q] * S.w[q] * gz[q] + G.ipw[5][q] * S.w[b] * gz[b];
    const F64 rg = S.rho[q + (long long)(D.g - 1) * D.fstride], y = rcp_near(rg);
    const F64 decay_constant = div_rn(decay_c * B.visc[q], rg, y), tke = B.tke[q];
    F64 t = tke + D.dtime * (-adv + div_rn(B.hd[q], rg, y) - decay_constant * tke);
    if (negative(t)) t = 0.0;
    B.tke_new[q] = t;
  }
}
// the coefficients of the scalar diffusion (scalar_diff_coeffs, mo_eff_diff_coeffs.F90:526-618) at a
// cell: kind 0 mass, 1 temperature (c_g_v = rho_g/rho_g*c_d_v is c_d_v)
__global__ void k64_diff_cells(Dims D, Grid<F64> G, StateT<F64> S, DiffBuf<F64> B, int kind, int vertical, F64* ch, F64* cv) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl);
  const F64 rg = S.rho[q + (long long)(D.g - 1) * D.fstride];
  ch[q] = kind == 0 ? B.visc[q] / rg : kC_D_V * B.visc[q];
  if (!vertical) return;
  const F64 t2v = B.vmol[q] + tke2vert<F64>(B.tke[q], B.nsq[q], G.layer_thickness[q]);
  cv[q] = kind == 0 ? t2v : rg * kC_D_V * t2v;
}
// at the faces and interfaces: the mean of the two cells
__global__ void k64_diff_face_coeffs(Dims D, const F64* ch, const F64* cv, int vertical, F64* hx, F64* hy, F64* hw) {
  LG_IDX3;
  const long long q = IX(D, ji, jk, jl);
  if (ji <= D.ny && jk <= D.nx + 1) {
    const bool inner = jk >= 2 && jk <= D.nx;
    hx[q] = half(ch[inner ? q - D.P : IX(D, ji, D.nx, jl)] + ch[inner ? q : IX(D, ji, 1, jl)]);
  }
  if (ji <= D.ny + 1 && jk <= D.nx) {
    const bool inner = ji >= 2 && ji <= D.ny;
    hy[q] = half(ch[inner ? q - 1 : IX(D, D.ny, jk, jl)] + ch[inner ? q : IX(D, 1, jk, jl)]);
  }
  if (vertical && jl >= 2 && ji <= D.ny && jk <= D.nx) hw[q] = half(cv[q - D.plane] + cv[q]);
}
// the diffusive flux of a scalar through the faces: coefficient times gradient
__global__ void k64_diff_faces(Dims D, Grid<F64> G, Recip R, const F64* s, const F64* w5, const F64* w6, const F64* hx,
                               const F64* hy, Faces F) {
  LG_IDX3;
  const long long q = IX(D, ji, jk, jl);
  F64 r;
  if (ji <= D.ny && jk <= D.nx + 1)
    face_x(D, G, grad_x64(D, G, R.dx, s, w5, w6, ji, jk, jl, &r) ? hx[q] * r : F64(0.0), F, jl, q);
  if (ji <= D.ny + 1 && jk <= D.nx)
    face_y(D, G, grad_y64(D, G, R.dy, s, w5, w6, ji, jk, jl, &r) ? hy[q] * r : F64(0.0), F, jl, q);
}
// its divergence, with the vertical part (add_vertical_div, mo_divergence_operators.F90:149-186)
__global__ void __launch_bounds__(128) k64_diff_div(Dims D, Grid<F64> G, const F64* rvol, Faces F, const F64* hw, const F64* gz,
                                                    int vertical, F64* out) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1, jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const int l0 = march_first(D, blockIdx.z), l1 = march_first(D, blockIdx.z + 1) - 1;
  if (l0 > l1) return;
  long long q = IX(D, ji, jk, l0);
  ColumnDiv c;
  c.start(D, G, F, q, l0);
  F64 up = 0.0;
  if (vertical && l0 >= 2) up = hw[q] * gz[q] * G.area_z[q];
  for (int jl = l0; jl <= l1; ++jl, q += D.plane) {
    const F64 V = G.volume[q], rV = rvol[q];
    F64 r = c.step(D, G, F, V, rV, q, jl);
    if (vertical) {
      const long long b = q + D.plane;
      F64 lo = 0.0;
      if (jl < D.nl) lo = hw[b] * gz[b] * G.area_z[b];
      r = r + div_rn(up - lo, V, rV);
      up = lo;
    }
    out[q] = r;
  }
}

}  // namespace

const DiffBuf<F64>& f64(const DiffBuf<double>& b) { return reinterpret_cast<const DiffBuf<F64>&>(b); }
void launch64_diff_tke(const Dims& D, const Grid<double>& G, const Recip& R, const State& S, const DiffBuf<double>& B,
                       const double* gx, const double* gy, const double* gz, double mva, cudaStream_t st) {
  k64_diff_tke<<<march_grid(D), kMarchBlock, 0, st>>>(D, f64(G), R.dz, f64(S), f64(B), f64(gx), f64(gy), f64(gz),
                                                      8.0 * (kPI * kPI) / mva);
}
void launch64_diff_coeffs(const Dims& D, const Grid<double>& G, const State& S, const DiffBuf<double>& B, int kind, int vertical,
                          double* ch, double* cv, cudaStream_t st) {
  k64_diff_cells<<<cell_grid(D.ny, D.nx, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(S), f64(B), kind, vertical, f64(ch), f64(cv));
}
void launch64_diff_face_coeffs(const Dims& D, const double* ch, const double* cv, int vertical, const DiffBuf<double>& B,
                               cudaStream_t st) {
  k64_diff_face_coeffs<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(ch), f64(cv), vertical, f64(B.flx),
                                                                                   f64(B.fly), f64(B.flw));
}
void launch64_diff_faces(const Dims& D, const Grid<double>& G, const Recip& R, const double* s, const double* w5,
                         const double* w6, const DiffBuf<double>& B, const Faces& F, cudaStream_t st) {
  k64_diff_faces<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(G), R, f64(s), f64(w5), f64(w6), f64(B.flx),
                                                                             f64(B.fly), F);
}
void launch64_diff_div(const Dims& D, const Grid<double>& G, const Recip& R, const Faces& F, const DiffBuf<double>& B,
                       const double* gz, int vertical, double* out, cudaStream_t st) {
  k64_diff_div<<<march_grid(D), kMarchBlock, 0, st>>>(D, f64(G), R.vol, F, f64(B.flw), f64(gz), vertical, f64(out));
}
// the closure's other kernels are the templates of diffusion.cuh
void launch64_diff_visc(const Dims& D, const Grid<double>& G, const State& S, const double* T, const DiffBuf<double>& B,
                        const DiffPar& P, cudaStream_t st) {
  k_diff_visc<F64, F64><<<cell_grid(D.ny, D.nx, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(S), f64(T), f64(B), P);
}
void launch64_diff_vz(const Dims& D, const Grid<double>& G, const State& S, const DiffBuf<double>& B, cudaStream_t st) {
  k_diff_vz<F64, F64><<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(S), f64(B));
}
void launch64_mom_diff_h(const Dims& D, const Grid<double>& G, const State& S, const DiffBuf<double>& B, cudaStream_t st) {
  k_mom_diff_h<F64, F64><<<cell_grid(D.ny, D.nx, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(S), f64(B));
}
void launch64_mom_diff_v(const Dims& D, const Grid<double>& G, const State& S, const DiffBuf<double>& B, cudaStream_t st) {
  k_mom_diff_v<F64, F64><<<cell_grid(D.ny, D.nx, D.nl - 1), kCellBlock, 0, st>>>(D, f64(G), f64(S), f64(B));
}
void launch64_diss_rate(const Dims& D, const Grid<double>& G, const State& S, const DiffBuf<double>& B, cudaStream_t st) {
  k_diss_rate<F64, F64><<<cell_grid(D.ny, D.nx, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(S), f64(B), f64(G.damp),
                                                                           (const F64*)nullptr);
}

void launch64_rot_grid(const Dims& D, const Grid<double>& G, double* const* a, cudaStream_t st) {
  k64_rot_grid<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(a[0]), f64(a[1]), f64(a[2]), f64(a[3]));
}
void launch64_zeta_z(const Dims& D, const Grid<double>& G, const RotGrid& X, const State& S, double* zz, cudaStream_t st) {
  k64_zeta_z<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(G), X, f64(S), f64(zz));
}
void launch64_eta_z(const Dims& D, const Grid<double>& G, const RotGrid& X, const State& S, double* ez, cudaStream_t st) {
  k64_eta_z<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(G), X, f64(S), f64(ez));
}
void launch64_covariant(const Dims& D, const Grid<double>& G, const State& S, double* cx, double* cy, cudaStream_t st) {
  k64_covariant<<<cell_grid(D.ny, D.nx, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(S), f64(cx), f64(cy));
}
void launch64_eta_xy(const Dims& D, const Grid<double>& G, const State& S, const double* cx, const double* cy, double* ex,
                     double* ey, cudaStream_t st) {
  k64_eta_xy<<<cell_grid(D.ny + 1, D.nx + 1, D.NL), kCellBlock, 0, st>>>(D, f64(G), f64(S), f64(cx), f64(cy), f64(ex), f64(ey));
}
void launch64_mass_flux(const Dims& D, const Grid<double>& G, const State& S, double* uph, double* vph, double* q5, double* q6,
                        cudaStream_t st) {
  k64_mass_flux<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(S), f64(uph), f64(vph), f64(q5), f64(q6));
}
void launch64_vort_flux(const Dims& D, const Grid<double>& G, const double* ex, const double* ey, const double* ez,
                        const double* uph, const double* vph, const double* q5, const double* q6, double* px, double* py,
                        double* pz, cudaStream_t st) {
  k64_vort_flux<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(ex), f64(ey), f64(ez), f64(uph), f64(vph),
                                                                           f64(q5), f64(q6), f64(px), f64(py), f64(pz));
}
void launch64_tend_wind(const Dims& D, const State& So, const State& Sn, const Tend<double>& Tn, const Carried<double>& C,
                        int rk_step, cudaStream_t st) {
  const Tend<F64> T{f64(Tn.rho), f64(Tn.rt), f64(Tn.u), f64(Tn.v), f64(Tn.w)};
  const CarriedF K{f64(C.nl_u), f64(C.nl_v), f64(C.nl_w), f64(C.l_u), f64(C.l_v), f64(C.l_w), f64(C.old_u), f64(C.old_v),
                   f64(C.pgcw), f64(C.vsg_x), f64(C.vsg_y), f64(C.vsg_z), f64(C.pvt_x), f64(C.pvt_y), f64(C.pvt_z),
                   f64(C.mdt_x), f64(C.mdt_y), f64(C.mdt_z)};
  k64_tend_wind<<<cell_grid(D.ny + 1, D.nx + 1, D.NL), kCellBlock, 0, st>>>(D, f64(So), f64(Sn), T, K, rk_step);
}

void launch64_pgrad_cells(const Dims& D, const Grid<double>& G, const State& S, double* th, double* decel, double* cond,
                          cudaStream_t st) {
  k64_pgrad_cells<<<cell_grid(D.ny, D.nx, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(S), f64(th), f64(decel), f64(cond));
}
void launch64_pgrad(const Dims& D, const Grid<double>& G, const State& S, const double* gx, const double* gy, const double* gz,
                    const double* th, const double* decel, const double* cond, const double* tvu, const double* tvv,
                    const double* tpu, const double* tpv, const PGrad<double>& P, int lfirst, cudaStream_t st) {
  k64_pgrad<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(S), f64(gx), f64(gy), f64(gz), f64(th), f64(decel), f64(cond), f64(tvu), f64(tvv), f64(tpu),
                                                                       f64(tpv), PGradF{f64(P.nl_u), f64(P.nl_v), f64(P.nl_w), f64(P.l_u), f64(P.l_v), f64(P.l_w), f64(P.old_u), f64(P.old_v), f64(P.pgcw)}, lfirst);
}
void launch64_recip(const Dims& D, const Grid<double>& G, double* rdx, double* rdy, double* rdz, cudaStream_t st) {
  k64_recip<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(rdx), f64(rdy), f64(rdz));
}
void launch64_grad_vert(const Dims& D, const Grid<double>& G, const Recip& R, const double* s, double* gz, double* w5,
                        double* w6, cudaStream_t st) {
  k64_grad_vert<<<march_grid(D), kMarchBlock, 0, st>>>(D, f64(G), R.dz, f64(s), f64(gz), f64(w5), f64(w6));
}
void launch64_grad_hor(const Dims& D, const Grid<double>& G, const Recip& R, const double* s, const double* w5,
                       const double* w6, double* rx, double* ry, cudaStream_t st) {
  k64_grad_hor<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(G), R, f64(s), f64(w5), f64(w6), f64(rx), f64(ry));
}
void launch64_grad_faces(const Dims& D, const Grid<double>& G, const Recip& R, const double* s, const double* w5,
                         const double* w6, const Faces& F, cudaStream_t st) {
  k64_grad_faces<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(G), R, f64(s), f64(w5), f64(w6), F);
}
void launch64_div(const Dims& D, const Grid<double>& G, const Recip& R, const Faces& F, double* out, cudaStream_t st) {
  k64_div<<<march_grid(D), kMarchBlock, 0, st>>>(D, f64(G), R.vol, F, f64(out));
}
void launch64_theta_edges(const Dims& D, const double* th, const double* dv, const double* u, const double* v, double* tvu,
                          double* tvv, cudaStream_t st) {
  k64_theta_edges<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(th), f64(dv), f64(u), f64(v), f64(tvu), f64(tvv));
}
void launch64_gas_faces(const Dims& D, const Grid<double>& G, const State& Ss, const double* u_new, const double* v_new,
                        const double* tvu, const double* tvv, const Faces& M, const Faces& T, cudaStream_t st) {
  k64_gas_faces<<<cell_grid(D.ny + 1, D.nx + 1, D.nl), kCellBlock, 0, st>>>(D, f64(G), f64(Ss), f64(u_new), f64(v_new), f64(tvu), f64(tvv), M, T);
}
void launch64_gas_theta(const Dims& D, const Grid<double>& G, const Recip& R, const State& Ss, const Faces& M, const Faces& T,
                        const double* cpi, const double* cpw, const double* hd, const double* rad, const double* csh,
                        double* t_rho, double* t_rt, const double* mdt, const double* tdh, const double* ptr,
                        const double* pth, cudaStream_t st) {
  k64_gas_theta<<<march_grid(D), kMarchBlock, 0, st>>>(D, f64(G), f64(Ss), R.vol, M, T, f64(cpi), f64(cpw), f64(hd), f64(rad), f64(csh), f64(t_rho), f64(t_rt), f64(mdt), f64(tdh),
                                                       f64(ptr), f64(pth));
}
void launch64_wind_slopes(const Dims& D, const Grid<double>& G, const double* u, const double* v, double* hx, double* hy,
                          cudaStream_t st) {
  k64_wind_slopes<<<cell_grid(D.ny + 1, D.nx + 1, D.nl - D.nf), kCellBlock, 0, st>>>(D, f64(G), f64(u), f64(v), f64(hx), f64(hy));
}
void launch64_contra(const Dims& D, const Grid<double>& G, const double* hx, const double* hy, double* cw, cudaStream_t st) {
  k64_contra<<<march_grid(D), kMarchBlock, 0, st>>>(D, f64(G), f64(hx), f64(hy), f64(cw));
}
void launch64_tracers(const Dims& D, const Grid<double>& G, const Recip& R, const State& Ss, const double* u_new,
                      const double* v_new, const double* cw, double* t_rho, int rk_step, const double* mdt, const double* ptr,
                      cudaStream_t st) {
  k64_tracers<<<cell_grid(D.ny, D.nx, D.nl), kCellBlock, 0, st>>>(D, f64(G), R.vol, f64(Ss), f64(u_new), f64(v_new), f64(cw), f64(t_rho), rk_step, f64(mdt), f64(ptr));
}

}  // namespace lg
