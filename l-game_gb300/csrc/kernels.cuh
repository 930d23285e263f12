// kernels.cuh -- pointwise helpers and the explicit-tendency kernels of the HEVI step,
// templated on the type T of the grid metrics, the intermediate fields and the
// arithmetic.  The state is always FP64.
//
//   T = double: the FP64 step (kernels_fp64.cu, -fmad=false): every expression keeps the
//               reference's operands and left-to-right order, so the results are the
//               reference's bits.
//   T = float:  the explicit stencils of the split-precision step (split.cu): the same
//               expressions in FP32 on FP32 copies of the metrics.
#pragma once

#include "dev.cuh"

namespace lg {

template <class T>
struct PGrad {  // pressure-gradient arrays of t_diag (mo_definitions.F90:137-146), always FP64
  double *nl_u, *nl_v, *nl_w, *l_u, *l_v, *l_w, *old_u, *old_v;
  T* pgcw;
};

template <class T>
struct Tend {  // t_tend (mo_definitions.F90:108-116)
  T *rho, *rt, *u, *v, *w;
};

template <class T>
struct Carried {  // read-only view of the diagnostics combined into the wind tendency
  const double *nl_u, *nl_v, *nl_w, *l_u, *l_v, *l_w, *old_u, *old_v;
  const T *pgcw, *vsg_x, *vsg_y, *vsg_z, *pvt_x, *pvt_y, *pvt_z;
  const T *mdt_x = nullptr, *mdt_y = nullptr, *mdt_z = nullptr;  // momentum diffusion (null: off)
};

// ---- edge operators with the reference's boundary branches --------------------
// Each returns false where the reference leaves the output point untouched
// (non-periodic boundary edges); periodic jk=nx+1 / ji=ny+1 evaluate the copy source.

// grad_hor_cov x-component at a u point, mo_gradient_operators.F90:33-52.  The difference
// is taken in the source type S and rounded to T afterwards (FP64 field, FP32 result).
template <class T, class S>
__device__ __forceinline__ bool grad_x_cov(const Dims& D, const Grid<T>& G, const S* s, int ji, int jk, int jl, T* r) {
  if (jk >= 2 && jk <= D.nx) {
    *r = cvt<T>(s[IX(D, ji, jk, jl)] - s[IX(D, ji, jk - 1, jl)]) / G.dx[IX(D, ji, jk, jl)];
    return true;
  }
  if (!D.periodic) return false;
  *r = cvt<T>(s[IX(D, ji, 1, jl)] - s[IX(D, ji, D.nx, jl)]) / G.dx[IX(D, ji, 1, jl)];
  return true;
}

// grad_hor_cov y-component at a v point, mo_gradient_operators.F90:39-60
template <class T, class S>
__device__ __forceinline__ bool grad_y_cov(const Dims& D, const Grid<T>& G, const S* s, int ji, int jk, int jl, T* r) {
  if (ji >= 2 && ji <= D.ny) {
    *r = cvt<T>(s[IX(D, ji - 1, jk, jl)] - s[IX(D, ji, jk, jl)]) / G.dy[IX(D, ji, jk, jl)];
    return true;
  }
  if (!D.periodic) return false;
  *r = cvt<T>(s[IX(D, D.ny, jk, jl)] - s[IX(D, 1, jk, jl)]) / G.dy[IX(D, 1, jk, jl)];
  return true;
}

// scalar_times_vector_h, mo_multiplications.F90:34-54 (state scalar and vector)
template <class T, class V>
__device__ __forceinline__ bool stv_h_x(const Dims& D, const V* s, const V* vx, int ji, int jk, int jl, T* r) {
  if (jk >= 2 && jk <= D.nx) {
    *r = half_of(T(s[IX(D, ji, jk - 1, jl)]) + T(s[IX(D, ji, jk, jl)])) * T(vx[IX(D, ji, jk, jl)]);
    return true;
  }
  if (!D.periodic) return false;
  *r = half_of(T(s[IX(D, ji, 1, jl)]) + T(s[IX(D, ji, D.nx, jl)])) * T(vx[IX(D, ji, 1, jl)]);
  return true;
}
template <class T, class V>
__device__ __forceinline__ bool stv_h_y(const Dims& D, const V* s, const V* vy, int ji, int jk, int jl, T* r) {
  if (ji >= 2 && ji <= D.ny) {
    *r = half_of(T(s[IX(D, ji - 1, jk, jl)]) + T(s[IX(D, ji, jk, jl)])) * T(vy[IX(D, ji, jk, jl)]);
    return true;
  }
  if (!D.periodic) return false;
  *r = half_of(T(s[IX(D, 1, jk, jl)]) + T(s[IX(D, D.ny, jk, jl)])) * T(vy[IX(D, 1, jk, jl)]);
  return true;
}
// sum(state%rho(:,:,:,1:nc+1),4) in constituent order
template <class T, class V>
__device__ __forceinline__ T rho_sum_cond_gas(const Dims& D, const V* rho, long long q) {
  T s = T(0);
  for (int jc = 0; jc <= D.nc; ++jc) s = s + T(rho[q + (long long)jc * D.fstride]);
  return s;
}

// c_p of the condensates, mo_dictionary.F90:112-189 (float: the same formulas in FP32)
__device__ __forceinline__ float c_p_water(float temperature) {
  float tc = temperature - float(kT_0), c;
  if (tc >= 0.f) {
    if (tc > 35.f) tc = 35.f;
    const float a = tc - 35.f, a2 = a * a;
    c = 0.9979f + 3.1e-6f * a2 + 3.8e-9f * (a2 * a2);
  } else {
    if (tc < -37.f) tc = -37.f;
    const float t2 = tc * tc;
    c = 1.000938f - 2.7052e-3f * tc - 2.3235e-5f * t2 + 4.3778e-6f * (t2 * tc) + 2.7136e-7f * (t2 * t2);
  }
  return 4186.8f * c;
}
__device__ __forceinline__ float c_p_ice(float temperature) {
  float tl = temperature;
  if (tl > float(kT_0)) tl = float(kT_0);
  if (tl < 20.f) tl = 20.f;
  const float q = tl * (1.f / 125.1f);
  const float c = -2.0572f + 0.14644f * tl + 0.06163f * tl * __expf(-(q * q));
  return c * float(1.0 / kM_V);
}
__device__ __forceinline__ float c_p_cond(int jc, float temperature) {
  return ((jc - 1) % 2 == 0) ? c_p_ice(temperature) : c_p_water(temperature);
}

// inner_product, mo_inner_product.F90:16-50 (both vectors the state wind)
template <class T, class V>
__device__ __forceinline__ T inner_product_at(const Dims& D, const Grid<T>& G, const V* u, const V* v,
                                              const V* w, int ji, int jk, int jl) {
  const T a = T(u[IX(D, ji, jk + 1, jl)]), b = T(v[IX(D, ji, jk, jl)]), c = T(u[IX(D, ji, jk, jl)]);
  const T d = T(v[IX(D, ji + 1, jk, jl)]), e = T(w[IX(D, ji, jk, jl)]), f = T(w[IX(D, ji, jk, jl + 1)]);
  return W_(1, ji, jk, jl) * a * a + W_(2, ji, jk, jl) * b * b + W_(3, ji, jk, jl) * c * c
       + W_(4, ji, jk, jl) * d * d + W_(5, ji, jk, jl) * e * e + W_(6, ji, jk, jl) * f * f;
}

// ---- potential vorticity, mo_vorticities.F90 -----------------------------------

// rel_vort x-component before the division by the area, mo_vorticities.F90:33-93
template <class T, class V>
__device__ __forceinline__ T zeta_x_raw(const Dims& D, const Grid<T>& G, const StateT<V>& S, int ji, int jk, int jl) {
  const V* v = S.v; const V* w = S.w;
  if (jl <= D.nl) {  // levels 2..nl
    const bool inner = ji >= 2 && ji <= D.ny;
    if (!inner && !D.periodic) return T(0);
    const int ii = inner ? ji : 1, im = inner ? ji - 1 : D.ny;
    return apart(G.dz[IX(D, im, jk, jl)], T(w[IX(D, im, jk, jl)]))
         - G.dy[IX(D, ii, jk, jl - 1)] * hcov_y<T, V>(D, G, v, w, ii, jk, jl - 1)
         - apart(G.dz[IX(D, ii, jk, jl)], T(w[IX(D, ii, jk, jl)]))
         + G.dy[IX(D, ii, jk, jl)] * hcov_y<T, V>(D, G, v, w, ii, jk, jl);
  }
  // surface level NL
  const int nl = D.nl, NL = D.NL;
  const bool inner = ji >= 2 && ji <= D.ny;
  int ii = ji;
  if (D.freeslip && D.periodic && ji == D.ny + 1) ii = 1;  // copy made after the free-slip addition
  T r = -G.dy[IX(D, ii, jk, nl)] * hcov_y<T, V>(D, G, v, w, ii, jk, nl);
  if (D.freeslip && (inner || (D.periodic && ii == 1))) {
    const int im = (ii == 1) ? D.ny : ii - 1;
    r = r + apart(half_of(G.dz[IX(D, im, jk, NL)]), T(w[IX(D, im, jk, NL)]))
          - apart(half_of(G.dz[IX(D, ii, jk, NL)]), T(w[IX(D, ii, jk, NL)]))
          + G.dy[IX(D, ii, jk, nl)] * (T(v[IX(D, ii, jk, nl)])
          + (T(v[IX(D, ii, jk, nl - 1)]) - T(v[IX(D, ii, jk, nl)])) / (G.z_v[IX(D, ii, jk, nl - 1)] - G.z_v[IX(D, ii, jk, nl)])
          * (half_of(G.z_w[IX(D, im, jk, NL)] + G.z_w[IX(D, ii, jk, NL)]) - G.z_v[IX(D, ii, jk, nl)])
          + half_of(T(w[IX(D, im, jk, NL)]) + T(w[IX(D, ii, jk, NL)]))
          * (G.z_w[IX(D, im, jk, NL)] - G.z_w[IX(D, ii, jk, NL)]) / G.dy[IX(D, ii, jk, nl)]);
  }
  return r;
}

// rel_vort y-component before the division, mo_vorticities.F90:104-165
template <class T, class V>
__device__ __forceinline__ T zeta_y_raw(const Dims& D, const Grid<T>& G, const StateT<V>& S, int ji, int jk, int jl) {
  const V* u = S.u; const V* w = S.w;
  if (jl <= D.nl) {
    const bool inner = jk >= 2 && jk <= D.nx;
    if (!inner && !D.periodic) return T(0);
    const int kk = inner ? jk : 1, km = inner ? jk - 1 : D.nx;
    return -apart(G.dz[IX(D, ji, kk, jl)], T(w[IX(D, ji, kk, jl)]))
         - G.dx[IX(D, ji, kk, jl)] * hcov_x<T, V>(D, G, u, w, ji, kk, jl)
         + apart(G.dz[IX(D, ji, km, jl)], T(w[IX(D, ji, km, jl)]))
         + G.dx[IX(D, ji, kk, jl - 1)] * hcov_x<T, V>(D, G, u, w, ji, kk, jl - 1);
  }
  const int nl = D.nl, NL = D.NL;
  const bool inner = jk >= 2 && jk <= D.nx;
  int kk = jk;
  if (D.freeslip && D.periodic && jk == D.nx + 1) kk = 1;
  T r = G.dx[IX(D, ji, kk, nl)] * hcov_x<T, V>(D, G, u, w, ji, kk, nl);
  if (D.freeslip && (inner || (D.periodic && kk == 1))) {
    const int km = (kk == 1) ? D.nx : kk - 1;
    r = r + apart(half_of(G.dz[IX(D, ji, km, NL)]), T(w[IX(D, ji, km, NL)]))
          - apart(half_of(G.dz[IX(D, ji, kk, NL)]), T(w[IX(D, ji, kk, NL)]))
          - G.dx[IX(D, ji, kk, nl)] * (T(u[IX(D, ji, kk, nl)])
          + (T(u[IX(D, ji, kk, nl - 1)]) - T(u[IX(D, ji, kk, nl)])) / (G.z_u[IX(D, ji, kk, nl - 1)] - G.z_u[IX(D, ji, kk, nl)])
          * (half_of(G.z_w[IX(D, ji, km, NL)] + G.z_w[IX(D, ji, kk, NL)]) - G.z_u[IX(D, ji, kk, nl)])
          + half_of(T(w[IX(D, ji, km, NL)]) + T(w[IX(D, ji, kk, NL)]))
          * (G.z_w[IX(D, ji, kk, NL)] - G.z_w[IX(D, ji, km, NL)]) / G.dx[IX(D, ji, kk, nl)]);
  }
  return r;
}

// density at a horizontal vorticity point (two scalar columns a and b), mo_vorticities.F90:240-266
template <class T, class V>
__device__ __forceinline__ T rho_avg_h(const Dims& D, const Grid<T>& G, const V* rho, int ia, int ka, int ib,
                                       int kb, int jl) {
  const T* zs = G.z_scalar;
  auto R = [&](int i, int k, int l) { return T(rho[IX(D, i, k, l)]); };
  if (jl == 1) {
    return half_of(R(ia, ka, jl)
      + (cvt<T>(D.toa) - zs[IX(D, ia, ka, jl)]) * (R(ia, ka, jl) - R(ia, ka, jl + 1))
        / (zs[IX(D, ia, ka, jl)] - zs[IX(D, ia, ka, jl + 1)])
      + R(ib, kb, jl)
      + (cvt<T>(D.toa) - zs[IX(D, ib, kb, jl)]) * (R(ib, kb, jl) - R(ib, kb, jl + 1))
        / (zs[IX(D, ib, kb, jl)] - zs[IX(D, ib, kb, jl + 1)]));
  }
  if (jl == D.NL) {
    const T* zw = G.z_w;
    return half_of(R(ia, ka, jl - 1)
      + (zw[IX(D, ia, ka, jl)] - zs[IX(D, ia, ka, jl - 1)]) * (R(ia, ka, jl - 2) - R(ia, ka, jl - 1))
        / (zs[IX(D, ia, ka, jl - 2)] - zs[IX(D, ia, ka, jl - 1)])
      + R(ib, kb, jl - 1)
      + (zw[IX(D, ib, kb, jl)] - zs[IX(D, ib, kb, jl - 1)]) * (R(ib, kb, jl - 2) - R(ib, kb, jl - 1))
        / (zs[IX(D, ib, kb, jl - 2)] - zs[IX(D, ib, kb, jl - 1)]));
  }
  return quarter_of(R(ia, ka, jl - 1) + R(ib, kb, jl - 1) + R(ia, ka, jl) + R(ib, kb, jl));
}

// eta_x at (ji,jk,jl), jl in 1..nl+1
template <class T, class V>
__device__ __forceinline__ T eta_x_at(const Dims& D, const Grid<T>& G, const StateT<V>& S, int ji, int jk, int jl) {
  if (D.periodic && ji == D.ny + 1) ji = 1;  // eta_x(ny+1,:,:) = eta_x(1,:,:) after the division
  T z = T(0);
  if (!D.llinear) {
    const int lev = (jl == 1) ? 2 : jl;  // zeta_x(:,:,1) = zeta_x(:,:,2) after the division
    z = zeta_x_raw<T>(D, G, S, ji, jk, lev) / G.area_dual_x[IX(D, ji, jk, lev)];
  }
  T e = D.lcorio ? z + G.fvec_x[IX(D, ji, jk, 1)] : z;
  const bool inner = ji >= 2 && ji <= D.ny;
  if (inner || D.periodic) {
    const int ia = inner ? ji - 1 : D.ny, ib = inner ? ji : 1;
    e = e / rho_avg_h<T>(D, G, S.rho + (long long)(D.g - 1) * D.fstride, ia, jk, ib, jk, jl);
  }
  return e;
}

// eta_y at (ji,jk,jl)
template <class T, class V>
__device__ __forceinline__ T eta_y_at(const Dims& D, const Grid<T>& G, const StateT<V>& S, int ji, int jk, int jl) {
  if (D.periodic && jk == D.nx + 1) jk = 1;
  T z = T(0);
  if (!D.llinear) {
    const int lev = (jl == 1) ? 2 : jl;
    z = zeta_y_raw<T>(D, G, S, ji, jk, lev) / G.area_dual_y[IX(D, ji, jk, lev)];
  }
  T e = D.lcorio ? z + G.fvec_y[IX(D, ji, jk, 1)] : z;
  const bool inner = jk >= 2 && jk <= D.nx;
  if (inner || D.periodic) {
    const int ka = inner ? jk - 1 : D.nx, kb = inner ? jk : 1;
    e = e / rho_avg_h<T>(D, G, S.rho + (long long)(D.g - 1) * D.fstride, ji, ka, ji, kb, jl);
  }
  return e;
}

// TRSK term for u, mo_vorticity_flux.F90:33-45 (km, kk, kp: columns jk-1, jk, jk+1)
template <class T>
__device__ __forceinline__ T trsk_u(const Dims& D, const Grid<T>& G, const T* vp, const T* up, const T* ez,
                                    int ji, int km, int kk, int kp, int jl) {
  const T w1 = G.trsk_u[0][ji - 1], w2 = G.trsk_u[1][ji - 1], w3 = G.trsk_u[2][ji - 1];
#define EZ(i, k) ez[IX(D, i, k, jl)]
  return quarter_of(w1 * vp[IX(D, ji, km, jl)]) * (EZ(ji, km) + EZ(ji, kk) + EZ(ji, kk) + EZ(ji + 1, kk))
       + quarter_of(w2 * up[IX(D, ji, km, jl)]) * (EZ(ji, km) + EZ(ji + 1, km) + EZ(ji, kk) + EZ(ji + 1, kk))
       + quarter_of(w3 * vp[IX(D, ji + 1, km, jl)]) * (EZ(ji + 1, km) + EZ(ji + 1, kk) + EZ(ji, kk) + EZ(ji + 1, kk))
       + quarter_of(w3 * vp[IX(D, ji + 1, kk, jl)]) * (EZ(ji + 1, kk) + EZ(ji + 1, kp) + EZ(ji, kk) + EZ(ji + 1, kk))
       + quarter_of(w2 * up[IX(D, ji, kp, jl)]) * (EZ(ji + 1, kp) + EZ(ji, kp) + EZ(ji, kk) + EZ(ji + 1, kk))
       + quarter_of(w1 * vp[IX(D, ji, kk, jl)]) * (EZ(ji, kk) + EZ(ji, kp) + EZ(ji, kk) + EZ(ji + 1, kk));
}

// TRSK term for v, mo_vorticity_flux.F90:72-80 (im, ii: rows ji-1, ji)
template <class T>
__device__ __forceinline__ T trsk_v(const Dims& D, const Grid<T>& G, const T* up, const T* ez, int im, int ii, int jk,
                                    int jl) {
  const T w1 = G.trsk_v[0][ii - 1], w2 = G.trsk_v[1][ii - 1];
  return quarter_of(w1 * up[IX(D, ii, jk, jl)]) * (EZ(ii, jk) + EZ(ii + 1, jk) + EZ(ii, jk) + EZ(ii, jk + 1))
       + quarter_of(w1 * up[IX(D, ii, jk + 1, jl)]) * (EZ(ii, jk + 1) + EZ(ii + 1, jk + 1) + EZ(ii, jk) + EZ(ii, jk + 1))
       + quarter_of(w2 * up[IX(D, im, jk + 1, jl)]) * (EZ(im, jk + 1) + EZ(ii, jk + 1) + EZ(ii, jk) + EZ(ii, jk + 1))
       + quarter_of(w2 * up[IX(D, im, jk, jl)]) * (EZ(im, jk) + EZ(ii, jk) + EZ(ii, jk) + EZ(ii, jk + 1));
#undef EZ
}

// 3-D launches: blockIdx.x tiles the rows (ji), blockIdx.y is the level and blockIdx.z tiles
// the columns (jk), so blocks launched one after another cover one level's row tiles and then
// the same rows one level down: the vertical neighbours a stencil reads are still in L2
// (with the columns in blockIdx.y they were a whole level plane of blocks apart)
#define LG_IDX3                                              \
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;  \
  const int jk = blockIdx.z * blockDim.y + threadIdx.y + 1;  \
  const int jl = blockIdx.y + 1

// ---- kernels --------------------------------------------------------------------

// temperature_diagnostics, mo_derived.F90:18-38
template <class T, class V = double>
__global__ void k_temperature(Dims D, Grid<T> G, StateT<V> S, T* Tm) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long i = IX(D, ji, jk, jl);
  T t = (G.theta_v_bg[i] + T(S.tp[i])) * (G.exner_bg[i] + T(S.ep[i]));
  if (D.lmoist) {
    const T rg = T(S.rho[i + (long long)(D.g - 1) * D.fstride]);
    const T rv = T(S.rho[i + (long long)D.g * D.fstride]);
    t = t / (T(1) + rv / rg * T(kM_D / kM_V - 1.0));
  }
  Tm[i] = t;
}

// diag%scalar_placeholder = theta_v_bg + theta_v_pert (mode 0) or theta_v_pert (mode 1)
template <class T, class V = double>
__global__ void k_theta(Dims D, Grid<T> G, const V* tp, T* out, int mode) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long i = IX(D, ji, jk, jl);
  out[i] = mode == 0 ? G.theta_v_bg[i] + T(tp[i]) : T(tp[i]);
}

// grad_vert, mo_gradient_operators.F90:65-83 (levels 2..nl); launched with blockIdx.y = jl-2
template <class T, class S>
__global__ void k_grad_vert(Dims D, Grid<T> G, const S* s, T* rz) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int jk = blockIdx.z * blockDim.y + threadIdx.y + 1;
  const int jl = blockIdx.y + 2;
  if (ji > D.ny || jk > D.nx || jl > D.nl) return;
  rz[IX(D, ji, jk, jl)] = cvt<T>(s[IX(D, ji, jk, jl - 1)] - s[IX(D, ji, jk, jl)]) / G.dz[IX(D, ji, jk, jl)];
}

// grad_hor, mo_gradient_operators.F90:17-63 + :85-130, u and v points of layer jl
template <class T, class S>
__global__ void k_grad_hor(Dims D, Grid<T> G, const S* s, const T* rz, T* rx, T* ry) {
  LG_IDX3;
  if (ji <= D.ny && jk <= D.nx + 1) {
    T r;
    if (grad_x_cov<T, S>(D, G, s, ji, jk, jl, &r)) {
      if (jl > D.nf) r = r - G.slope_x[IX(D, ji, jk, jl)] * remap_x<T, T>(D, G, rz, ji, jk, jl);
      rx[IX(D, ji, jk, jl)] = r;
    }
  }
  if (ji <= D.ny + 1 && jk <= D.nx) {
    T r;
    if (grad_y_cov<T, S>(D, G, s, ji, jk, jl, &r)) {
      if (jl > D.nf) r = r - G.slope_y[IX(D, ji, jk, jl)] * remap_y<T, T>(D, G, rz, ji, jk, jl);
      ry[IX(D, ji, jk, jl)] = r;
    }
  }
}

// div_h, mo_divergence_operators.F90:16-68
template <class T>
__global__ void k_div_h(Dims D, Grid<T> G, const T* vx, const T* vy, T* out) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  auto fx = [&](int i, int j, int k) { return vx[IX(D, i, j, k)]; };
  auto fy = [&](int i, int j, int k) { return vy[IX(D, i, j, k)]; };
  out[IX(D, ji, jk, jl)] = div_h_at<T>(D, G, fx, fy, ji, jk, jl);
}

// inner_product of the wind with itself, mo_inner_product.F90:16-50
template <class T, class V = double>
__global__ void k_ke(Dims D, Grid<T> G, StateT<V> S, T* out) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  out[IX(D, ji, jk, jl)] = inner_product_at<T>(D, G, S.u, S.v, S.w, ji, jk, jl);
}

}  // namespace lg
