// column_fp64.cu -- the vertically implicit part of the HEVI step, FP64, one thread per
// column (compiled with -fmad=false).
//
// A warp owns 32 adjacent columns of one x-row, so every level load of every field is
// one coalesced 256-byte access.  Each thread runs the Thomas algorithm of its column
// (mo_column_solvers.F90:606-640); the forward sweep and the back substitution are
// sequential in the level index, which is why the work is spread over the ~10^6
// columns of the domain instead of over the levels (parallel cyclic reduction would
// multiply the FP64 divisions by log2(n_layers), and FP64 throughput is the scarce
// resource of this GPU).
#include "kernels.cuh"

namespace lg {

constexpr int kMaxLayers = 128;

// a/b rounded to nearest for y = 1/b rounded to nearest: quotient, exact remainder, correction
// (Markstein, IBM J. Res. Dev. 34, 1990): three FP64-pipe operations instead of about seven.  The
// result is the correctly rounded quotient, except that a quotient within 2^-52 of its last place
// from the middle of two doubles may round the other way; a zero quotient's sign is not kept, and
// an infinite a gives NaN.
__device__ __forceinline__ double div_rn(double a, double b, double y) {
  const double q = a * y;
  return fma(fma(-b, q, a), y, q);
}

// the Thomas algorithm of mo_column_solvers.F90:606-640 (arrays 1-based)
__device__ __forceinline__ void thomas(const double* c, const double* d, const double* e, const double* r,
                                       double* sol, double* ep, double* rp, int n) {
  ep[1] = e[1] / d[1];
  rp[1] = r[1] / d[1];
  for (int jl = 2; jl <= n; ++jl) {
    const double den = d[jl] - ep[jl - 1] * c[jl - 1];
    if (jl <= n - 1) ep[jl] = e[jl] / den;
    rp[jl] = (r[jl] - rp[jl - 1] * c[jl - 1]) / den;
  }
  sol[n] = rp[n];
  for (int jl = n - 1; jl >= 1; --jl) sol[jl] = rp[jl] - ep[jl] * sol[jl + 1];
}

// three_band_solver_ver, mo_column_solvers.F90:21-351, plus the array-wide update of
// theta_v_pert (:346-349) and w_free_slip (mo_inner_product.F90:52-75) of this column,
// both of which only touch the column itself.
__global__ void k_column_ver(Dims D, Grid<double> G, State So, State Sn, Tend<double> Tn, int rk_step) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const int nl = D.nl;
  const double dtime = D.dtime;
  const long long goff = (long long)(D.g - 1) * D.fstride;
  const State& Su = (rk_step == 1) ? So : Sn;  // state_new_used
  const double* rho_o = So.rho + goff;
  const double* rho_u = Su.rho + goff;
  double* rho_n = Sn.rho + goff;
  const double* t_rho = Tn.rho + goff;
  const double pdw = 0.5;

  double alpha[kMaxLayers + 1], beta[kMaxLayers + 1], gammaa[kMaxLayers + 1];
  double rho_expl[kMaxLayers + 1], rt_expl[kMaxLayers + 1], ep_expl[kMaxLayers + 1], tp_expl[kMaxLayers + 1];
  double rio[kMaxLayers + 1], rie[kMaxLayers + 1], ti[kMaxLayers + 1];
  double cv[kMaxLayers + 1], dv[kMaxLayers + 1], evec[kMaxLayers + 1], rv[kMaxLayers + 1];
  double sol[kMaxLayers + 1], epr[kMaxLayers + 1], rpr[kMaxLayers + 1];

  for (int jl = 1; jl <= nl; ++jl) {
    const long long i = IX(D, ji, jk, jl);
    const double V = G.volume[i];
    rho_expl[jl] = rho_o[i] + dtime * t_rho[i];
    rt_expl[jl] = So.rt[i] + dtime * Tn.rt[i];
    if (rk_step == 1) {
      alpha[jl] = -So.rt[i] / (rho_o[i] * rho_o[i]) / V;
      beta[jl] = 1.0 / rho_o[i] / V;
      gammaa[jl] = kR_D / (kC_D_V * So.rt[i]) * (G.exner_bg[i] + So.ep[i]) / V;
    } else {
      const double alpha_old = -So.rt[i] / (rho_o[i] * rho_o[i]);
      const double beta_old = 1.0 / rho_o[i];
      const double gamma_old = kR_D / (kC_D_V * So.rt[i]) * (G.exner_bg[i] + So.ep[i]);
      const double alpha_new = -Su.rt[i] / (rho_u[i] * rho_u[i]);
      const double beta_new = 1.0 / rho_u[i];
      const double gamma_new = kR_D / (kC_D_V * Su.rt[i]) * (G.exner_bg[i] + Su.ep[i]);
      alpha[jl] = ((1.0 - pdw) * alpha_old + pdw * alpha_new) / V;
      beta[jl] = ((1.0 - pdw) * beta_old + pdw * beta_new) / V;
      gammaa[jl] = ((1.0 - pdw) * gamma_old + pdw * gamma_new) / V;
    }
    tp_expl[jl] = So.tp[i] + dtime * V * (alpha[jl] * t_rho[i] + beta[jl] * Tn.rt[i]);
    ep_expl[jl] = So.ep[i] + dtime * V * gammaa[jl] * Tn.rt[i];
  }
  for (int jl = 1; jl <= nl - 1; ++jl) {
    const long long a = IX(D, ji, jk, jl), b = IX(D, ji, jk, jl + 1);
    rio[jl] = 0.5 * (rho_o[a] + rho_o[b]);
    rie[jl] = 0.5 * (rho_expl[jl] + rho_expl[jl + 1]);
    ti[jl] = 0.5 * (Su.rt[a] / rho_u[a] + Su.rt[b] / rho_u[b]);
  }
  const double c_imp2 = kIMPL_THERMO_WEIGHT * (dtime * dtime) * kC_D_P;
  const double c_imp1 = kIMPL_THERMO_WEIGHT * dtime * kC_D_P;
  for (int jl = 1; jl <= nl - 1; ++jl) {
    const long long a = IX(D, ji, jk, jl), b = IX(D, ji, jk, jl + 1);
    const double zs0 = G.z_scalar[a], zs1 = G.z_scalar[b];
    const double eb0 = G.exner_bg[a], eb1 = G.exner_bg[b];
    const double dp = G.damp[b];  // prefactor at level jl+1
    const double wo = So.w[b];
    const double t = ti[jl];
    dv[jl] = -(t * t) * (gammaa[jl] + gammaa[jl + 1])
           + 0.5 * (eb0 - eb1) * (alpha[jl + 1] - alpha[jl] + t * (beta[jl + 1] - beta[jl]))
           - (zs0 - zs1) / (c_imp2 * rio[jl])
           * (2.0 / G.area_z[b] + dtime * wo * 0.5 * (-1.0 / G.volume[a] + 1.0 / G.volume[b])) * dp;
    rv[jl] = -(wo + dtime * Tn.w[b]) * (zs0 - zs1) / c_imp2
           + t * (ep_expl[jl] - ep_expl[jl + 1]) / dtime
           + 0.5 / dtime * (tp_expl[jl] + tp_expl[jl + 1]) * (eb0 - eb1)
           - (zs0 - zs1) / c_imp2 * wo * rie[jl] / rio[jl];
  }
  for (int jl = 1; jl <= nl - 2; ++jl) {
    const long long a = IX(D, ji, jk, jl), b = IX(D, ji, jk, jl + 1), c = IX(D, ji, jk, jl + 2);
    cv[jl] = ti[jl + 1] * gammaa[jl + 1] * ti[jl]
           + 0.5 * (G.exner_bg[b] - G.exner_bg[c]) * (alpha[jl + 1] + beta[jl + 1] * ti[jl])
           - (G.z_scalar[b] - G.z_scalar[c]) / c_imp1 * 0.5 * So.w[c] / (G.volume[b] * rio[jl + 1]) * G.damp[c];
    evec[jl] = ti[jl] * gammaa[jl + 1] * ti[jl + 1]
             - 0.5 * (G.exner_bg[a] - G.exner_bg[b]) * (alpha[jl + 1] + beta[jl + 1] * ti[jl + 1])
             + (G.z_scalar[a] - G.z_scalar[b]) / c_imp1 * 0.5 * So.w[b] / (G.volume[b] * rio[jl]) * G.damp[b];
  }
  thomas(cv, dv, evec, rv, sol, epr, rpr, nl - 1);
  for (int jl = 2; jl <= nl - 1; ++jl) {
    const long long i = IX(D, ji, jk, jl);
    rho_n[i] = rho_expl[jl] + dtime * (-sol[jl - 1] + sol[jl]) / G.volume[i];
    Sn.rt[i] = rt_expl[jl] + dtime * (-(ti[jl - 1] * sol[jl - 1]) + ti[jl] * sol[jl]) / G.volume[i];
  }
  {
    const long long i1 = IX(D, ji, jk, 1), iN = IX(D, ji, jk, nl);
    rho_n[i1] = rho_expl[1] + dtime * sol[1] / G.volume[i1];
    Sn.rt[i1] = rt_expl[1] + dtime * ti[1] * sol[1] / G.volume[i1];
    rho_n[iN] = rho_expl[nl] - dtime * sol[nl - 1] / G.volume[iN];
    Sn.rt[iN] = rt_expl[nl] - dtime * ti[nl - 1] * sol[nl - 1] / G.volume[iN];
  }
  for (int jl = 2; jl <= nl; ++jl) {
    const long long i = IX(D, ji, jk, jl);
    const double rin = 0.5 * (rho_n[IX(D, ji, jk, jl - 1)] + rho_n[i]);
    Sn.w[i] = (2.0 * sol[jl - 1] / G.area_z[i] - rin * So.w[i]) / rio[jl - 1];
  }
  for (int jl = 1; jl <= nl; ++jl) {
    const long long i = IX(D, ji, jk, jl);
    Sn.ep[i] = So.ep[i] + G.volume[i] * gammaa[jl] * (Sn.rt[i] - So.rt[i]);
    Sn.tp[i] = Sn.rt[i] / rho_n[i] - G.theta_v_bg[i];
  }
  if (D.freeslip) {
    const int n = nl;
    Sn.w[IX(D, ji, jk, n + 1)] =
        W_(1, ji, jk, n) * Sn.u[IX(D, ji, jk + 1, n)] * G.slope_x[IX(D, ji, jk + 1, n)]
      + W_(2, ji, jk, n) * Sn.v[IX(D, ji, jk, n)] * G.slope_y[IX(D, ji, jk, n)]
      + W_(3, ji, jk, n) * Sn.u[IX(D, ji, jk, n)] * G.slope_x[IX(D, ji, jk, n)]
      + W_(4, ji, jk, n) * Sn.v[IX(D, ji + 1, jk, n)] * G.slope_y[IX(D, ji + 1, jk, n)];
  }
}

// x < 0 by the bits (a comparison issues on the FP64 pipe); -0 counts as negative, NaN does not
__device__ __forceinline__ bool negative(double x) {
  const unsigned u = (unsigned)__double2hiint(x) - 0x80000000u;
  return u < 0x7FF00000u || (u == 0x7FF00000u && __double2loint(x) == 0);
}

// v_fall_liquid, mo_derived.F90:218-263 (state_old, diag%temperature)
__device__ __forceinline__ double v_fall_liquid(const Dims& D, const Grid<double>& G, const double* rho_g,
                                                const double* T, double radius, int ji, int jk, int jl) {
  double g;
  if (jl == 1) g = G.gm[IX(D, ji, jk, jl + 1)];
  else if (jl == D.nl) g = G.gm[IX(D, ji, jk, jl)];
  else g = W_(5, ji, jk, jl) * G.gm[IX(D, ji, jk, jl)] + W_(6, ji, jk, jl) * G.gm[IX(D, ji, jk, jl + 1)];
  const long long i = IX(D, ji, jk, jl);
  const double rg = rho_g[i];
  const double nu = calc_diff_coeff(T[i], rg);
  double v = 2.0 * (radius * radius) * (kRHO_H2O - rg) * g / (9.0 * rg * nu);
  const double re = v * radius / nu;
  if (re > 10.0) v = sqrt(8.0 * radius * kRHO_H2O * g / (3.0 * rg * 0.8));
  return v;
}

// v_fall_solid, mo_derived.F90:265-283 (threshold is the default-real literal 250.e-6)
__device__ __forceinline__ double v_fall_solid(double radius) {
  return (radius > (double)250.e-6f) ? 1.0 : 0.001;
}

// The quantities of a level that depend only on state_old and its temperature, formed once per
// step: the cloud droplets' fall speed, read by both substeps' tracer solves, and c_p of ice and
// water, read by the sediment heating and by both substeps' diabatic term (gas_theta).
__global__ void k_moist_aux(Dims D, Grid<double> G, State So, const double* T, double* vcloud, double* cpi, double* cpw) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl);
  const double cloud_r = 12.e-6;  // mo_dictionary.F90:276-318
  vcloud[q] = v_fall_liquid(D, G, So.rho + (long long)(D.g - 1) * D.fstride, T, cloud_r, ji, jk, jl);
  cpi[q] = c_p_ice(T[q]);
  cpw[q] = c_p_water(T[q]);
}

// three_band_solver_gen_densities, mo_column_solvers.F90:353-604, with the reference's operations
// in its order (the results are the reference's bits; divisions as div_rn).
//
// The upwind fluxes couple each interface's two cells in one direction only: of the coefficients
// e(jl) and c(jl) one is zero.  So the eliminated diagonal is the diagonal itself, and one number
// per interface holds both couplings: k >= 0 is -e/d (the row above couples down), k < 0 is c (the
// row below couples up).  Rain, graupel and vapour have no fall speed (their radius diag%a_rain is
// never set) and share one matrix.
//
// FP64 operations bound this kernel on large grids and chains of levels on small ones.  A block
// owns kTcCols columns and kTcChunks chunks of levels and takes the tracers in four groups of one
// matrix each (snow; rain, graupel, vapour; cloud ice; cloud water), in three phases a group: every
// thread forms its chunk's rows into shared memory, one thread per column and tracer runs the two
// sweeps, every thread clips and stores its chunk.  The level's own quantities come from k_moist_aux
// and from the grid (the reciprocal of the volume and itw*dtime/volume).  One thread per column with
// its arrays in local memory took 1530, 4887 us a launch at 65x97x33, 192x192x80; this 199, 1814 us.
constexpr int kTcCols = 16, kTcChunks = 16;
constexpr int kTcArrays = 8;  // k, d, 1/d, right-hand sides of up to three tracers, two heating sums (first substep)

template <int GROUP>
struct TracerGroup {
  __device__ static constexpr int n() { return GROUP == 1 ? 3 : 1; }
  __device__ static constexpr int jc(int q) { return GROUP == 0 ? 1 : GROUP == 2 ? 3 : GROUP == 3 ? 4 : q == 0 ? 2 : q == 1 ? 5 : 7; }
  __device__ static constexpr bool cond(int q) { return jc(q) <= 5; }
  __device__ static constexpr bool ice(int q) { return (jc(q) - 1) % 2 == 0; }
  __device__ static constexpr bool sfc_heat(int q) { return jc(q) > 1; }  // jc > nc/4: not snow
};

// one group of tracers of the block's columns; HEAT: the first substep, which forms the sediment
// heating (the sums over the condensates in their order, in hs; graupel's part waits in hx)
template <int GROUP, bool HEAT>
__device__ __forceinline__ void tracer_group(const Dims& D, const Grid<double>& G, const State& So, const State& Sn,
                                             const double* t_rho_all, const double* T, const double* rvol,
                                             const double* itwdtv, const double* vcloud, const double* cpi,
                                             const double* cpw, double* csh, int ji, int jk, bool valid, int lane, int w,
                                             double* sm) {
  using TG = TracerGroup<GROUP>;
  constexpr int N = TG::n(), S = kTcCols;
  const int nl = D.nl;
  const long long pl = D.plane, c0 = IX(D, ji, jk, 1);
  double* const sk = sm + lane;               // coupling of the interface below row jl at sk[S*(jl-1)]
  double* const sd = sm + S * nl + lane;      // diagonal
  double* const sy = sm + 2 * S * nl + lane;  // its reciprocal
  double* const sr = sm + 3 * S * nl + lane;  // right-hand side, then the solution: tracer q at + q*S*nl
  double* const hs = sm + 6 * S * nl + lane;
  double* const hx = sm + 7 * S * nl + lane;
  const double dtime = D.dtime;
  const double itw = 0.5, expl_weight = 1.0 - itw;
  const double ewdt = expl_weight * dtime;
  const int chunk = (nl + kTcChunks - 1) / kTcChunks, l0 = w * chunk + 1, l1 = min(nl, (w + 1) * chunk);
  const double vfix = GROUP == 0 ? v_fall_solid(500.e-6) : GROUP == 2 ? v_fall_solid(95.e-6) : 0.0;
  if (valid && l0 <= l1) {
    // interface between levels m and m+1: w point m+1
    struct Iface { double vfi, p0, p1, fr[N], ve[N]; };
    auto iface = [&](int m, const double* ro_a, const double* ro_b, double itwa, double itwb) {
      Iface f;
      const long long b = c0 + (long long)m * pl;
      double wo = So.w[b], wn = Sn.w[b];
      if (GROUP != 1) {
        const double vf = GROUP == 3 ? 0.5 * (vcloud[b - pl] + vcloud[b]) : vfix;
        wo = wo - vf;
        wn = wn - vf;
      }
      const double az = G.area_z[b];
      f.vfi = az * wo;
      const double vfr = az * wn;
      f.p0 = itwa * f.vfi;
      f.p1 = itwb * f.vfi;
      double cti = 0.0, ctw = 0.0;
      if (HEAT) {
        if (GROUP != 3) cti = cpi[b] * T[b];
        if (GROUP == 1 || GROUP == 3) ctw = cpw[b] * T[b];
      }
#pragma unroll
      for (int q = 0; q < N; ++q) {
        f.fr[q] = (negative(vfr) ? ro_a[q] : ro_b[q]) * vfr;
        f.ve[q] = (HEAT && TG::cond(q)) ? (TG::ice(q) ? cti : ctw) * f.fr[q] : 0.0;
      }
      return f;
    };
    auto load_rho = [&](int m, double* r) {
#pragma unroll
      for (int q = 0; q < N; ++q) r[q] = So.rho[c0 + (long long)(m - 1) * pl + (long long)(TG::jc(q) - 1) * D.fstride];
    };
    double ro[N], ro_n[N];
    load_rho(l0, ro);
    double itw_c = itwdtv[c0 + (long long)(l0 - 1) * pl];
    Iface up{}, dn{};
    if (l0 > 1) {
      double ro_u[N];
      load_rho(l0 - 1, ro_u);
      up = iface(l0 - 1, ro_u, ro, itwdtv[c0 + (long long)(l0 - 2) * pl], itw_c);
    }
    for (int jl = l0; jl <= l1; ++jl) {
      const long long i = c0 + (long long)(jl - 1) * pl;
      const double V = G.volume[i], rV = rvol[i];
      double itw_n = 0.0;
      if (jl < nl) {
        load_rho(jl + 1, ro_n);
        itw_n = itwdtv[i + pl];
        dn = iface(jl, ro, ro_n, itw_c, itw_n);
      }
      const double az_sfc = (jl == nl) ? G.area_z[i + pl] : 0.0;
      const double v_sfc = GROUP == 3 ? ((jl == nl) ? vcloud[i] : 0.0) : vfix;
      double d = 1.0;
      if (jl > 1 && !negative(up.vfi)) d = d + up.p1;
      if (jl < nl && negative(dn.vfi)) d = d - dn.p0;
      if (jl == nl && TG::cond(0) && GROUP != 1) d = d + div_rn(itw * v_sfc * dtime * az_sfc, V, rV);
      const double y = __drcp_rn(d);
      sd[S * (jl - 1)] = d;
      sy[S * (jl - 1)] = y;
      // (written as -e/d: e = -(itwdtv*vfi), so k = (itwdtv*vfi)/d)
      if (jl < nl) sk[S * (jl - 1)] = negative(dn.vfi) ? dn.p1 : div_rn(dn.p0, d, y);
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const double tr = t_rho_all[i + (long long)(TG::jc(q) - 1) * D.fstride];
        double r = ro[q] + dtime * tr;
        double h = 0.0, h2 = 0.0;
        if (jl == 1) {
          r = r + div_rn(ewdt * dn.fr[q], V, rV);
          if (HEAT && TG::cond(q)) h = div_rn(dn.ve[q], V, rV);
        } else if (jl == nl) {
          r = r - div_rn(ewdt * up.fr[q], V, rV);
          if (HEAT && TG::cond(q)) h = -div_rn(up.ve[q], V, rV);
          if (TG::cond(q) && GROUP != 1) {
            r = r - div_rn(expl_weight * v_sfc * dtime * ro[q] * az_sfc, V, rV);
            if (HEAT && TG::sfc_heat(q))
              h2 = div_rn(v_sfc * T[i] * (TG::ice(q) ? cpi[i] : cpw[i]) * ro[q] * az_sfc, V, rV);
          }
        } else {
          r = r + div_rn(ewdt * (-up.fr[q] + dn.fr[q]), V, rV);
          if (HEAT && TG::cond(q)) h = div_rn(-up.ve[q] + dn.ve[q], V, rV);
        }
        sr[S * (nl * q + jl - 1)] = r;
        if (HEAT && TG::cond(q)) {  // (the thread is the only one to touch its levels' sums)
          if (TG::jc(q) == 1) hs[S * (jl - 1)] = h;
          else if (TG::jc(q) == 5) hx[S * (jl - 1)] = h;  // its surface term is 0 (no fall speed)
          else {
            const double s = (hs[S * (jl - 1)] + h) - h2;
            if (TG::jc(q) == 4) csh[i] = s + hx[S * (jl - 1)];
            else hs[S * (jl - 1)] = s;
          }
        }
        ro[q] = ro_n[q];
      }
      itw_c = itw_n;
      up = dn;
    }
  }
  __syncthreads();
  // the two sweeps (mo_column_solvers.F90:606-640), a thread per column and tracer
  if (valid && w < N) {
    double* const r = sr + S * nl * w;
    double rp = r[0] = div_rn(r[0], sd[0], sy[0]);
#pragma unroll 4
    for (int jl = 2; jl <= nl; ++jl) {
      const double k = sk[S * (jl - 2)];
      const double x = negative(k) ? r[S * (jl - 1)] - rp * k : r[S * (jl - 1)];
      rp = div_rn(x, sd[S * (jl - 1)], sy[S * (jl - 1)]);
      r[S * (jl - 1)] = rp;
    }
#pragma unroll 4
    for (int jl = nl - 1; jl >= 1; --jl) {
      const double k = sk[S * (jl - 1)];
      rp = negative(k) ? r[S * (jl - 1)] : r[S * (jl - 1)] + k * rp;
      r[S * (jl - 1)] = rp;
    }
  }
  __syncthreads();
  if (valid)
    for (int jl = l0; jl <= l1; ++jl)
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const double s = sr[S * (nl * q + jl - 1)];
        Sn.rho[c0 + (long long)(jl - 1) * pl + (long long)(TG::jc(q) - 1) * D.fstride] = negative(s) ? 0.0 : s;
      }
  __syncthreads();  // the next group overwrites the arrays
}

template <bool HEAT>
__global__ void __launch_bounds__(kTcCols* kTcChunks, 2)
    k_column_tracers(Dims D, Grid<double> G, State So, State Sn, const double* t_rho_all, const double* T,
                     const double* rvol, const double* itwdtv, const double* vcloud, const double* cpi, const double* cpw,
                     double* csh) {
  extern __shared__ __align__(16) double sm_tc[];
  const int lane = threadIdx.x % kTcCols, w = threadIdx.x / kTcCols;
  const int col = blockIdx.x * kTcCols + lane;
  const bool valid = col < D.ny * D.nx;
  const int ji = valid ? col % D.ny + 1 : 1, jk = valid ? col / D.ny + 1 : 1;
#define TC_GROUP(g) \
  tracer_group<g, HEAT>(D, G, So, Sn, t_rho_all, T, rvol, itwdtv, vcloud, cpi, cpw, csh, ji, jk, valid, lane, w, sm_tc)
  TC_GROUP(0);
  TC_GROUP(1);
  TC_GROUP(2);
  TC_GROUP(3);
#undef TC_GROUP
}

int column_tracers_prepare() {
  for (auto k : {k_column_tracers<true>, k_column_tracers<false>})
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kTcArrays * kTcCols * kMaxLayers * (int)sizeof(double)) != cudaSuccess)
      return 1;
  return 0;
}

void launch_column_tracers(const Dims& D, const Grid<double>& G, const State& So, const State& Sn, const double* t_rho,
                           const double* T, const double* rvol, const double* itwdtv, const double* vcloud,
                           const double* cpi, const double* cpw, double* csh, int rk_step, cudaStream_t st) {
  const unsigned nb = (unsigned)(((long long)D.ny * D.nx + kTcCols - 1) / kTcCols);
  const dim3 b(kTcCols * kTcChunks);
  // the second substep keeps no heating sums
  const size_t lev = (size_t)kTcCols * D.nl * sizeof(double);
  if (rk_step == 1)
    k_column_tracers<true><<<nb, b, 8 * lev, st>>>(D, G, So, Sn, t_rho, T, rvol, itwdtv, vcloud, cpi, cpw, csh);
  else
    k_column_tracers<false><<<nb, b, 6 * lev, st>>>(D, G, So, Sn, t_rho, T, rvol, itwdtv, vcloud, cpi, cpw, csh);
}

}  // namespace lg
