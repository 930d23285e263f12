// column_fp64.cu -- the vertically implicit part of the HEVI step, FP64 (compiled with
// -fmad=false: only the fma written out are fused).
//
// A block owns a tile of columns, numbered through the plane, and cuts them into chunks of levels:
// what can be formed level by level is (matrices, right-hand sides, new state), and only the
// Thomas algorithm (mo_column_solvers.F90:606-640) is sequential in the level index, one thread
// per column from shared memory.  (Parallel cyclic reduction would multiply the FP64 divisions by
// log2(n_layers), and FP64 throughput is the scarce resource of this GPU.)
#include "fp64.cuh"

namespace lg {

// (The products stay the hardware's here: with a few warps an SM between barriers these kernels wait
// on chains of operations, and mul_int's longer chain made them slower, 1980 against 1811 us and 1716
// against 1662 us at 192x192x80.)
constexpr int kMaxLayers = 128;

// three_band_solver_ver, mo_column_solvers.F90:21-351, plus the array-wide update of
// theta_v_pert (:346-349) and w_free_slip (mo_inner_product.F90:52-75) of this column,
// both of which only touch the column itself, with the reference's operations in its order.
//
// A block owns kCvCols columns and kCvChunks chunks of levels: every thread forms its chunk's rows
// (matrix and right-hand side) into shared memory, one thread a column runs the Thomas algorithm
// (mo_column_solvers.F90:606-640), every thread the new state of its chunk.  FP64 operations bound it
// on large grids: grid-only factors come from arrays formed once (ColumnGrid), the reciprocals of
// rho and of the interface density are formed once and divide by div_rn.  One thread per column with
// fourteen arrays in local memory took 788, 2116 us a launch at 65x97x33, 192x192x80; two blocks an SM 158,
// 1591 us; three (80 registers) 139, 1523 us.
constexpr int kCvCols = 16, kCvChunks = 16;
constexpr int kCvArrays = 7;  // c (then c of the row above), d, e (then e/den), r (then the solution), interface
                              // theta, gamma, 1/(interface density)

template <int RK>
__global__ void __launch_bounds__(kCvCols* kCvChunks, 3)
    k_column_ver(Dims D, Grid<double> G, ColumnGrid X, StateT<double> So, StateT<double> Sn, Tend<double> Tn) {
  extern __shared__ __align__(16) double sm_cv[];
    constexpr int S = kCvCols;
  const int lane = threadIdx.x % S, w = threadIdx.x / S;
  const int col = blockIdx.x * S + lane;
  const bool valid = col < D.ny * D.nx;
  const int ji = valid ? col % D.ny + 1 : 1, jk = valid ? col / D.ny + 1 : 1;
  const int nl = D.nl, n = nl - 1;
  const double dtime = D.dtime, rdt = X.rdt;
  const long long goff = (long long)(D.g - 1) * D.fstride, pl = D.plane, c0 = IX(D, ji, jk, 1);
  const StateT<double>& Su = (RK == 1) ? So : Sn;  // state_new_used
  const double* rho_o = So.rho + goff;
  const double* rho_u = Su.rho + goff;
  double* rho_n = Sn.rho + goff;
  const double* t_rho = Tn.rho + goff;
  const double pdw = 0.5;
  double* const sc = sm_cv + lane;               // row jl at S*(jl-1)
  double* const sd = sm_cv + S * nl + lane;
  double* const se = sm_cv + 2 * S * nl + lane;
  double* const sr = sm_cv + 3 * S * nl + lane;
  double* const st = sm_cv + 4 * S * nl + lane;
  double* const sg = sm_cv + 5 * S * nl + lane;  // layer jl
  double* const sy = sm_cv + 6 * S * nl + lane;
  const double c_imp2 = kIMPL_THERMO_WEIGHT * (dtime * dtime) * kC_D_P;

  // alpha, beta, gamma over the volume, theta of state_new_used, explicit predictions
  struct Lay { double al, be, ga, th, ro, rhe, tpe, epe, V, rV; };
  auto layer = [&](int jl, bool predict) {
    Lay L{};
    const long long i = c0 + (long long)(jl - 1) * pl;
    L.V = G.volume[i];
    L.rV = X.rvol[i];
    const double ro = rho_o[i], rto = So.rt[i];
    L.ro = ro;
    const double yo = rcp(ro);
    double alpha = div_rn(-rto, ro * ro, yo * yo), beta = yo;
    double gamma = quot(kR_D, kC_D_V * rto) * (G.exner_bg[i] + So.ep[i]);
    if (RK == 2) {
      const double ru = rho_u[i], rtu = Su.rt[i];
      const double yu = rcp(ru);
      const double alpha_new = div_rn(-rtu, ru * ru, yu * yu);
      const double gamma_new = quot(kR_D, kC_D_V * rtu) * (G.exner_bg[i] + Su.ep[i]);
      alpha = (1.0 - pdw) * alpha + pdw * alpha_new;
      beta = (1.0 - pdw) * beta + pdw * yu;
      gamma = (1.0 - pdw) * gamma + pdw * gamma_new;
      L.th = div_rn(rtu, ru, yu);
    } else {
      L.th = div_rn(rto, ro, yo);
    }
    L.al = div_rn(alpha, L.V, L.rV);
    L.be = div_rn(beta, L.V, L.rV);
    L.ga = div_rn(gamma, L.V, L.rV);
    if (predict) {
      const double tr = t_rho[i], trt = Tn.rt[i], dtv = dtime * L.V;
      L.rhe = ro + dtime * tr;
      L.tpe = So.tp[i] + dtv * (L.al * tr + L.be * trt);
      L.epe = So.ep[i] + dtv * L.ga * trt;
    }
    return L;
  };

  const int chunk = (n + kCvChunks - 1) / kCvChunks, r0 = w * chunk + 1, r1 = min(n, (w + 1) * chunk);
  if (valid && r0 <= r1) {
    Lay L0 = layer(r0, true), L1 = layer(r0 + 1, true), L2{};
    double rio = 0.5 * (L0.ro + L1.ro), yrio = rcp_near(rio);
    double t = 0.5 * (L0.th + L1.th);
    for (int jl = r0; jl <= r1; ++jl) {
      const long long b = c0 + (long long)jl * pl;  // layer jl+1 and w level jl+1
      const double zs = X.zs[b], hdeb = X.hdeb[b], dp = G.damp[b], wo = So.w[b];
      const double rie = 0.5 * (L0.rhe + L1.rhe);
      const double dv = -(t * t) * (L0.ga + L1.ga) + hdeb * (L1.al - L0.al + t * (L1.be - L0.be))
                      - div_rn(zs, c_imp2 * rio, X.rc_imp2 * yrio)
                      * (2.0 * X.raz[b] + dtime * wo * 0.5 * (-L0.rV + L1.rV)) * dp;
      // (0.5/dtime * (...) * d(exner_bg), with hdeb half that difference: powers of two are exact)
      const double rv = div_rn(-(wo + dtime * Tn.w[b]) * zs, c_imp2, X.rc_imp2)
                      + div_rn(t * (L0.epe - L1.epe), dtime, rdt)
                      + 2.0 * (0.5 / dtime) * (L0.tpe + L1.tpe) * hdeb
                      - div_rn(X.zs_c2[b] * wo * rie, rio, yrio);
      double cv = 0.0, ev = 0.0, rio_n = 0.0, yrio_n = 0.0, tn = 0.0;
      if (jl < n) {
        L2 = layer(jl + 2, jl < r1);
        const long long cc = b + pl;
        tn = 0.5 * (L1.th + L2.th);
        rio_n = 0.5 * (L1.ro + L2.ro);
        yrio_n = rcp_near(rio_n);
        cv = tn * L1.ga * t + X.hdeb[cc] * (L1.al + L1.be * t)
           - div_rn(X.zs_c1h[cc] * So.w[cc], L1.V * rio_n, L1.rV * yrio_n) * G.damp[cc];
        ev = t * L1.ga * tn - hdeb * (L1.al + L1.be * tn)
           + div_rn(X.zs_c1h[b] * wo, L1.V * rio, L1.rV * yrio) * dp;
      }
      sc[S * (jl - 1)] = cv;
      sd[S * (jl - 1)] = dv;
      se[S * (jl - 1)] = ev;
      sr[S * (jl - 1)] = rv;
      st[S * (jl - 1)] = t;
      sg[S * (jl - 1)] = L0.ga;
      if (jl == n) sg[S * n] = L1.ga;
      sy[S * (jl - 1)] = yrio;
      L0 = L1;
      L1 = L2;
      rio = rio_n;
      yrio = yrio_n;
      t = tn;
    }
  }
  __syncthreads();
  if (valid && w == 0) {
    double y = rcp_near(sd[0]);
    double ep = div_rn(se[0], sd[0], y), rp = div_rn(sr[0], sd[0], y);
    se[0] = ep;
    sr[0] = rp;
#pragma unroll 2
    for (int jl = 2; jl <= n; ++jl) {
      const double c = sc[S * (jl - 2)];
      const double den = sd[S * (jl - 1)] - ep * c;
      y = rcp_near(den);
      ep = div_rn(se[S * (jl - 1)], den, y);  // (0 in the last row)
      rp = div_rn(sr[S * (jl - 1)] - rp * c, den, y);
      se[S * (jl - 1)] = ep;
      sr[S * (jl - 1)] = rp;
    }
#pragma unroll 4
    for (int jl = n - 1; jl >= 1; --jl) {
      rp = sr[S * (jl - 1)] - se[S * (jl - 1)] * rp;
      sr[S * (jl - 1)] = rp;
    }
  }
  __syncthreads();
  const int lchunk = (nl + kCvChunks - 1) / kCvChunks, l0 = w * lchunk + 1, l1 = min(nl, (w + 1) * lchunk);
  if (!valid || l0 > l1) return;
  auto new_rho = [&](int jl, double V, double rV) {
    const long long i = c0 + (long long)(jl - 1) * pl;
    const double rhe = rho_o[i] + dtime * t_rho[i];
    if (jl == 1) return rhe + div_rn(dtime * sr[0], V, rV);
    if (jl == nl) return rhe - div_rn(dtime * sr[S * (n - 1)], V, rV);
    return rhe + div_rn(dtime * (-sr[S * (jl - 2)] + sr[S * (jl - 1)]), V, rV);
  };
  double rn_up = 0.0, ro_up = 0.0;
  if (l0 > 1) {
    const long long a = c0 + (long long)(l0 - 2) * pl;
    rn_up = new_rho(l0 - 1, G.volume[a], X.rvol[a]);
    ro_up = rho_o[a];
  }
  for (int jl = l0; jl <= l1; ++jl) {
    const long long i = c0 + (long long)(jl - 1) * pl;
    const double V = G.volume[i], rV = X.rvol[i], rto = So.rt[i], ro = rho_o[i];
    const double rn = new_rho(jl, V, rV);
    const double rte = rto + dtime * Tn.rt[i];
    double rtn;
    if (jl == 1) rtn = rte + div_rn(dtime * st[0] * sr[0], V, rV);
    else if (jl == nl) rtn = rte - div_rn(dtime * st[S * (n - 1)] * sr[S * (n - 1)], V, rV);
    else rtn = rte + div_rn(dtime * (-(st[S * (jl - 2)] * sr[S * (jl - 2)]) + st[S * (jl - 1)] * sr[S * (jl - 1)]), V, rV);
    const double epn = So.ep[i] + V * sg[S * (jl - 1)] * (rtn - rto);
    const double tpn = quot(rtn, rn) - G.theta_v_bg[i];
    if (jl >= 2) {
      const double rin = 0.5 * (rn_up + rn);
      Sn.w[i] = div_rn(div_rn(2.0 * sr[S * (jl - 2)], G.area_z[i], X.raz[i]) - rin * So.w[i], 0.5 * (ro_up + ro),
                       sy[S * (jl - 2)]);
    }
    rho_n[i] = rn;
    Sn.rt[i] = rtn;
    Sn.ep[i] = epn;
    Sn.tp[i] = tpn;
    rn_up = rn;
    ro_up = ro;
  }
  if (D.freeslip && l1 == nl) {
    Sn.w[IX(D, ji, jk, nl + 1)] =
        W_(1, ji, jk, nl) * Sn.u[IX(D, ji, jk + 1, nl)] * G.slope_x[IX(D, ji, jk + 1, nl)]
      + W_(2, ji, jk, nl) * Sn.v[IX(D, ji, jk, nl)] * G.slope_y[IX(D, ji, jk, nl)]
      + W_(3, ji, jk, nl) * Sn.u[IX(D, ji, jk, nl)] * G.slope_x[IX(D, ji, jk, nl)]
      + W_(4, ji, jk, nl) * Sn.v[IX(D, ji + 1, jk, nl)] * G.slope_y[IX(D, ji + 1, jk, nl)];
  }
}

// the grid-only factors of the vertical solve, at w level jl = 2..nl (index of layer jl) and, the
// reciprocal of the volume, at every layer
__global__ void k_column_grid(Dims D, Grid<double> G, double* rvol, double* itwdtv, double* zs, double* zs_c2,
                              double* zs_c1h, double* hdeb, double* raz) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl), a = q - D.plane;
  rvol[q] = 1.0 / G.volume[q];
  itwdtv[q] = 0.5 * D.dtime / G.volume[q];
  if (jl == 1) return;
  const double c_imp2 = kIMPL_THERMO_WEIGHT * (D.dtime * D.dtime) * kC_D_P;
  const double c_imp1 = kIMPL_THERMO_WEIGHT * D.dtime * kC_D_P;
  const double z = G.z_scalar[a] - G.z_scalar[q];
  zs[q] = z;
  zs_c2[q] = z / c_imp2;
  zs_c1h[q] = z / c_imp1 * 0.5;
  hdeb[q] = 0.5 * (G.exner_bg[a] - G.exner_bg[q]);
  raz[q] = 1.0 / G.area_z[q];
}

void launch_column_grid(const Dims& D, const Grid<double>& G, double* rvol, double* itwdtv, double* zs, double* zs_c2,
                        double* zs_c1h, double* hdeb, double* raz, cudaStream_t st) {
  const dim3 g((unsigned)((D.ny + 31) / 32), (unsigned)D.nl, (unsigned)((D.nx + 7) / 8));
  k_column_grid<<<g, dim3(32, 8), 0, st>>>(D, G, rvol, itwdtv, zs, zs_c2, zs_c1h, hdeb, raz);
}

void launch_column_ver(const Dims& D, const Grid<double>& G, const ColumnGrid& X, const State& So, const State& Sn,
                       const Tend<double>& Tn, int rk_step, cudaStream_t st) {
  const unsigned nb = (unsigned)(((long long)D.ny * D.nx + kCvCols - 1) / kCvCols);
  const size_t sm = (size_t)kCvArrays * kCvCols * D.nl * sizeof(double);
  if (rk_step == 1) k_column_ver<1><<<nb, kCvCols * kCvChunks, sm, st>>>(D, G, X, So, Sn, Tn);
  else k_column_ver<2><<<nb, kCvCols * kCvChunks, sm, st>>>(D, G, X, So, Sn, Tn);
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
// its arrays in local memory took 1530, 4887 us a launch at 65x97x33, 192x192x80; two blocks an SM 187, 1772 us; three (80 registers) 138,
// 1571 us.
constexpr int kTcCols = 16, kTcChunks = 16;
constexpr int kTcArrays = 6;  // k, d, 1/d, right-hand sides of up to three tracers

template <int GROUP>
struct TracerGroup {
  __device__ static constexpr int n() { return GROUP == 1 ? 3 : 1; }
  __device__ static constexpr int jc(int q) { return GROUP == 0 ? 1 : GROUP == 2 ? 3 : GROUP == 3 ? 4 : q == 0 ? 2 : q == 1 ? 5 : 7; }
  __device__ static constexpr bool cond(int q) { return jc(q) <= 5; }
  __device__ static constexpr bool ice(int q) { return (jc(q) - 1) % 2 == 0; }
  __device__ static constexpr bool sfc_heat(int q) { return jc(q) > 1; }  // jc > nc/4: not snow
};

// one group of tracers of the block's columns; HEAT: the first substep, which forms the sediment
// heating (the sum over the condensates in their order, in csh; graupel's part waits in hx)
template <int GROUP, bool HEAT>
__device__ __forceinline__ void tracer_group(const Dims& D, const Grid<double>& G, const StateT<double>& So, const StateT<double>& Sn,
                                             const double* t_rho_all, const double* T, const double* rvol,
                                             const double* itwdtv, const double* vcloud, const double* cpi,
                                             const double* cpw, double* csh, double* hx, int ji, int jk, bool valid, int lane, int w,
                                             double* sm) {
  using TG = TracerGroup<GROUP>;
  constexpr int N = TG::n(), S = kTcCols;
  const int nl = D.nl;
  const long long pl = D.plane, c0 = IX(D, ji, jk, 1);
  double* const sk = sm + lane;               // coupling of the interface below row jl at sk[S*(jl-1)]
  double* const sd = sm + S * nl + lane;      // diagonal
  double* const sy = sm + 2 * S * nl + lane;  // its reciprocal
  double* const sr = sm + 3 * S * nl + lane;  // right-hand side, then the solution: tracer q at + q*S*nl
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
      const double y = rcp_near(d);
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
          if (TG::jc(q) == 1) csh[i] = h;
          else if (TG::jc(q) == 5) hx[i] = h;  // its surface term is 0 (no fall speed)
          else if (TG::jc(q) == 4) csh[i] = ((csh[i] + h) - h2) + hx[i];
          else csh[i] = (csh[i] + h) - h2;
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
__global__ void __launch_bounds__(kTcCols* kTcChunks, 3)
    k_column_tracers(Dims D, Grid<double> G, StateT<double> So, StateT<double> Sn, const double* t_rho_all, const double* T,
                     const double* rvol, const double* itwdtv, const double* vcloud, const double* cpi, const double* cpw,
                     double* csh, double* hx) {
  extern __shared__ __align__(16) double sm_tc[];
  const int lane = threadIdx.x % kTcCols, w = threadIdx.x / kTcCols;
  const int col = blockIdx.x * kTcCols + lane;
  const bool valid = col < D.ny * D.nx;
  const int ji = valid ? col % D.ny + 1 : 1, jk = valid ? col / D.ny + 1 : 1;
#define TC_GROUP(g) \
  tracer_group<g, HEAT>(D, G, So, Sn, t_rho_all, T, rvol, itwdtv, vcloud, cpi, cpw, csh, hx, ji, jk, valid, lane, w, sm_tc)
  TC_GROUP(0);
  TC_GROUP(1);
  TC_GROUP(2);
  TC_GROUP(3);
#undef TC_GROUP
}

int column_prepare() {
  for (auto k : {k_column_ver<1>, k_column_ver<2>})
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kCvArrays * kCvCols * kMaxLayers * (int)sizeof(double)) != cudaSuccess)
      return 1;
  for (auto k : {k_column_tracers<true>, k_column_tracers<false>})
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             kTcArrays * kTcCols * kMaxLayers * (int)sizeof(double)) != cudaSuccess)
      return 1;
  return 0;
}

void launch_column_tracers(const Dims& D, const Grid<double>& G, const State& So, const State& Sn, const double* t_rho,
                           const double* T, const double* rvol, const double* itwdtv, const double* vcloud,
                           const double* cpi, const double* cpw, double* csh, double* hx, int rk_step, cudaStream_t st) {
  const unsigned nb = (unsigned)(((long long)D.ny * D.nx + kTcCols - 1) / kTcCols);
  const dim3 b(kTcCols * kTcChunks);
  const size_t sm = (size_t)kTcArrays * kTcCols * D.nl * sizeof(double);
  if (rk_step == 1)
    k_column_tracers<true><<<nb, b, sm, st>>>(D, G, So, Sn, t_rho, T, rvol, itwdtv, vcloud, cpi, cpw, csh, hx);
  else
    k_column_tracers<false><<<nb, b, sm, st>>>(D, G, So, Sn, t_rho, T, rvol, itwdtv, vcloud, cpi, cpw, csh, hx);
}

}  // namespace lg
