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
constexpr int kCvArrays = 7;  // c, d, e (then e/den), r (then the solution), interface theta, gamma,
                              // 1/(interface density)

template <int RK>
__global__ void __launch_bounds__(kCvCols* kCvChunks, 3)
    k_column_ver(Dims D, Grid<F64> G, ColumnGrid X, StateT<F64> So, StateT<F64> Sn, Tend<F64> Tn) {
  extern __shared__ __align__(16) double sm_raw[];
  F64* const sm_cv = reinterpret_cast<F64*>(sm_raw);
  constexpr int S = kCvCols;
  const int lane = threadIdx.x % S, w = threadIdx.x / S;
  const int col = blockIdx.x * S + lane;
  const bool valid = col < D.ny * D.nx;
  const int ji = valid ? col % D.ny + 1 : 1, jk = valid ? col / D.ny + 1 : 1;
  const int nl = D.nl, n = nl - 1;
  const F64 dtime = D.dtime, rdt = X.rdt;
  const long long goff = (long long)(D.g - 1) * D.fstride, pl = D.plane, c0 = IX(D, ji, jk, 1);
  const StateT<F64>& Su = (RK == 1) ? So : Sn;  // state_new_used
  const F64* rho_o = So.rho + goff;
  const F64* rho_u = Su.rho + goff;
  F64* rho_n = Sn.rho + goff;
  const F64* t_rho = Tn.rho + goff;
  const F64 pdw = 0.5;
  F64* const sc = sm_cv + lane;               // row jl at S*(jl-1)
  F64* const sd = sm_cv + S * nl + lane;
  F64* const se = sm_cv + 2 * S * nl + lane;
  F64* const sr = sm_cv + 3 * S * nl + lane;
  F64* const st = sm_cv + 4 * S * nl + lane;
  F64* const sg = sm_cv + 5 * S * nl + lane;  // layer jl
  F64* const sy = sm_cv + 6 * S * nl + lane;
  const F64 c_imp2 = kIMPL_THERMO_WEIGHT * (dtime * dtime) * kC_D_P;

  // alpha, beta, gamma over the volume, theta of state_new_used, explicit predictions
  struct Lay { F64 al, be, ga, th, ro, rhe, tpe, epe, V, rV; };
  auto layer = [&](int jl, bool predict) {
    Lay L{};
    const long long i = c0 + (long long)(jl - 1) * pl;
    L.V = G.volume[i];
    L.rV = X.rvol[i];
    const F64 ro = rho_o[i], rto = So.rt[i];
    L.ro = ro;
    const F64 yo = rcp(ro);
    F64 alpha = div_rn(-rto, ro * ro, yo * yo), beta = yo;
    F64 gamma = F64(kR_D) / (kC_D_V * rto) * (G.exner_bg[i] + So.ep[i]);
    if (RK == 2) {
      const F64 ru = rho_u[i], rtu = Su.rt[i];
      const F64 yu = rcp(ru);
      const F64 alpha_new = div_rn(-rtu, ru * ru, yu * yu);
      const F64 gamma_new = F64(kR_D) / (kC_D_V * rtu) * (G.exner_bg[i] + Su.ep[i]);
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
      const F64 tr = t_rho[i], trt = Tn.rt[i], dtv = dtime * L.V;
      L.rhe = ro + dtime * tr;
      L.tpe = So.tp[i] + dtv * (L.al * tr + L.be * trt);
      L.epe = So.ep[i] + dtv * L.ga * trt;
    }
    return L;
  };

  const int chunk = (n + kCvChunks - 1) / kCvChunks, r0 = w * chunk + 1, r1 = min(n, (w + 1) * chunk);
  if (valid && r0 <= r1) {
    Lay L0 = layer(r0, true), L1 = layer(r0 + 1, true), L2{};
    F64 rio = 0.5 * (L0.ro + L1.ro), yrio = rcp_near(rio);
    F64 t = 0.5 * (L0.th + L1.th);
    // half of exner_bg(jl-1) - exner_bg(jl) at the interface above layer p
    auto half_deb = [&](long long p) { return half(G.exner_bg[p - pl] - G.exner_bg[p]); };
    F64 hdeb = half_deb(c0 + (long long)r0 * pl);
    for (int jl = r0; jl <= r1; ++jl) {
      const long long b = c0 + (long long)jl * pl;  // layer jl+1 and w level jl+1
      const F64 zs = G.z_scalar[b - pl] - G.z_scalar[b], dp = G.damp[b], wo = So.w[b];
      const F64 rie = 0.5 * (L0.rhe + L1.rhe);
      const F64 dv = -(t * t) * (L0.ga + L1.ga) + hdeb * (L1.al - L0.al + t * (L1.be - L0.be))
                      - div_rn(zs, c_imp2 * rio, X.rc_imp2 * yrio)
                      * (2.0 * X.raz[b] + dtime * wo * 0.5 * (-L0.rV + L1.rV)) * dp;
      // (0.5/dtime * (...) * d(exner_bg), with hdeb half that difference: powers of two are exact)
      const F64 rv = div_rn(-(wo + dtime * Tn.w[b]) * zs, c_imp2, X.rc_imp2)
                      + div_rn(t * (L0.epe - L1.epe), dtime, rdt)
                      + 2.0 * (0.5 / dtime) * (L0.tpe + L1.tpe) * hdeb
                      - div_rn(div_rn(zs, c_imp2, X.rc_imp2) * wo * rie, rio, yrio);
      F64 cv = 0.0, ev = 0.0, rio_n = 0.0, yrio_n = 0.0, tn = 0.0, hdeb_n = 0.0;
      if (jl < n) {
        L2 = layer(jl + 2, jl < r1);
        const long long cc = b + pl;
        tn = 0.5 * (L1.th + L2.th);
        rio_n = 0.5 * (L1.ro + L2.ro);
        yrio_n = rcp_near(rio_n);
        hdeb_n = half_deb(cc);
        cv = tn * L1.ga * t + hdeb_n * (L1.al + L1.be * t)
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
      hdeb = hdeb_n;
    }
  }
  __syncthreads();
  if (valid && w == 0) {  // (hardware products: a chain)
    const double *const dc = &sc->v, *const dd = &sd->v;
    double *const de = &se->v, *const dr = &sr->v;
    double y = rcp_near(dd[0]);
    double ep = div_rn(de[0], dd[0], y), rp = div_rn(dr[0], dd[0], y);
    de[0] = ep;
    dr[0] = rp;
#pragma unroll 2
    for (int jl = 2; jl <= n; ++jl) {
      const double c = dc[S * (jl - 2)];
      const double den = dd[S * (jl - 1)] - ep * c;
      y = rcp_near(den);
      ep = div_rn(de[S * (jl - 1)], den, y);  // (0 in the last row)
      rp = div_rn(dr[S * (jl - 1)] - rp * c, den, y);
      de[S * (jl - 1)] = ep;
      dr[S * (jl - 1)] = rp;
    }
#pragma unroll 4
    for (int jl = n - 1; jl >= 1; --jl) {
      rp = dr[S * (jl - 1)] - de[S * (jl - 1)] * rp;
      dr[S * (jl - 1)] = rp;
    }
  }
  __syncthreads();
  // (hardware products again, beside the other blocks' integer ones)
  const int lchunk = (nl + kCvChunks - 1) / kCvChunks, l0 = w * lchunk + 1, l1 = min(nl, (w + 1) * lchunk);
  if (!valid || l0 > l1) return;
  auto new_rho = [&](int jl, double V, double rV) {
    const long long i = c0 + (long long)(jl - 1) * pl;
    const double rhe = rho_o[i].v + D.dtime * t_rho[i].v;
    if (jl == 1) return rhe + div_rn(D.dtime * sr[0].v, V, rV);
    if (jl == nl) return rhe - div_rn(D.dtime * sr[S * (n - 1)].v, V, rV);
    return rhe + div_rn(D.dtime * (-sr[S * (jl - 2)].v + sr[S * (jl - 1)].v), V, rV);
  };
  double rn_up = 0.0, ro_up = 0.0;
  if (l0 > 1) {
    const long long a = c0 + (long long)(l0 - 2) * pl;
    rn_up = new_rho(l0 - 1, G.volume[a].v, X.rvol[a].v);
    ro_up = rho_o[a].v;
  }
  for (int jl = l0; jl <= l1; ++jl) {
    const long long i = c0 + (long long)(jl - 1) * pl;
    const double V = G.volume[i].v, rV = X.rvol[i].v, rto = So.rt[i].v, ro = rho_o[i].v;
    const double rn = new_rho(jl, V, rV);
    const double rte = rto + D.dtime * Tn.rt[i].v;
    double rtn;
    if (jl == 1) rtn = rte + div_rn(D.dtime * st[0].v * sr[0].v, V, rV);
    else if (jl == nl) rtn = rte - div_rn(D.dtime * st[S * (n - 1)].v * sr[S * (n - 1)].v, V, rV);
    else rtn = rte + div_rn(D.dtime * (-(st[S * (jl - 2)].v * sr[S * (jl - 2)].v) + st[S * (jl - 1)].v * sr[S * (jl - 1)].v), V, rV);
    const double epn = So.ep[i].v + V * sg[S * (jl - 1)].v * (rtn - rto);
    const double tpn = quot(rtn, rn) - G.theta_v_bg[i].v;
    if (jl >= 2) {
      const double rin = 0.5 * (rn_up + rn);
      Sn.w[i] = div_rn(div_rn(2.0 * sr[S * (jl - 2)].v, G.area_z[i].v, X.raz[i].v) - rin * So.w[i].v, 0.5 * (ro_up + ro),
                       sy[S * (jl - 2)].v);
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
        W_(1, ji, jk, nl).v * Sn.u[IX(D, ji, jk + 1, nl)].v * G.slope_x[IX(D, ji, jk + 1, nl)].v
      + W_(2, ji, jk, nl).v * Sn.v[IX(D, ji, jk, nl)].v * G.slope_y[IX(D, ji, jk, nl)].v
      + W_(3, ji, jk, nl).v * Sn.u[IX(D, ji, jk, nl)].v * G.slope_x[IX(D, ji, jk, nl)].v
      + W_(4, ji, jk, nl).v * Sn.v[IX(D, ji + 1, jk, nl)].v * G.slope_y[IX(D, ji + 1, jk, nl)].v;
  }
}

// the grid-only factors of the column solves (ColumnGrid; itwdtv may be null)
__global__ void k_column_grid(Dims D, Grid<double> G, double* rvol, double* itwdtv, double* zs_c1h, double* raz) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl);
  rvol[q] = 1.0 / G.volume[q];
  if (itwdtv) itwdtv[q] = 0.5 * D.dtime / G.volume[q];
  if (jl == 1) return;
  zs_c1h[q] = (G.z_scalar[q - D.plane] - G.z_scalar[q]) / (kIMPL_THERMO_WEIGHT * D.dtime * kC_D_P) * 0.5;
  raz[q] = 1.0 / G.area_z[q];
}

void launch_column_grid(const Dims& D, const Grid<double>& G, double* rvol, double* itwdtv, double* zs_c1h, double* raz,
                        cudaStream_t st) {
  const dim3 g((unsigned)((D.ny + 31) / 32), (unsigned)D.nl, (unsigned)((D.nx + 7) / 8));
  k_column_grid<<<g, dim3(32, 8), 0, st>>>(D, G, rvol, itwdtv, zs_c1h, raz);
}

void launch_column_ver(const Dims& D, const Grid<double>& G, const ColumnGrid& X, const State& So, const State& Sn,
                       const Tend<double>& Tn, int rk_step, cudaStream_t st) {
  const unsigned nb = (unsigned)(((long long)D.ny * D.nx + kCvCols - 1) / kCvCols);
  const size_t sm = (size_t)kCvArrays * kCvCols * D.nl * sizeof(double);
  const Tend<F64> T{f64(Tn.rho), f64(Tn.rt), f64(Tn.u), f64(Tn.v), f64(Tn.w)};
  if (rk_step == 1) k_column_ver<1><<<nb, kCvCols * kCvChunks, sm, st>>>(D, f64(G), X, f64(So), f64(Sn), T);
  else k_column_ver<2><<<nb, kCvCols * kCvChunks, sm, st>>>(D, f64(G), X, f64(So), f64(Sn), T);
}

// v_fall_liquid, mo_derived.F90:218-263 (state_old, diag%temperature)
__device__ __forceinline__ F64 v_fall_liquid(const Dims& D, const Grid<F64>& G, const F64* rho_g, const F64* T,
                                             double radius, int ji, int jk, int jl) {
  const long long i = IX(D, ji, jk, jl), b = i + D.plane;
  F64 g;
  if (jl == 1) g = G.gm[b];
  else if (jl == D.nl) g = G.gm[i];
  else g = G.ipw[4][i] * G.gm[i] + G.ipw[5][i] * G.gm[b];
  const F64 rg = rho_g[i];
  const F64 nu = calc_diff_coeff(T[i], rg);
  F64 v = 2.0 * (radius * radius) * (kRHO_H2O - rg) * g / (9.0 * rg * nu);
  // v*radius/nu > 10, the quotient formed only where v*radius is not clearly below 10 nu
  const F64 vr = v * radius;
  if (__double2hiint(vr.v) >= __double2hiint((9.99 * nu).v) && (vr / nu) > 10.0)
    v = root(8.0 * radius * kRHO_H2O * g / (3.0 * rg * 0.8));
  return v;
}
// c_p_water and c_p_ice, mo_dictionary.F90:112-173
__device__ __forceinline__ F64 c_p_water64(F64 temperature) {
  F64 tc = temperature - kT_0, c;
  if (upwind(tc)) {
    F64 a = tc - 35.0;
    if (positive(a)) a = 0.0;  // at most 35
    const F64 a2 = a * a;
    c = 0.9979 + 3.1e-6 * a2 + 3.8e-9 * (a2 * a2);
  } else {
    if (tc < -37.0) tc = -37.0;
    const F64 t2 = tc * tc;
    c = 1.000938 - 2.7052e-3 * tc - 2.3235e-5 * t2 + 4.3778e-6 * (t2 * tc) + 2.7136e-7 * (t2 * t2);
  }
  return 4186.8 * c;
}
__device__ __forceinline__ F64 c_p_ice64(F64 temperature) {
  F64 tl = temperature;
  if (tl > kT_0) tl = kT_0;
  if (tl < 20.0) tl = 20.0;
  const F64 q = div_rn(tl, 125.1, 1.0 / 125.1);
  const F64 c = -2.0572 + 0.14644 * tl + 0.06163 * tl * exp(-(q * q).v);
  return div_rn(c, kM_V, 1.0 / kM_V);
}

// v_fall_solid, mo_derived.F90:265-283 (threshold is the default-real literal 250.e-6)
__device__ __forceinline__ double v_fall_solid(double radius) {
  return (radius > (double)250.e-6f) ? 1.0 : 0.001;
}

// The quantities of a level that depend only on state_old and its temperature, formed once per
// step: the cloud droplets' fall speed, read by both substeps' tracer solves, and c_p of ice and
// water, read by the sediment heating and by both substeps' diabatic term (gas_theta).
__global__ void k_moist_aux(Dims D, Grid<F64> G, StateT<F64> So, const F64* T, F64* vcloud, F64* cpi, F64* cpw) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl);
  const double cloud_r = 12.e-6;  // mo_dictionary.F90:276-318
  vcloud[q] = v_fall_liquid(D, G, So.rho + (long long)(D.g - 1) * D.fstride, T, cloud_r, ji, jk, jl);
  cpi[q] = c_p_ice64(T[q]);
  cpw[q] = c_p_water64(T[q]);
}
void launch_moist_aux(const Dims& D, const Grid<double>& G, const State& So, const double* T, double* vcloud, double* cpi,
                      double* cpw, cudaStream_t st) {
  const dim3 g((unsigned)((D.ny + 31) / 32), (unsigned)D.nl, (unsigned)((D.nx + 7) / 8));
  k_moist_aux<<<g, dim3(32, 8), 0, st>>>(D, f64(G), f64(So), f64(T), f64(vcloud), f64(cpi), f64(cpw));
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
__device__ __forceinline__ void tracer_group(const Dims& D, const Grid<F64>& G, const StateT<F64>& So, const StateT<F64>& Sn,
                                             const F64* t_rho_all, const F64* T, const F64* rvol,
                                             const F64* itwdtv, const F64* vcloud, const F64* cpi,
                                             const F64* cpw, F64* csh, F64* hx, int ji, int jk, bool valid, int lane, int w,
                                             F64* sm) {
  using TG = TracerGroup<GROUP>;
  constexpr int N = TG::n(), S = kTcCols;
  const int nl = D.nl;
  const long long pl = D.plane, c0 = IX(D, ji, jk, 1);
  F64* const sk = sm + lane;               // coupling of the interface below row jl at sk[S*(jl-1)]
  F64* const sd = sm + S * nl + lane;      // diagonal
  F64* const sy = sm + 2 * S * nl + lane;  // its reciprocal
  F64* const sr = sm + 3 * S * nl + lane;  // right-hand side, then the solution: tracer q at + q*S*nl
  const F64 dtime = D.dtime;
  const F64 itw = 0.5, expl_weight = 1.0 - itw;
  const F64 ewdt = expl_weight * dtime;
  const int chunk = (nl + kTcChunks - 1) / kTcChunks, l0 = w * chunk + 1, l1 = min(nl, (w + 1) * chunk);
  const F64 vfix = GROUP == 0 ? v_fall_solid(500.e-6) : GROUP == 2 ? v_fall_solid(95.e-6) : 0.0;
  if (valid && l0 <= l1) {
    // interface between levels m and m+1: w point m+1
    struct Iface { F64 vfi, p0, p1, fr[N], ve[N]; };
    auto iface = [&](int m, const F64* ro_a, const F64* ro_b, F64 itwa, F64 itwb) {
      Iface f;
      const long long b = c0 + (long long)m * pl;
      F64 wo = So.w[b], wn = Sn.w[b];
      if (GROUP != 1) {
        const F64 vf = GROUP == 3 ? 0.5 * (vcloud[b - pl] + vcloud[b]) : vfix;
        wo = wo - vf;
        wn = wn - vf;
      }
      const F64 az = G.area_z[b];
      f.vfi = az * wo;
      const F64 vfr = az * wn;
      f.p0 = itwa * f.vfi;
      f.p1 = itwb * f.vfi;
      F64 cti = 0.0, ctw = 0.0;
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
    auto load_rho = [&](int m, F64* r) {
#pragma unroll
      for (int q = 0; q < N; ++q) r[q] = So.rho[c0 + (long long)(m - 1) * pl + (long long)(TG::jc(q) - 1) * D.fstride];
    };
    F64 ro[N], ro_n[N];
    load_rho(l0, ro);
    F64 itw_c = itwdtv[c0 + (long long)(l0 - 1) * pl];
    Iface up{}, dn{};
    if (l0 > 1) {
      F64 ro_u[N];
      load_rho(l0 - 1, ro_u);
      up = iface(l0 - 1, ro_u, ro, itwdtv[c0 + (long long)(l0 - 2) * pl], itw_c);
    }
    for (int jl = l0; jl <= l1; ++jl) {
      const long long i = c0 + (long long)(jl - 1) * pl;
      const F64 V = G.volume[i], rV = rvol[i];
      F64 itw_n = 0.0;
      if (jl < nl) {
        load_rho(jl + 1, ro_n);
        itw_n = itwdtv[i + pl];
        dn = iface(jl, ro, ro_n, itw_c, itw_n);
      }
      const F64 az_sfc = (jl == nl) ? G.area_z[i + pl] : 0.0;
      const F64 v_sfc = GROUP == 3 ? ((jl == nl) ? vcloud[i] : 0.0) : vfix;
      F64 d = 1.0;
      if (jl > 1 && !negative(up.vfi)) d = d + up.p1;
      if (jl < nl && negative(dn.vfi)) d = d - dn.p0;
      if (jl == nl && TG::cond(0) && GROUP != 1) d = d + div_rn(itw * v_sfc * dtime * az_sfc, V, rV);
      const F64 y = rcp_near(d);
      sd[S * (jl - 1)] = d;
      sy[S * (jl - 1)] = y;
      // (written as -e/d: e = -(itwdtv*vfi), so k = (itwdtv*vfi)/d)
      if (jl < nl) sk[S * (jl - 1)] = negative(dn.vfi) ? dn.p1 : div_rn(dn.p0, d, y);
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const F64 tr = t_rho_all[i + (long long)(TG::jc(q) - 1) * D.fstride];
        F64 r = ro[q] + dtime * tr;
        F64 h = 0.0, h2 = 0.0;
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
    double* const r = &sr->v + S * nl * w;
    const double *const dk = &sk->v, *const dd = &sd->v, *const dy = &sy->v;
    double rp = r[0] = div_rn(r[0], dd[0], dy[0]);
#pragma unroll 4
    for (int jl = 2; jl <= nl; ++jl) {
      const double k = dk[S * (jl - 2)];
      const double x = negative(k) ? r[S * (jl - 1)] - rp * k : r[S * (jl - 1)];
      rp = div_rn(x, dd[S * (jl - 1)], dy[S * (jl - 1)]);
      r[S * (jl - 1)] = rp;
    }
#pragma unroll 4
    for (int jl = nl - 1; jl >= 1; --jl) {
      const double k = dk[S * (jl - 1)];
      rp = negative(k) ? r[S * (jl - 1)] : r[S * (jl - 1)] + k * rp;
      r[S * (jl - 1)] = rp;
    }
  }
  __syncthreads();
  if (valid)
    for (int jl = l0; jl <= l1; ++jl)
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const F64 s = sr[S * (nl * q + jl - 1)];
        Sn.rho[c0 + (long long)(jl - 1) * pl + (long long)(TG::jc(q) - 1) * D.fstride] = negative(s) ? 0.0 : s;
      }
  __syncthreads();  // the next group overwrites the arrays
}

template <bool HEAT>
__global__ void __launch_bounds__(kTcCols* kTcChunks, 3)
    k_column_tracers(Dims D, Grid<F64> G, StateT<F64> So, StateT<F64> Sn, const F64* t_rho_all, const F64* T,
                     const F64* rvol, const F64* itwdtv, const F64* vcloud, const F64* cpi, const F64* cpw,
                     F64* csh, F64* hx) {
  extern __shared__ __align__(16) double sm_raw[];
  const int lane = threadIdx.x % kTcCols, w = threadIdx.x / kTcCols;
  const int col = blockIdx.x * kTcCols + lane;
  const bool valid = col < D.ny * D.nx;
  const int ji = valid ? col % D.ny + 1 : 1, jk = valid ? col / D.ny + 1 : 1;
#define TC_GROUP(g) \
  tracer_group<g, HEAT>(D, G, So, Sn, t_rho_all, T, rvol, itwdtv, vcloud, cpi, cpw, csh, hx, ji, jk, valid, lane, w, \
                        reinterpret_cast<F64*>(sm_raw))
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
    k_column_tracers<true><<<nb, b, sm, st>>>(D, f64(G), f64(So), f64(Sn), f64(t_rho), f64(T), f64(rvol), f64(itwdtv), f64(vcloud),
                                              f64(cpi), f64(cpw), f64(csh), f64(hx));
  else
    k_column_tracers<false><<<nb, b, sm, st>>>(D, f64(G), f64(So), f64(Sn), f64(t_rho), f64(T), f64(rvol), f64(itwdtv), f64(vcloud),
                                              f64(cpi), f64(cpw), f64(csh), f64(hx));
}

}  // namespace lg
