// split.cu -- FP32/FP64 split-precision HEVI step (compiled with -fmad=true, -prec-div=false).
//
// The explicit stencils are the templates of kernels.cuh instantiated for float.  They read
// an FP32 mirror of the state: a rounded copy of every prognostic field, written by the
// kernels that update the FP64 state (k_tend_wind for u and v, the two column solvers for
// the rest) and refreshed from the FP64 state whenever the host replaces it.  On this GPU a
// conversion between FP64 and FP32 costs as much as an FP64 operation (both ~2 per clock
// per SM, against 128 FP32 operations), so converting each state value once when it is
// written, instead of at every stencil use, takes the FP32 stencils off the FP64 pipe.
//
// This file adds the parts that stay in FP64 in this mode -- the pressure gradient and the
// two column solvers -- written to spend as few FP64 operations per cell as the precision
// split allows: coefficients that only scale an increment (the partial derivatives of the
// implicit system, fall speeds, fluxes) come from the FP32 mirror; the right-hand sides,
// the substitution sweeps of the tridiagonal solves and the state updates are FP64.
#include "split.cuh"
#include "common.h"
#include "fp64.cuh"
#include "lgame_gpu.h"
#include "tile_sweep.cuh"

#include <algorithm>
#include <string>
#include <vector>

namespace lg {

namespace {

struct GridX {  // FP64 reciprocal metrics and FP32 metric differences of the FP64 parts
  const double *inv_dx, *inv_dy, *inv_dz, *inv_volume, *inv_area_z;
  // FP32: 1/volume, 1/area_z, and at w level jl (2..nl) z_scalar(jl-1)-z_scalar(jl) and
  // exner_bg(jl-1)-exner_bg(jl), differenced in FP64 before rounding (no cancellation)
  const float *inv_volume_f, *inv_area_z_f, *dzs_f, *deb_f;
  // FP32: the swamp layer's deceleration per unit w, (1/damping_prefactor - 1)/dtime, formed in
  // FP64 (w/p - w would cancel where the prefactor is near 1); 0 at the top level
  const float* kdamp_f;
};

// x / d to FP64 accuracy for an FP32 divisor d in the normal range.  r = 1/d correctly
// rounded in FP32; the residual 1 - d*r of a correctly rounded reciprocal is exact in FP32,
// so r + (1 - d*r)*r is 1/d to ~2^-48 as an unevaluated pair of FP32 numbers (the
// correction step of Markstein's division), and x*(r + r_lo) costs one FP64-pipe operation and a
// product formed beside that pipe (relative error below 2^-47) instead of a conversion and an FP64 division.
__device__ __forceinline__ double div_f(double x, float d) {
  const float r = __frcp_rn(d);
  const float r_lo = __fmaf_rn(-d, r, 1.f) * r;
  return fma(x, wide(r_lo), mul_int(r, x));
}
}  // namespace

struct SplitCtx {
  std::vector<void*> allocs;
  Grid<float> GF{};
  GridX GX{};
  float *gf[40] = {};
  float *ipw[6] = {}, *trsk_u[3] = {}, *trsk_v[2] = {};
  double *inv_dx = nullptr, *inv_dy = nullptr, *inv_dz = nullptr, *inv_volume = nullptr, *inv_area_z = nullptr;
  // FP32 intermediates
  float *gx, *gy, *divf, *tvu, *tvv, *tpu, *tpv, *ex, *ey, *ez, *uph, *vph, *wph;
  // kinetic energy in FP64: its vertical differences over thin layers cancel most digits
  double* vsq = nullptr;
  // FP64 vertical gradient of exner' at w points (0 at the top and surface levels), and per
  // column and terrain-following layer l half its weighted sum 0.5*(W5*gz(l) + W6*gz(l+1))
  double* gzd = nullptr;
  double* rmz = nullptr;
  // sediment heating of each condensate (nc planes), summed into the carried csh
  float* csh_part = nullptr;
  float* cw = nullptr;  // contravariant wind correction times the interface area (moist)
  // divergence of the gradient of theta_bg (the third-order theta chain of the background),
  // and the background's x and y edge averages as FP32 pairs
  float* dbg = nullptr;
  float2 *tbu = nullptr, *tbv = nullptr;
  // horizontal gas mass fluxes and theta_v fluxes of the scalar tendency
  float *fu = nullptr, *fv = nullptr, *gu = nullptr, *gv = nullptr;
  // FP32 mirrors of the two state slots
  StateF mir[2]{};
  SplitCarriedF C{};
  // rhotheta_v of the background state, p_0/r_d*exner_bg^(c_d_v/r_d) (boundary relaxation)
  double* rtbg = nullptr;
  // the vertical acoustic solve with FP64 coefficients and elimination (precision mode
  // LGAME_PRECISION_SPLIT_FP64_COLUMN)
  bool column_fp64 = false;
  // diffusion closure: configuration and FP32 buffers (the carried ones are in C)
  SplitDiff diff{};
  DiffBuf<float> db{};
  // surface layer, PBL and soil (FP64 buffers of the FP64 step)
  SplitSfc sfc{};
  // the step's concurrent branches: two side streams and the events of their forks and joins
  cudaStream_t br[2] = {nullptr, nullptr};
  cudaEvent_t ev[9] = {};
};

namespace {

template <class P>
int salloc(SplitCtx* s, P** p, size_t n, long long* bytes) {
  void* q = nullptr;
  cudaError_t e = cudaMalloc(&q, n * sizeof(P));
  if (e != cudaSuccess) {
    lgame_set_error((std::string("cudaMalloc (split) failed: ") + cudaGetErrorString(e)).c_str());
    return LGAME_ERR_ALLOC;
  }
  if (cudaMemset(q, 0, n * sizeof(P)) != cudaSuccess) return LGAME_ERR_CUDA;
  s->allocs.push_back(q);
  *bytes += (long long)(n * sizeof(P));
  *p = (P*)q;
  return LGAME_OK;
}

__global__ void k_to_float(const double* a, float* b, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    b[i] = (float)a[i];
}
__global__ void k_net(const double* a, const double* b, float* net, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    net[i] = narrow(a[i] + b[i]);
}
__global__ void k_to_double(const float* a, double* b, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    b[i] = (double)a[i];
}
__global__ void k_recip(const double* a, double* b, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    b[i] = (a[i] != 0.0) ? 1.0 / a[i] : 0.0;
}
// FP32 metric reciprocals and vertical differences of the column solver (set-up only)
__global__ void k_grid_extra(Dims D, Grid<double> G, float* ivol, float* iaz, float* dzs, float* deb, float* kd) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx || jl > D.NL) return;
  const long long q = IX(D, ji, jk, jl);
  iaz[q] = (G.area_z[q] != 0.0) ? float(1.0 / G.area_z[q]) : 0.f;
  kd[q] = (jl >= 2) ? float((1.0 / G.damp[q] - 1.0) / D.dtime) : 0.f;
  if (jl <= D.nl) ivol[q] = float(1.0 / G.volume[q]);
  if (jl >= 2 && jl <= D.nl) {
    const long long a = IX(D, ji, jk, jl - 1);
    dzs[q] = float(G.z_scalar[a] - G.z_scalar[q]);
    deb[q] = float(G.exner_bg[a] - G.exner_bg[q]);
  }
}

// ---- edges ---------------------------------------------------------------------------------
// The kernels at u and v points read a thread's x and y edge both, at addresses that are valid
// everywhere, before they store either: branches around the loads, and stores between them, made
// each edge wait for memory on its own (ncu: 20 to 44 of 25 to 50 cycles an issue on loads, DRAM at
// 35 %).  At 768x768x80: gas fluxes 491 -> 305 us, theta edges 468 -> 393 us, gradients 508 -> 454 us.
//
// The two cells a and b of the x (y) edge at (ji, jk): a west (north), b east (south) of it, b also
// being where the reference evaluates the edge; periodic wrap edges join the first and last cell.
// q: the edge itself (where there is none, a cell's); in: an edge of the grid; flux: one the
// operators write (not a non-periodic boundary's).
struct Edge { long long a, b, q; bool in, flux; };
__device__ __forceinline__ Edge edge_x(const Dims& D, int ji, int jk, int jl) {
  const bool inner = jk >= 2 && jk <= D.nx;
  const int i = min(ji, D.ny);
  Edge e;
  e.in = ji <= D.ny;
  e.flux = e.in && (inner || D.periodic);
  e.a = IX(D, i, inner ? jk - 1 : D.nx, jl);
  e.b = IX(D, i, inner ? jk : 1, jl);
  e.q = IX(D, i, jk, jl);
  return e;
}
__device__ __forceinline__ Edge edge_y(const Dims& D, int ji, int jk, int jl) {
  const bool inner = ji >= 2 && ji <= D.ny;
  const int k = min(jk, D.nx);
  Edge e;
  e.in = jk <= D.nx;
  e.flux = e.in && (inner || D.periodic);
  e.a = IX(D, inner ? ji - 1 : D.ny, k, jl);
  e.b = IX(D, inner ? ji : 1, k, jl);
  e.q = IX(D, ji, k, jl);
  return e;
}

// ---- pressure gradient, mo_p_grad.F90:20-120, FP64 products ---------------------------
// gradient of the Exner pressure perturbation in FP64 (the small differences of a small
// field), theta edge values in FP32 (third order) or FP64 (second order), the background
// term theta'*grad(Pi_bg) in FP64, the condensate deceleration factor in FP32 from the
// mirror densities.  With plain products 32 FP64 operations a cell bound it: the products are
// formed beside that pipe (fp64.cuh), the loads of both edges and of the w point come first, and the
// condensate fractions of the six cells come from ks_gzp: 3.28 -> 2.03 ms at 768x768x80 with moisture
// (ks_gzp 0.52 -> 0.73 ms), 1.04 -> 0.74 ms at 512x512x50 without.

// nl = de*(te*grad), and l: de and an FP32 te (or theta') are widened; their product with the
// gradient is FP64 (an extra FP32 rounding of either product would unbalance the two terms, which
// cancel in an atmosphere at rest)
__device__ __forceinline__ double weighted(float de, float te, double grad) { return mul_int(de, mul_int(te, grad)); }
__device__ __forceinline__ double weighted(float de, double te, double grad) { return mul_int(de, mul_int(te, grad)); }

// cf: the cells' condensate mass fractions (ks_gzp; not read with a dry atmosphere).  TH: the type of
// the theta edges, float in the third order (tvu.., tpu..), double in the second, formed here.
template <class TH>
__global__ void __launch_bounds__(256, 4) ks_pgrad(Dims D, Grid<double> G, GridX X, State S, const double* gzd,
                                                  const double* rmz, const float* cf, const float* tvu,
                                                  const float* tvv, const float* tpu, const float* tpv,
                                                  PGrad<double> P, SplitCarriedF PF, float* pgcw, int lfirst) {
  LG_IDX3;
  if (ji > D.ny + 1 || jk > D.nx + 1) return;
  const bool bg = D.luse_bg, cell = ji <= D.ny && jk <= D.nx && jl >= 2;
  const Edge x = edge_x(D, ji, jk, jl), y = edge_y(D, ji, jk, jl);
  const long long q = IX(D, ji, jk, jl), qc = IX(D, min(ji, D.ny), min(jk, D.nx), jl), qa = jl >= 2 ? qc - D.plane : qc;
  const double *ep = S.ep, *tp = S.tp, *tb = G.theta_v_bg;
  const double exa = ep[x.a], exb = ep[x.b], eya = ep[y.a], eyb = ep[y.b];
  const double ix = X.inv_dx[x.b], iy = X.inv_dy[y.b];
  // theta at the edges, and theta' where there is a background
  TH tx, ty, px = 0, py = 0;
  if constexpr (sizeof(TH) == 4) {
    tx = tvu[x.b];
    ty = tvv[y.b];
    if (bg) {
      px = tpu[x.b];
      py = tpv[y.b];
    }
  } else {
    const double xa = tp[x.a], xb = tp[x.b], ya = tp[y.a], yb = tp[y.b];
    tx = half((tb[x.a] + xa) + (tb[x.b] + xb));
    ty = half((tb[y.a] + ya) + (tb[y.b] + yb));
    px = half(xa + xb);
    py = half(ya + yb);
  }
  const double tpa = tp[qa], tpb = tp[qc], tba = tb[qa], tbb = tb[qc], gzc = gzd[qc];
  double gu = 0.0, gv = 0.0, gw = 0.0;
  float net_u = 0.f, net_v = 0.f;
  if (bg) {
    gu = G.egu[x.b];
    gv = G.egv[y.b];
    gw = G.egw[qc];
    net_u = PF.pnet_u[q];
    net_v = PF.pnet_v[q];
  }
  const double gm = G.gm[qc];
  // condensate mass fraction sum(rho_cond)/sum(rho): the reference's rho_g/sum(rho) and
  // rho_g/sum(rho) - 1 (mo_p_grad.F90:86-87, :115-116) rewritten as 1 - f and -f, which
  // is exact for dry air and free of cancellation in FP32
  float fxa = 0.f, fxb = 0.f, fya = 0.f, fyb = 0.f, fa = 0.f, fb = 0.f;
  if (D.nc > 0) {
    fxa = cf[x.a];
    fxb = cf[x.b];
    fya = cf[y.a];
    fyb = cf[y.b];
    fa = cf[qa];
    fb = cf[qc];
  }
  auto decel = [](float a, float b) {
    return 0.5f * ((float(kC_D_P) - float(kC_D_P) * a) + (float(kC_D_P) - float(kC_D_P) * b));
  };
  double gx = mul_int(exb - exa, ix), gy = mul_int(eya - eyb, iy);
  // remap_ver2hor_x/_y (mo_averaging.F90:56-136) of the vertical gradient at a u or v face: the sum
  // over the face's two columns a and b of 0.5*(W5*gz(l) + W6*gz(l+1)), each column's term formed once
  // in ks_gzp (the reference adds the four products in the order W5a, W5b, W6a, W6b; here
  // the pairs of a column are added first, an FP64 rounding difference)
  if (jl > D.nf) {
    gx -= G.slope_x[x.b] * (rmz[x.a] + rmz[x.b]);
    gy -= G.slope_y[y.b] * (rmz[y.a] + rmz[y.b]);
  }
  // Both products are stored in FP64 (the reference's diagnostics).  With a background state
  // the wind update uses only the net nl + l and the previous substep's -(nl + l), both rounded
  // to FP32, so those are also kept in FP32 (net, old): the same values the update would round,
  // read at a third of the bytes.  p_grad_acc_old is updated in that form only.  Without a
  // background state nl alone carries the hydrostatic balance and the update reads the FP64
  // arrays.
  auto update = [&](const Edge& e, float de, TH te, TH tpe, double g, double gb, float net_prev, double* nl, double* l,
                    double* old, float* net_f, float* old_f) {
    const double nlv = weighted(de, te, g);
    if (bg) {
      float o = -net_prev;
      if (e.flux) {
        const double lv = weighted(de, tpe, gb);
        nl[q] = nlv;
        l[q] = lv;
        const float net = narrow(nlv + lv);
        net_f[q] = net;
        if (lfirst) o = -net;
      }
      old_f[q] = o;
    } else {
      const double nl_prev = nl[q];
      if (!lfirst) old[q] = -nl_prev;
      if (e.flux) {
        nl[q] = nlv;
        if (lfirst) old[q] = -nlv;
      } else if (lfirst) {
        old[q] = -nl_prev;
      }
    }
  };
  if (x.in) update(x, decel(fxa, fxb), tx, px, gx, gu, net_u, P.nl_u, P.l_u, P.old_u, PF.pnet_u, PF.pold_u);
  if (y.in) update(y, decel(fya, fyb), ty, py, gy, gv, net_v, P.nl_v, P.l_v, P.old_v, PF.pnet_v, PF.pold_v);
  if (cell) {
    const float de = decel(fa, fb);
    const double nlw = mul_int(de, half((tba + tpa) + (tbb + tpb)) * gzc);
    P.nl_w[q] = nlw;
    if (bg) {
      const double lw = mul_int(de, half(tpa + tpb) * gw);
      P.l_w[q] = lw;
      PF.pnet_w[q] = narrow(nlw + lw);
    }
    pgcw[q] = 0.5f * (-fa - fb) * narrow(gm);
  }
}

// vertical gradient of exner_pert at the w levels 2..nl (grad_vert, mo_gradient_operators.F90:65-83),
// and in the terrain-following layers l > nf the column's half of the remap of that gradient
// to the horizontal faces, 0.5*(W5(l)*gz(l) + W6(l)*gz(l+1)) (mo_averaging.F90:56-136; the W6
// term only where l < nl or with a free-slip surface), gz being 0 at levels 1 and nl+1; with
// condensates the cell's condensate mass fraction cf, which ks_pgrad reads at six cells
__global__ void ks_gzp(Dims D, Grid<double> G, GridX X, const double* ep, const float* mrho, double* gzd, double* rmz,
                       float* cf) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl);
  const double e0 = ep[jl >= 2 ? q - D.plane : q], e1 = ep[q];
  const double gz = jl >= 2 ? mul_int(e0 - e1, X.inv_dz[q]) : 0.0;
  double r = 0.0;
  if (jl > D.nf) {
    r = mul_int(G.ipw[4][q], gz);
    if (jl < D.nl || D.freeslip) {
      const double gz1 = (jl < D.nl) ? mul_int(e1 - ep[q + D.plane], X.inv_dz[q + D.plane]) : 0.0;
      r += G.ipw[5][q] * gz1;
    }
  }
  float c = 0.f;
  if (D.nc > 0) {
    for (int jc = 0; jc < D.nc; ++jc) c += mrho[q + (long long)jc * D.fstride];
    c = c / (c + mrho[q + (long long)(D.g - 1) * D.fstride]);
    cf[q] = c;
  }
  if (jl >= 2) gzd[q] = gz;
  if (jl > D.nf) rmz[q] = half(r);
}

// specific kinetic energy (inner_product, mo_inner_product.F90:15-50) in FP64: half of its products
// are formed beside the FP64 pipe (fp64.cuh): 0.75 against 1.02 ms at 768x768x80
__global__ void ks_ke(Dims D, Grid<double> G, State S, double* out) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl);
  const double a[6] = {S.u[IX(D, ji, jk + 1, jl)], S.v[q], S.u[q], S.v[IX(D, ji + 1, jk, jl)], S.w[q], S.w[q + D.plane]};
  double k = 0.0;
#pragma unroll
  for (int i = 0; i < 6; ++i) k = fma(mul_int(G.ipw[i][q], a[i]), a[i], k);
  out[q] = k;
}

// horizontal gas mass fluxes and theta_v fluxes of scalar_tend_expl, mo_scalar_tend_expl.F90:106-138:
// rho_g*u at u points, rho_g*v at v points (scalar_times_vector_h), times the theta_v edge
// values (third order: tvu, tvv; second order: the mean of the two cells).  Each face is
// computed once here and read by ks_gas_div; the reference's untouched boundary faces are 0.
__global__ void ks_gas_flux(Dims D, Grid<float> GF, StateF Ss, const float* u_new, const float* v_new,
                            const float* tvu, const float* tvv, float* fu, float* fv, float* gu, float* gv) {
  LG_IDX3;
  if (ji > D.ny + 1 || jk > D.nx + 1) return;
  const float* rg = Ss.rho + (long long)(D.g - 1) * D.fstride;
  const long long q = IX(D, ji, jk, jl);
  const Edge x = edge_x(D, ji, jk, jl), y = edge_y(D, ji, jk, jl);
  const float rxa = rg[x.a], rxb = rg[x.b], ux = u_new[x.b], rya = rg[y.a], ryb = rg[y.b], vy = v_new[y.b];
  float tx, ty;
  if (D.theta_order == 2) {
    auto th = [&](long long p) { return GF.theta_v_bg[p] + Ss.tp[p]; };
    tx = 0.5f * (th(x.a) + th(x.b));
    ty = 0.5f * (th(y.a) + th(y.b));
  } else {
    tx = tvu[x.q];
    ty = tvv[y.q];
  }
  const float f = x.flux ? 0.5f * (rxa + rxb) * ux : 0.f, h = y.flux ? 0.5f * (rya + ryb) * vy : 0.f;
  if (x.in) {
    fu[q] = f;
    gu[q] = x.flux ? tx * f : 0.f;
  }
  if (y.in) {
    fv[q] = h;
    gv[q] = y.flux ? ty * h : 0.f;
  }
}

// theta_v_adv_3rd_order edge values, mo_multiplications.F90:134-202, from theta' and dv, the
// divergence of the gradient of theta'.  The chain theta -> gradient -> divergence is linear,
// so the full theta_v edge is the background's part plus theta''s: 0.5*(theta_bg,a +
// theta_bg,b) - c*dbg, with dbg the background's divergence and both formed once in FP64 at
// set-up (split_set_grid; the face average is kept as an FP32 pair hi + lo), plus
// 0.5*(theta'_a + theta'_b) - c*dv.  Adding the small parts first and hi last rounds the
// ~300 K edge value once, where theta_bg + theta' rounded per cell cost one to two units of
// the last place; the FP32 differences are taken of theta' rather than of theta_v.  With
// tpu/tpv given, the edges of theta' alone (the background-subtracted edges of the pressure
// gradient) come from the same pass.  The upwind cell of the correction follows the face
// velocity as in the reference.
__global__ void ks_theta_edges(Dims D, const float* tp, const float* dv, const float* dbg, const float2* tbu,
                               const float2* tbv, const float* u, const float* v, float* tvu, float* tvv, float* tpu,
                               float* tpv) {
  LG_IDX3;
  if (ji > D.ny + 1 || jk > D.nx + 1) return;
  const float c = narrow(D.theta_edge_c);
  const long long q = IX(D, ji, jk, jl);
  const Edge x = edge_x(D, ji, jk, jl), y = edge_y(D, ji, jk, jl);
  const float xpa = tp[x.a], xpb = tp[x.b], ux = u[x.b], ypa = tp[y.a], ypb = tp[y.b], vy = v[y.b];
  const float2 bx = tbu[x.q], by = tbv[y.q];
  // the upwind cell: west (a) of an x edge, south (b) of a y edge for a velocity >= 0 (loading both
  // cells' values instead of waiting for the velocity: 0.51 against 0.39 ms at 768x768x80)
  const long long xu = ux >= 0.f ? x.a : x.b, yu = vy >= 0.f ? y.b : y.a;
  const float xd = dv[xu], xg = dbg[xu], yd = dv[yu], yg = dbg[yu];
  const float xe = 0.5f * (xpa + xpb), ye = 0.5f * (ypa + ypb);
  if (x.flux) {
    tvu[q] = bx.x + (bx.y + ((xe - c * xd) - c * xg));
    if (tpu) tpu[q] = xe - c * xd;
  }
  if (y.flux) {
    tvv[q] = by.x + (by.y + ((ye - c * yd) - c * yg));
    if (tpv) tpv[q] = ye - c * yd;
  }
}

// ks_theta_edges and ks_gas_flux in one, for the second substep, whose theta edges are those of the fluxes alone:
// they are not stored, and the winds are read once (1.23 -> 0.77 ms at 1024x1024x80)
__global__ void ks_theta_flux(Dims D, StateF S, const float* dv, const float* dbg, const float2* tbu, const float2* tbv,
                              float* fu, float* fv, float* gu, float* gv) {
  LG_IDX3;
  if (ji > D.ny + 1 || jk > D.nx + 1) return;
  const float c = narrow(D.theta_edge_c);
  const float *rg = S.rho + (long long)(D.g - 1) * D.fstride, *tp = S.tp;
  const long long q = IX(D, ji, jk, jl);
  const Edge x = edge_x(D, ji, jk, jl), y = edge_y(D, ji, jk, jl);
  const float ux = S.u[x.b], vy = S.v[y.b];
  const float xpa = tp[x.a], xpb = tp[x.b], ypa = tp[y.a], ypb = tp[y.b];
  const float rxa = rg[x.a], rxb = rg[x.b], rya = rg[y.a], ryb = rg[y.b];
  const float2 bx = tbu[x.q], by = tbv[y.q];
  const long long xu = ux >= 0.f ? x.a : x.b, yu = vy >= 0.f ? y.b : y.a;
  const float xd = dv[xu], xg = dbg[xu], yd = dv[yu], yg = dbg[yu];
  const float tx = bx.x + (bx.y + ((0.5f * (xpa + xpb) - c * xd) - c * xg));
  const float ty = by.x + (by.y + ((0.5f * (ypa + ypb) - c * yd) - c * yg));
  const float f = x.flux ? 0.5f * (rxa + rxb) * ux : 0.f, h = y.flux ? 0.5f * (rya + ryb) * vy : 0.f;
  if (x.in) {
    fu[q] = f;
    gu[q] = x.flux ? tx * f : 0.f;
  }
  if (y.in) {
    fv[q] = h;
    gv[q] = y.flux ? ty * h : 0.f;
  }
}

// the background's face averages 0.5*(theta_bg,a + theta_bg,b) at the x and y edges, in FP64,
// kept as FP32 pairs (hi = the rounded value, lo = the rounded remainder)
__global__ void k_bg_faces(Dims D, Grid<double> G, float2* tbu, float2* tbv) {
  LG_IDX3;
  auto pair = [](double x) {
    const float hi = narrow(x);
    return make_float2(hi, narrow(x - wide(hi)));
  };
  if (ji <= D.ny && jk <= D.nx + 1) {
    const bool in = jk >= 2 && jk <= D.nx;
    if (in || D.periodic) {
      const int ka = in ? jk - 1 : D.nx, kb = in ? jk : 1;
      tbu[IX(D, ji, jk, jl)] = pair(0.5 * (G.theta_v_bg[IX(D, ji, ka, jl)] + G.theta_v_bg[IX(D, ji, kb, jl)]));
    }
  }
  if (ji <= D.ny + 1 && jk <= D.nx) {
    const bool in = ji >= 2 && ji <= D.ny;
    if (in || D.periodic) {
      const int ia = in ? ji : 1, ib = in ? ji - 1 : D.ny;
      tbv[IX(D, ji, jk, jl)] = pair(0.5 * (G.theta_v_bg[IX(D, ia, jk, jl)] + G.theta_v_bg[IX(D, ib, jk, jl)]));
    }
  }
}

// simple_dissipation_rate, mo_momentum_diff_diss.F90:333-389, split step: the swamp layer's
// dissipative heating -sum(rho(1:nc+1))*(W5 w(jl) d(jl) + W6 w(jl+1) d(jl+1)), d = w*kdamp the
// deceleration at w levels 2..n_damping_levels, in FP32 from the mirror (a heating term, as
// the radiation and sediment heating it is added to)
__global__ void ks_heating_diss(Dims D, Grid<float> GF, GridX X, StateF M, float* hd) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx || jl > D.nl) return;
  const long long q = IX(D, ji, jk, jl), b = q + D.plane;
  const float wa = M.w[q], wb = M.w[b];
  const float da = (jl >= 2 && jl <= D.ndamp) ? wa * X.kdamp_f[q] : 0.f;
  const float db = (jl + 1 <= D.ndamp) ? wb * X.kdamp_f[b] : 0.f;
  const float ip = GF.ipw[4][q] * wa * da + GF.ipw[5][q] * wb * db;
  hd[q] = -rho_sum_cond_gas<float, float>(D, M.rho, q) * ip;
}

// ---- column-marching divergences -------------------------------------------------------
// div_h with the contravariant vertical correction (div_h_at above: div_h,
// mo_divergence_operators.F90:16-68, and vertical_contravariant_corr, mo_averaging.F90:16-54)
// evaluated by one thread per column walking down the levels.  The correction at the
// interface between layers l-1 and l is -(h(l-1) + h(l)), h(l) being half the slope-weighted
// sum of layer l's four face values (only h(l) at the top interface of the terrain-following
// layers, l = nf+1).  Each layer's faces are loaded once per column, each h once, and each
// interface's correction serves the cells on both sides of it; the next layer's loads are
// issued before the current layer's result is stored.

// the four face values of layer l of column (ji, jk) -- x at the east (jk+1) and west (jk)
// u points, y at the north (ji) and south (ji+1) v points -- and h(l)
struct LayerFaces { float xe, yn, xw, ys, h; };

// h(l) of a layer whose four face values are set
__device__ __forceinline__ void layer_h(const Dims& D, const Grid<float>& G, LayerFaces& f, int ji, int jk, int l) {
  f.h = 0.f;
  if (l >= D.nf + 1) {
    const long long p = IX(D, ji, jk, l);
    f.h = 0.5f * f.xe * G.slope_x[IX(D, ji, jk + 1, l)] * G.ipw[0][p] + 0.5f * f.yn * G.slope_y[p] * G.ipw[1][p]
        + 0.5f * f.xw * G.slope_x[p] * G.ipw[2][p] + 0.5f * f.ys * G.slope_y[IX(D, ji + 1, jk, l)] * G.ipw[3][p];
  }
}

template <class FX, class FY>
__device__ __forceinline__ LayerFaces layer_faces(const Dims& D, const Grid<float>& G, FX fx, FY fy, int ji, int jk,
                                                  int l) {
  LayerFaces f;
  f.xe = fx(ji, jk + 1, l);
  f.yn = fy(ji, jk, l);
  f.xw = fx(ji, jk, l);
  f.ys = fy(ji + 1, jk, l);
  layer_h(D, G, f, ji, jk, l);
  return f;
}

// contravariant corrections at the upper (cu, interface jl) and lower (cl, interface jl+1)
// face of cell jl, and which of them the reference's branches use (mo_divergence_operators.F90:
// the top terrain-following layer nf has only its lower face, the lowest layer only its upper
// one unless it is layer nf itself)
struct VertFaces { float cu, cl; bool up, lo; };
__device__ __forceinline__ VertFaces vert_faces(const Dims& D, float h_prev, float h_cur, float h_next, int jl) {
  VertFaces v;
  v.up = jl > D.nf;
  v.lo = jl == D.nf || (jl > D.nf && jl < D.nl);
  v.cu = (jl == D.nf + 1) ? -h_cur : -(h_prev + h_cur);
  v.cl = (jl + 1 == D.nf + 1) ? -h_next : -(h_cur + h_next);
  return v;
}

// the divergence of cell jl from its layer's faces and the corrections of its two interfaces
__device__ __forceinline__ float div_col(const Dims& D, const Grid<float>& G, const GridX& X, const LayerFaces& c,
                                         const VertFaces& v, int ji, int jk, int jl) {
  const long long q = IX(D, ji, jk, jl);
  const float comp_h = c.xe * G.area_x[IX(D, ji, jk + 1, jl)] + c.yn * G.area_y[q] - c.xw * G.area_x[q]
                     - c.ys * G.area_y[IX(D, ji + 1, jk, jl)];
  float comp_v = 0.f;
  if (v.up) comp_v += v.cu * G.area_z[q];
  if (v.lo) comp_v -= v.cl * G.area_z[IX(D, ji, jk, jl + 1)];
  return (comp_h + comp_v) * X.inv_volume_f[q];
}

// the levels l0..l1 of a marching thread: the column cut into gridDim.z chunks of equal length
// (a chunk forms h of the layer above it anew, so every cell has the bits of a whole column's walk)
struct LevelChunk { int l0, l1; };
__device__ __forceinline__ LevelChunk level_chunk(const Dims& D) {
  const int len = (D.nl + (int)gridDim.z - 1) / (int)gridDim.z;
  return LevelChunk{(int)blockIdx.z * len + 1, min(D.nl, ((int)blockIdx.z + 1) * len)};
}

// div_h of a stored horizontal vector field (the third-order theta chain); blockIdx.z is the
// chunk of levels (level_chunks)
__global__ void __launch_bounds__(128) ks_div_h(Dims D, Grid<float> GF, GridX X, const float* vx, const float* vy,
                                                float* out) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const LevelChunk lc = level_chunk(D);
  auto fx = [&](int i, int j, int k) { return vx[IX(D, i, j, k)]; };
  auto fy = [&](int i, int j, int k) { return vy[IX(D, i, j, k)]; };
  LayerFaces cur = layer_faces(D, GF, fx, fy, ji, jk, lc.l0), nxt{};
  float h_prev = 0.f;
  if (lc.l0 - 1 >= D.nf + 1) h_prev = layer_faces(D, GF, fx, fy, ji, jk, lc.l0 - 1).h;
  for (int jl = lc.l0; jl <= lc.l1; ++jl) {
    nxt.h = 0.f;
    if (jl < D.nl || jl == D.nf) nxt = layer_faces(D, GF, fx, fy, ji, jk, jl + 1);
    out[IX(D, ji, jk, jl)] = div_col(D, GF, X, cur, vert_faces(D, h_prev, cur.h, nxt.h, jl), ji, jk, jl);
    h_prev = cur.h;
    cur = nxt;
  }
}

constexpr int kTracers = 6;  // moist: five condensates and water vapour (the gas has its own kernels)
// divergences of the gas and theta_v fluxes and the diabatic rho*theta_v term,
// mo_scalar_tend_expl.F90:106-177 (the gas has old_weight 0, new_weight 1), column-marching.  A layer's
// fluxes, metrics and heating rates are loaded two layers ahead, and what only a layer with heating needs
// (its temperature, densities and exner) one layer ahead, so that a layer waits for memory once:
// 1053 us at 768x768x80 with six resident blocks (five 1252, and 1680 with each layer's loads in its own
// turn), with cw 1145 us.
// TRACERS: also cw, the contravariant correction of the wind through the interfaces nf+1..nl times their
// area, for ks_tracers, from the slopes and weights that are here already.
struct GasLoads {  // fluxes through the faces (layer_faces' order), metrics, the layer's heating
  float f[4], t[4], u[4], area[4], slope[4], w[4], az, iv, heat;
};
struct GasLayer {  // of a layer: horizontal parts, half the slope-weighted sums, upper area
  float fh, th, fs, ts, us, az, iv, heat;
};
struct GasHeat {  // of a layer with heating
  float T, rho[kTracers + 1], exner;
};
template <bool TRACERS>
__global__ void __launch_bounds__(128, 6) ks_gas_div(Dims D, Grid<float> GF, GridX X, StateF Ss, const float* fu,
                                                  const float* fv, const float* gu, const float* gv, const float* Tm,
                                                  const float* hd, const float* rad, const float* csh, float* t_rho,
                                                  float* t_rt, const float* mdt, const float* tdh,
                                                  const float* ptr, const float* pth, const float* u_new,
                                                  const float* v_new, float* cw) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const LevelChunk lc = level_chunk(D);
  const long long goff = (long long)(D.g - 1) * D.fstride;
  auto load = [&](int l) {
    GasLoads R{};
    if (l > D.nl) return R;
    const long long p = IX(D, ji, jk, l), e = IX(D, ji, jk + 1, l), s = IX(D, ji + 1, jk, l);
    R.f[0] = fu[e]; R.f[1] = fv[p]; R.f[2] = fu[p]; R.f[3] = fv[s];
    R.t[0] = gu[e]; R.t[1] = gv[p]; R.t[2] = gu[p]; R.t[3] = gv[s];
    R.area[0] = GF.area_x[e]; R.area[1] = GF.area_y[p]; R.area[2] = GF.area_x[p]; R.area[3] = GF.area_y[s];
    if (l > D.nf) {
      R.slope[0] = GF.slope_x[e]; R.slope[1] = GF.slope_y[p]; R.slope[2] = GF.slope_x[p]; R.slope[3] = GF.slope_y[s];
#pragma unroll
      for (int k = 0; k < 4; ++k) R.w[k] = GF.ipw[k][p];
      R.az = GF.area_z[p];
      if constexpr (TRACERS) {
        R.u[0] = u_new[e]; R.u[1] = v_new[p]; R.u[2] = u_new[p]; R.u[3] = v_new[s];
      }
    }
    R.iv = X.inv_volume_f[p];
    R.heat = hd[p] + rad[p];                 // dissipative, radiative heating
    if (pth) R.heat = R.heat + pth[p];       // phase transitions
    R.heat = R.heat + csh[p];                // sediment heating
    if (tdh) R.heat = R.heat + tdh[p];       // temperature diffusion
    return R;
  };
  auto reduce = [&](const GasLoads& R, int l) {
    GasLayer L;
    auto hor = [&](const float* f) {
      return fmaf(-f[3], R.area[3], fmaf(-f[2], R.area[2], fmaf(f[0], R.area[0], f[1] * R.area[1])));
    };
    L.fh = hor(R.f);
    L.th = hor(R.t);
    auto slopes = [&](const float* v) {
      return fmaf(0.5f * v[3] * R.slope[3], R.w[3],
                  fmaf(0.5f * v[2] * R.slope[2], R.w[2],
                       fmaf(0.5f * v[0] * R.slope[0], R.w[0], 0.5f * v[1] * R.slope[1] * R.w[1])));
    };
    L.fs = l > D.nf ? slopes(R.f) : 0.f;
    L.ts = l > D.nf ? slopes(R.t) : 0.f;
    L.us = TRACERS && l > D.nf ? slopes(R.u) : 0.f;
    L.az = R.az;
    L.iv = R.iv;
    L.heat = R.heat;
    return L;
  };
  auto heat_loads = [&](const GasLayer& L, int l) {
    GasHeat H{};
    if (l <= D.nl && L.heat != 0.f) {
      const long long p = IX(D, ji, jk, l);
      H.T = Tm[p];
#pragma unroll
      for (int k = 0; k < kTracers + 1; ++k)
        if (k < D.ncons) H.rho[k] = Ss.rho[p + (long long)k * D.fstride];
      H.exner = GF.exner_bg[p] + Ss.ep[p];
    }
    return H;
  };
  float fs_prev = 0.f, ts_prev = 0.f;
  if (lc.l0 - 1 >= D.nf + 1) {
    const GasLayer P = reduce(load(lc.l0 - 1), lc.l0 - 1);
    fs_prev = P.fs;
    ts_prev = P.ts;
  }
  GasLoads R = load(lc.l0 + 1);
  GasLayer cur = reduce(load(lc.l0), lc.l0);
  GasHeat H = heat_loads(cur, lc.l0);
  for (int jl = lc.l0; jl <= lc.l1; ++jl) {
    const long long q = IX(D, ji, jk, jl);
    const GasLayer nxt = reduce(R, jl + 1);
    if (jl < lc.l1) R = load(jl + 2);
    const GasHeat Hn = heat_loads(nxt, jl + 1);
    const VertFaces vm = vert_faces(D, fs_prev, cur.fs, nxt.fs, jl), vt = vert_faces(D, ts_prev, cur.ts, nxt.ts, jl);
    float cm = 0.f, ct = 0.f;
    if (vm.up) {
      cm += vm.cu * cur.az;
      ct += vt.cu * cur.az;
    }
    if (vm.lo) {
      cm -= vm.cl * nxt.az;
      ct -= vt.cl * nxt.az;
    }
    if (TRACERS && vm.lo) cw[q + D.plane] = ((jl == D.nf) ? -nxt.us : -(cur.us + nxt.us)) * nxt.az;
    const float div_m = (cur.fh + cm) * cur.iv, div_t = (cur.th + ct) * cur.iv;
    float x = 0.f;
    if (cur.heat != 0.f) {
      float cv = 0.f, rg;  // c_v_mass_weighted_air, mo_derived.F90:157-187
      if (D.lmoist) {
#pragma unroll
        for (int jc = 1; jc < kTracers; ++jc) cv = cv + H.rho[jc - 1] * c_p_cond(jc, H.T);
        cv = cv + (H.rho[kTracers - 1] - H.rho[kTracers]) * float(kC_D_V);
        cv = cv + H.rho[kTracers] * float(kC_V_V);
        rg = H.rho[kTracers - 1];
      } else {
        rg = H.rho[0];
        cv = rg * float(kC_D_V);
      }
      x = float(kC_D_V) * rg / cv * cur.heat / (float(kC_D_P) * H.exner);
    }
    if (ptr) {  // phase transitions' vapour rate and mass diffusion of the gas
      const float mdg = mdt ? mdt[q + goff] : 0.f, ptg = ptr[q + goff];
      t_rho[q + goff] = -div_m + mdg + ptg;
      t_rt[q] = -div_t + x + (ptg + mdg) * (GF.theta_v_bg[q] + Ss.tp[q]);
    } else if (mdt) {  // mass diffusion of the gas, in its tendency and times theta_v in rho*theta_v's
      const float mdg = mdt[q + goff];
      t_rho[q + goff] = -div_m + mdg;
      t_rt[q] = -div_t + x + mdg * (GF.theta_v_bg[q] + Ss.tp[q]);
    } else {
      t_rho[q + goff] = -div_m;
      t_rt[q] = -div_t + x;
    }
    fs_prev = cur.fs;
    ts_prev = cur.ts;
    cur = nxt;
    H = Hn;
  }
}

// scalar_tend_expl for the tracers, mo_scalar_tend_expl.F90:24-104 (upstream fluxes,
// mo_scalar_tend_expl.F90:56-82; vertical upstream term with the contravariant correction,
// mo_averaging.F90:16-54, whose product with the area ks_gas_div left in cw), split step.  The
// velocities through the six faces of the cell, times the face areas, and the indices of the
// faces' upwind cells are found once per cell; the tracer loop then only loads densities at known
// addresses, and every tracer's divergence is formed before the first tendency is stored, so no load
// waits on an earlier store.  The first substep (new weight 1) does not read the old tendency.
// 873 us at 768x768x80 with six resident blocks (five 918, four 951).  Forming the corrections here took
// half of the kernel's loads (1687 us); a column-marching form keeps too many values a tracer (1839 us).
__global__ void __launch_bounds__(256, 6) ks_tracers(Dims D, Grid<float> GF, GridX X, StateF Ss, const float* u_new,
                                                     const float* v_new, const float* cw, float* t_rho, int rk_step,
                                                     const float* mdt, const float* ptr) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl);
  // horizontal faces: flux = rho(upwind cell) * velocity, 0 on a non-periodic boundary; the periodic
  // wrap edges take the velocity at the first edge
  const Edge w = edge_x(D, ji, jk, jl), e = edge_x(D, ji, jk + 1, jl), n = edge_y(D, ji, jk, jl), so = edge_y(D, ji + 1, jk, jl);
  const bool up = jl > D.nf, lo = jl >= D.nf && jl < D.nl;  // the interfaces of the terrain-following layers
  const float ue = u_new[e.b], uw = u_new[w.b], vn = v_new[n.b], vs = v_new[so.b];
  const float ae = GF.area_x[e.q], aw = GF.area_x[w.q], an = GF.area_y[n.q], as = GF.area_y[so.q];
  float a_u = 0.f, a_l = 0.f;
  if (up) a_u = cw[q];
  if (lo) a_l = cw[q + D.plane];
  const float a_e = e.flux ? ue * ae : 0.f, a_w = w.flux ? uw * aw : 0.f;
  const float a_n = n.flux ? vn * an : 0.f, a_s = so.flux ? vs * as : 0.f;
  const long long i_e = ue >= 0.f ? e.a : e.b, i_w = uw >= 0.f ? w.a : w.b;
  const long long i_n = vn >= 0.f ? n.b : n.a, i_s = vs >= 0.f ? so.b : so.a;
  const long long i_u = up && a_u <= 0.f ? q - D.plane : q, i_l = lo && a_l > 0.f ? q + D.plane : q;
  const float iv = X.inv_volume_f[q];
  float dv[kTracers];
#pragma unroll
  for (int t = 0; t < kTracers; ++t) {
    const int jc = t + 1 + (t + 1 >= D.g ? 1 : 0);
    const float* r = Ss.rho + (long long)(jc - 1) * D.fstride;
    const float hor = fmaf(-r[i_s], a_s, fmaf(-r[i_w], a_w, fmaf(r[i_e], a_e, r[i_n] * a_n)));
    dv[t] = fmaf(-r[i_l], a_l, fmaf(r[i_u], a_u, hor)) * iv;
  }
  if (mdt) {  // mass diffusion: -div + mass_diff_tendency
#pragma unroll
    for (int t = 0; t < kTracers; ++t) {
      const int jc = t + 1 + (t + 1 >= D.g ? 1 : 0);
      dv[t] = dv[t] - mdt[q + (long long)(jc - 1) * D.fstride];
    }
  }
  if (ptr) {  // phase transitions: the condensates' own rates, vapour's rate nc+1
#pragma unroll
    for (int t = 0; t < kTracers; ++t) {
      const int jc = t + 1 + (t + 1 >= D.g ? 1 : 0);
      dv[t] = dv[t] - ptr[q + (long long)((jc < D.g ? jc : D.g) - 1) * D.fstride];
    }
  }
  if (rk_step == 1) {
#pragma unroll
    for (int t = 0; t < kTracers; ++t) {
      const int jc = t + 1 + (t + 1 >= D.g ? 1 : 0);
      t_rho[q + (long long)(jc - 1) * D.fstride] = -dv[t];
    }
  } else {
    float o[kTracers];
#pragma unroll
    for (int t = 0; t < kTracers; ++t) {
      const int jc = t + 1 + (t + 1 >= D.g ? 1 : 0);
      o[t] = t_rho[q + (long long)(jc - 1) * D.fstride];
    }
#pragma unroll
    for (int t = 0; t < kTracers; ++t) {
      const int jc = t + 1 + (t + 1 >= D.g ? 1 : 0);
      t_rho[q + (long long)(jc - 1) * D.fstride] = 0.5f * o[t] - 0.5f * dv[t];
    }
  }
}

// ---- potential vorticity and its flux, marching down the levels ------------------------------
// A thread walks a chunk of levels of one plane point (ji, jk).  Everything a level reads is loaded
// before anything is stored, at addresses that are valid everywhere (the edge kernels' reason), and what two
// levels share is carried.  The periodic copies at ny+1 and nx+1 evaluate the point they copy.
struct Around {  // the point (I, K) evaluated and its neighbours' plane offsets at level 1
  int I, K;
  bool fi, fk;  // not a non-periodic boundary row, column
  long long c, n, s, w, e, nw, sw, se, ne;
};
__device__ __forceinline__ Around around(const Dims& D, int ji, int jk) {
  Around A;
  A.fi = D.periodic || (ji >= 2 && ji <= D.ny);
  A.fk = D.periodic || (jk >= 2 && jk <= D.nx);
  A.I = D.periodic && ji == D.ny + 1 ? 1 : ji;
  A.K = D.periodic && jk == D.nx + 1 ? 1 : jk;
  const int im = A.I == 1 ? D.ny : A.I - 1, km = A.K == 1 ? D.nx : A.K - 1;
  const int ip = min(A.I + 1, D.ny + 1), kp = min(A.K + 1, D.nx + 1);
  A.c = IX(D, A.I, A.K, 1);
  A.n = IX(D, im, A.K, 1);
  A.s = IX(D, ip, A.K, 1);
  A.w = IX(D, A.I, km, 1);
  A.e = IX(D, A.I, kp, 1);
  A.nw = IX(D, im, km, 1);
  A.sw = IX(D, ip, km, 1);
  A.se = IX(D, ip, kp, 1);
  A.ne = IX(D, im, kp, 1);
  return A;
}

// grad_vert and grad_hor, mo_gradient_operators.F90:17-130, S the type of the scalar (FP64: the kinetic
// energy; its differences are taken in FP64 and rounded).  The vertical gradients at the interfaces of an
// edge's cells are formed here and carried; with VERT they are kept too (levels 2..nl of rz, whose first
// and surface levels, which no operator writes, are read as they are).  One kernel for the two, which wrote
// and read the vertical gradient in between: 3.31 -> 2.38 ms for the three of a step at 1024x1024x80.
template <class S, bool VERT>
__global__ void __launch_bounds__(128) ks_grad(Dims D, Grid<float> G, const S* s, float* rx, float* ry, float* rz) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny + 1 || jk > D.nx + 1) return;
  const LevelChunk lc = level_chunk(D);
  if (lc.l0 > D.nl) return;
  const Around A = around(D, ji, jk);
  const bool px = jk <= D.nx, py = ji <= D.ny;
  const long long pl = D.plane, q1 = IX(D, ji, jk, 1);
  const long long p[3] = {A.c, A.n, A.w};
  long long o = (long long)(lc.l0 - 1) * pl;
  S t[3];
  float g[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    t[m] = s[p[m] + o];
    g[m] = lc.l0 > 1 ? cvt<float>(s[p[m] + o - pl] - t[m]) / G.dz[p[m] + o] : VERT ? rz[p[m]] : 0.f;
  }
  for (int l = lc.l0; l <= lc.l1; ++l, o += pl) {
    const bool below = l < D.nl;
    S tn[3];
    float dz[3], w5[3], w6[3], gn[3], sx = 0.f, sy = 0.f;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      tn[m] = s[p[m] + (below ? o + pl : o)];
      dz[m] = below ? G.dz[p[m] + o + pl] : (VERT ? rz[p[m] + o + pl] : 0.f);
    }
    const float dx = G.dx[A.c + o], dy = G.dy[A.c + o];
    if (l > D.nf) {
#pragma unroll
      for (int m = 0; m < 3; ++m) {
        w5[m] = G.ipw[4][p[m] + o];
        w6[m] = G.ipw[5][p[m] + o];
      }
      sx = G.slope_x[q1 + o];
      sy = G.slope_y[q1 + o];
    }
#pragma unroll
    for (int m = 0; m < 3; ++m) gn[m] = below ? cvt<float>(t[m] - tn[m]) / dz[m] : dz[m];
    float x = cvt<float>(t[0] - t[2]) / dx, y = cvt<float>(t[1] - t[0]) / dy;
    if (l > D.nf) {
      float mx = w5[2] * g[2] + w5[0] * g[0], my = w5[1] * g[1] + w5[0] * g[0];
      if (below || D.freeslip) {
        mx = mx + w6[2] * gn[2] + w6[0] * gn[0];
        my = my + w6[1] * gn[1] + w6[0] * gn[0];
      }
      x = x - sx * (0.5f * mx);
      y = y - sy * (0.5f * my);
    }
    const long long q = q1 + o;
    if (py && A.fk) rx[q] = x;
    if (px && A.fi) ry[q] = y;
    if (VERT && px && py && l > 1) rz[q] = g[0];
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      t[m] = tn[m];
      g[m] = gn[m];
    }
  }
}

// calc_pot_vort (mo_vorticities.F90:19-421, with rel_vort and rel_vort_z_local) and the mass flux
// densities (mo_vector_tend_expl.F90:64-66).  Carried from level to level: the winds and heights at the
// dual point's four sides, w, the products length times covariant wind of the x and y vorticity, and the
// sums of the density.  One quotient a component, (zeta + f*A)/(A*rho), zeta before its division by the dual
// area A; the rescaled length (r_e + zd)/(r_e + z) of a dual point's side as 1 + (zd - z)/(r_e + z), since
// r_e + z has half a metre's resolution in FP32.  The last block in z does ex and ey at level 1 and at the
// surface, whose formulas are their own.  A thread a point, each term with its own branches, loads and
// quotients, took 3.37 ms at 1024x1024x80; so 1.80 ms (1.03 ms of memory traffic at the copy rate).
__global__ void __launch_bounds__(128, 4) ks_eta(Dims D, Grid<float> G, StateF S, float* ex, float* ey, float* ez,
                                                 float* uph, float* vph, float* wph) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny + 1 || jk > D.nx + 1) return;
  const bool px = jk <= D.nx, py = ji <= D.ny;
  const int chunks = (int)gridDim.z - 1;
  if ((int)blockIdx.z == chunks) {
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
      const int jl = k ? D.NL : 1;
      if (px) ex[IX(D, ji, jk, jl)] = eta_x_at<float>(D, G, S, ji, jk, jl);
      if (py) ey[IX(D, ji, jk, jl)] = eta_y_at<float>(D, G, S, ji, jk, jl);
    }
    return;
  }
  const int len = (D.nl + chunks - 1) / chunks, l0 = (int)blockIdx.z * len + 1, l1 = min(D.nl, l0 + len - 1);
  const Around A = around(D, ji, jk);
  const float* rg = S.rho + (long long)(D.g - 1) * D.fstride;
  const long long pl = D.plane, q1 = IX(D, ji, jk, 1);
  const bool zeta = !D.llinear;
  const float fx = D.lcorio ? G.fvec_x[A.c] : 0.f, fy = D.lcorio ? G.fvec_y[A.c] : 0.f, fz = D.lcorio ? G.fvec_z[A.c] : 0.f;
  // the dual point's sides: v at (I,K), u at (im,K), v at (I,km), u at (I,K); wind and height at the
  // level above, here and below
  float ua[4], ub[4], uc[4], za[4], zb[4], zc[4];
  auto sides = [&](long long o, float* u, float* z) {
    u[0] = S.v[A.c + o]; u[1] = S.u[A.n + o]; u[2] = S.v[A.w + o]; u[3] = S.u[A.c + o];
    z[0] = G.z_v[A.c + o]; z[1] = G.z_u[A.n + o]; z[2] = G.z_v[A.w + o]; z[3] = G.z_u[A.c + o];
  };
  struct W { float c, n, w; };
  auto cells = [&](const float* p, long long o) { return W{p[A.c + o], p[A.n + o], p[A.w + o]}; };
  // dx (dy) times the covariant wind at the u (v) point of layer l, horizontal_covariant_x/y
  // (mo_averaging.F90:56-176): wu, wl are w at the layer's upper and lower interface
  struct Cov { float x, y; };
  auto covariant = [&](int l, long long o, float u, float v, float dx, float dy, const W& wu, const W& wl) {
    Cov r{dx * u, dy * v};
    if (l > D.nf) {
      const W w5 = cells(G.ipw[4], o), w6 = cells(G.ipw[5], o);
      const float sx = G.slope_x[A.c + o], sy = G.slope_y[A.c + o];
      float mx = w5.w * wu.w + w5.c * wu.c, my = w5.n * wu.n + w5.c * wu.c;
      if (l < D.nl || D.freeslip) {
        mx = mx + w6.w * wl.w + w6.c * wl.c;
        my = my + w6.n * wl.n + w6.c * wl.c;
      }
      r.x = dx * (u + sx * (0.5f * mx));
      r.y = dy * (v + sy * (0.5f * my));
    }
    return r;
  };
  long long o = (long long)(l0 - 1) * pl;
  W w0 = cells(S.w, o);
  sides(o, ub, zb);
#pragma unroll
  for (int m = 0; m < 4; ++m) { ua[m] = ub[m]; za[m] = zb[m]; }
  Cov cp{0.f, 0.f};
  float rx = 0.f, ry = 0.f, rc0 = 0.f;  // density of the layer above: the u (v) point's two cells, the cell
  if (l0 > 1) {
    const long long a = o - pl;
    sides(a, ua, za);
    const W wa = cells(S.w, a), r = cells(rg, a);
    cp = covariant(l0 - 1, a, ua[3], ua[0], G.dx[A.c + a], G.dy[A.c + a], wa, w0);
    rx = r.w + r.c;
    ry = r.n + r.c;
    rc0 = r.c;
  }
  for (int l = l0; l <= l1; ++l, o += pl) {
    sides(o + pl, uc, zc);  // below the lowest layer: the padding level, not used
    const W w1 = cells(S.w, o + pl), r = cells(rg, o), dz = cells(G.dz, o);
    const float rnw = rg[A.nw + o], zd = G.z_area_dual_z[A.c + o];
    const float dxc = G.dx[A.c + o], dxn = G.dx[A.n + o], dyc = G.dy[A.c + o], dyw = G.dy[A.w + o];
    const float ax = G.area_dual_x[A.c + o], ay = G.area_dual_y[A.c + o], az = G.area_dual_z[A.c + o];
    const Cov cv = covariant(l, o, ub[3], ub[0], dxc, dyc, w0, w1);
    const float length[4] = {dyc, -dxn, -dyw, dxc};
    float zz = 0.f;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      if (l <= D.nf) {
        zz += apart(length[m], ub[m]);
      } else {
        const float d = zd - zb[m];
        const bool up = (d > 0.f || l == D.nl) && l > 1;
        const float zs = up ? za[m] : zc[m], us = up ? ua[m] : uc[m];
        const float rescaled = fmaf(length[m], d / (float(kR_E) + zb[m]), length[m]);
        zz += apart(rescaled, ub[m] + (ub[m] - us) * (d / (zb[m] - zs)));
      }
    }
    if (!zeta) zz = 0.f;
    const float ez_ = A.fi && A.fk ? (zz + fz * az) / (az * (0.25f * (r.w + r.c + r.n + rnw))) : fz;
    float ex_ = 0.f, ey_ = 0.f;
    if (l > 1) {
      const float zx = zeta ? apart(dz.n, w0.n) - cp.y - apart(dz.c, w0.c) + cv.y : 0.f;
      const float zy = zeta ? apart(dz.w, w0.w) + cp.x - apart(dz.c, w0.c) - cv.x : 0.f;
      ex_ = A.fi ? (zx + fx * ax) / (ax * (0.25f * (ry + r.n + r.c))) : fx;
      ey_ = A.fk ? (zy + fy * ay) / (ay * (0.25f * (rx + r.w + r.c))) : fy;
    }
    const long long q = q1 + o;
    ez[q] = ez_;
    if (l > 1 && px) ex[q] = ex_;
    if (l > 1 && py) ey[q] = ey_;
    if (py && A.fk) uph[q] = 0.5f * (r.w + r.c) * ub[3];
    if (px && A.fi) vph[q] = 0.5f * (r.n + r.c) * ub[0];
    if (l > 1 && px && py) wph[q] = 0.5f * (rc0 + r.c) * w0.c;
    cp = cv;
    w0 = w1;
    rx = r.w + r.c;
    ry = r.n + r.c;
    rc0 = r.c;
#pragma unroll
    for (int m = 0; m < 4; ++m) { ua[m] = ub[m]; ub[m] = uc[m]; za[m] = zb[m]; zb[m] = zc[m]; }
  }
}

// calc_vorticity_flux_term, mo_vorticity_flux.F90:16-171.  Carried from level to level: the vertical mass
// flux, eta_x and eta_y at the interface between, and the products weight times horizontal mass flux of the layer
// above, which the vertical component adds to this layer's before the vorticity multiplies both.
// 1.92 -> 1.18 ms at 1024x1024x80 against a thread a point (0.74 ms of memory traffic).
__global__ void __launch_bounds__(128, 4) ks_vort_flux(Dims D, Grid<float> G, StateF S, const float* ex,
                                                       const float* ey, const float* ez, const float* uph,
                                                       const float* vph, const float* wph, float* px, float* py,
                                                       float* pz) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny + 1 || jk > D.nx + 1) return;
  const LevelChunk lc = level_chunk(D);
  if (lc.l0 > D.nl) return;
  const Around A = around(D, ji, jk);
  const bool out_x = ji <= D.ny && A.fk, out_y = jk <= D.nx && A.fi, cell = ji <= D.ny && jk <= D.nx;
  const long long pl = D.plane, q1 = IX(D, ji, jk, 1);
  const int row = min(A.I, D.ny) - 1;
  const float u1 = 0.25f * G.trsk_u[0][row], u2 = 0.25f * G.trsk_u[1][row], u3 = 0.25f * G.trsk_u[2][row];
  const float v1 = 0.25f * G.trsk_v[0][row], v2 = 0.25f * G.trsk_v[1][row];
  // vertical mass flux at the surface: free slip, mo_vector_tend_expl.F90:68-80
  auto surface = [&](long long p1) {
    if (!D.freeslip) return 0.f;
    const float* rg = S.rho + (long long)(D.g - 1) * D.fstride;
    const long long b = p1 + (long long)(D.nl - 1) * pl, a = b - pl;
    const float dv = rg[b] + (rg[a] - rg[b]) / (G.z_scalar[a] - G.z_scalar[b]) * (G.z_w[b + pl] - G.z_scalar[b]);
    return dv * S.w[b + pl];
  };
  long long o = (long long)(lc.l0 - 1) * pl;
  float wc = wph[A.c + o], wn = wph[A.n + o], ww = wph[A.w + o], xc = ex[A.c + o], yc = ey[A.c + o];
  float fe = 0.f, fn = 0.f, fw = 0.f, fs = 0.f;  // weight times flux through the layer above's faces
  if (lc.l0 > 1) {
    const long long a = A.c + o - pl;
    fe = G.ipw[0][a] * uph[A.e + o - pl];
    fn = G.ipw[1][a] * vph[a];
    fw = G.ipw[2][a] * uph[a];
    fs = G.ipw[3][a] * vph[A.s + o - pl];
  }
  for (int l = lc.l0; l <= lc.l1; ++l, o += pl) {
    const float uc = uph[A.c + o], uw = uph[A.w + o], ue = uph[A.e + o], un = uph[A.n + o], une = uph[A.ne + o];
    const float vc = vph[A.c + o], vw = vph[A.w + o], vs = vph[A.s + o], vsw = vph[A.sw + o];
    const float zc = ez[A.c + o], zn = ez[A.n + o], zs = ez[A.s + o], zw = ez[A.w + o], ze = ez[A.e + o];
    const float zsw = ez[A.sw + o], zse = ez[A.se + o], zne = ez[A.ne + o];
    const float w1 = G.ipw[0][A.c + o], w2 = G.ipw[1][A.c + o], w3 = G.ipw[2][A.c + o], w4 = G.ipw[3][A.c + o];
    const float w5c = G.ipw[4][A.c + o], w5n = G.ipw[4][A.n + o], w5w = G.ipw[4][A.w + o];
    const float w6c = G.ipw[5][A.c + o], w6n = G.ipw[5][A.n + o], w6w = G.ipw[5][A.w + o];
    const float ye = ey[A.e + o], xs = ex[A.s + o], xd = ex[A.c + o + pl], yd = ey[A.c + o + pl];
    float dc, dn, dw;
    if (l < D.nl) {
      dc = wph[A.c + o + pl];
      dn = wph[A.n + o + pl];
      dw = wph[A.w + o + pl];
    } else {
      dc = surface(A.c);
      dn = surface(A.n);
      dw = surface(A.w);
    }
    // the TRSK terms, mo_vorticity_flux.F90:33-45, :72-80
    const float cs = zc + zs, ce = zc + ze;
    const float tx = u1 * vw * (zw + zc + cs) + u2 * uw * (zw + zsw + cs) + u3 * vsw * (zsw + zs + cs)
                   + u3 * vs * (zs + zse + cs) + u2 * ue * (zse + ze + cs) + u1 * vc * (zc + ze + cs);
    const float ty = v1 * uc * (zc + zs + ce) + v1 * ue * (ze + zse + ce) + v2 * une * (zne + ze + ce)
                   + v2 * un * (zn + zc + ce);
    const float rx = tx - 0.5f * (w5w * ww + w5c * wc) * yc - 0.5f * (w6w * dw + w6c * dc) * yd;
    const float ry = ty + 0.5f * (w5n * wn + w5c * wc) * xc + 0.5f * (w6n * dn + w6c * dc) * xd;
    const float ge = w1 * ue, gn = w2 * vc, gw = w3 * uc, gs = w4 * vs;
    const float rz = 0.5f * ((fe + ge) * ye - (fn + gn) * xc + (fw + gw) * yc - (fs + gs) * xs);
    const long long q = q1 + o;
    if (out_x) px[q] = rx;
    if (out_y) py[q] = ry;
    if (cell && l > 1) pz[q] = rz;
    wc = dc; wn = dn; ww = dw; xc = xd; yc = yd;
    fe = ge; fn = gn; fw = gw; fs = gs;
  }
}

// ---- update_n_squared and tke_update of the diffusion closure -----------------------------------
// (mo_eff_diff_coeffs.F90:620-669, mo_tke.F90:19-66; diffusion.cuh says what the reference's work arrays
// hold), marching like ks_eta: the vertical gradients of the TKE at the interfaces of the cell and its
// four neighbours are formed once and carried, and so are theta_v and its part of n_squared.  Reads the old
// TKE, viscosity and heating_diss; writes tke_new (neighbours still read the old one) and n_squared.
// A thread a cell formed the gradients at each of its four faces anew: 3.11 -> 1.52 ms at 1024x1024x80.
__global__ void __launch_bounds__(128, 4) ks_diff_tke(Dims D, Grid<float> G, StateF S, DiffBuf<float> B, DiffPar P) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const LevelChunk lc = level_chunk(D);
  if (lc.l0 > D.nl) return;
  // the cell, then its west, east, north and south neighbours (across the periodic edges), and whether the
  // edge towards them is a non-periodic boundary's, whose gradient is 0
  const bool per = D.periodic;
  const long long pl = D.plane, q1 = IX(D, ji, jk, 1);
  const long long p1[5] = {q1, IX(D, ji, jk == 1 ? D.nx : jk - 1, 1), IX(D, ji, jk == D.nx ? 1 : jk + 1, 1),
                           IX(D, ji == 1 ? D.ny : ji - 1, jk, 1), IX(D, ji == D.ny ? 1 : ji + 1, jk, 1)};
  const bool in_w = per || jk > 1, in_e = per || jk < D.nx, in_n = per || ji > 1, in_s = per || ji < D.ny;
  const long long e1 = q1 + D.P, s1 = q1 + 1;  // the east u point, the south v point
  const float* rg = S.rho + (long long)(D.g - 1) * D.fstride;
  const float decay = float(8.0 * (kPI * kPI)) / float(P.mva);
  auto theta = [&](long long p) { return G.theta_v_bg[p] + S.tp[p]; };
  long long o = (long long)(lc.l0 - 1) * pl;
  // t: TKE of layer l; g: its gradient at the layer's upper interface, 0 at the top
  float t[5], g[5], th = theta(q1 + o), nz = 0.f, w = S.w[q1 + o];
#pragma unroll
  for (int m = 0; m < 5; ++m) {
    t[m] = B.tke[p1[m] + o];
    g[m] = 0.f;
  }
  // g*0.5*(1/theta(l-1) + 1/theta(l))*dtheta/dz at the interface p between theta_v a and b
  auto n_squared = [&](long long p, float a, float b, float dz) {
    return G.gm[p] * (0.5f * (1.f / a + 1.f / b) * ((a - b) / dz));
  };
  if (lc.l0 > 1) {
#pragma unroll
    for (int m = 0; m < 5; ++m) g[m] = (B.tke[p1[m] + o - pl] - t[m]) / G.dz[p1[m] + o];
    nz = n_squared(q1 + o, theta(q1 + o - pl), th, G.dz[q1 + o]);
  }
  for (int l = lc.l0; l <= lc.l1; ++l, o += pl) {
    const bool below = l < D.nl;
    const long long d = below ? o + pl : o;
    float tn[5], dz[5], w5[5], w6[5], gn[5], h[5], sw = 0.f, se = 0.f, sn = 0.f, ss = 0.f;
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      tn[m] = B.tke[p1[m] + d];
      dz[m] = G.dz[p1[m] + d];
      w5[m] = m == 0 || l > D.nf ? G.ipw[4][p1[m] + o] : 0.f;
      w6[m] = m == 0 || l > D.nf ? G.ipw[5][p1[m] + o] : 0.f;
    }
    if (l > D.nf) {
      sw = G.slope_x[q1 + o];
      se = G.slope_x[e1 + o];
      sn = G.slope_y[q1 + o];
      ss = G.slope_y[s1 + o];
    }
    const long long q = q1 + o;
    const float dxw = G.dx[q], dxe = G.dx[p1[2] + o], dyn = G.dy[q], dys = G.dy[p1[4] + o];
    const float w1 = G.ipw[0][q], w2 = G.ipw[1][q], w3 = G.ipw[2][q], w4 = G.ipw[3][q];
    const float ue = S.u[e1 + o], uw = S.u[q], vn = S.v[q], vs = S.v[s1 + o], wn = S.w[q + pl];
    const float visc = B.visc[q], rho = rg[q], hd = B.hd[q], thn = theta(q1 + d), gm = G.gm[q1 + d];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      gn[m] = below ? (t[m] - tn[m]) / dz[m] : 0.f;
      h[m] = w5[m] * g[m] + w6[m] * gn[m];  // the column's part of the remap to its faces
    }
    const float nzn = below ? gm * (0.5f * (1.f / th + 1.f / thn) * ((th - thn) / dz[0])) : 0.f;
    const float gw = in_w ? (t[0] - t[1]) / dxw - sw * (0.5f * (h[1] + h[0])) : 0.f;
    const float ge = in_e ? (t[2] - t[0]) / dxe - se * (0.5f * (h[0] + h[2])) : 0.f;
    const float gN = in_n ? (t[3] - t[0]) / dyn - sn * (0.5f * (h[3] + h[0])) : 0.f;
    const float gS = in_s ? (t[0] - t[4]) / dys - ss * (0.5f * (h[0] + h[4])) : 0.f;
    const float adv = w1 * ue * ge + w2 * vn * gN + w3 * uw * gw + w4 * vs * gS + w5[0] * w * g[0] + w6[0] * wn * gn[0];
    const float r = t[0] + float(D.dtime) * (-adv + hd / rho - decay * visc / rho * t[0]);
    B.nsq[q] = l == 1 || l == D.nl ? 0.f : w5[0] * nz + w6[0] * nzn;
    B.tke_new[q] = r < 0.f ? 0.f : r;
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      t[m] = tn[m];
      g[m] = gn[m];
    }
    th = thn;
    nz = nzn;
    w = wn;
  }
}

// hor_viscosity (k_diff_visc, diffusion.cuh) with the divergence of the wind formed as in ks_div_h: 2.14 ->
// 1.13 ms at 1024x1024x80
__global__ void __launch_bounds__(128) ks_diff_visc(Dims D, Grid<float> G, GridX X, StateF S, const float* Tm,
                                                    DiffBuf<float> B, DiffPar P) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const LevelChunk lc = level_chunk(D);
  if (lc.l0 > D.nl) return;
  auto fx = [&](int i, int j, int k) { return S.u[IX(D, i, j, k)]; };
  auto fy = [&](int i, int j, int k) { return S.v[IX(D, i, j, k)]; };
  const float* rho = S.rho + (long long)(D.g - 1) * D.fstride;
  LayerFaces cur = layer_faces(D, G, fx, fy, ji, jk, lc.l0), nxt{};
  float h_prev = 0.f;
  if (lc.l0 - 1 >= D.nf + 1) h_prev = layer_faces(D, G, fx, fy, ji, jk, lc.l0 - 1).h;
  for (int jl = lc.l0; jl <= lc.l1; ++jl) {
    const long long q = IX(D, ji, jk, jl);
    const float rg = rho[q], t = Tm[q], tke = B.tke_new[q];
    float vac = 0.f;
    if (!P.tke_h) vac = 0.25f * (B.zz[q] + B.zz[q + D.P] + B.zz[q + 1] + B.zz[q + D.P + 1]);
    nxt.h = 0.f;
    if (jl < D.nl || jl == D.nf) nxt = layer_faces(D, G, fx, fy, ji, jk, jl + 1);
    const float dv = div_col(D, G, X, cur, vert_faces(D, h_prev, cur.h, nxt.h, jl), ji, jk, jl);
    const float vmol = diff_coeff_t<float>(t, rg);
    float eddy;
    if (P.tke_h) {
      eddy = tke2hor<float>(P, tke);
    } else {
      const float a = vac * vac + dv * dv, b = float(P.bg_shear) * float(P.bg_shear);
      eddy = float(P.c_s) * float(P.mva) * sqrtf(a > b ? a : b);
    }
    const float visc = rg * (vmol + eddy);
    B.vmol[q] = vmol;
    B.visc[q] = visc;
    B.vdiv[q] = visc * dv;
    B.tke[q] = tke;
    h_prev = cur.h;
    cur = nxt;
  }
}

// mom_diff_h (mo_momentum_diff_diss.F90:25-160; k_mom_diff_h, diffusion.cuh), marching like ks_eta: the
// dual points' viscosity times vorticity and heights, and the w points' accelerations, are carried: 2.32 ->
// 1.95 ms at 1024x1024x80.
__global__ void __launch_bounds__(128, 5) ks_mom_diff_h(Dims D, Grid<float> G, StateF S, DiffBuf<float> B) {
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const LevelChunk lc = level_chunk(D);
  if (lc.l0 > D.nl) return;
  const bool in_x = D.periodic || jk >= 2, in_y = D.periodic || ji >= 2;
  const long long pl = D.plane, c1 = IX(D, ji, jk, 1), w1 = IX(D, ji, jk >= 2 ? jk - 1 : D.nx, 1),
                  n1 = IX(D, ji >= 2 ? ji - 1 : D.ny, jk, 1);
  const long long d1[3] = {c1, c1 + 1, c1 + D.P};  // dual points (ji, jk), (ji+1, jk), (ji, jk+1)
  const long long x1 = IX(D, ji, D.nx + 1, 1), y1 = IX(D, D.ny + 1, jk, 1);
  const float* zd = G.z_area_dual_z;
  struct W { float c, w, n; };
  auto cells = [&](const float* p, long long o) { return W{p[c1 + o], p[w1 + o], p[n1 + o]}; };
  long long o = (long long)(lc.l0 - 1) * pl;
  float va[3], vb[3], vc[3], za[3], zb[3], zc[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const long long u = lc.l0 > 1 ? o - pl : o;
    va[m] = B.vz[d1[m] + u];
    za[m] = zd[d1[m] + u];
    vb[m] = B.vz[d1[m] + o];
    zb[m] = zd[d1[m] + o];
  }
  W mu = cells(B.mdtz, o);
  for (int l = lc.l0; l <= lc.l1; ++l, o += pl) {
    const long long q = c1 + o, d = l < D.nl ? o + pl : o;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      vc[m] = B.vz[d1[m] + d];
      zc[m] = zd[d1[m] + d];
    }
    const W ml = cells(B.mdtz, o + pl), sd = cells(B.vdiv, o);
    W r = cells(S.rho, o);
    for (int jc = 1; jc <= D.nc; ++jc) {
      const W x = cells(S.rho + (long long)jc * D.fstride, o);
      r.c = r.c + x.c;
      r.w = r.w + x.w;
      r.n = r.n + x.n;
    }
    const float dx = G.dx[q], dy = G.dy[q], dyd = G.dy_dual[q], dxd = G.dx_dual[q];
    float rx = in_x ? 0.f : B.mdtx[q], ry = in_y ? 0.f : B.mdty[q];
    float mx = 0.f, my = 0.f;
    if (l > D.nf) {
      const W w5 = cells(G.ipw[4], o), w6 = cells(G.ipw[5], o);
      const float sx = G.slope_x[q], sy = G.slope_y[q];
      mx = w5.w * mu.w + w5.c * mu.c;
      my = w5.n * mu.n + w5.c * mu.c;
      if (l < D.nl || D.freeslip) {
        mx = mx + w6.w * ml.w + w6.c * ml.c;
        my = my + w6.n * ml.n + w6.c * ml.c;
      }
      mx = sx * (0.5f * mx);
      my = sy * (0.5f * my);
    }
    float grad[3];  // half the vertical gradient over the layers above and below
#pragma unroll
    for (int m = 0; m < 3; ++m) grad[m] = 0.5f * (va[m] - vc[m]) / (za[m] - zc[m]);
    if (in_x) {
      const float up = (vb[1] - vb[0]) / dyd - (zb[1] - zb[0]) / dyd * (grad[1] + grad[0]);
      rx = ((sd.c - sd.w) / dx - mx + up) / (0.5f * (r.w + r.c));
    }
    if (in_y) {
      const float vp = (vb[2] - vb[0]) / dxd - (zb[2] - zb[0]) / dxd * (grad[2] + grad[0]);
      ry = ((sd.n - sd.c) / dy - my + vp) / (0.5f * (r.n + r.c));
    }
    B.mdtx[q] = rx;
    B.mdty[q] = ry;
    if (jk == 1) B.mdtx[x1 + o] = rx;
    if (ji == 1) B.mdty[y1 + o] = ry;
    mu = ml;
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      va[m] = vb[m];
      vb[m] = vc[m];
      za[m] = zb[m];
      zb[m] = zc[m];
    }
  }
}

// combination of the explicit wind tendencies, mo_vector_tend_expl.F90:258-310, and the
// forward step of the horizontal wind, mo_manage_pchevi.F90:86-89 (FP64 state), split step,
// with the pressure-gradient terms of a background state read in the FP32 form ks_pgrad keeps for it
// (net nl + l and the previous substep's -(nl + l)); without a background state the FP64 arrays.
// The three components' loads come first (the edge kernels' reason); the first substep (old weight 0) does
// not read the old tendency: 1.85 -> 1.49 ms at 1024x1024x80 (1.33 ms of memory traffic).  mu, mv: the FP32 mirrors of the new u, v.
__global__ void __launch_bounds__(256, 5) ks_tend_wind(Dims D, State So, State Sn, Tend<float> Tn, Carried<float> C,
                                                       SplitCarriedF PF, int rk_step, float* mu, float* mv) {
  LG_IDX3;
  if (ji > D.ny + 1 || jk > D.nx + 1) return;
  const double chw_d = 0.5 + kIMPL_THERMO_WEIGHT, ohw_d = 1.0 - (0.5 + kIMPL_THERMO_WEIGHT);
  const double cvw_d = 1.0 - kIMPL_THERMO_WEIGHT;
  const int i = min(ji, D.ny), k = min(jk, D.nx), l = min(jl, D.nl);
  const long long qu = IX(D, i, jk, l), qv = IX(D, ji, k, l), qw = IX(D, i, k, jl);
  float gu, gv, gw;
  if (D.luse_bg) {
    const float ou = PF.pold_u[qu], nu = PF.pnet_u[qu], ov = PF.pold_v[qv], nv = PF.pnet_v[qv], nw = PF.pnet_w[qw];
    gu = float(ohw_d) * ou - float(chw_d) * nu;
    gv = float(ohw_d) * ov - float(chw_d) * nv;
    gw = -(float(cvw_d) * nw);
  } else {
    const double ou = C.old_u[qu], nu = C.nl_u[qu], lu = C.l_u[qu], ov = C.old_v[qv], nv = C.nl_v[qv], lv = C.l_v[qv];
    const double nw = C.nl_w[qw], lw = C.l_w[qw];
    gu = narrow(ohw_d * ou - chw_d * (nu + lu));
    gv = narrow(ohw_d * ov - chw_d * (nv + lv));
    gw = narrow(-(cvw_d * (nw + lw)) - (1.0 - cvw_d) * lw);
  }
  const float ku = C.vsg_x[qu], kv = C.vsg_y[qv], kw = C.vsg_z[qw];
  const float vu = C.pvt_x[qu], vv = C.pvt_y[qv], vw = C.pvt_z[qw], cw = C.pgcw[qw];
  const double uo = So.u[qu], vo = So.v[qv];
  float du = 0.f, dv = 0.f, dw = 0.f, tu = 0.f, tv = 0.f, tw = 0.f;
  if (C.mdt_x) {
    du = C.mdt_x[qu];
    dv = C.mdt_y[qv];
    dw = C.mdt_z[qw];
  }
  if (rk_step == 2) {
    tu = Tn.u[qu];
    tv = Tn.v[qv];
    tw = Tn.w[qw];
  }
  float fu = gu - 0.5f * ku + vu, fv = gv - 0.5f * kv + vv, fw = gw - 0.5f * kw + vw + cw;
  if (C.mdt_x) {
    fu = fu + du;
    fv = fv + dv;
    fw = fw + dw;
  }
  if (rk_step == 2) {
    fu = 0.5f * tu + 0.5f * fu;
    fv = 0.5f * tv + 0.5f * fv;
    fw = 0.5f * tw + 0.5f * fw;
  }
  const double un = uo + D.dtime * wide(fu), vn = vo + D.dtime * wide(fv);
  if (jl <= D.nl && ji <= D.ny) {
    Tn.u[qu] = fu;
    Sn.u[qu] = un;
    mu[qu] = narrow(un);
  }
  if (jl <= D.nl && jk <= D.nx) {
    Tn.v[qv] = fv;
    Sn.v[qv] = vn;
    mv[qv] = narrow(vn);
  }
  if (ji <= D.ny && jk <= D.nx) Tn.w[qw] = fw;
}

// ---- three_band_solver_ver, mo_column_solvers.F90:21-351 --------------------------------
// The reference's implicit system for the vertical mass-flux increments at levels 2..nl of a
// column.  C = float (LGAME_PRECISION_SPLIT): from the FP32 mirror, the partial derivatives
// alpha, beta, gamma, the interface theta and density weights, the matrix and its elimination
// multipliers; FP64: the explicit predictions of theta' and exner', the right-hand side (where
// the pressure-gradient and buoyancy terms balance), the forward and back substitution, and the
// new rho_g, rho*theta_v, exner', w; theta' is formed as (rho*theta_v - theta_bg*rho)/rho with
// the small numerator in FP64.  C = double (LGAME_PRECISION_SPLIT_FP64_COLUMN): the same from
// the FP64 state, FP64 metric differences and reciprocals, with FP64 coefficients, multipliers
// and quotients -- the column solve wholly in FP64 (only the explicit tendencies it reads are
// FP32).
//
// Two kernels (the rule between them stands at their launch in split_step).  Large grids:
// ks_column_ver, one thread per column, streamed top to bottom and back, bound by about 20 FP64
// operations a cell and the latency of a level's loads: five more products are formed beside the FP64 pipe
// (fp64.cuh), the increment of rho*theta_v serves both it and exner', each layer's inputs are loaded a level
// ahead (five blocks of 96 registers an SM), and it is compiled with and without a background state (BG),
// whose absence costs two registers a layer and three FP64 operations: 1.57 -> 1.21 ms a launch at
// 512x512x80.  Small grids: ks_column_ver_tile below.
constexpr int kMaxLayers = 128;  // layers a context may have (lgame_gpu_create)

// the operators of the solve as functions of a column, for both kernels; what a level reads (LayIn, ItfIn) is
// loaded by functions of its own, so that a kernel can load ahead of its use.  (The order of the calls decides
// how a level's loads and divisions overlap: with the next layer formed before this row the thread-per-column
// kernel takes 1.37 ms at 512x512x80, with an interface loaded twice 1.30, as it is 1.21.)
template <class C>
struct ColVer {
  static constexpr bool F64 = sizeof(C) == 8;
  const Dims& D;
  const Grid<double>& G;
  const Grid<float>& GF;
  const GridX& X;
  const State &So, &Sn, &Su;  // Su: state_new_used, mo_column_solvers.F90:69-73
  const StateF &Mo, &Mn, &Mu;
  const Tend<float>& Tn;
  const bool bg;  // a background state
  const int rk_step, ji, jk;
  const long long goff;
  const C dtf, idtf, rdcv, ic2, ic1;
  const double idtd;

  __device__ __forceinline__ ColVer(const Dims& D_, const Grid<double>& G_, const Grid<float>& GF_, const GridX& X_,
                                    const State& So_, const State& Sn_, const StateF& Mo_, const StateF& Mn_,
                                    const Tend<float>& Tn_, bool bg_, int rk, int i, int j)
      : D(D_), G(G_), GF(GF_), X(X_), So(So_), Sn(Sn_), Su(rk == 1 ? So_ : Sn_), Mo(Mo_), Mn(Mn_),
        Mu(rk == 1 ? Mo_ : Mn_), Tn(Tn_), bg(bg_), rk_step(rk), ji(i), jk(j), goff((long long)(D_.g - 1) * D_.fstride),
        dtf(C(D_.dtime)), idtf(C(1.0 / D_.dtime)), rdcv(C(kR_D / kC_D_V)),
        ic2(C(1.0 / (kIMPL_THERMO_WEIGHT * (D_.dtime * D_.dtime) * kC_D_P))),
        ic1(C(1.0 / (kIMPL_THERMO_WEIGHT * D_.dtime * kC_D_P))), idtd(1.0 / D_.dtime) {}

  // the inputs of the coefficients, from the FP32 mirror or the FP64 state and metrics
  __device__ C rho_o(long long i) const { if constexpr (F64) return So.rho[goff + i]; else return Mo.rho[goff + i]; }
  __device__ C rt_o(long long i) const { if constexpr (F64) return So.rt[i]; else return Mo.rt[i]; }
  __device__ C ep_o(long long i) const { if constexpr (F64) return So.ep[i]; else return Mo.ep[i]; }
  __device__ C rho_u(long long i) const { if constexpr (F64) return Su.rho[goff + i]; else return Mu.rho[goff + i]; }
  __device__ C rt_u(long long i) const { if constexpr (F64) return Su.rt[i]; else return Mu.rt[i]; }
  __device__ C ep_u(long long i) const { if constexpr (F64) return Su.ep[i]; else return Mu.ep[i]; }
  __device__ C w_o(long long i) const { if constexpr (F64) return So.w[i]; else return Mo.w[i]; }
  __device__ C ebg(long long i) const { if constexpr (F64) return G.exner_bg[i]; else return GF.exner_bg[i]; }
  __device__ C ivol(long long i) const { if constexpr (F64) return X.inv_volume[i]; else return X.inv_volume_f[i]; }
  __device__ C iarz(long long i) const { if constexpr (F64) return X.inv_area_z[i]; else return X.inv_area_z_f[i]; }
  __device__ C damp(long long i) const { if constexpr (F64) return G.damp[i]; else return GF.damp[i]; }
  // at w level jl (2..nl): z_scalar(jl-1) - z_scalar(jl) and exner_bg(jl-1) - exner_bg(jl)
  __device__ C dzs(long long i) const {
    if constexpr (F64) return G.z_scalar[i - D.plane] - G.z_scalar[i]; else return X.dzs_f[i];
  }
  __device__ C debg(long long i) const {
    if constexpr (F64) return G.exner_bg[i - D.plane] - G.exner_bg[i]; else return X.deb_f[i];
  }
  static __device__ double W(C x) { if constexpr (F64) return x; else return wide(x); }
  static __device__ double M(C a, double x) { if constexpr (F64) return a * x; else return mul_int(a, x); }
  static __device__ double quot(double x, C d) { if constexpr (F64) return x / d; else return div_f(x, d); }

  // what a layer and an interface (w level) read
  struct LayIn { C ro, rt, eb, ep, iv, ru, rtu, epu, tr, trt; double tp, epd; };
  __device__ __forceinline__ LayIn layer_in(int jl) const {
    LayIn R{};
    if (jl > D.nl) return R;
    const long long i = IX(D, ji, jk, jl);
    R.ro = rho_o(i); R.rt = rt_o(i); R.eb = ebg(i); R.ep = ep_o(i); R.iv = ivol(i);
    if (rk_step == 2) { R.ru = rho_u(i); R.rtu = rt_u(i); R.epu = ep_u(i); }
    R.tr = C(Tn.rho[goff + i]); R.trt = C(Tn.rt[i]);
    R.tp = So.tp[i]; R.epd = So.ep[i];
    return R;
  }
  struct ItfIn { C dz, deb, dp, w, iaz, tw; double wd; };
  __device__ __forceinline__ ItfIn itf_in(int jl) const {
    ItfIn R{};
    if (jl > D.nl) return R;
    const long long i = IX(D, ji, jk, jl);
    R.dz = dzs(i); R.deb = debg(i); R.dp = damp(i); R.w = w_o(i); R.iaz = iarz(i); R.tw = C(Tn.w[i]);
    R.wd = So.w[i];
    return R;
  }
  // unscaled alpha, beta, gamma; theta of state_new_used (type C, and FP64 without a background
  // state, where theta * d(exner')/dz carries the whole hydrostatic balance); the explicit predictions of
  // theta_v' and exner' (FP64 state plus increments) and of rho_g
  struct Lay { C a, b, g, th, ro, iv, rhe; double thd, tpe, epe; };
  __device__ __forceinline__ Lay layer(int jl, const LayIn& R) const {
    Lay L;
    const long long i = IX(D, ji, jk, jl);
    L.thd = 0.0;
    if (!bg) L.thd = Su.rt[i] / Su.rho[goff + i];
    const C iro = C(1) / R.ro, irto = C(1) / R.rt;
    L.a = -R.rt * iro * iro;
    L.b = iro;
    L.g = rdcv * irto * (R.eb + R.ep);
    if (rk_step == 2) {
      const C iru = C(1) / R.ru, irtu = C(1) / R.rtu;
      L.a = C(0.5) * (L.a - R.rtu * iru * iru);
      L.b = C(0.5) * (L.b + iru);
      L.g = C(0.5) * (L.g + rdcv * irtu * (R.eb + R.epu));
      L.th = R.rtu * iru;
    } else {
      L.th = R.rt * iro;
    }
    L.ro = R.ro;
    L.iv = R.iv;
    L.tpe = R.tp + W(dtf * (L.a * R.tr + L.b * R.trt));
    L.epe = R.epd + W(dtf * L.g * R.trt);
    L.rhe = R.ro + dtf * R.tr;
    return L;
  }
  // at the interface between layers a and b: theta, and 2/(rho(a) + rho(b))
  struct Itf { C t, irho; };
  __device__ __forceinline__ Itf itf(const Lay& a, const Lay& b) const {
    return Itf{C(0.5) * (a.th + b.th), C(2) / (a.ro + b.ro)};
  }

  // row jl: the interface I (its inputs N) between layers jl (L0) and jl+1 (L1); diagonal and right-hand side
  struct Row { C dv; double rv; };
  __device__ __forceinline__ Row row(const Lay& L0, const Lay& L1, const ItfIn& N, const Itf& I) const {
    Row r;
    const C ti = I.t, irio = I.irho;
    const C dz = N.dz, deb = N.deb, dp = N.dp, wof = N.w;
    const double wo = N.wd;
    const C al0 = L0.a * L0.iv, al1 = L1.a * L1.iv, be0 = L0.b * L0.iv, be1 = L1.b * L1.iv;
    const C ga0 = L0.g * L0.iv, ga1 = L1.g * L1.iv;
    r.dv = -(ti * ti) * (ga0 + ga1) + C(0.5) * deb * (al1 - al0 + ti * (be1 - be0))
           - dz * ic2 * irio * (C(2) * N.iaz + dtf * wof * C(0.5) * (L1.iv - L0.iv)) * dp;
    const C rie = C(0.5) * (L0.rhe + L1.rhe);
    // The products of FP32 coefficients with FP64 values here and in the state update below
    // stay FP64 products of the FP32 factors: merging two FP32 factors into one rounded
    // coefficient (e.g. -dz*ic2*(1 + rie*irio) for w_old) saves two FP64 operations per cell
    // but lets an atmosphere at rest over hills drift about four times faster (1e-8 instead
    // of 3e-9 m/s of spurious wind after 3 h at 256 x 256 x 50).
    r.rv = M(-dz * ic2, wo + W(dtf * N.tw));
    r.rv = fma(bg ? W(ti * idtf) : 0.5 * (L0.thd + L1.thd) * idtd, L0.epe - L1.epe, r.rv);
    r.rv = fma(W(C(0.5) * idtf * deb), L0.tpe + L1.tpe, r.rv);
    r.rv = fma(W(-dz * ic2 * rie * irio), wo, r.rv);
    return r;
  }
  // and its couplings with row jl+1 by layer jl+1's derivatives, between the interfaces I1 above and I2 below it
  struct Coupling { C c, e; };
  __device__ __forceinline__ Coupling coupling(const Lay& L1, const ItfIn& N1, const ItfIn& N2, const Itf& I1,
                                               const Itf& I2) const {
    const C al1 = L1.a * L1.iv, be1 = L1.b * L1.iv, ga1 = L1.g * L1.iv;
    return Coupling{I2.t * ga1 * I1.t + C(0.5) * N2.deb * (al1 + be1 * I1.t)
                        - N2.dz * ic1 * C(0.5) * N2.w * L1.iv * I2.irho * N2.dp,
                    I1.t * ga1 * I2.t - C(0.5) * N1.deb * (al1 + be1 * I2.t)
                        + N1.dz * ic1 * C(0.5) * N1.w * L1.iv * I1.irho * N1.dp};
  }

  // the new state, mo_column_solvers.F90:300-345: layer jl from the solutions s0, s1 at the
  // interfaces above and below it (w levels jl, jl+1) and their products p0, p1 with the interface theta;
  // w at level jl+1 from the new densities of layers jl and jl+1
  struct StateIn { double rt, rho, ep, bg, w; C ivf, iaz, mro; float trho, trt; };
  __device__ __forceinline__ StateIn state_in(int m) const {
    StateIn r;
    const long long p = IX(D, ji, jk, m);
    r.rt = So.rt[p];
    r.rho = So.rho[goff + p];
    r.ep = So.ep[p];
    r.bg = G.theta_v_bg[p];
    r.w = So.w[p];
    r.ivf = ivol(p);
    r.iaz = iarz(p);
    r.mro = rho_o(p);
    r.trho = Tn.rho[goff + p];
    r.trt = Tn.rt[p];
    return r;
  }
  __device__ __forceinline__ double new_rho(const StateIn& c, double s0, double s1) const {
    return fma(W(dtf * c.ivf), s1 - s0, c.rho + W(dtf * C(c.trho)));
  }
  // new rho_g in the type of the coefficients (FP32: rounded)
  static __device__ __forceinline__ C rho_c(double rn) { if constexpr (F64) return rn; else return narrow(rn); }
  // returns rho_c of the layer's new density; below: the layer below and its rho_c
  __device__ __forceinline__ C new_state(int jl, const StateIn& c, const StateIn& below, C rnc_below, double s0,
                                         double s1, double p0, double p1, C g) const {
    const long long i = IX(D, ji, jk, jl);
    const double dtv = W(dtf * c.ivf);
    const double rn = new_rho(c, s0, s1);
    const double inc = fma(dtv, p1 - p0, W(dtf * C(c.trt)));
    const double rtn = c.rt + inc;
    const double epn = fma(W(g), inc, c.ep);
    const float rnf = narrow(rn);
    const C rnc = F64 ? C(rn) : C(rnf);
    if constexpr (F64) {
      const double tpn = fma(-c.bg, rn, rtn) / rn;
      Sn.tp[i] = tpn;
      Mn.tp[i] = narrow(tpn);
    } else {
      const float tpf = narrow(fma(-c.bg, rn, rtn)) / rnf;
      Sn.tp[i] = wide(tpf);
      Mn.tp[i] = tpf;
    }
    Sn.rho[goff + i] = rn;
    Sn.rt[i] = rtn;
    Sn.ep[i] = epn;
    Mn.rho[goff + i] = rnf;
    Mn.rt[i] = narrow(rtn);
    Mn.ep[i] = narrow(epn);
    if (jl < D.nl) {
      const long long ib = i + D.plane;
      const C rin = C(0.5) * (rnc + rnc_below);
      const C irio = C(2) / (c.mro + below.mro);
      const double wn = M(irio, fma(-W(rin), below.w, M(C(2) * below.iaz, s1)));
      Sn.w[ib] = wn;
      Mn.w[ib] = narrow(wn);
    }
    return rnc;
  }
  // w_free_slip, mo_inner_product.F90:52-75, with the new u, v
  __device__ __forceinline__ void free_slip() const {
    const int m = D.nl;
    const double wf =
        G.ipw[0][IX(D, ji, jk, m)] * Sn.u[IX(D, ji, jk + 1, m)] * G.slope_x[IX(D, ji, jk + 1, m)]
      + G.ipw[1][IX(D, ji, jk, m)] * Sn.v[IX(D, ji, jk, m)] * G.slope_y[IX(D, ji, jk, m)]
      + G.ipw[2][IX(D, ji, jk, m)] * Sn.u[IX(D, ji, jk, m)] * G.slope_x[IX(D, ji, jk, m)]
      + G.ipw[3][IX(D, ji, jk, m)] * Sn.v[IX(D, ji + 1, jk, m)] * G.slope_y[IX(D, ji + 1, jk, m)];
    Sn.w[IX(D, ji, jk, m + 1)] = wf;
    Mn.w[IX(D, ji, jk, m + 1)] = narrow(wf);
  }
};

// a thread a column; BG: with a background state
template <class C, bool BG>
__global__ void __launch_bounds__(128, 5) ks_column_ver(Dims D, Grid<double> G, Grid<float> GF, GridX X, State So,
                                                     State Sn, StateF Mo, StateF Mn, Tend<float> Tn, int rk_step) {
  using Cv = ColVer<C>;
  const int ji = blockIdx.x * blockDim.x + threadIdx.x + 1;
  const int jk = blockIdx.y * blockDim.y + threadIdx.y + 1;
  if (ji > D.ny || jk > D.nx) return;
  const Cv V(D, G, GF, X, So, Sn, Mo, Mn, Tn, BG, rk_step, ji, jk);
  const int nl = D.nl, n = nl - 1;
  C epr[kMaxLayers + 1];       // elimination multipliers
  double rpr[kMaxLayers + 1];  // substituted right-hand side, then the solution (FP64)
  C tis[kMaxLayers + 1];       // interface theta
  C gs[kMaxLayers + 1];        // gamma of each layer
  typename Cv::Lay L0 = V.layer(1, V.layer_in(1)), L1 = V.layer(2, V.layer_in(2)), L2{};
  typename Cv::LayIn R = V.layer_in(3);
  gs[1] = L0.g;
  C cv_prev = C(0), epr_prev = C(0);
  double rpr_prev = 0.0;
  typename Cv::Itf I1 = V.itf(L0, L1);
  typename Cv::ItfIn N1 = V.itf_in(2);
  for (int jl = 1; jl <= n; ++jl) {  // row jl: level jl+1 between layers jl and jl+1
    // (a layer's inputs are loaded a level ahead of their use; the interfaces' ahead too spills: 1.35 ms at
    // 512x512x80)
    const typename Cv::LayIn Rn = V.layer_in(jl + 3);
    const typename Cv::ItfIn N2 = V.itf_in(jl + 2);
    gs[jl + 1] = L1.g;
    tis[jl] = I1.t;
    const typename Cv::Row q = V.row(L0, L1, N1, I1);
    typename Cv::Itf I2{C(0), C(0)};
    typename Cv::Coupling k{C(0), C(0)};
    if (jl < n) {
      L2 = V.layer(jl + 2, R);
      I2 = V.itf(L1, L2);
      k = V.coupling(L1, N1, N2, I1, I2);
    }
    const C piv = q.dv - epr_prev * cv_prev;
    const double x = (jl == 1) ? q.rv : fma(-Cv::W(cv_prev), rpr_prev, q.rv);
    rpr_prev = Cv::quot(x, piv);
    rpr[jl] = rpr_prev;
    epr_prev = k.e / piv;
    epr[jl] = epr_prev;
    cv_prev = k.c;
    L0 = L1; L1 = L2;
    R = Rn;
    I1 = I2;
    N1 = N2;
  }
  // back substitution fused with the new state, bottom to top: layer jl needs the solutions of the rows above
  // (w level jl) and below it (w level jl+1), and w at level jl+1 the new densities of layers jl and jl+1,
  // all known once the substitution has reached row jl-1.  The inputs of the layer above are loaded before
  // the current layer's results are stored (a store may alias a later load, which stops the
  // compiler from moving the loads itself).
  typename Cv::StateIn in_cur = V.state_in(nl), in_up{}, in_below{};
  double s1 = 0.0;     // solution at the interface below the layer (w level jl+1)
  double p1 = 0.0;     // theta there times it
  C rnf_below = C(0);  // new rho_g of the layer below (FP32: rounded)
  for (int jl = nl; jl >= 1; --jl) {
    if (jl > 1) in_up = V.state_in(jl - 1);
    // solution of row jl-1 (w level jl), the interface above the layer
    double s0 = 0.0;
    if (jl >= 2) s0 = (jl - 1 == n) ? rpr[n] : fma(-Cv::W(epr[jl - 1]), s1, rpr[jl - 1]);
    const double p0 = (jl >= 2) ? Cv::M(tis[jl - 1], s0) : 0.0;
    rnf_below = V.new_state(jl, in_cur, in_below, rnf_below, s0, s1, p0, p1, gs[jl]);
    s1 = s0;
    p1 = p0;
    in_below = in_cur;
    in_cur = in_up;
  }
  if (D.freeslip) V.free_slip();
}

// Small grids: a block owns TC columns and NW chunks of levels (a lane per column, chunk w of a
// column in thread w*TC + lane), in phases:
//   1. every thread forms the rows of its chunk (matrix, right-hand side) into shared memory;
//   2. the first TC threads run the factorisation (pivot p, upper factor e/p, type C) and the forward
//      substitution y = r - (c/p)*y, c/p held in FP64 (tile_sweep.cuh), one multiply-add a row in the chain;
//   3. every thread its rows' y/p;  4. the first TC threads the back substitution;
//   5. every thread the new state of its chunk of layers.
// The chain of levels then waits on shared memory and arithmetic alone, and the levels' loads and
// FP64 operations run side by side.  Measured per launch, against ks_column_ver: 31 against 204
// us at 4 x 256 x 60, 124 against 275 us at 128 x 128 x 80, 245 against 322 us at 180 x 210 x 80, equal (363 us)
// at 243 x 240 x 80, and slower above (529 against 413 us at 288 x 288 x 80), where the phases in which one
// warp works cost more than the latency they hide.
template <class C, int TC, int NW>
__global__ void __launch_bounds__(TC * NW, sizeof(C) == 4 ? 768 / (TC * NW) : 1)
    ks_column_ver_tile(Dims D, Grid<double> G, Grid<float> GF, GridX X, State So, State Sn, StateF Mo, StateF Mn,
                       Tend<float> Tn, int rk_step) {
  using Cv = ColVer<C>;
  constexpr int kRow = kTileCoef * TC;  // coefficients of one level of the block's columns in shared memory
  const int lane = threadIdx.x % TC, w = threadIdx.x / TC;
  const int col = blockIdx.x * TC + lane;
  const bool valid = col < D.ny * D.nx;
  const Cv V(D, G, GF, X, So, Sn, Mo, Mn, Tn, D.luse_bg, rk_step, valid ? col % D.ny + 1 : 1, valid ? col / D.ny + 1 : 1);
  const int nl = D.nl, n = nl - 1;
  extern __shared__ __align__(16) unsigned char smem_cv[];
  double* const sr = (double*)smem_cv + lane;             // right-hand side, y, then the solution
  C* const sc = (C*)((double*)smem_cv + TC * nl) + lane;  // per row: diagonal (then the pivot), c, e (then
                                                          // e/p), interface theta, gamma of layer jl
  const int chunk = (n + NW - 1) / NW, r0 = w * chunk + 1, r1 = min(n, (w + 1) * chunk);
  if (valid && r0 <= r1) {
    typename Cv::Lay L0 = V.layer(r0, V.layer_in(r0)), L1 = V.layer(r0 + 1, V.layer_in(r0 + 1)), L2{};
    typename Cv::ItfIn N1 = V.itf_in(r0 + 1), N2{};
    typename Cv::Itf I1 = V.itf(L0, L1), I2{C(0), C(0)};
    for (int jl = r0; jl <= r1; ++jl) {
      const typename Cv::Row q = V.row(L0, L1, N1, I1);
      typename Cv::Coupling k{C(0), C(0)};
      if (jl < n) {
        L2 = V.layer(jl + 2, V.layer_in(jl + 2));
        N2 = V.itf_in(jl + 2);
        I2 = V.itf(L1, L2);
        k = V.coupling(L1, N1, N2, I1, I2);
      }
      C* const row = sc + kRow * (jl - 1);
      row[0] = q.dv;
      row[TC] = k.c;
      row[2 * TC] = k.e;
      row[3 * TC] = I1.t;
      row[4 * TC] = L0.g;
      if (jl == n) row[kRow + 4 * TC] = L1.g;
      sr[TC * (jl - 1)] = q.rv;
      L0 = L1; L1 = L2;
      N1 = N2;
      I1 = I2;
    }
  }
  __syncthreads();
  if (w == 0 && valid) tile_forward<C, TC>(sc, sr, n);
  __syncthreads();
  if (valid)
    for (int jl = r0; jl <= r1; ++jl) sr[TC * (jl - 1)] = Cv::quot(sr[TC * (jl - 1)], sc[kRow * (jl - 1)]);
  __syncthreads();
  if (w == 0 && valid) tile_back<C, TC>(sc, sr, n);
  __syncthreads();
  // the new state, each chunk of layers bottom to top; the chunk's first layer needs the new
  // density of the layer below it, formed anew
  const int lchunk = (nl + NW - 1) / NW, l0 = w * lchunk + 1, l1 = min(nl, (w + 1) * lchunk);
  if (!valid || l0 > l1) return;
  // solution and interface theta of row m (w level m+1), 0 at the model top and surface
  auto sol = [&](int m) -> double { return (m >= 1 && m <= n) ? sr[TC * (m - 1)] : 0.0; };
  auto tif = [&](int m) -> C { return (m >= 1 && m <= n) ? sc[kRow * (m - 1) + 3 * TC] : C(0); };
  typename Cv::StateIn in_cur = V.state_in(l1), in_up{}, in_below{};
  double s1 = sol(l1), p1 = Cv::M(tif(l1), s1);
  C rnf_below = C(0);
  if (l1 < nl) {
    in_below = V.state_in(l1 + 1);
    rnf_below = Cv::rho_c(V.new_rho(in_below, s1, sol(l1 + 1)));
  }
  for (int jl = l1; jl >= l0; --jl) {
    if (jl > l0) in_up = V.state_in(jl - 1);
    const double s0 = sol(jl - 1), p0 = Cv::M(tif(jl - 1), s0);
    rnf_below = V.new_state(jl, in_cur, in_below, rnf_below, s0, s1, p0, p1, sc[kRow * (jl - 1) + 4 * TC]);
    s1 = s0;
    p1 = p0;
    in_below = in_cur;
    in_cur = in_up;
  }
  if (D.freeslip && l1 == nl) V.free_slip();
}
template <class C, int TC>
constexpr size_t column_ver_smem(int nl) { return (size_t)nl * TC * (sizeof(double) + kTileCoef * sizeof(C)); }

// ---- three_band_solver_gen_densities, mo_column_solvers.F90:353-604 ----------------------
// The reference's system per (column, tracer)  d_l s_l + e_l s_{l+1} + c_{l-1} s_{l-1} = rho_l + inc_l
// (implicit-upwind vertical flux and sedimentation, inc = dt*tendency + explicit flux part) is
// solved for the increment delta = s - rho_old:
//   d_l delta_l + e_l delta_{l+1} + c_{l-1} delta_{l-1} = inc_l - (d_l - 1) rho_l - e_l rho_{l+1} - c_{l-1} rho_{l-1}
// in FP32 (coefficients from the mirror; the right-hand side's rounding is then relative to the
// flux terms, the size of delta, and not to the density), and the new density rho_old + delta
// is formed in FP64.  d - 1 is accumulated on its own, so the diagonal's rounding near 1 does
// not enter.  Each interface couples its two cells in one direction only (the upwind side:
// e_l = 0 or c_l = 0), so Thomas's pivots are the diagonal entries themselves and its sweeps
// are the affine recurrences
//   forward   r_l     = alpha_l r_{l-1} + beta_l,     alpha_l = -c_{l-1}/d_l, beta_l = rhs_l/d_l
//   backward  delta_l = r_l - e'_l delta_{l+1},        e'_l = e_l/d_l.
//
// A block owns 32 columns (a row tile, one per lane) and three tracers, in three phases:
//   1. the eight warps take contiguous chunks of levels (ten at 80 layers); a thread walks its
//      chunk top down and forms alpha, beta, e' of the three tracers into shared memory, and the
//      sediment heating.  What the three tracers share -- volume, area, old and new w,
//      temperature and heat capacities at each interface, the cloud droplets' fall speed -- is
//      loaded and formed once, the values of the interface below a level are carried to the next
//      level as the interface above it, and inputs are loaded two levels ahead;
//   2. three warps run the two sweeps of one tracer each, a lane per column, from shared memory
//      (no memory latency in the level chain), while the old FP64 densities of phase 3 arrive;
//   3. the chunks again: rho_old + delta in FP64, clipped (mo_column_solvers.F90:587-591), and
//      its rounded mirror.
// The elimination data never leave the chip: as a per-thread local stack (one thread per column
// and tracer walking all levels) they spilled through L2 to DRAM, 321 bytes per cell moved
// against 202.  The two blocks of a row tile are consecutive in the grid and read the tile's
// shared inputs once from DRAM.  The sediment heating of a set's condensates, added in their order, goes to the
// set's plane of csh_part (rk_step 1 only, FP32 heat capacities); ks_csh_sum adds the two (a plane a condensate:
// 0.48 -> 0.29 ms at 1024x1024x80, and 0.07 ms fewer here).
constexpr int kTrWarps = 8;   // level chunks in phases 1 and 3
constexpr int kTrSet = 3;     // tracers per block
constexpr int kTrPitch = 33;  // shared-memory row pitch (32 columns + 1)
constexpr int kTrPre = 10;    // levels per thread whose old densities are loaded before the sweeps
constexpr int kTrRow = 3 * kTrSet * kTrPitch;  // shared-memory floats per level

// inputs of one level m of a column for the three tracers of a block: the tracers' old mirror
// densities and tendencies, and at the interface above the level (w level m) area, old and
// new w; the level's 1/volume and temperature; for the cloud droplets' fall speed (second set
// only) the gas density, gravity at w levels m and m+1 and the two vertical weights
struct TrLevel { float ro[kTrSet], tr[kTrSet], az, wo, wn, iv, tm, rg, gm, gm1, w5, w6; };

// v_fall_liquid, mo_derived.F90:218-263, in FP32, at level m from its prefetched inputs
__device__ __forceinline__ float vfall_liquid_l(const TrLevel& L, float radius, int m, int nl) {
  const float g = (m == 1) ? L.gm1 : (m == nl) ? L.gm : L.w5 * L.gm + L.w6 * L.gm1;
  const float rg = L.rg;
  const float pm = float(kM_D / kN_A);
  const float tv = sqrtf(8.f * float(kK_B) / (float(kPI) * pm) * L.tm);
  const float mfp = 1.f / (1.41421356f * (rg / pm) * (4.f * float(kPI) * (130e-12f * 130e-12f)));
  const float nu = (1.f / 3.f) * tv * mfp;
  float v = 2.f * (radius * radius) * (float(kRHO_H2O) - rg) * g / (9.f * rg * nu);
  if (v * radius / nu > 10.f) v = sqrtf(8.f * radius * float(kRHO_H2O) * g / (3.f * rg * 0.8f));
  return v;
}

// properties of the block's tracers, fixed at compile time (the split path runs the moist
// constituent layout: 1 snow, 2 rain, 3 cloud ice, 4 cloud water, 5 graupel, 6 gas, 7 vapour):
// constituent index, condensate or not, ice or water heat capacity (odd constituents are ice,
// mo_dictionary.F90:175-189), fall speed (snow 1 m/s: radius 500 um above 250 um; cloud ice
// 0.001 m/s; cloud water v_fall_liquid at radius 12 um; rain, graupel and vapour 0, their
// radius never being set), and whether the surface sink's heat term applies (jc > nc/4)
template <int SET>
struct TrSet {
  __device__ static constexpr int jc(int q) { return SET == 0 ? q + 1 : (q == 2 ? 7 : q + 4); }
  __device__ static constexpr bool cond(int q) { return jc(q) <= 5; }
  __device__ static constexpr bool ice(int q) { return (jc(q) - 1) % 2 == 0; }
  __device__ static constexpr bool cloud(int q) { return jc(q) == 4; }
  __device__ static constexpr float vfix(int q) { return jc(q) == 1 ? 1.f : jc(q) == 3 ? 0.001f : 0.f; }
  __device__ static constexpr bool sfc_heat(int q) { return jc(q) > 1; }  // jc > nc/4 = 1
};

// One block: phases 1-3 above for tracer set SET; HEAT: the first substep, which also stores
// the sediment heating.  Shared memory [level-1][tracer q][alpha, beta, e'][33]: the nine values
// of a level sit at fixed offsets from one row address.
template <int SET, bool HEAT>
__device__ __forceinline__ void tracer_block(const Dims& D, const Grid<float>& GF, const GridX& X, const State& So,
                                             const State& Sn, const StateF& Mo, const StateF& Mn,
                                             const float* t_rho_all, const float* Tm, float* csh_part, float* sm) {
  using P = TrSet<SET>;
  const int nl = D.nl;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int ji = blockIdx.y * 32 + lane + 1;
  const int jk = blockIdx.z + 1;
  const bool valid = ji <= D.ny;
  const float dt = float(D.dtime);
  const float itw = 0.5f, ew = 0.5f;
  const int pl = (int)D.plane;  // level stride; fstride*ncons < 2^31 for every supported grid
  // 32-bit element indices off the arrays' base addresses, which stay kernel parameters: level
  // jl of tracer q is at tq[q] + (jl-1)*pl
  const int c32 = (int)IX(D, valid ? ji : 1, jk, 1);
  int tq[kTrSet];
#pragma unroll
  for (int q = 0; q < kTrSet; ++q) tq[q] = (P::jc(q) - 1) * (int)D.fstride + c32;
  const int grg = (D.g - 1) * (int)D.fstride + c32;
  const int chunk = (nl + kTrWarps - 1) / kTrWarps;
  const int l0 = w * chunk + 1, l1 = min(nl, (w + 1) * chunk);
  auto load = [&](int m, TrLevel& L) {
    const int o = (m - 1) * pl;
#pragma unroll
    for (int q = 0; q < kTrSet; ++q) {
      L.ro[q] = Mo.rho[tq[q] + o];
      L.tr[q] = t_rho_all[tq[q] + o];
    }
    const int e = c32 + o;
    L.az = GF.area_z[e];
    L.wo = Mo.w[e];
    L.wn = Mn.w[e];
    L.iv = X.inv_volume_f[e];
    if (HEAT || SET == 1) L.tm = Tm[e];
    if (SET == 1) {
      L.rg = Mo.rho[grg + o];
      L.gm = GF.gm[e];
      L.gm1 = GF.gm[e + pl];
      L.w5 = GF.ipw[4][e];
      L.w6 = GF.ipw[5][e];
    }
  };
  auto vf_of = [&](int q, float vcl) -> float { return P::cloud(q) ? vcl : P::vfix(q); };
  auto cp_t = [&](int q, float tm) -> float { return (P::ice(q) ? c_p_ice(tm) : c_p_water(tm)) * tm; };
  // ---- phase 1: coefficients, a thread walking its chunk of levels ----------------------------
  // ring of level inputs: level jl in slot k, jl+1 in k+1, jl+2 and jl+3 loading (two levels of
  // look-ahead: the interface below level jl+1 needs level jl+2 in the next iteration)
  if (valid && l0 <= l1) {
    TrLevel ring[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) ring[k] = TrLevel{};
    load(l0, ring[0]);
    if (l0 + 1 <= nl) load(l0 + 1, ring[1]);
    if (l0 + 2 <= min(l1 + 1, nl)) load(l0 + 2, ring[2]);
    // carried from the interface above the current level: flux coefficient, flux, heat flux of
    // each tracer, the densities of the level above, and the cloud droplets' fall speed at the
    // current level
    float vfi_up[kTrSet], vfr_up[kTrSet], vefv_up[kTrSet], ro_up[kTrSet];
    float vcl_cur = (SET == 1) ? vfall_liquid_l(ring[0], 12.e-6f, l0, nl) : 0.f;
#pragma unroll
    for (int q = 0; q < kTrSet; ++q) vfi_up[q] = vfr_up[q] = vefv_up[q] = ro_up[q] = 0.f;
    if (l0 >= 2) {  // the interface above the chunk's first level, formed from scratch
      TrLevel up{};
      load(l0 - 1, up);
      const TrLevel& cur = ring[0];
      const float vcl_i = (SET == 1) ? 0.5f * (vfall_liquid_l(up, 12.e-6f, l0 - 1, nl) + vcl_cur) : 0.f;
#pragma unroll
      for (int q = 0; q < kTrSet; ++q) {
        const float vf = vf_of(q, vcl_i);
        vfi_up[q] = cur.az * (cur.wo - vf);
        float fr = cur.az * (cur.wn - vf);
        fr = ((fr >= 0.f) ? cur.ro[q] : up.ro[q]) * fr;
        vfr_up[q] = fr;
        if (HEAT && P::cond(q)) vefv_up[q] = cp_t(q, cur.tm) * fr;
        ro_up[q] = up.ro[q];
      }
    }
    for (int base = l0; base <= l1; base += 4) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int jl = base + k;
        if (jl > l1) break;
        if (jl + 3 <= min(l1 + 1, nl)) load(jl + 3, ring[(k + 3) % 4]);
        const TrLevel& cur = ring[k];
        const TrLevel& nxt = ring[(k + 1) % 4];
        const int o = (jl - 1) * pl;
        const float iv = cur.iv;
        const float itv_a = itw * dt * iv;
        const bool below = jl <= nl - 1;
        // shared parts of the interface below the level (w level jl+1)
        float vcl_b = 0.f, vcl_i = 0.f;
        if (SET == 1 && below) {
          vcl_b = vfall_liquid_l(nxt, 12.e-6f, jl + 1, nl);
          vcl_i = 0.5f * (vcl_cur + vcl_b);
        }
        const float az_sfc = (jl == nl) ? GF.area_z[c32 + o + pl] : 0.f;
        float* row = sm + (jl - 1) * kTrRow + lane;
        float heat = 0.f;
#pragma unroll
        for (int q = 0; q < kTrSet; ++q) {
          const float ro = cur.ro[q];
          float vfi = 0.f, vfr = 0.f, vefv = 0.f, ro_dn = 0.f;
          if (below) {
            const float vf = vf_of(q, vcl_i);
            ro_dn = nxt.ro[q];
            vfi = nxt.az * (nxt.wo - vf);
            float fr = nxt.az * (nxt.wn - vf);
            fr = ((fr >= 0.f) ? ro_dn : ro) * fr;
            vfr = fr;
            if (HEAT && P::cond(q)) vefv = cp_t(q, nxt.tm) * fr;
          }
          // d - 1, explicit flux part and sediment heating of cell jl
          float dm1, fl, h = 0.f;
          if (jl == 1) {
            dm1 = (vfi >= 0.f) ? 0.f : -itv_a * vfi;
            fl = ew * dt * vfr * iv;
            h = vefv * iv;
          } else if (jl == nl) {
            dm1 = (vfi_up[q] >= 0.f) ? itv_a * vfi_up[q] : 0.f;
            fl = -ew * dt * vfr_up[q] * iv;
            h = -vefv_up[q] * iv;
            if (P::cond(q)) {
              const float vsurf = vf_of(q, vcl_cur);  // the lowest layer's own fall speed
              dm1 += itw * vsurf * dt * az_sfc * iv;
              fl -= ew * vsurf * dt * ro * az_sfc * iv;
              if (HEAT && P::sfc_heat(q)) {
                const float tn = cur.tm;
                h -= vsurf * tn * (P::ice(q) ? c_p_ice(tn) : c_p_water(tn)) * ro * az_sfc * iv;
              }
            }
          } else {
            dm1 = 0.f;
            if (vfi_up[q] >= 0.f) dm1 += itv_a * vfi_up[q];
            if (vfi < 0.f) dm1 -= itv_a * vfi;
            fl = ew * dt * (vfr - vfr_up[q]) * iv;
            h = (vefv - vefv_up[q]) * iv;
          }
          if (HEAT && P::cond(q)) heat += h;
          // couplings: row jl to jl+1 (upward flux below), row jl to jl-1 (downward flux above);
          // the pivot is the diagonal 1 + (d - 1)
          const float ev = (below && vfi >= 0.f) ? -(itv_a * vfi) : 0.f;
          const float cv_up = (jl >= 2 && vfi_up[q] < 0.f) ? itv_a * vfi_up[q] : 0.f;
          const float rhs = (dt * cur.tr[q] + fl) - dm1 * ro - ev * ro_dn - cv_up * ro_up[q];
          const float ip = 1.f / (1.f + dm1);
          row[(3 * q + 0) * kTrPitch] = -cv_up * ip;
          row[(3 * q + 1) * kTrPitch] = rhs * ip;
          row[(3 * q + 2) * kTrPitch] = ev * ip;
          vfi_up[q] = vfi;
          vfr_up[q] = vfr;
          vefv_up[q] = vefv;
          ro_up[q] = ro;
        }
        if (HEAT) csh_part[SET * (int)D.fstride + c32 + o] = heat;
        vcl_cur = vcl_b;
      }
    }
  }
  // the old FP64 densities of phase 3, loaded before the sweeps so that they arrive meanwhile
  // (the registers of phase 1 are free by now); chunks longer than kTrPre levels load the rest
  // in phase 3
  double rq[kTrPre][kTrSet];
#pragma unroll
  for (int k = 0; k < kTrPre; ++k)
#pragma unroll
    for (int q = 0; q < kTrSet; ++q) rq[k][q] = (valid && l0 + k <= l1) ? So.rho[tq[q] + (l0 + k - 1) * pl] : 0.0;
  __syncthreads();
  // ---- phase 2: the sweeps, warp q for tracer q, a lane per column -----------------------------
  if (w < kTrSet) {
    float* row = sm + lane + 3 * w * kTrPitch;
    float r = 0.f;
#pragma unroll 4
    for (int jl = 1; jl <= nl; ++jl, row += kTrRow) {
      r = row[0] * r + row[kTrPitch];
      row[kTrPitch] = r;
    }
    float dl = 0.f;
#pragma unroll 4
    for (int jl = nl; jl >= 1; --jl) {
      row -= kTrRow;
      dl = row[kTrPitch] - row[2 * kTrPitch] * dl;
      row[kTrPitch] = dl;
    }
  }
  __syncthreads();
  // ---- phase 3: new densities rho_old + delta (FP64), clipped, and their mirror ---------------
  if (!valid || l0 > l1) return;
  // the mirror is rounded by the hardware conversion here (the bits of narrow() in one issue
  // slot): the FP64 pipe carries only this and the addition per value, against a dozen integer
  // operations for narrow()
  auto update = [&](int jl, int q, double ro_old) {
    const int e = tq[q] + (jl - 1) * pl;
    const double sn = ro_old + wide(sm[(jl - 1) * kTrRow + lane + (3 * q + 1) * kTrPitch]);
    const double v = __double2hiint(sn) < 0 ? 0.0 : sn;
    Sn.rho[e] = v;
    Mn.rho[e] = __double2float_rn(v);
  };
#pragma unroll
  for (int k = 0; k < kTrPre; ++k)
#pragma unroll
    for (int q = 0; q < kTrSet; ++q)
      if (l0 + k <= l1) update(l0 + k, q, rq[k][q]);
  for (int jl = l0 + kTrPre; jl <= l1; ++jl)
#pragma unroll
    for (int q = 0; q < kTrSet; ++q) update(jl, q, So.rho[tq[q] + (jl - 1) * pl]);
}

// grid (2 tracer sets, row tiles, nx), 256 threads, dynamic shared memory tracer_smem(D.nl);
// HEAT: the first substep
template <bool HEAT>
__global__ void __launch_bounds__(kTrWarps * 32, 2) ks_column_tracers(Dims D, Grid<float> GF, GridX X, State So,
                                                                      State Sn, StateF Mo, StateF Mn,
                                                                      const float* t_rho_all, const float* Tm,
                                                                      float* csh_part) {
  extern __shared__ float sm[];
  if (blockIdx.x == 0) tracer_block<0, HEAT>(D, GF, X, So, Sn, Mo, Mn, t_rho_all, Tm, csh_part, sm);
  else tracer_block<1, HEAT>(D, GF, X, So, Sn, Mo, Mn, t_rho_all, Tm, csh_part, sm);
}

// sediment heating of all condensates: the sums of ks_column_tracers' two tracer sets
__global__ void ks_csh_sum(Dims D, const float* csh_part, float* csh) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl);
  csh[q] = csh_part[q] + csh_part[q + D.fstride];
}

// dynamic shared memory of ks_column_tracers: alpha, beta and e' of three tracers, 32 columns
size_t tracer_smem(int nl) { return (size_t)nl * kTrRow * sizeof(float); }

// the tile kernel's shared memory is allowed for the most layers a context may have: contexts of
// different heights share the function's attribute
template <class C, int TC, int NW>
bool column_ver_attr() {
  return cudaFuncSetAttribute(ks_column_ver_tile<C, TC, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)column_ver_smem<C, TC>(kMaxLayers)) == cudaSuccess;
}

constexpr int kSMs = 152;  // streaming multiprocessors of the GB300

dim3 sblk() { return dim3(32, 8, 1); }
// x: row tiles, y: levels, z: column tiles (see LG_IDX3)
dim3 sgrd(int rows, int cols, int levs) {
  return dim3((unsigned)((rows + 31) / 32), (unsigned)levs, (unsigned)((cols + 7) / 8));
}
// column kernels: 128 threads, 32 rows x 4 columns
dim3 cblk() { return dim3(32, 4, 1); }
dim3 cgrd(int rows, int cols) { return dim3((unsigned)((rows + 31) / 32), (unsigned)((cols + 3) / 4), 1u); }
// the marching divergences: the column in as many chunks as give the device about 128 warps an SM,
// of at least 4 levels.  (One chunk: ks_gas_div 187, 421, 505, 1772 us at 4x256x60, 128x128x80,
// 256x256x80, 768x768x80; so: 24, 62, 245, 1718 us, and 50, 198, 1145 us at the last three since it
// loads layers ahead.  64 warps an SM: 72 us at 128x128x80, 1899 us at 768x768x80; two levels a chunk at
// least: 64 us at 128x128x80, both before that.)
dim3 cgrd_levels(const Dims& D, int rows, int cols) {
  dim3 g = cgrd(rows, cols);
  const long long warps = 4LL * g.x * g.y;
  const int chunks = (int)std::min<long long>((kSMs * 128LL + warps - 1) / warps, D.nl);
  const int len = std::max((D.nl + chunks - 1) / chunks, 4);
  g.z = (unsigned)((D.nl + len - 1) / len);
  return g;
}

}  // namespace

int split_create(const Dims& D, bool column_fp64, const SplitDiff& diff, const SplitSfc& sfc, SplitCtx** out,
                 long long* bytes) {
  if (D.ncons > 1 && D.ncons != kTracers + 1) {
    lgame_set_error("split precision: the tracer kernel is built for five condensates and water vapour");
    return LGAME_ERR_UNSUPPORTED;
  }
  if (D.ncons > 1 &&
      (D.nl > kMaxLayers ||
       cudaFuncSetAttribute(ks_column_tracers<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)tracer_smem(kMaxLayers)) != cudaSuccess ||
       cudaFuncSetAttribute(ks_column_tracers<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)tracer_smem(kMaxLayers)) != cudaSuccess)) {
    lgame_set_error("split precision: the tracer solver supports at most 128 layers");
    return LGAME_ERR_UNSUPPORTED;
  }
  if (!(column_fp64 ? column_ver_attr<double, 8, 32>() && column_ver_attr<double, 16, 16>()
                    : column_ver_attr<float, 8, 32>() && column_ver_attr<float, 32, 12>())) {
    lgame_set_error("split precision: shared memory of the vertical solver refused");
    return LGAME_ERR_CUDA;
  }
  if (diff.mom_h &&
      (cudaFuncSetAttribute(k_diff_scalar_col<7, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)diff_scalar_smem(8)) != cudaSuccess ||
       cudaFuncSetAttribute(k_diff_scalar_col<7, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)diff_scalar_smem(7)) != cudaSuccess)) {
    lgame_set_error("split precision: shared memory of the scalar diffusion kernel refused");
    return LGAME_ERR_CUDA;
  }
  auto* s = new SplitCtx();
  s->column_fp64 = column_fp64;
  const size_t F = (size_t)D.fstride;
  int rc = LGAME_OK;
  auto fail = [&](int code) { split_destroy(s); *out = nullptr; return code; };
  for (int k = 0; k < 40; ++k) if ((rc = salloc(s, &s->gf[k], F, bytes))) return fail(rc);
  for (int k = 0; k < 6; ++k) if ((rc = salloc(s, &s->ipw[k], F, bytes))) return fail(rc);
  for (int k = 0; k < 3; ++k) if ((rc = salloc(s, &s->trsk_u[k], (size_t)D.P, bytes))) return fail(rc);
  for (int k = 0; k < 2; ++k) if ((rc = salloc(s, &s->trsk_v[k], (size_t)D.P, bytes))) return fail(rc);
  if ((rc = salloc(s, &s->inv_dx, F, bytes)) || (rc = salloc(s, &s->inv_dy, F, bytes)) ||
      (rc = salloc(s, &s->inv_dz, F, bytes)) || (rc = salloc(s, &s->inv_volume, F, bytes)) ||
      (rc = salloc(s, &s->inv_area_z, F, bytes)))
    return fail(rc);
  float** scratch[] = {&s->gx, &s->gy, &s->divf, &s->tvu, &s->tvv, &s->tpu, &s->tpv,
                       &s->ex, &s->ey, &s->ez, &s->uph, &s->vph, &s->wph};
  for (float** p : scratch) if ((rc = salloc(s, p, F, bytes))) return fail(rc);
  s->sfc = sfc;
  if (sfc.vsq) s->vsq = sfc.vsq;
  else if ((rc = salloc(s, &s->vsq, F, bytes))) return fail(rc);
  if ((rc = salloc(s, &s->gzd, F, bytes)) || (rc = salloc(s, &s->rmz, F, bytes))) return fail(rc);
  if (D.nc > 0 && (rc = salloc(s, &s->csh_part, F * 2, bytes))) return fail(rc);
  if (D.ncons > 1 && (rc = salloc(s, &s->cw, F, bytes))) return fail(rc);
  if ((rc = salloc(s, &s->dbg, F, bytes)) || (rc = salloc(s, &s->tbu, F, bytes)) || (rc = salloc(s, &s->tbv, F, bytes)))
    return fail(rc);
  float** fl[] = {&s->fu, &s->fv, &s->gu, &s->gv};
  for (float** p : fl) if ((rc = salloc(s, p, F, bytes))) return fail(rc);
  for (int k = 0; k < 2; ++k) {
    StateF& M = s->mir[k];
    if ((rc = salloc(s, &M.rho, F * D.ncons, bytes))) return fail(rc);
    float** mf[] = {&M.rt, &M.tp, &M.ep, &M.u, &M.v, &M.w};
    for (float** p : mf) if ((rc = salloc(s, p, F, bytes))) return fail(rc);
  }
  SplitCarriedF& C = s->C;
  float** car[] = {&C.pgcw, &C.vsg_x, &C.vsg_y, &C.vsg_z, &C.pvt_x, &C.pvt_y, &C.pvt_z, &C.csh, &C.rad, &C.temperature,
                   &C.hdiss,
                   &C.tend.rt, &C.tend.u, &C.tend.v, &C.tend.w, &C.pnet_u, &C.pnet_v, &C.pnet_w, &C.pold_u,
                   &C.pold_v};
  for (float** p : car) if ((rc = salloc(s, p, F, bytes))) return fail(rc);
  if ((rc = salloc(s, &C.tend.rho, F * D.ncons, bytes))) return fail(rc);
  s->diff = diff;
  if (diff.mom_h) {
    DiffBuf<float>& B = s->db;
    float** dfl[] = {&C.tke, &C.visc, &C.mdtx, &C.mdty, &C.mdtz, &B.tke_new, &B.vmol, &B.nsq, &B.vz, &B.tdh,
                     &B.zz, &B.vdiv};
    for (float** p : dfl) if ((rc = salloc(s, p, F, bytes))) return fail(rc);
    if ((rc = salloc(s, &B.mdt, F * D.ncons, bytes))) return fail(rc);
    // (no flux density arrays: the scalar diffusion forms its faces in shared memory)
    B.tke = C.tke; B.visc = C.visc; B.mdtx = C.mdtx; B.mdty = C.mdty; B.mdtz = C.mdtz; B.hd = C.hdiss;
    C.tdh = B.tdh; C.mdt = B.mdt;
  }
  if (sfc.phase) {  // the phase transitions' rates (graupel's is never written: stays zero) and heating
    if ((rc = salloc(s, &C.ptr, F * (size_t)(D.nc + 1), bytes)) || (rc = salloc(s, &C.pth, F, bytes))) return fail(rc);
  }
  for (cudaStream_t& b : s->br)
    if (cudaStreamCreateWithFlags(&b, cudaStreamNonBlocking) != cudaSuccess) {
      lgame_set_error("split precision: cudaStreamCreate failed");
      return fail(LGAME_ERR_CUDA);
    }
  for (cudaEvent_t& e : s->ev)
    if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
      lgame_set_error("split precision: cudaEventCreate failed");
      return fail(LGAME_ERR_CUDA);
    }
  *out = s;
  return LGAME_OK;
}

void split_set_diff_par(SplitCtx* s, const DiffPar& par) { s->diff.par = par; }
void split_set_sfc_par(SplitCtx* s, const SfcPar& par) { s->sfc.par = par; }

void split_destroy(SplitCtx* s) {
  if (!s) return;
  for (void* p : s->allocs) cudaFree(p);
  for (cudaEvent_t e : s->ev) if (e) cudaEventDestroy(e);
  for (cudaStream_t b : s->br) if (b) cudaStreamDestroy(b);
  delete s;
}

SplitCarriedF split_carried(SplitCtx* s) { return s->C; }
StateF split_mirror(SplitCtx* s, int slot) { return s->mir[slot]; }

int split_net(const double* a, const double* b, float* net, long long n, cudaStream_t stream) {
  k_net<<<1216, 256, 0, stream>>>(a, b, net, n);
  return cudaGetLastError() == cudaSuccess ? LGAME_OK : LGAME_ERR_CUDA;
}

int split_convert(const double* src, float* dst, long long n, cudaStream_t stream) {
  k_to_float<<<1216, 256, 0, stream>>>(src, dst, n);
  return cudaGetLastError() == cudaSuccess ? LGAME_OK : LGAME_ERR_CUDA;
}
int split_convert_back(const float* src, double* dst, long long n, cudaStream_t stream) {
  k_to_double<<<1216, 256, 0, stream>>>(src, dst, n);
  return cudaGetLastError() == cudaSuccess ? LGAME_OK : LGAME_ERR_CUDA;
}

// ---- lateral boundary relaxation (mo_boundaries.F90:19-97) in split precision -------------
namespace {
__global__ void k_rtbg(const double* exner_bg, double* rtbg, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    rtbg[i] = kP_0 / kR_D * pow(exner_bg[i], kC_D_V / kR_D);
}

// Two kernels.  ks_bc_rim relaxes the swamp layer only: one thread per (listed plane point,
// level), the points being those where any of the three rescale factors is nonzero, with the
// FP64 blend x = f*(w_old*x_old + w_new*x_new) + (1 - f)*x of every field (FP32 mirror rounded
// from it).  Everywhere else the reference's 0*(...) + 1*x is x (for finite boundary data and
// a nonzero x), so nothing is written there.  ks_bc_thermo then recomputes theta_v_pert and
// exner_pert at every scalar point with one FP64 operation each:
//   theta_v_pert = (rhotheta_v - rho_gas*theta_v_bg)/rho_gas, the numerator in FP64 and
//                  the division in FP32 (relative error ~1e-7 of theta_v_pert),
//   exner_pert   = (r_d*rhotheta_v/p_0)^(r_d/c_d_v) - exner_bg
//                = exner_bg*((1 + d)^kappa - 1) = exner_bg*expm1(kappa*log1p(d)),
//                  d = (rhotheta_v - rt_bg)/rt_bg with rt_bg the background's rhotheta_v,
//                  in FP32 after the FP64 difference (relative error ~1e-7 of exner_pert).
// Keeping the blend out of the second kernel matters on this GPU: a warp covers 32 rows, so
// with one kernel every warp that touches the swamp layer issued the whole FP64 blend.

// (1 + d)^kappa - 1 in FP32 for |d| <= 0.25 from series with multiply-adds only:
// log1p(d) = 2 atanh(s) = 2 (s + s^3/3 + ... + s^13/13), s = d/(2 + d), |s| <= 1/7, and
// expm1(y) = y + y^2/2! + ... + y^8/8!, |y| = |kappa log1p(d)| <= 0.12 (truncation errors
// below 1e-11 relative); larger |d| goes through log1pf and expm1f.
__device__ __forceinline__ float pow1p_m1(float d, float kappa) {
  if (fabsf(d) > 0.25f) return expm1f(kappa * log1pf(d));
  const float sv = d / (2.f + d), s2 = sv * sv;
  float t = 1.f / 13.f;
  t = fmaf(t, s2, 1.f / 11.f);
  t = fmaf(t, s2, 1.f / 9.f);
  t = fmaf(t, s2, 1.f / 7.f);
  t = fmaf(t, s2, 1.f / 5.f);
  t = fmaf(t, s2, 1.f / 3.f);
  t = fmaf(t, s2, 1.f);
  const float y = kappa * (2.f * sv * t);
  float e = 1.f / 40320.f;
  e = fmaf(e, y, 1.f / 5040.f);
  e = fmaf(e, y, 1.f / 720.f);
  e = fmaf(e, y, 1.f / 120.f);
  e = fmaf(e, y, 1.f / 24.f);
  e = fmaf(e, y, 1.f / 6.f);
  e = fmaf(e, y, 0.5f);
  e = fmaf(e, y, 1.f);
  return y * e;
}
// the factors are +0 or positive: a bit test instead of an FP64 comparison

// grid (ceil(nrim/128), NL), 128 threads; rim[r] = plane index (ji-1) + P*(jk-1)
__global__ void __launch_bounds__(128) ks_bc_rim(Dims D, State S, StateF M, State B0, State B1, const int* rim, int nrim,
                                                 const double* fs, const double* fu, const double* fv, double ow,
                                                 double nw) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrim) return;
  const int p = rim[r], ji = p % D.P + 1, jk = p / D.P + 1, jl = blockIdx.y + 1;
  const bool mir = M.rho != nullptr;
  auto relax = [&](double f, const double* b0, const double* b1, double* x, float* xm, long long q) {
    const double v = f * (ow * b0[q] + nw * b1[q]) + (1.0 - f) * x[q];
    x[q] = v;
    if (mir) xm[q] = narrow(v);
  };
  const long long q = IX(D, ji, jk, jl);
  if (ji <= D.ny && jk <= D.nx && nonzero(fs[p])) {
    const double f = fs[p];
    if (jl <= D.nl) {
      for (int jc = 0; jc < D.ncons; ++jc) relax(f, B0.rho, B1.rho, S.rho, M.rho, q + (long long)jc * D.fstride);
      relax(f, B0.rt, B1.rt, S.rt, M.rt, q);
    }
    relax(f, B0.w, B1.w, S.w, M.w, q);
  }
  if (jl <= D.nl && ji <= D.ny && jk <= D.nx + 1 && nonzero(fu[p])) relax(fu[p], B0.u, B1.u, S.u, M.u, q);
  if (jl <= D.nl && ji <= D.ny + 1 && jk <= D.nx && nonzero(fv[p])) relax(fv[p], B0.v, B1.v, S.v, M.v, q);
}

__global__ void __launch_bounds__(256) ks_bc_thermo(Dims D, State S, StateF M, const double* theta_v_bg,
                                                    const double* exner_bg, const double* rtbg) {
  LG_IDX3;
  if (ji > D.ny || jk > D.nx) return;
  const long long q = IX(D, ji, jk, jl);
  const double rho_g = S.rho[q + (long long)(D.g - 1) * D.fstride], rt = S.rt[q];
  const double tb = theta_v_bg[q], rb = rtbg[q], eb = exner_bg[q];
  const float tpf = narrow(fma(-rho_g, tb, rt)) / narrow(rho_g);
  const float d = narrow(rt - rb) / narrow(rb);
  const float epf = narrow(eb) * pow1p_m1(d, (float)(kR_D / kC_D_V));
  S.tp[q] = wide(tpf);
  S.ep[q] = wide(epf);
  if (M.tp) {
    M.tp[q] = tpf;
    M.ep[q] = epf;
  }
}
}  // namespace

int split_bc_prepare(SplitCtx* s, const Dims& D, const Grid<double>& G, cudaStream_t stream) {
  if (!s->rtbg) {
    long long bytes = 0;
    if (salloc(s, &s->rtbg, (size_t)D.fstride, &bytes)) return LGAME_ERR_ALLOC;
  }
  k_rtbg<<<1216, 256, 0, stream>>>(G.exner_bg, s->rtbg, D.fstride);
  return cudaGetLastError() == cudaSuccess ? LGAME_OK : LGAME_ERR_CUDA;
}

int split_bc_update(SplitCtx* s, const Dims& D, const Grid<double>& G, const State& S, const StateF& M, const State& B0,
                    const State& B1, const int* rim, int nrim, const double* fs, const double* fu, const double* fv,
                    double ow, double nw, cudaStream_t stream) {
  if (!s->rtbg) return LGAME_ERR_STATE;
  if (nrim > 0)
    ks_bc_rim<<<dim3((unsigned)((nrim + 127) / 128), (unsigned)D.NL), 128, 0, stream>>>(D, S, M, B0, B1, rim, nrim, fs, fu,
                                                                                        fv, ow, nw);
  ks_bc_thermo<<<sgrd(D.ny, D.nx, D.nl), dim3(32, 8), 0, stream>>>(D, S, M, G.theta_v_bg, G.exner_bg, s->rtbg);
  return cudaGetLastError() == cudaSuccess ? LGAME_OK : LGAME_ERR_CUDA;
}

int split_refresh_mirror(SplitCtx* s, const Dims& D, int slot, const State& S, cudaStream_t stream) {
  const long long F = D.fstride;
  const StateF& M = s->mir[slot];
  if (split_convert(S.rho, M.rho, F * D.ncons, stream)) return LGAME_ERR_CUDA;
  const double* src[] = {S.rt, S.tp, S.ep, S.u, S.v, S.w};
  float* dst[] = {M.rt, M.tp, M.ep, M.u, M.v, M.w};
  for (int k = 0; k < 6; ++k)
    if (split_convert(src[k], dst[k], F, stream)) return LGAME_ERR_CUDA;
  return LGAME_OK;
}

int split_set_grid(SplitCtx* s, const Dims& D, const Grid<double>& G, cudaStream_t stream) {
  const long long F = D.fstride;
  const double* src[] = {G.z_scalar, G.z_u, G.z_v, G.z_w, G.dx, G.dy, G.dz, G.volume, G.area_x, G.area_y, G.area_z,
                         G.area_dual_x, G.area_dual_y, G.area_dual_z, G.z_area_dual_z, G.slope_x, G.slope_y,
                         G.theta_v_bg, G.exner_bg, G.egu, G.egv, G.egw, G.gm, G.gp, G.fvec_x, G.fvec_y, G.fvec_z,
                         G.damp};
  const double* src2[] = {G.dx_dual, G.dy_dual, G.layer_thickness};  // -> gf[33..35]
  const int nsrc = sizeof(src) / sizeof(src[0]);
  for (int k = 0; k < nsrc; ++k) {
    const long long n = (src[k] == G.fvec_x || src[k] == G.fvec_y || src[k] == G.fvec_z) ? D.plane : F;
    if (split_convert(src[k], s->gf[k], n, stream)) return LGAME_ERR_CUDA;
  }
  for (int k = 0; k < 3; ++k) if (split_convert(src2[k], s->gf[33 + k], F, stream)) return LGAME_ERR_CUDA;
  for (int k = 0; k < 6; ++k) if (split_convert(G.ipw[k], s->ipw[k], F, stream)) return LGAME_ERR_CUDA;
  for (int k = 0; k < 3; ++k) if (split_convert(G.trsk_u[k], s->trsk_u[k], D.P, stream)) return LGAME_ERR_CUDA;
  for (int k = 0; k < 2; ++k) if (split_convert(G.trsk_v[k], s->trsk_v[k], D.P, stream)) return LGAME_ERR_CUDA;
  k_recip<<<1216, 256, 0, stream>>>(G.dx, s->inv_dx, F);
  k_recip<<<1216, 256, 0, stream>>>(G.dy, s->inv_dy, F);
  k_recip<<<1216, 256, 0, stream>>>(G.dz, s->inv_dz, F);
  k_recip<<<1216, 256, 0, stream>>>(G.volume, s->inv_volume, F);
  k_recip<<<1216, 256, 0, stream>>>(G.area_z, s->inv_area_z, F);
  float* ivol = s->gf[28];
  float* iaz = s->gf[29];
  float* dzs = s->gf[30];
  float* deb = s->gf[31];
  float* kd = s->gf[32];
  k_grid_extra<<<sgrd(D.ny, D.nx, D.NL), sblk(), 0, stream>>>(D, G, ivol, iaz, dzs, deb, kd);
  if (cudaGetLastError() != cudaSuccess) return LGAME_ERR_CUDA;
  Grid<float>& GF = s->GF;
  float** g = s->gf;
  GF.z_scalar = g[0]; GF.z_u = g[1]; GF.z_v = g[2]; GF.z_w = g[3]; GF.dx = g[4]; GF.dy = g[5]; GF.dz = g[6];
  GF.volume = g[7]; GF.area_x = g[8]; GF.area_y = g[9]; GF.area_z = g[10]; GF.area_dual_x = g[11];
  GF.area_dual_y = g[12]; GF.area_dual_z = g[13]; GF.z_area_dual_z = g[14]; GF.slope_x = g[15]; GF.slope_y = g[16];
  GF.theta_v_bg = g[17]; GF.exner_bg = g[18]; GF.egu = g[19]; GF.egv = g[20]; GF.egw = g[21]; GF.gm = g[22];
  GF.gp = g[23]; GF.fvec_x = g[24]; GF.fvec_y = g[25]; GF.fvec_z = g[26]; GF.damp = g[27];
  GF.dx_dual = g[33]; GF.dy_dual = g[34]; GF.layer_thickness = g[35];
  for (int k = 0; k < 6; ++k) GF.ipw[k] = s->ipw[k];
  for (int k = 0; k < 3; ++k) GF.trsk_u[k] = s->trsk_u[k];
  for (int k = 0; k < 2; ++k) GF.trsk_v[k] = s->trsk_v[k];
  s->GX = GridX{s->inv_dx, s->inv_dy, s->inv_dz, s->inv_volume, s->inv_area_z, ivol, iaz, dzs, deb, kd};
  // the third-order theta chain of the background, in FP64 on temporary arrays that start at 0
  // (the levels and boundary faces the chain does not write are read as 0)
  double* tmp[4] = {};
  bool ok = true;
  for (double*& t : tmp) {
    ok = ok && cudaMalloc(&t, (size_t)F * sizeof(double)) == cudaSuccess &&
         cudaMemsetAsync(t, 0, (size_t)F * sizeof(double), stream) == cudaSuccess;
  }
  if (ok) {
    const dim3 B = sblk();
    k_grad_vert<double, double><<<sgrd(D.ny, D.nx, D.nl - 1), B, 0, stream>>>(D, G, G.theta_v_bg, tmp[0]);
    k_grad_hor<double, double><<<sgrd(D.ny + 1, D.nx + 1, D.nl), B, 0, stream>>>(D, G, G.theta_v_bg, tmp[0], tmp[1],
                                                                                  tmp[2]);
    k_div_h<double><<<sgrd(D.ny, D.nx, D.nl), B, 0, stream>>>(D, G, tmp[1], tmp[2], tmp[3]);
    k_to_float<<<1216, 256, 0, stream>>>(tmp[3], s->dbg, F);
    k_bg_faces<<<sgrd(D.ny + 1, D.nx + 1, D.nl), B, 0, stream>>>(D, G, s->tbu, s->tbv);
    ok = cudaGetLastError() == cudaSuccess && cudaStreamSynchronize(stream) == cudaSuccess;
  }
  for (double* t : tmp) if (t) cudaFree(t);
  if (!ok) {
    lgame_set_error("split set-up: theta chain of the background state failed");
    return LGAME_ERR_CUDA;
  }
  return LGAME_OK;
}

int split_step(SplitCtx* s, const Dims& D, const Grid<double>& G, const State& So, const State& Sn, int so, int sn,
               const PGrad<double>& pg, int step, cudaStream_t stream, int* nk,
               int (*tb)(void*, const char*), void (*te)(void*, int), void* tracer, bool serial) {
  const Grid<float>& GF = s->GF;
  const SplitCarriedF& C = s->C;
  const Tend<float> T = C.tend;
  const StateF& Mo = s->mir[so];
  const StateF& Mn = s->mir[sn];
  int launches = 0;
  // Kernels that do not depend on each other run on side streams, forked from and joined back
  // into `stream` by events:
  //   first substep:  the closure, swamp-layer heating and phase transitions (FP32 and
  //                   latency-bound) beside the theta edges and the FP64 pressure gradient;
  //   both substeps:  the tracer tendencies beside the vertical solve;
  //   between them:   the first substep's tracer solver beside the second substep's vorticity,
  //                   kinetic energy (FP64, on a second side stream) and wind update, which waits
  //                   for the first substep's tracer tendencies (they read the wind it overwrites).
  // Every two kernels of which one writes what the other reads or writes are ordered
  // (tests/test_split_order.py); with `serial` (per-kernel tracing, and the caller's graph capture,
  // where the serial order measured faster) everything runs on `stream` in the same order.
  const bool conc = !serial;
  cudaStream_t cur = stream;
  cudaStream_t side = conc ? s->br[0] : stream, side2 = conc ? s->br[1] : stream;
  enum { EV_A = 0, EV_JA, EV_B, EV_C, EV_CSH, EV_KE, EV_JKE, EV_END, EV_TR };
  // `to` starts after everything enqueued on `from` so far
  auto after = [&](cudaStream_t to, cudaStream_t from, int k) -> int {
    if (!conc || to == from) return LGAME_OK;
    if (cudaEventRecord(s->ev[k], from) != cudaSuccess || cudaStreamWaitEvent(to, s->ev[k], 0) != cudaSuccess) {
      lgame_set_error("split step: fork/join event failed");
      return LGAME_ERR_CUDA;
    }
    return LGAME_OK;
  };
#define SL(name, kernel, grid_, block_, ...) SLS(name, kernel, grid_, block_, 0, __VA_ARGS__)
#define SLS(name, kernel, grid_, block_, smem_, ...)                            \
  do {                                                                          \
    const int tr_ = tb ? tb(tracer, name) : -1;                                 \
    kernel<<<grid_, block_, smem_, cur>>>(__VA_ARGS__);                         \
    if (tr_ >= 0) te(tracer, tr_);                                              \
    cudaError_t e_ = cudaGetLastError();                                        \
    if (e_ != cudaSuccess) {                                                    \
      lgame_set_error((std::string("launch of ") + name + ": " + cudaGetErrorString(e_)).c_str()); \
      return LGAME_ERR_CUDA;                                                    \
    }                                                                           \
    ++launches;                                                                 \
  } while (0)
#define SYNC(call)                   \
  do {                               \
    const int rc_ = (call);          \
    if (rc_ != LGAME_OK) return rc_; \
  } while (0)
  const dim3 B = sblk();
  // third-order theta edges: the gradient of theta' (read from the mirror) and its divergence
  auto theta_div = [&](const float* tp) -> int {
    SL("ks_grad", (ks_grad<float, false>), cgrd_levels(D, D.ny + 1, D.nx + 1), cblk(), D, GF, tp, s->gx, s->gy,
       (float*)nullptr);
    SL("ks_div_h", ks_div_h, cgrd_levels(D, D.ny, D.nx), cblk(), D, GF, s->GX, s->gx, s->gy, s->divf);
    return LGAME_OK;
  };
  SL("ks_temperature", (k_temperature<float, float>), sgrd(D.ny, D.nx, D.nl), B, D, GF, Mo, C.temperature);
  // the surface parts in FP64 on the FP64 state (two-dimensional): update_sfc_turb_quantities
  // before the substeps (mo_manage_pchevi.F90:51-53)
  const SplitSfc& SF = s->sfc;
  if (SF.turb) SL("ks_sfc_turb", k_sfc_turb<float>, sgrd(D.ny, D.nx, 1), B, D, G, So, s->vsq, SF.buf, SF.par);
  Carried<float> CC{pg.nl_u, pg.nl_v, pg.nl_w, pg.l_u, pg.l_v, pg.l_w, pg.old_u, pg.old_v, C.pgcw,
                    C.vsg_x, C.vsg_y, C.vsg_z, C.pvt_x, C.pvt_y, C.pvt_z};
  const SplitDiff& SD = s->diff;
  const DiffBuf<float>& DB = s->db;
  const bool vort = !D.llinear || D.lcorio, tracers = D.ncons > 1;
  const float* mdt = (SD.mom_h && SD.mass_h) ? DB.mdt : nullptr;
  const float* tdh = (SD.mom_h && SD.temp_h) ? DB.tdh : nullptr;
  const float* ptr = SF.phase ? C.ptr : nullptr;
  const float* pth = SF.phase ? C.pth : nullptr;
  if (SD.mom_h) { CC.mdt_x = DB.mdtx; CC.mdt_y = DB.mdty; CC.mdt_z = DB.mdtz; }
  // the vorticity flux and the kinetic-energy gradient of state Sv (mirror Mv); with `branch`
  // the kinetic energy (FP64) runs on the second side stream beside the vorticity (FP32)
  auto vector_terms = [&](const State& Sv, const StateF& Mv, bool branch) -> int {
    if (!vort) return LGAME_OK;
    const bool ke = !D.llinear;
    if (ke && branch) {
      SYNC(after(side2, stream, EV_KE));
      cur = side2;
    }
    if (ke) {
      SL("ks_ke", ks_ke, sgrd(D.ny, D.nx, D.nl), B, D, G, Sv, s->vsq);
      SL("ks_grad", (ks_grad<double, true>), cgrd_levels(D, D.ny + 1, D.nx + 1), cblk(), D, GF, s->vsq, C.vsg_x, C.vsg_y,
         C.vsg_z);
    }
    cur = stream;
    const dim3 gp = cgrd_levels(D, D.ny + 1, D.nx + 1), ge(gp.x, gp.y, gp.z + 1);
    SL("ks_eta", ks_eta, ge, cblk(), D, GF, Mv, s->ex, s->ey, s->ez, s->uph, s->vph, s->wph);
    SL("ks_vort_flux", ks_vort_flux, gp, cblk(), D, GF, Mv, s->ex, s->ey, s->ez, s->uph, s->vph, s->wph, C.pvt_x,
       C.pvt_y, C.pvt_z);
    if (ke && branch) SYNC(after(stream, side2, EV_JKE));
    return LGAME_OK;
  };
  for (int rk = 1; rk <= 2; ++rk) {
    const StateF& Ms = (rk == 1) ? Mo : Mn;
    if (rk == 1) {
      // side: the closure (momentum diffusion, dissipation, scalar diffusion), or the swamp
      // layer's heating, and the phase transitions: they read the old mirror, its temperature
      // and the surface quantities, and write only their own buffers (DB, hdiss, ptr/pth, the
      // latent fluxes).  main: theta edges, gzp, pressure gradient (scratch gx..divf, tvu..tpv,
      // gzd, rmz, the pressure-gradient arrays).  Joined before the wind update.
      const bool side_work = SD.mom_h || (D.lklemp && D.ndamp > 0) || SF.phase;
      // step 0 forms the vector terms at the first substep too (mo_vector_tend_expl.F90:41-98),
      // before the closure: the PBL reads the kinetic energy they form
      if (step == 0) SYNC(vector_terms(So, Mo, false));
      if (side_work) {
        SYNC(after(side, stream, EV_A));
        cur = side;
      }
      if (SD.mom_h) {
        const dim3 gs = sgrd(D.ny, D.nx, D.nl);
        SL("ks_diff_tke", ks_diff_tke, cgrd_levels(D, D.ny, D.nx), cblk(), D, GF, Mo, DB, SD.par);
        SL("ks_diff_zeta", (k_diff_zeta<float, float>), sgrd(D.ny + 1, D.nx + 1, D.nl), B, D, GF, Mo, DB);
        SL("ks_diff_visc", ks_diff_visc, cgrd_levels(D, D.ny, D.nx), cblk(), D, GF, s->GX, Mo, (const float*)C.temperature,
           DB, SD.par);
        SL("ks_diff_vz", (k_diff_vz<float, float>), sgrd(D.ny + 1, D.nx + 1, D.nl), B, D, GF, Mo, DB);
        SL("ks_mom_diff_h", ks_mom_diff_h, cgrd_levels(D, D.ny, D.nx), cblk(), D, GF, Mo, DB);
        if (SD.mom_v) SL("ks_mom_diff_v", (k_mom_diff_v<float, float>), sgrd(D.ny, D.nx, D.nl - 1), B, D, GF, Mo, DB);
        if (SF.pbl)
          SL("ks_pbl", (k_pbl<float, float>), sgrd(D.ny, D.nx, 1), B, D, G, So, s->vsq, SF.buf, SF.par, DB.mdtx, DB.mdty);
        SL("ks_diss_rate", (k_diss_rate<float, float>), gs, B, D, GF, Mo, DB, GF.damp, s->GX.kdamp_f);
        // temperature and mass diffusion (mo_scalar_tend_expl.F90:60-101): fluxes and divergence of
        // every constituent and the temperature in one column-marching launch; the second
        // substep's temperature diffusion is the same (same temperature and coefficients)
        const dim3 gd((D.ny + DS_X - 1) / DS_X, (D.nx + DS_Y - 1) / DS_Y);
        if (SD.temp_h || SD.mass_h) {
          const float* tm = (const float*)C.temperature;
          const float* rm = (const float*)Mo.rho;
          const int vm = SD.mass_v ? 1 : 0, vt = SD.temp_v ? 1 : 0;
          const dim3 bd(DS_THREADS);
          if (SD.temp_h && SD.mass_h && D.ncons == 7)
            SLS("ks_diff_scalar", (k_diff_scalar_col<7, 1>), gd, bd, diff_scalar_smem(8), D, GF, Mo, DB, rm, vm, DB.mdt,
                tm, vt, DB.tdh);
          else if (SD.temp_h && SD.mass_h)
            SLS("ks_diff_scalar", (k_diff_scalar_col<1, 1>), gd, bd, diff_scalar_smem(2), D, GF, Mo, DB, rm, vm, DB.mdt,
                tm, vt, DB.tdh);
          else if (SD.temp_h)
            SLS("ks_diff_scalar", (k_diff_scalar_col<0, 1>), gd, bd, diff_scalar_smem(1), D, GF, Mo, DB, rm, 0,
                (float*)nullptr, tm, vt, DB.tdh);
          else if (D.ncons == 7)
            SLS("ks_diff_scalar", (k_diff_scalar_col<7, 0>), gd, bd, diff_scalar_smem(7), D, GF, Mo, DB, rm, vm, DB.mdt,
                tm, 0, (float*)nullptr);
          else
            SLS("ks_diff_scalar", (k_diff_scalar_col<1, 0>), gd, bd, diff_scalar_smem(1), D, GF, Mo, DB, rm, vm, DB.mdt,
                tm, 0, (float*)nullptr);
        }
      } else if (D.lklemp && D.ndamp > 0) {
        SL("ks_heating_diss", ks_heating_diss, sgrd(D.ny, D.nx, std::min(D.nl, D.ndamp)), B, D, GF, s->GX, Mo, C.hdiss);
      }
      // the phase transitions (extension) from state_old and its temperature, in FP64 on the FP64
      // state; both substeps read the rates
      if (SF.phase)
        SL("ks_phase_trans", (k_phase_trans<float, float>), sgrd(D.ny, D.nx, D.nl), B, D, G, So,
           (const float*)C.temperature, SF.buf, SF.tsoil[so], SF.phase_sfc ? 1 : 0, D.dtime, C.ptr, C.pth);
      cur = stream;
      if (D.theta_order == 3) {  // the edges of theta_v and, with a background state, of theta'
        SYNC(theta_div(Mo.tp));
        SL("ks_theta_edges", ks_theta_edges, sgrd(D.ny + 1, D.nx + 1, D.nl), B, D, Mo.tp, s->divf, s->dbg, s->tbu, s->tbv,
           Mo.u, Mo.v, s->tvu, s->tvv, D.luse_bg ? s->tpu : nullptr, D.luse_bg ? s->tpv : nullptr);
      }
      SL("ks_gzp", ks_gzp, sgrd(D.ny, D.nx, D.nl), B, D, G, s->GX, So.ep, Mo.rho, s->gzd, s->rmz, s->gu);
      SL("ks_pgrad", (D.theta_order == 2 ? ks_pgrad<double> : ks_pgrad<float>), sgrd(D.ny + 1, D.nx + 1, D.nl), B, D, G,
         s->GX, So, s->gzd, s->rmz, s->gu, s->tvu, s->tvv, s->tpu, s->tpv, pg, C, C.pgcw, step == 0 ? 1 : 0);
      if (side_work) SYNC(after(stream, side, EV_JA));
    } else {
      // main: vorticity of the new state; side 2: its kinetic energy (FP64); both read the state
      // of the first substep (u, v from its wind update, w and rho_g from its vertical solve),
      // which the tracer tendencies and the tracer solver still running on the side stream do not write
      SYNC(vector_terms(Sn, Mn, true));
      // the first substep's tracer tendencies, on the side stream, read the wind written next
      if (tracers && conc && cudaStreamWaitEvent(stream, s->ev[EV_TR], 0) != cudaSuccess) {
        lgame_set_error("split step: join event failed");
        return LGAME_ERR_CUDA;
      }
    }
    SL("ks_tend_wind", ks_tend_wind, sgrd(D.ny + 1, D.nx + 1, D.NL), B, D, So, Sn, T, CC, C, rk, Mn.u, Mn.v);
    // gas fluxes with third-order theta edges of the state used here; in the first substep that is the
    // old state, whose edges the pressure gradient's call above already left in tvu/tvv (nothing
    // in between writes the old mirror or tvu/tvv), so only the second substep forms them anew
    if (D.theta_order == 3 && rk == 2) {
      SYNC(theta_div(Ms.tp));
      SL("ks_theta_flux", ks_theta_flux, sgrd(D.ny + 1, D.nx + 1, D.nl), B, D, Ms, s->divf, s->dbg, s->tbu, s->tbv, s->fu,
         s->fv, s->gu, s->gv);
    } else {
      SL("ks_gas_flux", ks_gas_flux, sgrd(D.ny + 1, D.nx + 1, D.nl), B, D, GF, Ms, Mn.u, Mn.v, s->tvu, s->tvv, s->fu,
         s->fv, s->gu, s->gv);
    }
    // the second substep's gas divergence reads every density of the new mirror (the heat
    // capacity) and the sediment heating: it waits for the first substep's tracer solver
    if (rk == 2 && tracers && conc) {
      if (cudaStreamWaitEvent(stream, s->ev[EV_CSH], 0) != cudaSuccess) {
        lgame_set_error("split step: join event failed");
        return LGAME_ERR_CUDA;
      }
    }
    SL("ks_gas_div", (tracers ? ks_gas_div<true> : ks_gas_div<false>), cgrd_levels(D, D.ny, D.nx), cblk(), D, GF, s->GX, Ms, s->fu,
       s->fv, s->gu, s->gv, C.temperature, C.hdiss, C.rad, C.csh, T.rho, T.rt, mdt, tdh, ptr, pth, Mn.u, Mn.v, s->cw);
    // side: the tracer tendencies (read the tracer densities of Ms and the new u, v; write the
    // tracer fields of T.rho), after the gas divergence, which leaves cw, beside the vertical solve, which
    // writes the gas density, theta', exner', rhotheta_v and w
    if (tracers) {
      SYNC(after(side, stream, EV_B));
      cur = side;
      SL("ks_tracers", ks_tracers, sgrd(D.ny, D.nx, D.nl), B, D, GF, s->GX, Ms, Mn.u, Mn.v, s->cw, T.rho, rk, mdt, ptr);
      if (rk == 1 && conc && cudaEventRecord(s->ev[EV_TR], side) != cudaSuccess) {
        lgame_set_error("split step: event record failed");
        return LGAME_ERR_CUDA;
      }
      cur = stream;
    }
    if (SF.sens || SF.soil)
      SL("ks_sfc_column", k_sfc_column_split<float>, sgrd(D.ny, D.nx, 1), B, D, G, So, rk == 1 ? So : Sn, T.rt,
         SF.buf, SF.par, SF.tsoil[so], SF.tsoil[rk == 1 ? so : sn], SF.tsoil[sn]);
    // The vertical solve by the number of columns: up to 8 columns an SM, 8 a block with 32 chunks of
    // levels (31 us at 1,024 columns of 60 layers; 45 with 32 x 12); up to the size that gives
    // every SM sub-partition three warps of columns, 32 a block with 12 chunks (124 us at 16,384
    // columns of 80 layers; 202 with 8 x 32); above, a thread a column (equal, 363 us, at 58,320 columns of
    // 80 layers; 171 against 296 at 22,500).  The FP64-coefficient solve keeps twice the shared memory
    // a column and takes 16 columns a block.
    const long long cols = (long long)D.ny * D.nx;
#define CV_ARGS D, G, GF, s->GX, So, Sn, Mo, Mn, T, rk
#define CV_TILE(C, TC, NW)                                                                              \
  SLS("ks_column_ver", (ks_column_ver_tile<C, TC, NW>), dim3((unsigned)((cols + TC - 1) / TC)), dim3(TC * NW), \
      (column_ver_smem<C, TC>(D.nl)), CV_ARGS)
    const bool tiny = cols <= kSMs * 8LL, small = cols <= kSMs * 4LL * 32 * 3;
    if (s->column_fp64) {
      if (tiny) CV_TILE(double, 8, 32);
      else if (small) CV_TILE(double, 16, 16);
      else SL("ks_column_ver", (D.luse_bg ? ks_column_ver<double, true> : ks_column_ver<double, false>), cgrd(D.ny, D.nx),
              cblk(), CV_ARGS);
    } else {
      if (tiny) CV_TILE(float, 8, 32);
      else if (small) CV_TILE(float, 32, 12);
      else SL("ks_column_ver", (D.luse_bg ? ks_column_ver<float, true> : ks_column_ver<float, false>), cgrd(D.ny, D.nx),
              cblk(), CV_ARGS);
    }
#undef CV_TILE
#undef CV_ARGS
    if (tracers) {
      // the two tracer sets fastest (the blocks of a row tile run together), row tiles, columns
      const dim3 gt(2u, (unsigned)((D.ny + 31) / 32), (unsigned)D.nx);
      if (rk == 1) {
        // side (after its tracer tendencies): the first substep's tracer solver and sediment
        // heating, which read w old and new and the gas density (final now) and write the
        // tracer densities and csh, beside the second substep's vorticity and wind update
        SYNC(after(side, stream, EV_C));
        cur = side;
        SLS("ks_column_tracers", ks_column_tracers<true>, gt, dim3(kTrWarps * 32), tracer_smem(D.nl), D, GF, s->GX, So,
            Sn, Mo, Mn, T.rho, C.temperature, s->csh_part);
        if (D.nc > 0) SL("ks_csh_sum", ks_csh_sum, sgrd(D.ny, D.nx, D.nl), B, D, s->csh_part, C.csh);
        if (conc && cudaEventRecord(s->ev[EV_CSH], side) != cudaSuccess) {
          lgame_set_error("split step: event record failed");
          return LGAME_ERR_CUDA;
        }
        cur = stream;
      } else {
        SYNC(after(stream, side, EV_END));
        SLS("ks_column_tracers", ks_column_tracers<false>, gt, dim3(kTrWarps * 32), tracer_smem(D.nl), D, GF, s->GX, So,
            Sn, Mo, Mn, T.rho, C.temperature, s->csh_part);
      }
    }
  }
#undef SL
#undef SLS
#undef SYNC
  *nk = launches;
  return LGAME_OK;
}

}  // namespace lg
