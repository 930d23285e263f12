// fp64.cuh -- FP64 arithmetic of the FP64 step in fewer operations of the FP64 pipe, which issues
// 1.6 operations per clock and SM on this GPU against 64 integer ones: with plain expressions every
// kernel of the step had that pipe at 80-88 % and everything else below 10 %, so its time was the
// number of these operations.  Every function returns the bits of the plain expression, with the exceptions
// stated beside it (tests/test_fp64_device.py compares them on the GPU).
#pragma once

#include <cstdint>

#include "kernels.cuh"

namespace lg {

// The hardware product, out of line: as a select the compiler would issue it beside the integer path.
static __device__ __noinline__ double mul_hw(double x, double y) { return x * y; }

// x*y rounded to nearest even in integer operations: the 53-bit mantissas multiplied in four 32 x 32
// bit products, normalised, the dropped bits folded into one.  On this GPU the FP64 pipe runs beside
// the integer ones, so a product formed here costs it nothing: chains of a product and a sum run at 3.15
// operations per clock and SM, against 1.60 with the hardware's product (1.89 for this product
// alone).  Factors outside 2^-510..2^511 take the hardware's, but zeros.
__device__ __forceinline__ double mul_int(double x, double y) {
  const uint32_t xh = (uint32_t)__double2hiint(x), xl = (uint32_t)__double2loint(x);
  const uint32_t yh = (uint32_t)__double2hiint(y), yl = (uint32_t)__double2loint(y);
  const uint32_t xe = xh & 0x7FF00000u, ye = yh & 0x7FF00000u;
  if (max(xe - (513u << 20), ye - (513u << 20)) >= (1022u << 20)) {
    const bool x0 = ((xh << 1) | xl) == 0u, y0 = ((yh << 1) | yl) == 0u;
    if ((x0 && ye < 0x7FF00000u) || (y0 && xe < 0x7FF00000u)) return __hiloint2double((int)((xh ^ yh) & 0x80000000u), 0);
    return mul_hw(x, y);
  }
  // mantissas as a < 2^54 and b < 2^64: the product is in [2^116, 2^118), its upper 64 bits hold 53 or 54
  const uint32_t ah = (__funnelshift_l(xl, xh, 1) & 0x1FFFFFu) | 0x200000u, al = xl << 1;
  const uint32_t bh = __funnelshift_l(yl, yh, 11) | 0x80000000u, bl = yl << 11;
  const uint64_t p00 = (uint64_t)al * bl;
  const uint64_t p01 = (uint64_t)al * bh + (p00 >> 32);
  const uint64_t p10 = (uint64_t)ah * bl + (uint32_t)p01;
  const uint64_t up = (uint64_t)ah * bh + (p01 >> 32) + (p10 >> 32);
  uint32_t hh = (uint32_t)(up >> 32), hl = (uint32_t)up;
  const uint32_t big = hh >> 21, sh = 1u - big, mid = (uint32_t)p10;
  // to 54 bits: the mantissa and the first dropped bit; t rounds (to even at a tie)
  hh = __funnelshift_l(hl, hh, sh);
  hl = __funnelshift_l(mid, hl, sh);
  const uint32_t t = ((hl >> 1) & 1u) | (((mid << sh) | (uint32_t)p00) != 0u ? 1u : 0u);
  const uint64_t r = ((((uint64_t)hh << 32) | hl) + t) >> 1;
  const uint32_t e = xe + ye - 0x3FF00000u - 0x00100000u + (big << 20);
  return __hiloint2double((int)(((uint32_t)(r >> 32) + e) ^ ((xh ^ yh) & 0x80000000u)), (int)(uint32_t)r);
}

// The same with a single-precision factor x, whose 24 bits leave two of the four partial products;
// subnormal and non-finite x take the hardware's.
__device__ __forceinline__ double mul_int(float x, double y) {
  const uint32_t xu = __float_as_uint(x), yh = (uint32_t)__double2hiint(y), yl = (uint32_t)__double2loint(y);
  const uint32_t xe = xu & 0x7F800000u, ye = yh & 0x7FF00000u;
  if ((xe - (1u << 23) >= (254u << 23)) | (ye - (513u << 20) >= (1022u << 20))) {
    const bool x0 = xu << 1 == 0u, y0 = ((yh << 1) | yl) == 0u;
    if ((x0 && ye < 0x7FF00000u) || (y0 && xe < 0x7F800000u)) return __hiloint2double((int)((xu ^ yh) & 0x80000000u), 0);
    return mul_hw(wide(x), y);
  }
  // mantissas as a < 2^32 and b < 2^54: the product is in [2^84, 2^86), its upper 64 bits hold 53 or 54
  const uint32_t a = (xu << 8) | 0x80000000u;
  const uint32_t bh = (__funnelshift_l(yl, yh, 1) & 0x1FFFFFu) | 0x200000u, bl = yl << 1;
  const uint64_t low = (uint64_t)a * bl, up = (uint64_t)a * bh + (low >> 32);
  uint32_t hh = (uint32_t)(up >> 32), hl = (uint32_t)up;
  const uint32_t big = hh >> 21, sh = 1u - big, mid = (uint32_t)low;
  hh = __funnelshift_l(hl, hh, sh);
  hl = __funnelshift_l(mid, hl, sh);
  const uint32_t t = ((hl >> 1) & 1u) | ((mid << sh) != 0u ? 1u : 0u);
  const uint64_t r = ((((uint64_t)hh << 32) | hl) + t) >> 1;
  const uint32_t e = (xe >> 3) + (896u << 20) + ye - 0x3FF00000u - 0x00100000u + (big << 20);
  return __hiloint2double((int)(((uint32_t)(r >> 32) + e) ^ ((xu ^ yh) & 0x80000000u)), (int)(uint32_t)r);
}

// x < 0 by the bits (a comparison issues on the FP64 pipe); -0 counts as negative, NaN does not
__device__ __forceinline__ bool negative(double x) {
  const unsigned u = (unsigned)__double2hiint(x) - 0x80000000u;
  return u < 0x7FF00000u || (u == 0x7FF00000u && __double2loint(x) == 0);
}
// x != 0 by the bits (NaN counts as nonzero)
__device__ __forceinline__ bool nonzero(double x) {
  return (((unsigned)__double2hiint(x) & 0x7FFFFFFFu) | (unsigned)__double2loint(x)) != 0u;
}

// x >= 0 by the bits (-0 included; true for a positive NaN too)
__device__ __forceinline__ bool upwind(double x) { return __double2hiint(x) >= 0 || !nonzero(x); }
// x > 0, but by the bits true for NaN too
__device__ __forceinline__ bool positive(double x) { return __double2hiint(x) >= 0 && nonzero(x); }

// x*2^-K, K = 1 or 2: the exponent lowered by K where it stays normal
template <int K>
__device__ __forceinline__ double scale_down(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), e = hi & 0x7FF00000u;
  if (e - ((unsigned)(K + 1) << 20) < ((2046u - K) << 20)) return __hiloint2double((int)(hi - ((unsigned)K << 20)), __double2loint(x));
  if (!nonzero(x)) return x;
  return (K == 1 ? 0.5 : 0.25) * x;
}
__device__ __forceinline__ double half(double x) { return scale_down<1>(x); }
__device__ __forceinline__ double quarter(double x) { return scale_down<2>(x); }

// a double whose products are formed by mul_int; sums are the hardware's.  Arrays of
// double are read and written as arrays of it.
struct F64 {
  double v;
  F64() = default;
  __host__ __device__ __forceinline__ constexpr F64(double x) : v(x) {}
};
__device__ __forceinline__ F64 operator-(F64 a) { return -a.v; }
__device__ __forceinline__ F64 operator+(F64 a, F64 b) { return a.v + b.v; }
__device__ __forceinline__ F64 operator-(F64 a, F64 b) { return a.v - b.v; }
__device__ __forceinline__ F64 operator*(F64 a, F64 b) { return mul_int(a.v, b.v); }
__device__ __forceinline__ bool operator>(F64 a, F64 b) { return a.v > b.v; }
__device__ __forceinline__ bool operator<(F64 a, F64 b) { return a.v < b.v; }
__device__ __forceinline__ bool operator>=(F64 a, F64 b) { return a.v >= b.v; }
__device__ __forceinline__ F64 half(F64 a) { return half(a.v); }
__device__ __forceinline__ F64 half_of(F64 a) { return half(a.v); }
__device__ __forceinline__ F64 quarter_of(F64 a) { return quarter(a.v); }
__device__ __forceinline__ bool negative(F64 a) { return negative(a.v); }
__device__ __forceinline__ bool nonzero(F64 a) { return nonzero(a.v); }
__device__ __forceinline__ bool upwind(F64 a) { return upwind(a.v); }
__device__ __forceinline__ bool positive(F64 a) { return positive(a.v); }
// 1/b to about a unit of the last place, b within 2^-100..2^99: the single-precision reciprocal of b's leading
// 24 bits (to 2^-21: the cut and two units of __fdividef) and one step of Halley's iteration, y(1 + e + e^2)
// with e = 1 - b*y, to e^3: three operations of the FP64 pipe
__device__ __forceinline__ bool near_range(double b) {
  return ((uint32_t)__double2hiint(b) & 0x7FF00000u) - (923u << 20) < (200u << 20);
}
__device__ __forceinline__ double rcp_start(double b) {
  const uint32_t hi = (uint32_t)__double2hiint(b), lo = (uint32_t)__double2loint(b);
  const float f = __uint_as_float((hi & 0x80000000u) | ((((hi & 0x7FFFFFFFu) - (896u << 20)) << 3) | (lo >> 29)));
  const double y = wide(__fdividef(1.f, f));
  const double e = fma(-b, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
static __device__ __noinline__ double div_hw(double a, double b) { return a / b; }
// the same for any b, the hardware's quotient outside that range
__device__ __forceinline__ double rcp_near(double b) { return near_range(b) ? rcp_start(b) : div_hw(1.0, b); }
// a remainder that is not finite (infinite or NaN operands, a zero divisor, overflow) corrects nothing: the
// quotient as it is then is the hardware's
__device__ __forceinline__ double corrected(double q, double r, double y) {
  return ((uint32_t)__double2hiint(r) & 0x7FF00000u) == 0x7FF00000u ? q : fma(r, y, q);
}
// 1/b and a/b rounded to nearest: value, remainder, correction (Markstein, IBM J. Res. Dev. 34, 1990).
// div_rn: b within 2^-100..2^99, 0, infinite or NaN, and y its reciprocal to 2^-50 (four units of the last
// place: also a product of two such reciprocals, for a rounded product of two divisors); the corrected quotient
// is off by the product of y's and q's errors, at most 2^-99, before it is rounded.  So the result is the
// correctly rounded one, except that
//   a value within 2^-46 of its last place from the middle of two doubles may round the other way;
//   a quotient below 2^-1022, and one of a dividend below 2^-960, whose remainder is not exact, may be off by
//   a unit of its last place;
//   a zero quotient's sign is not kept.
__device__ __forceinline__ double rcp(double b) {
  const double y = rcp_near(b);
  return corrected(y, fma(-b, y, 1.0), y);
}
__device__ __forceinline__ F64 rcp(F64 b) { return rcp(b.v); }
__device__ __forceinline__ F64 rcp_near(F64 b) { return rcp_near(b.v); }
__device__ __forceinline__ double div_rn(double a, double b, double y) {
  const double q = a * y;
  return corrected(q, fma(-b, q, a), y);
}
__device__ __forceinline__ F64 div_rn(F64 a, F64 b, F64 y) {
  const double q = mul_int(a.v, y.v);
  return corrected(q, fma(-b.v, q, a.v), y.v);
}
__device__ __forceinline__ double quot(double a, double b) { return near_range(b) ? div_rn(a, b, rcp_start(b)) : div_hw(a, b); }
__device__ __forceinline__ F64 operator/(F64 a, F64 b) {
  if (near_range(b.v)) return div_rn(a, b, rcp_start(b.v));
  return div_hw(a.v, b.v);
}

__device__ __forceinline__ F64 root(F64 a) { return sqrt(a.v); }
// calc_diff_coeff, mo_derived.F90:189-216
__device__ __forceinline__ F64 calc_diff_coeff(F64 temperature, F64 density) {
  constexpr double pm = kM_D / kN_A, c1 = kPI * pm, cross_section = 4.0 * kPI * (130e-12 * 130e-12);
  const F64 tv = root(div_rn(8.0 * kK_B * temperature, c1, 1.0 / c1));
  const F64 mfp = rcp(1.4142135623730951 * div_rn(density, pm, 1.0 / pm) * cross_section);
  return 1.0 / 3.0 * tv * mfp;
}

// the same arrays, read as F64
inline const F64* f64(const double* p) { return reinterpret_cast<const F64*>(p); }
inline F64* f64(double* p) { return reinterpret_cast<F64*>(p); }
inline const Grid<F64>& f64(const Grid<double>& g) { return reinterpret_cast<const Grid<F64>&>(g); }
inline const StateT<F64>& f64(const StateT<double>& s) { return reinterpret_cast<const StateT<F64>&>(s); }

// reciprocals of the metrics at their own points, formed once with the grid
struct Recip {
  const F64 *vol, *dx, *dy, *dz;
};
// what a face hands to the divergences of its two cells: flux times area and the slope term
// 0.5*f*slope, x at u points, y at v points
struct Faces {
  F64 *px, *py, *hx, *hy;
};

// grid-only factors of the vorticity: in the terrain-following layers, for each side of a dual point,
// (r_e + z_dual)/(r_e + z_side) times its length, with the side's sign
struct RotGrid {
  const F64 *m0, *m1, *m2, *m3;
};

// the explicit kernels (kernels_fp64.cu)
void launch64_rot_grid(const Dims& D, const Grid<double>& G, double* const* a, cudaStream_t st);
void launch64_zeta_z(const Dims& D, const Grid<double>& G, const RotGrid& X, const State& S, double* zz, cudaStream_t st);
void launch64_eta_z(const Dims& D, const Grid<double>& G, const RotGrid& X, const State& S, double* ez, cudaStream_t st);
void launch64_covariant(const Dims& D, const Grid<double>& G, const State& S, double* cx, double* cy, cudaStream_t st);
void launch64_eta_xy(const Dims& D, const Grid<double>& G, const State& S, const double* cx, const double* cy, double* ex,
                     double* ey, cudaStream_t st);
void launch64_mass_flux(const Dims& D, const Grid<double>& G, const State& S, double* uph, double* vph, double* q5, double* q6,
                        cudaStream_t st);
void launch64_vort_flux(const Dims& D, const Grid<double>& G, const double* ex, const double* ey, const double* ez,
                        const double* uph, const double* vph, const double* q5, const double* q6, double* px, double* py,
                        double* pz, cudaStream_t st);
void launch64_tend_wind(const Dims& D, const State& So, const State& Sn, const Tend<double>& Tn, const Carried<double>& C,
                        int rk_step, cudaStream_t st);
void launch64_recip(const Dims& D, const Grid<double>& G, double* rdx, double* rdy, double* rdz, cudaStream_t st);
void launch64_grad_vert(const Dims& D, const Grid<double>& G, const Recip& R, const double* s, double* gz, double* w5,
                        double* w6, cudaStream_t st);
void launch64_grad_hor(const Dims& D, const Grid<double>& G, const Recip& R, const double* s, const double* w5,
                       const double* w6, double* rx, double* ry, cudaStream_t st);
void launch64_grad_faces(const Dims& D, const Grid<double>& G, const Recip& R, const double* s, const double* w5,
                         const double* w6, const Faces& F, cudaStream_t st);
void launch64_div(const Dims& D, const Grid<double>& G, const Recip& R, const Faces& F, double* out, cudaStream_t st);
void launch64_theta_edges(const Dims& D, const double* th, const double* dv, const double* u, const double* v, double* tvu,
                          double* tvv, cudaStream_t st);
void launch64_gas_faces(const Dims& D, const Grid<double>& G, const State& Ss, const double* u_new, const double* v_new,
                        const double* tvu, const double* tvv, const Faces& M, const Faces& T, cudaStream_t st);
void launch64_gas_theta(const Dims& D, const Grid<double>& G, const Recip& R, const State& Ss, const Faces& M, const Faces& T,
                        const double* cpi, const double* cpw, const double* hd, const double* rad, const double* csh,
                        double* t_rho, double* t_rt, const double* mdt, const double* tdh, const double* ptr,
                        const double* pth, cudaStream_t st);
void launch64_wind_slopes(const Dims& D, const Grid<double>& G, const double* u, const double* v, double* hx, double* hy,
                          cudaStream_t st);
void launch64_contra(const Dims& D, const Grid<double>& G, const double* hx, const double* hy, double* cw, cudaStream_t st);
void launch64_tracers(const Dims& D, const Grid<double>& G, const Recip& R, const State& Ss, const double* u_new,
                      const double* v_new, const double* cw, double* t_rho, int rk_step, const double* mdt, const double* ptr,
                      cudaStream_t st);
void launch64_pgrad_cells(const Dims& D, const Grid<double>& G, const State& S, double* th, double* decel, double* cond,
                          cudaStream_t st);
void launch64_pgrad(const Dims& D, const Grid<double>& G, const State& S, const double* gx, const double* gy, const double* gz,
                    const double* th, const double* decel, const double* cond, const double* tvu, const double* tvv,
                    const double* tpu, const double* tpv, const PGrad<double>& P, int lfirst, cudaStream_t st);

// the diffusion closure; of DiffBuf's flux arrays one field each is used, for the coefficients at the
// faces and interfaces
template <class T>
struct DiffBuf;
struct DiffPar;
void launch64_diff_tke(const Dims& D, const Grid<double>& G, const Recip& R, const State& S, const DiffBuf<double>& B,
                       const double* gx, const double* gy, const double* gz, double mva, cudaStream_t st);
void launch64_diff_coeffs(const Dims& D, const Grid<double>& G, const State& S, const DiffBuf<double>& B, int kind, int vertical,
                          double* ch, double* cv, cudaStream_t st);
void launch64_diff_face_coeffs(const Dims& D, const double* ch, const double* cv, int vertical, const DiffBuf<double>& B,
                               cudaStream_t st);
void launch64_diff_faces(const Dims& D, const Grid<double>& G, const Recip& R, const double* s, const double* w5,
                         const double* w6, const DiffBuf<double>& B, const Faces& F, cudaStream_t st);
void launch64_diff_div(const Dims& D, const Grid<double>& G, const Recip& R, const Faces& F, const DiffBuf<double>& B,
                       const double* gz, int vertical, double* out, cudaStream_t st);
void launch64_diff_visc(const Dims& D, const Grid<double>& G, const State& S, const double* T, const DiffBuf<double>& B,
                        const DiffPar& P, cudaStream_t st);
void launch64_diff_vz(const Dims& D, const Grid<double>& G, const State& S, const DiffBuf<double>& B, cudaStream_t st);
void launch64_mom_diff_h(const Dims& D, const Grid<double>& G, const State& S, const DiffBuf<double>& B, cudaStream_t st);
void launch64_mom_diff_v(const Dims& D, const Grid<double>& G, const State& S, const DiffBuf<double>& B, cudaStream_t st);
void launch64_diss_rate(const Dims& D, const Grid<double>& G, const State& S, const DiffBuf<double>& B, cudaStream_t st);

// the column solves (column_fp64.cu)
// grid-only factors of the column solves: 1/volume at the layers; at w level jl = 2..nl (index of
// layer jl) half of z_scalar(jl-1) - z_scalar(jl) over c_imp1 (= impl_thermo_weight*dtime*c_d_p), 1/area_z;
// 1/c_imp2 (c_imp2 = c_imp1*dtime) and 1/dtime
struct ColumnGrid {
  const F64 *rvol, *zs_c1h, *raz;
  double rc_imp2, rdt;
};
// itwdtv: 0.5*dtime/volume, of moist runs (null: not formed)
void launch_column_grid(const Dims& D, const Grid<double>& G, double* rvol, double* itwdtv, double* zs_c1h, double* raz,
                        cudaStream_t st);
// once per step of a moist run, from state_old and its temperature: the cloud droplets' fall speed
// and c_p of ice and water
void launch_moist_aux(const Dims& D, const Grid<double>& G, const State& So, const double* T, double* vcloud, double* cpi,
                      double* cpw, cudaStream_t st);
int column_prepare();
void launch_column_ver(const Dims& D, const Grid<double>& G, const ColumnGrid& X, const State& So, const State& Sn,
                       const Tend<double>& Tn, int rk_step, cudaStream_t st);
// the tracer solve: rvol = 1/volume, itwdtv = 0.5*dtime/volume; csh is written at rk_step 1, with
// hx as work space
void launch_column_tracers(const Dims& D, const Grid<double>& G, const State& So, const State& Sn, const double* t_rho,
                           const double* T, const double* rvol, const double* itwdtv, const double* vcloud,
                           const double* cpi, const double* cpw, double* csh, double* hx, int rk_step, cudaStream_t st);

}  // namespace lg
