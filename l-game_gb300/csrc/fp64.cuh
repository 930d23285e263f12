// fp64.cuh -- FP64 arithmetic of the FP64 step in fewer operations of the FP64 pipe, which issues
// 1.7 operations per clock and SM on this GPU against 64 integer ones: with every kernel of the
// step at 80-88 % of that pipe and below 10 % of everything else, its time is the number of these
// operations.  Every function returns the bits of the plain expression (exceptions as stated).
#pragma once

#include "kernels.cuh"

namespace lg {

// a/b rounded to nearest for y within two units of the last place of 1/b: quotient, remainder,
// correction (Markstein, IBM J. Res. Dev. 34, 1990): three FP64-pipe operations instead of about
// seven.  The result is the correctly rounded quotient, except that a quotient within 2^-50 of its
// last place from the middle of two doubles may round the other way; a zero quotient's sign is not
// kept, and an infinite a gives NaN.
__device__ __forceinline__ double div_rn(double a, double b, double y) {
  const double q = a * y;
  return fma(fma(-b, q, a), y, q);
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

// reciprocals of the metrics at their own points, formed once with the grid
struct Recip {
  const double *vol, *dx, *dy, *dz;
};
// what a face hands to the divergences of its two cells: flux times area and the slope term
// 0.5*f*slope, x at u points, y at v points
struct Faces {
  double *px, *py, *hx, *hy;
};

// the explicit kernels (kernels_fp64.cu)
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

}  // namespace lg
