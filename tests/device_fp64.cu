// the arithmetic of fp64.cuh on given arrays, beside CUDA's own operations
#include "fp64.cuh"

namespace {
using lg::F64;
enum Op { kMul, kMulF, kDiv, kRcp, kDivStored, kDivTwo, kHalf, kQuarter, kNegative, kNonzero, kUpwind, kPositive, kOps };
// one operation on (a, b, c): fp64.cuh's in r, the plain one in s
__global__ void k_op(int op, long long n, const double* a, const double* b, const double* c, double* r, double* s) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = a[i], y = b[i], z = c[i];
  double p = 0.0, q = 0.0;
  switch (op) {
    case kMul: p = lg::mul_int(x, y); q = x * y; break;
    case kMulF: p = lg::mul_int((float)x, y); q = (double)(float)x * y; break;
    case kDiv: p = (F64(x) / F64(y)).v; q = x / y; break;
    case kRcp: p = lg::rcp(y); q = 1.0 / y; break;
    case kDivStored: p = lg::div_rn(F64(x), F64(y), F64(1.0 / y)).v; q = x / y; break;
    // a rounded product of two divisors, and the product of a stored reciprocal and a formed one
    case kDivTwo: p = lg::div_rn(F64(x), F64(y) * F64(z), F64(1.0 / y) * lg::rcp_near(F64(z))).v; q = x / (y * z); break;
    case kHalf: p = lg::half(x); q = 0.5 * x; break;
    case kQuarter: p = lg::quarter(x); q = 0.25 * x; break;
    case kNegative: p = lg::negative(x); q = x < 0.0; break;
    case kNonzero: p = lg::nonzero(x); q = x != 0.0; break;
    case kUpwind: p = lg::upwind(x); q = x >= 0.0; break;
    case kPositive: p = lg::positive(x); q = x > 0.0; break;
  }
  r[i] = p;
  s[i] = q;
}
}  // namespace

extern "C" int fp64_op(int op, long long n, const double* a, const double* b, const double* c, double* r, double* s) {
  double* d[5];
  const double* src[3] = {a, b, c};
  if (op < 0 || op >= kOps || n < 1) return 9;
  for (double*& p : d)
    if (cudaMalloc(&p, n * sizeof(double))) return 1;
  for (int k = 0; k < 3; ++k)
    if (cudaMemcpy(d[k], src[k], n * sizeof(double), cudaMemcpyHostToDevice)) return 2;
  k_op<<<(unsigned)((n + 255) / 256), 256>>>(op, n, d[0], d[1], d[2], d[3], d[4]);
  if (cudaGetLastError() || cudaMemcpy(r, d[3], n * sizeof(double), cudaMemcpyDeviceToHost) ||
      cudaMemcpy(s, d[4], n * sizeof(double), cudaMemcpyDeviceToHost))
    return 3;
  for (double* p : d) cudaFree(p);
  return 0;
}
