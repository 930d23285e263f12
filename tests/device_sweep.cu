// ks_column_ver_tile's sweeps (tile_sweep.cuh) on given systems, and the same elimination with every row
// divided in FP64, a thread a column.
#include "tile_sweep.cuh"

namespace {
constexpr int TC = 32;
template <class C>
__global__ void k_sweeps(int n, int cols, const C* d, const C* c, const C* e, const double* rhs, double* tile,
                         double* plain) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x, col = blockIdx.x * TC + lane;
  if (col >= cols) return;
  double* const r = (double*)smem + lane;
  C* const row = (C*)((double*)smem + TC * n) + lane;
  for (int l = 0; l < n; ++l) {
    const int i = l * cols + col;
    row[lg::kTileCoef * TC * l] = d[i];
    row[lg::kTileCoef * TC * l + TC] = c[i];
    row[lg::kTileCoef * TC * l + 2 * TC] = e[i];
    r[TC * l] = rhs[i];
  }
  lg::tile_forward<C, TC>(row, r, n);
  // the same pivots and upper factors, each row's quotient in the chain
  double q = 0.0;
  for (int l = 0; l < n; ++l) {
    const int i = l * cols + col;
    const double cp = l ? (double)c[i - cols] : 0.0, p = (double)row[lg::kTileCoef * TC * l];
    q = (rhs[i] - cp * q) / p;
    plain[i] = q;
    r[TC * l] /= p;
  }
  for (int l = n - 2; l >= 0; --l)
    plain[l * cols + col] -= (double)row[lg::kTileCoef * TC * l + 2 * TC] * plain[(l + 1) * cols + col];
  lg::tile_back<C, TC>(row, r, n);
  for (int l = 0; l < n; ++l) tile[l * cols + col] = r[TC * l];
}

template <class C>
int run(int n, int cols, const C* d, const C* c, const C* e, const double* rhs, double* tile, double* plain) {
  const size_t m = (size_t)n * cols;
  C* a[3];
  double* b[3];
  const C* src[3] = {d, c, e};
  for (int k = 0; k < 3; ++k) {
    if (cudaMalloc(&a[k], m * sizeof(C)) || cudaMemcpy(a[k], src[k], m * sizeof(C), cudaMemcpyHostToDevice)) return 1;
    if (cudaMalloc(&b[k], m * sizeof(double))) return 1;
  }
  if (cudaMemcpy(b[0], rhs, m * sizeof(double), cudaMemcpyHostToDevice)) return 1;
  const size_t sm = (size_t)n * TC * (sizeof(double) + lg::kTileCoef * sizeof(C));
  if (cudaFuncSetAttribute(k_sweeps<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm)) return 2;
  k_sweeps<C><<<(cols + TC - 1) / TC, TC, sm>>>(n, cols, a[0], a[1], a[2], b[0], b[1], b[2]);
  if (cudaGetLastError()) return 3;
  if (cudaMemcpy(tile, b[1], m * sizeof(double), cudaMemcpyDeviceToHost)) return 4;
  if (cudaMemcpy(plain, b[2], m * sizeof(double), cudaMemcpyDeviceToHost)) return 4;
  for (int k = 0; k < 3; ++k) {
    cudaFree(a[k]);
    cudaFree(b[k]);
  }
  return 0;
}
}  // namespace

extern "C" int sweeps_f32(int n, int cols, const float* d, const float* c, const float* e, const double* rhs, double* tile,
                          double* plain) {
  return run(n, cols, d, c, e, rhs, tile, plain);
}
extern "C" int sweeps_f64(int n, int cols, const double* d, const double* c, const double* e, const double* rhs,
                          double* tile, double* plain) {
  return run(n, cols, d, c, e, rhs, tile, plain);
}
