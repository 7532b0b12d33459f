// The pivot search and reciprocal of the direct solver on given values, a warp each.
#include "mic_pivot.cuh"

static __global__ void k_best(const double *a, int *lane) {
  const int w = blockIdx.x, l = threadIdx.x;
  const int best = mic::warp_best(mic::pivot_key(a[32 * w + l]));
  if (l == 0) lane[w] = best;
}
static __global__ void k_rcp(const double *p, double *r, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) r[i] = mic::pivot_rcp(p[i]);
}

// host arrays: best[warps] of a[32 warps]; r[n] of p[n]
extern "C" int pivot_probe(const double *a, int warps, int *best, const double *p, int n, double *r) {
  double *da = nullptr, *dp = nullptr, *dr = nullptr;
  int *db = nullptr;
  bool ok = cudaMalloc(&da, sizeof(double) * 32 * warps) == cudaSuccess &&
            cudaMalloc(&db, sizeof(int) * warps) == cudaSuccess && cudaMalloc(&dp, sizeof(double) * n) == cudaSuccess &&
            cudaMalloc(&dr, sizeof(double) * n) == cudaSuccess &&
            cudaMemcpy(da, a, sizeof(double) * 32 * warps, cudaMemcpyHostToDevice) == cudaSuccess &&
            cudaMemcpy(dp, p, sizeof(double) * n, cudaMemcpyHostToDevice) == cudaSuccess;
  if (ok) {
    k_best<<<warps, 32>>>(da, db);
    k_rcp<<<(n + 255) / 256, 256>>>(dp, dr, n);
    ok = cudaMemcpy(best, db, sizeof(int) * warps, cudaMemcpyDeviceToHost) == cudaSuccess &&
         cudaMemcpy(r, dr, sizeof(double) * n, cudaMemcpyDeviceToHost) == cudaSuccess;
  }
  cudaFree(da);
  cudaFree(db);
  cudaFree(dp);
  cudaFree(dr);
  return ok ? 0 : 1;
}
