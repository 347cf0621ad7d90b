// The library's scalar device functions over arrays, for
// tests/device_probe.py: one thread per element, bounds checked.
// Compiled by the test from the library's own headers.
#include "../../hbtplus_gb300/csrc/walk_ops.cuh"

using namespace hbtu;

namespace {

__global__ void k_f2d(const float *x, int n, double *got, double *want)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  got[i] = f2d(x[i]);
  want[i] = (double)x[i];
}

__global__ void k_d2f(const double *x, int n, float *got, float *want)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  got[i] = d2f(x[i]);
  want[i] = __double2float_rn(x[i]);
}

__global__ void k_fp64_contrib(const double *r2, const float *m, int n, DevParams P, double *got,
                               double *want)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  got[i] = fp64_contrib(r2[i], m[i], P);
  want[i] = fp64_contrib_any(r2[i], (double)m[i], P.h, P.h_inv);
}

// x (n elements) to the device, f(device pointer) and the two outputs back.
template <typename In, typename In2, typename Out, typename F>
int run(const In *x, const In2 *x2, int n, Out *got, Out *want, F launch)
{
  if (n <= 0) return 0;
  In *dx = nullptr;
  In2 *dx2 = nullptr;
  Out *dg = nullptr, *dw = nullptr;
  cudaError_t e = cudaMalloc(&dx, sizeof(In) * n);
  if (e == cudaSuccess) e = cudaMalloc(&dx2, sizeof(In2) * n);
  if (e == cudaSuccess) e = cudaMalloc(&dg, sizeof(Out) * n);
  if (e == cudaSuccess) e = cudaMalloc(&dw, sizeof(Out) * n);
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, sizeof(In) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && x2) e = cudaMemcpy(dx2, x2, sizeof(In2) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    launch((n + 127) / 128, dx, dx2, dg, dw);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(got, dg, sizeof(Out) * n, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(want, dw, sizeof(Out) * n, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dx2);
  cudaFree(dg);
  cudaFree(dw);
  return (int)e;
}

DevParams softening_params(double h)
{
  DevParams P = {};
  P.h = h;
  P.h_inv = 1.0 / h;
  return P;
}

}  // namespace

extern "C" {

int probe_f2d(const float *x, int n, double *got, double *want)
{
  return run(x, (const float *)nullptr, n, got, want,
             [&](int nb, float *dx, float *, double *g, double *w) {
               k_f2d<<<nb, 128>>>(dx, n, g, w);
             });
}

int probe_d2f(const double *x, int n, float *got, float *want)
{
  return run(x, (const float *)nullptr, n, got, want,
             [&](int nb, double *dx, float *, float *g, float *w) {
               k_d2f<<<nb, 128>>>(dx, n, g, w);
             });
}

int probe_fp64_contrib(const double *r2, const float *m, int n, double h, double *got, double *want)
{
  const DevParams P = softening_params(h);
  return run(r2, m, n, got, want, [&](int nb, double *dx, float *dm, double *g, double *w) {
    k_fp64_contrib<<<nb, 128>>>(dx, dm, n, P, g, w);
  });
}

}  // extern "C"
