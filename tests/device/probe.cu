// The library's scalar device functions over arrays, for
// tests/device_probe.py: one thread per element (or sum), bounds checked.
// Compiled by the test from the library's own headers.
#include "../../hbtplus_gb300/csrc/loop_ops.cuh"
#include "../../hbtplus_gb300/csrc/tree_ops.cuh"
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

__global__ void k_over_scale(const double *x, int n, DevParams P, double *got, double *want)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  got[i] = over_scale(x[i], P);
  want[i] = __ddiv_rn(x[i], P.ad);
}

__global__ void k_fp64_contrib(const double *r2, const float *m, int n, DevParams P, double *got,
                               double *want)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  got[i] = fp64_contrib(r2[i], m[i], P);
  want[i] = fp64_contrib_any(r2[i], (double)m[i], P.h, P.h_inv);
}

__global__ void k_quot_float(const double *c, const double *m, int n, float *got, float *want)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  bool ok;
  const double r = recip_refined(m[i], ok);
  got[i] = quot_float(c[i], m[i], r, ok);
  want[i] = __double2float_rn(__ddiv_rn(c[i], m[i]));
}

// fold_chunks as launch_fold launches it, and the loop of additions.
__global__ void __launch_bounds__(128) k_fold(Ctx c, int K)
{
  fold_chunks(c, K, (blockIdx.x * 128 + threadIdx.x) >> 5, threadIdx.x & 31);
}

__global__ void k_loop(Ctx c, int K, double *out)
{
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= c.nlong * K) return;
  const int s = c.seg_order[w / K];
  double t = 0.;
  for (int b = c.bchunk_base[s]; b < c.bchunk_base[s + 1]; b++)
    t = __dadd_rn(t, c.chunk_sums[(size_t)b * kSums + w % K]);
  out[w] = t;
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

DevParams scale_params(float a)
{
  DevParams P = {};
  P.a = a;
  P.ad = (double)a;
  P.a_inv = 1.0 / (double)a;
  return P;
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

int probe_over_scale(const double *x, int n, float a, double *got, double *want)
{
  const DevParams P = scale_params(a);
  return run(x, (const float *)nullptr, n, got, want,
             [&](int nb, double *dx, float *, double *g, double *w) {
               k_over_scale<<<nb, 128>>>(dx, n, P, g, w);
             });
}

int probe_fp64_contrib(const double *r2, const float *m, int n, double h, double *got, double *want)
{
  const DevParams P = softening_params(h);
  return run(r2, m, n, got, want, [&](int nb, double *dx, float *dm, double *g, double *w) {
    k_fp64_contrib<<<nb, 128>>>(dx, dm, n, P, g, w);
  });
}

int probe_quot_float(const double *c, const double *m, int n, float *got, float *want)
{
  return run(c, m, n, got, want, [&](int nb, double *dc, double *dm, float *g, float *w) {
    k_quot_float<<<nb, 128>>>(dc, dm, n, g, w);
  });
}

// sums: kSums per chunk, changed by the fold; base: nsub + 1 first chunks; order: the
// subhaloes whose sums are made, nlong of them; loop: nlong * K
int probe_fold(double *sums, const int *base, const int *order, int nsub, int nlong, int K,
               double *loop)
{
  const int nchunks = base[nsub];
  if (nlong <= 0 || nlong > nsub || K <= 0 || K > kSums || nchunks <= 0) return -1;
  Ctx c = {};
  double *out = nullptr;
  const size_t bytes = sizeof(double) * kSums * nchunks;
  cudaError_t e = cudaMalloc(&c.chunk_sums, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&c.bchunk_base, sizeof(int) * (nsub + 1));
  if (e == cudaSuccess) e = cudaMalloc(&c.seg_order, sizeof(int) * nlong);
  if (e == cudaSuccess) e = cudaMalloc(&out, sizeof(double) * nlong * K);
  if (e == cudaSuccess) e = cudaMemcpy(c.chunk_sums, sums, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(c.bchunk_base, base, sizeof(int) * (nsub + 1), cudaMemcpyHostToDevice);
  if (e == cudaSuccess)
    e = cudaMemcpy(c.seg_order, order, sizeof(int) * nlong, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    c.S = nsub;
    c.nlong = nlong;
    k_loop<<<(nlong * K + 127) / 128, 128>>>(c, K, out);
    k_fold<<<(32 * nlong * K + 127) / 128, 128>>>(c, K);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(sums, c.chunk_sums, bytes, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(loop, out, sizeof(double) * nlong * K, cudaMemcpyDeviceToHost);
  cudaFree(c.chunk_sums);
  cudaFree(c.bchunk_base);
  cudaFree(c.seg_order);
  cudaFree(out);
  return (int)e;
}

}  // extern "C"
