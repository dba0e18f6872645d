// Test-only probe: the flux arithmetic of physics.cuh item by item, so that a
// test can measure its rounding against extended precision.  Built by
// tests/test_gpu_flux_rounding.py; not part of the library.
#include <cuda_runtime.h>

#include "../../include/aerof_gpu.h"

#include "../../aerof_dev_b200/csrc/physics.cuh"

// in: V(5) n(3) Ub(5); out: the far-field flux as the residual forms it, and
// with divisions and roots throughout
__global__ void k_farfield(int n, const double* in, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* q = in + 13 * (size_t)i;
  const aerof::Gas g = aerof::make_gas(1.4);
  aerof::sw_flux(g, q[5], q[6], q[7], q, q + 8, out + 10 * (size_t)i);
  aerof::sw_flux<true>(g, q[5], q[6], q[7], q, q + 8, out + 10 * (size_t)i + 5);
}
// in: Ug(5) Ud(5) n(3) gphi(5); out: cotangents of Ug, Ud, n
__global__ void k_roe_adjoint(int n, const double* in, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* q = in + 18 * (size_t)i;
  double* o = out + 13 * (size_t)i;
  for (int k = 0; k < 13; ++k) o[k] = 0.0;
  aerof::roe_flux_adj(aerof::make_gas(1.4), q[10], q[11], q[12], q, q + 5, q + 13, o, o + 5, o + 10);
}
// in: Vi, ddVij, Vj, ddVji; out: both reconstructed values
__global__ void k_vanalbada(int n, const double* in, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* q = in + 4 * (size_t)i;
  aerof::vanalbada(1.0 / 3.0, q[0], q[1], q[2], q[3], out[2 * (size_t)i], out[2 * (size_t)i + 1]);
}

// in: a, b; out: sqrt b and a / b as corrected products
__global__ void k_products(int n, const double* in, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = in[2 * (size_t)i], b = in[2 * (size_t)i + 1];
  out[2 * (size_t)i] = aerof::sqrt_(b, aerof::rsqrt_(b));
  out[2 * (size_t)i + 1] = aerof::quot_(a, b, aerof::rcp_(b));
}

// what: 0 far-field flux, 1 adjoint of the Roe flux, 2 limiter, 3 products.  Returns 0 or a cudaError_t.
extern "C" int flux_probe(int what, int n, const double* in, double* out) {
  const size_t ni[4] = {13, 18, 4, 2}, no[4] = {10, 13, 2, 2};
  double *di = nullptr, *dout = nullptr;
  cudaError_t e = cudaMalloc(&di, sizeof(double) * ni[what] * n);
  if (e == cudaSuccess) e = cudaMalloc(&dout, sizeof(double) * no[what] * n);
  if (e == cudaSuccess) e = cudaMemcpy(di, in, sizeof(double) * ni[what] * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    const int b = (n + 127) / 128;
    if (what == 0) k_farfield<<<b, 128>>>(n, di, dout);
    else if (what == 1) k_roe_adjoint<<<b, 128>>>(n, di, dout);
    else if (what == 2) k_vanalbada<<<b, 128>>>(n, di, dout);
    else k_products<<<b, 128>>>(n, di, dout);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, dout, sizeof(double) * no[what] * n, cudaMemcpyDeviceToHost);
  cudaFree(di);
  cudaFree(dout);
  return (int)e;
}
