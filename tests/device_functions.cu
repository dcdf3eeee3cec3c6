// The hand-written device functions of the kernels, over arrays: for
// test_gpu_device_functions.py.
#include <stdint.h>

#include "gbdx_f2.cuh"
#include "gbdx_f64i.cuh"
#include "gbdx_vbt.cuh"

using namespace gbdx;

__global__ void k_tanh2(const float *x, float *y, int pairs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < pairs) f2_unpack(tanh2(x[2 * i], x[2 * i + 1]), y[2 * i], y[2 * i + 1]);
}

__global__ void k_tanh_lib(const float *x, float *y, int pairs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 2 * pairs) y[i] = tanhf(x[i]);
}

// z: four values a pair of (u, v) words
__global__ void k_box(const uint32_t *u, const uint32_t *v, float *z, int pairs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= pairs) return;
  float o[4];
  box_muller2(u[2 * i], v[2 * i], u[2 * i + 1], v[2 * i + 1], o);
  for (int q = 0; q < 4; q++) z[4 * i + q] = o[q];
}

// the same with the CUDA library's functions
__global__ void k_box_lib(const uint32_t *u, const uint32_t *v, float *z, int pairs) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2 * pairs) return;
  const float a = (float(u[i] >> 8) + 0.5f) * 0x1p-24f, b = (float(v[i] >> 8) + 0.5f) * 0x1p-24f;
  const float rad = sqrtf(-2.0f * logf(a));
  float s, c;
  sincospif(2.0f * b, &s, &c);
  z[2 * i] = rad * c;
  z[2 * i + 1] = rad * s;
}

__global__ void k_quotient(const double *a, const double *b, float *q, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) q[i] = f64i_quotient_f32(a[i], b[i]);
}

static int done() { return int(cudaDeviceSynchronize()) | int(cudaGetLastError()); }

extern "C" {
int run_tanh2(const float *x, float *y, int pairs) {
  k_tanh2<<<(pairs + 255) / 256, 256>>>(x, y, pairs);
  return done();
}
int run_tanh_lib(const float *x, float *y, int pairs) {
  k_tanh_lib<<<(2 * pairs + 255) / 256, 256>>>(x, y, pairs);
  return done();
}
int run_box(const uint32_t *u, const uint32_t *v, float *z, int pairs) {
  k_box<<<(pairs + 255) / 256, 256>>>(u, v, z, pairs);
  return done();
}
int run_box_lib(const uint32_t *u, const uint32_t *v, float *z, int pairs) {
  k_box_lib<<<(2 * pairs + 255) / 256, 256>>>(u, v, z, pairs);
  return done();
}
int run_quotient(const double *a, const double *b, float *q, int n) {
  k_quotient<<<(n + 255) / 256, 256>>>(a, b, q, n);
  return done();
}
}
