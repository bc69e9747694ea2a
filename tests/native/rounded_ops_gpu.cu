// Device check of cr_math.cuh: the seeds' errors against the bounds that the
// sequences' analysis takes, and the sequences from those seeds beside the IEEE
// operators, bit for bit (tests/test_rounded_ops_gpu.py).
#include <cuda_runtime.h>

#include <cmath>

#include "cr_math.cuh"

using namespace dgswem;

namespace {

struct Found {
  unsigned long long rcp_seed, rsqrt_seed, log2_start, exp2_start;  // largest errors, as double bits
  unsigned long long rcp_bad, sqrt_bad, quot_bad, pow_bad, pow_left;
};

__device__ void largest(unsigned long long* at, double err) {
  atomicMax(at, (unsigned long long)__double_as_longlong(err));  // errors are not negative
}
__device__ unsigned mix(unsigned long long i) {  // a hash, for low words
  i ^= i >> 33;
  i *= 0xff51afd7ed558ccdull;
  i ^= i >> 33;
  i *= 0xc4ceb9fe1a85ec53ull;
  return (unsigned)(i >> 16);
}
__device__ bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }

__device__ void check_ops(double x, double a, Found* f) {
  const double y = rcp_seed(x), z = rsqrt_seed(x);
  largest(&f->rcp_seed, fabs(fma(-x, y, 1.0)));
  largest(&f->rsqrt_seed, 0.5 * fabs(fma(-(x * z), z, 1.0)));
  if (!mid_range(x)) return;
  const double r = rcp_from(x, y);
  if (!same(r, 1.0 / x)) atomicAdd(&f->rcp_bad, 1ull);
  if (!same(sqrt_from(x, z), sqrt(x))) atomicAdd(&f->sqrt_bad, 1ull);
  if (mid_range(a) && !same(quot_from(a, x, r), a / x)) atomicAdd(&f->quot_bad, 1ull);
}

// every high word of the binades [2^-256, 2^-254) and those scaled into eight
// others, each with low words of all zeros, ones but the last bit, and hashes
__global__ void sweep_high_words(Found* f) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 2u << 20) return;
  for (int k = 0; k < 8; ++k) {
    const unsigned hi = 0x2ff00000u + i + (unsigned)(k * 63) * 0x100000u;
    for (int j = 0; j < 6; ++j) {
      const unsigned h = mix(((unsigned long long)i << 8) | (unsigned)(k * 8 + j));
      const unsigned lo = j == 0 ? 0u : j == 1 ? 0xfffffffeu : h;
      const unsigned ahi = 0x2ff00000u + mix(((unsigned long long)h << 32) | i) % 0x20000000u;
      check_ops(__hiloint2double((int)hi, (int)lo), __hiloint2double((int)ahi, (int)mix(h)), f);
    }
  }
}

__global__ void listed(const double* x, int n, Found* f) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) check_ops(x[i], 1.0, f);
}

// every single-precision number of [2^-30, 2^30], with hashed low bits below it
__global__ void sweep_depths(Found* f) {
  const unsigned m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= 1u << 23) return;
  double el = 0.0, ey = 0.0;
  unsigned long long bad = 0, left = 0;
  for (int e = -30; e < 30; ++e) {
    const unsigned long long low = mix(((unsigned long long)m << 8) | (unsigned)(e + 30)) & 0x1fffffffu;
    const double x =
        __longlong_as_double((long long)(((unsigned long long)(1023 + e) << 52) | ((unsigned long long)m << 29) | low));
    // the start as pow_third_try forms it
    const float l2 = __log2f((float)x);
    float y0;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(l2 * (-1.0f / 3.0f)));
    el = fmax(el, fabs((double)l2 - log2(x)));
    const double y = (double)y0;
    ey = fmax(ey, fabs(fma(-(x * y), y * y, 1.0)) / 3.0);
    double r;
    const bool near = pow_third_try(x, &r);
    const double full = pow_third_any(x);
    left += near ? 0 : 1;
    bad += near && !same(r, full) ? 1 : 0;
  }
  largest(&f->log2_start, el);
  largest(&f->exp2_start, ey);
  if (bad) atomicAdd(&f->pow_bad, bad);
  if (left) atomicAdd(&f->pow_left, left);
}

}  // namespace

// out[0..3]: the seeds' and starts' largest errors; counts[0..4]: mismatches of
// the reciprocal, root, quotient and cube root, and cube roots left to the
// general method.  Returns the CUDA status.
extern "C" int rounded_ops_gpu(const double* hard, int n, double* out, unsigned long long* counts) {
  Found *d = nullptr, h{};
  double* x = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof(Found));
  if (e == cudaSuccess) e = cudaMalloc(&x, (size_t)n * sizeof(double));
  if (e == cudaSuccess) e = cudaMemset(d, 0, sizeof(Found));
  if (e == cudaSuccess) e = cudaMemcpy(x, hard, (size_t)n * sizeof(double), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    sweep_high_words<<<(2u << 20) / 256, 256>>>(d);
    listed<<<(unsigned)((n + 255) / 256), 256>>>(x, n, d);
    sweep_depths<<<(1u << 23) / 256, 256>>>(d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(&h, d, sizeof(Found), cudaMemcpyDeviceToHost);
  cudaFree(x);
  cudaFree(d);
  const unsigned long long errs[4] = {h.rcp_seed, h.rsqrt_seed, h.log2_start, h.exp2_start};
  for (int i = 0; i < 4; ++i) {
    union {
      unsigned long long u;
      double v;
    } c;
    c.u = errs[i];
    out[i] = c.v;
  }
  counts[0] = h.rcp_bad;
  counts[1] = h.sqrt_bad;
  counts[2] = h.quot_bad;
  counts[3] = h.pow_bad;
  counts[4] = h.pow_left;
  return (int)e;
}
