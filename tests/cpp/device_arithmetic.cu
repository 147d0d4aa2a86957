// Device arithmetic of common.cuh, entry by entry, for tests/test_division.py
// and tests/test_determinism.py.
#include "../../aprl_b200/csrc/common.cuh"

using namespace aprl_gpu;

namespace {

template <class T>
__global__ void divide_kernel(const T* x, const T* h, T* out, long long n) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = divide_by(x[i], h[i], T(1.) / h[i]);
}

__global__ void fixed_kernel(const double* v, long long n, double scale, int merged,
                             unsigned long long* pairs, int* accepted) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  accepted[i] = merged ? fixed_add<true>(pairs + 2 * i, v[i], scale)
                       : fixed_add(pairs + 2 * i, v[i], scale);
}

template <class T>
struct Device {
  T* p = nullptr;
  explicit Device(long long n) {
    if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess) p = nullptr;
  }
  ~Device() { cudaFree(p); }
};

template <class T>
int divide(const T* x, const T* h, T* out, long long n) {
  Device<T> a(n), b(n), c(n);
  if (!a.p || !b.p || !c.p) return 1;
  cudaMemcpy(a.p, x, n * sizeof(T), cudaMemcpyHostToDevice);
  cudaMemcpy(b.p, h, n * sizeof(T), cudaMemcpyHostToDevice);
  divide_kernel<T><<<(unsigned)((n + 255) / 256), 256>>>(a.p, b.p, c.p, n);
  return cudaMemcpy(out, c.p, n * sizeof(T), cudaMemcpyDeviceToHost) != cudaSuccess;
}

}  // namespace

extern "C" int test_divide64(const double* x, const double* h, double* out, long long n) {
  return divide(x, h, out, n);
}
extern "C" int test_divide32(const float* x, const float* h, float* out, long long n) {
  return divide(x, h, out, n);
}

// Each value added to a pair of its own, which starts at zero.
extern "C" int test_fixed_add(const double* v, long long n, double scale, int merged,
                              unsigned long long* pairs, int* accepted) {
  Device<double> a(n);
  Device<unsigned long long> b(2 * n);
  Device<int> c(n);
  if (!a.p || !b.p || !c.p) return 1;
  cudaMemcpy(a.p, v, n * 8, cudaMemcpyHostToDevice);
  cudaMemset(b.p, 0, 2 * n * 8);
  fixed_kernel<<<(unsigned)((n + 255) / 256), 256>>>(a.p, n, scale, merged, b.p, c.p);
  cudaMemcpy(pairs, b.p, 2 * n * 8, cudaMemcpyDeviceToHost);
  return cudaMemcpy(accepted, c.p, n * 4, cudaMemcpyDeviceToHost) != cudaSuccess;
}
