// Device functions that no entry point returns by themselves, one value per
// thread, for tests/test_gpu_device_math.py.
#include "../../pdds_gb300/csrc/k_fast64.cu"
#include "../../pdds_gb300/csrc/pair_sum.cuh"

// sums of n rows of `len` values, two rows per thread
__global__ void k_pair_sum(const float* x, int n, int len, double* out) {
  const int i = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (i + 1 >= n) return;
  const float2 z = make_float2(0.f, 0.f);
  pdds::PairSum p = {z, z, z};
  for (int q = 0; q < len; q++) pdds::pair_add(p, make_float2(x[(size_t)i * len + q], x[(size_t)(i + 1) * len + q]));
  out[i] = pdds::pair_total(p, 0);
  out[i + 1] = pdds::pair_total(p, 1);
}

// the table functions (tab = 1) and the math library's: 0 sin and cos of pi x,
// 1 sin and cos of x, 2 exp; two outputs per argument
__global__ void k_math(const double* x, int n, int fn, int tab, pdds::Fast64 T, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0, c = 0.0;
  if (fn == 0) {
    if (tab) pdds::f64::sincospi(T, x[i], s, c);
    else ::sincospi(x[i], &s, &c);
  } else if (fn == 1) {
    if (tab) pdds::f64::sincos(T, x[i], s, c);
    else ::sincos(x[i], &s, &c);
  } else {
    s = tab ? pdds::f64::exp(T, x[i]) : ::exp(x[i]);
  }
  out[2 * i] = s;
  out[2 * i + 1] = c;
}

namespace {

template <typename T, typename F>
int on_device(const T* x, size_t n_x, double* out, size_t n_out, F launch) {
  T* dx = nullptr;
  double* d = nullptr;
  cudaError_t e = cudaMalloc(&dx, n_x * sizeof(T));
  if (e == cudaSuccess) e = cudaMalloc(&d, n_out * sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, n_x * sizeof(T), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    launch(dx, d);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d, n_out * sizeof(double), cudaMemcpyDeviceToHost);
  if (dx) cudaFree(dx);
  if (d) cudaFree(d);
  return (int)e;
}

}  // namespace

extern "C" int check_pair_sum(const float* x, int n, int len, double* out) {  // n even
  return on_device(x, (size_t)n * len, out, n, [&](const float* dx, double* d) {
    k_pair_sum<<<(n / 2 + 127) / 128, 128>>>(dx, n, len, d);
  });
}

extern "C" int check_math(const double* x, int n, int fn, int tab, double* out) {
  void* block = nullptr;
  cudaError_t e = cudaMalloc(&block, pdds::fast64_bytes());
  if (e == cudaSuccess) e = pdds::launch_fast64_tables(block, 0);
  int st = (int)e;
  if (st == 0)
    st = on_device(x, (size_t)n, out, (size_t)2 * n, [&](const double* dx, double* d) {
      k_math<<<(n + 127) / 128, 128>>>(dx, n, fn, tab, pdds::fast64_view(block), d);
    });
  if (block) cudaFree(block);
  return st;
}
