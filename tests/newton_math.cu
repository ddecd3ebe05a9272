// The branch-free operators of the face states (NewtonMath) and CUDA's own, on
// arrays of operands; built and called by test_gpu_newton_math.py.
#include "../raishinsource_b200/csrc/rg_device.cuh"

__global__ void k_newton(const double* a, const double* b, int n, double* out, int* ok) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  rg::NewtonMath r, d, s;
  out[i] = r.rcp(b[i]);
  out[n + i] = d.div(a[i], b[i]);
  out[2 * n + i] = s.sqrt(b[i]);
  out[3 * n + i] = 1.0 / b[i];
  out[4 * n + i] = a[i] / b[i];
  out[5 * n + i] = sqrt(b[i]);
  ok[i] = (r.ok() ? 1 : 0) | (d.ok() ? 2 : 0) | (s.ok() ? 4 : 0);
}

// a, b: n host doubles; out: 6 n doubles, ok: n ints (host).  Returns a cudaError_t.
extern "C" int newton_math(const double* a, const double* b, int n, double* out, int* ok) {
  double* d = nullptr;
  int* f = nullptr;
  const size_t m = (size_t)n * sizeof(double);
  cudaError_t e = cudaMalloc(&d, 8 * m);
  if (e == cudaSuccess) e = cudaMalloc(&f, (size_t)n * sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpy(d, a, m, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(d + n, b, m, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    k_newton<<<(n + 255) / 256, 256>>>(d, d + n, n, d + 2 * (size_t)n, f);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(out, d + 2 * (size_t)n, 6 * m, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(ok, f, (size_t)n * sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(d);
  cudaFree(f);
  return (int)e;
}
