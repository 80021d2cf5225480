// The quotients and roots of harm_exact.cuh over arrays, on the host (with a
// shifted seed) and on the device.  root: 0 a / b, 1 sqrt(a), 2 a / b down to
// subnormal numbers, 3 the same for normal ones, 4 and 5 a / (b b) and
// a / ((b b) b) with reciprocals from that of b.
#include <cuda_runtime.h>

#include "../harm_ramt_b200/csrc/harm_exact.cuh"

using namespace harm;

HD_INLINE void one(int root, double a, double b, int nudge, double* q, unsigned char* ok)
{
  if (root == 2) {
    ExactTiny ex;
    *q = ex.div(a, ex.rcp(b, nudge));
    *ok = ex.ok();
  } else if (root > 2) {
    ExactTiny ex;
    const Recip r1 = ex.rcp(b, nudge), r2 = ex.rcp_from(b * b, r1.y * r1.y), r3 = ex.rcp_from((b * b) * b, r2.y * r1.y);
    *q = ex.div_normal(a, root == 3 ? r1 : (root == 4 ? r2 : r3));
    *ok = ex.ok();
  } else {
    Exact ex;
    *q = root ? ex.sqrt_of(a, nudge) : ex.div(a, ex.rcp(b, nudge));
    *ok = ex.ok();
  }
}

__global__ void k_ops(int root, int n, const double* a, const double* b, double* q, unsigned char* ok)
{
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < n) one(root, a[k], b[k], 0, q + k, ok + k);
}

extern "C" void exact_host(int root, int n, const double* a, const double* b, int nudge, double* q, unsigned char* ok)
{
  for (int k = 0; k < n; k++) one(root, a[k], b[k], nudge, q + k, ok + k);
}

extern "C" int exact_device(int root, int n, const double* a, const double* b, double* q, unsigned char* ok)
{
  double* d = nullptr;
  unsigned char* f = nullptr;
  const size_t m = n * sizeof(double);
  int rc = cudaMalloc(&d, 3 * m) != cudaSuccess || cudaMalloc(&f, n) != cudaSuccess;
  if (!rc) {
    cudaMemcpy(d, a, m, cudaMemcpyHostToDevice);
    cudaMemcpy(d + n, b, m, cudaMemcpyHostToDevice);
    k_ops<<<(n + 255) / 256, 256>>>(root, n, d, d + n, d + 2 * n, f);
    cudaMemcpy(q, d + 2 * n, m, cudaMemcpyDeviceToHost);
    rc = cudaMemcpy(ok, f, n, cudaMemcpyDeviceToHost) != cudaSuccess;
  }
  cudaFree(d);
  cudaFree(f);
  return rc;
}
