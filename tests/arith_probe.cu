// The scalar arithmetic of the kernels (ec2d_dev.cuh, k_turb.cu) over arrays, for
// test_gpu_arith.py: out[k] = op(a[k], b[k]).
#include "k_turb.cu"

namespace ec2d {
// launchers that k_turb.cu refers to (contexts with FP32 parts)
void launch_sa_rows_mixed(const Lvl &, cudaStream_t) {}
void launch_sst_rows_mixed(const Lvl &, cudaStream_t) {}
void launch_fdm_mixed(const Lvl &, cudaStream_t) {}

__device__ double op(int k, double a, double b) {
  switch (k) {
    case 0: return recip(a);
    case 1: return recip_any(a);
    case 2: return rroot(a);
    case 3: return root(a);
    case 4: return root_t(a);
    case 5: return root_ratio(a, b);
    case 6: return quot(a, b, rcp_seed(b));
    case 7: return quot_any(a, b, rcp_seed(b));
    case 8: return div_r(a, b);
    case 9: return sqrt_r(a);
    case 10: return (double)to<float>(a);
    case 11: return to_double((float)a);
    case 12: return pow2<1>(a);
    case 13: return half(a);
    case 14: return pow2<-3>(a);
    case 15: return neg(a);
    case 16: return below(a, b);
    case 17: return at_least(a, b);
    case 18: return above(a, b);
    case 19: return minmod(a, b);
    case 20: return tanh_pos(a);
    case 21: return sixth_root(a, 1.0 / a, b);
    case 22: return pos_part(a);
    case 23: return neg_part(a);
  }
  return 0.0;
}
__global__ void k_op(int k, long long n, const double *a, const double *b, double *out) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = op(k, a[i], b[i]);
}
}  // namespace ec2d

extern "C" int arith(int k, long long n, const double *a, const double *b, double *out) {
  double *d = nullptr;
  if (cudaMalloc(&d, 3 * n * sizeof(double)) != cudaSuccess) return 1;
  cudaMemcpy(d, a, n * sizeof(double), cudaMemcpyHostToDevice);
  cudaMemcpy(d + n, b, n * sizeof(double), cudaMemcpyHostToDevice);
  ec2d::k_op<<<(unsigned)((n + 255) / 256), 256>>>(k, n, d, d + n, d + 2 * n);
  cudaMemcpy(out, d + 2 * n, n * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return cudaGetLastError() != cudaSuccess;
}
