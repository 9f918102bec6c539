// Kernels that no entry point runs alone, for the tests (conftest.py, kernels).
#include "../../bem_gmsh_gb300/csrc/bem_crmath.cuh"
#include "../../bem_gmsh_gb300/csrc/bem_lu.h"

#include <vector>

// One Gram-Schmidt step, all pointers on the device but host (page-locked, 64
// doubles): bem::gram_schmidt64.
extern "C" int h_gram_schmidt(const double* V, int N, int m, double* w, double* vn, double* host) {
  int *info = nullptr, *hinfo = nullptr;
  int rc = cudaMalloc(&info, 16) || cudaMemset(info, 0, 16) || cudaMallocHost(&hinfo, 16);
  if (!rc) rc = bem::gram_schmidt64(V, N, N, m, w, vn, host, info, hinfo, 0);
  if (cudaDeviceSynchronize() != cudaSuccess) rc = -1;
  cudaFree(info);
  cudaFreeHost(hinfo);
  return rc;
}

// The look-ahead LU of a column-major FP64 matrix: A32 receives L\U, cs the
// column scales; n a multiple of 128.
extern "C" int h_factor(const double* A64, int n, float* A32, double* cs, int variant) {
  using namespace bem;
  const int K = n / LU_NB;
  int lo = 0, hi = 0, rc = 1;
  cudaDeviceGetStreamPriorityRange(&lo, &hi);
  cudaStream_t st[3];
  for (int i = 0; i < 3; ++i) cudaStreamCreateWithPriority(&st[i], cudaStreamNonBlocking, i ? hi : lo);
  std::vector<cudaEvent_t> ev(3 * K + 1);
  for (auto& e : ev) cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
  float* Dinv = nullptr;
  int *info = nullptr, h[2] = {1, 1};
  const size_t op = (size_t)n * LU_NB;
  float* ops = nullptr;
  TcPlan tc[LU_PLANS];
  bool ok = cudaMalloc(&Dinv, sizeof(float) * lu_dinv_floats(K)) == cudaSuccess &&
            cudaMalloc(&info, 256) == cudaSuccess && cudaMemset(info, 0, 256) == cudaSuccess &&
            cudaMalloc(&ops, sizeof(float) * op * 3 * LU_PLANS) == cudaSuccess;
  for (int i = 0; ok && i < LU_PLANS; ++i)
    ok = tc_plan(tc[i], A32, n, n, ops + op * 3 * i, ops + op * (3 * i + 1), ops + op * (3 * i + 2), variant) &&
         tc[i].variant == variant;
  if (ok) {
    cudaDeviceSynchronize();
    lu_prepare(A64, n, n, n, cs, A32, n, st[0]);
    rc = lu_factor_lookahead(A32, n, n, Dinv, info, st[0], st[1], ev[3 * K], ev.data(), ev.data() + K, st[2],
                             ev.data() + 2 * K, tc, info + 1, info + 16);
    if (cudaDeviceSynchronize() != cudaSuccess) rc = 2;
    cudaMemcpy(h, info, sizeof(h), cudaMemcpyDeviceToHost);
  }
  cudaFree(Dinv);
  cudaFree(info);
  cudaFree(ops);
  for (auto& e : ev) cudaEventDestroy(e);
  for (auto& s : st) cudaStreamDestroy(s);
  return rc ? rc : (h[0] || h[1] ? 3 : 0);
}

// The FP64 functions of fast64.cuh and the tangent of bem_crmath.cuh on the
// device, x, y, o device arrays of n: 0 log, 1 x / y, 2 1 / x, 3 sqrt, 4 tan,
// 5 tan in full.
__global__ void k_function(int which, const double* x, const double* y, int n, double* o) {
  using namespace bem;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  switch (which) {
    case 0: o[i] = f64::log(x[i]); break;
    case 1: o[i] = f64::div(x[i], y[i]); break;
    case 2: o[i] = f64::rcp(x[i]); break;
    case 3: o[i] = f64::sqrt(x[i]); break;
    case 4: o[i] = crm::cr_tan(x[i]); break;
    default: o[i] = crm::cr_tan_full(x[i]); break;
  }
}
extern "C" int h_function(int which, const double* x, const double* y, int n, double* o) {
  k_function<<<(n + 255) / 256, 256>>>(which, x, y, n, o);
  const int rc = (int)cudaGetLastError();
  return cudaDeviceSynchronize() != cudaSuccess ? -1 : rc;
}
