// C entry points to the library's internal launch wrappers, for tests that hold one kernel to its
// reference by itself. Linked against libwbgpu.so.
#include "wb_kernels.h"

using namespace wb;

namespace {
__global__ void rsqrt_kernel(int n, const double* v, double* start, double* full, double* cuda) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  start[i] = rsqrt_start(v[i]);
  full[i] = rsqrt64(v[i]);
  cuda[i] = rsqrt(v[i]);
}
}  // namespace

extern "C" {

int ops_rsqrt(int n, const double* v, double* start, double* full, double* cuda) {
  rsqrt_kernel<<<(n + 255) / 256, 256>>>(n, v, start, full, cuda);
  return (int)cudaGetLastError();
}

int ops_getrf(int is_double, int batch, int n, void* A, long long a_bs, int* piv, int* status) {
  if (is_double) getrf<double>(0, batch, n, (Cx<double>*)A, n, a_bs, piv, n, status, 1);
  else getrf<float>(0, batch, n, (Cx<float>*)A, n, a_bs, piv, n, status, 1);
  return (int)cudaGetLastError();
}

int ops_getrs(int is_double, int batch, int n, const void* LU, long long a_bs, const int* piv, void* B, int nrhs,
              int trans) {
  const long long b_bs = (long long)n * nrhs;
  if (is_double) getrs<double>(0, batch, n, (const Cx<double>*)LU, n, a_bs, piv, n, (Cx<double>*)B, nrhs, n, b_bs, trans);
  else getrs<float>(0, batch, n, (const Cx<float>*)LU, n, a_bs, piv, n, (Cx<float>*)B, nrhs, n, b_bs, trans);
  return (int)cudaGetLastError();
}

// Schur form: A (n x n, by columns) becomes T, Z its vectors, w its eigenvalues
int ops_schur(int batch, int n, void* A, void* Z, void* w, void* tau, int* status) {
  geev_schur<double>(0, batch, n, (Cx<double>*)A, n, (long long)n * n, (Cx<double>*)Z, n, (long long)n * n,
                     (Cx<double>*)w, (Cx<double>*)tau, status, 1);
  return (int)cudaGetLastError();
}

// C = (ar + i ai) op(A) op(B) + (br + i bi) C; strides in elements (rows, columns, batch). idx: A's batch index
int ops_zgemm(int batch, int m, int n, int k, double ar, double ai, const void* A, const long long* as, const int* idx,
              int conj_a, const void* B, const long long* bs, int conj_b, double br, double bi, void* C,
              const long long* cs) {
  const double2 alpha = make_double2(ar, ai), beta = make_double2(br, bi);
  if (idx)
    gemm_idx<double>(0, batch, m, n, k, alpha, (const Cx<double>*)A, as[0], as[1], as[2], idx, (const Cx<double>*)B,
                     bs[0], bs[1], bs[2], beta, (Cx<double>*)C, cs[0], cs[1], cs[2]);
  else
    zgemm_conj(0, batch, m, n, k, alpha, (const cplx*)A, as[0], as[1], as[2], conj_a, (const cplx*)B, bs[0], bs[1],
               bs[2], conj_b, beta, (cplx*)C, cs[0], cs[1], cs[2]);
  return (int)cudaGetLastError();
}
}
