// C entry points to the library's internal launch wrappers, for tests that hold one kernel to its
// reference by itself. Linked against libwbgpu.so.
#include "wb_kernels.h"

using namespace wb;

extern "C" {

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
}
