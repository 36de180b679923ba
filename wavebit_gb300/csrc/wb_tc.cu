// Host side of the tensor-core complex products, FP32 (wb_tc.cuh) and FP64 (wb_oz.cuh): the dispatch
// that gemm<float> and gemm<double> try first, and the error counter of timed-out CTAs.
#include "wb_oz.cuh"
#include "wb_tc.cuh"
#include "wb_kernels.h"

namespace wb {

bool tc_cgemm(cudaStream_t s, int batch, int m, int n, int k, double2 alpha, const Cx<float>* A, long long a_rs,
              long long a_cs, long long a_bs, const Cx<float>* B, long long b_rs, long long b_cs, long long b_bs,
              double2 beta, Cx<float>* C, long long c_rs, long long c_cs, long long c_bs) {
  if (tuning(kTuneTensorCores) == 1) return false;          // switched off
  if (batch <= 0 || m < tc::kTileM || n < 64 || k < tc::kKb) return false;   // small: the SIMT kernel
  if (allow_shared(tc::cgemm_kernel, (int)tc::kSmemBytes) !=
      cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  dim3 grid((m + tc::kTileM - 1) / tc::kTileM, (n + tc::kTileN - 1) / tc::kTileN, batch);
  tc::cgemm_kernel<<<grid, tc::kThreads, tc::kSmemBytes, s>>>(
      m, n, k, make_float2((float)alpha.x, (float)alpha.y), make_float2((float)beta.x, (float)beta.y), A, a_rs, a_cs,
      a_bs, B, b_rs, b_cs, b_bs, C, c_rs, c_cs, c_bs);
  note_launch();
  return true;
}

// The exact-slice product serves any strides, real alpha and beta and conjugated operands. Its cost is
// flat (about 17 us a 64 x 64 tile and 64 of K, an FP64 tile of that size 270 us), so only the thinnest
// products stay on the FP64 pipes: a dimension under 8 (the right-hand-side blocks of gemm_narrow_kernel).
bool oz_zgemm(cudaStream_t s, int batch, int m, int n, int k, double2 alpha, const cplx* A, long long a_rs,
              long long a_cs, long long a_bs, const int* a_idx, bool conj_a, const cplx* B, long long b_rs,
              long long b_cs, long long b_bs, bool conj_b, double2 beta, cplx* C, long long c_rs, long long c_cs,
              long long c_bs) {
  if (tuning(kTuneTensorCores) == 1) return false;          // switched off
  if (alpha.y != 0.0 || beta.y != 0.0 || m < 8 || n < 8 || k < 8) return false;
  if (allow_shared(oz::zgemm_kernel, (int)oz::kSmem) !=
      cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  oz::Args g;
  g.m = m; g.n = n; g.k = k; g.alpha = alpha.x; g.beta = beta.x;
  g.A = A; g.B = B; g.C = C;
  g.a_rs = a_rs; g.a_cs = a_cs; g.a_bs = a_bs; g.b_rs = b_rs; g.b_cs = b_cs; g.b_bs = b_bs;
  g.c_rs = c_rs; g.c_cs = c_cs; g.c_bs = c_bs;
  g.a_idx = a_idx; g.conj_a = conj_a; g.conj_b = conj_b;
  dim3 grid((m + oz::kT - 1) / oz::kT, (n + oz::kT - 1) / oz::kT, batch);
  oz::zgemm_kernel<<<grid, oz::kThreads, oz::kSmem, s>>>(g);
  note_launch();
  return true;
}

long long tc_errors() {
  unsigned int v = 0, z = 0;
  if (cudaMemcpyFromSymbol(&v, tc::g_tc_error, sizeof(v)) != cudaSuccess ||
      cudaMemcpyFromSymbol(&z, oz::g_oz_error, sizeof(z)) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return (long long)v + (long long)z;
}

}  // namespace wb
