// Batched complex non-Hermitian eigen-decomposition, templated over the
// real type R in {double, float, df64} (wb_num.cuh).
//
// The layer operator Omega^2 of every (solve, layer) pair is decomposed as
//   Omega^2 = Z T Z^H  (Hessenberg reduction, then Francis single-shift QR to Schur form)
//   Omega^2 W = W diag(w),  W = Z X  (X: eigenvectors of the triangular T by back-substitution)
// which is the factorisation LAPACK's zgeev performs for numpy.linalg.eig (right vectors only).
//
// GB300 note: FP64 runs at ~1 TFLOP/s, about 2 FP64 FMAs per clock per SM, and an FP64 instruction
// holds a scheduler for 64 cycles whatever its active lanes: FP64 work is spread over lanes, warps and
// the CTAs of a cluster (wb_hrd.cuh, wb_qr.cuh), whose sums keep one order whatever their number. The
// df64 instantiation runs the same algorithm on the FP32 pipes, one CTA a matrix in the reduction.
//
// Every iteration is capped; a matrix that hits the cap gets WB_ST_NOCONV in its status word
// and NaN eigenvalues, and the kernel returns normally.
#include <mutex>
#include <type_traits>
#include <utility>
#include <vector>
#include "wb_common.cuh"
#include "wb_num.cuh"
#include "wb_kernels.h"
#include "wb_qr.cuh"

namespace wb {


__device__ __forceinline__ double shfl_xor(double v, int off) { return __shfl_xor_sync(0xffffffffu, v, off); }
__device__ __forceinline__ float shfl_xor(float v, int off) { return __shfl_xor_sync(0xffffffffu, v, off); }
__device__ __forceinline__ df64 shfl_xor(df64 v, int off) {
  return df64(__shfl_xor_sync(0xffffffffu, v.hi, off), __shfl_xor_sync(0xffffffffu, v.lo, off));
}
__device__ __forceinline__ double shfl_idx(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ float shfl_idx(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ df64 shfl_idx(df64 v, int src) {
  return df64(__shfl_sync(0xffffffffu, v.hi, src), __shfl_sync(0xffffffffu, v.lo, src));
}
template <class R> __device__ __forceinline__ R warp_sum(R v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = v + shfl_xor(v, off);
  return v;
}

template <class R> __device__ R block_sum(R v, R* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    R s = R(0.0);
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s = s + red[w];
    red[0] = s;
  }
  __syncthreads();
  R r = red[0];
  __syncthreads();
  return r;
}

__device__ int block_max_int(int v, int* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = max(v, __shfl_down_sync(0xffffffffu, v, off));
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = red[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) s = max(s, red[w]);
    red[0] = s;
  }
  __syncthreads();
  int r = red[0];
  __syncthreads();
  return r;
}

// Householder reflector for (alpha, x): returns beta (real), tau and the scale of x so that
// (I - tau v v^H)^H (alpha; x) = (beta; 0), v = (1; x * scale).
template <class R> struct Refl { R beta; Cx<R> tau; Cx<R> scale; bool identity; };
template <class R> __device__ __forceinline__ Refl<R> make_reflector(Cx<R> alpha, R xnorm) {
  Refl<R> r;
  if (xnorm == R(0.0) && alpha.y == R(0.0)) {
    r.identity = true; r.beta = alpha.x; r.tau = cxzero<R>(); r.scale = cxzero<R>();
    return r;
  }
  R ax = rabs(alpha.x), ay = rabs(alpha.y);
  R m = rmax(rmax(ax, ay), xnorm);
  R u = ax / m, v = ay / m, w = xnorm / m;
  R nrm = m * rsqrt_(u * u + v * v + w * w);
  R beta = (alpha.x >= R(0.0)) ? -nrm : nrm;
  r.identity = false;
  r.beta = beta;
  r.tau = cxmk<R>((beta - alpha.x) / beta, -alpha.y / beta);
  r.scale = cxinv(cxmk<R>(alpha.x - beta, alpha.y));
  return r;
}

}  // namespace wb
#include "wb_hrd.cuh"
namespace wb {
// ------------------------------------------------------------- 1. Hessenberg reduction
// H := Q^H A Q, reflectors stored below the subdiagonal (v_0 = 1 implicit), tau[k].
//
// Both sides of reflector k are applied in one pass over the trailing columns. With y = A v
// (all rows) and c = v^H y, the right update A' = A - t y v^H and the left update
// A'' = A' - conj(t) v (v^H A') combine, column by column, into
//   A''[:, j] = A[:, j] - t y conj(v_j) - conj(t) v z_j,   z_j = v^H A[:, j] - t c conj(v_j),
// so each step reads the trailing matrix twice (y, then each column's z_j and its update) and
// writes it once. Every load-modify-store sweep issues kUnroll loads before its stores, so one
// memory latency serves kUnroll elements per lane.
constexpr int kUnroll = 4;

template <class R>
__device__ __forceinline__ Cx<R> block_sum_cx(Cx<R> v, R* red) {
  Cx<R> r;
  r.x = block_sum(v.x, red);
  r.y = block_sum(v.y, red);
  return r;
}

// sum_i conj(v_i) c_i over i < m by one warp, the total in every lane. The FP32 form issues four
// loads per lane before it accumulates (four partial sums), the other forms one.
template <class R>
__device__ __forceinline__ Cx<R> column_dot(const Cx<R>* v, const Cx<R>* c, int m, int lane) {
  Cx<R> acc = cxzero<R>();
  int i = lane;
  if constexpr (sizeof(R) == 4) {
    Cx<R> acc1 = cxzero<R>(), acc2 = cxzero<R>(), acc3 = cxzero<R>();
    for (; i + 96 < m; i += 128) {
      const Cx<R> c0 = c[i], c1 = c[i + 32], c2 = c[i + 64], c3 = c[i + 96];
      acc = cxfma_conj(v[i], c0, acc);
      acc1 = cxfma_conj(v[i + 32], c1, acc1);
      acc2 = cxfma_conj(v[i + 64], c2, acc2);
      acc3 = cxfma_conj(v[i + 96], c3, acc3);
    }
    acc = (acc + acc2) + (acc1 + acc3);
  }
  for (; i < m; i += 32) acc = cxfma_conj(v[i], c[i], acc);
  acc.x = warp_sum(acc.x);
  acc.y = warp_sum(acc.y);
  return acc;
}

template <class R>
__global__ void __launch_bounds__(1024) gehrd_kernel(Cx<R>* __restrict__ Aall, int n, int lda,
                                                     long long a_bs, Cx<R>* __restrict__ tau_all,
                                                     const int* __restrict__ live) {
  using C_ = Cx<R>;
  if (live && (int)blockIdx.x >= *live) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  C_* sv = reinterpret_cast<C_*>(smraw);          // v (n), then y = A v (n)
  __shared__ R red[32];
  __shared__ C_ s_tau;
  C_* A = Aall + blockIdx.x * a_bs;
  C_* tau = tau_all + (long long)blockIdx.x * n;
  C_* sy = sv + n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  for (int k = 0; k + 2 < n; ++k) {
    const int m = n - k - 1;
    C_* col = A + (long long)k * lda;
    R part = R(0.0);
    for (int i = k + 2 + tid; i < n; i += blockDim.x) part = part + cxabs2(col[i]);
    R xn2 = block_sum(part, red);
    C_ alpha = col[k + 1];
    Refl<R> r = make_reflector(alpha, rsqrt_(xn2));
    if (r.identity) {
      if (tid == 0) tau[k] = cxzero<R>();
      __syncthreads();
      continue;
    }
    for (int i = k + 2 + tid; i < n; i += blockDim.x) {
      C_ v = col[i] * r.scale;
      col[i] = v;
      sv[i - k - 1] = v;
    }
    if (tid == 0) {
      sv[0] = cxone<R>();
      tau[k] = r.tau;
      s_tau = r.tau;
    }
    __syncthreads();
    // every thread has read alpha = A(k+1, k) by now; column k is not touched again in this step
    if (tid == 0) col[k + 1] = cxmk<R>(r.beta, R(0.0));
    const C_ t = s_tau, tc = cxconj(t);
    // y = A[:, k+1:n] v, one row per thread (loads only: they pipeline). The FP32 form keeps four
    // loads in flight per thread (its registers allow it; the FP64-sized forms are at the limit).
    for (int i = tid; i < n; i += blockDim.x) {
      const C_* ai = A + i + (long long)(k + 1) * lda;
      C_ acc0 = cxzero<R>(), acc1 = cxzero<R>();
      int j = 0;
      if constexpr (sizeof(R) == 4) {
        C_ acc2 = cxzero<R>(), acc3 = cxzero<R>();
        for (; j + 3 < m; j += 4) {
          const C_ a0 = ai[(long long)j * lda], a1 = ai[(long long)(j + 1) * lda];
          const C_ a2 = ai[(long long)(j + 2) * lda], a3 = ai[(long long)(j + 3) * lda];
          acc0 = cxfma(a0, sv[j], acc0);
          acc1 = cxfma(a1, sv[j + 1], acc1);
          acc2 = cxfma(a2, sv[j + 2], acc2);
          acc3 = cxfma(a3, sv[j + 3], acc3);
        }
        acc0 = acc0 + acc2;
        acc1 = acc1 + acc3;
      }
      for (; j + 1 < m; j += 2) {
        acc0 = cxfma(ai[(long long)j * lda], sv[j], acc0);
        acc1 = cxfma(ai[(long long)(j + 1) * lda], sv[j + 1], acc1);
      }
      if (j < m) acc0 = cxfma(ai[(long long)j * lda], sv[j], acc0);
      sy[i] = acc0 + acc1;
    }
    __syncthreads();
    C_ cp = cxzero<R>();
    for (int i = tid; i < m; i += blockDim.x) cp = cxfma_conj(sv[i], sy[k + 1 + i], cp);
    const C_ c = block_sum_cx(cp, red);
    const C_ tcoef = t * c;
    // both sides, one warp per trailing column
    for (int jj = warp; jj < m; jj += nw) {
      C_* cj = A + (long long)(k + 1 + jj) * lda;
      const C_ acc = column_dot<R>(sv, cj + k + 1, m, lane);
      const C_ vjc = cxconj(sv[jj]);
      const C_ z = acc - tcoef * vjc;
      const C_ a1 = t * vjc, a2 = tc * z;
      for (int i0 = lane; i0 < n; i0 += 32 * kUnroll) {
        C_ val[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          const int i = i0 + 32 * u;
          if (i < n) val[u] = cj[i];
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
          const int i = i0 + 32 * u;
          if (i >= n) continue;
          C_ nv = val[u] - sy[i] * a1;
          if (i > k) nv = nv - sv[i - k - 1] * a2;
          cj[i] = nv;
        }
      }
    }
    __syncthreads();
  }
}

// --------------------------------------- 1b. blocked Hessenberg reduction (FP32 form)
// The same reflectors and storage as gehrd_kernel, kHrdPanel columns at a time in WY form. With
// the panel's reflectors so far Q_j = I - V_j T_j V_j^H and Y_j = A V_j T_j (A as at the panel's
// start), column c = k + j of Q_j^H A Q_j is
//   b = a_c - Y_j V_j(c, :)^H,   then   b <- b - V_j T_j^H (V_j^H b)   (rows below k),
// its reflector (tau_j, v_j) extends T (T[:j, j] = -tau_j T_j V_j^H v_j, T[j, j] = tau_j) and Y
// (Y[:, j] = tau_j (A v_j - Y_j V_j^H v_j)); a_c and A v_j read columns the panel has not yet
// written, so the panel makes one pass over the trailing columns per column. After the panel,
// A <- Q^H (A - Y V^H) on the columns right of it, as batched products (geev_schur). Scratch per
// matrix (column-major, ld n): V, conj(V), Y (n x kHrdPanel), W, X (kHrdPanel x n), T^H.
constexpr int kHrdPanel = 32;

// A row times v by four lanes, one a partial sum (q % 4), UN loads in flight: (s0 + s2) + (s1 + s3) in each
// of the four. The tail past the last multiple of four belongs to the first.
template <int UN>
__device__ __forceinline__ Cx<float> row_times(const Cx<float>* ar, int lda, const Cx<float>* vv, int m) {
  using C_ = Cx<float>;
  const int m4 = m & ~3, s4 = threadIdx.x & 3;
  C_ acc = cxzero<float>();
  int q = s4;
  for (; q + 4 * (UN - 1) < m4; q += 4 * UN) {
    C_ a[UN];
#pragma unroll
    for (int u = 0; u < UN; ++u) a[u] = ar[(long long)(q + 4 * u) * lda];
#pragma unroll
    for (int u = 0; u < UN; ++u) acc = cxfma(a[u], vv[q + 4 * u], acc);
  }
  for (; q < m4; q += 4) acc = cxfma(ar[(long long)q * lda], vv[q], acc);
  if (s4 == 0)
    for (q = m4; q < m; ++q) acc = cxfma(ar[(long long)q * lda], vv[q], acc);
  acc = acc + cxmk<float>(__shfl_xor_sync(0xffffffffu, acc.x, 2), __shfl_xor_sync(0xffffffffu, acc.y, 2));
  return acc + cxmk<float>(__shfl_xor_sync(0xffffffffu, acc.x, 1), __shfl_xor_sync(0xffffffffu, acc.y, 1));
}

__global__ void __launch_bounds__(1024) gehrd_panel_kernel(Cx<float>* __restrict__ Aall, int n, int lda, long long a_bs,
                                                           Cx<float>* __restrict__ tau_all, int k, int bb,
                                                           Cx<float>* __restrict__ Wsall, long long ws_bs) {
  using R = float;
  using C_ = Cx<R>;
  extern __shared__ __align__(16) unsigned char smraw[];
  C_* sb = reinterpret_cast<C_*>(smraw);          // (n) the column being reduced
  C_* sv = sb + n;                                 // (n) its reflector
  __shared__ C_ T[kHrdPanel][kHrdPanel + 1];
  __shared__ C_ s_vc[kHrdPanel], s_w[kHrdPanel], s_u[kHrdPanel];
  __shared__ R red[32];
  __shared__ C_ s_tau, s_scale;
  __shared__ R s_beta;
  __shared__ int s_id;
  C_* A = Aall + blockIdx.x * a_bs;
  C_* tau = tau_all + (long long)blockIdx.x * n;
  C_* ws = Wsall + blockIdx.x * ws_bs;
  const long long nB = (long long)n * kHrdPanel;
  C_* V = ws;
  C_* Vc = ws + nB;
  C_* Y = ws + 2 * nB;
  C_* TH = ws + 5 * nB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
  for (int e = tid; e < kHrdPanel * (kHrdPanel + 1); e += nt) T[e / (kHrdPanel + 1)][e % (kHrdPanel + 1)] = cxzero<R>();
  __syncthreads();
  for (int j = 0; j < bb; ++j) {
    const int c = k + j;
    if (tid < j) s_vc[tid] = cxconj(V[c + (long long)tid * n]);
    __syncthreads();
    // b = a_c - Y_j conj(V_j(c, :))
    for (int r = tid; r < n; r += nt) {
      C_ acc = A[r + (long long)c * lda];
#pragma unroll 8
      for (int l = 0; l < j; ++l) acc = acc - Y[r + (long long)l * n] * s_vc[l];
      sb[r] = acc;
    }
    __syncthreads();
    if (j > 0) {
      // w = V_j^H b (rows below k), u = T_j^H w, b <- b - V_j u
      for (int l = warp; l < j; l += nw) {
        C_ acc = cxzero<R>();
        for (int r = k + 1 + lane; r < n; r += 32) acc = cxfma_conj(V[r + (long long)l * n], sb[r], acc);
        acc.x = warp_sum(acc.x);
        acc.y = warp_sum(acc.y);
        if (lane == 0) s_w[l] = acc;
      }
      __syncthreads();
      if (tid < j) {
        C_ acc = cxzero<R>();
        for (int lp = 0; lp <= tid; ++lp) acc = cxfma_conj(T[lp][tid], s_w[lp], acc);
        s_u[tid] = acc;
      }
      __syncthreads();
      for (int r = k + 1 + tid; r < n; r += nt) {
        C_ acc = sb[r];
#pragma unroll 8
        for (int l = 0; l < j; ++l) acc = acc - V[r + (long long)l * n] * s_u[l];
        sb[r] = acc;
      }
      __syncthreads();
    }
    // the reflector of (b[c+1]; b[c+2:])
    R part = R(0.0);
    for (int r = c + 2 + tid; r < n; r += nt) part = part + cxabs2(sb[r]);
    const R xn2 = block_sum(part, red);
    if (tid == 0) {
      const Refl<R> rf = make_reflector(sb[c + 1], rsqrt_(xn2));
      s_id = rf.identity ? 1 : 0;
      s_tau = rf.identity ? cxzero<R>() : rf.tau;
      s_scale = rf.scale;
      s_beta = rf.beta;
      tau[c] = s_tau;
    }
    __syncthreads();
    const bool ident = s_id != 0;
    const C_ tj = s_tau, scl = s_scale;
    // v, V[:, j] and conj(V[:, j]), and column c in its final form
    for (int r = tid; r < n; r += nt) {
      C_ v = cxzero<R>();
      if (!ident) {
        if (r == c + 1) v = cxone<R>();
        else if (r > c + 1) v = sb[r] * scl;
      }
      sv[r] = v;
      V[r + (long long)j * n] = v;
      Vc[r + (long long)j * n] = cxconj(v);
      C_ a = sb[r];
      if (!ident && r == c + 1) a = cxmk<R>(s_beta, R(0.0));
      else if (!ident && r > c + 1) a = v;
      A[r + (long long)c * lda] = a;
    }
    __syncthreads();
    // w2 = V_j^H v, T[:j, j] = -tau T_j w2, T[j, j] = tau
    if (j > 0) {
      for (int l = warp; l < j; l += nw) {
        C_ acc = cxzero<R>();
        for (int r = c + 1 + lane; r < n; r += 32) acc = cxfma_conj(V[r + (long long)l * n], sv[r], acc);
        acc.x = warp_sum(acc.x);
        acc.y = warp_sum(acc.y);
        if (lane == 0) s_w[l] = acc;
      }
      __syncthreads();
      if (tid < j) {
        C_ acc = cxzero<R>();
        for (int lp = tid; lp < j; ++lp) acc = acc + T[tid][lp] * s_w[lp];
        T[tid][j] = -(tj * acc);
      }
    }
    if (tid == 0) T[j][j] = tj;
    __syncthreads();
    // Y[:, j] = tau (A[:, c+1:] v[c+1:] - Y_j w2): four threads a row, eight loads in flight each (a
    // thread a row and four loads ran on their latency)
    const int m = n - c - 1;
    for (int i0 = 0; i0 < n; i0 += nt / 4) {
      const int r = i0 + (tid >> 2);
      const bool in = r < n;
      C_ y = row_times<8>(A + (in ? r : 0) + (long long)(c + 1) * lda, lda, sv + c + 1, m);
      if (in && (tid & 3) == 0) {
#pragma unroll 8
        for (int l = 0; l < j; ++l) y = y - Y[r + (long long)l * n] * s_w[l];
        Y[r + (long long)j * n] = ident ? cxzero<R>() : tj * y;
      }
    }
    __syncthreads();
  }
  // T^H, column-major kHrdPanel x kHrdPanel, for the trailing update's X = T^H W
  for (int e = tid; e < kHrdPanel * kHrdPanel; e += nt) {
    const int r = e % kHrdPanel, cc = e / kHrdPanel;
    TH[e] = (r < bb && cc < bb) ? cxconj(T[cc][r]) : cxzero<R>();
  }
}

// The same panel by a cluster of CTAs a matrix, its rows shared out: one CTA pulls the trailing matrix through
// one SM once a column (21 of a column's 45 us at n = 798) and runs the panel's products on its latencies.
// Every CTA has the column and its reflector whole, its own rows of V and Y in shared memory, and the columns
// l = rank, rank + ctas, .. of V whole; rows of b, and the sums V^H b and V^H v, go to all by shared memory of
// the cluster. A row of A v is four threads, one a partial sum. Every sum has the order of gehrd_panel_kernel
// (the norm's that of its `vthreads` threads), so the bits are its.
constexpr int kHrdClusterThreads = 512;
static size_t hrd_panel_shared(int n, int ctas) {
  const int rp = (n + ctas - 1) / ctas;
  return sizeof(Cx<float>) * ((size_t)2 * n + (size_t)2 * kHrdPanel * rp + (size_t)(kHrdPanel / ctas) * n);
}

__device__ __forceinline__ void send32(Cx<float>* p, Cx<float> v, unsigned ctas) {
  const unsigned src = (unsigned)__cvta_generic_to_shared(p);
  for (unsigned c = 0; c < ctas; ++c) {
    unsigned dst;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(src), "r"(c));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(v.x) : "memory");
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + 4), "f"(v.y) : "memory");
  }
}

__global__ void __launch_bounds__(kHrdClusterThreads) gehrd_panel_cluster_kernel(
    Cx<float>* __restrict__ Aall, int n, int lda, long long a_bs, Cx<float>* __restrict__ tau_all, int k, int bb,
    Cx<float>* __restrict__ Wsall, long long ws_bs, int vthreads) {
  using R = float;
  using C_ = Cx<float>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const unsigned ctas = qr::cta_count(), rank = qr::cta_rank();
  const int rp = (n + (int)ctas - 1) / (int)ctas, r0 = (int)rank * rp, rows = max(0, min(rp, n - r0));
  C_* sb = reinterpret_cast<C_*>(smraw);          // (n) the column being reduced
  C_* sv = sb + n;                                 // (n) its reflector
  C_* sV = sv + n;                                 // [kHrdPanel][rp] this CTA's rows
  C_* sY = sV + kHrdPanel * rp;
  C_* sF = sY + kHrdPanel * rp;                    // [kHrdPanel / ctas][n] whole columns of V
  __shared__ C_ T[kHrdPanel][kHrdPanel + 1];
  __shared__ C_ top[kHrdPanel][kHrdPanel];         // [l][i]: V(k + i, l)
  __shared__ C_ s_vc[kHrdPanel], s_w[kHrdPanel], s_u[kHrdPanel];
  __shared__ R red[32];
  __shared__ C_ s_tau, s_scale;
  __shared__ R s_beta;
  __shared__ int s_id;
  C_* A = Aall + (blockIdx.x / ctas) * a_bs;
  C_* tau = tau_all + (long long)(blockIdx.x / ctas) * n;
  C_* ws = Wsall + (blockIdx.x / ctas) * ws_bs;
  const long long nB = (long long)n * kHrdPanel;
  C_* V = ws;
  C_* Vc = ws + nB;
  C_* Y = ws + 2 * nB;
  C_* TH = ws + 5 * nB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
  for (int e = tid; e < kHrdPanel * (kHrdPanel + 1); e += nt) T[e / (kHrdPanel + 1)][e % (kHrdPanel + 1)] = cxzero<R>();
  qr::barrier_all(ctas);
  for (int j = 0; j < bb; ++j) {
    const int c = k + j;
    if (tid < j) s_vc[tid] = cxconj(top[tid][j]);
    __syncthreads();
    // b = a_c - Y_j conj(V_j(c, :))
    for (int i = tid; i < rows; i += nt) {
      C_ acc = A[r0 + i + (long long)c * lda];
      for (int l = 0; l < j; ++l) acc = acc - sY[l * rp + i] * s_vc[l];
      send32(sb + r0 + i, acc, ctas);
    }
    qr::barrier_all(ctas);
    if (j > 0) {
      // w = V_j^H b (rows below k), u = T_j^H w, b <- b - V_j u
      for (int l = (int)rank + warp * (int)ctas; l < j; l += nw * (int)ctas) {
        const C_* f = sF + (l / (int)ctas) * n;
        C_ acc = cxzero<R>();
        for (int r = k + 1 + lane; r < n; r += 32) acc = cxfma_conj(f[r], sb[r], acc);
        acc.x = warp_sum(acc.x);
        acc.y = warp_sum(acc.y);
        if (lane == 0) send32(s_w + l, acc, ctas);
      }
      qr::barrier_all(ctas);
      if (tid < j) {
        C_ acc = cxzero<R>();
        for (int lp = 0; lp <= tid; ++lp) acc = cxfma_conj(T[lp][tid], s_w[lp], acc);
        s_u[tid] = acc;
      }
      __syncthreads();
      for (int i = tid; i < rows; i += nt) {
        if (r0 + i < k + 1) continue;
        C_ acc = sb[r0 + i];
        for (int l = 0; l < j; ++l) acc = acc - sV[l * rp + i] * s_u[l];
        send32(sb + r0 + i, acc, ctas);
      }
      qr::barrier_all(ctas);
    }
    // the reflector of (b[c+1]; b[c+2:])
    for (int vw = warp; vw < vthreads / 32; vw += nw) {
      R part = R(0.0);
      for (int r = c + 2 + 32 * vw + lane; r < n; r += vthreads) part = part + cxabs2(sb[r]);
      part = warp_sum(part);
      if (lane == 0) red[vw] = part;
    }
    __syncthreads();
    if (tid == 0) {
      R xn2 = R(0.0);
      for (int w = 0; w < vthreads / 32; ++w) xn2 = xn2 + red[w];
      const Refl<R> rf = make_reflector(sb[c + 1], rsqrt_(xn2));
      s_id = rf.identity ? 1 : 0;
      s_tau = rf.identity ? cxzero<R>() : rf.tau;
      s_scale = rf.scale;
      s_beta = rf.beta;
      if (rank == 0) tau[c] = s_tau;
    }
    __syncthreads();
    const bool ident = s_id != 0;
    const C_ tj = s_tau, scl = s_scale;
    // v whole, V[:, j] and conj(V[:, j]), and column c in its final form
    const bool keep = j % (int)ctas == (int)rank;
    for (int r = tid; r < n; r += nt) {
      C_ v = cxzero<R>();
      if (!ident) {
        if (r == c + 1) v = cxone<R>();
        else if (r > c + 1) v = sb[r] * scl;
      }
      sv[r] = v;
      if (keep) sF[(j / (int)ctas) * n + r] = v;
      if (r >= k && r < k + kHrdPanel) top[j][r - k] = v;
      const int i = r - r0;
      if (i >= 0 && i < rows) {
        sV[j * rp + i] = v;
        V[r + (long long)j * n] = v;
        Vc[r + (long long)j * n] = cxconj(v);
        C_ a = sb[r];
        if (!ident && r == c + 1) a = cxmk<R>(s_beta, R(0.0));
        else if (!ident && r > c + 1) a = v;
        A[r + (long long)c * lda] = a;
      }
    }
    __syncthreads();
    // w2 = V_j^H v, T[:j, j] = -tau T_j w2, T[j, j] = tau
    if (j > 0) {
      for (int l = (int)rank + warp * (int)ctas; l < j; l += nw * (int)ctas) {
        const C_* f = sF + (l / (int)ctas) * n;
        C_ acc = cxzero<R>();
        for (int r = c + 1 + lane; r < n; r += 32) acc = cxfma_conj(f[r], sv[r], acc);
        acc.x = warp_sum(acc.x);
        acc.y = warp_sum(acc.y);
        if (lane == 0) send32(s_w + l, acc, ctas);
      }
    }
    qr::barrier_all(ctas);
    if (tid < j) {
      C_ acc = cxzero<R>();
      for (int lp = tid; lp < j; ++lp) acc = acc + T[tid][lp] * s_w[lp];
      T[tid][j] = -(tj * acc);
    }
    if (tid == 0) T[j][j] = tj;
    // Y[:, j] = tau (A[:, c+1:] v[c+1:] - Y_j w2), four threads a row
    for (int i0 = 0; i0 < rows; i0 += nt / 4) {
      const int i = i0 + (tid >> 2);
      const bool in = i < rows;
      C_ y = row_times<16>(A + (in ? r0 + i : r0) + (long long)(c + 1) * lda, lda, sv + c + 1, n - c - 1);
      if (in && (tid & 3) == 0) {
        for (int l = 0; l < j; ++l) y = y - sY[l * rp + i] * s_w[l];
        y = ident ? cxzero<R>() : tj * y;
        sY[j * rp + i] = y;
        Y[r0 + i + (long long)j * n] = y;
      }
    }
    __syncthreads();
  }
  // T^H, column-major kHrdPanel x kHrdPanel, for the trailing update's X = T^H W
  if (rank == 0)
    for (int e = tid; e < kHrdPanel * kHrdPanel; e += nt) {
      const int r = e % kHrdPanel, cc = e / kHrdPanel;
      TH[e] = (r < bb && cc < bb) ? cxconj(T[cc][r]) : cxzero<R>();
    }
  qr::barrier_all(ctas);                                        // no CTA leaves while another may still send to it
}

// --------------------------------------------- 2b. Q from the reflectors in panels (FP32 form)
// Q = H_0 H_1 ... H_{n-3} is formed as unghr_kernel forms it, last reflectors first, but
// kHrdPanel reflectors at a time: their product is I - V T V^H (T upper triangular, built
// forward: T[:j, j] = -tau_j T_j V_j^H v_j, T[j, j] = tau_j), and Z's trailing block gets
// Z <- Z - V (T (V^H Z)) as batched products. This kernel writes the panel's V, conj(V) (n x
// kHrdPanel) and T (column-major kHrdPanel x kHrdPanel) into the scratch.
__global__ void __launch_bounds__(1024) unghr_panel_kernel(const Cx<float>* __restrict__ Aall, int n, int lda,
                                                           long long a_bs, const Cx<float>* __restrict__ tau_all, int k0,
                                                           int bb, Cx<float>* __restrict__ Wsall, long long ws_bs) {
  using R = float;
  using C_ = Cx<R>;
  __shared__ C_ T[kHrdPanel][kHrdPanel + 1];
  __shared__ C_ s_w[kHrdPanel];
  const C_* A = Aall + blockIdx.x * a_bs;
  const C_* tau = tau_all + (long long)blockIdx.x * n;
  C_* ws = Wsall + blockIdx.x * ws_bs;
  const long long nB = (long long)n * kHrdPanel;
  C_* V = ws;
  C_* Vc = ws + nB;
  C_* Tm = ws + 4 * nB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
  for (int e = tid; e < kHrdPanel * (kHrdPanel + 1); e += nt) T[e / (kHrdPanel + 1)][e % (kHrdPanel + 1)] = cxzero<R>();
  for (long long e = tid; e < nB; e += nt) {
    const int r = (int)(e % n), j = (int)(e / n), c = k0 + j;
    C_ v = cxzero<R>();
    if (j < bb) {
      const C_ t = tau[c];
      if (!(t.x == R(0.0) && t.y == R(0.0))) {
        if (r == c + 1) v = cxone<R>();
        else if (r > c + 1) v = A[r + (long long)c * lda];
      }
    }
    V[e] = v;
    Vc[e] = cxconj(v);
  }
  __syncthreads();
  for (int j = 0; j < bb; ++j) {
    const int c = k0 + j;
    const C_ tj = tau[c];
    for (int l = warp; l < j; l += nw) {
      C_ acc = cxzero<R>();
      for (int r = c + 1 + lane; r < n; r += 32) acc = cxfma_conj(V[r + (long long)l * n], V[r + (long long)j * n], acc);
      acc.x = warp_sum(acc.x);
      acc.y = warp_sum(acc.y);
      if (lane == 0) s_w[l] = acc;
    }
    __syncthreads();
    if (tid < j) {
      C_ acc = cxzero<R>();
      for (int lp = tid; lp < j; ++lp) acc = acc + T[tid][lp] * s_w[lp];
      T[tid][j] = -(tj * acc);
    }
    if (tid == 0) T[j][j] = tj;
    __syncthreads();
  }
  for (int e = tid; e < kHrdPanel * kHrdPanel; e += nt) {
    const int r = e % kHrdPanel, cc = e / kHrdPanel;
    Tm[e] = (r < bb && cc < bb) ? T[r][cc] : cxzero<R>();
  }
}

// the reflectors' storage below the subdiagonal cleared, leaving H
template <class R>
__global__ void clear_below_subdiag_kernel(Cx<R>* __restrict__ Aall, int n, int lda, long long a_bs) {
  Cx<R>* A = Aall + blockIdx.y * a_bs;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < (long long)n * n;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e % n), j = (int)(e / n);
    if (i > j + 1) A[i + (long long)j * lda] = cxzero<R>();
  }
}

// ------------------------------------------------------------------ 2. form Q = Z
template <class R>
__global__ void __launch_bounds__(1024) unghr_kernel(Cx<R>* __restrict__ Aall, int n, int lda,
                                                            long long a_bs, const Cx<R>* __restrict__ tau_all,
                                                            Cx<R>* __restrict__ Zall, int ldz, long long z_bs,
                                                            const int* __restrict__ live) {
  using C_ = Cx<R>;
  if (live && (int)blockIdx.x >= *live) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  C_* sv = reinterpret_cast<C_*>(smraw);
  C_* A = Aall + blockIdx.x * a_bs;
  C_* Z = Zall + blockIdx.x * z_bs;
  const C_* tau = tau_all + (long long)blockIdx.x * n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  for (long long e = tid; e < (long long)n * n; e += blockDim.x) {
    int i = (int)(e % n), j = (int)(e / n);
    Z[i + (long long)j * ldz] = (i == j) ? cxone<R>() : cxzero<R>();
  }
  __syncthreads();
  for (int k = n - 3; k >= 0; --k) {
    const int m = n - k - 1;
    const C_ t = tau[k];
    if (t.x == R(0.0) && t.y == R(0.0)) continue;
    for (int i = tid; i < m; i += blockDim.x) sv[i] = (i == 0) ? cxone<R>() : A[k + 1 + i + (long long)k * lda];
    __syncthreads();
    for (int j = warp; j < m; j += nw) {
      C_* cj = Z + (long long)(k + 1 + j) * ldz;
      const C_ acc = column_dot<R>(sv, cj + k + 1, m, lane);
      const C_ f = t * acc;
      for (int i0 = lane; i0 < m; i0 += 32 * kUnroll) {
        C_ val[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
          if (i0 + 32 * u < m) val[u] = cj[k + 1 + i0 + 32 * u];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u)
          if (i0 + 32 * u < m) cj[k + 1 + i0 + 32 * u] = val[u] - sv[i0 + 32 * u] * f;
      }
    }
    __syncthreads();
  }
  for (long long e = tid; e < (long long)n * n; e += blockDim.x) {
    int i = (int)(e % n), j = (int)(e / n);
    if (i > j + 1) A[i + (long long)j * lda] = cxzero<R>();
  }
}

// ---------------------------------------------------------- 3. Schur form by shifted QR: wb_qr.cuh
// FP64 matrices of up to kQrSmall, and some double-float ones (qr_small), take the sweep element by
// element, one CTA a matrix and one barrier a reflector: the windows of wb_qr.cuh are 16 reflectors wide
// and their two ticks a sweep (a window, and its far updates before the next sweep) cost more there. The
// FP64 ones are the 32 x 32 group blocks of the mixed form's Newton steps, most of them diagonal.
constexpr int kQrSmall = 32;

// MT, its largest CTA, sets the registers: 85 a thread for 768, so that CTAs run side by side; 255 for 256.
template <class R, int MT>
__global__ void __launch_bounds__(MT) hseqr_small_kernel(Cx<R>* __restrict__ Hall, int n, int ldh,
                                                            long long h_bs, Cx<R>* __restrict__ Zall, int ldz,
                                                            long long z_bs, Cx<R>* __restrict__ w_all,
                                                            int32_t* __restrict__ status, int st_div, int itmax, const int* __restrict__ live) {
  using C_ = Cx<R>;
  if (live && (int)blockIdx.x >= *live) return;
  extern __shared__ __align__(16) unsigned char smraw[];
  C_* sphase = reinterpret_cast<C_*>(smraw);
  __shared__ int ired[32];
  __shared__ C_ s_t1[2], s_v2[2], s_sc;
  __shared__ R s_t2[2];
  __shared__ int s_done;
  constexpr int kChunk = sizeof(R) <= 4 ? 4 : 2;   // worker items whose loads are issued together
  C_* H = Hall + blockIdx.x * h_bs;
  C_* Z = Zall + blockIdx.x * z_bs;
  C_* w = w_all + (long long)blockIdx.x * n;
  int32_t* st = status ? status + blockIdx.x / st_div : nullptr;
  const int tid = threadIdx.x, warp = tid >> 5;
  const R ulp = RealT<R>::eps();
  const R smlnum = RealT<R>::tiny() * (R((double)n) / ulp);
  auto h = [&](int i, int j) -> C_& { return H[i + (long long)j * ldh]; };
  // subdiagonal made real by a diagonal similarity D^-1 H D, |d_i| = 1, d_i = d_{i-1} sd_i/|sd_i|
  if (tid == 0) {
    C_ d = cxone<R>();
    sphase[0] = d;
    for (int r = 1; r < n; ++r) {
      C_ sd = h(r, r - 1);
      R a = cxabs(sd);
      // a subdiagonal below the safe range keeps a unit phase (its imaginary part is dropped)
      if (a > RealT<R>::tiny() && sd.y != R(0.0)) d = d * (sd * (R(1.0) / a));
      sphase[r] = d;
    }
  }
  __syncthreads();
  for (long long e = tid; e < (long long)n * n; e += blockDim.x) {
    int r = (int)(e % n), c = (int)(e / n);
    if (r <= c + 1) h(r, c) = (cxconj(sphase[r]) * h(r, c)) * sphase[c];
    Z[r + (long long)c * ldz] = Z[r + (long long)c * ldz] * sphase[c];
  }
  __syncthreads();
  for (int r = 1 + tid; r < n; r += blockDim.x) h(r, r - 1) = cxmk<R>(h(r, r - 1).x, R(0.0));
  __syncthreads();
  int i = n - 1;
  int total = 0;
  long long steps = 0;
  bool failed = false;
  while (i >= 0 && !failed) {
    int its = 0;
    for (;;) {
      // --- deflation: largest k in [1, i] with a negligible subdiagonal H(k, k-1)
      int cand = 0;
      for (int k = 1 + tid; k <= i; k += blockDim.x) {
        C_ sub = h(k, k - 1);
        bool small = false;
        if (cxabs1(sub) <= smlnum) {
          small = true;
        } else {
          R tst = cxabs1(h(k - 1, k - 1)) + cxabs1(h(k, k));
          if (tst == R(0.0)) {
            if (k - 2 >= 0) tst = tst + rabs(h(k - 1, k - 2).x);
            if (k + 1 <= i) tst = tst + rabs(h(k + 1, k).x);
          }
          if (rabs(sub.x) <= ulp * tst) {
            R ab = rmax(cxabs1(sub), cxabs1(h(k - 1, k)));
            R ba = rmin(cxabs1(sub), cxabs1(h(k - 1, k)));
            C_ dd = h(k - 1, k - 1) - h(k, k);
            R aa = rmax(cxabs1(h(k, k)), cxabs1(dd));
            R bb = rmin(cxabs1(h(k, k)), cxabs1(dd));
            R sx = aa + ab;
            if (ba * (ab / sx) <= rmax(smlnum, ulp * (bb * (aa / sx)))) small = true;
          }
        }
        if (small) cand = max(cand, k);
      }
      const int l = block_max_int(cand, ired);
      if (l >= i) break;
      if (tid == 0 && l > 0) h(l, l - 1) = cxzero<R>();
      if (its >= 60 || total >= itmax) { failed = true; break; }
      ++its; ++total;
      steps += i - l;
      // --- shift and first reflector vector (thread 0)
      if (tid == 0) {
        C_ t;
        if (its % 20 == 10) {
          R sx = R(0.75) * rabs(h(l + 1, l).x);
          t = cxmk<R>(sx, R(0.0)) + h(l, l);
        } else if (its % 20 == 0) {
          R sx = R(0.75) * rabs(h(i, i - 1).x);
          t = cxmk<R>(sx, R(0.0)) + h(i, i);
        } else {
          t = h(i, i);
          C_ u = cxsqrt(h(i - 1, i)) * cxsqrt(h(i, i - 1));
          R sx = cxabs1(u);
          if (sx != R(0.0)) {
            C_ x = (h(i - 1, i - 1) - t) * R(0.5);
            R sxx = cxabs1(x);
            sx = rmax(sx, cxabs1(x));
            C_ xs = x * (R(1.0) / sx), us = u * (R(1.0) / sx);
            C_ y = cxsqrt(xs * xs + us * us) * sx;
            if (sxx > R(0.0)) {
              C_ xn = x * (R(1.0) / sxx);
              if (xn.x * y.x + xn.y * y.y < R(0.0)) y = -y;
            }
            t = t - u * cxdiv(u, x + y);
          }
        }
        C_ h11s = h(l, l) - t;
        R h21 = h(l + 1, l).x;
        R sc = cxabs1(h11s) + rabs(h21);
        if (sc == R(0.0)) sc = R(1.0);
        R isc = R(1.0) / sc;
        // the first reflector of the sweep, from the shifted first column
        Rot<R> rf = householder(h11s * isc, h21 * isc);
        s_t1[l & 1] = rf.t1; s_v2[l & 1] = rf.v2; s_t2[l & 1] = rf.t2;
      }
      __syncthreads();
      // Bulge chase, one CTA barrier per step. Reflector k acts on rows/columns (k, k+1). The core
      // lane (thread 0) owns the elements where its left and right applications meet -- rows
      // k..min(k+2, i) of columns k, k+1 -- and, having updated them, builds reflector k+1 from
      // its own (k+1, k), (k+2, k) and publishes it (double-buffered in shared memory). The worker
      // warps (all but warp 0) apply reflector k everywhere else, in one phase, since those
      // elements are disjoint: rows k, k+1 of columns k+2..n-1 (left), rows 0..k-1 of columns
      // k, k+1 (right) and Z's columns k, k+1. Each worker issues the loads of up to kChunk items
      // before it updates any, so that one memory latency serves the chunk.
      for (int k = l; k < i; ++k) {
        const int sl = k & 1;
        const C_ t1 = s_t1[sl], v2 = s_v2[sl];
        const R t2 = s_t2[sl];
        const C_ t1c = cxconj(t1), v2c = cxconj(v2);
        if (warp == 0) {
          if (tid == 0) {
            const bool has2 = (k + 2 <= i);
            C_ h00 = h(k, k), h01 = h(k, k + 1), h10 = h(k + 1, k), h11 = h(k + 1, k + 1);
            C_ h21 = has2 ? h(k + 2, k + 1) : cxzero<R>();
            C_ sum = t1c * h00 + h10 * t2;             // left on columns k, k+1
            h00 = h00 - sum; h10 = h10 - sum * v2;
            sum = t1c * h01 + h11 * t2;
            h01 = h01 - sum; h11 = h11 - sum * v2;
            sum = t1 * h00 + h01 * t2;                 // right on rows k, k+1, k+2
            h00 = h00 - sum; h01 = h01 - sum * v2c;
            sum = t1 * h10 + h11 * t2;
            h10 = h10 - sum; h11 = h11 - sum * v2c;
            sum = h21 * t2;                            // (k+2, k) is zero before this step
            C_ h20 = -sum;
            h21 = h21 - sum * v2c;
            h(k, k) = h00; h(k, k + 1) = h01; h(k + 1, k + 1) = h11;
            if (has2) h(k + 2, k + 1) = h21;
            if (k + 1 < i) {
              Rot<R> rn = householder(h10, h20.x);
              h(k + 1, k) = rn.identity ? h10 : cxmk<R>(rn.beta, R(0.0));
              h(k + 2, k) = cxzero<R>();
              s_t1[sl ^ 1] = rn.t1; s_v2[sl ^ 1] = rn.v2; s_t2[sl ^ 1] = rn.t2;
            } else {
              h(k + 1, k) = h10;
              if (has2) h(k + 2, k) = h20;
            }
          }
        } else {
          const int wt = blockDim.x - 32, wid = tid - 32;
          const int nL = max(0, n - (k + 2)), nR = k, total = nL + nR + n;
          for (int base = wid; base < total; base += kChunk * wt) {
            C_* pa[kChunk];
            C_* pb[kChunk];
            C_ a[kChunk], b[kChunk];
#pragma unroll
            for (int u = 0; u < kChunk; ++u) {
              int e = base + u * wt;
              if (e < nL) { pa[u] = &h(k, k + 2 + e); pb[u] = pa[u] + 1; }
              else if (e < nL + nR) { e -= nL; pa[u] = &h(e, k); pb[u] = &h(e, k + 1); }
              else if (e < total) { e -= nL + nR; pa[u] = Z + e + (long long)k * ldz; pb[u] = pa[u] + ldz; }
              else { pa[u] = nullptr; pb[u] = nullptr; }
            }
#pragma unroll
            for (int u = 0; u < kChunk; ++u)
              if (pa[u]) { a[u] = *pa[u]; b[u] = *pb[u]; }
#pragma unroll
            for (int u = 0; u < kChunk; ++u) {
              if (!pa[u]) continue;
              if (base + u * wt < nL) {
                const C_ sum = t1c * a[u] + b[u] * t2;
                *pa[u] = a[u] - sum; *pb[u] = b[u] - sum * v2;
              } else {
                const C_ sum = t1 * a[u] + b[u] * t2;
                *pa[u] = a[u] - sum; *pb[u] = b[u] - sum * v2c;
              }
            }
          }
        }
        __syncthreads();
      }
      // make H(i, i-1) real again
      if (tid == 0) {
        C_ sd = h(i, i - 1);
        s_done = 0;
        if (sd.y != R(0.0)) {
          R a = cxabs(sd);
          if (a > RealT<R>::tiny()) {
            h(i, i - 1) = cxmk<R>(a, R(0.0));
            s_sc = sd * (R(1.0) / a);
            s_done = 1;
          } else {
            h(i, i - 1) = cxmk<R>(sd.x, R(0.0));      // below the safe range: negligible
          }
        }
      }
      __syncthreads();
      if (s_done) {
        const C_ sc = s_sc;
        for (int j = i + 1 + tid; j < n; j += blockDim.x) h(i, j) = cxconj(sc) * h(i, j);
        for (int j = tid; j < i; j += blockDim.x) h(j, i) = sc * h(j, i);
        for (int j = tid; j < n; j += blockDim.x) Z[j + (long long)i * ldz] = sc * Z[j + (long long)i * ldz];
      }
      __syncthreads();
    }
    if (failed) break;
    if (tid == 0) w[i] = h(i, i);
    __syncthreads();
    i -= 1;
  }
  if (failed) {
    for (int j = tid; j <= i; j += blockDim.x) w[j] = cxmk<R>(R(NAN), R(NAN));
    if (tid == 0) wb_flag(st, WB_ST_NOCONV);
  }
  if (tid == 0)
    atomicAdd(&g_qr_bytes[QrSlot<R>::v],
              (unsigned long long)steps * (unsigned long long)(2 * n - 2) * 2ULL * sizeof(C_));
}

// -------------------------------------------------- 4. eigenvectors of the triangular T
// X[:, k] solves (T[0:k,0:k] - T(k,k) I) x = -T[0:k, k] with x_k = 1, x_j = 0 for j > k.
// One warp per column; tiny pivots are replaced by max(ulp |T(k,k)|, smlnum).
template <class R>
__global__ void __launch_bounds__(256) trevc_kernel(const Cx<R>* __restrict__ Tall, int n, int ldt,
                                                    long long t_bs, Cx<R>* __restrict__ Xall, int ldx,
                                                    long long x_bs, int batch, const int* __restrict__ live) {
  using C_ = Cx<R>;
  const int warps_per_block = blockDim.x >> 5;
  long long gw = (long long)blockIdx.x * warps_per_block + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (gw >= (long long)batch * n) return;
  const int b = (int)(gw / n), k = (int)(gw % n);
  if (live && b >= *live) return;
  const C_* T = Tall + b * t_bs;
  C_* x = Xall + b * x_bs + (long long)k * ldx;
  const R ulp = RealT<R>::eps();
  const R smlnum = RealT<R>::tiny() * (R((double)n) / ulp);
  const C_ lam = T[k + (long long)k * ldt];
  const R smin = rmax(ulp * cxabs1(lam), smlnum);
  for (int r = lane; r < n; r += 32) {
    C_ v;
    if (r < k) v = -T[r + (long long)k * ldt];
    else v = (r == k) ? cxone<R>() : cxzero<R>();
    x[r] = v;
  }
  __syncwarp();
  // back-substitution with rescaling: whenever a component exceeds `big`, the whole column (the
  // solved part and the remaining right-hand side) is scaled down, since an eigenvector is only
  // defined up to scale. This keeps the double-float form (FP32 exponent range) finite where
  // nearly equal eigenvalues make the triangular solve grow.
  const R big = RealT<R>::big();
  for (int j = k - 1; j >= 0; --j) {
    C_ xj = cxzero<R>();
    if (lane == (j & 31)) {
      C_ d = T[j + (long long)j * ldt] - lam;
      if (cxabs1(d) < smin) d = cxmk<R>(smin, R(0.0));
      xj = cxdiv(x[j], d);
      x[j] = xj;
    }
    xj.x = shfl_idx(xj.x, j & 31);
    xj.y = shfl_idx(xj.y, j & 31);
    R mag = cxabs1(xj);
    if (mag > big) {
      const R sc = R(1.0) / mag;
      __syncwarp();
      for (int r = lane; r <= k; r += 32) x[r] = x[r] * sc;
      xj = xj * sc;
      __syncwarp();
    }
    const C_* tc = T + (long long)j * ldt;
    for (int r = lane; r < j; r += 32) x[r] = x[r] - xj * tc[r];
    __syncwarp();
  }
}

// ------------------------------------------------------------- 5. column normalisation
template <class R>
__global__ void normalize_columns_kernel(Cx<R>* __restrict__ Wall, int n, int ldw, long long w_bs, int batch,
                                         const int* __restrict__ live) {
  using C_ = Cx<R>;
  const int warps_per_block = blockDim.x >> 5;
  long long gw = (long long)blockIdx.x * warps_per_block + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (gw >= (long long)batch * n) return;
  const int b = (int)(gw / n), k = (int)(gw % n);
  if (live && b >= *live) return;
  C_* c = Wall + b * w_bs + (long long)k * ldw;
  R s = R(0.0);
  for (int r = lane; r < n; r += 32) s = s + cxabs2(c[r]);
  s = warp_sum(s);
  R inv = (s > R(0.0)) ? R(1.0) / rsqrt_(s) : R(1.0);
  for (int r = lane; r < n; r += 32) c[r] = c[r] * inv;
}

// Live timing of the QR-sweep launches (per real type), for the benchmark's roofline: CUDA
// events recorded on the launching stream around every hseqr launch while profiling is on.
namespace {
struct QrProfile {
  bool on = false;
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ev[3];
};
QrProfile g_qrp;
std::mutex g_qrp_mutex;
}  // namespace

void qr_profile(bool on) {
  std::lock_guard<std::mutex> lock(g_qrp_mutex);
  for (auto& v : g_qrp.ev)
    for (auto& e : v) { cudaEventDestroy(e.first); cudaEventDestroy(e.second); }
  for (auto& v : g_qrp.ev) v.clear();
  unsigned long long zero[3] = {0, 0, 0};
  cudaMemcpyToSymbol(g_qr_bytes, zero, sizeof(zero));
  g_qrp.on = on;
}

int qr_profile_read(int slot, double* ms, long long* launches, double* bytes) {
  if (slot < 0 || slot > 2) return 1;
  std::lock_guard<std::mutex> lock(g_qrp_mutex);
  double t = 0.0;
  for (auto& e : g_qrp.ev[slot]) {
    float x = 0.f;
    if (cudaEventSynchronize(e.second) != cudaSuccess || cudaEventElapsedTime(&x, e.first, e.second) != cudaSuccess) {
      cudaGetLastError();
      return 2;
    }
    t += x;
  }
  unsigned long long b[3] = {0, 0, 0};
  if (cudaMemcpyFromSymbol(b, g_qr_bytes, sizeof(b)) != cudaSuccess) { cudaGetLastError(); return 2; }
  *ms = t;
  *launches = (long long)g_qrp.ev[slot].size();
  *bytes = (double)b[slot];
  return 0;
}

// CTAs a matrix (a cluster) and threads a CTA of the QR sweep. A window's far updates are about
// 2 n / 32 warp tasks; the chase of a window takes as long as a few rounds of them, so a small
// matrix needs one task a warp and no second CTA. WB_TUNE_QR_THREADS overrides the threads (the
// autotuner sets it).
struct QrShape { int ctas, threads; size_t smem; };
template <class R> static QrShape qr_shape(int batch, int n) {
  const int sms = sm_count(), tasks = 2 * ((n + 31) / 32) + 1;
  int want;
  if (sizeof(R) == 4) want = n < 320 ? 1 : n < 640 ? 2 : 4;
  else want = n < 24 ? 1 : n < 160 ? 2 : n < 480 ? 4 : 8;
  int c = 1;
  while (2 * c <= want && 2LL * c * batch <= sms) c *= 2;
  const long long per_sm = ((long long)batch * c + sms - 1) / sms;
  // More matrices than SMs: small CTAs side by side, as many as the registers take (modes of 600 matrices of
  // 242, FP32: 4 warps 231 ms, 6 206, 8 221; FP64: 4 warps 1.23 s, 5 1.59, 8 1.33), until a tick's far updates
  // outlast its chase and the largest CTA wins (sweep of 512 of 450, FP32: 4 warps 784 ms, 8 656, 16 451;
  // FP64: 4 warps 5.0 s, 5 8.1, 8 4.2). In FP64 two of 4 warps fit an SM, so three matrices an SM take one of 8 at a
  // time (modes of 450 of 162 / 242: 4 warps 417 / 1133 ms, 8 389 / 1027).
  const int cap = sizeof(R) == 4 ? (per_sm <= 1 || n >= 256 ? 16 : per_sm <= 2 ? 7 : 6)
                                 : (per_sm <= 1 || n >= 320 || (per_sm == 3 && n >= 160) ? 8 : 4);
  int warps = (tasks + c - 1) / c + 1;
  warps = warps > cap ? cap : warps < 4 ? 4 : warps;
  QrShape s;
  s.ctas = c;
  s.threads = 32 * warps;
  const int forced = tuning(kTuneQrThreads);
  if (forced >= 64 && forced % 32 == 0)
    s.threads = forced < 128 ? 128 : forced < QrMaxThreads<R>::v ? forced : QrMaxThreads<R>::v;
  const size_t work = 2 * (size_t)QrWin<R>::m * QrTile<R>::ld + (size_t)(s.threads / 32) * 32 * (QrWin<R>::m + 1);
  s.smem = sizeof(Cx<R>) * (work > (size_t)n ? work : (size_t)n);
  return s;
}

// The element-by-element sweep where it is taken (threads, 0 where not; wide: by the instance with 255 registers): FP64
// matrices of up to kQrSmall, and of double-float (the same bits either way; modes in ms)
//   n <= 22: one matrix of 14 / 18 1.5 / 2.4, in windows 1.8 / 2.8;
//   one matrix an SM from n = 144 on, by as many threads as have pairs: 152 of 162 / 242 / 450 173 / 394 / 1714, in windows
//     185 / 424 / 2219; where windows still have two CTAs' room they win below n = 400 (100 of 202: 205, 198 in windows;
//     of 450: 1595, 1777);
//   k > 1 matrices an SM (600 of 50 / 126 / 242: 24 / 169 / 1080, in windows 35 / 228 / 1260), by threads and registers that
//     fill whole waves: 255 registers let two CTAs of 256 threads or four of 128 run side by side, 85 three of 256
//     or six of 128, each at less.
//     n >= 126: two wide of 256 for k = 2 (200 of 242: 463; 478 narrow, 536 by 128), four wide of 128 for k = 4 (600 of
//     450: 5584; 5778 narrow of 256), else three narrow of 256 (450 of 338: 1904; 2111 and 2374 wide; 760 of 242: 1264; 1681, 1443).
//     n = 65..125: three narrow of 256 for k <= 3 (400 of 70: 45; 48 wide of 128), else four wide or six narrow of 128, 1.4 times
//     as long, whichever takes its waves in less (600 / 1500 of 66: 47 / 128 and 63 / 123).
struct QrSmall { int threads; bool wide; };
template <class R> static QrSmall qr_small(int batch, int n) {
  const bool fp64 = std::is_same<R, double>::value;
  const int sms = sm_count(), k = (batch + sms - 1) / sms;
  const bool each = n >= 144 && 4LL * batch > (n >= 400 ? 2LL : 3LL) * sms;
  if (!(fp64 ? n <= kQrSmall : n <= 22 || k > 1 || each)) return {0, false};
  QrSmall q = {128, fp64};
  if (!fp64 && k > 1) {
    if (n >= 126) q = {k == 4 ? 128 : 256, k == 2 || k == 4};
    else if (n > 64 && k <= 3) q = {256, false};
    else q = {128, 10 * ((k + 3) / 4) <= 14 * ((k + 5) / 6)};
  } else if (n > 64) {
    q = {768, false};
    while (q.threads > 128 && q.threads / 2 >= 2 * n) q.threads /= 2;
  }
  const int most = q.wide ? 256 : 768, forced = tuning(kTuneQrThreads);
  if (forced >= 64 && forced % 32 == 0) q.threads = forced < most ? forced : most;
  return q;
}

// Threads of one Hessenberg-reduction (and Q-forming) CTA: one warp per trailing column, so as
// many warps as fit when few matrices share an SM. WB_TUNE_HRD_THREADS overrides the choice.
int hrd_threads(int batch, int n) {
  const int forced = tuning(kTuneHrdThreads);
  if (forced >= 64 && forced <= 1024 && forced % 32 == 0) return forced;
  const int per_sm = (batch + sm_count() - 1) / sm_count();
  int t = per_sm <= 1 ? 1024 : per_sm <= 2 ? 512 : 256;
  while (t > 128 && t / 32 > n) t /= 2;
  return t;
}

// Launches kernel with `ctas` CTAs a matrix as one cluster; `most`: its largest dynamic shared memory.
template <class... P, class... Q>
static void launch_cluster(cudaStream_t s, void (*kernel)(P...), int most, int ctas, int batch, int threads, size_t smem,
                           Q... args) {
  allow_shared(kernel, most);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(batch * ctas));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)ctas;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);
  note_launch();
}

// FP64, n > kQrSmall: H and Q by wb_hrd.cuh; false where its shared memory does not reach.
static bool reduce64(cudaStream_t s, int batch, int n, Cx<double>* A, int lda, long long a_bs, Cx<double>* Z, int ldz,
                     long long z_bs, Cx<double>* tau) {
  const size_t smem = hrd::shared_elements(n) * sizeof(Cx<double>);
  constexpr int most = 200 * 1024;
  if (n > 512 || smem > most) return false;
  const int sms = sm_count();
  int c = 1;
  while (2 * c <= hrd::kParts && 2LL * c * batch <= sms) c *= 2;
  if (n <= 64) launch_cluster(s, hrd::gehrd64_kernel<2>, most, c, batch, hrd::kThreads, smem, A, n, lda, a_bs, tau);
  else if (n <= 128) launch_cluster(s, hrd::gehrd64_kernel<4>, most, c, batch, hrd::kThreads, smem, A, n, lda, a_bs, tau);
  else launch_cluster(s, hrd::gehrd64_kernel<8>, most, c, batch, hrd::kThreads, smem, A, n, lda, a_bs, tau);
  const int groups = n <= 256 ? (n + 1) / 2 : n;
  const unsigned gx = (unsigned)max(1LL, min((long long)(groups + 3) / 4, (2LL * sms + batch - 1) / batch));
  const dim3 grid(gx, (unsigned)batch);
  if (n <= 64) hrd::unghr64_kernel<2, 2><<<grid, 128, 0, s>>>(A, n, lda, a_bs, tau, Z, ldz, z_bs);
  else if (n <= 128) hrd::unghr64_kernel<4, 2><<<grid, 128, 0, s>>>(A, n, lda, a_bs, tau, Z, ldz, z_bs);
  else if (n <= 256) hrd::unghr64_kernel<8, 2><<<grid, 128, 0, s>>>(A, n, lda, a_bs, tau, Z, ldz, z_bs);
  else hrd::unghr64_kernel<16, 1><<<grid, 128, 0, s>>>(A, n, lda, a_bs, tau, Z, ldz, z_bs);
  note_launch();
  const unsigned cx = (unsigned)min((long long)sms, ((long long)n * n + 255) / 256);
  clear_below_subdiag_kernel<double><<<dim3(cx, (unsigned)batch), 256, 0, s>>>(A, n, lda, a_bs); note_launch();
  return true;
}

// FP32: H in panels (ws: the panels' scratch), Q in panels
static void reduce_panels(cudaStream_t s, int batch, int n, Cx<float>* A, int lda, long long a_bs, Cx<float>* ws,
                          long long ws_bs, Cx<float>* tau, int th) {
  using C_ = Cx<float>;
  constexpr int BB = kHrdPanel, most = 200 * 1024;
  allow_shared(gehrd_panel_kernel, kVectorShared / 2);
  const long long nB = (long long)n * BB;
  C_ *V = ws, *Vc = ws + nB, *Y = ws + 2 * nB, *Wm = ws + 3 * nB, *Xm = ws + 4 * nB, *TH = ws + 5 * nB;
  const double2 one = make_double2(1.0, 0.0), mone = make_double2(-1.0, 0.0), zero = make_double2(0.0, 0.0);
  int ctas = 1;
  while (2 * ctas <= 8 && 2LL * ctas * batch <= sm_count()) ctas *= 2;
  const size_t spread = hrd_panel_shared(n, ctas), sm = 2 * (size_t)n * sizeof(C_);
  for (int k = 0; k + 2 < n; k += BB) {
    const int bb = min(BB, n - 2 - k);
    if (ctas > 1 && spread <= most) {
      launch_cluster(s, gehrd_panel_cluster_kernel, most, ctas, batch, kHrdClusterThreads, spread, A, n, lda, a_bs, tau, k, bb,
                     ws, ws_bs, th);
    } else {
      gehrd_panel_kernel<<<batch, th, sm, s>>>(A, n, lda, a_bs, tau, k, bb, ws, ws_bs); note_launch();
    }
    const int c0 = k + bb, m = n - c0, rows = n - k - 1;
    if (m <= 0) continue;
    C_* Ac = A + (long long)c0 * lda;
    // A[:, c0:] -= Y conj(V[c0:, :])^T
    gemm<float>(s, batch, n, m, bb, mone, Y, 1, n, ws_bs, Vc + c0, n, 1, ws_bs, one, Ac, 1, lda, a_bs);
    // W = V[k+1:, :]^H A[k+1:, c0:];  X = T^H W;  A[k+1:, c0:] -= V[k+1:, :] X
    gemm<float>(s, batch, bb, m, rows, one, Vc + (k + 1), n, 1, ws_bs, Ac + (k + 1), 1, lda, a_bs, zero, Wm, 1, BB, ws_bs);
    gemm<float>(s, batch, bb, m, bb, one, TH, 1, BB, ws_bs, Wm, 1, BB, ws_bs, zero, Xm, 1, BB, ws_bs);
    gemm<float>(s, batch, rows, m, bb, mone, V + (k + 1), 1, n, ws_bs, Xm, 1, BB, ws_bs, one, Ac + (k + 1), 1, lda, a_bs);
  }
}

static void form_panels(cudaStream_t s, int batch, int n, Cx<float>* A, int lda, long long a_bs, Cx<float>* Z, int ldz,
                        long long z_bs, const Cx<float>* tau, Cx<float>* ws, long long ws_bs, int th) {
  using C_ = Cx<float>;
  constexpr int BB = kHrdPanel;
  const long long nB = (long long)n * BB;
  C_ *V = ws, *Vc = ws + nB, *Wm = ws + 2 * nB, *Xm = ws + 3 * nB, *Tm = ws + 4 * nB;
  const double2 one = make_double2(1.0, 0.0), mone = make_double2(-1.0, 0.0), zero = make_double2(0.0, 0.0);
  set_identity<float>(s, batch, n, Z, ldz, z_bs);
  const int nk = n - 2;                                    // reflectors 0 .. n - 3
  for (int k0 = ((nk - 1) / BB) * BB; k0 >= 0; k0 -= BB) {
    const int bb = min(BB, nk - k0), rows = n - k0 - 1;
    unghr_panel_kernel<<<batch, th, 0, s>>>(A, n, lda, a_bs, tau, k0, bb, ws, ws_bs); note_launch();
    C_* Zb = Z + (k0 + 1) + (long long)(k0 + 1) * ldz;
    // W = V[k0+1:, :]^H Z_blk;  X = T W;  Z_blk -= V[k0+1:, :] X
    gemm<float>(s, batch, bb, rows, rows, one, Vc + (k0 + 1), n, 1, ws_bs, Zb, 1, ldz, z_bs, zero, Wm, 1, BB, ws_bs);
    gemm<float>(s, batch, bb, rows, bb, one, Tm, 1, BB, ws_bs, Wm, 1, BB, ws_bs, zero, Xm, 1, BB, ws_bs);
    gemm<float>(s, batch, rows, rows, bb, mone, V + (k0 + 1), 1, n, ws_bs, Xm, 1, BB, ws_bs, one, Zb, 1, ldz, z_bs);
  }
  const unsigned gx = (unsigned)min((long long)sm_count(), ((long long)n * n + 255) / 256);
  clear_below_subdiag_kernel<float><<<dim3(gx, batch), 256, 0, s>>>(A, n, lda, a_bs); note_launch();
}

template <class R>
void geev_schur(cudaStream_t s, int batch, int n, Cx<R>* A, int lda, long long a_bs, Cx<R>* Z, int ldz,
                long long z_bs, Cx<R>* w, Cx<R>* tau, int32_t* status, int st_div, Cx<R>* ws, long long ws_bs,
                const int* live) {
  if (batch <= 0 || n <= 0) return;
  size_t sm = 2 * (size_t)n * sizeof(Cx<R>);
  allow_shared(gehrd_kernel<R>, kVectorShared);
  allow_shared(unghr_kernel<R>, kVectorShared);
  const int th = hrd_threads(batch, n);
  bool hessenberg = false, formed = false;                 // H, Q
  if constexpr (std::is_same<R, double>::value)
    if (n > kQrSmall) hessenberg = formed = reduce64(s, batch, n, A, lda, a_bs, Z, ldz, z_bs, tau);
  // the FP32 form at n >= 192 reduces in panels (Z, not yet formed, holds the panels' scratch:
  // 5 n kHrdPanel + kHrdPanel^2 elements, within n * ldz from n = 161 on)
  if constexpr (std::is_same<R, float>::value)
    if (n >= 192 && ldz >= n && tuning(kTuneHrdBlocked) != 1) {
      reduce_panels(s, batch, n, A, lda, a_bs, Z, z_bs, tau, th);
      hessenberg = true;
      // Q in panels when the caller lends scratch (5 n kHrdPanel + kHrdPanel^2 elements a matrix)
      if (ws && ws_bs >= 5LL * n * kHrdPanel + kHrdPanel * kHrdPanel) {
        form_panels(s, batch, n, A, lda, a_bs, Z, ldz, z_bs, tau, ws, ws_bs, th);
        formed = true;
      }
    }
  if (!hessenberg) { gehrd_kernel<R><<<batch, th, sm, s>>>(A, n, lda, a_bs, tau, live); note_launch(); }
  if (!formed) { unghr_kernel<R><<<batch, th, sm, s>>>(A, n, lda, a_bs, tau, Z, ldz, z_bs, live); note_launch(); }
  int itmax = 30 * (n > 10 ? n : 10);
  const QrShape shape = qr_shape<R>(batch, n);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  bool timed = false;
  {
    std::lock_guard<std::mutex> lock(g_qrp_mutex);
    if (g_qrp.on && cudaEventCreate(&e0) == cudaSuccess && cudaEventCreate(&e1) == cudaSuccess) {
      timed = true;
      g_qrp.ev[QrSlot<R>::v].push_back({e0, e1});
    }
  }
  if (timed) cudaEventRecord(e0, s);
  bool launched = false;
  if constexpr (sizeof(R) > 4) {
    const QrSmall small = qr_small<R>(batch, n);
    if (small.threads) {
      auto kernel = hseqr_small_kernel<R, 256>;
      if constexpr (!std::is_same<R, double>::value)
        if (!small.wide) kernel = hseqr_small_kernel<R, 768>;
      allow_shared(kernel, kVectorShared / 2);
      kernel<<<batch, small.threads, (size_t)n * sizeof(Cx<R>), s>>>(A, n, lda, a_bs, Z, ldz, z_bs, w, status,
                                                                    st_div < 1 ? 1 : st_div, itmax, live);
      launched = true;
    }
  }
  if (launched) note_launch();
  else
    launch_cluster(s, hseqr_kernel<R>, kVectorShared, shape.ctas, batch, shape.threads, shape.smem, A, n, lda, a_bs, Z, ldz, z_bs, w,
                   status, st_div < 1 ? 1 : st_div, itmax);
  if (timed) cudaEventRecord(e1, s);
}

template <class R>
void trevc(cudaStream_t s, int batch, int n, const Cx<R>* T, int ldt, long long t_bs, Cx<R>* X, int ldx,
           long long x_bs, const int* live) {
  long long warps = (long long)batch * n;
  if (warps <= 0) return;
  trevc_kernel<R><<<(unsigned)((warps + 7) / 8), 256, 0, s>>>(T, n, ldt, t_bs, X, ldx, x_bs, batch, live); note_launch();
}

template <class R>
void normalize_columns(cudaStream_t s, int batch, int n, Cx<R>* W, int ldw, long long w_bs, const int* live) {
  long long warps = (long long)batch * n;
  if (warps <= 0) return;
  normalize_columns_kernel<R><<<(unsigned)((warps + 7) / 8), 256, 0, s>>>(W, n, ldw, w_bs, batch, live); note_launch();
}

// double2 wrappers of the plain FP64 path
void zgeev_schur(cudaStream_t s, int batch, int n, cplx* A, int lda, long long a_bs, cplx* Z, int ldz,
                 long long z_bs, cplx* w, cplx* tau, int32_t* status, int st_div) {
  geev_schur<double>(s, batch, n, (Cx<double>*)A, lda, a_bs, (Cx<double>*)Z, ldz, z_bs, (Cx<double>*)w,
                     (Cx<double>*)tau, status, st_div);
}
void ztrevc(cudaStream_t s, int batch, int n, const cplx* T, int ldt, long long t_bs, cplx* X, int ldx,
            long long x_bs) {
  trevc<double>(s, batch, n, (const Cx<double>*)T, ldt, t_bs, (Cx<double>*)X, ldx, x_bs);
}
void znormalize_columns(cudaStream_t s, int batch, int n, cplx* W, int ldw, long long w_bs) {
  normalize_columns<double>(s, batch, n, (Cx<double>*)W, ldw, w_bs);
}

#define WB_EIG_INST(R)                                                                                   \
  template void geev_schur<R>(cudaStream_t, int, int, Cx<R>*, int, long long, Cx<R>*, int, long long,     \
                              Cx<R>*, Cx<R>*, int32_t*, int, Cx<R>*, long long, const int*);              \
  template void trevc<R>(cudaStream_t, int, int, const Cx<R>*, int, long long, Cx<R>*, int, long long,   \
                         const int*);                                                                    \
  template void normalize_columns<R>(cudaStream_t, int, int, Cx<R>*, int, long long, const int*);
WB_EIG_INST(double)
WB_EIG_INST(float)
WB_EIG_INST(df64)

}  // namespace wb
