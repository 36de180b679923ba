// The panel, interchange and triangular-block kernels of the batched LU and its solves (wb_linalg.cu):
// everything that is not a product. FP64 instructions hold a scheduler for 64 cycles on GB300, so in
// FP64 each kernel spreads its elements over as many warps and CTAs as it can; in FP32 the chains'
// latency counts, and the order and rounding of every element's operations are fixed (the mixed
// form's answers move by up to 1e-7 of their size with the last bits of its FP32 factors).
#pragma once
#include <type_traits>
#include "wb_common.cuh"
#include "wb_num.cuh"

namespace wb {
namespace tri {

// a - l x. FP32: each product pair rounded once and fused once, V saying which product is the fused one
// (bit 0: real part, bit 1: imaginary part; 0: the first).
template <int V, class R> __device__ __forceinline__ Cx<R> sub_mul(Cx<R> a, Cx<R> l, Cx<R> x) { return a - l * x; }
template <int V> __device__ __forceinline__ Cx<float> sub_mul(Cx<float> a, Cx<float> l, Cx<float> x) {
  const float re = (V & 1) ? __fmaf_rn(-l.y, x.y, __fmul_rn(l.x, x.x)) : __fmaf_rn(l.x, x.x, -__fmul_rn(l.y, x.y));
  const float im = (V & 2) ? __fmaf_rn(l.y, x.x, __fmul_rn(l.x, x.y)) : __fmaf_rn(l.x, x.y, __fmul_rn(l.y, x.x));
  return cxmk<float>(__fsub_rn(a.x, re), __fsub_rn(a.y, im));
}
template <int V> __device__ __forceinline__ Cx<double> sub_mul(Cx<double> a, Cx<double> l, Cx<double> x) {
  return cxmk<double>(fma(-l.x, x.x, fma(l.y, x.y, a.x)), fma(-l.x, x.y, fma(-l.y, x.x, a.y)));
}
template <int V, class R> __device__ __forceinline__ Cx<R> mul(Cx<R> a, Cx<R> b) { return a * b; }
template <int V> __device__ __forceinline__ Cx<float> mul(Cx<float> a, Cx<float> b) {
  const float re = (V & 1) ? __fmaf_rn(-a.y, b.y, __fmul_rn(a.x, b.x)) : __fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y));
  const float im = (V & 2) ? __fmaf_rn(a.y, b.x, __fmul_rn(a.x, b.y)) : __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x));
  return cxmk<float>(re, im);
}
// a / b (Smith), every multiply-add fused
template <class R> __device__ __forceinline__ Cx<R> quotient(Cx<R> a, Cx<R> b) { return cxdiv(a, b); }
__device__ __forceinline__ Cx<float> quotient(Cx<float> a, Cx<float> b) {
  if (fabsf(b.y) <= fabsf(b.x)) {
    const float r = b.y / b.x, d = __fmaf_rn(b.y, r, b.x);
    return cxmk<float>(__fmaf_rn(a.y, r, a.x) / d, __fmaf_rn(-a.x, r, a.y) / d);
  }
  const float r = b.x / b.y, d = __fmaf_rn(b.x, r, b.y);
  return cxmk<float>(__fmaf_rn(a.x, r, a.y) / d, __fmaf_rn(a.y, r, -a.x) / d);
}

__device__ __forceinline__ float shf(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ double shf(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ df64 shf(df64 v, int src) {
  return df64(__shfl_sync(0xffffffffu, v.hi, src), __shfl_sync(0xffffffffu, v.lo, src));
}
template <class R> __device__ __forceinline__ Cx<R> shf(Cx<R> v, int src) { return cxmk<R>(shf(v.x, src), shf(v.y, src)); }

// which products are fused in FP32: an update's real part the first, its imaginary part the second; a
// multiplier's both the first
constexpr int kUpdate = 2, kScale = 0;

// ------------------------------------------------------------------------------------ LU panel
// Partial pivoting down a panel of kPB columns, by a cluster of C CTAs a matrix: the panel's rows in the
// CTAs' shared memory (column by column, `rows` each), `slices` threads a row. Per column: every CTA sends
// its largest |re| + |im| (first index on ties) with that row to the others, the owner of row j its row,
// and after one cluster barrier each picks the pivot, exchanges its rows, scales its multipliers and
// updates; the threads that update column j + 1 start its search. What they receive is buffered twice,
// so the next column's barrier is the only one.
//
// The magnitudes are compared as integers (an FP64 compare holds a scheduler for 64 cycles, as any FP64
// instruction; the search and its exchange took half of a column's 13000 cycles with them).
constexpr int kPB = 32;
constexpr int kPanelThreads = 512;
constexpr int kPanelMaxCluster = 8;

// Magnitudes in order: non-negative values' bits are; NaN and nothing below them all.
template <class R> struct Mag {
  R v;
  static __device__ __forceinline__ Mag none() { Mag m; m.v = R(-1.0); return m; }
  static __device__ __forceinline__ Mag of(R a) { Mag m; m.v = a >= R(0.0) ? a : R(-1.0); return m; }
  __device__ __forceinline__ bool operator>(const Mag& o) const { return v > o.v; }
  __device__ __forceinline__ bool operator==(const Mag& o) const { return v == o.v; }
  __device__ __forceinline__ Mag lane(int src) const { Mag m; m.v = shf(v, src); return m; }
};
template <> struct Mag<float> {
  int v;
  static __device__ __forceinline__ Mag none() { return {-1}; }
  static __device__ __forceinline__ Mag of(float a) { const int b = __float_as_int(a); return {b > 0x7f800000 ? -1 : b}; }
  __device__ __forceinline__ bool operator>(const Mag& o) const { return v > o.v; }
  __device__ __forceinline__ bool operator==(const Mag& o) const { return v == o.v; }
  __device__ __forceinline__ Mag lane(int src) const { return {__shfl_sync(0xffffffffu, v, src)}; }
};
template <> struct Mag<double> {
  long long v;
  static __device__ __forceinline__ Mag none() { return {-1}; }
  static __device__ __forceinline__ Mag of(double a) {
    const long long b = __double_as_longlong(a);
    return {b > 0x7ff0000000000000ll ? -1 : b};
  }
  __device__ __forceinline__ bool operator>(const Mag& o) const { return v > o.v; }
  __device__ __forceinline__ bool operator==(const Mag& o) const { return v == o.v; }
  __device__ __forceinline__ Mag lane(int src) const { return {__shfl_sync(0xffffffffu, v, src)}; }
};
template <class R> struct Pivot {
  Mag<R> m;
  int i;
  __device__ __forceinline__ void take(const Mag<R>& om, int oi) {
    if (om > m || (om == m && oi < i)) { m = om; i = oi; }
  }
  __device__ __forceinline__ void meet(int o, int lane) {
    const Mag<R> om = m.lane(lane ^ o);
    take(om, __shfl_xor_sync(0xffffffffu, i, o));
  }
};

// 1 / p: in FP64 r = conj(p) / |p|^2 to 21 bits, then r (1 + d + d^2) with d = 1 - p r (the geometric series
// of 1 / (1 - d); Smith's three divisions cost 1400 cycles of a column's chain). A quotient formed with it is off by
// 0.74 units of 2^-53 in the mean square, 2.9 at the most; by Smith's reciprocal 0.81 and 2.8, by his division 0.75 and
// 2.6, by conj(p) / |p|^2 rounded 1.33 and 5.6.
template <class R> __device__ __forceinline__ Cx<R> reciprocal(Cx<R> p) { return quotient(cxone<R>(), p); }
template <> __device__ __forceinline__ Cx<double> reciprocal(Cx<double> p) {
  const int e = max(__double2hiint(p.x) & 0x7fffffff, __double2hiint(p.y) & 0x7fffffff) >> 20;
  if ((unsigned)(e - (1023 - 400)) > 800u) return quotient(cxone<double>(), p);
  const double r = rsqrt_start(fma(p.x, p.x, p.y * p.y)), ir = r * r, x = p.x * ir, y = p.y * ir;
  const double d = fma(-p.x, x, fma(-p.y, y, 1.0)), f = fma(d, d, d);
  return cxmk<double>(fma(x, f, x), -fma(y, f, y));
}
template <class R> struct PanelShared {
  Mag<R> val[2][kPanelMaxCluster];         // the CTAs' candidates, their indices and rows
  int idx[2][kPanelMaxCluster];
  Cx<R> row[2][kPanelMaxCluster][kPB];
  Cx<R> jrow[2][kPB];                      // row j before the exchange
  Mag<R> wv[kPanelThreads / 32];
  int wi[kPanelThreads / 32];
  Cx<R> rp;
};

template <class T> __device__ __forceinline__ void put_remote(T* local, unsigned rank, const T& v) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(local);
  unsigned d;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(rank));
  const int* w = reinterpret_cast<const int*>(&v);
#pragma unroll
  for (int e = 0; e < (int)(sizeof(T) / 4); ++e)
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(d + 4 * e), "r"(w[e]) : "memory");
}
__device__ __forceinline__ void barrier_all(unsigned ctas) {
  if (ctas == 1) { __syncthreads(); return; }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <class R>
__global__ void __launch_bounds__(kPanelThreads) lu_panel_kernel(Cx<R>* __restrict__ Aall, int n, int lda, long long a_bs,
                                                                int* __restrict__ ipiv_all, long long piv_bs,
                                                                int32_t* __restrict__ status, int st_div, int k0, int kb,
                                                                int rows, int slices) {
  using C_ = Cx<R>;
  constexpr int kNone = 0x7fffffff;
  extern __shared__ __align__(16) unsigned char smraw[];
  C_* P = reinterpret_cast<C_*>(smraw);                       // (kb, rows), column by column
  __shared__ PanelShared<R> sh;
  unsigned rank, ctas;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ctas));
  const int mat = blockIdx.x / ctas;
  C_* A = Aall + mat * a_bs;
  int* ipiv = ipiv_all + (long long)mat * piv_bs;
  int32_t* st = status ? status + mat / st_div : nullptr;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
  const int g0 = k0 + (int)rank * rows, m = max(0, min(rows, n - g0));      // this CTA's rows g0 .. g0 + m - 1
  for (int c = warp; c < kb; c += nw)
    for (int r = lane; r < m; r += 32) P[c * rows + r] = A[g0 + r + (long long)(k0 + c) * lda];
  const int rstep = nt / slices, tr = tid % rstep, sl = tid / rstep;        // a thread's rows and its column slice
  barrier_all(ctas);                                          // (and every CTA of the cluster runs)
  Pivot<R> best = {Mag<R>::none(), kNone};
  if (sl == 0)
    for (int r = tr; r < m; r += rstep) best.take(Mag<R>::of(cxabs1(P[r])), g0 + r);
  for (int j = 0; j < kb; ++j) {
    const int gj = k0 + j, buf = j & 1;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) best.meet(o, lane);
    if (lane == 0) { sh.wv[warp] = best.m; sh.wi[warp] = best.i; }
    __syncthreads();
    const int jr = gj - g0;
    if (warp == 0) {
      best.m = lane < nw ? sh.wv[lane] : Mag<R>::none();
      best.i = lane < nw ? sh.wi[lane] : kNone;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) best.meet(o, lane);
      if (best.m == Mag<R>::none()) best.i = kNone;
      if (best.i != kNone && lane < kb) {
        const C_ v = P[lane * rows + best.i - g0];
        for (unsigned c = 0; c < ctas; ++c) put_remote(&sh.row[buf][rank][lane], c, v);
      }
      if (lane < (int)ctas) {
        put_remote(&sh.val[buf][rank], (unsigned)lane, best.m);
        put_remote(&sh.idx[buf][rank], (unsigned)lane, best.i);
      }
    }
    if (warp == 1 && jr >= 0 && jr < m && lane < kb) {
      const C_ v = P[lane * rows + jr];
      for (unsigned c = 0; c < ctas; ++c) put_remote(&sh.jrow[buf][lane], c, v);
    }
    barrier_all(ctas);
    const int cand = lane & ((int)ctas - 1);                  // (a power of two)
    Pivot<R> top = {sh.val[buf][cand], sh.idx[buf][cand]};
    for (int o = (int)ctas / 2; o > 0; o >>= 1) top.meet(o, lane);
    const int from = ctas == 1 ? 0 : (top.i - k0) / rows;     // the CTA with that row
    // no finite candidate (NaN): the row itself, as a search that finds nothing larger
    const bool found = top.i != kNone;
    const int p = found ? top.i : gj;
    const C_* prow = found ? sh.row[buf][from] : sh.jrow[buf];
    if (rank == 0 && tid == 0) ipiv[gj] = p;
    const C_ piv = prow[j];
    const bool zero = piv.x == R(0.0) && piv.y == R(0.0);
    const int pr = p - g0;
    if (p != gj) {
      if (warp == 0 && pr >= 0 && pr < m && lane < kb) P[lane * rows + pr] = sh.jrow[buf][lane];
      if (warp == 1 && jr >= 0 && jr < m && lane < kb) P[lane * rows + jr] = prow[lane];
    }
    if (zero && rank == 0 && tid == 0) wb_flag(st, WB_ST_SINGULAR);
    if (!zero && warp == nw - 1) {
      const C_ r = reciprocal(piv);
      if (lane == 0) sh.rp = r;
    }
    __syncthreads();
    if (!zero) {
      const C_ rp = sh.rp;
      for (int r = tid; r < m; r += nt)
        if (g0 + r > gj) P[j * rows + r] = mul<kScale>(P[j * rows + r], rp);
    }
    __syncthreads();
    best.m = Mag<R>::none(); best.i = kNone;
    for (int r = tr; r < m; r += rstep) {
      if (g0 + r <= gj) continue;
      const C_ l = P[j * rows + r];
      int c = j + 1 + sl;
      if (sl == 0 && c < kb) {                                // column j + 1, and its search
        C_ v = P[c * rows + r];
        if (!zero) {
          v = sub_mul<kUpdate>(v, l, prow[c]);
          P[c * rows + r] = v;
        }
        best.take(Mag<R>::of(cxabs1(v)), g0 + r);
        c += slices;
      }
      if (zero) continue;
#pragma unroll 4
      for (; c < kb; c += slices) P[c * rows + r] = sub_mul<kUpdate>(P[c * rows + r], l, prow[c]);
    }
  }
  __syncthreads();
  for (int c = warp; c < kb; c += nw)
    for (int r = lane; r < m; r += 32) A[g0 + r + (long long)(k0 + c) * lda] = P[c * rows + r];
}

// ------------------------------------------------------------- interchanges of a panel and U12
// Columns outside the panel [k0, k0 + kb): the panel's row swaps, and U12 = L11^-1 A12 for the trailing
// ones. The swaps are composed once a CTA into moves dest <- src (the kb block rows first, then the rows
// below that a swap touched); 8 threads a column carry them, thread g the block rows g, g + 8, ... in
// registers, and substitute with shuffles.
constexpr int kSwapThreads = 128;          // 16 columns

template <class R>
__global__ void __launch_bounds__(kSwapThreads) lu_swap_trsm_kernel(Cx<R>* __restrict__ Aall, int n, int lda,
                                                                   long long a_bs, const int* __restrict__ ipiv_all,
                                                                   long long piv_bs, int k0, int kb) {
  using C_ = Cx<R>;
  __shared__ C_ sL[kPB][kPB + 1];          // [column t][row r]
  __shared__ int s_dst[2 * kPB], s_src[2 * kPB], s_n;
  C_* A = Aall + blockIdx.y * a_bs;
  const int* ipiv = ipiv_all + (long long)blockIdx.y * piv_bs;
  const int tid = threadIdx.x, lane = tid & 31, g = lane & 7;
  for (int e = tid; e < kb * kb; e += kSwapThreads) {
    const int r = e % kb, t = e / kb;
    sL[t][r] = A[k0 + r + (long long)(k0 + t) * lda];
  }
  if (tid < 32) {
    // lane j: swap j's row; the rows' contents are followed through the swaps in order
    const int pj = lane < kb ? ipiv[k0 + lane] : -1;
    int src = k0 + lane, below = -1, bsrc = -1;               // block row lane; a row below first met at swap lane
    for (int j = 0; j < kb; ++j) {
      const int p = __shfl_sync(0xffffffffu, pj, j);
      if (p < k0 + kb) {                                      // both in the block
        const int a = __shfl_sync(0xffffffffu, src, j), b = __shfl_sync(0xffffffffu, src, p - k0);
        if (lane == j) src = b;
        if (lane == p - k0) src = a;
      } else {
        const unsigned have = __ballot_sync(0xffffffffu, below == p);
        const int a = __shfl_sync(0xffffffffu, src, j);
        if (have) {
          const int o = __ffs(have) - 1, b = __shfl_sync(0xffffffffu, bsrc, o);
          if (lane == j) src = b;
          if (lane == o) bsrc = a;
        } else if (lane == j) {
          src = p;
          below = p; bsrc = a;
        }
      }
    }
    const unsigned m = __ballot_sync(0xffffffffu, below >= 0);
    if (lane < kb) { s_dst[lane] = k0 + lane; s_src[lane] = src; }
    if (below >= 0) {
      const int at = kb + __popc(m & ((1u << lane) - 1u));
      s_dst[at] = below; s_src[at] = bsrc;
    }
    if (lane == 0) s_n = kb + __popc(m);
  }
  __syncthreads();
  int c = (blockIdx.x * kSwapThreads + tid) >> 3;
  const bool live = c < n - kb;
  if (c >= k0) c += kb;                                       // skip the panel
  C_* col = A + (long long)(live ? c : 0) * lda;
  const int nd = s_n;
  C_ x[4], y[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int j = g + 8 * q, e = kb + g + 8 * q;
    x[q] = (live && j < kb) ? col[s_src[j]] : cxzero<R>();
    y[q] = (live && e < nd) ? col[s_src[e]] : cxzero<R>();
  }
  __syncwarp();                                               // every source read before a destination is written
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (live && kb + g + 8 * q < nd) col[s_dst[kb + g + 8 * q]] = y[q];
  const bool solve = live && c >= k0;
  const unsigned any = __ballot_sync(0xffffffffu, solve);
  if (any) {
    const int first = lane & ~7;
#pragma unroll
    for (int qt = 0; qt < 4; ++qt)
      for (int gt = 0; gt < 8; ++gt) {
        const int t = 8 * qt + gt;
        if (t >= kb) break;
        const C_ xt = shf(x[qt], first + gt);
#pragma unroll
        for (int q = qt; q < 4; ++q) {
          const int r = g + 8 * q;
          if (solve && r > t && r < kb) x[q] = sub_mul<kUpdate>(x[q], sL[t][r], xt);
        }
      }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (live && g + 8 * q < kb) col[k0 + g + 8 * q] = x[q];
}

// ------------------------------------------------------------------------ all row interchanges
// B's rows in the order of the interchanges (forward) or of their inverse: composed once a CTA in shared
// memory, then each column gathered through a copy of it there.
template <class R>
__global__ void __launch_bounds__(256) laswp_kernel(Cx<R>* __restrict__ Ball, int n, int nrhs, int ldb, long long b_bs,
                                                    const int* __restrict__ ipiv_all, long long piv_bs, int forward,
                                                    int cols) {
  extern __shared__ __align__(16) unsigned char smraw[];
  Cx<R>* buf = reinterpret_cast<Cx<R>*>(smraw);               // a column
  int* perm = reinterpret_cast<int*>(buf + n);
  int* piv = perm + n;
  const int* ipiv = ipiv_all + (long long)blockIdx.y * piv_bs;
  Cx<R>* B = Ball + blockIdx.y * b_bs;
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int i = tid; i < n; i += nt) { perm[i] = i; piv[i] = ipiv[i]; }
  __syncthreads();
  if (tid == 0) {
    for (int s = 0; s < n; ++s) {
      const int j = forward ? s : n - 1 - s, p = piv[j];
      const int a = perm[j], b = perm[p];
      perm[j] = b; perm[p] = a;
    }
  }
  __syncthreads();
  const int c1 = min(nrhs, (int)(blockIdx.x + 1) * cols);
  for (int c = blockIdx.x * cols; c < c1; ++c) {
    Cx<R>* col = B + (long long)c * ldb;
    for (int i = tid; i < n; i += nt) buf[i] = col[i];
    __syncthreads();
    for (int i = tid; i < n; i += nt)
      if (perm[i] != i) col[i] = buf[perm[i]];
    __syncthreads();
  }
}

// ------------------------------------------------------------------- a diagonal block's solve
// op(A)'s diagonal block [i0, i0 + ib) (ib <= 64) against 128 / T columns a CTA: T threads a column, thread
// g its rows g, g + T, ... in registers; a solved row goes to the others by shuffles and is taken off
// theirs at once (right-looking; the operations on an element and their order do not depend on T).
// In FP64 a warp's work is FP64 issue, 1152 (T = 8), 640 (16) or 384 (32) instructions of 64 cycles for
// 32 / T columns: the host takes the T whose rounds over the GPU's schedulers cost least.
constexpr int kTB = 64;
constexpr int kTriThreads = 128;

template <class R, int T>
__global__ void __launch_bounds__(kTriThreads) trsm_diag_kernel(const Cx<R>* __restrict__ LUall, int lda, long long a_bs,
                                                               Cx<R>* __restrict__ Ball, int nrhs, int ldb,
                                                               long long b_bs, int i0, int ib, int lower, int unit,
                                                               int trans) {
  using C_ = Cx<R>;
  constexpr int Q = kTB / T;
  extern __shared__ __align__(16) unsigned char smraw[];
  C_* sT = reinterpret_cast<C_*>(smraw);                      // [t][r], ld kTB + 1: element (r, t) of op(A)
  __shared__ C_ sD[kTB];                                      // reciprocal diagonal (FP64), diagonal (others)
  const C_* LU = LUall + blockIdx.y * a_bs;
  C_* B = Ball + blockIdx.y * b_bs;
  const int tid = threadIdx.x, lane = tid & 31, g = lane % T, first = lane - g;
  const int c = (blockIdx.x * kTriThreads + tid) / T;
  const bool live = c < nrhs;
  C_* col = B + i0 + (long long)(live ? c : 0) * ldb;
  C_ x[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) x[q] = (live && g + T * q < ib) ? col[g + T * q] : cxzero<R>();
#pragma unroll
  for (int b0 = 0; b0 < kTB; b0 += 16) {                      // a warp four columns of LU, eight loads in flight
    C_ v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int a = lane + 32 * (u & 1), b = b0 + (tid >> 5) + 4 * (u >> 1);
      if (a < ib && b < ib) v[u] = LU[i0 + a + (long long)(i0 + b) * lda];
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int a = lane + 32 * (u & 1), b = b0 + (tid >> 5) + 4 * (u >> 1);
      if (a < ib && b < ib) sT[trans ? a * (kTB + 1) + b : b * (kTB + 1) + a] = v[u];   // op(A)(b, a) or (a, b)
    }
  }
  __syncthreads();
  if (tid < ib && !unit) {
    const C_ d = sT[tid * (kTB + 1) + tid];
    sD[tid] = std::is_same<R, double>::value ? reciprocal(d) : d;
  }
  __syncthreads();
  constexpr bool kInv = std::is_same<R, double>::value;
  if (lower) {
#pragma unroll
    for (int qt = 0; qt < Q; ++qt)
#pragma unroll 1
      for (int gt = 0; gt < T; ++gt) {
        const int t = T * qt + gt;
        if (t >= ib) break;
        if (!unit) {
          const C_ v = kInv ? x[qt] * sD[t] : quotient(x[qt], sD[t]);
          if (g == gt) x[qt] = v;
        }
        const C_ xt = shf(x[qt], first + gt);
        const C_* l = sT + t * (kTB + 1) + g;
        if (g > gt) x[qt] = sub_mul<kUpdate>(x[qt], l[T * qt], xt);
#pragma unroll
        for (int q = qt + 1; q < Q; ++q) x[q] = sub_mul<kUpdate>(x[q], l[T * q], xt);
      }
  } else {
#pragma unroll
    for (int qt = Q - 1; qt >= 0; --qt)
#pragma unroll 1
      for (int gt = T - 1; gt >= 0; --gt) {
        const int t = T * qt + gt;
        if (t >= ib) continue;
        if (!unit) {
          const C_ v = kInv ? x[qt] * sD[t] : quotient(x[qt], sD[t]);
          if (g == gt) x[qt] = v;
        }
        const C_ xt = shf(x[qt], first + gt);
        const C_* l = sT + t * (kTB + 1) + g;
        if (g < gt) x[qt] = sub_mul<kUpdate>(x[qt], l[T * qt], xt);
#pragma unroll
        for (int q = 0; q < qt; ++q) x[q] = sub_mul<kUpdate>(x[q], l[T * q], xt);
      }
  }
#pragma unroll
  for (int q = 0; q < Q; ++q)
    if (live && g + T * q < ib) col[g + T * q] = x[q];
}

// The upper solve in FP32: the row's sum runs over the later unknowns in ascending order, so its first
// term is the one solved last and each row is one chain. One thread a column; the block's unknowns stay in
// the thread's column of shared memory but for the last one, so that no load is on the chain.
__global__ void __launch_bounds__(32) trsm_upper_f32_kernel(const Cx<float>* __restrict__ LUall, int lda, long long a_bs,
                                                           Cx<float>* __restrict__ Ball, int nrhs, int ldb,
                                                           long long b_bs, int i0, int ib, int unit, int trans) {
  using C_ = Cx<float>;
  extern __shared__ __align__(16) unsigned char smraw[];
  C_* sT = reinterpret_cast<C_*>(smraw);                      // [r][t], ld kTB + 1
  C_* sX = sT + kTB * (kTB + 1);                              // [column][r], ld kTB + 1
  const C_* LU = LUall + blockIdx.y * a_bs;
  C_* B = Ball + blockIdx.y * b_bs;
  const int lane = threadIdx.x, c0 = blockIdx.x * 32, w = min(32, nrhs - c0);
#pragma unroll 8
  for (int b = 0; b < ib; ++b)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int a = lane + 32 * u;
      if (a < ib) sT[trans ? b * (kTB + 1) + a : a * (kTB + 1) + b] = LU[i0 + a + (long long)(i0 + b) * lda];
    }
#pragma unroll 8
  for (int c = 0; c < w; ++c)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = lane + 32 * u;
      if (r < ib) sX[c * (kTB + 1) + r] = B[i0 + r + (long long)(c0 + c) * ldb];
    }
  __syncwarp();
  if (lane < w) {
    C_* mine = sX + lane * (kTB + 1);
    C_ last = cxzero<float>();
    for (int r = ib - 1; r >= 0; --r) {
      const C_* l = sT + r * (kTB + 1);
      C_ acc = mine[r];
      if (r + 1 < ib) acc = sub_mul<kUpdate>(acc, l[r + 1], last);
#pragma unroll 8
      for (int t = r + 2; t < ib; ++t) acc = sub_mul<kUpdate>(acc, l[t], mine[t]);
      if (!unit) acc = quotient(acc, l[r]);
      last = acc;
      mine[r] = acc;
    }
  }
  __syncwarp();
  for (int c = 0; c < w; ++c)
    for (int r = lane; r < ib; r += 32) B[i0 + r + (long long)(c0 + c) * ldb] = sX[c * (kTB + 1) + r];
}

// ------------------------------------------------------------------- few right-hand sides
// A X = B for NC <= 6 columns by a cluster of C CTAs a matrix. X (n x NC) is in every CTA's shared memory;
// rows are taken 32 at a time, block b by CTA b % C. Per block: its owner solves the diagonal block, one
// warp a column (the rows in its lanes), and sends the solution to every CTA; then each CTA takes the
// block's part off its own blocks still to solve, a warp 32 rows (in FP64 one column of them), with the
// loads of a row's 32 elements in flight together, while the next diagonal block comes in.
constexpr int kNarrowThreads = 512;

// x / d with what depends on d alone formed ahead (Smith)
template <class R> struct Divisor {
  R r, d;
  bool swap;
  __device__ __forceinline__ void set(Cx<R> b) {
    swap = !(rabs(b.y) <= rabs(b.x));
    r = swap ? b.x / b.y : b.y / b.x;
    d = swap ? rfma(b.x, r, b.y) : rfma(b.y, r, b.x);
  }
  __device__ __forceinline__ Cx<R> of(Cx<R> a) const {
    if (!swap) return cxmk<R>(rfma(a.y, r, a.x) / d, rfma(-a.x, r, a.y) / d);
    return cxmk<R>(rfma(a.x, r, a.y) / d, rfma(a.y, r, -a.x) / d);
  }
};
template <> struct Divisor<double> {       // FP64: times the reciprocal (a division is 7 multiply-adds)
  Cx<double> r;
  __device__ __forceinline__ void set(Cx<double> b) { r = cxinv(b); }
  __device__ __forceinline__ Cx<double> of(Cx<double> a) const { return a * r; }
};
template <> struct Divisor<df64> {
  Cx<df64> b;
  __device__ __forceinline__ void set(Cx<df64> v) { b = v; }
  __device__ __forceinline__ Cx<df64> of(Cx<df64> a) const { return cxdiv(a, b); }
};

template <class R, int NC>
__global__ void __launch_bounds__(kNarrowThreads) getrs_narrow_kernel(const Cx<R>* __restrict__ LUall, int n, int lda,
                                                                     long long a_bs, const int* __restrict__ ipiv_all,
                                                                     long long piv_bs, Cx<R>* __restrict__ Ball,
                                                                     int nrhs, int ldb, long long b_bs) {
  using C_ = Cx<R>;
  constexpr int NB = 32, CG = std::is_same<R, double>::value ? 1 : NC, G = NC / CG, U = sizeof(R) == 4 ? 32 : 16;
  extern __shared__ __align__(16) unsigned char smraw[];
  C_* X = reinterpret_cast<C_*>(smraw);                       // [column][row]
  unsigned short* perm = reinterpret_cast<unsigned short*>(X + (size_t)n * NC);
  int* piv = reinterpret_cast<int*>(X);                       // until the fill
  __shared__ C_ sD[NB][NB + 1];                               // [t][r]
  unsigned rank, ctas;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ctas));
  const int mat = blockIdx.x / ctas;
  const C_* LU = LUall + mat * a_bs;
  const int* ipiv = ipiv_all + (long long)mat * piv_bs;
  C_* B = Ball + mat * b_bs;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = blockDim.x, nw = nt >> 5;
  for (int i = tid; i < n; i += nt) { perm[i] = (unsigned short)i; piv[i] = ipiv[i]; }
  __syncthreads();
  if (tid == 0)
    for (int j = 0; j < n; ++j) {
      const int p = piv[j];
      const unsigned short a = perm[j], b = perm[p];
      perm[j] = b; perm[p] = a;
    }
  __syncthreads();
  for (int e = tid; e < n * NC; e += nt) {
    const int r = e % n, c = e / n;
    X[e] = (c < nrhs) ? B[perm[r] + (long long)c * ldb] : cxzero<R>();
  }
  barrier_all(ctas);                                          // every copy of X is filled before a solution is sent to it
  const int nblk = (n + NB - 1) / NB;
  for (int sweep = 0; sweep < 2; ++sweep) {
    const bool fwd = sweep == 0;                              // L (unit lower), then U (upper)
    auto begin = [&](int b) { return fwd ? b * NB : max(0, n - (b + 1) * NB); };
    auto size = [&](int b) { return fwd ? min(NB, n - b * NB) : (n - b * NB) - begin(b); };
    auto bring = [&](int b) {                                 // block b's diagonal (its owner)
      const int i0 = begin(b), ib = size(b);
      for (int e = tid; e < NB * NB; e += nt) {
        const int r = e % NB, t = e / NB;
        sD[t][r] = (r < ib && t < ib) ? LU[i0 + r + (long long)(i0 + t) * lda] : cxzero<R>();
      }
    };
    if (rank == 0) bring(0);
    __syncthreads();
    for (int b = 0; b < nblk; ++b) {
      const int i0 = begin(b), ib = size(b);
      if (rank == (unsigned)(b % (int)ctas) && warp < NC) {
        C_* xc = X + (size_t)warp * n + i0;
        C_ x = lane < ib ? xc[lane] : cxzero<R>();
        if (fwd) {
          for (int t = 0; t < ib; ++t) {
            const C_ l = sD[t][lane], xt = shf(x, t);
            if (lane > t) x = sub_mul<kUpdate>(x, l, xt);
          }
        } else {
          Divisor<R> dv;
          dv.set(lane < ib ? sD[lane][lane] : cxone<R>());
          for (int t = ib - 1; t >= 0; --t) {
            const C_ u = sD[t][lane];
            if (lane == t) x = dv.of(x);
            __syncwarp();
            const C_ xt = shf(x, t);
            if (lane < t) x = sub_mul<kUpdate>(x, u, xt);
          }
        }
        if (lane < ib) {
          if (ctas == 1) xc[lane] = x;
          else
            for (unsigned c = 0; c < ctas; ++c) put_remote(&xc[lane], c, x);
        }
      }
      barrier_all(ctas);
      // the block's part of the blocks still to solve (CTA k's: k, k + C, ...)
      const int nb = b + 1;
      if (nb < nblk && rank == (unsigned)(nb % (int)ctas)) bring(nb);
      const int first = nb + (int)((rank + ctas - (unsigned)(nb % (int)ctas)) % ctas);
      const int mine = first < nblk ? (nblk - first + (int)ctas - 1) / (int)ctas : 0;
      for (int q = warp; q < mine * G; q += nw) {
        const int rb = first + (q / G) * (int)ctas, cg = (q % G) * CG;
        const int r0 = begin(rb), rn = size(rb);
        if (lane < rn) {
          const C_* li = LU + r0 + lane + (long long)i0 * lda;
          C_ acc[CG];
#pragma unroll
          for (int c = 0; c < CG; ++c) acc[c] = X[(size_t)(cg + c) * n + r0 + lane];
#pragma unroll 1
          for (int t0 = 0; t0 < ib; t0 += U) {
            C_ l[U];
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (t0 + u < ib) l[u] = li[(long long)(t0 + u) * lda];
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (t0 + u < ib) {
#pragma unroll
                for (int c = 0; c < CG; ++c)
                  acc[c] = sub_mul<kUpdate>(acc[c], l[u], X[(size_t)(cg + c) * n + i0 + t0 + u]);
              }
          }
#pragma unroll
          for (int c = 0; c < CG; ++c) X[(size_t)(cg + c) * n + r0 + lane] = acc[c];
        }
      }
      __syncthreads();
    }
    barrier_all(ctas);
  }
  if (rank == 0)
    for (int e = tid; e < n * nrhs; e += nt) B[e % n + (long long)(e / n) * ldb] = X[e];
}

}  // namespace tri
}  // namespace wb
