// Schur form of a complex Hessenberg matrix by shifted QR (Francis single-shift sweeps), the
// Schur vectors accumulated into Z: T in H. The subdiagonal is kept real so that every 2-element
// reflector has a real second coefficient. Deflation uses the standard small-subdiagonal test
// with the Ahues-Tisseur refinement; shifts are Wilkinson shifts with exceptional shifts after
// 10 and 20 stalled iterations.
//
// A sweep over the active block [l, i] is a chain of reflectors k = l .. i-1, reflector k acting
// on rows and columns (k, k+1); each is built from elements the previous ones have just changed,
// so the chain is serial (a square root and three divisions deep). Everything else a reflector
// touches -- rows k, k+1 of the columns to the right, columns k, k+1 of the rows above, Z -- only
// has to see the reflectors in order. The chain is therefore cut into windows of QrWin<R>::m
// reflectors [k0, k1):
//   chase   one warp runs the window's reflectors. In FP32 every lane carries the 2 x 2 core and the
//           reflector (no hand-over, no barrier); lane j also carries column k0 + 2 + j of the
//           window down its rows, and the element it finishes joins the core by a shuffle. In FP64
//           four lanes share a pair (chase64_step). The window's columns sit in shared memory (the tile).
//   far     the other warps apply the window before: one thread a row (of Z, and of H above the
//           window) carries its element through the window's columns; one thread a column to the
//           right carries it down the window's rows, through a 32-column tile in shared memory.
// One barrier a window separates them, so the chase of window w + 1 overlaps the far updates of
// window w. The columns that window w + 1 chases get window w's reflectors from the chasing warp
// itself (the near columns). Each element sees exactly the operations of the element-by-element
// sweep in the same order, so the result does not depend on the window, the threads or the CTAs.
//
// A matrix is worked on by a cluster of C CTAs (qr_shape): its far updates are spread over their
// warps, the reflectors and the window's record are written to every CTA's shared memory, and the
// barrier is the cluster's.
//
// The chase holds 74..220 registers a thread and has to have them: spilled, a reflector takes three
// times as long. So every role is a function of its own, its state kept in shared memory between
// windows, and a CTA has at most 512 (FP32) or 256 threads.
//
// What bounds it: the chase's latency. In FP32 a reflector (a square root and three reciprocals, two of
// them at once) and the core's update take 670 cycles a step, 900 with the windows' and sweeps' starts,
// against 2400..4500 for one barrier a reflector over the whole CTA; in FP64, where an instruction holds a
// scheduler for 64 cycles whatever its active lanes, 2140 and 2500 against 11000..19000 (some 16 FP64
// instructions a step, each handing over to shuffles). Measured on a GB300 (one layer matrix an SM or
// fewer): the sweep of 2 matrices of 798 in FP32 some 760 -> 215 ms, of 32 of 242 in FP64 446 -> 95 ms; at
// n = 1250 and one matrix per SM the far updates' memory traffic (2 (2n - 2) complex values a reflector)
// is next.
#pragma once
#include <type_traits>
#include "wb_common.cuh"
#include "wb_num.cuh"

namespace wb {

// The sweep's operations. In FP32 every multiply-add is written out (which product is rounded first
// and which is fused), so that a result depends neither on how the compiler contracts an expression
// in one place or another nor on which warp applies a reflector: the mixed form's answers move by up
// to 1e-7 of their size when the FP32 Schur form's last bits do.
namespace qr {
template <class R> __device__ __forceinline__ Cx<R> scaled_column(Cx<R> sc, Cx<R> a) { return sc * a; }
template <class R> __device__ __forceinline__ Cx<R> product(Cx<R> a, Cx<R> b) { return a * b; }
template <class R> __device__ __forceinline__ Cx<R> scaled_row(Cx<R> sc, Cx<R> a) { return cxconj(sc) * a; }
template <class R> __device__ __forceinline__ R sum_squares(R a, R b, R c) { return a * a + b * b + c * c; }
template <class R> __device__ __forceinline__ R sum_squares2(R a, R b) { return a * a + b * b; }
template <class R> __device__ __forceinline__ R modulus(Cx<R> a) { return cxabs(a); }
template <class R> __device__ __forceinline__ R plain_sub(R a, R b) { return a - b; }
template <class R> __device__ __forceinline__ R plain_mul(R a, R b) { return a * b; }

__device__ __forceinline__ float fma2(float a, float b, float c, float d) { return __fmaf_rn(a, b, __fmul_rn(c, d)); }
__device__ __forceinline__ Cx<float> left_sum(Cx<float> t, Cx<float> a, Cx<float> b, float t2) {
  return cxmk<float>(__fmaf_rn(b.x, t2, fma2(t.x, a.x, -t.y, a.y)), __fmaf_rn(b.y, t2, fma2(t.x, a.y, t.y, a.x)));
}
__device__ __forceinline__ Cx<float> right_sum(Cx<float> t, Cx<float> a, Cx<float> b, float t2) {
  return cxmk<float>(__fmaf_rn(b.x, t2, fma2(t.x, a.x, -t.y, a.y)), __fmaf_rn(b.y, t2, fma2(t.y, a.x, t.x, a.y)));
}
__device__ __forceinline__ Cx<float> left_sub(Cx<float> n, Cx<float> s, Cx<float> w) {
  return cxmk<float>(__fsub_rn(n.x, fma2(s.x, w.x, -s.y, w.y)), __fsub_rn(n.y, fma2(s.x, w.y, s.y, w.x)));
}
__device__ __forceinline__ Cx<float> right_sub(Cx<float> n, Cx<float> s, Cx<float> w) {
  return cxmk<float>(__fsub_rn(n.x, fma2(s.x, w.x, -s.y, w.y)), __fsub_rn(n.y, fma2(s.y, w.x, s.x, w.y)));
}

// (a, b) <- the reflector's left application to rows (k, k + 1) of a column, or its right one to
// columns (k, k + 1) of a row.
// FP32 and double-float: H = I - t1 (1; v2)(1; v2)^H with t1 v2 = t2 real.
template <class R> __device__ __forceinline__ void left_pair(Cx<R> t1, Cx<R> v2, R t2, Cx<R>& a, Cx<R>& b) {
  const Cx<R> sum = cxconj(t1) * a + b * t2;
  a = a - sum; b = b - sum * v2;
}
template <class R> __device__ __forceinline__ void right_pair(Cx<R> t1, Cx<R> v2, R t2, Cx<R>& a, Cx<R>& b) {
  const Cx<R> sum = t1 * a + b * t2;
  a = a - sum; b = b - sum * cxconj(v2);
}
__device__ __forceinline__ void left_pair(Cx<float> t1, Cx<float> v2, float t2, Cx<float>& a, Cx<float>& b) {
  const Cx<float> sum = left_sum(cxconj(t1), a, b, t2);
  a = a - sum; b = left_sub(b, sum, v2);
}
__device__ __forceinline__ void right_pair(Cx<float> t1, Cx<float> v2, float t2, Cx<float>& a, Cx<float>& b) {
  const Cx<float> sum = right_sum(t1, a, b, t2);
  a = a - sum; b = right_sub(b, sum, cxconj(v2));
}
// FP64: the rotation G = [[conj(c), s], [-s, c]] with c = t1, s = t2 real: 12 operations instead of
// 14, and no division to form it (chase64_step, chase_reflector). An FP64 instruction holds a scheduler for 64
// cycles on GB300, so their number is the cost.
__device__ __forceinline__ void left_pair(Cx<double> c, Cx<double>, double s, Cx<double>& a, Cx<double>& b) {
  const Cx<double> p = a, q = b;
  a.x = fma(c.x, p.x, fma(c.y, p.y, s * q.x));
  a.y = fma(c.x, p.y, fma(-c.y, p.x, s * q.y));
  b.x = fma(c.x, q.x, fma(-c.y, q.y, -s * p.x));
  b.y = fma(c.x, q.y, fma(c.y, q.x, -s * p.y));
}
__device__ __forceinline__ void right_pair(Cx<double> c, Cx<double>, double s, Cx<double>& a, Cx<double>& b) {
  const Cx<double> p = a, q = b;
  a.x = fma(c.x, p.x, fma(-c.y, p.y, s * q.x));
  a.y = fma(c.x, p.y, fma(c.y, p.x, s * q.y));
  b.x = fma(c.x, q.x, fma(c.y, q.y, -s * p.x));
  b.y = fma(c.x, q.y, fma(-c.y, q.x, -s * p.y));
}
__device__ __forceinline__ Cx<float> scaled_column(Cx<float> a, Cx<float> b) {
  return cxmk<float>(fma2(a.x, b.x, -a.y, b.y), fma2(a.y, b.x, a.x, b.y));
}
__device__ __forceinline__ Cx<float> product(Cx<float> a, Cx<float> b) {
  return cxmk<float>(fma2(a.x, b.x, -a.y, b.y), fma2(a.x, b.y, a.y, b.x));
}
__device__ __forceinline__ Cx<float> scaled_row(Cx<float> a, Cx<float> b) {
  return cxmk<float>(fma2(a.x, b.x, a.y, b.y), fma2(a.x, b.y, -a.y, b.x));
}
__device__ __forceinline__ float sum_squares(float a, float b, float c) { return __fmaf_rn(c, c, fma2(a, a, b, b)); }
__device__ __forceinline__ float sum_squares2(float a, float b) { return fma2(b, b, a, a); }
__device__ __forceinline__ float plain_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float plain_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float modulus(Cx<float> a) {
  const float ax = fabsf(a.x), ay = fabsf(a.y), m = fmaxf(ax, ay);
  if (!(m > RealT<float>::tiny())) return m;
  const float s = 1.0f / m, u = __fmul_rn(ax, s), v = __fmul_rn(ay, s);
  return __fmul_rn(m, sqrtf(fma2(u, u, v, v)));
}

// Wilkinson shift of the block's last 2 x 2: the eigenvalue of [[p, u1], [u2, t]] closer to t
template <class R> __device__ __forceinline__ Cx<R> wilkinson(Cx<R> p, Cx<R> u1, Cx<R> u2, Cx<R> t) {
  using C_ = Cx<R>;
  const C_ u = cxsqrt(u1) * cxsqrt(u2);
  R sx = cxabs1(u);
  if (sx == R(0.0)) return t;
  const C_ x = (p - t) * R(0.5);
  const R sxx = cxabs1(x);
  sx = rmax(sx, cxabs1(x));
  const C_ xs = x * (R(1.0) / sx), us = u * (R(1.0) / sx);
  C_ y = cxsqrt(xs * xs + us * us) * sx;
  if (sxx > R(0.0)) {
    const C_ xn = x * (R(1.0) / sxx);
    if (xn.x * y.x + xn.y * y.y < R(0.0)) y = -y;
  }
  return t - u * cxdiv(u, x + y);
}
__device__ __forceinline__ Cx<float> root(Cx<float> z) {      // principal square root
  if (z.x == 0.f && z.y == 0.f) return cxmk<float>(0.f, z.y);
  const float t = sqrtf(__fmul_rn(0.5f, __fadd_rn(fabsf(z.x), modulus(z))));
  if (!(t > 0.f)) return cxmk<float>(0.f, 0.f);
  const float t2 = __fmul_rn(2.f, t);
  if (z.x >= 0.f) return cxmk<float>(t, z.y / t2);
  return cxmk<float>(fabsf(z.y) / t2, z.y < 0.f ? -t : t);
}
__device__ __forceinline__ Cx<float> wilkinson(Cx<float> p, Cx<float> u1, Cx<float> u2, Cx<float> t) {
  const Cx<float> r1 = root(u1), r2 = root(u2);
  const Cx<float> u = cxmk<float>(fma2(r1.x, r2.x, -r1.y, r2.y), fma2(r1.x, r2.y, r1.y, r2.x));
  float sx = cxabs1(u);
  if (sx == 0.f) return t;
  const Cx<float> x = cxmk<float>(__fmul_rn(__fsub_rn(p.x, t.x), 0.5f), __fmul_rn(__fsub_rn(p.y, t.y), 0.5f));
  const float sxx = cxabs1(x);
  sx = fmaxf(sx, sxx);
  const float is = 1.0f / sx;
  const Cx<float> xs = cxmk<float>(__fmul_rn(x.x, is), __fmul_rn(x.y, is)), us = cxmk<float>(__fmul_rn(u.x, is), __fmul_rn(u.y, is));
  Cx<float> y = root(cxmk<float>(__fadd_rn(fma2(xs.x, xs.x, -xs.y, xs.y), fma2(us.x, us.x, -us.y, us.y)),
                                 __fadd_rn(fma2(xs.x, xs.y, xs.y, xs.x), fma2(us.x, us.y, us.y, us.x))));
  y = cxmk<float>(__fmul_rn(y.x, sx), __fmul_rn(y.y, sx));
  if (sxx > 0.f) {
    const float ix = 1.0f / sxx;
    if (fma2(__fmul_rn(x.x, ix), y.x, __fmul_rn(x.y, ix), y.y) < 0.f) y = -y;
  }
  const Cx<float> b = cxmk<float>(__fadd_rn(x.x, y.x), __fadd_rn(x.y, y.y));
  Cx<float> q;                                                // u / b
  if (fabsf(b.y) <= fabsf(b.x)) {
    const float r = b.y / b.x, d = __fmaf_rn(b.y, r, b.x);
    q = cxmk<float>(__fmaf_rn(u.y, r, u.x) / d, __fmaf_rn(-u.x, r, u.y) / d);
  } else {
    const float r = b.x / b.y, d = __fmaf_rn(b.x, r, b.y);
    q = cxmk<float>(__fmaf_rn(u.x, r, u.y) / d, __fmaf_rn(u.y, r, -u.x) / d);
  }
  return left_sub(t, u, q);
}
// The same eigenvalue in FP64: t - u1 u2 / (x + y), y^2 = x^2 + u1 u2, x = (p - t) / 2. In FP64 a division
// or a root costs 7 to 10 multiply-adds of 64 cycles; these are three of the reciprocal roots above. Entries
// out of 2^+-200 go the scaled way.
__device__ __forceinline__ Cx<double> wilkinson(Cx<double> p, Cx<double> u1, Cx<double> u2, Cx<double> t) {
  auto hi = [](double v) { return __double2hiint(v) & 0x7fffffff; };
  const Cx<double> x = (p - t) * 0.5;
  const int e = max(max(hi(x.x), hi(x.y)), max(max(hi(u1.x), hi(u1.y)), max(hi(u2.x), hi(u2.y)))) >> 20;
  if ((unsigned)(e - (1023 - 200)) > 400u) return wilkinson<double>(p, u1, u2, t);
  const Cx<double> w = u1 * u2, z = x * x + w;
  Cx<double> y = cxzero<double>();
  if (max(hi(z.x), hi(z.y)) >> 20 > 1023 - 500) {               // principal root of z
    const double m2 = fma(z.x, z.x, z.y * z.y), t2 = 0.5 * fma(m2, rsqrt64(m2), fabs(z.x));
    const double rt = rsqrt64(t2), a = t2 * rt, b = 0.5 * (z.y * rt);
    y = z.x >= 0.0 ? cxmk<double>(a, b) : cxmk<double>(fabs(b), z.y < 0.0 ? -a : a);
  }
  if (fma(x.x, y.x, x.y * y.y) < 0.0) y = -y;
  const Cx<double> d = x + y;
  const double dd = fma(d.x, d.x, d.y * d.y);
  if (hi(dd) >> 20 < 1023 - 900) return t;                      // x = 0 = u1 u2
  const double r = rsqrt64(dd);
  return t - w * cxconj(d) * (r * r);
}
}  // namespace qr

// Reflector of (alpha, x) with x real, as used by the chase: beta = -sign(Re alpha)|(alpha, x)|,
// tau = (beta - alpha)/beta, v2 = x/(alpha - beta); one square root and two reciprocals.
template <class R> struct Rot { Cx<R> t1, v2; R t2, beta; bool identity; };
// Called by a whole warp with the same values in every lane.
template <class R> __device__ __forceinline__ Rot<R> householder(Cx<R> alpha, R x) {
  Rot<R> r;
  // scaled by m = max(|Re a|, |Im a|, |x|) so that squares stay in range (the double-float form
  // has FP32's exponent range, where a nearly converged bulge of 1e-25 would square to zero)
  const R m = rmax(rmax(rabs(alpha.x), rabs(alpha.y)), rabs(x));
  if ((x == R(0.0) && alpha.y == R(0.0)) || !(m > RealT<R>::tiny())) {
    r.identity = true; r.t1 = cxzero<R>(); r.v2 = cxzero<R>(); r.t2 = R(0.0); r.beta = alpha.x;
    return r;
  }
  const R im = R(1.0) / m;
  const R ax = qr::plain_mul(alpha.x, im), ay = qr::plain_mul(alpha.y, im), xs = qr::plain_mul(x, im);
  R nrm = rsqrt_(qr::sum_squares(ax, ay, xs));
  R bs = (ax >= R(0.0)) ? -nrm : nrm;                         // beta / m
  Cx<R> d = cxmk<R>(qr::plain_sub(ax, bs), ay);                              // (alpha - beta) / m
  const R dd = qr::sum_squares2(d.x, d.y);
  R ib, idd;
  if constexpr (sizeof(R) == 4) {
    // one reciprocal a half of the warp: the two are a subroutine each and would run one after the other
    const bool upper = threadIdx.x & 16;
    const R r = R(1.0) / (upper ? dd : bs), o = __shfl_xor_sync(0xffffffffu, r, 16);
    ib = upper ? o : r;
    idd = upper ? r : o;
  } else {
    ib = R(1.0) / bs;
    idd = R(1.0) / dd;
  }
  r.identity = false;
  r.beta = bs * m;
  r.t1 = cxmk<R>(qr::plain_sub(bs, ax) * ib, -(ay * ib));
  r.v2 = cxmk<R>(xs * d.x * idd, -(xs * d.y * idd));            // x / (alpha - beta)
  r.t2 = -(xs * ib);                                           // Re(t1 v2) = -x / beta
  return r;
}

template <class R> __device__ __forceinline__ Rot<R> chase_reflector(Cx<R> alpha, R x) { return householder<R>(alpha, x); }
// FP64: the rotation of (alpha, x) onto (|(alpha, x)|, 0): c = alpha / beta, s = x / beta, from one
// reciprocal square root (a division costs as much as 7 multiply-adds here, a square root 10).
template <> __device__ __forceinline__ Rot<double> chase_reflector<double>(Cx<double> alpha, double x) {
  Rot<double> r;
  const int e = max(max(__double2hiint(alpha.x) & 0x7fffffff, __double2hiint(alpha.y) & 0x7fffffff),
                    __double2hiint(x) & 0x7fffffff) >> 20;     // exponent of the largest part
  r.v2 = cxzero<double>();
  if ((x == 0.0 && alpha.y == 0.0) || e == 0) {
    r.identity = true; r.t1 = cxone<double>(); r.t2 = 0.0; r.beta = alpha.x;
    return r;
  }
  double f = 1.0;
  if (e < 1023 - 400 || e > 1023 + 400) {                      // squares kept in range
    f = __hiloint2double((2046 - min(e, 2045)) << 20, 0);      // 2^(1023 - e)
    alpha.x *= f; alpha.y *= f; x *= f;
  }
  const double ss = fma(x, x, fma(alpha.x, alpha.x, alpha.y * alpha.y)), rs = rsqrt(ss);
  r.identity = false;
  r.beta = ss * rs;
  if (f != 1.0) r.beta /= f;
  r.t1 = cxmk<double>(alpha.x * rs, alpha.y * rs);
  r.t2 = x * rs;
  return r;
}

// Reflectors of a window: 32 in FP32, 16 in the 16-byte forms (the same tile bytes).
template <class R> struct QrWin { static constexpr int m = sizeof(R) == 4 ? 32 : 16; };

// largest QR-sweep CTA: 128 (255) registers a thread, so that neither the chase nor the far updates spill
template <class R> struct QrMaxThreads { static constexpr int v = sizeof(R) == 4 ? 512 : 256; };

// One window (or none) as every CTA of the cluster reads it.
enum { kQrIdle = 0, kQrWindow = 1, kQrDone = 2 };
template <class R> struct QrRecord {
  int type, k0, k1;
  int cfar;            // first column of the far left update
  int scaled;          // last window of a sweep whose final subdiagonal is made real by sc
  Cx<R> sc;
  Cx<R> t1[QrWin<R>::m], v2[QrWin<R>::m];
  R t2[QrWin<R>::m];
};

// The chase between two windows: the core (rows and columns k, k + 1 and (k+2, k+1)), row k - 1 of
// columns k, k + 1, the next reflector, the active block [l, i] and the next window.
template <class R> struct QrChase {
  Cx<R> c00, c01, c10, c11, c21, x, y, t1, v2;
  R t2;
  int i, its, total, k0, kp, failed;
  int drain;           // first column of a sweep's last window that is still being applied
  int tile, base;      // the tile of the next window and its first row
  long long steps;
};

// Algorithmic bytes of the QR sweeps, per real type (0 double, 1 float, 2 df64): every bulge step
// reads and writes each of its 2n - 2 element pairs' moving element once (the minimum of the
// single-shift sweep: Z's row, H's row or column carries the other element), so a step moves
// 2 (2n - 2) complex values. Each matrix adds its steps' bytes at the end.
__device__ unsigned long long g_qr_bytes[3];
template <class R> struct QrSlot;
template <> struct QrSlot<double> { static constexpr int v = 0; };
template <> struct QrSlot<float> { static constexpr int v = 1; };
template <> struct QrSlot<df64> { static constexpr int v = 2; };

// Leading dimension of a chase tile: the rows of two windows before the columns', theirs and two
// below (odd, so that lanes a column apart fall on different banks).
template <class R> struct QrTile { static constexpr int ld = 3 * QrWin<R>::m + 5; };

namespace qr {

__device__ __forceinline__ unsigned cta_rank() { unsigned r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ unsigned cta_count() { unsigned r; asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r)); return r; }
// the barrier of every thread that works on the matrix
__device__ __forceinline__ void barrier_all(unsigned ctas) {
  if (ctas == 1) { __syncthreads(); return; }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void helper_barrier(int threads) {
  asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}
// Matrix elements change hands between SMs at the window barriers: loads bypass L1.
template <class R> __device__ __forceinline__ Cx<R> ldg(const Cx<R>* p);
template <> __device__ __forceinline__ Cx<float> ldg<float>(const Cx<float>* p) {
  const float2 v = __ldcg(reinterpret_cast<const float2*>(p));
  return cxmk<float>(v.x, v.y);
}
template <> __device__ __forceinline__ Cx<double> ldg<double>(const Cx<double>* p) {
  const double2 v = __ldcg(reinterpret_cast<const double2*>(p));
  return cxmk<double>(v.x, v.y);
}
template <> __device__ __forceinline__ Cx<df64> ldg<df64>(const Cx<df64>* p) {
  const float4 v = __ldcg(reinterpret_cast<const float4*>(p));
  Cx<df64> c;
  c.x = df64(v.x, v.y); c.y = df64(v.z, v.w);
  return c;
}
__device__ __forceinline__ float shf(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ double shf(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ df64 shf(df64 v, int src) {
  return df64(__shfl_sync(0xffffffffu, v.hi, src), __shfl_sync(0xffffffffu, v.lo, src));
}
template <class R> __device__ __forceinline__ Cx<R> shf(Cx<R> v, int src) { return cxmk<R>(shf(v.x, src), shf(v.y, src)); }

// The far update of 32 rows (one a lane, `row` < 0: none): columns k0 .. k1, reflectors from
// max(k0, kst) on. M is Z, or H with kst = row + 2.
template <class R>
__device__ __forceinline__ void far_rows(Cx<R>* M, int ld, int row, int kst, const QrRecord<R>& g) {
  using C_ = Cx<R>;
  constexpr int U = sizeof(R) == 4 ? 8 : 4;
  const int k1 = g.k1;
  int k = g.k0;
  if (row < 0) return;
  if (kst > k) k = kst;
  if (k >= k1) return;
  C_* p = M + row + (long long)k * ld;
  C_ a = ldg<R>(p);
  int q = k - g.k0;
  C_ b[U];
  if (k + U <= k1) {
#pragma unroll
    for (int u = 0; u < U; ++u) b[u] = ldg<R>(p + (long long)(u + 1) * ld);
  }
  for (; k + U <= k1; k += U, q += U) {
    C_ nb[U];                                          // the next U elements, in flight meanwhile
    const bool more = k + 2 * U <= k1;
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (more) nb[u] = ldg<R>(p + (long long)(U + u + 1) * ld);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      right_pair(g.t1[q + u], g.v2[q + u], g.t2[q + u], a, b[u]);
      p[(long long)u * ld] = a;
      a = b[u];
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (more) b[u] = nb[u];
    p += (long long)U * ld;
  }
  for (; k < k1; ++k, ++q) {
    C_ nx = ldg<R>(p + ld);
    right_pair(g.t1[q], g.v2[q], g.t2[q], a, nx);
    *p = a;
    a = nx;
    p += ld;
  }
  if (g.scaled) a = scaled_column(g.sc, a);
  *p = a;
}

// The far update of columns c0 .. c0 + 31 (those below n): rows k0 .. k1, through the warp's tile
// (rows down a column are contiguous in memory, columns are the lanes').
template <class R>
__device__ __forceinline__ void far_columns(Cx<R>* H, int ld, int n, int c0, const QrRecord<R>& g, Cx<R>* tile) {
  using C_ = Cx<R>;
  constexpr int MW = QrWin<R>::m, S = MW + 1, PER = 32 / MW;   // columns a load instruction covers
  const int lane = threadIdx.x & 31, k0 = g.k0, mm = g.k1 - k0, nc = min(32, n - c0);
  const int r = lane % MW, cc = lane / MW;
  const bool mine = r < mm;
  C_* base = H + k0 + r + (long long)(c0 + cc) * ld;
  for (int j0 = 0; j0 < nc; j0 += 8 * PER) {
    C_ v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = j0 + u * PER;
      if (mine && j + cc < nc) v[u] = ldg<R>(base + (long long)j * ld);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int j = j0 + u * PER;
      if (mine && j + cc < nc) tile[(j + cc) * S + r] = v[u];
    }
  }
  __syncwarp();
  if (lane < nc) {
    C_* t = tile + lane * S;
    C_* end = H + g.k1 + (long long)(c0 + lane) * ld;
    const C_ fin = ldg<R>(end);                       // row k1, the last one the window reaches
    C_ a = t[0];
#pragma unroll 4
    for (int q = 0; q < mm; ++q) {
      C_ b = (q + 1 < mm) ? t[q + 1] : fin;
      left_pair(g.t1[q], g.v2[q], g.t2[q], a, b);
      t[q] = a;
      a = b;
    }
    if (g.scaled) a = scaled_row(g.sc, a);
    *end = a;
  }
  __syncwarp();
  for (int j = 0; j < nc; j += PER)
    if (mine && j + cc < nc) base[(long long)j * ld] = tile[(j + cc) * S + r];
  __syncwarp();
}

// What the chase's helpers do in a tick: the window [k0, k1) of the sweep over [., i], the window
// before from kp on (kp = k0: none), the tile that holds the window's columns and its first row.
struct Request { int k0, k1, kp, i, tile, base, first; };

// The rows base .. e + 2 of columns c0 .. cmax into a tile, zero below the subdiagonal and past i;
// warp `part` of `parts`. Every load of a batch is issued before its first store.
template <class R>
__device__ __forceinline__ void load_tile(const Cx<R>* H, int ldh, Cx<R>* tile, int c0, int cmax, int base, int e,
                                          int i, int part, int parts) {
  using C_ = Cx<R>;
  constexpr int TL = QrTile<R>::ld, CB = 4, RB = (TL + 31) / 32;
  const int lane = threadIdx.x & 31, nrow = e + 3 - base;
  for (int j0 = part; c0 + j0 <= cmax; j0 += CB * parts) {
    C_ v[CB][RB];
#pragma unroll
    for (int b = 0; b < CB; ++b) {
      const int c = c0 + j0 + b * parts;
      const C_* col = H + base + (long long)c * ldh;
#pragma unroll
      for (int u = 0; u < RB; ++u) {
        const int rr = lane + 32 * u;
        v[b][u] = cxzero<R>();
        if (c <= cmax && rr < nrow && base + rr <= min(c + 1, i)) v[b][u] = ldg<R>(col + rr);
      }
    }
#pragma unroll
    for (int b = 0; b < CB; ++b) {
      const int j = j0 + b * parts;
#pragma unroll
      for (int u = 0; u < RB; ++u) {
        const int rr = lane + 32 * u;
        if (c0 + j <= cmax && rr < nrow) tile[j * TL + rr] = v[b][u];
      }
    }
  }
}

// Progress of the chase within a window that is not a sweep's last (it has all m reflectors), from
// the chasing warp to the near one: an mbarrier every kQrStride reflectors, which the lane that
// wrote them to the record arrives on. (A fence before a flag waits for the global stores in
// flight: 500 cycles and more.)
constexpr int kQrStride = 4;
__device__ __forceinline__ uint32_t bar_addr(uint64_t* bars, int j) { return (uint32_t)__cvta_generic_to_shared(bars + j); }
__device__ __forceinline__ void publish(uint64_t* bars, int j) {
  asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}\n" ::"r"(bar_addr(bars, j)) : "memory");
}
__device__ __forceinline__ bool await(uint64_t* bars, int j, uint32_t parity) {
  for (int it = 0; it < (1 << 22); ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(bar_addr(bars, j)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// The near columns k1 + 2 .. : those of the window after [k0, k1). Their rows from the window
// before on come into the tile, see its reflectors (gp), then this window's (g) as the chase
// publishes them; rows above k1 go back to H, row k1 and the untouched ones below stay in the tile.
template <class R>
__device__ __noinline__ bool near_columns(Cx<R>* H, int ldh, Cx<R>* tile, const Request& rq, const QrRecord<R>& g,
                                          const QrRecord<R>& gp, uint64_t* bars, uint32_t parity) {
  using C_ = Cx<R>;
  constexpr int MW = QrWin<R>::m, TL = QrTile<R>::ld;
  __builtin_assume(__isShared(tile)); __builtin_assume(__isShared(&g)); __builtin_assume(__isShared(&gp));
  const int lane = threadIdx.x & 31, k0 = rq.k0, k1 = rq.k1, kp = rq.kp, i = rq.i;
  const int k2 = min(k1 + MW, i), cmax = min(k2 + 1, i);
  load_tile<R>(H, ldh, tile, k1 + 2, cmax, kp, k2, i, 0, 1);
  __syncwarp();
  const bool mine = lane < MW && k1 + 2 + lane <= cmax;
  C_* col = tile + min(lane, MW - 1) * TL;
  C_* out = H + kp + (long long)(k1 + 2 + lane) * ldh;
  C_ a = col[0];
  int r = 0;
  for (int q = 0; q < k0 - kp; ++q, ++r) {
    C_ b = col[r + 1];
    left_pair(gp.t1[q], gp.v2[q], gp.t2[q], a, b);
    if (mine) out[r] = a;
    a = b;
  }
  bool ok = true;
  for (int q = 0; q < k1 - k0; ++q, ++r) {
    if (q % kQrStride == 0) {
      ok = ok && await(bars, q / kQrStride, parity);
      __syncwarp();
    }
    C_ b = col[r + 1];
    left_pair(g.t1[q], g.v2[q], g.t2[q], a, b);
    if (mine) out[r] = a;
    a = b;
  }
  if (mine) col[r] = a;
  return ok;
}

// One window of the chase: the tile holds columns k0 + 2 .. min(k1 + 1, i) from row rq.base on, with
// every reflector below k0 applied; the reflectors go to g.
//
// FP32: every lane carries the core (rows and columns k, k + 1) and computes the reflector, lane j
// the window's column k0 + 2 + j as well; no hand-over is on the chain, which is the core's update
// and the reflector (670 cycles a step with the stores and the next step's loads).
// Double-float: an operation is 8 to 20 FP32 instructions, so the elements of the core are spread over the
// lanes: lane j carries column k0 + j for the left application, lanes 0 .. 3 the rows k - 1 .. k + 2 for the
// right one. (FP64: chase_window64.)
template <class R>
__device__ __noinline__ void chase_window(Cx<R>* H, int ldh, const Cx<R>* tile, const Request& rq, QrChase<R>& cs,
                                          QrRecord<R>& g, uint64_t* bars) {
  using C_ = Cx<R>;
  constexpr int MW = QrWin<R>::m, TL = QrTile<R>::ld;
  __builtin_assume(__isShared(tile)); __builtin_assume(__isShared(&cs)); __builtin_assume(__isShared(&g));
  const int lane = threadIdx.x & 31;
  const int i = rq.i, k0 = rq.k0, k1 = rq.k1, o = k0 - rq.base, cmax = min(k1 + 1, i);
  const bool lastw = k1 == i;
  C_ c00 = cs.c00, c01 = cs.c01, c10 = cs.c10, c11 = cs.c11, c21 = cs.c21, x = cs.x, y = cs.y;
  C_ t1 = cs.t1, v2 = cs.v2;
  R t2 = cs.t2;
  C_ sc = cxone<R>();
  int scaled = 0;
  // a sweep's last subdiagonal made real (step i - 1)
  auto finish = [&](C_ h10, C_& sub) {
    sub = h10;
    if (h10.y != R(0.0)) {
      const R am = modulus(h10);
      if (am > RealT<R>::tiny()) {
        sub = cxmk<R>(am, R(0.0));
        sc = h10 * (R(1.0) / am);
        scaled = 1;
      } else {
        sub = cxmk<R>(h10.x, R(0.0));                         // below the safe range: negligible
      }
    }
  };
  if constexpr (sizeof(R) == 4) {
    const bool mine = lane < MW && k0 + 2 + lane <= cmax;
    const C_* col = tile + min(lane, MW - 1) * TL + o;
    C_* out = H + k0 + (long long)(k0 + 2 + lane) * ldh;
    C_ a = col[0], b = col[1];
    // lane q keeps what step k0 + q leaves on the band
    C_ s00 = c00, ssub = c00, sxf = c00, syf = c00;
    C_ h01 = c01, h11 = c11;
#pragma unroll 1
    for (int q = 0; q < k1 - k0; ++q) {
      const int k = k0 + q;
      const C_ t1c = cxconj(t1), v2c = cxconj(v2);
      g.t1[q] = t1; g.v2[q] = v2; g.t2[q] = t2;               // the same value from every lane: no branch
      // raw diagonal and subdiagonal of column k + 2 (zero past i), for the next step's core
      const C_ p22 = tile[q * TL + o + q + 2], p32 = tile[q * TL + o + q + 3];
      // the lane's column, rows k and k + 1
      C_ sum = left_sum(t1c, a, b, t2);
      const C_ an = a - sum, bn = left_sub(b, sum, v2);
      const C_ yn = shf(an, q), cn = shf(bn, q);              // column k + 2: (k, k+2), (k+1, k+2)
      if (mine && lane > q) out[q] = an;
      a = bn;
      b = col[q + 2];
      // the core: left on columns k, k + 1, right on rows k, k + 1, k + 2
      sum = left_sum(t1c, c00, c10, t2);
      C_ h00 = c00 - sum, h10 = left_sub(c10, sum, v2);
      sum = left_sum(t1c, c01, c11, t2);
      h01 = c01 - sum; h11 = left_sub(c11, sum, v2);
      sum = right_sum(t1, h00, h01, t2);
      h00 = h00 - sum; h01 = right_sub(h01, sum, v2c);
      sum = left_sum(t1, h10, h11, t2);
      h10 = h10 - sum; h11 = right_sub(h11, sum, v2c);
      sum = cxmk<R>(plain_mul(c21.x, t2), plain_mul(c21.y, t2));
      const C_ h20 = -sum;
      const C_ h21 = left_sub(c21, sum, v2c);
      // row k - 1, columns k, k + 1 (right): its superdiagonal is final
      sum = right_sum(t1, x, y, t2);
      const C_ xf = x - sum, yf = right_sub(y, sum, v2c);
      C_ sub = h10;
      if (k + 1 < i) {
        const Rot<R> rn = chase_reflector(h10, h20.x);
        if (!rn.identity) sub = cxmk<R>(rn.beta, R(0.0));
        t1 = rn.t1; v2 = rn.v2; t2 = rn.t2;
        c00 = h11; c10 = h21; c01 = cn; c11 = p22; c21 = p32;
        x = h01; y = yn;
      }
      s00.x = lane == q ? h00.x : s00.x; s00.y = lane == q ? h00.y : s00.y;
      ssub.x = lane == q ? sub.x : ssub.x; ssub.y = lane == q ? sub.y : ssub.y;
      sxf.x = lane == q ? xf.x : sxf.x; sxf.y = lane == q ? xf.y : sxf.y;
      syf.x = lane == q ? yf.x : syf.x; syf.y = lane == q ? yf.y : syf.y;
      if (!lastw && (q + 1) % kQrStride == 0 && lane == 0) publish(bars, q / kQrStride);
    }
    if (lane < k1 - k0) {
      const int k = k0 + lane;
      if (lastw && k == i - 1) {
        finish(ssub, ssub);
        if (scaled) { h01 = scaled_column(sc, h01); syf = scaled_column(sc, syf); }
        H[i - 1 + (long long)i * ldh] = h01;
        H[i + (long long)i * ldh] = h11;
        g.sc = sc; g.scaled = scaled;
      }
      C_* d = H + k + (long long)k * ldh;
      d[0] = s00;
      d[1] = ssub;
      if (k > 0) { d[-1] = sxf; d[ldh - 1] = syf; }
    }
    if (!lastw && lane == 0) g.scaled = 0;
  } else {
    // lane j: column k0 + j
    const bool mine = lane < MW + 2 && k0 + lane <= cmax;
    const C_* col = tile + min(max(lane - 2, 0), MW - 1) * TL + o;
    C_* out = H + k0 + (long long)(k0 + lane) * ldh;
    C_ a = lane == 0 ? c00 : lane == 1 ? c01 : col[0];
    C_ b = lane == 0 ? c10 : lane == 1 ? c11 : col[1];
    C_* band = H + (k0 - 1 + lane) + (long long)k0 * ldh;     // lanes 0 .. 2: rows k - 1 .. k + 1 of column k
#pragma unroll 1
    for (int q = 0; q < k1 - k0; ++q) {
      const int k = k0 + q;
      g.t1[q] = t1; g.v2[q] = v2; g.t2[q] = t2;               // the same value from every lane: no branch
      const C_ p22 = tile[q * TL + o + q + 2], p32 = tile[q * TL + o + q + 3];
      C_ an = a, bn = b;
      left_pair(t1, v2, t2, an, bn);
      const C_ a0 = shf(an, q), a1 = shf(an, q + 1), b0 = shf(bn, q), b1 = shf(bn, q + 1);
      const C_ yn = shf(an, q + 2), cn = shf(bn, q + 2);
      if (mine && lane > q + 2) out[q] = an;
      // right on rows k - 1 (lane 0), k, k + 1, k + 2 (lane 3) of columns k, k + 1
      C_ p = cxzero<R>(), w = c21;
      if (lane == 0) { p = x; w = y; }
      if (lane == 1) { p = a0; w = a1; }
      if (lane == 2) { p = b0; w = b1; }
      right_pair(t1, v2, t2, p, w);
      const C_ pn = p, wn = w;
      const C_ h10 = shf(pn, 2), h11 = shf(wn, 2), h21 = shf(wn, 3), h01 = shf(wn, 1);
      const R h20 = shf(pn.x, 3);
      C_ sub = h10;
      const bool more = k + 1 < i;
      if (more) {
        const Rot<R> rn = chase_reflector(h10, h20);
        if (!rn.identity) sub = cxmk<R>(rn.beta, R(0.0));
        t1 = rn.t1; v2 = rn.v2; t2 = rn.t2;
        a = bn;
        b = col[q + 2];
        if (lane == q + 1) { a = h11; b = h21; }
        c00 = h11; c10 = h21; c01 = cn; c11 = p22; c21 = p32;
        x = h01; y = yn;
      } else {
        finish(h10, sub);
      }
      C_ top = h01, yf = wn;
      if (scaled) { top = sc * top; yf = sc * yf; }
      if (lane < 3 && (lane > 0 || k > 0)) *band = lane == 2 ? sub : pn;
      if (lane == 0) {
        if (k > 0) band[ldh] = yf;
        if (!more) { H[i - 1 + (long long)i * ldh] = top; H[i + (long long)i * ldh] = h11; }
      }
      __syncwarp();
      band += ldh + 1;
      if (!lastw && (q + 1) % kQrStride == 0 && lane == 0) publish(bars, q / kQrStride);
    }
    if (lane == 0) { g.sc = sc; g.scaled = scaled; }
  }
  if (lane == 0) {
    const int k2 = min(k1 + MW, i), k3 = min(k2 + MW, i);
    g.k0 = k0; g.k1 = k1;
    g.cfar = min(k3 + 1, i) + 1;
    cs.c00 = c00; cs.c01 = c01; cs.c10 = c10; cs.c11 = c11; cs.c21 = c21; cs.x = x; cs.y = y;
    cs.t1 = t1; cs.v2 = v2; cs.t2 = t2;
    if (lastw) { cs.drain = k0; cs.k0 = -1; }
    else { cs.kp = k0; cs.k0 = k1; cs.base = rq.kp; cs.tile ^= 1; }
  }
  __syncwarp();
}

// FP64: an instruction takes 64 cycles of a warp's issue on GB300 whatever its active lanes, so the
// elements are spread over the lanes by their real components. For the left application lane 4 j + c
// carries component c of column k + j's pair (c = 0, 1: row k; 2, 3: row k + 1), 8 columns a set, the
// window's columns in up to three sets that move down a slot a step; for the right one lane 4 r + c
// carries row k - 1 + r of columns k, k + 1. Each application is then three operations
// (cx u + (+-cy) v + (+-s) w, the partners v and w by shuffles) instead of twelve, in the order of
// left_pair and right_pair: the bits are theirs.
__device__ __forceinline__ double flip(double v, int mask) {    // v with its sign changed by mask (0 or 1 << 31)
  return __hiloint2double(__double2hiint(v) ^ mask, __double2loint(v));
}
__device__ __forceinline__ double shx(double v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }

struct Chase64 {
  double L[3];                 // left layout: this lane's component of its pair in every set
  double e;                    // right layout: rows k - 1 and k + 2
  double cx, cy, s;            // the rotation
  const double* in;            // left layout, set 0: row k + 2 of column k + 1 + slot (the next step's) in the tile
  const double* sub;           // (k + 3, k + 2) in the tile
  double* out;                 // row k of column k + slot in H
  double* band;                // right layout: row k - 1 + slot of column k + c / 2 in H
  double* rec;                 // lanes 0 .. 2: the rotation's parts in the record
};

template <int NS>
__device__ __forceinline__ void chase64_step(Chase64& v, Cx<double>* H, int ldh, int k, int i, int cmax,
                                             QrRecord<double>& g) {
  constexpr int TL = QrTile<double>::ld;
  const int lane = threadIdx.x & 31, c = lane & 3, slot = lane >> 2;
  const int left = (c == 1 || c == 2) ? 1 << 31 : 0, rest = c >= 2 ? 1 << 31 : 0;
  const int col2 = ((c >> 1) * 4 + (c & 1)) | (lane & 8 ? 2 : 0);   // slot 1: row k, slot 2: row k + 1 of column k + c / 2
  // left on columns k ..
  const double cyl = flip(v.cy, left), sl = flip(v.s, rest);
  double Ln[NS], nb[NS];
  Ln[0] = fma(v.cx, v.L[0], fma(cyl, shx(v.L[0], 1), sl * shx(v.L[0], 2)));
  if (lane < 3) *v.rec = lane == 0 ? v.cx : lane == 1 ? v.cy : v.s;
  // right on rows k - 1 .. k + 2 of columns k, k + 1; lane 16 makes the square of (k + 2, k)
  const double ev = shx(v.e, 1), ew = shx(v.e, 2);
  double u = shf(Ln[0], col2), pv = shf(Ln[0], col2 ^ 1), pw = shf(Ln[0], col2 ^ 4);
  if (slot != 1 && slot != 2) { u = v.e; pv = ev; pw = ew; }
  const double r1 = sl * pw;
  const bool sq = slot == 4;
  const double r2 = fma(sq ? r1 : flip(cyl, 1 << 31), sq ? r1 : pv, sq ? 0.0 : r1);
  const double Rn = fma(v.cx, u, r2);
  // the rows the next step needs: row k + 2 of its columns, (k + 3, k + 2). A column past the window's
  // reads what the tile happens to hold there: it never joins the core.
#pragma unroll
  for (int t = 0; t < NS; ++t) nb[t] = v.in[t == 0 && slot == 0 ? 2 * TL : 16 * t * TL];
  const double n21 = v.sub[c & 1];
#pragma unroll
  for (int t = 1; t < NS; ++t) Ln[t] = fma(v.cx, v.L[t], fma(cyl, shx(v.L[t], 1), sl * shx(v.L[t], 2)));
  const double ax = shf(Rn, 8), ay = shf(Rn, 9), xx = shf(Rn, 12), x2 = shf(Rn, 16);
  double top = Rn;                                              // what the band keeps, right layout
  if (k + 1 < i) {
    const int e = max(max(__double2hiint(ax) & 0x7fffffff, __double2hiint(ay) & 0x7fffffff), __double2hiint(xx) & 0x7fffffff) >> 20;
    double beta, z0 = 0.0;
    if ((unsigned)(e - (1023 - 400)) > 800u) {
      const Rot<double> rn = chase_reflector<double>(cxmk<double>(ax, ay), xx);
      beta = rn.beta;
      if (rn.identity) z0 = ay;
      v.cx = rn.t1.x; v.cy = rn.t1.y; v.s = rn.t2;
    } else {
      // (ax, ay, xx, ss) / sqrt(ss), one a lane, by one third-order step from a 22-bit start
      const double ss = fma(ax, ax, fma(ay, ay, x2)), y = rsqrt_start(ss);
      const double z = (c == 0 ? ax : c == 1 ? ay : c == 2 ? xx : ss) * y;
      const double d = fma(-shf(z, 3), y, 1.0);
      beta = fma(z, d * fma(d, 0.375, 0.5), z);
      v.cx = shf(beta, 0); v.cy = shf(beta, 1); v.s = shf(beta, 2);   // c == 3 keeps sqrt(ss)
    }
    // the pairs of step k + 1
    double m[NS];
#pragma unroll
    for (int t = 0; t < NS; ++t) m[t] = shf(Ln[t], (lane + 6) & 31);
    const double core = shf(Rn, 10 + (c & 1) + 4 * (c >> 1));
    const double xy = shf(slot == 1 ? Rn : Ln[0], 6 + c);       // (k, k + 1), (k, k + 2)
#pragma unroll
    for (int t = 0; t < NS; ++t) v.L[t] = c >= 2 ? nb[t] : slot < 7 ? m[t] : t + 1 < NS ? m[t + 1 < NS ? t + 1 : t] : 0.0;
    if (slot == 0) v.L[0] = core;
    v.e = slot == 0 ? xy : c >= 2 ? n21 : 0.0;
    if (slot < 2 && (slot == 0 || c < 2) && (slot > 0 || k > 0)) *v.band = top;
    if (slot == 2 && c >= 2) v.band[c == 3 ? -1 : 0] = c == 3 ? beta : z0;
  } else {
    // the sweep's last subdiagonal made real; the factor goes to column k + 1
    Cx<double> sc = cxone<double>();
    double subx = ax;
    int scaled = 0;
    if (ay != 0.0) {
      const double am = modulus(cxmk<double>(ax, ay));
      if (am > RealT<double>::tiny()) {
        subx = am;
        sc = cxmk<double>(ax, ay) * (1.0 / am);
        scaled = 1;
      }
    }
    const double other = shx(Rn, 1);
    if (scaled && c >= 2 && slot <= 1) {
      const Cx<double> p = c == 2 ? cxmk<double>(Rn, other) : cxmk<double>(other, Rn);
      const Cx<double> w = sc * p;
      top = c == 2 ? w.x : w.y;
    }
    if (lane == 0) { g.sc = sc; g.scaled = scaled; }
    if (slot == 2 && c < 2) top = c ? 0.0 : subx;
    double* at = slot == 2 && c >= 2 ? v.band + 2 * ldh - 3 + c : v.band;
    if (slot < 3 && (slot > 0 || k > 0)) *at = top;             // rows k, k + 1 of column k + 1 too
  }
  // the finished row k of the columns past k + 2
#pragma unroll
  for (int t = 0; t < NS; ++t)
    if (c < 2 && 8 * t + slot >= 3 && k + 8 * t + slot <= cmax) v.out[16LL * t * ldh] = Ln[t];
  v.in += 2 * (TL + 1);
  v.sub += 2 * (TL + 1);
  v.out += 2 * (ldh + 1);
  v.band += 2 * (ldh + 1);
  v.rec += lane < 2 ? 2 : 1;
}

__device__ __noinline__ void chase_window64(Cx<double>* H, int ldh, const Cx<double>* tile, const Request& rq,
                                            QrChase<double>& cs, QrRecord<double>& g, uint64_t* bars) {
  constexpr int MW = QrWin<double>::m, TL = QrTile<double>::ld;
  static_assert(MW + 2 <= 24, "three sets of columns");
  __builtin_assume(__isShared(tile)); __builtin_assume(__isShared(&cs)); __builtin_assume(__isShared(&g));
  const int lane = threadIdx.x & 31, c = lane & 3, slot = lane >> 2;
  const int i = rq.i, k0 = rq.k0, k1 = rq.k1, o = k0 - rq.base, cmax = min(k1 + 1, i);
  const bool lastw = k1 == i;
  const double* td = reinterpret_cast<const double*>(tile);
  Chase64 v;
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const int jj = 8 * t + slot - 2;
    v.L[t] = (jj >= 0 && jj < MW && k0 + 2 + jj <= cmax) ? td[2 * (jj * TL + o + (c >> 1)) + (c & 1)] : 0.0;
  }
  auto part = [](const Cx<double>& a, int p) { return p ? a.y : a.x; };
  if (slot == 0) v.L[0] = part(c < 2 ? cs.c00 : cs.c10, c & 1);
  if (slot == 1) v.L[0] = part(c < 2 ? cs.c01 : cs.c11, c & 1);
  v.e = slot == 0 ? part(c < 2 ? cs.x : cs.y, c & 1) : c >= 2 ? part(cs.c21, c & 1) : 0.0;
  v.cx = cs.t1.x; v.cy = cs.t1.y; v.s = cs.t2;
  v.in = td + 2 * ((slot - 1) * TL + o + 2) + (c & 1);         // the core's column (slot 0, set 0) reads the next one's
  v.sub = td + 2 * (o + 3);
  v.out = reinterpret_cast<double*>(H + k0 + (long long)(k0 + slot) * ldh) + (c & 1);
  v.band = reinterpret_cast<double*>(H + (k0 - 1 + slot) + (long long)(k0 + (c >> 1)) * ldh) + (c & 1);
  if (slot == 2 && c >= 2) v.band = reinterpret_cast<double*>(H + k0 + 1 + (long long)k0 * ldh) + 1;
  v.rec = lane < 2 ? reinterpret_cast<double*>(g.t1) + lane : g.t2;
  __syncwarp();
  if (lane == 0) { g.sc = cxone<double>(); g.scaled = 0; }
  const int nc = cmax - k0 + 1;                                 // columns at the window's first step
  int q = 0;
  auto done = [&]() {
    ++q;
    if (q % kQrStride == 0) {
      __syncwarp();
      if (!lastw && lane == 0) publish(bars, q / kQrStride - 1);
    }
  };
#pragma unroll 1
  while (q < k1 - k0 && nc - q > 16) { chase64_step<3>(v, H, ldh, k0 + q, i, cmax, g); done(); }
#pragma unroll 1
  while (q < k1 - k0 && nc - q > 8) { chase64_step<2>(v, H, ldh, k0 + q, i, cmax, g); done(); }
#pragma unroll 1
  while (q < k1 - k0) { chase64_step<1>(v, H, ldh, k0 + q, i, cmax, g); done(); }
  __syncwarp();
  if (slot < 2) reinterpret_cast<double*>(slot ? (c < 2 ? &cs.c01 : &cs.c11) : (c < 2 ? &cs.c00 : &cs.c10))[c & 1] = v.L[0];
  if (slot == 0) reinterpret_cast<double*>(c < 2 ? &cs.x : &cs.y)[c & 1] = v.e;
  if (slot == 3 && c >= 2) reinterpret_cast<double*>(&cs.c21)[c & 1] = v.e;
  if (lane == 0) {
    const int k2 = min(k1 + MW, i), k3 = min(k2 + MW, i);
    g.k0 = k0; g.k1 = k1;
    g.cfar = min(k3 + 1, i) + 1;
    cs.t1 = cxmk<double>(v.cx, v.cy); cs.v2 = cxzero<double>(); cs.t2 = v.s;
    if (lastw) { cs.drain = k0; cs.k0 = -1; }
    else { cs.kp = k0; cs.k0 = k1; cs.base = rq.kp; cs.tile ^= 1; }
  }
  __syncwarp();
}

// The near columns in FP64: warp `part` (0, 1) carries eight of them, four lanes a column as above.
__device__ __noinline__ bool near_columns64(Cx<double>* H, int ldh, Cx<double>* tile, const Request& rq, int part,
                                            const QrRecord<double>& g, const QrRecord<double>& gp, uint64_t* bars,
                                            uint32_t parity) {
  constexpr int MW = QrWin<double>::m, TL = QrTile<double>::ld;
  static_assert(MW == 16, "two warps of eight columns");
  __builtin_assume(__isShared(tile)); __builtin_assume(__isShared(&g)); __builtin_assume(__isShared(&gp));
  const int lane = threadIdx.x & 31, c = lane & 3, slot = lane >> 2;
  const int k0 = rq.k0, k1 = rq.k1, kp = rq.kp, i = rq.i;
  const int k2 = min(k1 + MW, i), c0 = k1 + 2 + 8 * part, cmax = min(min(k2 + 1, i), c0 + 7);
  tile += 8 * part * TL;
  load_tile<double>(H, ldh, tile, c0, cmax, kp, k2, i, 0, 1);
  __syncwarp();
  const bool mine = c0 + slot <= cmax;
  double* col = reinterpret_cast<double*>(tile + slot * TL) + (c & 1);
  double* out = reinterpret_cast<double*>(H + kp + (long long)(c0 + slot) * ldh) + (c & 1);
  const int left = (c == 1 || c == 2) ? 1 << 31 : 0, rest = c >= 2 ? 1 << 31 : 0;
  double L = c < 2 ? col[0] : col[2];
  bool ok = true;
  const int np = k0 - kp, nt = k1 - kp;
  for (int r = 0; r < nt; ++r) {
    const int q = r - np;
    if (q >= 0 && q % kQrStride == 0) {
      ok = ok && await(bars, q / kQrStride, parity);
      __syncwarp();
    }
    const QrRecord<double>& gr = q < 0 ? gp : g;
    const int e = q < 0 ? r : q;
    const Cx<double> t1 = gr.t1[e];
    const double s = gr.t2[e], nb = col[2 * (r + 2)];
    const double Ln = fma(t1.x, L, fma(flip(t1.y, left), shx(L, 1), flip(s, rest) * shx(L, 2)));
    const double dn = shx(Ln, 2);
    if (mine && c < 2) out[2 * r] = Ln;
    L = c < 2 ? dn : nb;
  }
  if (mine && c < 2) col[2 * nt] = L;
  return ok;
}

// A subdiagonal below one unit of roundoff of its neighbours' diagonal deflates if the refined test
// agrees (Ahues and Tisseur). Where both diagonal entries are the same number (equal eigenvalues of a
// uniform layer, split by rounding alone) that test never does, and when the shift rounds to them too
// a sweep only swaps the two: after 10 sweeps the FP64 form also deflates a pair that cannot be told apart, its
// diagonal entries within tol = one unit of roundoff of their sum and its split, the root of the two off-diagonal
// entries' product, below tol too. Any other block keeps the refined test, however slow.
template <class R> struct QrStall { static constexpr int its = 1 << 30; };
template <> struct QrStall<double> { static constexpr int its = 10; };
template <class R> __device__ __forceinline__ bool same_pair(Cx<R> dd, Cx<R> sub, Cx<R> sup, R tol) {
  return cxabs1(dd) <= tol && cxabs1(sub) * cxabs1(sup) <= tol * tol;
}

// What the chase does next, decided by the chasing warp: continue the sweep, or find the active
// block of the next one (deflating converged eigenvalues into w), its shift and first reflector.
template <class R>
__device__ __noinline__ int next_window(Cx<R>* H, int n, int ldh, Cx<R>* w, int itmax, QrChase<R>& cs, Request& rq) {
  using C_ = Cx<R>;
  constexpr int MW = QrWin<R>::m;
  __builtin_assume(__isShared(&cs));
  const int lane = threadIdx.x & 31;
  const R ulp = RealT<R>::eps();
  const R smlnum = RealT<R>::tiny() * (R((double)n) / ulp);
  auto h = [&](int i, int j) -> C_& { return H[i + (long long)j * ldh]; };
  auto hl = [&](int i, int j) -> C_ { return ldg<R>(H + i + (long long)j * ldh); };
  int type = kQrWindow;
  int i = cs.i, k0 = cs.k0;
  if (k0 < 0) {                                          // a new sweep: deflate, shift
    int its = cs.its, l = 0, failed = 0;
    const int total = cs.total;
    for (;;) {
      if (i < 0) { type = kQrDone; break; }
      // largest k in [1, i] with a negligible subdiagonal H(k, k-1), 0 when there is none
      int cand = 0;
      unsigned maybe = ~0u;                                // chunks of 32 of the next 128 that have to be looked at
      for (int kb = i; kb >= 1; kb -= 32) {
        if constexpr (std::is_same<R, double>::value) {
          // By the exponents alone (integers): |sub| > 2^-49 of the largest part of its neighbours stays.
          if (((i - kb) & 96) == 0) {
            bool any[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int k = kb - 32 * u - lane;
              any[u] = false;
              if (k >= 1) {
                const C_ hd = hl(k, k), hp = hl(k - 1, k - 1);
                auto hi = [](double v) { return __double2hiint(v) & 0x7fffffff; };
                const int es = hi(hl(k, k - 1).x) >> 20, em = max(max(hi(hd.x), hi(hd.y)), max(hi(hp.x), hi(hp.y))) >> 20;
                any[u] = es <= max(em - 48, 100) || em == 0;
              }
            }
            maybe = 0;
#pragma unroll
            for (int u = 0; u < 4; ++u) maybe |= __any_sync(0xffffffffu, any[u]) ? 1u << u : 0u;
          }
          if (!(maybe >> (((i - kb) >> 5) & 3) & 1u)) continue;
        }
        const int k = kb - lane;
        bool small = false;
        if (k >= 1) {
          const C_ sub = hl(k, k - 1), hd = hl(k, k), hp = hl(k - 1, k - 1), hu = hl(k - 1, k);
          if (cxabs1(sub) <= smlnum) {
            small = true;
          } else {
            R tst = cxabs1(hp) + cxabs1(hd);
            if (tst == R(0.0)) {
              if (k - 2 >= 0) tst = tst + rabs(hl(k - 1, k - 2).x);
              if (k + 1 <= i) tst = tst + rabs(hl(k + 1, k).x);
            }
            if (rabs(sub.x) <= ulp * tst) {
              R ab = rmax(cxabs1(sub), cxabs1(hu));
              R ba = rmin(cxabs1(sub), cxabs1(hu));
              C_ dd = hp - hd;
              R aa = rmax(cxabs1(hd), cxabs1(dd));
              R bb = rmin(cxabs1(hd), cxabs1(dd));
              R sx = aa + ab;
              if (ba * (ab / sx) <= rmax(smlnum, ulp * (bb * (aa / sx)))) small = true;
              else if (its >= QrStall<R>::its && same_pair<R>(dd, sub, hu, ulp * tst)) small = true;
            }
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, small);
        if (m) { cand = kb - (__ffs(m) - 1); break; }
      }
      l = cand;
      if (l < i) break;
      if (lane == 0) w[i] = hl(i, i);
      i -= 1;
      its = 0;
    }
    if (type == kQrWindow) {
      if (lane == 0 && l > 0) h(l, l - 1) = cxzero<R>();
      if (its >= 60 || total >= itmax) { failed = 1; type = kQrDone; }
    }
    if (type == kQrWindow && min(l + 2 * MW + 1, i) >= cs.drain) type = kQrIdle;   // let the last window drain
    if (type == kQrWindow) {
      ++its;
      C_ t;
      if (its % 20 == 10) {
        R sx = R(0.75) * rabs(hl(l + 1, l).x);
        t = cxmk<R>(sx, R(0.0)) + hl(l, l);
      } else if (its % 20 == 0) {
        R sx = R(0.75) * rabs(hl(i, i - 1).x);
        t = cxmk<R>(sx, R(0.0)) + hl(i, i);
      } else {
        t = wilkinson(hl(i - 1, i - 1), hl(i - 1, i), hl(i, i - 1), hl(i, i));
      }
      const C_ c00 = hl(l, l), c01 = hl(l, l + 1), c10 = hl(l + 1, l), c11 = hl(l + 1, l + 1);
      const C_ c21 = (l + 2 <= i) ? hl(l + 2, l + 1) : cxzero<R>();
      C_ x = cxzero<R>(), y = x;
      if (l > 0) { x = hl(l - 1, l); y = hl(l - 1, l + 1); }
      C_ h11s = c00 - t;
      R h21 = c10.x;
      R sc = cxabs1(h11s) + rabs(h21);
      if (sc == R(0.0)) sc = R(1.0);
      R isc = R(1.0) / sc;
      // the first reflector of the sweep, from the shifted first column
      Rot<R> rf;
      if constexpr (std::is_same<R, double>::value) rf = chase_reflector<R>(h11s, h21);   // scales by itself
      else rf = chase_reflector(h11s * isc, h21 * isc);
      k0 = l;
      __syncwarp();
      if (lane == 0) {
        cs.c00 = c00; cs.c01 = c01; cs.c10 = c10; cs.c11 = c11; cs.c21 = c21; cs.x = x; cs.y = y;
        cs.t1 = rf.t1; cs.v2 = rf.v2; cs.t2 = rf.t2;
        cs.k0 = l; cs.kp = l; cs.base = l; cs.total = total + 1; cs.steps += i - l;
      }
    }
    __syncwarp();
    if (lane == 0) { cs.i = i; cs.its = its; cs.failed = failed; }
  }
  __syncwarp();
  if (lane == 0) {
    cs.drain = 0x7fffffff;
    rq.k0 = type == kQrWindow ? k0 : -1;
    rq.k1 = min(k0 + MW, i); rq.kp = cs.kp; rq.i = i; rq.tile = cs.tile; rq.base = cs.base;
    rq.first = cs.kp == k0;
  }
  __syncwarp();
  return type;
}

// The window of record g everywhere but in the chase's columns: this warp's share of the tasks.
template <class R>
__device__ __noinline__ void far_update(Cx<R>* H, int ldh, Cx<R>* Z, int ldz, int n, const QrRecord<R>& g, Cx<R>* tile,
                                        int worker, int nworkers) {
  __builtin_assume(__isShared(tile)); __builtin_assume(__isShared(&g));
  const int lane = threadIdx.x & 31;
  const int tz = (n + 31) / 32, rows = max(0, g.k1 - 2), th = (rows + 31) / 32;
  const int tc = (max(0, n - g.cfar) + 31) / 32;
#pragma unroll 1
  for (int t = worker; t < tz + th + tc; t += nworkers) {
    if (t < tc) {
      far_columns<R>(H, ldh, n, g.cfar + 32 * t, g, tile);
    } else {
      const bool z = t >= tc + th;
      const int r = 32 * (t - (z ? tc + th : tc)) + lane;
      far_rows<R>(z ? Z : H, z ? ldz : ldh, r < (z ? n : rows) ? r : -1, z ? 0 : r + 2, g);
    }
  }
}

// The record to the other CTAs of the cluster
template <class R> __device__ __noinline__ void send_record(QrRecord<R>& g, unsigned ctas) {
  const int lane = threadIdx.x & 31;
  const unsigned src = (unsigned)__cvta_generic_to_shared(&g);
  constexpr int words = sizeof(QrRecord<R>) / 4;
  const int* rw = reinterpret_cast<const int*>(&g);
  for (unsigned c = 1; c < ctas; ++c) {
    unsigned dst;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(src), "r"(c));
    for (int e = lane; e < words; e += 32)
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(dst + 4 * e), "r"(rw[e]) : "memory");
  }
}

// The unit factors of the diagonal similarity that makes the subdiagonal real, applied to H and Z
// (d_i = d_{i-1} sd_i / |sd_i|): the factors in parallel, then their running product.
template <class R>
__device__ __noinline__ void real_subdiagonal(Cx<R>* H, int ldh, Cx<R>* Z, int ldz, int n, Cx<R>* sphase, unsigned rank,
                                              unsigned ctas) {
  using C_ = Cx<R>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nw = blockDim.x >> 5;
  for (int r = tid; r < n; r += blockDim.x) {
    C_ f = cxone<R>();
    if (r > 0) {
      const C_ sd = ldg<R>(H + r + (long long)(r - 1) * ldh);
      const R a = modulus(sd);
      // a subdiagonal below the safe range keeps a unit phase (its imaginary part is dropped)
      if (a > RealT<R>::tiny() && sd.y != R(0.0)) f = sd * (R(1.0) / a);
      else f = cxzero<R>();                                  // zero: no factor
    }
    sphase[r] = f;
  }
  __syncthreads();
  if (tid == 0) {
    C_ d = cxone<R>();
    for (int r = 1; r < n; ++r) {
      const C_ f = sphase[r];
      if (f.x != R(0.0) || f.y != R(0.0)) d = product(d, f);
      sphase[r] = d;
    }
  }
  barrier_all(ctas);
  const int warps = nw * (int)ctas;
  for (int c = warp * (int)ctas + (int)rank; c < n; c += warps) {
    const C_ pc = sphase[c];
    C_* hc = H + (long long)c * ldh;
    C_* zc = Z + (long long)c * ldz;
    for (int r = lane; r < n; r += 32) {
      if (r <= c + 1) {
        C_ v = product(product(cxconj(sphase[r]), hc[r]), pc);
        if (r == c + 1) v = cxmk<R>(v.x, R(0.0));
        hc[r] = v;
      }
      zc[r] = scaled_column(zc[r], pc);
    }
  }
  barrier_all(ctas);
}

}  // namespace qr

template <class R>
__global__ void __launch_bounds__(QrMaxThreads<R>::v) hseqr_kernel(Cx<R>* __restrict__ Hall, int n, int ldh,
                                                            long long h_bs, Cx<R>* __restrict__ Zall, int ldz,
                                                            long long z_bs, Cx<R>* __restrict__ w_all,
                                                            int32_t* __restrict__ status, int st_div, int itmax) {
  using C_ = Cx<R>;
  constexpr int MW = QrWin<R>::m, TL = QrTile<R>::ld, TS = MW * TL;
  extern __shared__ __align__(16) unsigned char smraw[];
  C_* tile = reinterpret_cast<C_*>(smraw);                   // chase: two of MW columns x TL rows
  __shared__ QrRecord<R> rec[2];
  __shared__ QrChase<R> cs;
  __shared__ qr::Request s_req;                              // k0 < 0: no window in this tick
  __shared__ uint64_t s_bar[MW / qr::kQrStride];
  __shared__ int s_late;
  const unsigned ctas = qr::cta_count(), rank = qr::cta_rank();
  const int warp = threadIdx.x >> 5;
  C_* H = Hall + (blockIdx.x / ctas) * h_bs;
  C_* Z = Zall + (blockIdx.x / ctas) * z_bs;
  qr::real_subdiagonal<R>(H, ldh, Z, ldz, n, tile, rank, ctas);

  // Warps of the chasing CTA: 0 chases, 1 follows with the near columns, 0 .. 3 bring in a sweep's
  // first tile. Its far updates keep off the chasing warp's scheduler (every fourth warp); in the
  // 16-byte forms of a cluster the CTA leaves them to the others.
  constexpr bool f64 = std::is_same<R, double>::value;
  const bool chaser = rank == 0 && warp == 0, near = rank == 0 && warp >= 1 && warp <= (f64 ? 2 : 1);
  const bool helper = rank == 0 && warp < 4;
  int worker = -1, nworkers;                                 // CTA by CTA within each round of tasks
  {
    const int nw = blockDim.x >> 5, own = (sizeof(R) > 4 && ctas > 1) ? 0 : nw - (nw + 3) / 4 - 1, c = (int)ctas;
    nworkers = own + nw * (c - 1);
    if (f64 && c == 1 && n >= 160) {                         // far updates bound a tick: the chase's scheduler too
      nworkers = nw - 2;
      worker = warp - 2;
    }
    else if (rank > 0) worker = warp < own ? warp * c + (int)rank : own * c + (warp - own) * (c - 1) + (int)rank - 1;
    else if (warp > 1 && warp % 4 != 0 && own > 0) worker = (warp - 2 - warp / 4) * c;
  }
  if (threadIdx.x == 0) {
    cs.i = n - 1; cs.its = 0; cs.total = 0; cs.k0 = -1; cs.kp = 0; cs.failed = 0; cs.drain = 0x7fffffff; cs.steps = 0;
    cs.x = cxzero<R>(); cs.y = cxzero<R>();
    cs.tile = 0; cs.base = 0; s_late = 0;
    for (int j = 0; j < MW / qr::kQrStride; ++j)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(qr::bar_addr(s_bar, j)) : "memory");
  }
  __syncthreads();

  uint32_t followed = 0;                                     // windows the near warp has followed
  for (int tick = 0;; ++tick) {
    const int buf = tick & 1, prev = buf ^ 1;
    int type = kQrIdle;
    if (chaser) type = qr::next_window<R>(H, n, ldh, w_all + (long long)(blockIdx.x / ctas) * n, itmax, cs, s_req);
    if (helper) {
      qr::helper_barrier(128);
      if (s_req.k0 >= 0 && s_req.first) {                    // a new sweep: its first window's columns
        qr::load_tile<R>(H, ldh, tile + s_req.tile * TS, s_req.k0 + 2, min(s_req.k1 + 1, s_req.i), s_req.base,
                         s_req.k1, s_req.i, warp, 4);
        qr::helper_barrier(128);
      }
    }
    if (near && s_req.k0 >= 0 && s_req.k1 < s_req.i) {
      bool ok;
      if constexpr (f64)
        ok = qr::near_columns64(H, ldh, tile + (s_req.tile ^ 1) * TS, s_req, warp - 1, rec[buf], rec[prev], s_bar, followed & 1u);
      else
        ok = qr::near_columns<R>(H, ldh, tile + (s_req.tile ^ 1) * TS, s_req, rec[buf], rec[prev], s_bar, followed & 1u);
      ++followed;
      if (!ok) s_late = 1;
    }
    if (chaser) {
      if (type == kQrWindow) {
        if constexpr (f64) qr::chase_window64(H, ldh, tile + s_req.tile * TS, s_req, cs, rec[buf], s_bar);
        else qr::chase_window<R>(H, ldh, tile + s_req.tile * TS, s_req, cs, rec[buf], s_bar);
      }
      rec[buf].type = type;
      __syncwarp();
      if (ctas > 1) qr::send_record<R>(rec[buf], ctas);
    }
    // the window before, everywhere else
    if (worker >= 0 && tick > 0 && rec[prev].type == kQrWindow)
      qr::far_update<R>(H, ldh, Z, ldz, n, rec[prev], tile + 2 * TS + warp * 32 * (MW + 1), worker, nworkers);
    qr::barrier_all(ctas);
    if (rec[buf].type == kQrDone) break;
  }
  if (chaser) {
    C_* w = w_all + (long long)(blockIdx.x / ctas) * n;
    const int lane = threadIdx.x & 31;
    if (cs.failed || s_late) {
      for (int j = lane; j <= (s_late ? n - 1 : cs.i); j += 32) w[j] = cxmk<R>(R(NAN), R(NAN));
      if (lane == 0) wb_flag(status ? status + blockIdx.x / ctas / st_div : nullptr, WB_ST_NOCONV);
    }
    if (lane == 0)
      atomicAdd(&g_qr_bytes[QrSlot<R>::v],
                (unsigned long long)cs.steps * (unsigned long long)(2 * n - 2) * 2ULL * sizeof(C_));
  }
}

}  // namespace wb
