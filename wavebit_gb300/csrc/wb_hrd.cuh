// FP64 Hessenberg reduction A = Q H Q^H and the forming of Q, for matrices past the 32 x 32 group blocks.
//
// What bounds them: FP64 issue (an instruction holds a scheduler for 64 cycles on GB300, some 2
// multiply-adds a cycle and SM), 6.7 n^3 multiply-adds for H and 2.7 n^3 for Q, and in a small matrix the
// serial part of a step (a norm, a reflector, two sums). One CTA a matrix ran them at half that rate: every
// warp formed the reflector (eight divisions and roots) for itself, and A was read twice a step.
//
// Reduction: a cluster of up to 8 CTAs a matrix. Column j belongs to one warp for good: part j % 8 (the CTA
// is part % ctas), warp j / 8 % 8. A step k, with v its reflector, t its tau:
//   A  every warp reads its columns once: its share of y = A v (lanes own rows) and z_j = v^H A_j.
//      The shares of a part's eight warps are summed in shared memory and sent to every CTA.
//   B  after a cluster barrier: A_j -= y (t conj v_j) + v (conj t)(z_j - t c conj v_j), c = v^H A v. The
//      warp with column k + 1 takes that one first and then forms the next reflector beside the others'
//      updates, and sends it to every CTA.
// The sums run over parts and warps in the same order whatever the cluster, so the bits do not depend on
// it. Only v and y change hands: a column is read and written by one warp.
//
// Measured (H; Q): 32 matrices of 242 51 -> 11.7 ms; 19.6 -> 6.0 ms, 4 of them 51 -> 7.2; 19.6 -> 1.2 ms, one of 50
// 2.4 -> 0.45; 0.47 -> 0.08 ms.
//
// Q: column j of H_0 H_1 .. H_{n-3} is e_j with the reflectors j - 1 .. 0 applied, so columns need nothing
// from one another: a warp keeps two of them in registers through all its reflectors.
#pragma once
#include "wb_common.cuh"
#include "wb_num.cuh"
#include "wb_qr.cuh"

namespace wb {
namespace hrd {

using C64 = Cx<double>;
constexpr int kParts = 8, kWarps = 8, kThreads = 32 * kWarps;

__device__ __forceinline__ C64 fmac(C64 a, C64 b, C64 c) {        // a b + c
  return cxmk<double>(fma(a.x, b.x, fma(-a.y, b.y, c.x)), fma(a.x, b.y, fma(a.y, b.x, c.y)));
}
__device__ __forceinline__ C64 fmac_conj(C64 a, C64 b, C64 c) {   // conj(a) b + c
  return cxmk<double>(fma(a.x, b.x, fma(a.y, b.y, c.x)), fma(a.x, b.y, fma(-a.y, b.x, c.y)));
}
__device__ __forceinline__ C64 nmac(C64 a, C64 b, C64 c) {        // c - a b
  return cxmk<double>(fma(-a.x, b.x, fma(a.y, b.y, c.x)), fma(-a.x, b.y, fma(-a.y, b.x, c.y)));
}
__device__ __forceinline__ C64 shf(C64 v, int src) {
  return cxmk<double>(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
// The sums over the warp of a.x, a.y, b.x, b.y in lanes 0 .. 3 of every four, by six additions.
__device__ __forceinline__ double sum_pair(C64 a, C64 b) {
  const int lane = threadIdx.x & 31;
  const bool hi = lane & 2, odd = lane & 1;
  const double x = (hi ? b.x : a.x) + qr::shx(hi ? a.x : b.x, 2), y = (hi ? b.y : a.y) + qr::shx(hi ? a.y : b.y, 2);
  double s = (odd ? y : x) + qr::shx(odd ? x : y, 1);
#pragma unroll
  for (int off = 4; off < 32; off <<= 1) s += qr::shx(s, off);
  return s;
}
// v to address p (a multiple of 16 bytes) of every CTA's shared memory
__device__ __forceinline__ void send(C64* p, C64 v, unsigned ctas) {
  if (ctas == 1) { *p = v; return; }
  const unsigned src = (unsigned)__cvta_generic_to_shared(p);
  for (unsigned c = 0; c < ctas; ++c) {
    unsigned dst;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(src), "r"(c));
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(dst), "d"(v.x), "d"(v.y) : "memory");
  }
}

// The reflector of (alpha; x), |x|^2 = xn2: beta, tau, 1 / (alpha - beta), from two reciprocal roots
// (make_reflector's eight divisions and root cost 4000 cycles); entries out of 2^+-200 go that way.
__device__ __forceinline__ Refl<double> reflector(C64 alpha, double xn2) {
  auto hi = [](double v) { return __double2hiint(v) & 0x7fffffff; };
  const double ss = fma(alpha.x, alpha.x, fma(alpha.y, alpha.y, xn2));
  if ((unsigned)((hi(ss) >> 20) - (1023 - 400)) > 800u || xn2 == 0.0) return make_reflector<double>(alpha, sqrt(xn2));
  Refl<double> r;
  const double rs = rsqrt64(ss), nrm = ss * rs;
  const bool neg = alpha.x < 0.0;
  r.identity = false;
  r.beta = neg ? nrm : -nrm;
  const double ib = neg ? rs : -rs;
  r.tau = cxmk<double>(fma(-alpha.x, ib, 1.0), -alpha.y * ib);
  const C64 d = cxmk<double>(alpha.x - r.beta, alpha.y);
  const double rd = rsqrt64(fma(d.x, d.x, d.y * d.y)), ir = rd * rd;
  r.scale = cxmk<double>(d.x * ir, -d.y * ir);
  return r;
}

struct __align__(16) Meta { C64 tau; int identity; };

// Reflector k by the warp that has column k: to every CTA's v (zeros above row k + 1), the column's storage
// (v below the subdiagonal, beta on it) and tau.
__device__ __forceinline__ void next_reflector(C64* A, int n, int lda, int k, C64* tau, C64* v, Meta* meta, unsigned ctas) {
  const int lane = threadIdx.x & 31;
  C64* col = A + (long long)k * lda;
  __syncwarp();
  double s = 0.0;
  for (int i = k + 2 + lane; i < n; i += 32) { const C64 x = col[i]; s = fma(x.x, x.x, fma(x.y, x.y, s)); }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) s += qr::shx(s, off);
  const C64 alpha = col[k + 1];
  const Refl<double> r = reflector(alpha, s);
  __syncwarp();
  if (!r.identity) {
    for (int i = lane; i < n; i += 32) {
      C64 x = cxzero<double>();
      if (i == k + 1) {
        x = cxone<double>();
        col[i] = cxmk<double>(r.beta, 0.0);
      } else if (i > k + 1) {
        x = col[i] * r.scale;
        col[i] = x;
      }
      send(v + i, x, ctas);
    }
  }
  if (lane == 0) {
    const C64 t = r.identity ? cxzero<double>() : r.tau;
    tau[k] = t;
    send(&meta->tau, t, ctas);
    for (unsigned c = 0; c < ctas; ++c) {
      unsigned dst;
      asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"((unsigned)__cvta_generic_to_shared(&meta->identity)), "r"(c));
      asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(dst), "r"(r.identity ? 1 : 0) : "memory");
    }
  }
}

// Elements of dynamic shared memory: v twice, y's parts, the warps' shares of 16 / U parts, z.
__host__ __device__ constexpr size_t shared_elements(int n) {
  return (size_t)n * (2 + kParts) + 16 * kWarps * 32 + (size_t)n + kParts * kWarps;
}

// U: rows a lane holds (32 U rows at a time)
template <int U>
__global__ void __launch_bounds__(kThreads, 1) gehrd64_kernel(C64* __restrict__ Aall, int n, int lda, long long a_bs,
                                                              C64* __restrict__ tau_all) {
  constexpr int VP = 16 / U, ROWS = 32 * U;             // parts summed at a time
  extern __shared__ __align__(16) unsigned char smraw[];
  C64* sv = reinterpret_cast<C64*>(smraw);              // [2][n]
  C64* yp = sv + 2 * n;                                 // [kParts][n]
  C64* yw = yp + kParts * n;                            // [VP][kWarps][ROWS]
  C64* z = yw + 16 * kWarps * 32;                       // z_j
  __shared__ Meta meta[2];
  __shared__ __align__(16) C64 cpart[kParts];
  const unsigned ctas = qr::cta_count(), rank = qr::cta_rank();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  C64* A = Aall + (blockIdx.x / ctas) * a_bs;
  C64* tau = tau_all + (long long)(blockIdx.x / ctas) * n;
  const int mine = kParts / (int)ctas;                  // parts rank, rank + ctas, ..
  qr::barrier_all(ctas);                                // every CTA of the cluster runs
  if (rank == 0 && warp == 0) next_reflector(A, n, lda, 0, tau, sv, meta, ctas);
  qr::barrier_all(ctas);
  for (int k = 0; k + 2 < n; ++k) {
    const C64* v = sv + (k & 1) * n;
    const bool step = !meta[k & 1].identity;
    const C64 t = meta[k & 1].tau;
    if (step) {
      for (int p0 = 0; p0 < mine; p0 += VP) {
        const int np = min(VP, mine - p0);
        for (int r0 = 0; r0 < n; r0 += ROWS) {
          C64 vu[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int r = r0 + 32 * u + lane;
            vu[u] = r < n ? v[r] : cxzero<double>();
          }
          for (int p = 0; p < np; ++p) {
            const int part = (int)rank + (p0 + p) * (int)ctas;
            C64 y[U];
#pragma unroll
            for (int u = 0; u < U; ++u) y[u] = cxzero<double>();
            int j = part + kParts * warp;
            if (j < k + 1) j += (k + 1 - j + kParts * kWarps - 1) / (kParts * kWarps) * (kParts * kWarps);
            for (; j < n; j += 2 * kParts * kWarps) {
              const int j2 = j + kParts * kWarps;
              const bool two = j2 < n;
              const C64* a = A + (long long)j * lda + r0 + lane;
              const C64* b = two ? a + (long long)kParts * kWarps * lda : a;
              C64 au[U], bu[U];
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const bool in = r0 + 32 * u + lane < n;
                au[u] = in ? a[32 * u] : cxzero<double>();
                bu[u] = in && two ? b[32 * u] : cxzero<double>();
              }
              const C64 va = v[j], vb = two ? v[j2] : cxzero<double>();
              C64 da = cxzero<double>(), db = cxzero<double>();
#pragma unroll
              for (int u = 0; u < U; ++u) {
                y[u] = fmac(au[u], va, y[u]);
                if (r0 + 32 * u + 31 > k) da = fmac_conj(vu[u], au[u], da);
              }
              if (two) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                  y[u] = fmac(bu[u], vb, y[u]);
                  if (r0 + 32 * u + 31 > k) db = fmac_conj(vu[u], bu[u], db);
                }
              }
              const double s = sum_pair(da, db);
              if (lane < (two ? 4 : 2)) {
                double* zj = reinterpret_cast<double*>(z + (lane < 2 ? j : j2)) + (lane & 1);
                *zj = r0 == 0 ? s : *zj + s;
              }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) yw[(p * kWarps + warp) * ROWS + 32 * u + lane] = y[u];
          }
          __syncthreads();
          for (int e = tid; e < np * ROWS; e += kThreads) {
            const int p = e / ROWS, r = e % ROWS;
            if (r0 + r < n) {
              C64 s = yw[p * kWarps * ROWS + r];
#pragma unroll
              for (int w = 1; w < kWarps; ++w) s = s + yw[(p * kWarps + w) * ROWS + r];
              send(yp + ((int)rank + (p0 + p) * (int)ctas) * n + r0 + r, s, ctas);
            }
          }
          // c's part: sum of z_j v_j, one warp a part
          if (r0 + ROWS >= n && warp < np) {
            const int part = (int)rank + (p0 + warp) * (int)ctas;
            C64 s = cxzero<double>();
            for (int j = part + kParts * lane; j < n; j += kParts * 32)
              if (j > k) s = fmac(z[j], v[j], s);
            const double r = sum_pair(s, s);
            const double im = __shfl_sync(0xffffffffu, r, 1);
            if (lane == 0) send(cpart + part, cxmk<double>(r, im), ctas);
          }
          __syncthreads();
        }
      }
      qr::barrier_all(ctas);
      for (int r = tid; r < n; r += kThreads) {
        C64 s = yp[r];
#pragma unroll
        for (int p = 1; p < kParts; ++p) s = s + yp[p * n + r];
        yp[r] = s;
      }
      C64 c = cpart[lane & (kParts - 1)];
#pragma unroll
      for (int off = 1; off < kParts; off <<= 1) { c.x += qr::shx(c.x, off); c.y += qr::shx(c.y, off); }
      const C64 tc = t * c;
      __syncthreads();
      // the warp's columns, 32 at a time: lane l has the coefficients of column l of them
      for (int p = 0; p < mine; ++p) {
        const int part = (int)rank + p * (int)ctas, first = part + kParts * warp;
        for (int g = first; g < n; g += 32 * kParts * kWarps) {
          const int jl = g + lane * kParts * kWarps;
          C64 a1 = cxzero<double>(), a2 = a1;
          if (jl > k && jl < n) {
            const C64 vc = cxconj(v[jl]);
            a1 = t * vc;
            a2 = cxconj(t) * nmac(tc, vc, z[jl]);
          }
          for (int q = 0; q < 32; ++q) {
            const int j = g + q * kParts * kWarps;
            if (j >= n) break;
            if (j <= k) continue;
            const C64 c1 = shf(a1, q), c2 = shf(a2, q);
            for (int r0 = 0; r0 < n; r0 += ROWS) {
              C64* a = A + (long long)j * lda + r0 + lane;
              C64 au[U];
#pragma unroll
              for (int u = 0; u < U; ++u)
                if (r0 + 32 * u + lane < n) au[u] = a[32 * u];
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const int r = r0 + 32 * u + lane;
                if (r0 + 32 * u >= n) continue;
                const int rr = r < n ? r : n - 1;
                au[u] = nmac(yp[rr], c1, au[u]);
                if (r0 + 32 * u + 31 > k) au[u] = nmac(v[rr], c2, au[u]);
                if (r < n) a[32 * u] = au[u];
              }
            }
            if (j == k + 1 && k + 3 < n) next_reflector(A, n, lda, k + 1, tau, sv + ((k + 1) & 1) * n, meta + ((k + 1) & 1), ctas);
          }
        }
      }
    } else if (k + 3 < n && (k + 1) % kParts % (int)ctas == (int)rank && (k + 1) / kParts % kWarps == warp) {
      next_reflector(A, n, lda, k + 1, tau, sv + ((k + 1) & 1) * n, meta + ((k + 1) & 1), ctas);
    }
    qr::barrier_all(ctas);
  }
}

// G columns a warp, U rows a lane: n <= 32 U. Reads the reflectors below A's subdiagonal.
template <int U, int G>
__global__ void __launch_bounds__(128) unghr64_kernel(const C64* __restrict__ Aall, int n, int lda, long long a_bs,
                                                      const C64* __restrict__ tau_all, C64* __restrict__ Zall, int ldz,
                                                      long long z_bs) {
  const C64* A = Aall + blockIdx.y * a_bs;
  const C64* tau = tau_all + (long long)blockIdx.y * n;
  C64* Z = Zall + blockIdx.y * z_bs;
  const int lane = threadIdx.x & 31, warps = gridDim.x * 4;
  for (int p = blockIdx.x * 4 + (threadIdx.x >> 5); G * p < n; p += warps) {
    const int j1 = n - 1 - G * p;                       // the group's last column; the one before (G = 2) may be -1
    C64 z[G][U], v[U], nv[U];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
      for (int u = 0; u < U; ++u) z[g][u] = lane + 32 * u == j1 - g ? cxone<double>() : cxzero<double>();
    auto load = [&](int k, C64 (&x)[U]) {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = lane + 32 * u;
        x[u] = i == k + 1 ? cxone<double>() : cxzero<double>();
        if (i > k + 1 && i < n) x[u] = A[i + (long long)k * lda];
      }
    };
    int k = min(n - 3, j1 - 1);
    C64 nt = cxzero<double>();
    if (k >= 0) { load(k, nv); nt = tau[k]; }
    for (; k >= 0; --k) {
      const C64 t = nt;
#pragma unroll
      for (int u = 0; u < U; ++u) v[u] = nv[u];
      if (k > 0) { load(k - 1, nv); nt = tau[k - 1]; }
      if (t.x == 0.0 && t.y == 0.0) continue;
      C64 d[G];
#pragma unroll
      for (int g = 0; g < G; ++g) d[g] = cxzero<double>();
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (32 * u + 31 > k)
#pragma unroll
          for (int g = 0; g < G; ++g) d[g] = fmac_conj(v[u], z[g][u], d[g]);
      // lanes 0 .. 3 of every four: the sums' components, then those of t times them
      const double s = sum_pair(d[0], d[G - 1]), o = qr::shx(s, 1);
      const double f = fma(t.x, s, (lane & 1) ? t.y * o : -t.y * o);
      C64 fg[G];
#pragma unroll
      for (int g = 0; g < G; ++g)
        fg[g] = cxmk<double>(__shfl_sync(0xffffffffu, f, 2 * g), __shfl_sync(0xffffffffu, f, 2 * g + 1));
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (32 * u + 31 > k)
#pragma unroll
          for (int g = 0; g < G; ++g) z[g][u] = nmac(v[u], fg[g], z[g][u]);
    }
#pragma unroll
    for (int g = 0; g < G; ++g)
      if (j1 - g >= 0)
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (lane + 32 * u < n) Z[lane + 32 * u + (long long)(j1 - g) * ldz] = z[g][u];
  }
}

}  // namespace hrd
}  // namespace wb
