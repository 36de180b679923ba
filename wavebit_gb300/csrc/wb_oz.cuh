// Complex FP64 products on the tensor cores of sm_103a (tcgen05, kind::f16), to FP64 accuracy.
//
// GB300 issues about two FP64 FMAs per clock and SM; its tensor cores have no FP64 kind but multiply
// small integers exactly. C = alpha op(A) op(B) + beta C therefore runs on exact slices (the splitting
// of Ozaki, Ogita, Oishi and Rump, "Error-free transformations of matrix multiplication", 2012, in its
// tensor-core form of Mukunoki, Ozaki, Ogita and Imamura, 2020):
//   - a row of A (a column of B) is scaled by the power of two of its largest entry to fixed point, by
//     integer operations on the doubles' bits, its largest entry in [2^61, 2^62), and cut into 8 balanced
//     digits of 8 bits, |d| <= 128, kept as FP16;
//   - the products of digit planes i and j with i + j = w < 8 go to one FP32 accumulator per w. K is
//     taken 64 complex (128 real) at a time, so an accumulator holds at most 8 x 128 products of at
//     most 2^14: integers up to 2^24, exact in FP32;
//   - the eight accumulators are put together as integers and rounded once to FP64.
//
// Operands graded along k (modes scaled by any factors against their inverse, the columns of U against the
// rows of a solution) would lose what lies far below a line's largest entry, though its partner is as far
// above: so each k of a tile's panel is first scaled by a power of two too, its column of A by 2^s and its row
// of B by 2^-s, with s half of how much further below their lines' largest the column's entries stay
// than the row's. The product of two lines' largest entries only falls by it. Powers of two on rows and columns
// change no bits; on a k (against its inverse) they move the error by a binary order at most.
//
// Error of a panel: an entry keeps 2^-62 of its scaled line's largest, the dropped pairs (w >= 8) are below
// 2^-57 of the two lines' largest a term, and the sum is rounded once. Where a line's entries, scaled so,
// stay within some four binary orders, that is below a chain of FP64 FMAs' error; beyond, the error is normwise:
// K 2^-56 of the two scaled lines' largest entries, not of each sum |a||b|. Subnormal entries and results count
// in full. An infinity or NaN in a row or column makes that row or column of C NaN.
//
// A complex product is one real product of twice the size, [Re -Im; Im Re] [Re; Im], so a CTA's 64 x 64
// complex tile is one 128 x 64 accumulator for each of 8 weights: all 512 columns of tensor memory.
//
// Per CTA (8 warps and a ninth that issues the MMAs): a pass over the K panel finds the scales; then, 16
// complex k at a time, warps 0..3 split A and warps 4..7 split B into the canonical no-swizzle
// K-major layout (two stages of 96 KB) while the MMAs of the chunk before run (36 pairs, 72 MMAs a
// chunk).
//
// What bounds it: a tile's own latencies. One CTA an SM (192 KB, all of tensor memory) takes about 17 us a
// tile of K = 64: the scales' pass, the splitting and the 288 MMAs (5 us alone), the eight accumulators'
// assembly, and C read and written; FP64 FMAs take 270 us. 450 x 450 x 64, 8 matrices, C read and written: 126 us
// (6.6 TFLOP/s), 121 without the k's scales; x 450 5% longer with them too; K = 31 the same with and without.
// Holding C's entries during the MMAs spills at 168 registers and was 10% slower.
// Every mbarrier wait is bounded, as in wb_tc.cuh.
#pragma once
#include "wb_tc.cuh"

namespace wb {
namespace oz {

constexpr int kT = 64;                 // complex rows and columns of a CTA's tile
constexpr int kKc = 16;                // complex k of a chunk (32 real: two MMA steps)
constexpr int kKp = 64;                // complex k of a panel: 8 * 2 * kKp * 2^14 = 2^24
constexpr int kDig = 8;
constexpr int kWorkers = 256, kThreads = kWorkers + 32;
constexpr int kPlaneA = 128 * 64, kPlaneB = 64 * 64;          // bytes: rows x 32 halves
constexpr int kStage = kDig * (kPlaneA + kPlaneB);
constexpr size_t kSmem = 2 * (size_t)kStage;
constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(kT >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);   // FP32 += FP16 x FP16

// byte offset of 8 halves (row, k = 8 kc ..) of a plane: 8-row x 16-byte cores, K-adjacent ones
// 128 bytes apart, 8-row groups 512
__device__ __forceinline__ uint32_t core_off(int row, int kc) {
  return (uint32_t)((row & 7) * 16 + (row >> 3) * 512 + kc * 128);
}

__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(kIdesc), "r"(acc));
}

// Exponents of lines and entries are kept with this added (0: none); kBad: an infinity or NaN in the line.
constexpr int kOff = 4096, kBad = 1 << 20;
// the shift of a k that contributes nothing (its column of A or row of B is zero)
constexpr int kDropped = -30000;

// The exponent of a complex entry's larger component, biased (subnormals' by their leading bit, down to -51),
// + kSub; 0 for zero, which stays below kSome under any shift, as no other entry does but a dropped one.
constexpr int kSub = 8192 + 64, kSome = 6144;
__device__ __forceinline__ int entry_exponent(double2 v) {
  const int hx = __double2hiint(v.x) & 0x7fffffff, hy = __double2hiint(v.y) & 0x7fffffff;
  const int e = max(hx, hy) >> 20;
  if (e) return e + kSub;
  const uint64_t b = ((uint64_t)(uint32_t)(hx | hy) << 32) | (uint32_t)(__double2loint(v.x) | __double2loint(v.y));
  return b ? kSub + 12 - __clzll((long long)b) : 0;
}

// x in fixed point for the biased exponent eb of its line's largest entry (x not scaled: eb less the k's
// shift), every byte biased by 128: byte 7 - i is digit i + 128
__device__ __forceinline__ uint64_t fixed_bytes(double x, int eb) {
  const int hi = __double2hiint(x), e = (hi >> 20) & 0x7ff;
  uint64_t m = ((uint64_t)((hi & 0xfffff) | (min(e, 1) << 20)) << 32) | (uint32_t)__double2loint(x);
  const int sh = max(e, 1) - eb + 9;
  if (sh < -54) m = 0;
  else if (sh >= 0) m <<= sh;
  else m = (m + (1ull << (-sh - 1))) >> -sh;
  const uint64_t q = hi < 0 ? 0ull - m : m;
  return q + 0x8080808080808080ull;
}

// the digits in byte b (0 lowest) of 8 words, as 8 FP16 numbers
__device__ __forceinline__ uint4 halves(const uint32_t* w, int b) {
  uint32_t o[4];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    uint32_t v = __byte_perm(w[2 * p], w[2 * p + 1], b | (b << 4) | ((b + 4) << 8) | ((b + 4) << 12));
    v = (v & 0x00ff00ffu) | 0x64006400u;                       // 1024 + byte
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(o[p]) : "r"(v), "r"(0x64806480u));   // - 1152
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ uint4 negated(uint4 v) {
  return make_uint4(v.x ^ 0x80008000u, v.y ^ 0x80008000u, v.z ^ 0x80008000u, v.w ^ 0x80008000u);
}

// m (its top bit set) of biased exponent e where that is no normal number's: subnormal, or infinite
__device__ __noinline__ double range_end(uint64_t m, int e, bool neg) {
  uint64_t bits = 0x7ffull << 52;
  if (e < 1) {
    const int drop = 12 - e;
    bits = drop > 64 ? 0 : (drop < 64 ? m >> drop : 0) + ((m >> (drop - 1)) & 1);
  }
  return __longlong_as_double((long long)(((uint64_t)neg << 63) | bits));
}

// sum over w of a[w] 256^(7 - w), times 2^(ea + eb) (biased exponents of the row and the column)
__device__ __forceinline__ double assemble(const float* a, int ea, int eb) {
  long long h = 0, l = 0;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    h = h * 256 + (long long)__float2int_rn(a[w]);
    l = l * 256 + (long long)__float2int_rn(a[w + 4]);
  }
  h += l >> 32;
  uint32_t lo = (uint32_t)l;
  const bool neg = h < 0;
  if (neg) {
    h = -h;
    if (lo) { h -= 1; lo = 0u - lo; }
  }
  int shift = 0;
  if (h == 0) { h = (long long)lo; lo = 0; shift = 32; }
  if (h == 0) return 0.0;
  const int n = __clzll(h);
  uint64_t m = (uint64_t)h << n;
  m |= n >= 32 ? (uint64_t)lo << (n - 32) : (uint64_t)lo >> (32 - n);
  int e = ea + eb - n - 994 - shift;
  uint64_t r = (m >> 11) + ((m >> 10) & 1);                    // 53 bits, rounded
  const int up = (int)(r >> 53);
  if ((unsigned)(e + up - 1) >= 2046u) return range_end(m, e, neg);
  const uint64_t bits = ((uint64_t)neg << 63) | ((uint64_t)(e + up) << 52) | ((r >> up) & 0xfffffffffffffull);
  return __longlong_as_double((long long)bits);
}

__device__ unsigned int g_oz_error;

struct Args {
  int m, n, k;
  double alpha, beta;
  const double2 *A, *B;
  double2* C;
  long long a_rs, a_cs, a_bs, b_rs, b_cs, b_bs, c_rs, c_cs, c_bs;
  const int* a_idx;
  int conj_a, conj_b;
};

__global__ void __launch_bounds__(kThreads) zgemm_kernel(const Args g) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ uint64_t bars[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int s_fail[3];                                    // thread 0's wait ran out: by a chunk's buffer, a panel's end
  __shared__ int s_top[2 * kT], s_line[2 * kT];                // the lines' exponents before and after the k's shifts
  __shared__ int s_k[2 * kT];                                  // a k's largest entry, against its line's largest
  __shared__ __align__(16) short s_shift[2 * kT];              // its shift
  __shared__ __align__(16) short s_half[2 * kT];               // the same, even k before odd ones
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool issuer = warp == 8;
  const int row0 = blockIdx.x * kT, col0 = blockIdx.y * kT;
  const double2* A = g.A + (g.a_idx ? (long long)g.a_idx[blockIdx.z] : (long long)blockIdx.z) * g.a_bs;
  const double2* B = g.B + blockIdx.z * g.b_bs;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(&tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    tc::mbar_init(&bars[0]);
    tc::mbar_init(&bars[1]);
    asm volatile("fence.mbarrier_init.release.cluster;");
    s_fail[0] = s_fail[1] = s_fail[2] = 0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_slot;

  // a worker's line: row row0 + line of A (threads 0 .. 127) or column col0 + line of B, halves of a chunk
  const bool onB = tid >= 128;
  const int line = tid & 63, part = (tid >> 6) & 1;
  const long long ls = onB ? g.b_cs : g.a_rs, ks = onB ? g.b_rs : g.a_cs;
  const bool live = !issuer && (onB ? col0 + line < g.n : row0 + line < g.m);
  const double2* src = onB ? B + (long long)(col0 + line) * ls : A + (long long)(row0 + line) * ls;
  const int side = onB ? kT : 0;
  const bool flip = (onB ? g.conj_b : g.conj_a) != 0;

  // an accumulator row (real or imaginary part of a complex row) and 32 columns a thread
  const int arow = (warp & 3) * 32 + lane, acol0 = (warp >> 2) * 32;
  double acc[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) acc[j] = 0.0;

  uint32_t uses = 0;                    // chunks staged so far: buffer uses & 1, its use uses >> 1
  bool ok = true;
  for (int p0 = 0; p0 < g.k && ok; p0 += kKp) {
    const int kk = min(kKp, g.k - p0), nchunk = (kk + kKc - 1) / kKc;
    // the panel's scales: the lines' largest entries, the k's shifts, the lines' largest with them
    if (tid < 2 * kT) s_top[tid] = s_line[tid] = s_k[tid] = 0;
    __syncthreads();
    // this thread's 32 exponents, two a word, in the stages' memory (their last readers were waited for)
    uint32_t* ex = reinterpret_cast<uint32_t*>(smem) + tid;
    const int tk = kk > 32 ? 32 : 16;
    int top = 0;
    bool bad = false;
    if (!issuer) {
      // (q = part, part + 2, ..: the two halves of a line read its sectors together)
#pragma unroll 1
      for (int t = 0; t < tk; t += 4) {
        double2 w[4];
        uint32_t e[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int q = part + 2 * (t + u);
          w[u] = make_double2(0.0, 0.0);
          if (live && q < kk) w[u] = src[(p0 + q) * ks];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          int x = entry_exponent(w[u]);
          if (x == 0x7ff + kSub) { bad = true; x = 0; }
          top = max(top, x);
          e[u] = (uint32_t)x;
        }
        ex[kWorkers * (t / 2)] = e[0] | e[1] << 16;
        ex[kWorkers * (t / 2 + 1)] = e[2] | e[3] << 16;
      }
      if (top) atomicMax(&s_top[side + line], top);
    }
    __syncthreads();
    if (!issuer) {
      // the largest of the warp's 32 lines for each of its k, 16 at a time: pairs of 16 bits, halved from lane to
      // lane until a lane holds one pair
      const int own = s_top[side + line];
      const uint32_t base = own ? (uint32_t)(kSub + kOff - own) * 0x10001u : 0u;
#pragma unroll 1
      for (int t0 = 0; t0 < tk; t0 += 16) {
        uint32_t w[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) w[t] = ex[kWorkers * (t0 / 2 + t)] + base;
#pragma unroll
        for (int h = 4, bit = 1; h >= 1; h >>= 1, bit <<= 1)
#pragma unroll
          for (int t = 0; t < h; ++t) {
            const bool up = lane & bit;
            const uint32_t give = up ? w[t] : w[t + h], keep = up ? w[t + h] : w[t];
            w[t] = __vmaxu2(keep, __shfl_xor_sync(0xffffffffu, give, bit));
          }
        w[0] = __vmaxu2(w[0], __shfl_xor_sync(0xffffffffu, w[0], 8));
        w[0] = __vmaxu2(w[0], __shfl_xor_sync(0xffffffffu, w[0], 16));
        const int t = t0 + (((lane & 1) << 3) | ((lane & 2) << 1) | ((lane & 4) >> 1) | (lane >> 4));
        const int m = (int)(lane >> 4 ? w[0] >> 16 : w[0] & 0xffffu);
        if (m >= kSub && !(lane & 8)) atomicMax(&s_k[side + part + 2 * t], m);
      }
    }
    __syncthreads();
    if (tid < kT) {
      const int a = s_k[tid], b = s_k[kT + tid], h = (b - a) >> 1;
      const int at = (tid & 1) * 32 + (tid >> 1);
      s_shift[tid] = s_half[at] = (short)(a && b ? h : kDropped);
      s_shift[kT + tid] = s_half[kT + at] = (short)(a && b ? -h : kDropped);
    }
    __syncthreads();
    if (!issuer) {
      uint32_t most = (uint32_t)(kDropped & 0xffff) * 0x10001u;
#pragma unroll 1
      for (int t = 0; t < tk; t += 8) {
        const uint4 sv = *reinterpret_cast<const uint4*>(s_half + side + part * 32 + t);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          most = __viaddmax_s16x2(ex[kWorkers * (t / 2 + u)], u == 0 ? sv.x : u == 1 ? sv.y : u == 2 ? sv.z : sv.w, most);
      }
      int mx = max((int)(short)most, (int)most >> 16);
      mx = mx >= kSome ? mx - kSub + kOff : 0;
      if (bad) mx = kBad;
      if (mx > 0) atomicMax(&s_line[side + line], mx);
    }
    __syncthreads();
    const int eb = issuer ? 0 : s_line[side + line] - kOff;
    double2 v[8];
    uint4 shift;                                               // of the 8 k, 16 bits each
    auto load = [&](int c) {
      shift = *reinterpret_cast<const uint4*>(s_shift + side + c * kKc + part * 8);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int q = c * kKc + part * 8 + u;
        v[u] = make_double2(0.0, 0.0);
        if (live && q < kk) v[u] = src[(p0 + q) * ks];
      }
    };
    if (!issuer) load(0);
    for (int c = 0; c < nchunk; ++c, ++uses) {
      const int buf = uses & 1;
      unsigned char* st = smem + buf * kStage;
      if (!issuer) {
        if (uses >= 2 && tid == 0 && !tc::mbar_wait(&bars[buf], ((uses >> 1) - 1) & 1)) s_fail[buf] = 1;
        // split: words of 4 digit bytes, high (digits 0..3) and low (4..7), of the 8 real and 8 imaginary parts
        uint32_t rh[8], rl[8], ih[8], il[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const uint32_t h = u < 2 ? shift.x : u < 4 ? shift.y : u < 6 ? shift.z : shift.w;
          const int ek = eb - ((u & 1) ? (int)h >> 16 : (int)(short)h);
          const uint64_t a = fixed_bytes(v[u].x, ek), b = fixed_bytes(flip ? -v[u].y : v[u].y, ek);
          rh[u] = (uint32_t)(a >> 32); rl[u] = (uint32_t)a;
          ih[u] = (uint32_t)(b >> 32); il[u] = (uint32_t)b;
        }
        if (c + 1 < nchunk) load(c + 1);
        asm volatile("bar.sync 1, 256;" ::: "memory");         // the workers' buffer is free
        if (onB) {
          unsigned char* pb = st + kDig * kPlaneA;
#pragma unroll
          for (int d = 0; d < kDig; ++d) {
            const uint4 re = halves(d < 4 ? rh : rl, 3 - (d & 3)), im = halves(d < 4 ? ih : il, 3 - (d & 3));
            *reinterpret_cast<uint4*>(pb + d * kPlaneB + core_off(line, part)) = re;
            *reinterpret_cast<uint4*>(pb + d * kPlaneB + core_off(line, part + 2)) = im;
          }
        } else {
#pragma unroll
          for (int d = 0; d < kDig; ++d) {
            const uint4 re = halves(d < 4 ? rh : rl, 3 - (d & 3)), im = halves(d < 4 ? ih : il, 3 - (d & 3));
            unsigned char* pa = st + d * kPlaneA;
            *reinterpret_cast<uint4*>(pa + core_off(line, part)) = re;
            *reinterpret_cast<uint4*>(pa + core_off(line, part + 2)) = negated(im);
            *reinterpret_cast<uint4*>(pa + core_off(line + 64, part)) = im;
            *reinterpret_cast<uint4*>(pa + core_off(line + 64, part + 2)) = re;
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      __syncthreads();
      if (s_fail[buf]) { ok = false; break; }                  // (the next chunk's wait sets the other flag)
      if (issuer && lane == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        // descriptors differ by their start address alone (bits 0..13, in 16-byte units)
        const uint64_t da = tc::sdesc(tc::smem_u32(st)), db = tc::sdesc(tc::smem_u32(st) + kDig * kPlaneA);
#pragma unroll 1
        for (int j = 0; j < 2; ++j) {                          // K = 16 halves each
          const uint64_t ja = da + 16 * j, jb = db + 16 * j;
          const uint32_t first = (c > 0 || j > 0) ? 1u : 0u;
#pragma unroll
          for (int w = 0; w < kDig; ++w)
#pragma unroll
            for (int i = 0; i <= w; ++i)
              mma_f16(tmem + w * kT, ja + i * (kPlaneA / 16), jb + (w - i) * (kPlaneB / 16), i > 0 ? 1u : first);
        }
        tc::mma_commit(&bars[buf]);
      }
    }
    if (!ok) break;
    // the panel's MMAs are done: the last commit on each buffer
    if (tid == 0) {
      for (int b = 0; b < 2; ++b) {
        const uint32_t last = uses - 1 - ((uses - 1 - b) & 1);  // the latest chunk in buffer b
        if (uses > (uint32_t)b && !tc::mbar_wait(&bars[b], (last >> 1) & 1)) s_fail[2] = 1;
      }
    }
    __syncthreads();
    if (s_fail[2]) { ok = false; break; }
    asm volatile("tcgen05.fence::after_thread_sync;");
    if (!issuer) {
      const int ea = s_line[arow & 63];
#pragma unroll
      for (int c8 = 0; c8 < 32; c8 += 4) {
        float t[kDig][4];
#pragma unroll
        for (int w = 0; w < kDig; ++w) {
          const uint32_t addr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(w * kT + acol0 + c8);
          uint32_t r0, r1, r2, r3;
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                       : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                       : "r"(addr));
          t[w][0] = __uint_as_float(r0); t[w][1] = __uint_as_float(r1);
          t[w][2] = __uint_as_float(r2); t[w][3] = __uint_as_float(r3);
        }
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float a8[kDig];
#pragma unroll
          for (int w = 0; w < kDig; ++w) a8[w] = t[w][j];
          const int ec = s_line[kT + acol0 + c8 + j];
          double x = 0.0;
          if (ea == kBad || ec == kBad) x = NAN;
          else if (ea && ec) x = assemble(a8, ea - kOff, ec - kOff);
          acc[c8 + j] = p0 == 0 ? x : acc[c8 + j] + x;
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
  }
  if (tid == 0 && !ok) {
    // wait (bounded) for the MMAs still in flight before the tensor memory goes back
    for (int b = 0; b < 2; ++b)
      if (uses > (uint32_t)b) tc::mbar_wait(&bars[b], ((uses - 1 - ((uses - 1 - b) & 1)) >> 1) & 1);
    atomicAdd(&g_oz_error, 1u);
  }
  if (!issuer && ok) {
    const int gr = row0 + (arow & 63), comp = arow >> 6;
    if (gr < g.m) {
      double* out = reinterpret_cast<double*>(g.C + blockIdx.z * g.c_bs + gr * g.c_rs + (long long)(col0 + acol0) * g.c_cs) + comp;
      const long long step = 2 * g.c_cs;
      const int nc = min(32, g.n - col0 - acol0);
      const bool keep = g.beta != 0.0;
#pragma unroll
      for (int j0 = 0; j0 < 32; j0 += 8) {
        double old[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) old[j] = (keep && j0 + j < nc) ? out[(j0 + j) * step] : 0.0;
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (j0 + j < nc) {
            const double x = g.alpha == 1.0 ? acc[j0 + j] : g.alpha == -1.0 ? -acc[j0 + j] : g.alpha * acc[j0 + j];
            out[(j0 + j) * step] = !keep ? x : g.beta == 1.0 ? old[j] + x : fma(g.beta, old[j], x);
          }
      }
    }
  }
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

}  // namespace oz
}  // namespace wb
