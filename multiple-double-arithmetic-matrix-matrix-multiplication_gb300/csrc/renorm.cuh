// Renormalisation of diagonal sums to P limbs, shared by the single-problem
// and batched kernels (renorm.cu).
//
// W = sum_d C_d 256^(D-1-d), C_d the sum of diagonal d's chunk planes, is
// built from the least significant diagonal up, eight diagonals (two 32-bit
// pieces) per pass, and rounded to P limbs.  W lives in shared memory and the
// passes are a loop: with W in registers every word position had to be
// unrolled, and the code outgrew the instruction cache (registers / shared
// memory: dd 64 x 64 29 / 8 us, qd 256 x 256 49 / 14 us, dd 16001 x 96 142 /
// 58 us; the cross form of qd 8192 x 8192 16.3 / 6.8 ms).  It also makes the
// limb count and the width run-time numbers, so one kernel serves every P
// and one launch a whole batch (four launches before; 64 mixed problems of
// 32 .. 512: 3.84 -> 3.42 ms a call).
// Cutting limbs from 32-bit pieces with funnel shifts, from a bound on W's
// top bit down, instead of from 64-bit words: qd 1024^2, cross form, 90 -> 83
// us, od 2048^2 775 -> 693, hd 1024^2 583 -> 553, dd 16001 x 96 48 -> 42 us.
//
// In the cross form (cross_sums.cuh) the planes are the squares P_i and the
// chunks S of products of sums: a chunk holds the pairs i in [i0, i1) of
// diagonal d, and
//   sum over the chunk of A_i B_j + A_j B_i
//     = S - sum_{i0 <= i < i1} P_i - sum_{d-i1 < j <= d-i0} P_j   (mod 2^32),
// two differences of prefix sums Q_i = P_0 + .. + P_{i-1}; diagonal d has
// its chunks, and P_{d/2} for even d.  Where a chunk holds all pairs of its
// diagonal ("whole") that is S - Q_{d+1}, plus P_{d/2} for even d: Q_D is summed
// first and reduced by P_d after diagonal d, at the price of loading the squares
// again, which L2 then holds.
#pragma once

#include <stdint.h>

#include "cross_sums.cuh"
#include "slice_tc.cuh"

namespace mdgi {

constexpr int RENORM_THREADS = 128;

// Chunks of each diagonal, by value to a kernel.
struct ChunkCounts {
  unsigned of[128];
  int pairs_per_chunk;  // cross form
};

// Where renorm_columns has the chunk counts from: chunks of CHUNK_STEPS
// k-steps (a batch), a table, a table of the cross form, one with at most one
// chunk a diagonal.
enum { kPlainChunks = 0, kTableChunks = 1, kCrossChunks = 2, kCrossWhole = 3 };

// 32-bit pieces of W per column: the diagonals' (eight diagonals make two),
// the carry out of them (two), two of sign.
__host__ __device__ inline int renorm_pieces(int D) { return 2 * ((D + 7) / 8) + 4; }

// Shared memory of a block: W, and in the cross form the prefix sums.
__host__ __device__ inline int renorm_smem(int D, int V, bool cross) {
  return RENORM_THREADS * V * 4 * (renorm_pieces(D) + (cross ? D + 1 : 0));
}

// A bit position from which W is all sign: a diagonal is the sum of at most
// `terms` int32, and the diagonals' weights add up to less than 256/255 of the
// first one's.
inline int renorm_top(int D, int terms) {
  int bits = 0;
  while ((1 << bits) < terms) ++bits;
  return 8 * (D - 1) + 33 + bits;
}

// V adjacent int32.
template <int V>
struct Ints;
template <>
struct Ints<1> {
  using T = int;
  static __device__ __forceinline__ int get(T t, int) { return t; }
  static __device__ __forceinline__ T put(const int (&x)[1]) { return x[0]; }
};
template <>
struct Ints<2> {
  using T = int2;
  static __device__ __forceinline__ int get(T t, int v) { return v ? t.y : t.x; }
  static __device__ __forceinline__ T put(const int (&x)[2]) { return make_int2(x[0], x[1]); }
};

// 64 bits of W (piece i at w[i * STRIDE]) from bit pos.
template <int STRIDE>
__device__ __forceinline__ uint64_t bits64(const uint32_t *w, int pos) {
  const uint32_t *p = w + (pos >> 5) * STRIDE;
  const int r = pos & 31;
  const uint32_t a = p[0], b = p[STRIDE], c = p[2 * STRIDE];
  return (uint64_t)__funnelshift_r(b, c, r) << 32 | __funnelshift_r(a, b, r);
}

// The P limbs of W 2^scale: limb l is the residual R_l = W - (limbs 0..l-1),
// rounded to nearest-even to 53 bits.  W itself is never modified: after a
// limb rounded at bit sh, the residual is W's bits below sh with every bit
// from sh up equal to f, where f is all ones if that limb was rounded up and
// zero otherwise (rounding up leaves a negative remainder, rounding down a
// non-negative one, and |R| is below 2^sh either way).  So each limb needs:
// the highest bit t of R that differs from f (its magnitude), found 64 bits
// at a time from the cut h down, mostly at once; the 54 bits from t down,
// with f above; and whether any bit of W lies below them (the sticky bit,
// from W's lowest set bit lsb).  Bits of W from h up are f at the start.
// wide: out is 16-byte aligned and limbs leave in pairs.
template <int STRIDE>
__device__ __forceinline__ void emit_limbs(int P, const uint32_t *w, int h, int lsb, uint64_t f,
                                           int scale, double *out, bool wide) {
  double even = 0.0;
#pragma unroll 1
  for (int l = 0; l < P; ++l) {
    double val = 0.0;
    if (f != 0 || lsb < h) {  // else R = 0
      int t;
      for (;;) {
        const int b = h > 64 ? h - 64 : 0;
        uint64_t x = bits64<STRIDE>(w, b) ^ f;
        if (h < 64) x &= (1ull << h) - 1;
        if (x) {
          t = b + 63 - __clzll((long long)x);
          break;
        }
        if (b == 0) {
          t = -1;  // R = -1
          break;
        }
        h = b;
      }
      // rounding position sh; m = floor(R / 2^sh), |m| <= 2^53
      const int sh = t > 52 ? t - 52 : 0;
      int64_t m;
      bool up = false;
      if (sh > 0) {
        const uint64_t y = bits64<STRIDE>(w, sh - 1);
        const int64_t x = (int64_t)((y & ((1ull << 54) - 1)) | f << 54);
        m = x >> 1;
        up = (x & 1) && (lsb < sh - 1 || (m & 1));
      } else {
        const uint64_t keep = (2ull << t) - 1;  // t = -1: none
        m = (int64_t)((bits64<STRIDE>(w, 0) & (t < 0 ? 0ull : keep)) | (f & ~(t < 0 ? 0ull : keep)));
      }
      if (up) ++m;
      f = up ? ~0ull : 0ull;
      h = sh;
      // m 2^(sh + scale): with its top bit at 52, or 53 after rounding up,
      // and a normal exponent the bits are put together as integers (the
      // leading bit, and a carry into bit 53, add to the exponent field)
      const bool neg = m < 0;
      const uint64_t mm = neg ? (uint64_t)(-m) : (uint64_t)m;
      const int be = sh + scale + 52 + 1023;
      if (mm >> 52 && be >= 1 && be <= 2045) {
        const int hi = (int)(mm >> 32) + ((be - 1) << 20);
        val = __hiloint2double(neg ? hi | (int)0x80000000 : hi, (int)mm);
      } else {
        val = ldexp((double)mm, sh + scale);
        if (neg) val = -val;
      }
    }
    if (!wide)
      out[l] = val;
    else if (l & 1)
      *reinterpret_cast<double2 *>(out + l - 1) = make_double2(even, val);
    even = val;
  }
}

// val += c 2^(8 j) for |c| < 2^54, what would pass 2^63 into `up`, whose
// unit is 2^32.
__device__ __forceinline__ void add_at(long long &val, long long &up, long long c, int j) {
  if (j < 2) {
    val += (c & 0xffffff) * (1ll << (8 * j)) + (c >> 24) * (1ll << (24 + 8 * j));
  } else {
    val += (c & 0xffffff) * (1ll << (8 * j));
    up += (c >> 24) * (1ll << (8 * j - 8));
  }
}

// One thread: row r, columns c0 .. c0 + V - 1 (c0 < n) of one problem.
// planes: chunk planes in all.  top: renorm_top.  The sums of a pass are loaded together, the
// first chunks of each of its eight diagonals, so that the DRAM latency
// is paid once per eight to sixteen loads; in the cross form all D squares go
// to shared memory first, where the thread turns its own columns into prefix
// sums.
template <int V, int CHUNKS>
__device__ __forceinline__ void renorm_columns(int P, int s, int D, int KB, int planes, int top,
                                               int n,
                                               const ChunkCounts *counts,
                                               const int *__restrict__ chunks, long long plane_c,
                                               int ldcd, const int *__restrict__ E,
                                               const int *__restrict__ F, double *__restrict__ C,
                                               int ldc, int r, int c0, bool wide, void *smem) {
  using I = Ints<V>;
  using Vec = typename I::T;
  constexpr int T = RENORM_THREADS;
  constexpr bool CROSS = CHUNKS == kCrossChunks, WHOLE = CHUNKS == kCrossWhole;
  // chunks of a diagonal loaded ahead; four for small outputs (one column),
  // whose diagonals are cut into more chunks for the GEMM's sake
  constexpr int kAhead = CHUNKS == kTableChunks && V == 1 ? 4 : 2;
  const int dwords = (D + 7) / 8;
  // piece i of column v at W[(i * V + v) * T]; Q_i at Q[i * T]
  uint32_t *W = reinterpret_cast<uint32_t *>(smem) + threadIdx.x;
  Vec *Q = reinterpret_cast<Vec *>(reinterpret_cast<uint32_t *>(smem) + (2 * dwords + 4) * V * T) +
           threadIdx.x;
  const int *src = chunks + (size_t)r * ldcd + c0;
  const int ppc = CROSS ? counts->pairs_per_chunk : 0;
  if constexpr (CROSS) {
    for (int i = 0; i < D; ++i) {
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(Q + i * T);
      asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst),
                   "l"(src + (size_t)i * plane_c), "n"(4 * V)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    int run[V];
#pragma unroll
    for (int v = 0; v < V; ++v) run[v] = 0;
#pragma unroll 4
    for (int i = 0; i < D; ++i) {
      const Vec x = Q[i * T];
      Q[i * T] = I::put(run);
#pragma unroll
      for (int v = 0; v < V; ++v) run[v] = (int)((unsigned)run[v] + (unsigned)I::get(x, v));
    }
    Q[D * T] = I::put(run);
  }

  unsigned all[V];  // WHOLE: P_0 + .. + P_d of the diagonal at hand
#pragma unroll
  for (int v = 0; v < V; ++v) all[v] = 0;
  if constexpr (WHOLE) {
#pragma unroll 8
    for (int i = 0; i < D; ++i) {
      const Vec x = __ldcg(reinterpret_cast<const Vec *>(src + (size_t)i * plane_c));
#pragma unroll
      for (int v = 0; v < V; ++v) all[v] += (unsigned)I::get(x, v);
    }
  }

  long long carry[V];
  int lsb[V];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    carry[v] = 0;
    lsb[v] = 1 << 20;
  }
  int q = planes;  // the chunk planes of the diagonals above the current one start here
#pragma unroll 1
  for (int wi = 0; wi < dwords; ++wi) {
    Vec x0[8], x1[8], x2[kAhead > 2 ? 8 : 1], x3[kAhead > 2 ? 8 : 1];
    Vec p[WHOLE ? 8 : 1], mid[WHOLE ? 4 : 1];  // P_d; P_{d/2} of every other d
    int first[8], nc[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int d = D - 1 - (wi * 8 + b);
      nc[b] = d < 0 ? 0 : CHUNKS == kPlainChunks ? diag_chunks(d, s, KB) : (int)counts->of[d];
      q -= nc[b];
      first[b] = q;
      if (nc[b] > 0) x0[b] = __ldcs(reinterpret_cast<const Vec *>(src + (size_t)q * plane_c));
      if constexpr (WHOLE) {
        if (d >= 0) p[b] = __ldcg(reinterpret_cast<const Vec *>(src + (size_t)d * plane_c));
        if (d >= 0 && !(d & 1))
          mid[b >> 1] = __ldcg(reinterpret_cast<const Vec *>(src + (size_t)(d / 2) * plane_c));
      } else if (nc[b] > 1)
        x1[b] = __ldcs(reinterpret_cast<const Vec *>(src + (size_t)(q + 1) * plane_c));
      if constexpr (kAhead > 2) {
        if (nc[b] > 2)
          x2[b] = __ldcs(reinterpret_cast<const Vec *>(src + (size_t)(q + 2) * plane_c));
        if (nc[b] > 3)
          x3[b] = __ldcs(reinterpret_cast<const Vec *>(src + (size_t)(q + 3) * plane_c));
      }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      long long val[V], up[V];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        val[v] = carry[v];
        up[v] = 0;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int b = 4 * half + j, d = D - 1 - (wi * 8 + b);
        if (d < 0) continue;
        const long long unit = 1ll << (8 * j);
        if constexpr (WHOLE) {
          const bool even = !(d & 1);
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const int square = even ? I::get(mid[b >> 1], v) : 0;
            const unsigned sums = nc[b] ? (unsigned)I::get(x0[b], v) : 0u;
            val[v] += square * unit;
            val[v] += (int)(sums - all[v] + (unsigned)square) * unit;
            all[v] -= (unsigned)I::get(p[b], v);
          }
        } else if constexpr (CROSS) {
          const bool even = !(d & 1);
          int square[V];  // P_{d/2}
          if (even) {
            const Vec lo = Q[(d / 2) * T], hi = Q[(d / 2 + 1) * T];
#pragma unroll
            for (int v = 0; v < V; ++v) {
              square[v] = (int)((unsigned)I::get(hi, v) - (unsigned)I::get(lo, v));
              val[v] += square[v] * unit;
            }
          }
          if (nc[b] == 1) {  // all pairs: every P_i, i <= d, but the middle one
            const Vec all = Q[(d + 1) * T];
#pragma unroll
            for (int v = 0; v < V; ++v)
              val[v] += (int)((unsigned)I::get(x0[b], v) - (unsigned)I::get(all, v) +
                              (even ? (unsigned)square[v] : 0u)) *
                        unit;
            continue;
          }
          const int pairs = cross_pairs(d);
          for (int c = 0; c < nc[b]; ++c) {
            const int i0 = c * ppc, i1 = min(pairs, i0 + ppc);
            const Vec x = c == 0   ? x0[b]
                          : c == 1 ? x1[b]
                                   : __ldcs(reinterpret_cast<const Vec *>(
                                         src + (size_t)(first[b] + c) * plane_c));
            const Vec a0 = Q[i0 * T], a1 = Q[i1 * T];
            const Vec b0 = Q[(d - i1 + 1) * T], b1 = Q[(d - i0 + 1) * T];
#pragma unroll
            for (int v = 0; v < V; ++v) {
              const int t = (int)((unsigned)I::get(x, v) + (unsigned)I::get(a0, v) -
                                  (unsigned)I::get(a1, v) + (unsigned)I::get(b0, v) -
                                  (unsigned)I::get(b1, v));
              if (c < 2)
                val[v] += t * unit;
              else
                add_at(val[v], up[v], t, j);
            }
          }
        } else {
          // at most 2^31 2^24 each: the first four chunks of four diagonals
          // stay below 2^59
#pragma unroll
          for (int v = 0; v < V; ++v) {
            val[v] += I::get(x0[b], v) * unit;
            if (nc[b] > 1) val[v] += I::get(x1[b], v) * unit;
            if constexpr (kAhead > 2) {
              if (nc[b] > 2) val[v] += I::get(x2[b], v) * unit;
              if (nc[b] > 3) val[v] += I::get(x3[b], v) * unit;
            }
          }
          if (nc[b] > kAhead) {
            long long rest[V];
#pragma unroll
            for (int v = 0; v < V; ++v) rest[v] = 0;
            for (int c = kAhead; c < nc[b]; ++c) {
              const Vec x =
                  __ldcs(reinterpret_cast<const Vec *>(src + (size_t)(first[b] + c) * plane_c));
#pragma unroll
              for (int v = 0; v < V; ++v) rest[v] += I::get(x, v);
            }
#pragma unroll
            for (int v = 0; v < V; ++v) add_at(val[v], up[v], rest[v], j);
          }
        }
      }
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const uint32_t bits = (uint32_t)val[v];
        W[((2 * wi + half) * V + v) * T] = bits;
        if (bits && lsb[v] == 1 << 20) lsb[v] = 64 * wi + 32 * half + __ffs((int)bits) - 1;
        carry[v] = (val[v] >> 32) + up[v];
      }
    }
  }
  const int scale = E[r] - 14 - 8 * (D - 1);
#pragma unroll
  for (int v = 0; v < V; ++v) {
    uint32_t *above = W + (2 * dwords * V + v) * T;
    const uint32_t f = (uint32_t)(carry[v] >> 63);
    above[0] = (uint32_t)carry[v];
    above[V * T] = (uint32_t)(carry[v] >> 32);
    above[2 * V * T] = f;
    above[3 * V * T] = f;
    if (carry[v] && lsb[v] == 1 << 20) lsb[v] = 64 * dwords + __ffsll(carry[v]) - 1;
  }
#pragma unroll 1
  for (int v = 0; v < V; ++v) {
    if (c0 + v >= n) break;
    const int low = V == 2 && v ? lsb[V - 1] : lsb[0];
    const long long over = V == 2 && v ? carry[V - 1] : carry[0];
    emit_limbs<V * T>(P, W + v * T, top, low, (uint64_t)(over >> 63), scale + F[c0 + v],
                      C + ((size_t)r * ldc + c0 + v) * P, wide);
  }
}

}  // namespace mdgi
