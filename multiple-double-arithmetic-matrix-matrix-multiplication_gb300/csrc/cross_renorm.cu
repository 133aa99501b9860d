// Renormalisation of the cross form's output planes (cross_sums.cuh).
//
// The diagonal sums come back from the squares P_i and the chunks S of
// products of sums: a chunk holds pairs i in [i0, i1) of diagonal d, and
//   sum over the chunk of A_i B_j + A_j B_i
//     = S - sum_{i0 <= i < i1} P_i - sum_{d-i1 < j <= d-i0} P_j   (mod 2^32),
// two differences of prefix sums Q_i = P_0 + .. + P_{i-1}.  Diagonal d adds
// its chunks, and P_{d/2} for even d, in 64 bits; from there on it is the
// renormalisation of renorm_elems (slice_stages.cuh).
#include <algorithm>

#include "common.cuh"
#include "cross_sums.cuh"
#include "slice_common.cuh"
#include "slice_stages.cuh"
#include "slice_tc.cuh"

namespace {

constexpr int THREADS = 128;

// chunks of each diagonal, by value to the kernel
struct ChunkCounts {
  unsigned char of[128];
};

template <int V>
struct Ints;
template <>
struct Ints<1> {
  using T = int;
};
template <>
struct Ints<2> {
  using T = int2;
};

template <int V>
__device__ __forceinline__ void get(const typename Ints<V>::T &t, int (&x)[V]) {
  if constexpr (V == 2) {
    x[0] = t.x;
    x[1] = t.y;
  } else {
    x[0] = t;
  }
}

template <int V>
__device__ __forceinline__ typename Ints<V>::T put(const int (&x)[V]) {
  if constexpr (V == 2)
    return make_int2(x[0], x[1]);
  else
    return x[0];
}

// The P limbs of W 2^scale, as emit_limbs (slice_stages.cuh) rounds them, from
// W's words in shared memory (word i at w[i * stride], two words of sign
// above the last): the word that a limb's window starts in depends on the
// data, and shared memory takes a run-time index where registers would need
// a barrel shift over all words for every window.
template <int P>
__device__ __forceinline__ void emit_limbs_shared(const uint64_t *w, int stride, int top, int lsb,
                                                  uint64_t f, int scale, double *out, bool wide) {
  int h = top;  // bits of the residual from h up all equal f
  double even = 0.0;
#pragma unroll 1
  for (int l = 0; l < P; ++l) {
    double val = 0.0;
    if (f != 0 || lsb < h) {
      int b0, t;
      uint64_t lo, hi;
      for (;;) {
        b0 = h > 128 ? h - 128 : 0;
        const uint64_t *p = w + (b0 >> 6) * stride;
        const int r = b0 & 63;
        const uint64_t w0 = p[0], w1 = p[stride], w2 = p[2 * stride];
        lo = r ? ((w0 >> r) | (w1 << (64 - r))) : w0;
        hi = r ? ((w1 >> r) | (w2 << (64 - r))) : w1;
        const int cut = h - b0;  // 0..128: window bits from cut up are f
        if (cut < 64) {
          const uint64_t keep = cut ? ((1ull << cut) - 1) : 0ull;
          lo = (lo & keep) | (f & ~keep);
          hi = f;
        } else if (cut < 128) {
          const uint64_t keep = cut > 64 ? ((1ull << (cut - 64)) - 1) : 0ull;
          hi = (hi & keep) | (f & ~keep);
        }
        const uint64_t xh = hi ^ f, xl = lo ^ f;
        if (xh) {
          t = b0 + 127 - __clzll((long long)xh);
          break;
        }
        if (b0 == 0) {
          t = xl ? 63 - __clzll((long long)xl) : -1;
          break;
        }
        h = b0 + 64;
      }
      const int sh = t > 52 ? t - 52 : 0;
      uint64_t x;
      if (sh == 0) {
        x = lo << 1;
      } else {
        const int o = sh - 1 - b0;
        if (o < 64)
          x = o ? ((lo >> o) | (hi << (64 - o))) : lo;
        else
          x = o > 64 ? ((hi >> (o - 64)) | (f << (128 - o))) : hi;
      }
      const int64_t m = (int64_t)x >> 1;
      const bool up = sh > 0 && (x & 1ull) && (lsb < sh - 1 || (m & 1));
      const int64_t mr = up ? m + 1 : m;
      f = up ? ~0ull : 0ull;
      h = sh;
      const bool neg = mr < 0;
      const uint64_t mm = neg ? (uint64_t)(-mr) : (uint64_t)mr;
      const bool carry = mm >> 53;
      const uint64_t frac = carry ? (mm >> 1) : mm;
      const int be = sh + scale + 52 + (carry ? 1 : 0) + 1023;
      if ((frac >> 52) == 1 && be >= 1 && be <= 2046)
        val = __longlong_as_double((long long)(((uint64_t)be << 52) | (frac & ((1ull << 52) - 1))));
      else
        val = ldexp((double)mm, sh + scale);
      if (neg) val = -val;
    }
    if (!wide)
      out[l] = val;
    else if (l & 1)
      *reinterpret_cast<double2 *>(out + l - 1) = make_double2(even, val);
    even = val;
  }
}

// V adjacent columns per thread.  The squares go to shared memory (all D
// loads of a thread in flight at once), where each thread turns its own
// columns into prefix sums; the sums are loaded eight diagonals at a time,
// one 64-bit word of W per pass, so that the DRAM latency is paid once per
// eight to sixteen loads.  The pass is a loop and W lives in shared memory:
// unrolled over all words the code outgrew the instruction cache.  Unrolled /
// loop: qd 8192^3 16.3 / 6.7 ms (19.3 GB in, 2.1 GB out), qd 1024^3 258 / 94
// us, hd 1024 x 1024 x 512 1644 / 648 us.
template <int P, int NW, int V>
__global__ void __launch_bounds__(THREADS)
    cross_renorm_kernel(int D, int ppc, int planes, const __grid_constant__ ChunkCounts counts,
                        int m, int n, const int *__restrict__ out, long long plane_c, int ldcd,
                        const int *__restrict__ E, const int *__restrict__ F,
                        double *__restrict__ C, int ldc, int wide) {
  using Vec = typename Ints<V>::T;
  extern __shared__ int4 prefix_raw[];
  // word i of column v at W[(i * V + v) * THREADS]; Q_i at Q[i * THREADS]
  uint64_t *W = reinterpret_cast<uint64_t *>(prefix_raw) + threadIdx.x;
  Vec *Q = reinterpret_cast<Vec *>(reinterpret_cast<uint64_t *>(prefix_raw) +
                                   (NW + 2) * V * THREADS) + threadIdx.x;
  const int r = blockIdx.y, c0 = (blockIdx.x * THREADS + threadIdx.x) * V;
  if (c0 >= n) return;
  const int *src = out + (size_t)r * ldcd + c0;
  for (int i = 0; i < D; ++i) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(Q + i * THREADS);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst),
                 "l"(src + (size_t)i * plane_c), "n"(4 * V)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  {
    unsigned run[V];
#pragma unroll
    for (int v = 0; v < V; ++v) run[v] = 0;
#pragma unroll 4
    for (int i = 0; i < D; ++i) {
      int x[V], q[V];
      get<V>(Q[i * THREADS], x);
#pragma unroll
      for (int v = 0; v < V; ++v) {
        q[v] = (int)run[v];
        run[v] += (unsigned)x[v];
      }
      Q[i * THREADS] = put<V>(q);
    }
    int q[V];
#pragma unroll
    for (int v = 0; v < V; ++v) q[v] = (int)run[v];
    Q[D * THREADS] = put<V>(q);
  }

  long long T[V];
  int lsb[V];
#pragma unroll
  for (int v = 0; v < V; ++v) {
    T[v] = 0;
    lsb[v] = 64 * NW;
  }
  int q = planes;  // the chunk planes of the diagonals above the current one start here
#pragma unroll 1
  for (int wi = 0; wi * 8 < D - 1; ++wi) {
    // the first two chunks of the word's eight diagonals
    Vec x0[8], x1[8];
    int first[8];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int d = D - 1 - (wi * 8 + b);
      const int nc = d > 0 ? counts.of[d] : 0;
      q -= nc;
      first[b] = q;
      if (nc > 0) x0[b] = __ldcs(reinterpret_cast<const Vec *>(src + (size_t)q * plane_c));
      if (nc > 1) x1[b] = __ldcs(reinterpret_cast<const Vec *>(src + (size_t)(q + 1) * plane_c));
    }
    uint64_t word[V];
#pragma unroll
    for (int v = 0; v < V; ++v) word[v] = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int d = D - 1 - (wi * 8 + b);
      if (d > 0) {
        const int nc = counts.of[d];
        const int pairs = mdgi::cross_pairs(d);
        unsigned corr[V];  // what the squares add to the first chunk, negated
        {
          const int i1 = min(pairs, ppc);
          int a1[V], b0[V], b1[V];
          get<V>(Q[i1 * THREADS], a1);
          get<V>(Q[(d - i1 + 1) * THREADS], b0);
          get<V>(Q[(d + 1) * THREADS], b1);
          int s[V];
          get<V>(x0[b], s);
#pragma unroll
          for (int v = 0; v < V; ++v) {
            corr[v] = (unsigned)a1[v] + (unsigned)b1[v] - (unsigned)b0[v];
            T[v] += (int)((unsigned)s[v] - corr[v]);
          }
        }
        for (int c = 1; c < nc; ++c) {
          const int i0 = c * ppc, i1 = min(pairs, i0 + ppc);
          int s[V], a0[V], a1[V], b0[V], b1[V];
          if (c == 1)
            get<V>(x1[b], s);
          else
            get<V>(__ldcs(reinterpret_cast<const Vec *>(src + (size_t)(first[b] + c) * plane_c)),
                   s);
          get<V>(Q[i0 * THREADS], a0);
          get<V>(Q[i1 * THREADS], a1);
          get<V>(Q[(d - i1 + 1) * THREADS], b0);
          get<V>(Q[(d - i0 + 1) * THREADS], b1);
#pragma unroll
          for (int v = 0; v < V; ++v)
            T[v] += (int)((unsigned)s[v] - ((unsigned)a1[v] - (unsigned)a0[v]) -
                          ((unsigned)b1[v] - (unsigned)b0[v]));
        }
        if (!(d & 1)) {
          int lo[V], hi[V];
          get<V>(Q[(d / 2) * THREADS], lo);
          get<V>(Q[(d / 2 + 1) * THREADS], hi);
#pragma unroll
          for (int v = 0; v < V; ++v) T[v] += (int)((unsigned)hi[v] - (unsigned)lo[v]);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
          word[v] |= (uint64_t)(T[v] & 255) << (8 * b);
          T[v] >>= 8;
        }
      }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) {
      W[(wi * V + v) * THREADS] = word[v];
      if (word[v] && lsb[v] == 64 * NW)
        lsb[v] = 64 * wi + __ffsll((long long)word[v]) - 1;
    }
  }
  // diagonal 0 (the square of the leading digits), then T on top of the bytes
  {
    int p0[V];
    get<V>(Q[THREADS], p0);
#pragma unroll
    for (int v = 0; v < V; ++v) T[v] += p0[v];
  }
  const int at = 8 * (D - 1), aw = at >> 6, ar = at & 63;
  const int scale = E[r] - 14 - at;
#pragma unroll 1
  for (int v = 0; v < V; ++v) {
    const int c = c0 + v;
    if (c >= n) break;
    long long t = T[0];
    int low = lsb[0];
    if (V == 2 && v == 1) {
      t = T[V - 1];
      low = lsb[V - 1];
    }
    uint64_t *w = W + v * THREADS;
    const uint64_t f = (uint64_t)(t >> 63);
    const uint64_t below = ar ? w[aw * V * THREADS] : 0ull;
    w[aw * V * THREADS] = below | (uint64_t)t << ar;
    w[(aw + 1) * V * THREADS] = ar ? (uint64_t)(t >> (64 - ar)) : f;
    w[(aw + 2) * V * THREADS] = f;
    w[(aw + 3) * V * THREADS] = f;
    if (low == 64 * NW && t) low = at + __ffsll(t) - 1;
    emit_limbs_shared<P>(w, V * THREADS, at + 64, low, f, scale + F[c],
                         C + ((size_t)r * ldc + c) * P, wide);
  }
}

template <int P, int NW, int V>
int launch(int D, int KB, int m, int n, const int *out, long long plane_c, int ldcd, const int *E,
           const int *F, double *C, int ldc, cudaStream_t st) {
  const int ppc = mdgi::cross_pairs_per_chunk(KB);
  ChunkCounts counts{};
  for (int d = 1; d < D; ++d) counts.of[d] = (unsigned char)mdgi::cross_chunks(d, ppc);
  const int smem = (D + 1) * THREADS * V * 4 + (NW + 2) * V * THREADS * 8;
  MDG_TRY_CUDA(cudaFuncSetAttribute(cross_renorm_kernel<P, NW, V>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  cross_renorm_kernel<P, NW, V>
      <<<dim3(mdgi::ceil_div(mdgi::ceil_div(n, V), THREADS), m), THREADS, smem, st>>>(
          D, ppc, mdgi::cross_outputs(D, KB), counts, m, n, out, plane_c, ldcd, E, F, C, ldc,
          reinterpret_cast<uintptr_t>(C) % 16 == 0);
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

constexpr int kWords[4] = {4, 6, 10, 16};  // P = 2, 4, 8, 16

}  // namespace

namespace mdgi {

bool cross_renorm_supported(int p, int s, int D) {
  const int words = p == 2 ? kWords[0] : p == 4 ? kWords[1] : p == 8 ? kWords[2] : kWords[3];
  return D <= s && D >= 2 && D <= 127 && words_for(1, D) == words;
}

int launch_cross_renorm(int p, int D, int KB, int m, int n, const int *out, long long plane_c,
                        int ldcd, const int *E, const int *F, double *C, int ldc,
                        cudaStream_t st) {
  if (m == 0 || n == 0) return MDG_SUCCESS;
  switch (p) {
    case 2: return launch<2, 4, 2>(D, KB, m, n, out, plane_c, ldcd, E, F, C, ldc, st);
    case 4: return launch<4, 6, 2>(D, KB, m, n, out, plane_c, ldcd, E, F, C, ldc, st);
    case 8: return launch<8, 10, 2>(D, KB, m, n, out, plane_c, ldcd, E, F, C, ldc, st);
    case 16: return launch<16, 16, 1>(D, KB, m, n, out, plane_c, ldcd, E, F, C, ldc, st);
  }
  return MDG_ERROR_INVALID_LIMBS;
}

}  // namespace mdgi
