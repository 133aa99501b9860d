// Bodies of the scale and digit stages of the slice-digit form, shared by the
// single-problem kernels (slice_tc.cu) and the batched kernels
// (batched_stages.cu).  See slice_tc.cu for what each stage computes.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

#include "slice_common.cuh"
#include "slice_tc.cuh"

namespace mdgi {

// ------------------------------------------------------------ exponents --
__device__ __forceinline__ unsigned long long umax64(unsigned long long a, unsigned long long b) {
  return a > b ? a : b;
}

// sum_l |x_l| of one entry (FP64 additions in limb order), as its bit
// pattern: maxima of non-negative doubles are taken as 64-bit unsigned
// integers, which orders them like the doubles and keeps the reductions off
// the FP64 pipe (narrow on this GPU).  A NaN sum counts as 0, so that a
// maximum skips it as a floating-point comparison would.
template <int P>
__device__ __forceinline__ unsigned long long abs_sum_bits(const double (&x)[P]) {
  double v = fabs(x[0]);
#pragma unroll
  for (int l = 1; l < P; ++l) v = v + fabs(x[l]);
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return b > 0x7ff0000000000000ull ? 0ull : b;
}

// An entry's P limbs; wide: 16-byte aligned.
template <int P>
__device__ __forceinline__ void load_entry(const double *__restrict__ p, bool wide,
                                           double (&x)[P]) {
  if (wide) {
#pragma unroll
    for (int l = 0; l < P; l += 2) {
      const double2 t = __ldg(reinterpret_cast<const double2 *>(p + l));
      x[l] = t.x;
      x[l + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int l = 0; l < P; ++l) x[l] = __ldg(p + l);
  }
}

// Largest entry of `count` at p, p + step, .. : loads of about 16 doubles are
// issued together.  With one entry at a time and 8-byte loads the stage
// waited for DRAM: qd 1024^3 35 -> 21 us for both operands, dd 16001 x 96 x
// 3001 227 -> 139 us, qd 8192^3 1104 -> 811 us (5.3 TB/s).
template <int P>
__device__ __forceinline__ unsigned long long strided_max(const double *__restrict__ p,
                                                          size_t step, int count, bool wide) {
  constexpr int N = P >= 16 ? 1 : 16 / P;
  unsigned long long mx = 0;
  int i = 0;
  for (; i + N <= count; i += N) {
    double x[N][P];
#pragma unroll
    for (int e = 0; e < N; ++e) load_entry<P>(p + (i + e) * step, wide, x[e]);
#pragma unroll
    for (int e = 0; e < N; ++e) mx = umax64(mx, abs_sum_bits<P>(x[e]));
  }
  for (; i < count; ++i) {
    double x[P];
    load_entry<P>(p + i * step, wide, x);
    mx = umax64(mx, abs_sum_bits<P>(x));
  }
  return mx;
}

__device__ __forceinline__ unsigned long long strided_max(int P, const double *p, size_t step,
                                                          int count, bool wide) {
  switch (P) {
    case 2: return strided_max<2>(p, step, count, wide);
    case 4: return strided_max<4>(p, step, count, wide);
    case 8: return strided_max<8>(p, step, count, wide);
    default: return strided_max<16>(p, step, count, wide);
  }
}

// The rows of A are taken a warp each, the columns of B 8 to a block, so
// that a stage writes every maximum once: no atomics, nothing cleared first.
constexpr int SCALE_THREADS = 256, SCALE_ROWS = SCALE_THREADS / 32, SCALE_COLS = 8;

__device__ __forceinline__ bool wide_entries(const double *X) {
  return reinterpret_cast<uintptr_t>(X) % 16 == 0;
}

// Largest entry of row r over the columns [c0, c1), in every lane.
__device__ __forceinline__ unsigned long long row_max(int P, const double *__restrict__ X, int ldx,
                                                      int r, int c0, int c1) {
  const int c = c0 + (int)(threadIdx.x & 31);
  unsigned long long mx = strided_max(P, X + ((size_t)r * ldx + c) * P, (size_t)32 * P,
                                      c < c1 ? (c1 - c + 31) / 32 : 0, wide_entries(X));
#pragma unroll
  for (int o = 16; o; o >>= 1) mx = umax64(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  return mx;
}

// Largest entry of column c0 + (thread % 8) over the rows [r0, r1), valid in
// the block's first 8 threads.  A warp reads four rows of 8 adjacent entries.
__device__ __forceinline__ unsigned long long col_max(int P, const double *__restrict__ X, int ldx,
                                                      int c0, int cols, int r0, int r1) {
  __shared__ unsigned long long part[SCALE_THREADS / 32][SCALE_COLS];
  const int c = c0 + (int)(threadIdx.x & 7), r = r0 + (int)(threadIdx.x >> 3);
  const int lanes = SCALE_THREADS / 8;
  const int count = c < cols && r < r1 ? (r1 - r + lanes - 1) / lanes : 0;
  unsigned long long mx = strided_max(P, X + ((size_t)r * ldx + c) * P, (size_t)lanes * ldx * P,
                                      count, wide_entries(X));
#pragma unroll
  for (int o = 8; o < 32; o <<= 1) mx = umax64(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) < SCALE_COLS) part[threadIdx.x >> 5][threadIdx.x & 7] = mx;
  __syncthreads();
  if (threadIdx.x < SCALE_COLS)
#pragma unroll
    for (int w = 1; w < SCALE_THREADS / 32; ++w) mx = umax64(mx, part[w][threadIdx.x]);
  return mx;
}

// --------------------------------------------------------------- digits --
constexpr int DIGIT_THREADS = 128;

// 32-bit words of an entry's integer V: the s - 1 low digits, then the 32
// bits that the leading digit is read from.
__host__ __device__ inline int digit_words(int s) { return (s - 1) / 4 + 2; }
__host__ __device__ inline int digit_smem(int s, int V) {
  return digit_words(s) * V * DIGIT_THREADS * 8;
}

// One operand: X rows x cols (trans: cols x rows), E its rows' exponents,
// digit planes of rows x ld_out, of which cols_pad columns are written (the
// ones from cols on with zeros).
struct DigitSide {
  const double *X;
  const int *E;
  __nv_bfloat16 *planes;
  int ldx, trans, rows, cols, ld_out, cols_pad;
  long long plane_stride;
};

// Digit rows that neighbouring threads take together: in a transposed operand
// the entries of one k lie side by side along the rows, up to four of them in
// a 128-byte line, which a row per 128 threads fetched for each of them.  (A
// warp then stores 32 bytes of each row of a plane: eight rows, for P = 2,
// would be half sectors.)  Both operands: qd 1024^3 53 -> 45 us, qd 8192^3
// 3.06 -> 2.6 ms, od 2048^3 393 -> 353 us.
__host__ __device__ inline int digit_row_shift(int P, int trans) {
  return !trans || P == 16 ? 0 : P == 8 ? 1 : 2;  // log2 of their number
}

// Threads of a side whose rows take `groups` groups of k-positions each, and
// the row and group of thread e.
__host__ __device__ inline long long digit_threads(int P, int trans, int rows, int groups) {
  const int shift = digit_row_shift(P, trans);
  return (((long long)rows + (1 << shift) - 1) >> shift << shift) * groups;
}
__device__ __forceinline__ void digit_place(int P, int trans, long long e, int groups, int &row,
                                            int &group) {
  const int shift = digit_row_shift(P, trans);
  const long long v = e >> shift;
  // (a 64-bit division is a hundred instructions)
  const int band = v >> 32 ? (int)(v / groups) : (int)((uint32_t)v / (uint32_t)groups);
  row = (band << shift) + ((int)e & ((1 << shift) - 1));
  group = (int)(v - (long long)band * groups);
}

// One thread: the digits of V adjacent entries (row, pc0 ..) of one side.
//
// V = sum_l floor(a_l 2^(S-E)) is collected in 32-bit pieces, one signed
// 64-bit sum per piece in shared memory: a limb touches the three pieces it
// covers and needs no carry, whatever the width.  One pass from the bottom
// then settles the carries.  Adding 128 at every digit but the leading one
// turns the balanced digits d in [-128, 127] into plain bytes d + 128, so the
// bytes of a piece need no carry among them either; byte b becomes BF16 by
// writing it into the significand of 2^23 and subtracting 2^23 + 128, and
// the top half of that float is d in BF16.
//
// Bound by the traffic, 8 P bytes in and 2 s out an entry.  With V's words in
// registers (positions unrolled, per width) most of the time went to
// instruction fetches and to 4 .. 16 carry steps a limb; both operands, so /
// from shared memory: qd 8192^3 4.96 / 3.06 ms (11.8 GB, 3.9 TB/s), od 2048^3
// 909 / 393 us, hd 1024 x 1024 x 512 880 / 116 us, dd 16001 x 96 x 3001 773 /
// 515 us, qd 256^3 26 / 8 us.
template <int V, int PL>
__device__ __forceinline__ void digits_group(int P, int s, const DigitSide &d, int row, int pc0,
                                             bool wide, void *smem) {
  constexpr int T = DIGIT_THREADS;
  const int words = digit_words(s);
  // piece j of entry v at acc[(j * V + v) * T]
  long long *acc = reinterpret_cast<long long *>(smem) + threadIdx.x;
  for (int j = 0; j < words * V; ++j) acc[j * T] = 0;
  const int base = 7 + 8 * (s - 1) - d.E[row];
  const double *a[V];
#pragma unroll
  for (int v = 0; v < V; ++v)
    a[v] = d.X + (d.trans ? (size_t)(pc0 + v) * d.ldx + row : (size_t)row * d.ldx + pc0 + v) * P;
  for (int l0 = 0; l0 < P; l0 += PL) {
    double x[V][PL];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (pc0 + v >= d.cols) {
#pragma unroll
        for (int l = 0; l < PL; ++l) x[v][l] = 0.0;
      } else if (wide) {
#pragma unroll
        for (int l = 0; l < PL; l += 2) {
          const double2 t = __ldg(reinterpret_cast<const double2 *>(a[v] + l0 + l));
          x[v][l] = t.x;
          x[v][l + 1] = t.y;
        }
      } else {
#pragma unroll
        for (int l = 0; l < PL; ++l) x[v][l] = __ldg(a[v] + l0 + l);
      }
    }
#pragma unroll
    for (int v = 0; v < V; ++v)
#pragma unroll
      for (int l = 0; l < PL; ++l) {
        int e2;
        int64_t m = exact_significand(x[v][l], e2);
        int q = e2 + base;
        if (q < 0) {
          m >>= q > -63 ? -q : 63;
          q = 0;
        }
        if (m == 0) continue;
        const int j = q >> 5, r = q & 31;
        const uint64_t lo = (uint64_t)m << r;
        const int64_t hi = r ? m >> (64 - r) : m >> 63;
        // pieces above the leading digit's 32 bits do not count
        long long *p = acc + (j * V + v) * T;
        if (j < words) p[0] += (uint32_t)lo;
        if (j + 1 < words) p[V * T] += (uint32_t)(lo >> 32);
        if (j + 2 < words) p[2 * V * T] += hi;
      }
  }
  __nv_bfloat16 *out = d.planes + (size_t)row * d.ld_out + pc0;
  long long carry[V];
#pragma unroll
  for (int v = 0; v < V; ++v) carry[v] = 0;
#pragma unroll 1
  for (int j = 0;; ++j) {
    const int low = min(s - 1 - 4 * j, 4);  // digits below the leading one in this piece
    const uint32_t offset = low > 0 ? 0x80808080u >> (8 * (4 - low)) : 0u;
    long long t[V];
#pragma unroll
    for (int v = 0; v < V; ++v) {
      t[v] = acc[(j * V + v) * T] + carry[v] + offset;
      carry[v] = t[v] >> 32;
    }
    __nv_bfloat16 *o = out + (s - 1 - 4 * j) * d.plane_stride;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      if (b >= low) continue;
      uint32_t f[V];
#pragma unroll
      for (int v = 0; v < V; ++v)
        f[v] = __float_as_uint(
            __int_as_float(__byte_perm((uint32_t)t[v], 0x4B000000u, 0x7440 | b)) - 8388736.0f);
      if constexpr (V == 2)
        *reinterpret_cast<uint32_t *>(o) = __byte_perm(f[0], f[1], 0x7632);
      else
        *reinterpret_cast<unsigned short *>(o) = (unsigned short)(f[0] >> 16);
      o -= d.plane_stride;
    }
    if (low < 4) {
      unsigned short top[V];
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const uint64_t above = (uint64_t)acc[((j + 1) * V + v) * T] << (32 - 8 * low);
        top[v] = __bfloat16_as_ushort(
            __float2bfloat16_rn((float)(int)(uint32_t)((uint64_t)(t[v] >> (8 * low)) + above)));
      }
      if constexpr (V == 2)
        *reinterpret_cast<uint32_t *>(out) = top[0] | (uint32_t)top[1] << 16;
      else
        *reinterpret_cast<unsigned short *>(out) = top[0];
      return;
    }
  }
}

}  // namespace mdgi
