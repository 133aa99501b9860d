// Per-element / per-block bodies of the slice-digit stage kernels, shared
// by the single-problem kernels (slice_tc.cu) and the batched kernels
// (batched.cu).  See slice_tc.cu for what each stage computes.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

#include "slice_common.cuh"
#include "slice_tc.cuh"

namespace mdgi {

// ------------------------------------------------------------ exponents --
// sum_l |x_l| of one entry (FP64 additions in limb order), as its bit
// pattern: maxima of non-negative doubles are taken as 64-bit unsigned
// integers, which orders them like the doubles and keeps the reductions off
// the FP64 pipe (narrow on this GPU).  A NaN sum counts as 0, so that a
// maximum skips it as a floating-point comparison would.
__device__ __forceinline__ unsigned long long abs_sum_bits(const double *x, int P) {
  double v = fabs(x[0]);
  for (int l = 1; l < P; ++l) v = v + fabs(x[l]);
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  return b > 0x7ff0000000000000ull ? 0ull : b;
}
__device__ __forceinline__ unsigned long long umax64(unsigned long long a, unsigned long long b) {
  return a > b ? a : b;
}

// Block 32 x 8 covers 32 columns x 256 rows; each warp walks 32 rows of
// one 32-column strip.  Row maxima: warp reduction, one atomic per row per
// warp.  Column maxima: one atomic per thread.
__device__ __forceinline__ void absmax_block(int P, int R, int Cn, const double *__restrict__ X,
                                             int ldx, unsigned long long *rowbits,
                                             unsigned long long *colbits, int bx, int by) {
  const int c = bx * 32 + threadIdx.x;
  const int r0 = by * 256 + threadIdx.y * 32;
  unsigned long long cm = 0;
  for (int rr = 0; rr < 32; ++rr) {
    const int r = r0 + rr;
    if (r >= R) break;
    const unsigned long long v = c < Cn ? abs_sum_bits(X + ((size_t)r * ldx + c) * P, P) : 0ull;
    cm = umax64(cm, v);
    if (rowbits) {
      unsigned long long w = v;
#pragma unroll
      for (int o = 16; o; o >>= 1) w = umax64(w, __shfl_xor_sync(0xffffffffu, w, o));
      if (threadIdx.x == 0) atomicMax(rowbits + r, w);
    }
  }
  if (colbits && c < Cn) atomicMax(colbits + c, cm);
}

// --------------------------------------------------------------- digits --
// BF16 bits of an integer d in [-128, 127] without a conversion instruction
// (conversions run at a fraction of the FP32 rate): 2^23 + 128 + d written
// into the bit pattern of 2^23 is that integer as a float, and subtracting
// 2^23 + 128 in FP32 leaves d exactly; a float with at most 8 significant
// bits has its low 16 bits clear, so its top half is d in BF16.
__device__ __forceinline__ uint32_t bf16_bits_of_digit(int d) {
  const float f = __int_as_float(0x4B000000 + 128 + d) - 8388736.0f;
  return __float_as_uint(f) >> 16;
}

// One thread per element of the padded plane (prow, pcol); pcol (the k
// index) is the fastest, so plane stores are coalesced.  Outside the valid
// region every digit is zero.
template <int NW>
__device__ __forceinline__ void digits_elem(int P, int s, int rows, int cols,
                                            const double *__restrict__ X, int ldx,
                                            const int *__restrict__ E, int trans,
                                            __nv_bfloat16 *__restrict__ planes, int ld_out,
                                            long long plane_stride, int rows_pad, int cols_pad,
                                            int pr, int pc) {
  if (pc >= cols_pad || pr >= rows_pad) return;
  __nv_bfloat16 *out = planes + (size_t)pr * ld_out + pc;
  if (pr >= rows || pc >= cols) {
    for (int i = 0; i < s; ++i) out[i * plane_stride] = __float2bfloat16_rn(0.0f);
    return;
  }
  const double *a = trans ? X + ((size_t)pc * ldx + pr) * P : X + ((size_t)pr * ldx + pc) * P;
  const int S = 7 + 8 * (s - 1);
  const int Er = E[pr];
  uint64_t w[NW];
#pragma unroll
  for (int i = 0; i < NW; ++i) w[i] = 0;
  for (int l = 0; l < P; ++l) {
    int e2;
    const int64_t m = mdgi::exact_significand(a[l], e2);
    if (m == 0) continue;
    const int q = e2 + S - Er;
    if (q >= 0) {
      mdgi::wide_add_shifted<NW>(w, m, q);
    } else if (q > -64) {
      mdgi::wide_add_shifted<NW>(w, m >> (-q), 0);
    } else {
      mdgi::wide_add_shifted<NW>(w, m < 0 ? -1 : 0, 0);
    }
  }
  // balanced digits from the bottom: t = byte + carry, t >= 128 -> t - 256
  int carry = 0;
#pragma unroll
  for (int wi = 0; wi < NW; ++wi) {
    const uint64_t word = w[wi];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int p = wi * 8 + b;
      if (p < s - 1) {
        const int t = (int)((word >> (8 * b)) & 255) + carry;
        const int d = t >= 128 ? t - 256 : t;
        carry = t >= 128 ? 1 : 0;
        out[(s - 1 - p) * plane_stride] =
            __ushort_as_bfloat16((unsigned short)bf16_bits_of_digit(d));
      }
    }
  }
  const int top = (int)(int64_t)mdgi::wide_bits64<NW>(w, 8 * (s - 1)) + carry;
  out[0] = __float2bfloat16_rn((float)top);
}

// Four consecutive k-positions per thread: the same digits as digits_elem,
// written as one 8-byte vector (4 BF16) per plane.  pc0 is a multiple of 4;
// cols_pad, ld_out and plane_stride are multiples of 4.
template <int NW>
__device__ __forceinline__ void digits_elem4(int P, int s, int rows, int cols,
                                             const double *__restrict__ X, int ldx,
                                             const int *__restrict__ E, int trans,
                                             __nv_bfloat16 *__restrict__ planes, int ld_out,
                                             long long plane_stride, int rows_pad, int cols_pad,
                                             int pr, int pc0) {
  if (pc0 >= cols_pad || pr >= rows_pad) return;
  uint2 *out = reinterpret_cast<uint2 *>(planes + (size_t)pr * ld_out + pc0);
  const long long vstride = plane_stride / 4;
  if (pr >= rows || pc0 >= cols) {
    for (int i = 0; i < s; ++i) out[i * vstride] = make_uint2(0, 0);
    return;
  }
  const int S = 7 + 8 * (s - 1);
  const int Er = E[pr];
  uint64_t w[4][NW];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
#pragma unroll
    for (int i = 0; i < NW; ++i) w[e][i] = 0;
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int pc = pc0 + e;
    const double *a = trans ? X + ((size_t)pc * ldx + pr) * P : X + ((size_t)pr * ldx + pc) * P;
    for (int l = 0; l < P; ++l) {
      int e2;
      const int64_t m = pc < cols ? mdgi::exact_significand(a[l], e2) : 0;
      if (m == 0) continue;
      const int q = e2 + S - Er;
      if (q >= 0) {
        mdgi::wide_add_shifted<NW>(w[e], m, q);
      } else if (q > -64) {
        mdgi::wide_add_shifted<NW>(w[e], m >> (-q), 0);
      } else {
        mdgi::wide_add_shifted<NW>(w[e], m < 0 ? -1 : 0, 0);
      }
    }
  }
  int carry[4] = {0, 0, 0, 0};
#pragma unroll
  for (int wi = 0; wi < NW; ++wi) {
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int p = wi * 8 + b;
      if (p < s - 1) {
        uint32_t packed[2];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int t = (int)((w[e][wi] >> (8 * b)) & 255) + carry[e];
          const int d = t >= 128 ? t - 256 : t;
          carry[e] = t >= 128 ? 1 : 0;
          const uint32_t bits = bf16_bits_of_digit(d);
          if (e & 1) packed[e >> 1] |= bits << 16; else packed[e >> 1] = bits;
        }
        out[(s - 1 - p) * vstride] = make_uint2(packed[0], packed[1]);
      }
    }
  }
  uint32_t packed[2];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int top = (int)(int64_t)mdgi::wide_bits64<NW>(w[e], 8 * (s - 1)) + carry[e];
    const uint32_t bits = __bfloat16_as_ushort(__float2bfloat16_rn((float)top));
    if (e & 1) packed[e >> 1] |= bits << 16; else packed[e >> 1] = bits;
  }
  out[0] = make_uint2(packed[0], packed[1]);
}

}  // namespace mdgi
