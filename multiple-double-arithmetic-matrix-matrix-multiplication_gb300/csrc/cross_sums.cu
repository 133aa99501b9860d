// Sum planes of the cross form (cross_sums.cuh).
#include <algorithm>

#include <cuda_bf16.h>

#include "common.cuh"
#include "cross_sums.cuh"
#include "slice_tc.cuh"

namespace {

constexpr int SUM_WARPS = 8;
// 16-byte vectors of a digit row's window: at most 8 k-steps of 64 BF16
constexpr int MAX_WINDOW = 64;

// a + b of two BF16 pairs, exact for integers of magnitude <= 128 each
__device__ __forceinline__ uint32_t add_pair(uint32_t a, uint32_t b) {
  __nv_bfloat162 x, y;
  *reinterpret_cast<uint32_t *>(&x) = a;
  *reinterpret_cast<uint32_t *>(&y) = b;
  const __nv_bfloat162 z = __hadd2(x, y);
  return *reinterpret_cast<const uint32_t *>(&z);
}

__device__ __forceinline__ float add_squares(uint32_t z, float acc) {
  const float lo = __uint_as_float(z << 16), hi = __uint_as_float(z & 0xffff0000u);
  return __fmaf_rn(hi, hi, __fmaf_rn(lo, lo, acc));
}

// Block (x, y): digit row x (rows of A, then rows of B^T), window y of half a
// flush group (at most 512 k).  The row's window of every digit plane is
// staged in shared memory once; each warp then writes whole sum rows.
// Writing bounds it: 2 bytes out per sum against 2 digits in per D / 2 sums.
// qd 8192^3: 52.6 GB of sums in 11.6 ms (4.5 TB/s); qd 1024^3: 0.82 GB in
// 140 us, 6.2 TB/s of DRAM traffic.
// Digit rows lie `stride` vectors apart, the longest window's: with 64 for every
// size the 110 digits of a hexa-double row let two blocks on an SM (hd 1024 x 1024
// x 512 1272 us, 1022 now).
__global__ void __launch_bounds__(32 * SUM_WARPS)
    cross_sums_kernel(int s, int plo, int phi, int digits, int KB, int windows, int stride, int rows_a,
                      __nv_bfloat16 *dA, __nv_bfloat16 *dB, long long plane_a, long long plane_b,
                      unsigned *norms) {
  extern __shared__ uint4 digit_rows[];
  __shared__ unsigned warp_max[SUM_WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool side_b = (int)blockIdx.x >= rows_a;
  const int row = side_b ? (int)blockIdx.x - rows_a : (int)blockIdx.x;
  const long long plane = (side_b ? plane_b : plane_a) / 8;  // in vectors
  const int v0 = (int)blockIdx.y * KB / windows * 8, v1 = ((int)blockIdx.y + 1) * KB / windows * 8;
  const int nv = v1 - v0;
  uint4 *base = reinterpret_cast<uint4 *>(side_b ? dB : dA) + (size_t)row * KB * 8 + v0;

  for (int i = warp; i < digits; i += SUM_WARPS)
    for (int v = lane; v < nv; v += 32) {
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(digit_rows + i * stride + v);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst),
                   "l"(base + i * plane + v)
                   : "memory");
    }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  unsigned top = 0;
  for (int q = plo + warp; q < phi; q += SUM_WARPS) {
    // diagonal of sum q: the largest d with d^2 / 4 <= q (4 q + 3 is never
    // a square, so the rounded root has the right integer part)
    const int d = (int)sqrtf((float)(4 * q + 3));
    const int i = q - mdgi::cross_offset(d), j = d - i;
    const uint4 *xi = digit_rows + i * stride, *xj = digit_rows + j * stride;
    uint4 *out = base + (s + q - plo) * plane;
    float sq = 0.0f;  // at most 16 squares of 2^16 a lane: exact
    for (int v = lane; v < nv; v += 32) {
      const uint4 a = xi[v], b = xj[v];
      uint4 z;
      z.x = add_pair(a.x, b.x);
      z.y = add_pair(a.y, b.y);
      z.z = add_pair(a.z, b.z);
      z.w = add_pair(a.w, b.w);
      out[v] = z;
      sq = add_squares(z.w, add_squares(z.z, add_squares(z.y, add_squares(z.x, sq))));
    }
    top = max(top, __reduce_add_sync(0xffffffffu, (unsigned)sq));
  }
  if (lane == 0) warp_max[warp] = top;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < SUM_WARPS; ++w) top = max(top, warp_max[w]);
    unsigned *norm = norms + (side_b ? 1 : 0);
    if (top > *reinterpret_cast<volatile unsigned *>(norm)) atomicMax(norm, top);
  }
}

}  // namespace

namespace mdgi {

int launch_cross_sums(int s, int dlo, int dhi, int Kp, int rows_a, int rows_b, void *dA, void *dB,
                      long long plane_a, long long plane_b, unsigned *norms, cudaStream_t st) {
  const int KB = Kp / 64, windows = 2 * cross_groups(KB);
  // vectors of the longest window
  const int stride = (KB + windows - 1) / windows * 8;
  const int smem = dhi * stride * 16;
  MDG_TRY(allow_smem(cross_sums_kernel, smem, MAX_DIAGONALS * MAX_WINDOW * 16));
  cross_sums_kernel<<<dim3(rows_a + rows_b, windows), 32 * SUM_WARPS, smem, st>>>(
      s, cross_offset(dlo), cross_offset(dhi), dhi, KB, windows, stride, rows_a,
      reinterpret_cast<__nv_bfloat16 *>(dA), reinterpret_cast<__nv_bfloat16 *>(dB), plane_a,
      plane_b, norms);
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

}  // namespace mdgi
