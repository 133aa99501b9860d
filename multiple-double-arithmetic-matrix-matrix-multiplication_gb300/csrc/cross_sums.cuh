// Sum planes of the slice-digit GEMM ("cross" form of the diagonal sums).
//
// With digit planes A_0 .. A_{D-1}, B_0 .. B_{D-1} and P_i = A_i B_i^T, the
// two products of an unordered digit pair i < j come from one product of
// sums:
//   A_i B_j^T + A_j B_i^T = (A_i + A_j)(B_i + B_j)^T - P_i - P_j,
// so the D (D + 1) / 2 digit pairs of the diagonals d < D need D squares and
// floor(D^2 / 4) products of sums (quad-double: 224 instead of 406).  The
// sums lie in [-256, 256], which BF16 holds exactly.
//
// Order: sums of diagonal 1, 2, ..; within diagonal d = i + j by i.  Output
// planes of the diagonal GEMM: P_0 .. P_{D-1}, then per diagonal its pairs
// in chunks of pairs_per_chunk.  All int32 arithmetic on them is modulo
// 2^32: what must fit an int32 is the sum of A_i B_j + A_j B_i over a chunk,
// at most 2 x pairs x KB x 64 products of 2^14, below 2^31 for pairs x KB <=
// 1016 (the 2032 k-steps of the plain chunks).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace mdgi {

constexpr int CROSS_CHUNK_STEPS = 1016;

__host__ __device__ inline int cross_pairs(int d) { return (d + 1) >> 1; }
// sums of the diagonals before d
__host__ __device__ inline int cross_offset(int d) { return d * d / 4; }
__host__ __device__ inline int cross_pairs_per_chunk(int KB) { return CROSS_CHUNK_STEPS / KB; }
__host__ __device__ inline int cross_chunks(int d, int ppc) {
  return (cross_pairs(d) + ppc - 1) / ppc;
}
inline int cross_outputs(int D, int KB) {
  int c = D;
  for (int d = 1; d < D; ++d) c += cross_chunks(d, cross_pairs_per_chunk(KB));
  return c;
}
// FP32 flush groups of a plane's KB k-steps: ceil(KB / 16) groups of at most
// 16 k-steps, each cut again into 2 or 4 where the data asks for it (level).
// Group j of `groups` starts at k-step j KB / groups; the cuts are nested.
__host__ __device__ inline int cross_groups(int KB) { return (KB + 15) / 16; }

// End of the diagonal group that starts at dlo when the buffer holds `cap`
// sum planes (cap >= cross_pairs(D - 1)).
inline int cross_group_end(int dlo, int D, int cap) {
  int e = dlo;
  while (e < D && cross_offset(e + 1) - cross_offset(dlo) <= cap) ++e;
  return e;
}

// Sum planes of the diagonals [dlo, dhi) into planes s.. of both operands'
// buffers (s digit planes of rows x Kp first), and in norms[0] / norms[1]
// the maxima, over the rows of A / B, the sum planes and the windows of half
// a flush group, of the sums of squares.
// One operand alone: the other's rows 0.
int launch_cross_sums(int s, int dlo, int dhi, int Kp, int rows_a, int rows_b, void *dA, void *dB,
                      long long plane_a, long long plane_b, unsigned *norms, cudaStream_t st);

// The diagonal GEMM over sum planes: the squares (squares = D, or 0 where
// an earlier launch did them) and the diagonals [dlo, dhi).
int launch_diag_gemm_cross(int s, int D, int dlo, int dhi, int squares, int sum_planes, int Mp,
                           int Np, int Kp, const void *dA, const void *dB, const unsigned *norm_a,
                           const unsigned *norm_b, int *out, int parts, int raster, int pace,
                           cudaStream_t st);

// Renormalisation from the cross form's output planes (renorm.cu).
int launch_cross_renorm(int p, int D, int KB, int m, int n, const int *out, long long plane_c,
                        int ldcd, const int *E, const int *F, double *C, int ldc,
                        cudaStream_t st);

}  // namespace mdgi
