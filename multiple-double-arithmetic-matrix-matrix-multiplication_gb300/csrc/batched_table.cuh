// The problem table of the batched slice-digit GEMM (batched.cu) and the
// lookup of a block's problem, shared by the planning code and the stage
// kernels (batched_stages.cu, renorm.cu).
#pragma once

#include <cuda_bf16.h>

#include "common.cuh"

namespace mdgi {

// Every stage kernel runs over a flat list of work units (thread blocks);
// each problem owns a contiguous range of units in every list.
//   scale:  blocks of SCALE_ROWS rows of A, then of SCALE_COLS columns of B
//   digits: blocks of DIGIT_THREADS threads over A's digit rows, two
//           k-positions a thread, then over B's
//   renorm: blocks of RENORM_THREADS threads over C, two columns a thread
struct BatchProblem {
  int p, s, D, m, n, k, Mp, Np, Kp;
  const double *A, *B;
  double *C;
  int lda, ldb, ldc;
  int offE, offF;  // exponents of A's rows at offE, of B's columns at offF
  __nv_bfloat16 *dA, *dB;
  int *chunks;
  int planes, top, wide;  // chunk planes in all; renorm_top; C is 16-byte aligned
  long long plane_a, plane_b, plane_c;
  int scale_begin, scale_b_off;  // first scale unit; units of A's rows
  int dig_begin, dig_b_off;      // first digit unit; units of A's digit rows
  int out_begin;                 // first renormalisation unit
};

enum { kScaleUnits = 0, kDigitUnits = 1, kRenormUnits = 2 };

// The problem whose range of units (Field) holds unit x: the last problem
// whose first unit is <= x.
template <int Field>
__device__ __forceinline__ int find_problem(const BatchProblem *pr, int count, int x) {
  int lo = 0, hi = count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    const int b = Field == kScaleUnits ? pr[mid].scale_begin
                  : Field == kDigitUnits ? pr[mid].dig_begin
                                         : pr[mid].out_begin;
    if (b <= x) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// One launch each over every problem of the batch (batched_stages.cu); max_s:
// the most digits of any problem.
int launch_batch_scale(const BatchProblem *pr, int count, int units, int *exps, cudaStream_t st);
int launch_batch_digits(const BatchProblem *pr, int count, int units, int max_s, const int *exps,
                        cudaStream_t st);
// The renormalisation, whatever the limb counts (renorm.cu); max_d: the most
// diagonals of any problem.
int launch_batch_renorm(const BatchProblem *pr, int count, int units, int max_d, const int *exps,
                        cudaStream_t st);

}  // namespace mdgi
