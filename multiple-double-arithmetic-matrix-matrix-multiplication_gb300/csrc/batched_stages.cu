// Scale and digit kernels of the batched slice-digit GEMM: one launch each
// over every problem, whatever its limb count (the stages take it as a
// number); each block finds its problem in the table (batched_table.cuh).
#include "batched_table.cuh"
#include "slice_stages.cuh"

namespace {

using mdgi::BatchProblem;
using mdgi::DIGIT_THREADS;
using mdgi::SCALE_COLS;
using mdgi::SCALE_ROWS;
using mdgi::SCALE_THREADS;

__global__ void __launch_bounds__(SCALE_THREADS)
    batch_scale_kernel(const BatchProblem *__restrict__ pr, int count, int *__restrict__ exps) {
  const BatchProblem &b = pr[mdgi::find_problem<mdgi::kScaleUnits>(pr, count, blockIdx.x)];
  const int lu = blockIdx.x - b.scale_begin;
  if (lu < b.scale_b_off) {
    const int r = SCALE_ROWS * lu + (int)(threadIdx.x >> 5);
    if (r >= b.m) return;
    const unsigned long long mx = mdgi::row_max(b.p, b.A, b.lda, r, 0, b.k);
    if ((threadIdx.x & 31) == 0)
      exps[b.offE + r] = mdgi::scale_exp(__longlong_as_double((long long)mx));
  } else {
    const int c0 = SCALE_COLS * (lu - b.scale_b_off), c = c0 + (int)threadIdx.x;
    const unsigned long long mx = mdgi::col_max(b.p, b.B, b.ldb, c0, b.n, 0, b.k);
    if (threadIdx.x < SCALE_COLS && c < b.n)
      exps[b.offF + c] = mdgi::scale_exp(__longlong_as_double((long long)mx));
  }
}

// Valid rows and k-positions (an odd last one with its neighbour) only: the
// padding of every plane was cleared when the plan was made.
__global__ void __launch_bounds__(DIGIT_THREADS)
    batch_digits_kernel(const BatchProblem *__restrict__ pr, int count,
                        const int *__restrict__ exps) {
  extern __shared__ uint4 smem[];
  const BatchProblem &b = pr[mdgi::find_problem<mdgi::kDigitUnits>(pr, count, blockIdx.x)];
  int lu = blockIdx.x - b.dig_begin;
  const bool side_b = lu >= b.dig_b_off;
  if (side_b) lu -= b.dig_b_off;
  const mdgi::DigitSide d =
      side_b ? mdgi::DigitSide{b.B, exps + b.offF, b.dB, b.ldb, 1, b.n, b.k, b.Kp, b.Kp, b.plane_b}
             : mdgi::DigitSide{b.A, exps + b.offE, b.dA, b.lda, 0, b.m, b.k, b.Kp, b.Kp, b.plane_a};
  const int groups = (b.k + 1) / 2;
  const long long e = lu * (long long)DIGIT_THREADS + threadIdx.x;
  int row, group;
  mdgi::digit_place(b.p, d.trans, e, groups, row, group);
  if (row >= d.rows) return;
  const bool wide = reinterpret_cast<uintptr_t>(d.X) % 16 == 0;
  mdgi::digits_group<2, 2>(b.p, b.s, d, row, group * 2, wide, smem);
}

}  // namespace

namespace mdgi {

int launch_batch_scale(const BatchProblem *pr, int count, int units, int *exps, cudaStream_t st) {
  if (units == 0) return MDG_SUCCESS;
  batch_scale_kernel<<<units, SCALE_THREADS, 0, st>>>(pr, count, exps);
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

int launch_batch_digits(const BatchProblem *pr, int count, int units, int max_s, const int *exps,
                        cudaStream_t st) {
  if (units == 0) return MDG_SUCCESS;
  const int smem = digit_smem(max_s, 2);
  MDG_TRY(allow_smem(batch_digits_kernel, smem, digit_smem(MAX_SLICES, 2)));
  batch_digits_kernel<<<units, DIGIT_THREADS, smem, st>>>(pr, count, exps);
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

}  // namespace mdgi
