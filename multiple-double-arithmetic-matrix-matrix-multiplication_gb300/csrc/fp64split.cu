// Truncated slice convolution on FP64 tensor cores (DMMA m8n8k4).
//
// Cq[r][c][i] = sum_k sum_{j<=i} Aq[r][k][j] * Bq[k][c][i-j]
//
// This is the product the reference forms with one FP64 wmma GEMM against
// the block-Toeplitz matrix bigB2 (TCtest.cu:21-46, TCcuda.cu:79-95): its
// K index is the flattened (k, j) = k*pp + j, consumed four at a time by
// each m8n8k4 DMMA.  Here bigB2 is never formed.  For every output entry the
// DMMAs run over the same chunks (k, j0..j0+3), k outer, j0 inner, with the
// same four operands per chunk, and the chunks whose B part is zero for the
// whole tile (j0 > i) are skipped, which removes half of the reference's
// tensor work.  Operands are addressed through element strides: the
// reference's AoS layout (m x k x pp; four consecutive slices of one entry
// per 32-byte sector) for mdg_slice_conv, and slice planes (pp planes of
// m x k, the layout of the CPU convolution driver TCcudant.cpp:172-276) for
// mdg_plane_conv.
//
// GB300 note: FP64 tensor throughput on this part is a small fraction of its
// BF16 rate; this kernel is the baseline the BF16 slice form is measured
// against, and it is DMMA-bound, not memory-bound.
#include "common.cuh"

namespace {

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// Element (row, k, slice) of A sits at row * ar + kk * ak + j * aj, and so
// on for B (k, column, slice) and C (row, column, slice).
struct ConvStrides {
  long long ar, ak, aj, bk, bc, bj, cr, cc, ci;
};

// One warp per block, an 8 x 8 tile of diagonal i = pp - 1 - blockIdx.z.  An
// SM's FP64 tensor unit takes a DMMA in about 135 cycles and one quarter of
// the SM alone in 540, so the two operand loads of a DMMA need no reuse; what
// counts is that every SM quarter gets an equal share to the end.  Diagonal i
// costs i / 4 + 1 chunks a k: so the tiles are the smallest, the dear
// diagonals come first, and kDynamicSmem holds back all but 16 blocks per
// SM, so that an SM takes its next block as it finishes one.  With 64 x 32
// tiles of four warps, all resident at once: qd 251 x 300 x 277 8.98 -> 6.49
// ms a call, qd 100^3 1.02 -> 0.42, dd 64^3 0.35 -> 0.08, qd 512^3 41.1 ->
// 39.9 (1.02 of the DGEMM rate for the chunks done).  On slice planes, whose
// loads touch a sector each: 16 planes of 251 x 300 x 277 8.86 -> 6.34 ms, 512^3
// 41.8 -> 39.5, 12 of 300 x 100 x 900 10.3 -> 5.1.
constexpr int kDynamicSmem = 13000;

__global__ void __launch_bounds__(32)
    slice_conv_kernel(int pp, int m, int n, int k, int col_tiles, const double *__restrict__ Aq,
                      const double *__restrict__ Bq, double *__restrict__ Cq,
                      const ConvStrides sd) {
  const int i = (int)(gridDim.z - 1 - blockIdx.z);
  const int g = threadIdx.x >> 2, t = threadIdx.x & 3;
  const int row_tile = blockIdx.x / col_tiles, col_tile = blockIdx.x - row_tile * col_tiles;
  const int row = row_tile * 8 + g, col = col_tile * 8 + g;  // of the operands
  double acc[2] = {0.0, 0.0};
#pragma unroll 2
  for (int kk = 0; kk < k; ++kk) {
    for (int j0 = 0; j0 <= i; j0 += 4) {
      const int ja = j0 + t, jb = i - ja;
      const double a =
          (row < m && ja < pp) ? __ldg(Aq + row * sd.ar + kk * sd.ak + ja * sd.aj) : 0.0;
      const double b = (col < n && jb >= 0) ? __ldg(Bq + kk * sd.bk + col * sd.bc + jb * sd.bj) : 0.0;
      dmma(acc, a, b);
    }
  }
  if (row >= m) return;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int c = col_tile * 8 + 2 * t + h;
    if (c < n) Cq[row * sd.cr + c * sd.cc + i * sd.ci] = acc[h];
  }
}

}  // namespace

namespace mdgi {

int launch_slice_conv(int pp, int m, int n, int k, const double *Aq, const double *Bq,
                      double *Cq, int planes, cudaStream_t st) {
  if (m == 0 || n == 0 || pp == 0) return MDG_SUCCESS;
  if (pp > 65535) return MDG_ERROR_INVALID_SIZE;
  const long long P = pp, M = m, N = n, K = k;
  const ConvStrides aos{K * P, P, 1, N * P, P, 1, N * P, P, 1};
  const ConvStrides soa{K, 1, M * K, N, 1, K * N, N, 1, M * N};
  const long long col_tiles = ceil_div(n, 8), tiles = col_tiles * ceil_div(m, 8);
  if (tiles > 0x7fffffff) return MDG_ERROR_INVALID_SIZE;
  slice_conv_kernel<<<dim3((unsigned)tiles, 1, pp), 32, kDynamicSmem, st>>>(
      pp, m, n, k, (int)col_tiles, Aq, Bq, Cq, planes ? soa : aos);
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

}  // namespace mdgi
