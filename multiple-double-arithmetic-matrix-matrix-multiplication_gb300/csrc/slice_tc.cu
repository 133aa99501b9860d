// The slice-digit form of the multi-double GEMM: split, diagonal GEMM on
// BF16 tensor cores, renormalisation.
//
// 1. scale exponents.  E[r] for each row of A and F[c] for each column of B
//    from the largest sum of absolute limbs; 2^E bounds every entry.
// 2. digits.  Each P-double a of row r becomes the integer
//       V = sum_l floor(a_l * 2^(S - E[r])),  S = 7 + 8 (s - 1),
//    written as s balanced base-256 digits d_0 (most significant) ..
//    d_{s-1} in [-128, 128].  Digit i of every entry forms one BF16 plane
//    (the integers up to 256 are exact in BF16).  A's planes are m x k,
//    B's are transposed to n x k so both operands are K-major.
// 3. diagonal GEMM.  C_d = sum_{i+j=d} A_i B_j^T for d < D.  One product
//    of two digits is at most 2^14, so an FP32 accumulator holds the exact
//    sum of 1024 of them (|sum| <= 2^24); every 1024 products (256 in the
//    mma.sync engine) the FP32 accumulator is flushed into 32-bit
//    integers, and every 2032 k-steps (130048 products) the integers are
//    stored as one "chunk" plane (|sum| < 2^31).  All sums are exact.
// 4. renormalisation.  W = sum_d C_d 256^(D-1-d), C_d the sum of the
//    chunks of diagonal d, is formed exactly in
//    wide integers and rounded to P limbs, each to nearest, scaled by
//    2^(E[r] + F[c] - 14 - 8 (D - 1)).
// The reference has no counterpart of steps 1-4; its split form cuts limbs
// into FP64 slices for FP64 DMMA (floatybits.cu, TCtest.cu).  The oracle's
// section 8 restates these steps on the CPU, and the GPU result equals it
// bit for bit.
#include "common.cuh"
#include "cross_sums.cuh"
#include "slice_common.cuh"
#include "slice_tc.cuh"
#include "slice_stages.cuh"

#include <cuda_bf16.h>

namespace {

using mdgi::DIGIT_THREADS;
using mdgi::DigitSide;
using mdgi::SCALE_COLS;
using mdgi::SCALE_ROWS;
using mdgi::SCALE_THREADS;

// ------------------------------------------------------------ exponents --
// One operand of the scale stage: the exponents of `count` rows of X (count x
// k), or, trans, of `count` columns (k x count).
struct ScaleSide {
  const double *X;
  int ld, trans, count;
  int *E;
};

// Blocks of 8 rows or columns of the first side, then of the second, each cut
// into `cuts` ranges of k.  One range: the exponents, at once.  More: maxima
// by atomics into bits (first side, then second), and exps_kernel after.  Bound
// by reading A and B once; on small problems one launch instead of two
// clears, two maxima and two exponent launches (dd 64^3 56 -> 6 us, qd 256^3
// 64 -> 8 us, qd 8192^3 1.06 -> 0.81 ms, 5.3 TB/s).
__global__ void __launch_bounds__(SCALE_THREADS)
    scale_kernel(int P, int k, const ScaleSide a, const ScaleSide b, int blocks_a, int cuts,
                 unsigned long long *bits) {
  static_assert(SCALE_ROWS == SCALE_COLS, "a block takes as many rows as columns");
  int blk = blockIdx.x / cuts;
  const int cut = blockIdx.x - blk * cuts;
  const int k0 = (int)((long long)k * cut / cuts), k1 = (int)((long long)k * (cut + 1) / cuts);
  const bool second = blk >= blocks_a;
  const ScaleSide &d = second ? b : a;
  if (second) blk -= blocks_a;
  int i;  // this thread's row or column, where it holds the maximum
  unsigned long long mx;
  bool holds;
  if (d.trans) {
    i = blk * SCALE_COLS + (int)threadIdx.x;
    mx = mdgi::col_max(P, d.X, d.ld, blk * SCALE_COLS, d.count, k0, k1);
    holds = threadIdx.x < SCALE_COLS && i < d.count;
  } else {
    i = blk * SCALE_ROWS + (int)(threadIdx.x >> 5);
    if (i >= d.count) return;
    mx = mdgi::row_max(P, d.X, d.ld, i, k0, k1);
    holds = (threadIdx.x & 31) == 0;
  }
  if (!holds) return;
  if (cuts == 1)
    d.E[i] = mdgi::scale_exp(__longlong_as_double((long long)mx));
  else
    atomicMax(bits + (second ? a.count : 0) + i, mx);
}

__global__ void exps_kernel(int m, int n, const unsigned long long *__restrict__ bits,
                            int *__restrict__ E, int *__restrict__ F) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m + n) return;
  const int e = mdgi::scale_exp(__longlong_as_double((long long)bits[i]));
  if (i < m)
    E[i] = e;
  else
    F[i - m] = e;
}

// --------------------------------------------------------------- digits --
// Both operands in one launch; threads run over the sides' groups of V
// k-positions (digit_place), so plane stores are coalesced for A and B alike.  norms: two counters of a later stage, cleared on the way.
template <int V, int PL>
__global__ void __launch_bounds__(DIGIT_THREADS)
    digits_kernel(int P, int s, const DigitSide a, const DigitSide b, long long of_a, bool wide,
                  unsigned *norms) {
  extern __shared__ uint4 smem[];
  const long long e = blockIdx.x * (long long)DIGIT_THREADS + threadIdx.x;
  if (norms && e < 2) norms[e] = 0;
  const int groups = a.cols_pad / V;
  const DigitSide &d = e < of_a ? a : b;
  int row, group;
  mdgi::digit_place(P, d.trans, e < of_a ? e : e - of_a, groups, row, group);
  if (row >= d.rows) return;
  mdgi::digits_group<V, PL>(P, s, d, row, group * V, wide, smem);
}

// ---------------------------------------------------- diagonal GEMM v0 --
// mma.sync m16n8k16 BF16 -> FP32.  Block 128 x 64, 8 warps as 4 x 2, warp
// tile 32 x 32 (2 x 4 MMA tiles), K chunk 32 through shared memory.
constexpr int BM = 128, BN = 64, BK = 32, SK = BK + 8;
// k-steps of 64 per FP32 flush in this engine: 256 products, |sum| <= 2^22,
// the range of the exact_int conversion below
constexpr int V0_GROUP_STEPS = 4;

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4],
                                         const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// x is an integer-valued float with |x| <= 2^22: adding 1.5 * 2^23 puts it
// in the significand exactly; the bits minus those of 1.5 * 2^23 are x.
__device__ __forceinline__ int64_t exact_int(float x) {
  return (int64_t)(__float_as_int(x + 12582912.0f) - 0x4B400000);
}

__global__ void __launch_bounds__(256)
    diag_gemm_v0(int s, int D, int Kp, const __nv_bfloat16 *__restrict__ dA,
                 const __nv_bfloat16 *__restrict__ dB, int ld, long long plane_a,
                 long long plane_b, int *__restrict__ out, long long plane_c, int ldc, int cs) {
  __shared__ __align__(16) __nv_bfloat16 As[BM][SK];
  __shared__ __align__(16) __nv_bfloat16 Bs[BN][SK];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
  const int KB = Kp / 64;
  int chunk = 0;

  for (int d = 0; d < D; ++d) {
    float acc[2][4][4];
    int tot[2][4][4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          acc[a][b][c] = 0.f;
          tot[a][b][c] = 0;
        }
    const int ilo = max(0, d - (s - 1));
    const int S = mdgi::diag_pairs(d, s) * KB;
    for (int step = 0; step < S; ++step) {
      const int i = ilo + step / KB, kb = step % KB;
      const __nv_bfloat16 *Ai = dA + i * plane_a + (size_t)row0 * ld + kb * 64;
      const __nv_bfloat16 *Bj = dB + (d - i) * plane_b + (size_t)col0 * ld + kb * 64;
      for (int half = 0; half < 2; ++half) {
#pragma unroll
        for (int v = tid; v < BM * BK / 8; v += 256) {
          const int r = v >> 2, cc = (v & 3) * 8;
          *reinterpret_cast<uint4 *>(&As[r][cc]) =
              *reinterpret_cast<const uint4 *>(Ai + (size_t)r * ld + half * BK + cc);
        }
        {
          const int r = tid >> 2, cc = (tid & 3) * 8;
          *reinterpret_cast<uint4 *>(&Bs[r][cc]) =
              *reinterpret_cast<const uint4 *>(Bj + (size_t)r * ld + half * BK + cc);
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; kk += 16) {
          uint32_t af[2][4], bf[4][2];
#pragma unroll
          for (int mt = 0; mt < 2; ++mt) {
            const int r = wm + mt * 16 + g;
            af[mt][0] = *reinterpret_cast<const uint32_t *>(&As[r][kk + 2 * t]);
            af[mt][1] = *reinterpret_cast<const uint32_t *>(&As[r + 8][kk + 2 * t]);
            af[mt][2] = *reinterpret_cast<const uint32_t *>(&As[r][kk + 8 + 2 * t]);
            af[mt][3] = *reinterpret_cast<const uint32_t *>(&As[r + 8][kk + 8 + 2 * t]);
          }
#pragma unroll
          for (int nt = 0; nt < 4; ++nt) {
            const int c = wn + nt * 8 + g;
            bf[nt][0] = *reinterpret_cast<const uint32_t *>(&Bs[c][kk + 2 * t]);
            bf[nt][1] = *reinterpret_cast<const uint32_t *>(&Bs[c][kk + 8 + 2 * t]);
          }
#pragma unroll
          for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int nt = 0; nt < 4; ++nt) mma_bf16(acc[mt][nt], af[mt], bf[nt]);
        }
        __syncthreads();
      }
      const bool chunk_end = step % cs == cs - 1 || step == S - 1;
      const bool group_end = step % V0_GROUP_STEPS == V0_GROUP_STEPS - 1 || chunk_end;
      if (group_end) {
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              tot[a][b][c] += (int)exact_int(acc[a][b][c]);
              acc[a][b][c] = 0.f;
            }
      }
      if (chunk_end) {
        int *o = out + (size_t)chunk * plane_c;
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
          for (int nt = 0; nt < 4; ++nt)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int r = row0 + wm + mt * 16 + g + h * 8;
              const int c = col0 + wn + nt * 8 + 2 * t;
              *reinterpret_cast<int2 *>(o + (size_t)r * ldc + c) =
                  make_int2(tot[mt][nt][2 * h], tot[mt][nt][2 * h + 1]);
              tot[mt][nt][2 * h] = tot[mt][nt][2 * h + 1] = 0;
            }
        ++chunk;
      }
    }
  }
}

}  // namespace

namespace mdgi {

// kCrossSumBytes: sums of both operands held at once (beyond that the
// diagonals are done in groups that reuse the buffer).  kCrossMaxBytes:
// workspace beyond which the digit pairs are used, so that problems which
// fill the device still fit.
// kCrossBlockBytes: workspace of a column strip of the host entry, whose
// sums are all kept for the row panels to come.
// Each group has a last wave of tiles of its own and its sums are short, so a
// smaller buffer costs time.  ms a call with 1 / 2 / 4 / 8 / 16 GiB of sums: hd 1024
// x 1024 x 512 4.28 / 4.00 / 4.05 / 3.93 / 3.93, od 2048^3 13.2 / 12.4 / 11.9 / 12.0 /
// 12.2, qd 4096^3 27.0 / 24.6 / 24.3 / 23.9 / 23.5, qd 8192^3 183 / 184 / 183 / 180 /
// 176; 0.25 and 1: qd 1024^3 0.82 / 0.62.
constexpr size_t kCrossSumBytes = 16ull << 30, kCrossMaxBytes = 160ull << 30;
constexpr size_t kCrossBlockBytes = 32ull << 30;

// Where sum planes beat digit pairs.  They save half the products (time as
// Mp Np Kp) and cost the writing of the sums (as (Mp + Np) Kp) and a dearer
// renormalisation (as Mp Np): so a least Mp Np / (Mp + Np) and a least k.
// Measured whole calls, pairs against sums: qd 1024 x 768 x 1024 718 / 653
// us, 1024 x 768 x 512 486 / 468, 1024 x 1024 x 256 421 / 517, 256 x 4096 x
// 1024 1029 / 1073; dd 1024 x 768 x 1024 301 / 282, 512 x 2048 x 1024 347 /
// 352.  Up to four 256 x 256 tiles leave most of the chip idle and the
// length of a tile's work is what counts: qd 512 x 512 x 1024 571 / 431,
// but x 512 370 / 332 and x 256 236 / 310.
static bool cross_pays(int p, int Mp, int Np, int KB) {
  const double tile = (double)Mp * Np / ((double)Mp + Np);
  if (KB >= 16) return tile >= (p == 2 ? 500.0 : 384.0) || (p > 2 && Mp * (long long)Np <= 512 * 512);
  return KB >= 8 && tile >= (p == 2 ? 1000.0 : 500.0);
}

int words_for(int s, int D) {
  // digits need S + 2 bits plus a word of headroom; W needs 8 (D - 1) + 64
  const int bits = std::max(7 + 8 * (s - 1) + 2, 8 * (D - 1) + 72);
  const int w = (bits + 63) / 64 + 1;
  if (w <= 4) return 4;
  if (w <= 6) return 6;
  if (w <= 10) return 10;
  if (w <= 16) return 16;
  return 0;
}

// sums: sum planes per operand (0: digit pairs alone)
static SlicePlan layout_slice_plan(int p, int s, int D, int m, int n, int k, int sums,
                                   int cs = CHUNK_STEPS) {
  SlicePlan pl{};
  pl.p = p;
  pl.s = s;
  pl.D = D;
  pl.m = m;
  pl.n = n;
  pl.k = k;
  pl.Mp = (int)align_up(std::max(m, 1), 256);
  pl.Np = (int)align_up(std::max(n, 1), 256);
  pl.Kp = (int)align_up(std::max(k, 1), 64);
  pl.sums = sums;
  pl.cs = cs;
  pl.chunks = sums ? cross_outputs(D, pl.Kp / 64) : total_chunks(s, D, pl.Kp / 64, cs);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t o = off;
    off = align_up(off + bytes, 256);
    return o;
  };
  pl.off_bits = take(sizeof(unsigned long long) * ((size_t)pl.Mp + pl.Np));
  pl.off_E = take(sizeof(int) * pl.Mp);
  pl.off_F = take(sizeof(int) * pl.Np);
  pl.off_norms = sums ? take(2 * sizeof(unsigned)) : 0;
  pl.plane_a = (long long)pl.Mp * pl.Kp;
  pl.plane_b = (long long)pl.Np * pl.Kp;
  pl.plane_c = (long long)pl.Mp * pl.Np;
  pl.off_dA = take(sizeof(__nv_bfloat16) * (size_t)(s + sums) * pl.plane_a);
  pl.off_dB = take(sizeof(__nv_bfloat16) * (size_t)(s + sums) * pl.plane_b);
  pl.off_Cd = take(sizeof(int) * (size_t)pl.chunks * pl.plane_c);
  pl.total = off;
  return pl;
}

SlicePlan make_slice_plan(int p, int s, int D, int m, int n, int k) {
  return layout_slice_plan(p, s, D, m, n, k, 0);
}

// What the diagonal GEMM takes on a problem of few tiles, in us: k-steps of the
// busiest worker.  A k-step of 32 KiB of operands a CTA takes 0.43 us where
// all 152 SMs ask L2 for them (11 TB/s), 48 KiB 0.62, and 0.27 by itself; 16
// k-steps go to the ends of a run.  Estimated / measured whole calls,
// short chunks against two diagonals an accumulator: qd 2000 x 100 x 500 154 -
// 86 / 218 - 160 us, 100 x 2000 x 500 116 - 86 / 190 - 158, 500 x 64 x 500 44 -
// 65 / 88 - 117, od 300 x 128 x 700 150 - 168 / 247 - 269, 3000 x 64 x 1000
// 1680 - 880 / 1899 - 977, dd 300 x 300 x 2000 83 - 125 / 159 - 204.
static double chunked_us(int s, int D, int KB, long long tiles, int tn) {
  long long steps = 0;
  for (int d = 0; d < D; ++d) steps += (long long)diag_pairs(d, s) * KB;
  const double share = (double)steps * tiles / (tn ? 152 : 76) + 16.0;
  return share * (tn == 256 ? 0.62 : 0.43);
}

static double stacked_us(int s, int D, int m, int n, int KB) {
  const int stack = stacked_tiles(s, D, m, n, KB);
  if (!stack) return 1e30;
  const long long tiles = stack == 1 ? (long long)ceil_div(m, 256) * ceil_div(n, 128)
                                     : (long long)ceil_div(m, 128) * ceil_div(n, 256);
  long long steps = 0;
  for (int d = -(D & 1); d < D; d += 2) steps += (long long)(d + 2) * KB + 16;
  return std::max(0.43 * (double)steps * tiles / 76, 0.27 * ((D + 1.0) * KB + 16.0));
}

int narrow_tile(int s, int D, int m, int n, int KB) {
  const int tn = n <= 128 ? 128 : m <= 128 ? 256 : 0;
  if (!tn) return 0;
  const long long tiles = (long long)ceil_div(m, 128) * ceil_div(n, tn);
  // a full chip of them asks more operand bytes of L2 than pairs do (tall dd
  // 16001 x 96 x 3001: 1.84 ms against 1.74)
  if (tiles > 76 || stacked_us(s, D, m, n, KB) < chunked_us(s, D, KB, tiles, tn)) return 0;
  return tn;
}

AutoTiles auto_tiles(int s, int D, int m, int n, int KB, int cs) {
  const int narrow = narrow_tile(s, D, m, n, KB);
  return AutoTiles{narrow, !narrow && cs == CHUNK_STEPS ? stacked_tiles(s, D, m, n, KB) : 0};
}

// Measured, chunks of 2032 k-steps and at most 8 parts / this: qd 256^3 107 /
// 28 us for the GEMM (plan 136 / 61 us a call), dd 64^3 26 / 11 us.
//
// k-steps per chunk that let the CTAs of a chip (152, or 76 pairs) share a
// problem of few tiles: about the steps each can have.  Where a chunk per
// CTA fits at up to twice that length it is taken, so that none gets two.
static int chunk_steps(int s, int D, int m, int n, int KB) {
  const int tn = narrow_tile(s, D, m, n, KB);
  const long long tiles = tn ? (long long)ceil_div(m, 128) * ceil_div(n, tn)
                             : (long long)ceil_div(m, 256) * ceil_div(n, 256);
  const int workers = tn ? 152 : 76;
  long long steps = 0;
  for (int d = 0; d < D; ++d) steps += (long long)diag_pairs(d, s) * KB;
  const long long share = (steps * tiles + workers - 1) / workers;
  if (2 * tiles > workers || share >= CHUNK_STEPS / 2 ||
      stacked_us(s, D, m, n, KB) < chunked_us(s, D, KB, tiles, tn))
    return CHUNK_STEPS;
  const int least = std::max(8, (int)(share + 3) / 4 * 4);
  // (longer chunks are never more)
  int lo = 0, hi = least / 4 + 1;
  while (lo < hi) {
    const int mid = (lo + hi) / 2;
    if (tiles * total_chunks(s, D, KB, least + 4 * mid) <= workers)
      hi = mid;
    else
      lo = mid + 1;
  }
  return lo <= least / 4 ? least + 4 * lo : least;
}

SlicePlan best_slice_plan(int p, int s, int D, int m, int n, int k) {
  SlicePlan pairs = make_slice_plan(p, s, D, m, n, k);
  const int KB = pairs.Kp / 64;
  const int cs = chunk_steps(s, D, std::max(m, 1), std::max(n, 1), KB);
  if (cs != CHUNK_STEPS) pairs = layout_slice_plan(p, s, D, m, n, k, 0, cs);
  if (D < 2 || D > s || KB > CROSS_CHUNK_STEPS || !cross_pays(p, pairs.Mp, pairs.Np, KB))
    return pairs;
  const int all = cross_offset(D), least = cross_pairs(D - 1);
  const double plane_bytes = 2.0 * ((double)pairs.plane_a + pairs.plane_b);
  int sums = all;
  if (all * plane_bytes > (double)kCrossSumBytes)
    sums = std::max(least, (int)((double)kCrossSumBytes / plane_bytes));
  const SlicePlan pl = layout_slice_plan(p, s, D, m, n, k, sums);
  return pl.total <= kCrossMaxBytes && pl.total >= pairs.total ? pl : pairs;
}

int launch_scale_exponents(int p, int m, int n, int k, const double *A, int lda,
                           const double *B, int ldb, unsigned long long *bits, int *E, int *F,
                           cudaStream_t st, int trans_a, int trans_b) {
  m = std::max(m, 0);
  n = std::max(n, 0);
  if (m == 0 && n == 0) return MDG_SUCCESS;
  // B first: its few columns of a tall problem take longest
  const ScaleSide b{B, ldb, !trans_b, n, F}, a{A, lda, trans_a, m, E};
  const int blocks_b = ceil_div(n, SCALE_COLS);
  const long long blocks = (long long)blocks_b + ceil_div(m, SCALE_ROWS);
  // a thread takes k / 32 entries one after another: ranges of k where that
  // is long and the blocks leave SMs idle (four 256-thread blocks fill one
  // of 152)
  const int cuts = (int)std::min<long long>(std::max<long long>(1, 608 / blocks),
                                            std::max(1, k / 1024));
  if (cuts > 1)
    MDG_TRY_CUDA(cudaMemsetAsync(bits, 0, sizeof(unsigned long long) * ((size_t)m + n), st));
  scale_kernel<<<(unsigned)(blocks * cuts), SCALE_THREADS, 0, st>>>(p, k, b, a, blocks_b, cuts,
                                                                    bits);
  MDG_TRY_LAUNCH();
  if (cuts > 1) {
    exps_kernel<<<ceil_div((long long)m + n, 256), 256, 0, st>>>(n, m, bits, F, E);
    MDG_TRY_LAUNCH();
  }
  return MDG_SUCCESS;
}

template <int V, int PL>
static int launch_digits_v(int p, int s, const DigitSide &a, const DigitSide &b, bool wide,
                           unsigned *norms, cudaStream_t st) {
  const int smem = digit_smem(s, V);
  MDG_TRY(allow_smem(digits_kernel<V, PL>, smem, digit_smem(MAX_SLICES, V)));
  const long long of_a = digit_threads(p, a.trans, a.rows, a.cols_pad / V);
  const long long threads = of_a + digit_threads(p, b.trans, b.rows, a.cols_pad / V);
  digits_kernel<V, PL>
      <<<ceil_div(threads, DIGIT_THREADS), DIGIT_THREADS, smem, st>>>(p, s, a, b, of_a, wide, norms);
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

int launch_digits(int p, int s, const DigitSide &a, const DigitSide &b, unsigned *norms,
                  cudaStream_t st) {
  if (!words_for(s, 1)) return MDG_ERROR_NOT_SUPPORTED;
  if (b.rows && b.cols_pad != a.cols_pad) return MDG_ERROR_INVALID_SIZE;
  if (a.rows + b.rows == 0 || a.cols_pad == 0) return MDG_SUCCESS;
  auto addr = [](const void *x) { return reinterpret_cast<uintptr_t>(x); };
  const bool wide = (addr(a.X) | addr(b.X)) % 16 == 0;
  // two k-positions a thread where planes take 4-byte stores
  auto even = [&](const DigitSide &d) {
    return d.rows == 0 || (d.cols_pad % 2 == 0 && d.ld_out % 2 == 0 && d.plane_stride % 2 == 0 &&
                           addr(d.planes) % 4 == 0);
  };
  if (even(a) && even(b))
    return p == 2 ? launch_digits_v<2, 2>(p, s, a, b, wide, norms, st)
                  : launch_digits_v<2, 4>(p, s, a, b, wide, norms, st);
  return p == 2 ? launch_digits_v<1, 2>(p, s, a, b, wide, norms, st)
                : launch_digits_v<1, 4>(p, s, a, b, wide, norms, st);
}

static unsigned long long *plan_bits(const SlicePlan &pl, void *ws) {
  return reinterpret_cast<unsigned long long *>(reinterpret_cast<char *>(ws) + pl.off_bits);
}

static DigitSide side_a(const SlicePlan &pl, int rows, const double *A, int lda, const int *E,
                        void *planes, int trans = 0) {
  return DigitSide{A, E, reinterpret_cast<__nv_bfloat16 *>(planes), lda, trans, rows, pl.k, pl.Kp,
                   pl.Kp, pl.plane_a};
}

static DigitSide side_b(const SlicePlan &pl, const double *B, int ldb, const int *F,
                        void *planes, int trans = 0) {
  return DigitSide{B, F, reinterpret_cast<__nv_bfloat16 *>(planes), ldb, !trans, pl.n, pl.k, pl.Kp,
                   pl.Kp, pl.plane_b};
}

int launch_diag_gemm_v0(int s, int D, int Mp, int Np, int Kp, const void *dA, const void *dB,
                        int ld, long long plane_a, long long plane_b, int *chunks,
                        long long plane_c, int cs, cudaStream_t st) {
  if (Mp % BM || Np % BN || Kp % 64) return MDG_ERROR_INVALID_SIZE;
  dim3 grid(Np / BN, Mp / BM);
  diag_gemm_v0<<<grid, 256, 0, st>>>(s, D, Kp, reinterpret_cast<const __nv_bfloat16 *>(dA),
                                     reinterpret_cast<const __nv_bfloat16 *>(dB), ld, plane_a,
                                     plane_b, chunks, plane_c, Np, cs);
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

SlicePlan block_slice_plan(int p, int s, int D, int m, int n, int k) {
  const SlicePlan pairs = make_slice_plan(p, s, D, m, n, k);
  const int KB = pairs.Kp / 64;
  if (D < 2 || D > s || KB > CROSS_CHUNK_STEPS || !cross_pays(p, pairs.Mp, pairs.Np, KB))
    return pairs;
  const SlicePlan pl = layout_slice_plan(p, s, D, m, n, k, cross_offset(D));
  return pl.total <= kCrossBlockBytes ? pl : pairs;
}

// All sums of one side of a block plan, and its norm.
static int block_sums(const SlicePlan &pl, int rows_a, int rows_b, void *ws, cudaStream_t st) {
  if (!pl.sums) return MDG_SUCCESS;
  char *base = reinterpret_cast<char *>(ws);
  auto *norms = reinterpret_cast<unsigned *>(base + pl.off_norms);
  MDG_TRY_CUDA(cudaMemsetAsync(norms + (rows_b ? 1 : 0), 0, sizeof(unsigned), st));
  return launch_cross_sums(pl.s, 1, pl.D, pl.Kp, rows_a, rows_b, base + pl.off_dA,
                           base + pl.off_dB, pl.plane_a, pl.plane_b, norms, st);
}

int slice_prepare_b(const SlicePlan &pl, const double *B, int ldb, void *ws, cudaStream_t st) {
  char *base = reinterpret_cast<char *>(ws);
  int *F = reinterpret_cast<int *>(base + pl.off_F);
  MDG_TRY(launch_scale_exponents(pl.p, 0, pl.n, pl.k, nullptr, 1, B, ldb, plan_bits(pl, ws),
                                 nullptr, F, st));
  const DigitSide b = side_b(pl, B, ldb, F, base + pl.off_dB);
  DigitSide none = b;
  none.rows = 0;
  MDG_TRY(launch_digits(pl.p, pl.s, none, b, nullptr, st));
  return block_sums(pl, 0, pl.n, ws, st);
}

int slice_panel_a(const SlicePlan &pl, int rows, const double *A, int lda, void *ws,
                  cudaStream_t st) {
  if (rows <= 0) return MDG_SUCCESS;
  if (rows > pl.m) return MDG_ERROR_INVALID_SIZE;
  char *base = reinterpret_cast<char *>(ws);
  int *E = reinterpret_cast<int *>(base + pl.off_E);
  MDG_TRY(launch_scale_exponents(pl.p, rows, 0, pl.k, A, lda, nullptr, 1, plan_bits(pl, ws), E,
                                 nullptr, st));
  const DigitSide a = side_a(pl, rows, A, lda, E, base + pl.off_dA);
  DigitSide none = a;
  none.rows = 0;
  MDG_TRY(launch_digits(pl.p, pl.s, a, none, nullptr, st));
  return block_sums(pl, rows, 0, ws, st);
}

int slice_block(const SlicePlan &pla, const void *wsa, const SlicePlan &plb, void *wsb, int rows,
                double *C, int ldc, int engine, int parts, int raster, cudaStream_t st,
                int pace) {
  if (rows <= 0) return MDG_SUCCESS;
  if (rows > pla.m || pla.Mp != plb.Mp || pla.Kp != plb.Kp || pla.s != plb.s ||
      pla.D != plb.D || pla.p != plb.p || pla.sums != plb.sums)
    return MDG_ERROR_INVALID_SIZE;
  const char *abase = reinterpret_cast<const char *>(wsa);
  char *bbase = reinterpret_cast<char *>(wsb);
  const int *E = reinterpret_cast<const int *>(abase + pla.off_E);
  const int *F = reinterpret_cast<const int *>(bbase + plb.off_F);
  const void *dA = abase + pla.off_dA;
  const void *dB = bbase + plb.off_dB;
  auto *Cd = reinterpret_cast<int *>(bbase + plb.off_Cd);
  const SlicePlan &pl = plb;
  if (pl.sums) {
    const auto *norm_a = reinterpret_cast<const unsigned *>(abase + pla.off_norms);
    const auto *norm_b = reinterpret_cast<const unsigned *>(bbase + plb.off_norms) + 1;
    MDG_TRY(launch_diag_gemm_cross(pl.s, pl.D, 1, pl.D, pl.D, pl.sums, pl.Mp, pl.Np, pl.Kp, dA, dB,
                                   norm_a, norm_b, Cd, parts, raster, pace, st));
    return launch_cross_renorm(pl.p, pl.D, pl.Kp / 64, rows, pl.n, Cd, pl.plane_c, pl.Np, E, F, C,
                               ldc, st);
  }
  if (engine != 0) {
    MDG_TRY(launch_diag_gemm_tc(pl.s, pl.D, pl.Mp, pl.Np, pl.Kp, rows, pl.n, pl.k, dA, dB, pl.Kp,
                                pla.plane_a, pl.plane_b, Cd, pl.plane_c, pl.cs, engine, parts,
                                raster, st, pace));
  } else {
    MDG_TRY(launch_diag_gemm_v0(pl.s, pl.D, pl.Mp, pl.Np, pl.Kp, dA, dB, pl.Kp, pla.plane_a,
                                pl.plane_b, Cd, pl.plane_c, pl.cs, st));
  }
  return launch_renorm(pl.p, pl.s, pl.D, pl.Kp / 64, pl.cs, rows, pl.n, Cd, pl.plane_c, pl.Np, E, F, C,
                       ldc, st);
}

int run_slice_gemm(const SlicePlan &pl, const double *A, int lda, const double *B, int ldb,
                   double *C, int ldc, void *ws, int engine, int parts, int raster,
                   cudaStream_t st, int pace, int trans_a, int trans_b) {
  char *base = reinterpret_cast<char *>(ws);
  int *E = reinterpret_cast<int *>(base + pl.off_E);
  int *F = reinterpret_cast<int *>(base + pl.off_F);
  void *dA = base + pl.off_dA;
  void *dB = base + pl.off_dB;
  auto *Cd = reinterpret_cast<int *>(base + pl.off_Cd);
  unsigned *norms = pl.sums ? reinterpret_cast<unsigned *>(base + pl.off_norms) : nullptr;
  NvtxRange range("mdg slice_bf16");
  {
    NvtxRange r("split: scale exponents and digits");
    MDG_TRY(launch_scale_exponents(pl.p, pl.m, pl.n, pl.k, A, lda, B, ldb, plan_bits(pl, ws), E,
                                   F, st, trans_a, trans_b));
    MDG_TRY(launch_digits(pl.p, pl.s, side_a(pl, pl.m, A, lda, E, dA, trans_a),
                          side_b(pl, B, ldb, F, dB, trans_b), norms, st));
  }
  NvtxRange r2("diagonal GEMM and renormalisation");
  if (pl.sums) {
    for (int lo = 1, hi; lo < pl.D; lo = hi) {
      hi = cross_group_end(lo, pl.D, pl.sums);
      if (hi == lo) return MDG_ERROR_NOT_SUPPORTED;
      MDG_TRY(launch_cross_sums(pl.s, lo, hi, pl.Kp, pl.m, pl.n, dA, dB, pl.plane_a, pl.plane_b,
                                norms, st));
      MDG_TRY(launch_diag_gemm_cross(pl.s, pl.D, lo, hi, lo == 1 ? pl.D : 0, pl.sums, pl.Mp,
                                     pl.Np, pl.Kp, dA, dB, norms, norms + 1, Cd, parts, raster,
                                     pace, st));
    }
    return launch_cross_renorm(pl.p, pl.D, pl.Kp / 64, pl.m, pl.n, Cd, pl.plane_c, pl.Np, E, F, C,
                               ldc, st);
  }
  if (engine != 0) {
    MDG_TRY(launch_diag_gemm_tc(pl.s, pl.D, pl.Mp, pl.Np, pl.Kp, pl.m, pl.n, pl.k, dA, dB, pl.Kp,
                                pl.plane_a, pl.plane_b, Cd, pl.plane_c, pl.cs, engine, parts,
                                raster, st, pace));
  } else {
    MDG_TRY(launch_diag_gemm_v0(pl.s, pl.D, pl.Mp, pl.Np, pl.Kp, dA, dB, pl.Kp, pl.plane_a,
                                pl.plane_b, Cd, pl.plane_c, pl.cs, st));
  }
  MDG_TRY(launch_renorm(pl.p, pl.s, pl.D, pl.Kp / 64, pl.cs, pl.m, pl.n, Cd, pl.plane_c, pl.Np, E, F,
                        C, ldc, st));
  return MDG_SUCCESS;
}

}  // namespace mdgi
