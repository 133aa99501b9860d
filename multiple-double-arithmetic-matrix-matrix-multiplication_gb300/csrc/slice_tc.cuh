// Internal interface of the slice-digit form (slice_tc.cu, diag_gemm_tc.cu).
#pragma once

#include <string>
#include <vector>

#include <cuda_runtime.h>
#include <stddef.h>

#include "mdgemm.h"

namespace mdgi {

// The diagonal sums are written as int32 "chunk" planes: the products of
// diagonal d (pairs_d digit pairs times Kp/64 k-steps of 64) are cut into
// runs of CHUNK_STEPS k-steps, at most 2032 x 64 = 130048 products of
// |d_i d_j| <= 2^14, so every chunk sum is an exact int32 with |sum| <=
// 2032 x 2^20 = 2130706432 < 2^31.  2032 is the longest run of 16-step
// flush groups that int32 holds: fewer chunk planes to write and to read
// back.  Chunks are numbered diagonal by diagonal.
constexpr int CHUNK_STEPS = 2032;
// k-steps of 64 per FP32 accumulator flush in the tcgen05 engines: 1024
// products of magnitude <= 2^14, so every partial sum is an integer with
// |sum| <= 2^24, exactly representable in FP32.
constexpr int GROUP_STEPS = 16;

__host__ __device__ inline int diag_pairs(int d, int s) {
  const int lo = d - (s - 1) > 0 ? d - (s - 1) : 0, hi = d < s - 1 ? d : s - 1;
  return hi - lo + 1;
}
// Small problems cut the diagonals into shorter chunks (`cs` k-steps), so
// that more CTAs share them.
__host__ __device__ inline int diag_chunks(int d, int s, int KB, int cs = CHUNK_STEPS) {
  return (diag_pairs(d, s) * KB + cs - 1) / cs;
}
inline int total_chunks(int s, int D, int KB, int cs = CHUNK_STEPS) {
  int c = 0;
  for (int d = 0; d < D; ++d) c += diag_chunks(d, s, KB, cs);
  return c;
}

// Workspace layout of one slice-digit GEMM (byte offsets, 256-aligned).
struct SlicePlan {
  int p, s, D, m, n, k;
  int Mp, Np, Kp;  // padded to 256, 256, 64
  int chunks;
  long long plane_a, plane_b, plane_c;  // elements between digit / chunk planes
  // sum planes behind each operand's digit planes (cross_sums.cuh); 0: the
  // diagonal sums come from digit pairs alone.  off_norms: two unsigned.
  int sums;
  int cs;  // k-steps per chunk (digit pairs)
  size_t off_bits, off_E, off_F, off_norms, off_dA, off_dB, off_Cd, total;
};

// The plan over digit pairs.
SlicePlan make_slice_plan(int p, int s, int D, int m, int n, int k);
// The plan over sum planes where that is faster; over digit pairs in shorter
// chunks for small problems; else make_slice_plan's.  Never smaller than
// make_slice_plan's.
SlicePlan best_slice_plan(int p, int s, int D, int m, int n, int k);
// The plan of a row panel by column strip block (slice_block): over sum planes,
// all of them held, where that is faster and of bounded size, else
// make_slice_plan's.
SlicePlan block_slice_plan(int p, int s, int D, int m, int n, int k);
// Tiles of the single-CTA kernel for small problems of up to 128 rows or
// columns: 128 rows by tn columns over the valid part (0: CTA pairs).
int narrow_tile(int s, int D, int m, int n, int KB);
// What engine 1 makes of a plan over digit pairs beyond 256 x 256 tiles: narrow
// tiles, or two diagonals an accumulator (stacked_tiles; chunks of CHUNK_STEPS).
// The forced engines have neither.
struct AutoTiles {
  int narrow, stack;
};
AutoTiles auto_tiles(int s, int D, int m, int n, int KB, int cs);
// 64-bit words for s digits and D diagonals, 0 where they are too many: no call
// comes with more than MAX_SLICES and MAX_DIAGONALS.
int words_for(int s, int D);
constexpr int MAX_SLICES = 119, MAX_DIAGONALS = 112;

// The FP64-DMMA slice-digit form (digits64.cu): default digits per P
// (19-bit), integer words, workspace layout and the whole GEMM.
struct Digits64Plan {
  int p, s, D, m, n, k;
  size_t off_bits, off_E, off_F, off_dA, off_dB, off_Cd, total;
};
int digits64_default(int p);
int words64_for(int s, int D);
Digits64Plan make_digits64_plan(int p, int s, int D, int m, int n, int k);
int run_digits64_gemm(const Digits64Plan &pl, const double *A, int lda, const double *B, int ldb,
                      double *C, int ldc, void *ws, cudaStream_t st);

// Scale exponents of op(A)'s rows (m of them) and op(B)'s columns (n); bits:
// m + n words of scratch.  trans_a: A is k x m; trans_b: B is n x k.
int launch_scale_exponents(int p, int m, int n, int k, const double *A, int lda,
                           const double *B, int ldb, unsigned long long *bits, int *E, int *F,
                           cudaStream_t st, int trans_a = 0, int trans_b = 0);
// Digit planes of two operands (slice_stages.cuh; rows = 0: none), and zeros
// into norms[0], norms[1] where given.
struct DigitSide;
int launch_digits(int p, int s, const DigitSide &a, const DigitSide &b, unsigned *norms,
                  cudaStream_t st);
// Engines write chunk planes of Mp x Np int32 (row stride Np).
// mma.sync engine (Mp % 128, Np % 64, Kp % 64)
int launch_diag_gemm_v0(int s, int D, int Mp, int Np, int Kp, const void *dA, const void *dB,
                        int ld, long long plane_a, long long plane_b, int *chunks,
                        long long plane_c, int cs, cudaStream_t st);
// tcgen05 engine (Mp % 128, Np % 256, Kp % 64, ld == Kp; m x n x k valid).
// engine: 2 forces 128 x 256 tiles on one CTA, 3 CTA pairs where Mp % 256 ==
// 0, else pairs or narrow tiles by size.  parts: ranges of a tile's chunks, 0
// = chosen to fill the chip.  raster:
// pair tiles run across strips this many 256-column blocks wide (0 = auto).
// pace: cross-cluster pacing window of the pair kernel in k-steps (0 = the
// default, or MDG_TC_PACE when set; -1 = off).
int launch_diag_gemm_tc(int s, int D, int Mp, int Np, int Kp, int m, int n, int k, const void *dA,
                        const void *dB, int ld, long long plane_a, long long plane_b, int *chunks,
                        long long plane_c, int cs, int engine, int parts, int raster,
                        cudaStream_t st, int pace = 0);
// Renormalisation of chunk planes (renorm.cu).
int launch_renorm(int p, int s, int D, int KB, int cs, int m, int n, const int *chunks,
                  long long plane_c, int ldcd, const int *E, const int *F, double *C, int ldc,
                  cudaStream_t st);
// One problem of a grouped diagonal GEMM: the single-CTA tcgen05 kernel
// (tiles of 128 rows x tn columns, tn = 256 or 128) or the CTA-pair kernel
// (tiles of 256 x 256; B box of 128 rows, one half per CTA).  Tensor maps of
// its digit planes, sizes, first global work unit, row tiles mt and column
// tiles nt, parts per tile, output chunk planes.  The problem's units are
// its mt x nt tiles times `parts` ranges of diagonals (whose digit-pair
// counts add up to about 1/parts of a tile's pairs each), numbered part
// after part.  ktail: MMAs of K = 16 that reach data in the last 64-deep
// k-block (1..4).  stack: stacked_tiles (pair kernel).  Lives in global memory, 64-byte
// aligned.
struct alignas(64) GroupedProblem {
  unsigned char tmA[128];  // CUtensorMap, A planes, box 64 x 128
  unsigned char tmB[128];  // CUtensorMap, B planes, box 64 x tn (pairs: 64 x 128)
  unsigned char tmC[128];  // CUtensorMap, int32 output chunk planes, box 32 x 32
  int s, D, Mp, Np, KB, unit_begin, tn, mt, nt, ktail, parts, stack;
};
// Tile shape of the pair kernel that pads an m x n problem least: 0 256 x 256,
// 1 256 x 128, 2 128 x 256 (two diagonals in one accumulator).
int stacked_tiles(int s, int D, int m, int n, int KB);
int encode_plane_map(void *map128, const void *base, int Kp, long long rows_total, int box_rows);
int encode_out_map(void *map128, const void *base, int Np, long long rows_total);
// The batched plan's entries in the tuning cache (plan.cu), under the
// current device: the tile policy and split mode recorded for a batch key,
// if any (left alone otherwise; a record without a split mode sets only the
// policy), and a new record.
void tune_lookup_batch(const std::string &key, int *policy, int *split);
void tune_record_batch(const std::string &key, int policy, int split, double ms);
// The units of the table over the workers (CTAs, or CTA pairs): worker w takes
// order[starts[w]] .. order[starts[w + 1] - 1].
int deal_units(const std::vector<GroupedProblem> &probs, int workers, std::vector<int> *starts,
               std::vector<int> *order);
// pair: the CTA-pair kernel (Mp of every problem a multiple of 256).
int launch_diag_gemm_grouped(const GroupedProblem *dev_probs, int count, int workers,
                             const int *dev_starts, const int *dev_order, int pair,
                             cudaStream_t st);

// Waits for the device; MDG_ERROR_TIMEOUT if a bounded wait of the tcgen05
// engine gave up since the last call (the flag is then cleared).
int tc_device_status();

// engine: 0 = mma.sync, 1 = tcgen05 auto tiles, 2 = tcgen05 single CTA,
// 3 = tcgen05 CTA pairs
int run_slice_gemm(const SlicePlan &pl, const double *A, int lda, const double *B, int ldb,
                   double *C, int ldc, void *ws, int engine, int parts, int raster,
                   cudaStream_t st, int pace = 0, int trans_a = 0, int trans_b = 0);

// mdg_gemm of the BF16 form on checked arguments, m, n, k > 0, with operands
// that may be given transposed (A k x m, B n x k): the digit planes are
// formed from either layout.
int slice_gemm(int p, int m, int n, int k, const double *A, int lda, int trans_a, const double *B,
               int ldb, int trans_b, double *C, int ldc, const mdg_options *opt, void *workspace,
               size_t workspace_bytes, void *stream);

// run_slice_gemm in parts, for the host entry, which splits A into row panels and
// B into column strips (each with its own plan and workspace): slice_prepare_b
// computes a strip's exponents, digits and sums once, slice_panel_a those of
// rows (<= pl.m) rows of A into wsa, slice_block then those rows of C against the
// strip of plb / wsb (plans of equal m, k, s, D).  A row of C depends only on its
// row of A and a column only on its column of B, so blocks give the bits of one
// run_slice_gemm.
int slice_prepare_b(const SlicePlan &pl, const double *B, int ldb, void *ws, cudaStream_t st);
int slice_panel_a(const SlicePlan &pl, int rows, const double *A, int lda, void *ws,
                  cudaStream_t st);
int slice_block(const SlicePlan &pla, const void *wsa, const SlicePlan &plb, void *wsb, int rows,
                double *C, int ldc, int engine, int parts, int raster, cudaStream_t st,
                int pace = 0);

// Which engine mdg_gemm uses for the BF16 form (MDG_SLICE_ENGINE=0/1 overrides).
int default_engine();
// mdg_options.engine -> run_slice_gemm engine code.
int engine_choice(int opt);

}  // namespace mdgi
