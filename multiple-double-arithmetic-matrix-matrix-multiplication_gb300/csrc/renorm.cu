// Renormalisation kernels of one problem (renorm.cuh).
#include <algorithm>

#include "batched_table.cuh"
#include "common.cuh"
#include "renorm.cuh"

namespace {

using mdgi::RENORM_THREADS;

// Two columns a thread halve the loads and the address work, one column
// doubles the threads and leaves more blocks their shared memory.  Two / one:
// dd 16001 x 96 58 / 68 us, qd 8192 x 8192 (cross form) 6.8 / 7.6 ms, qd 1024
// x 1024 92 / 92 us; with the prefix sums of 55 and 110 diagonals od 2048 x
// 2048 1275 / 833, hd 1024 x 1024 1120 / 630 us.  Beyond 32 diagonals the kernel
// that keeps no prefix sums, where each diagonal is one chunk: od 2048 x 2048
// one column with prefix sums 690, without 691, two columns 593 us; hd 1024 x
// 1024 549, 324, 296; but qd 2048 x 2048 308 (two columns), 350, 313, dd 3000 x
// 3000 293, 459, 417.
//
// From 2^17 entries on.  The kernel alone, one / two: dd 14 diagonals 512 x 512
// 18.5 / 10.4, 256 x 512 11.1 / 8.3 us; qd 28 of them 512 x 512 31.9 / 18.4, 256 x
// 512 18.5 / 12.4, 256 x 256 12.1 / 10.3.  But problems below cut their diagonals
// into short chunks, which one column loads four at a time: whole calls qd 256^3
// 57.4 / 59.4, 128^3 49.3 / 53.2, od 128^3 63.7 / 69.8, qd 400^3 122 / 110, 700 x
// 700 x 256 172 / 142, hd 500 x 500 x 70 425 / 378.
constexpr long long kTwoColumnEntries = 1 << 17;
constexpr int kTwoColumnDiagonals = 32;

// Threads run over the rows' groups of V columns, row after row.  (Blocks per
// SM: with two columns the registers otherwise leave 5, and the kernel waits
// for its loads: dd 16001 x 96 60 -> 48 us with 7, qd 8192 x 8192, cross form,
// 6.97 -> 6.30 ms with 6, 64 mixed problems 375 -> 325 us with 7.)
template <int V>
__global__ void __launch_bounds__(RENORM_THREADS, V == 2 ? 7 : 1)
    renorm_kernel(int P, int D, int planes, int top, const __grid_constant__ mdgi::ChunkCounts counts,
                  int m, int n, const int *__restrict__ chunks, long long plane_c, int ldcd,
                  const int *__restrict__ E, const int *__restrict__ F, double *__restrict__ C,
                  int ldc, bool wide) {
  extern __shared__ uint4 smem[];
  const int groups = (n + V - 1) / V;
  const long long e = blockIdx.x * (long long)RENORM_THREADS + threadIdx.x;
  const int r = (int)(e / groups), c0 = (int)(e - (long long)r * groups) * V;
  if (r >= m) return;
  mdgi::renorm_columns<V, mdgi::kTableChunks>(P, 0, D, 0, planes, top, n, &counts, chunks, plane_c, ldcd,
                                              E, F, C, ldc, r, c0, wide, smem);
}

template <int V>
__global__ void __launch_bounds__(RENORM_THREADS, V == 2 ? 6 : 1)
    cross_renorm_kernel(int P, int D, int planes, int top, const __grid_constant__ mdgi::ChunkCounts counts,
                        int m, int n, const int *__restrict__ out, long long plane_c, int ldcd,
                        const int *__restrict__ E, const int *__restrict__ F,
                        double *__restrict__ C, int ldc, bool wide) {
  extern __shared__ uint4 smem[];
  const int groups = (n + V - 1) / V;
  const long long e = blockIdx.x * (long long)RENORM_THREADS + threadIdx.x;
  const int r = (int)(e / groups), c0 = (int)(e - (long long)r * groups) * V;
  if (r >= m) return;
  mdgi::renorm_columns<V, mdgi::kCrossChunks>(P, 0, D, 0, planes, top, n, &counts, out, plane_c, ldcd, E,
                                              F, C, ldc, r, c0, wide, smem);
}

// The same where no diagonal has more than one chunk, without prefix sums in
// shared memory: those of 110 diagonals left 12 warps on an SM.
template <int V>
__global__ void __launch_bounds__(RENORM_THREADS, V == 2 ? 5 : 8)
    whole_renorm_kernel(int P, int D, int planes, int top, const __grid_constant__ mdgi::ChunkCounts counts,
                        int m, int n, const int *__restrict__ out, long long plane_c, int ldcd,
                        const int *__restrict__ E, const int *__restrict__ F,
                        double *__restrict__ C, int ldc, bool wide) {
  extern __shared__ uint4 smem[];
  const int groups = (n + V - 1) / V;
  const long long e = blockIdx.x * (long long)RENORM_THREADS + threadIdx.x;
  const int r = (int)(e / groups), c0 = (int)(e - (long long)r * groups) * V;
  if (r >= m) return;
  mdgi::renorm_columns<V, mdgi::kCrossWhole>(P, 0, D, 0, planes, top, n, &counts, out, plane_c, ldcd, E,
                                             F, C, ldc, r, c0, wide, smem);
}

// Every problem of a batch: block x belongs to the problem whose units hold x.
__global__ void __launch_bounds__(RENORM_THREADS, 7)
    batch_renorm_kernel(const mdgi::BatchProblem *__restrict__ pr, int count,
                        const int *__restrict__ exps) {
  extern __shared__ uint4 smem[];
  const int x = blockIdx.x;
  const mdgi::BatchProblem &b = pr[mdgi::find_problem<mdgi::kRenormUnits>(pr, count, x)];
  const int groups = (b.n + 1) / 2;
  const long long e = (x - b.out_begin) * (long long)RENORM_THREADS + threadIdx.x;
  const int r = (int)(e / groups), c0 = (int)(e - (long long)r * groups) * 2;
  if (r >= b.m) return;
  mdgi::renorm_columns<2, mdgi::kPlainChunks>(b.p, b.s, b.D, b.Kp / 64, b.planes, b.top, b.n, nullptr,
                                              b.chunks, b.plane_c, b.Np, exps + b.offE,
                                              exps + b.offF, b.C, b.ldc, r, c0, b.wide, smem);
}

bool aligned16(const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// The chip is filled anyway and the planes are aligned for 8-byte loads.
bool two_columns(int m, int n, const int *chunks, long long plane_c, int ldcd) {
  return (long long)m * n >= kTwoColumnEntries && ldcd % 2 == 0 && plane_c % 2 == 0 &&
         reinterpret_cast<uintptr_t>(chunks) % 8 == 0;
}

unsigned blocks(int m, int n, int V) {
  return mdgi::ceil_div((long long)m * ((n + V - 1) / V), RENORM_THREADS);
}

template <int V>
int launch_direct(int p, int s, int D, int KB, int cs, int m, int n, const int *chunks,
                  long long plane_c, int ldcd, const int *E, const int *F, double *C, int ldc,
                  cudaStream_t st) {
  mdgi::ChunkCounts counts{};
  int planes = 0, most = 1;
  for (int d = 0; d < D; ++d) {
    const int nc = mdgi::diag_chunks(d, s, KB, cs);
    counts.of[d] = nc;
    planes += nc;
    most = std::max(most, nc);
  }
  const int smem = mdgi::renorm_smem(D, V, false);
  MDG_TRY(mdgi::allow_smem(renorm_kernel<V>, smem, mdgi::renorm_smem(mdgi::MAX_DIAGONALS, V, false)));
  renorm_kernel<V><<<blocks(m, n, V), RENORM_THREADS, smem, st>>>(
      p, D, planes, mdgi::renorm_top(D, most), counts, m, n, chunks, plane_c, ldcd, E, F, C, ldc, aligned16(C));
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

template <int V>
int launch_cross(int p, int D, int KB, int m, int n, const int *out, long long plane_c, int ldcd,
                 const int *E, const int *F, double *C, int ldc, cudaStream_t st) {
  mdgi::ChunkCounts counts{};
  counts.pairs_per_chunk = mdgi::cross_pairs_per_chunk(KB);
  int most = 0;
  for (int d = 1; d < D; ++d) {
    counts.of[d] = mdgi::cross_chunks(d, counts.pairs_per_chunk);
    most = std::max(most, (int)counts.of[d]);
  }
  const bool whole = most <= 1 && D > kTwoColumnDiagonals;
  const int smem = mdgi::renorm_smem(D, V, !whole);
  const auto kernel = whole ? whole_renorm_kernel<V> : cross_renorm_kernel<V>;
  MDG_TRY(mdgi::allow_smem(kernel, smem, mdgi::renorm_smem(mdgi::MAX_DIAGONALS, V, !whole)));
  kernel<<<blocks(m, n, V), RENORM_THREADS, smem, st>>>(
      p, D, mdgi::cross_outputs(D, KB), mdgi::renorm_top(D, most + 1), counts, m, n, out, plane_c, ldcd, E, F, C, ldc,
      aligned16(C));
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

}  // namespace

namespace mdgi {

int launch_renorm(int p, int s, int D, int KB, int cs, int m, int n, const int *chunks,
                  long long plane_c, int ldcd, const int *E, const int *F, double *C, int ldc,
                  cudaStream_t st) {
  if (m == 0 || n == 0) return MDG_SUCCESS;
  if (!words_for(1, D) || D > 128) return MDG_ERROR_NOT_SUPPORTED;
  if (two_columns(m, n, chunks, plane_c, ldcd))
    return launch_direct<2>(p, s, D, KB, cs, m, n, chunks, plane_c, ldcd, E, F, C, ldc, st);
  return launch_direct<1>(p, s, D, KB, cs, m, n, chunks, plane_c, ldcd, E, F, C, ldc, st);
}

int launch_cross_renorm(int p, int D, int KB, int m, int n, const int *out, long long plane_c,
                        int ldcd, const int *E, const int *F, double *C, int ldc,
                        cudaStream_t st) {
  if (m == 0 || n == 0) return MDG_SUCCESS;
  if (!words_for(1, D) || KB > CROSS_CHUNK_STEPS) return MDG_ERROR_NOT_SUPPORTED;
  // 'whole', beyond kTwoColumnDiagonals: the last diagonal's pairs fit a chunk
  const bool two = D <= kTwoColumnDiagonals || cross_pairs(D - 1) <= cross_pairs_per_chunk(KB);
  if (two && two_columns(m, n, out, plane_c, ldcd))
    return launch_cross<2>(p, D, KB, m, n, out, plane_c, ldcd, E, F, C, ldc, st);
  return launch_cross<1>(p, D, KB, m, n, out, plane_c, ldcd, E, F, C, ldc, st);
}

int launch_batch_renorm(const BatchProblem *pr, int count, int units, int max_d, const int *exps,
                        cudaStream_t st) {
  if (units == 0) return MDG_SUCCESS;
  const int smem = renorm_smem(max_d, 2, false);
  MDG_TRY(allow_smem(batch_renorm_kernel, smem, renorm_smem(MAX_DIAGONALS, 2, false)));
  batch_renorm_kernel<<<units, RENORM_THREADS, smem, st>>>(pr, count, exps);
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

}  // namespace mdgi
