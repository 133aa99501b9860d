// Diagonal GEMM of digit planes on the 5th-generation tensor cores.
//
// For every output tile (128 rows x 256 columns) and every diagonal d < D,
// the products A_i B_j^T with i + j = d are summed over k exactly: BF16
// digits in [-128, 128], FP32 accumulation in tensor memory (TMEM), flushed
// every 1024 products (|partial| <= 2^24) into int32 registers, stored every
// 2032 k-steps (130048 products) as one int32 chunk plane (|sum| < 2^31).
//
// One CTA per SM, persistent over tiles; 10 warps with fixed roles:
//   warp 0      TMA producer: A_i (128 x 64) and B_j (256 x 64) k-blocks
//               into a 4-stage shared-memory ring (128-byte swizzle),
//   warp 1      TMEM allocator and MMA issuer: tcgen05.mma kind::f16,
//               M=128 N=256 K=16, BF16 x BF16 -> FP32, into one of two
//               256-column accumulators (all 512 TMEM columns),
//   warps 2-9   epilogue: tcgen05.ld of the accumulator (warp w reads TMEM
//               lanes 32 (w % 4) .. +31, columns 128 ((w - 2) / 4) .. +127)
//               every 16 k-steps, exact float -> int conversion, int32
//               accumulation, chunk stores.
// Barriers: full/empty per stage (TMA <-> MMA), accfull/accempty per
// accumulator (MMA <-> epilogue).  Every wait is bounded (2 s of
// %globaltimer); on a timeout the CTA records the error, stops issuing,
// waits (bounded) for its copies and MMAs in flight, frees TMEM and exits.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <functional>
#include <queue>
#include <utility>
#include <vector>

#include "common.cuh"
#include "cross_sums.cuh"
#include "slice_tc.cuh"

namespace {

constexpr int TM = 128, TN = 256, TK = 64;
constexpr int STAGES = 4;
constexpr int A_BYTES = TM * TK * 2;  // 16 KiB
constexpr int B_BYTES = TN * TK * 2;  // 32 KiB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 32 * (2 + EPI_WARPS);
constexpr int TMEM_COLS = 512;
// per epilogue warp: a 32 x 32 int32 block on its way out
constexpr int OUT_BYTES = 32 * 32 * 4;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + EPI_WARPS * OUT_BYTES + 1024 /* align */ +
                           256 /* barriers */;
constexpr unsigned long long TIMEOUT_NS = 2000000000ull;

// kind::f16 instruction descriptor: D F32 (bits 4-5 = 1), A BF16 (7-9 = 1),
// B BF16 (10-12 = 1), both K-major (bits 15, 16 = 0), N >> 3 at bit 17,
// M >> 4 at bit 24.
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) |
                           ((uint32_t)(TM >> 4) << 24);

__device__ int g_tc_error = 0;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait.  Returns false on a timeout (and raises the CTA's abort
// flag) or when another role has already aborted.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort) {
  if (mbar_test(bar, parity)) return true;
  const unsigned long long t0 = now_ns();
  while (true) {
    if (mbar_test(bar, parity)) return true;
    if (*abort) return false;
    if (now_ns() - t0 > TIMEOUT_NS) {
      *abort = 1;
      return false;
    }
  }
}

// Bounded wait that ignores the abort flag (draining in-flight work).
__device__ __forceinline__ void mbar_drain(uint32_t bar, uint32_t parity) {
  const unsigned long long t0 = now_ns();
  while (!mbar_test(bar, parity) && now_ns() - t0 < TIMEOUT_NS) {
  }
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *tm, int x, int y,
                                            uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: start address
// >> 4 (bits 0-13), leading byte offset 16 B (unused for this layout,
// bits 16-29), stride byte offset 1024 B between 8-row groups (bits 32-45),
// descriptor version 1 (bits 46-47), swizzle mode 2 = 128 B (bits 61-63).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFF) >> 4) | ((uint64_t)(16 >> 4) << 16) |
         ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

// idesc: IDESC with the tile width of the job.
__device__ __forceinline__ void mma_bf16_n(uint32_t d_tmem, uint64_t a, uint64_t b,
                                           uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
      : "memory");
}

__device__ __forceinline__ void fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Asynchronous TMEM load of 32 columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
      "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
        "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]),
        "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
        "=r"(r[31])
      : "r"(taddr));
}

// Waits for this thread's outstanding TMEM loads.  The registers of the
// last load are operands, so no read of them can move above the wait.
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                 "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]),
                 "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]),
                 "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]),
                 "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// The accumulator holds integer-valued floats with |x| <= 2^24; the
// conversion to int32 is exact.  Sums of sum planes' products are taken modulo
// 2^32 (cross_sums.cuh), so without sign.
__device__ __forceinline__ void add_exact(int *acc, const uint32_t (&r)[32]) {
#pragma unroll
  for (int j = 0; j < 32; ++j)
    acc[j] = (int)((uint32_t)acc[j] + (uint32_t)__float2int_rn(__uint_as_float(r[j])));
}

// Adds 128 accumulator columns (starting at taddr) into acc: four 32-column
// loads, each issued before the previous block is converted so that the
// load latency overlaps the integer work.
__device__ __forceinline__ void drain128(uint32_t taddr, int (&acc)[128]) {
  uint32_t ra[32], rb[32];
  tmem_ld32(taddr, ra);
  tmem_wait(ra);
  tmem_ld32(taddr + 32, rb);
  add_exact(acc, ra);
  tmem_wait(rb);
  tmem_ld32(taddr + 64, ra);
  add_exact(acc + 32, rb);
  tmem_wait(ra);
  tmem_ld32(taddr + 96, rb);
  add_exact(acc + 64, ra);
  tmem_wait(rb);
  add_exact(acc + 96, rb);
}

// Stores a warp's 32 rows x 128 columns of int32 sums (row = lane) at (x, y)
// of the output planes and clears them.  Through shared memory and the TMA,
// 32 columns at a time: a thread holds a row, so storing from registers
// touches 32 lines per instruction and the L1 takes them one a cycle (8192
// cycles for a CTA's 128 x 256 block, as long as a whole flush group, during
// which the accumulators are not drained).  The staging block has the
// 128-byte swizzle of the tensor map, so the 16-byte writes of eight rows
// hit different banks.  Against stores from registers: double-double 64^3
// 119 -> 106 us, a batch of 64 mixed problems 4.09 -> 3.84 ms a call.
__device__ __forceinline__ void store_rows(uint32_t staging, int lane, int (&acc)[128],
                                           const CUtensorMap *tm, int x, int y) {
  const uint32_t line = staging + lane * 128;
#pragma unroll
  for (int cb = 0; cb < 4; ++cb) {
    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    __syncwarp();
#pragma unroll
    for (int v = 0; v < 8; ++v) {
      int *a = acc + 32 * cb + 4 * v;
      asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(
                       line + ((uint32_t)(v ^ (lane & 7)) << 4)),
                   "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3])
                   : "memory");
      a[0] = a[1] = a[2] = a[3] = 0;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
      asm volatile(
          "cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
              reinterpret_cast<uint64_t>(tm)),
          "r"(x + 32 * cb), "r"(y), "r"(staging)
          : "memory");
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
  }
}

// Waits until this thread's stores have been written.
__device__ __forceinline__ void stores_done() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// A run of plane products that goes into one output plane: `steps` k-steps
// from step t0 of the products of planes (a0 + astep p, b0 + bstep p), KB
// k-steps each, p = 0, 1, ..  cuts: flush groups per plane (sums form).
struct Run {
  int a0, astep, b0, bstep, t0, steps, chunk, cuts;
};

// Two diagonals in one 256 x 256 accumulator, for problems that waste less on
// tiles of 128: the second half of B's rows (kStackN), or of A's (kStackM),
// is the next digit plane instead of the next 128 columns (rows), so that
// the halves of the accumulator are diagonals d and d + 1 of a 256 x 128
// (128 x 256) tile.  A step too many at one end of d is a plane -1, which the
// TMA fills with zeros.  Pair kernel, D <= s, one chunk per diagonal.  Dd 14
// digits: 56 steps for the tile of 128 instead of 105 for one of 256 that is
// half padding; dd 16001 x 96 x 3001 2.50 -> 1.73 ms a call (its GEMM streams
// A's planes from DRAM, 56 instead of 105 times 97 MB), 64 mixed problems of
// 32 .. 512 3.15 -> 2.69 ms.
enum { kStackNone = 0, kStackN = 1, kStackM = 2 };

// Runs over digit planes: the chunks (cs k-steps) of the diagonals; stacked,
// pairs of diagonals from the top down, an odd first one with d = -1.
struct DigitRuns {
  int s, D, KB, cs, stack, d, c, chunk, left;
  __host__ __device__ bool next(Run &r) {
    if (left <= 0 || d >= D) return false;
    if (stack) {
      r = stack == kStackN ? Run{0, 1, d, -1, 0, (d + 2) * KB, d, 0}
                           : Run{d, -1, 0, 1, 0, (d + 2) * KB, d, 0};
      d += 2;
      --left;
      return true;
    }
    const int S = mdgi::diag_pairs(d, s) * KB;
    r.a0 = d - (s - 1) > 0 ? d - (s - 1) : 0;
    r.b0 = d - r.a0;
    r.astep = 1;
    r.bstep = -1;
    r.t0 = c * cs;
    r.steps = S - r.t0 < cs ? S - r.t0 : cs;
    r.chunk = chunk++;
    --left;
    if (r.t0 + cs < S) {
      ++c;
    } else {
      ++d;
      c = 0;
    }
    return true;
  }
  // FP32 flushes every GROUP_STEPS k-steps, whatever plane they fall in
  struct Groups {
    int left;
    __device__ Groups(const Run &r, int) : left(r.steps) {}
    __device__ int next() {  // k-steps of the next flush group, 0 at the end
      const int n = left < mdgi::GROUP_STEPS ? left : mdgi::GROUP_STEPS;
      left -= n;
      return n;
    }
    __device__ bool last() const { return left == 0; }
  };
};

// Part `part` of a tile's runs: run `part` itself where there are as many
// parts as runs, else the runs that start in the part's 1/parts of the
// tile's k-steps (none when parts exceeds what the runs allow).
__host__ __device__ __forceinline__ DigitRuns part_runs(int s, int D, int KB, int cs, int stack, int part,
                                               int parts) {
  DigitRuns all{s, D, KB, cs, stack, stack ? -(D & 1) : 0, 0, 0, 1 << 30};
  if (parts == 1) return all;
  long long steps = 0;
  int runs = 0;
  if (stack) {
    for (int d = -(D & 1); d < D; d += 2, ++runs) steps += (d + 2) * KB;
  } else {
    for (int d = 0; d < D; ++d) {
      steps += mdgi::diag_pairs(d, s) * KB;
      runs += mdgi::diag_chunks(d, s, KB, cs);
    }
  }
  const bool one = parts == runs;
  const long long lo = one ? part : steps * part / parts;
  const long long hi = one ? part + 1 : steps * (part + 1) / parts;
  Run r;
  long long at = 0;
  while (at < lo && all.next(r)) at += one ? 1 : r.steps;
  DigitRuns first = all;
  first.left = 0;
  while (at < hi && all.next(r)) {
    at += one ? 1 : r.steps;
    ++first.left;
  }
  return first;
}

// One unit of work: where its operands and output live, which of its
// problem's rows / columns it covers and which runs it computes.  tn: tile
// width, 256 or 128 columns (the B box of tmB is tn rows); ktail: MMAs of
// K = 16 issued for the last k-block (1..4; the rest of that block is the
// zero padding of k).
struct TileJob {
  const CUtensorMap *tmA, *tmB, *tmC;
  int Mp, Np, KB, row, col, tn, ktail;
  DigitRuns runs;
};

// Workers (CTAs or clusters) take the units of a single problem in turn.
struct DealtInTurn {
  __device__ int first(int worker, int) const { return worker; }
  __device__ int step(int workers) const { return workers; }
  __device__ int unit(int i) const { return i; }
};

// A single problem cut into mt x nt tiles of 128 x tn, each into parts.
struct SingleJobs : DealtInTurn {
  const CUtensorMap *tmA, *tmB, *tmC;
  int s, D, Mp, Np, KB, cs, tn, mt, nt, parts;
  __device__ int last(int) const { return mt * nt * parts; }
  __device__ TileJob job(int u) const {
    const int tiles = mt * nt, tile = u % tiles;
    return TileJob{tmA, tmB, tmC, Mp, Np, KB, (tile % mt) * TM, (tile / mt) * tn, tn, TK / 16,
                   part_runs(s, D, KB, cs, kStackNone, u / tiles, parts)};
  }
};

template <class Jobs>
__device__ __forceinline__ void tc1_body(const Jobs &jobs) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t *bars = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE_BYTES + EPI_WARPS * OUT_BYTES);
  // bars: [0,4) full, [4,8) empty, [8,10) accfull, [10,12) accempty, 12 mma drain
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bars + 16);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 17);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t smem_base = smem_u32(smem);
  auto full = [&](int st) { return smem_u32(bars + st); };
  auto empty = [&](int st) { return smem_u32(bars + STAGES + st); };
  auto accfull = [&](int b) { return smem_u32(bars + 2 * STAGES + b); };
  auto accempty = [&](int b) { return smem_u32(bars + 2 * STAGES + 2 + b); };
  const uint32_t drain_bar = smem_u32(bars + 2 * STAGES + 4);

  if (threadIdx.x == 0) {
    for (int st = 0; st < STAGES; ++st) {
      mbar_init(full(st), 1);
      mbar_init(empty(st), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(accfull(b), 1);
      mbar_init(accempty(b), EPI_WARPS);
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_holder)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem_base = *tmem_holder;

  const int worker = blockIdx.x, first = jobs.first(worker, gridDim.x);
  const int last = jobs.last(worker), step = jobs.step(gridDim.x);

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------------ producer --
      int st = 0;
      uint32_t ph = 0;
      // per stage: a copy was issued (bit of `issued`), parity of its phase
      // (bit of `last_par`); bit masks so that they stay in registers
      uint32_t issued = 0, last_par = 0;
      for (int i = first; i < last; i += step) {
        TileJob jb = jobs.job(jobs.unit(i));
        const int KB = jb.KB;
        Run r;
        while (jb.runs.next(r)) {
          for (int t = r.t0; t < r.t0 + r.steps; ++t) {
            const int q = t / KB, kb = t - q * KB, pa = r.a0 + q, pb = r.b0 - q;
            if (!mbar_wait(empty(st), ph ^ 1, abort_flag)) goto producer_done;
            mbar_expect_tx(full(st), A_BYTES + jb.tn * TK * 2);
            const uint32_t a_dst = smem_base + st * STAGE_BYTES;
            tma_load_2d(a_dst, jb.tmA, kb * TK, pa * jb.Mp + jb.row, full(st));
            tma_load_2d(a_dst + A_BYTES, jb.tmB, kb * TK, pb * jb.Np + jb.col, full(st));
            last_par = (last_par & ~(1u << st)) | (ph << st);
            issued |= 1u << st;
            if (++st == STAGES) {
              st = 0;
              ph ^= 1;
            }
          }
        }
      }
    producer_done:
      if (*abort_flag)
        for (int i = 0; i < STAGES; ++i)
          if ((issued >> i) & 1u) mbar_drain(full(i), (last_par >> i) & 1u);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ---------------------------------------------------- MMA issuer --
      int st = 0, buf = 0;
      uint32_t ph = 0, aph[2] = {0, 0};
      bool any = false;
      for (int i = first; i < last; i += step) {
        TileJob jb = jobs.job(jobs.unit(i));
        const uint32_t idesc = (IDESC & ~(0x3Fu << 17)) | ((uint32_t)(jb.tn >> 3) << 17);
        Run r;
        while (jb.runs.next(r)) {
          int kb = r.t0 % jb.KB;  // k-block of a step within its digit pair
          DigitRuns::Groups groups(r, jb.KB);
          for (int steps; (steps = groups.next()) > 0;) {
            if (!mbar_wait(accempty(buf), aph[buf] ^ 1, abort_flag)) goto mma_done;
            fence_after();
            const uint32_t dt = tmem_base + buf * TN;
            for (int t = 0; t < steps; ++t) {
              if (!mbar_wait(full(st), ph, abort_flag)) goto mma_done;
              fence_after();
              const uint32_t a_addr = smem_base + st * STAGE_BYTES;
              const uint64_t da = sw128_desc(a_addr), db = sw128_desc(a_addr + A_BYTES);
              // the last k-block of a pair: only the MMAs that reach data
              const bool short_block = kb == jb.KB - 1 && jb.ktail < TK / 16;
              if (++kb == jb.KB) kb = 0;
              if (!short_block) {
#pragma unroll
                for (int kk = 0; kk < TK / 16; ++kk)
                  mma_bf16_n(dt, da + 2 * kk, db + 2 * kk, idesc, (t > 0 || kk > 0) ? 1u : 0u);
              } else {
                for (int kk = 0; kk < jb.ktail; ++kk)
                  mma_bf16_n(dt, da + 2 * kk, db + 2 * kk, idesc, (t > 0 || kk > 0) ? 1u : 0u);
              }
              mma_commit(empty(st));
              any = true;
              if (++st == STAGES) {
                st = 0;
                ph ^= 1;
              }
            }
            mma_commit(accfull(buf));
            aph[buf] ^= 1;
            buf ^= 1;
          }
        }
      }
    mma_done:
      if (*abort_flag && any) {
        mma_commit(drain_bar);
        mbar_drain(drain_bar, 0);
      }
    }
  } else {
    // -------------------------------------------------------- epilogue --
    const int q = warp & 3, h = (warp - 2) >> 2;
    const uint32_t staging = smem_base + STAGES * STAGE_BYTES + (warp - 2) * OUT_BYTES;
    int acc[128];
#pragma unroll
    for (int j = 0; j < 128; ++j) acc[j] = 0;
    int buf = 0;
    uint32_t aph[2] = {0, 0};
    for (int i = first; i < last; i += step) {
      TileJob jb = jobs.job(jobs.unit(i));
      // a 128-column tile is drained by the warps of the first column half
      // alone (128 columns each, as for a 256-column tile); the others only
      // release the accumulator
      const bool active = jb.tn == TN || h == 0;
      const int row = jb.row + 32 * q;
      const int col = jb.col + 128 * h;
      Run r;
      while (jb.runs.next(r)) {
        DigitRuns::Groups groups(r, jb.KB);
        while (groups.next() > 0) {
          // lane 0 waits; the outcome is broadcast so the warp stays
          // converged for the .sync.aligned TMEM loads
          int ok = 1;
          if (lane == 0) ok = mbar_wait(accfull(buf), aph[buf], abort_flag) ? 1 : 0;
          ok = __shfl_sync(0xffffffffu, ok, 0);
          if (!ok) goto epi_done;
          aph[buf] ^= 1;
          fence_after();
          const uint32_t taddr = tmem_base + ((uint32_t)(32 * q) << 16) + buf * TN + 128 * h;
          if (active) drain128(taddr, acc);
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(accempty(buf));
          buf ^= 1;
          if (groups.last() && active)
            store_rows(staging, lane, acc, jb.tmC, col, r.chunk * jb.Mp + row);
        }
      }
    }
  epi_done:
    if (lane == 0) stores_done();
  }
  __syncwarp();
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(TMEM_COLS)
                 : "memory");
  if (threadIdx.x == 0 && *abort_flag) atomicExch(&g_tc_error, 1);
}


__global__ void __launch_bounds__(THREADS, 1)
    diag_gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA,
                        const __grid_constant__ CUtensorMap tmB,
                        const __grid_constant__ CUtensorMap tmC, int s, int D, int Mp, int Np,
                        int KB, int cs, int tn, int mt, int nt, int parts) {
  tc1_body(SingleJobs{{}, &tmA, &tmB, &tmC, s, D, Mp, Np, KB, cs, tn, mt, nt, parts});
}

// Many problems: a table of GroupedProblem in global memory (tensor maps
// included, 64-byte aligned), units numbered problem after problem and,
// within a problem, part after part (all tiles of one diagonal range, then
// the next range).
__device__ __forceinline__ const mdgi::GroupedProblem &grouped_find(
    const mdgi::GroupedProblem *probs, int count, int u) {
  int lo = 0, hi = count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (probs[mid].unit_begin <= u) lo = mid; else hi = mid - 1;
  }
  return probs[lo];
}

// Units dealt by the host: worker w takes order[starts[w]] .. .
struct DealtByHost {
  const int *starts, *order;
  __device__ int first(int worker, int) const { return starts[worker]; }
  __device__ int last(int worker) const { return starts[worker + 1]; }
  __device__ int step(int) const { return 1; }
  __device__ int unit(int i) const { return order[i]; }
};

struct GroupedJobs : DealtByHost {
  const mdgi::GroupedProblem *probs;
  int count;
  __device__ TileJob job(int u) const {
    const mdgi::GroupedProblem &g = grouped_find(probs, count, u);
    const int lt = u - g.unit_begin, tiles = g.mt * g.nt;
    const int tile = lt % tiles, part = lt / tiles;
    return TileJob{reinterpret_cast<const CUtensorMap *>(g.tmA),
                   reinterpret_cast<const CUtensorMap *>(g.tmB),
                   reinterpret_cast<const CUtensorMap *>(g.tmC), g.Mp, g.Np, g.KB,
                   (tile % g.mt) * TM, (tile / g.mt) * g.tn, g.tn, g.ktail,
                   part_runs(g.s, g.D, g.KB, mdgi::CHUNK_STEPS, kStackNone, part, g.parts)};
  }
};

__global__ void __launch_bounds__(THREADS, 1)
    diag_gemm_tc_grouped_kernel(const mdgi::GroupedProblem *__restrict__ probs, int count,
                                const int *__restrict__ starts, const int *__restrict__ order) {
  tc1_body(GroupedJobs{{starts, order}, probs, count});
}

// ------------------------------------------------------------------------
// The same computation on CTA pairs (cta_group::2): a cluster of two CTAs
// owns a 256 x 256 output tile; CTA r holds rows r*128..+127 of the A
// k-block and rows r*128..+127 of the B k-block (the N half), and the pair's
// tensor cores compute M=256 N=256 K=16 per instruction, issued by one thread
// of the even CTA.  Each CTA streams 32 KiB per k-step instead of 48 and its
// tensor core reads 8 KiB of operands per 128-cycle MMA instead of 12, which
// halves the shared-memory traffic that bounds the single-CTA kernel.
// Synchronisation: both CTAs' TMA loads complete on the even CTA's full
// barrier (cp.async.bulk.tensor .cta_group::2); the even CTA's MMA commits
// arrive, multicast, on the empty and accumulator-full barriers of both
// CTAs; the epilogue warps of both CTAs arrive on the even CTA's
// accumulator-empty barrier (16 arrivals).  Each CTA's TMEM holds its 128
// rows of both accumulators.  Warps: 0 producer, 1 MMA issuer (even CTA),
// 2-9 epilogue, 10 the pacer (even CTA; see "Pacing across clusters").
// Work units are tiles, or parts of tiles (ranges of diagonals), taken in
// strips of `raster` column blocks.
constexpr int TN2 = 256, BH = 128;
constexpr int STAGES2 = 6;
constexpr int A2_BYTES = TM * TK * 2;  // 16 KiB
constexpr int B2_BYTES = BH * TK * 2;  // 16 KiB
constexpr int STAGE2_BYTES = A2_BYTES + B2_BYTES;
constexpr int SMEM2_BYTES = STAGES2 * STAGE2_BYTES + EPI_WARPS * OUT_BYTES + 1024 + 256;
constexpr uint32_t IDESC2 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN2 >> 3) << 17) |
                            ((uint32_t)(256 >> 4) << 24);

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}

__device__ __forceinline__ uint32_t map_to_rank0(uint32_t addr) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
  return r;
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}

__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *tm, int x, int y,
                                                 uint32_t bar_cluster) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(bar_cluster)
      : "memory");
}

__device__ __forceinline__ void mma_bf16_pair(uint32_t d_tmem, uint64_t a, uint64_t b,
                                              uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(IDESC2), "r"(acc));
}

__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {
  const uint16_t mask = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;" ::"r"(bar),
      "h"(mask)
      : "memory");
}

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster)
               : "memory");
}

// Pacing across clusters.  Clusters that keep the same pace read the same
// k-blocks of the same digit planes at about the same time, so each block
// comes from DRAM once and from L2 for the others; left alone they drift
// apart by more than L2 holds and most blocks come from DRAM again.  An
// eleventh warp of the even CTA (the pacer) publishes its producer's
// progress (k-steps issued, tagged with the launch's epoch) to a slot per
// cluster and posts, in shared memory, how far the producer may go: the
// slowest running cluster's progress plus `pace` k-steps.  The producer
// holds before a k-step beyond that.  Only the timing depends on it: a hold
// longer than PACE_WAIT_NS turns the pacing off for the rest of the launch
// in that CTA, so a cluster that is not resident (or a concurrent launch
// using the slots) costs at most that.
constexpr int PACE_EVERY = 32, PACE_SLOTS = 128;
constexpr int PACER_WARP = 2 + EPI_WARPS, THREADS2 = THREADS + 32;
constexpr unsigned long long PACE_WAIT_NS = 50000, PACE_STALE_NS = 2000000000ull;
constexpr uint32_t PACE_DONE = 0xFFFFFFFFu;
// 64 and 128 k-steps ran equally well on quad-double 4096^3 and 8192^3
// (8192^3: 289 ms per GEMM paced, 326 ms unpaced); 32 holds too often
constexpr int kDefaultPace = 64;
// one slot per 128-byte line, so that the clusters' stores and the pacers'
// polling spread over L2 slices instead of contending for a few lines
constexpr int PACE_STRIDE = 16;
constexpr unsigned PACE_POLL_NS = 2000;
__device__ unsigned long long g_pace[PACE_SLOTS * PACE_STRIDE];

__device__ __forceinline__ void pace_publish(int slot, uint32_t epoch, uint32_t steps) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(g_pace + slot * PACE_STRIDE),
               "l"(((unsigned long long)epoch << 32) | steps)
               : "memory");
}

// Published progress of a cluster in this launch (0 before it publishes).
__device__ __forceinline__ uint32_t pace_load(int slot, int ncl, uint32_t epoch) {
  if (slot >= ncl) return PACE_DONE;
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];"
               : "=l"(v)
               : "l"(g_pace + slot * PACE_STRIDE)
               : "memory");
  return (uint32_t)(v >> 32) == epoch ? (uint32_t)v : 0u;
}

// One unit of work of the pair kernel over digit planes: a 256 x 256 tile
// of one problem (rows row0.., columns col0..) and the runs it computes.
// ktail: as in TileJob.
struct PairJob {
  const CUtensorMap *tmA, *tmB, *tmC;
  int Mp, Np, KB, row0, col0, stack, ktail;
  DigitRuns runs;
};

// One unit of work over digit and sum planes (cross_sums.cuh): a tile and
// `planes` consecutive products of its list, which is the squares [sq, nsq),
// then the sums of the diagonals from d on, chunk by chunk.  The same plane
// index on both sides; flush groups never span two planes, because their
// exactness rests on the norms of windows of single sum planes.
struct CrossRuns {
  int sq, nsq, d, i, chunk, planes;  // where the list goes on, planes left
  int plane0, ppc, KB;               // plane of diagonal d's pair 0 is plane0 + cross_offset(d)
  int cuts1, cuts;                   // flush groups per square, per sum
  __host__ __device__ bool next(Run &r) {
    if (planes <= 0) return false;
    if (sq < nsq) {
      r = Run{sq, 1, sq, 1, 0, KB, sq, cuts1};
      ++sq;
      --planes;
    } else {
      const int left = mdgi::cross_pairs(d) - i;
      const int np = left < ppc ? left : ppc;
      const int t = plane0 + mdgi::cross_offset(d) + i;
      r = Run{t, 1, t, 1, 0, np * KB, chunk, cuts};
      ++chunk;
      planes -= np;
      i += np;
      if (np == left) {
        ++d;
        i = 0;
      }
    }
    return true;
  }
  struct Groups {
    int left, KB, cuts, j, at;
    __device__ Groups(const Run &r, int KB_) : left(r.steps), KB(KB_), cuts(r.cuts), j(0), at(0) {}
    __device__ int next() {
      if (left == 0) return 0;
      const int to = ++j * KB / cuts, n = to - at;
      at = to;
      if (j == cuts) j = at = 0;
      left -= n;
      return n;
    }
    __device__ bool last() const { return left == 0; }
  };
};

// Part `part` of a tile's list over the squares (nsq of them) and the diagonals
// [dlo, dhi): the runs that start in the part's 1/parts of its products.
__host__ __device__ __forceinline__ CrossRuns cross_part(int D, int dlo, int dhi, int nsq,
                                                         int plane0, int ppc, int KB, int cuts,
                                                         int part, int parts) {
  const int total = nsq + mdgi::cross_offset(dhi) - mdgi::cross_offset(dlo);
  const int lo = (int)((long long)total * part / parts);
  const int hi = (int)((long long)total * (part + 1) / parts);
  CrossRuns it{0, nsq, dlo, 0, D, total, plane0, ppc, KB, mdgi::cross_groups(KB), cuts};
  for (int d = 1; d < dlo; ++d) it.chunk += mdgi::cross_chunks(d, ppc);
  Run r;
  while (total - it.planes < lo && it.next(r)) {
  }
  CrossRuns first = it;
  while (total - it.planes < hi && it.next(r)) {
  }
  first.planes -= it.planes;
  return first;
}

struct CrossJob {
  static constexpr int stack = kStackNone, ktail = TK / 16;
  const CUtensorMap *tmA, *tmB, *tmC;
  int Mp, Np, KB, row0, col0;
  CrossRuns runs;
};

// The units of one problem as the host deals them (deal_single): cluster w takes
// order[starts[w]] .. order[starts[w + 1] - 1].  Travels as a kernel argument.
constexpr int kDealtUnits = 1024, kDealtWorkers = 80;
struct UnitDeal {
  unsigned short starts[kDealtWorkers + 1], order[kDealtUnits];
};

// Units of a single problem: as dealt, or (null) in turn.
struct MaybeDealt {
  const UnitDeal *deal;
  __device__ int first(int worker, int) const { return deal ? deal->starts[worker] : worker; }
  __device__ int end(int worker, int units) const { return deal ? deal->starts[worker + 1] : units; }
  __device__ int step(int workers) const { return deal ? 1 : workers; }
  __device__ int unit(int i) const { return deal ? deal->order[i] : i; }
};

// A single problem: units are tiles, or parts of tiles (ranges of
// diagonals whose digit-pair counts add up to about 1/parts of the tile's
// work), taken in strips of `raster` column blocks: tiles run across a strip
// of `raster` column blocks, then down the rows, so that the clusters busy at
// the same time read few distinct A row blocks and B column blocks and share
// them in L2 (raster = 1 walks each column block top to bottom).
struct PairSingle : MaybeDealt {
  const CUtensorMap *tmA, *tmB, *tmC;
  int s, D, Mp, Np, KB, cs, stack, ktail, mt, nt;
  int parts, raster;
  __device__ int last(int worker) const { return end(worker, mt * nt * parts); }
  __device__ PairJob job(int u) const {
    const int tiles = mt * nt, tile = u % tiles, part = u / tiles;
    const int strip = tile / (mt * raster);
    const int idx = tile - strip * mt * raster;
    const int c0 = strip * raster;
    const int g = nt - c0 < raster ? nt - c0 : raster;
    const int rb = idx / g, cb = c0 + idx - rb * g;
    return PairJob{tmA, tmB, tmC, Mp, Np, KB, rb * (stack == kStackM ? 128 : 256),
                   cb * (stack == kStackN ? 128 : 256), stack, ktail,
                   part_runs(s, D, KB, cs, stack, part, parts)};
  }
};

// Many problems (GroupedProblem table in global memory, tensor maps with
// 128-row boxes for A and B, Mp a multiple of 256): units are 256 x 256
// tiles times diagonal ranges, numbered as for the single-CTA kernel.
struct PairGrouped : DealtByHost {
  const mdgi::GroupedProblem *probs;
  int count;
  __device__ PairJob job(int u) const {
    const mdgi::GroupedProblem &g = grouped_find(probs, count, u);
    const int lt = u - g.unit_begin, tiles = g.mt * g.nt;
    const int tile = lt % tiles, part = lt / tiles;
    return PairJob{reinterpret_cast<const CUtensorMap *>(g.tmA),
                   reinterpret_cast<const CUtensorMap *>(g.tmB),
                   reinterpret_cast<const CUtensorMap *>(g.tmC), g.Mp, g.Np, g.KB,
                   (tile % g.mt) * (g.stack == kStackM ? 128 : 256),
                   (tile / g.mt) * (g.stack == kStackN ? 128 : 256), g.stack, g.ktail,
                   part_runs(g.s, g.D, g.KB, mdgi::CHUNK_STEPS, g.stack, part, g.parts)};
  }
};

// A single problem over digit and sum planes: units are tiles, or parts of
// tiles whose lists hold about 1/parts of its products each (cut between
// output planes), in the order of PairSingle's.
struct PairCross : MaybeDealt {
  const CUtensorMap *tmA, *tmB, *tmC;
  int D, dlo, dhi, nsq, plane0, ppc, Mp, Np, KB;
  int parts, raster;
  const unsigned *norm_a, *norm_b;
  __device__ int last(int worker) const {
    return end(worker, (Mp / 256) * (Np / TN2) * parts);
  }
  // Flush groups per sum plane.  |sum over a group| <= |a| |b| (Cauchy and
  // Schwarz; every partial sum too) with |a|^2 <= 2 *norm_a, |b|^2 <= 2
  // *norm_b over a whole group (two windows), <= *norm_a, *norm_b over half
  // of one; a quarter holds at most 256 products of 2^16.  FP32 is exact up
  // to 2^24, so whole groups where 4 *norm_a *norm_b <= 2^48.  (Rows of non-finite
  // entries can have any norm; n2 cannot wrap, 4 n2 could.)
  __device__ int cuts() const {
    const unsigned long long n2 = (unsigned long long)*norm_a * *norm_b;
    return mdgi::cross_groups(KB) * (n2 <= 1ull << 46 ? 1 : n2 <= 1ull << 48 ? 2 : 4);
  }
  __device__ CrossJob job(int u) const {
    const int MB = Mp / 256, NB = Np / TN2, tiles = MB * NB;
    const int tile = u % tiles, part = u / tiles;
    const int strip = tile / (MB * raster);
    const int idx = tile - strip * MB * raster;
    const int c0 = strip * raster;
    const int g = NB - c0 < raster ? NB - c0 : raster;
    const int rb = idx / g, cb = c0 + idx - rb * g;
    return CrossJob{tmA, tmB, tmC, Mp, Np, KB, rb * 256, cb * TN2,
                    cross_part(D, dlo, dhi, nsq, plane0, ppc, KB, cuts(), part, parts)};
  }
};

template <class Jobs>
__device__ __forceinline__ void tc2_body(const Jobs &jobs, int pace, uint32_t epoch,
                                         int no_loads) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = reinterpret_cast<uint8_t *>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t *bars =
      reinterpret_cast<uint64_t *>(smem + STAGES2 * STAGE2_BYTES + EPI_WARPS * OUT_BYTES);
  // bars: STAGES2 full, STAGES2 empty, 2 accfull, 2 accempty, 1 drain, then
  // the TMEM address and the abort flag
  static_assert(2 * STAGES2 + 9 <= 32, "barrier area holds 32 words of 8 bytes");
  uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bars + 2 * STAGES2 + 5);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars + 2 * STAGES2 + 6);
  // pacing: k-steps issued by the producer (every PACE_EVERY), k-steps it
  // may issue (posted by the pacer warp)
  volatile uint32_t *pace_steps = reinterpret_cast<volatile uint32_t *>(bars + 2 * STAGES2 + 7);
  volatile uint32_t *pace_allowed = reinterpret_cast<volatile uint32_t *>(bars + 2 * STAGES2 + 8);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_rank();
  const bool leader = rank == 0;
  const uint32_t smem_base = smem_u32(smem);
  auto full = [&](int st) { return smem_u32(bars + st); };
  auto empty = [&](int st) { return smem_u32(bars + STAGES2 + st); };
  auto accfull = [&](int b) { return smem_u32(bars + 2 * STAGES2 + b); };
  auto accempty = [&](int b) { return smem_u32(bars + 2 * STAGES2 + 2 + b); };
  const uint32_t drain_bar = smem_u32(bars + 2 * STAGES2 + 4);

  if (threadIdx.x == 0) {
    for (int st = 0; st < STAGES2; ++st) {
      mbar_init(full(st), 1);
      mbar_init(empty(st), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(accfull(b), 1);
      mbar_init(accempty(b), 2 * EPI_WARPS);
    }
    mbar_init(drain_bar, 1);
    *abort_flag = 0;
    *pace_steps = 0;
    *pace_allowed = PACE_DONE;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_holder)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  fence_before();
  cluster_sync();
  fence_after();
  const uint32_t tmem_base = *tmem_holder;

  const int cid = blockIdx.x >> 1, ncl = gridDim.x >> 1;
  const int first = jobs.first(cid, ncl), last = jobs.last(cid), step = jobs.step(ncl);
  const bool pacer = leader && pace > 0 && ncl <= PACE_SLOTS;
  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------------------------------ producer --
      int st = 0;
      uint32_t ph = 0;
      // per stage: a copy was issued (bit of `issued`), parity of its phase
      // (bit of `last_par`); bit masks so that they stay in registers
      uint32_t issued = 0, last_par = 0;
      bool pacing = pacer;
      uint32_t steps = 0;  // k-steps issued by this cluster
      // no_loads (self-test of the bounded waits): issue no copy, so the
      // MMA thread's wait for data runs out, it raises the abort flag and
      // every role leaves with nothing in flight
      for (int n = no_loads ? last : first; n < last; n += step) {
        auto jb = jobs.job(jobs.unit(n));
        const int KB = jb.KB;
        // the odd CTA: the next 128 rows and columns, or the next plane
        const int next_a = jb.stack == kStackM ? (int)rank : 0;
        const int next_b = jb.stack == kStackN ? (int)rank : 0;
        const int row = jb.row0 + ((int)rank - next_a) * TM;
        const int col = jb.col0 + ((int)rank - next_b) * BH;
        Run r;
        while (jb.runs.next(r)) {
          for (int t = r.t0; t < r.t0 + r.steps; ++t) {
            const int q = t / KB, kb = t - q * KB;
            const int i = r.a0 + r.astep * q + next_a, j = r.b0 + r.bstep * q + next_b;
            if (pacing && steps > *pace_allowed) {
              const unsigned long long t0 = now_ns();
              while (steps > *pace_allowed) {
                if (*abort_flag) break;
                if (now_ns() - t0 > PACE_WAIT_NS) {
                  pacing = false;
                  break;
                }
              }
            }
            if (!mbar_wait(empty(st), ph ^ 1, abort_flag)) goto producer_done;
            if (leader) mbar_expect_tx(full(st), 2 * STAGE2_BYTES);
            const uint32_t a_dst = smem_base + st * STAGE2_BYTES;
            const uint32_t bar0 = map_to_rank0(full(st));
            tma_load_2d_pair(a_dst, jb.tmA, kb * TK, i * jb.Mp + row, bar0);
            tma_load_2d_pair(a_dst + A2_BYTES, jb.tmB, kb * TK, j * jb.Np + col, bar0);
            last_par = (last_par & ~(1u << st)) | (ph << st);
            issued |= 1u << st;
            if (++st == STAGES2) {
              st = 0;
              ph ^= 1;
            }
            if ((++steps & (PACE_EVERY - 1)) == 0) *pace_steps = steps;
          }
        }
      }
    producer_done:
      *pace_steps = PACE_DONE;
      if (*abort_flag && leader)
        for (int i = 0; i < STAGES2; ++i)
          if ((issued >> i) & 1u) mbar_drain(full(i), (last_par >> i) & 1u);
    }
  } else if (warp == 1) {
    if (lane == 0 && leader) {
      // ---------------------------------------------------- MMA issuer --
      int st = 0, buf = 0;
      uint32_t ph = 0, aph[2] = {0, 0};
      bool any = false;
      for (int n = first; n < last; n += step) {
        auto jb = jobs.job(jobs.unit(n));
        Run r;
        while (jb.runs.next(r)) {
          int kb = r.t0 % jb.KB;
          typename decltype(jb.runs)::Groups groups(r, jb.KB);
          for (int steps; (steps = groups.next()) > 0;) {
            if (!mbar_wait(accempty(buf), aph[buf] ^ 1, abort_flag)) goto mma_done;
            fence_after();
            const uint32_t dt = tmem_base + buf * TN2;
            for (int t = 0; t < steps; ++t) {
              if (!mbar_wait(full(st), ph, abort_flag)) goto mma_done;
              fence_after();
              const uint32_t a_addr = smem_base + st * STAGE2_BYTES;
              const uint64_t da = sw128_desc(a_addr), db = sw128_desc(a_addr + A2_BYTES);
              // the last k-block of a plane: only the MMAs that reach data
              const bool short_block = kb == jb.KB - 1 && jb.ktail < TK / 16;
              if (++kb == jb.KB) kb = 0;
              if (!short_block) {
#pragma unroll
                for (int kk = 0; kk < TK / 16; ++kk)
                  mma_bf16_pair(dt, da + 2 * kk, db + 2 * kk, (t > 0 || kk > 0) ? 1u : 0u);
              } else {
                for (int kk = 0; kk < jb.ktail; ++kk)
                  mma_bf16_pair(dt, da + 2 * kk, db + 2 * kk, (t > 0 || kk > 0) ? 1u : 0u);
              }
              mma_commit_pair(empty(st));
              any = true;
              if (++st == STAGES2) {
                st = 0;
                ph ^= 1;
              }
            }
            mma_commit_pair(accfull(buf));
            aph[buf] ^= 1;
            buf ^= 1;
          }
        }
      }
    mma_done:
      if (*abort_flag && any) {
        mma_commit_pair(drain_bar);
        mbar_drain(drain_bar, 0);
      }
    }
  } else if (warp == PACER_WARP) {
    if (pacer) {
      // --------------------------------------------------------- pacer --
      // publishes the producer's progress and posts the number of k-steps
      // it may issue (slowest running cluster + pace) until the producer
      // is done; bounded by PACE_STALE_NS without news from the producer
      uint32_t last = 0;
      unsigned long long t_last = now_ns();
      while (true) {
        const uint32_t mine = __shfl_sync(0xffffffffu, *pace_steps, 0);
        if (mine != last) {
          last = mine;
          t_last = now_ns();
        }
        if (lane == 0) pace_publish(cid, epoch, mine);
        if (mine == PACE_DONE) break;
        uint32_t m = PACE_DONE;
#pragma unroll
        for (int k = 0; k < PACE_SLOTS / 32; ++k) m = min(m, pace_load(lane + 32 * k, ncl, epoch));
        m = __reduce_min_sync(0xffffffffu, m);
        if (lane == 0)
          *pace_allowed = m == PACE_DONE || m > PACE_DONE - (uint32_t)pace ? PACE_DONE
                                                                           : m + (uint32_t)pace;
        int stop = 0;
        if (lane == 0) stop = (*abort_flag || now_ns() - t_last > PACE_STALE_NS) ? 1 : 0;
        if (__shfl_sync(0xffffffffu, stop, 0)) break;
        __nanosleep(PACE_POLL_NS);
      }
      if (lane == 0) {
        *pace_allowed = PACE_DONE;
        pace_publish(cid, epoch, PACE_DONE);
      }
    }
  } else {
    // -------------------------------------------------------- epilogue --
    const int q = warp & 3, h = (warp - 2) >> 2;
    const uint32_t staging = smem_base + STAGES2 * STAGE2_BYTES + (warp - 2) * OUT_BYTES;
    int acc[128];
#pragma unroll
    for (int j = 0; j < 128; ++j) acc[j] = 0;
    int buf = 0;
    uint32_t aph[2] = {0, 0};
    const uint32_t accempty0[2] = {map_to_rank0(accempty(0)), map_to_rank0(accempty(1))};
    for (int n = first; n < last; n += step) {
      auto jb = jobs.job(jobs.unit(n));
      const int next = jb.stack == kStackM ? (int)rank : jb.stack == kStackN ? h : 0;
      const int row = jb.row0 + (jb.stack == kStackM ? 0 : (int)rank * TM) + 32 * q;
      const int col = jb.col0 + (jb.stack == kStackN ? 0 : 128 * h);
      Run r;
      while (jb.runs.next(r)) {
        typename decltype(jb.runs)::Groups groups(r, jb.KB);
        while (groups.next() > 0) {
          int ok = 1;
          if (lane == 0) ok = mbar_wait(accfull(buf), aph[buf], abort_flag) ? 1 : 0;
          ok = __shfl_sync(0xffffffffu, ok, 0);
          if (!ok) goto epi_done;
          aph[buf] ^= 1;
          fence_after();
          const uint32_t taddr = tmem_base + ((uint32_t)(32 * q) << 16) + buf * TN2 + 128 * h;
          drain128(taddr, acc);
          fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(accempty0[buf]);
          buf ^= 1;
          // (a diagonal -1 is all zeros)
          if (groups.last() && r.chunk + next >= 0)
            store_rows(staging, lane, acc, jb.tmC, col, (r.chunk + next) * jb.Mp + row);
        }
      }
    }
  epi_done:
    if (lane == 0) stores_done();
  }
  __syncwarp();
  fence_before();
  cluster_sync();
  fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(TMEM_COLS)
                 : "memory");
  if (threadIdx.x == 0 && *abort_flag) atomicExch(&g_tc_error, 1);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS2, 1)
    diag_gemm_tc2_kernel(const __grid_constant__ CUtensorMap tmA,
                         const __grid_constant__ CUtensorMap tmB,
                         const __grid_constant__ CUtensorMap tmC, int s, int D, int Mp, int Np,
                         int KB, int cs, int stack, int ktail, int mt, int nt, int parts,
                         int raster, int pace, uint32_t epoch, int no_loads, int dealt,
                         const __grid_constant__ UnitDeal deal) {
  tc2_body(PairSingle{{dealt ? &deal : nullptr}, &tmA, &tmB, &tmC, s, D, Mp, Np, KB, cs, stack, ktail, mt, nt, parts, raster},
           pace, epoch, no_loads);
}

// The diagonal GEMM over digit and sum planes (cross_sums.cuh).  Bound by the
// tensor cores as the kernel above, at 224 instead of 406 products of planes
// for quad-double: qd 8192^3 146 instead of 268 ms (1684 TFLOP/s done), od
// 2048^3 8.5 instead of 16.4 ms, qd 1024^3 312 instead of 607 us.  Flush
// groups of 16, 8 and 4 k-steps (whole, halves, quarters) cost 17.0, 17.9
// and 27.7 ms on the same quad-double 4096 x 4096 x 2048 digit pairs: reading
// the accumulators back takes about 4000 cycles, 4 k-steps of products 2048.
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS2, 1)
    diag_gemm_cross_kernel(const __grid_constant__ CUtensorMap tmA,
                           const __grid_constant__ CUtensorMap tmB,
                           const __grid_constant__ CUtensorMap tmC, int D, int dlo, int dhi,
                           int nsq, int plane0, int ppc, int Mp, int Np, int KB, int parts,
                           int raster, const unsigned *__restrict__ norm_a,
                           const unsigned *__restrict__ norm_b, int pace, uint32_t epoch,
                           int no_loads, int dealt, const __grid_constant__ UnitDeal deal) {
  tc2_body(PairCross{{dealt ? &deal : nullptr}, &tmA, &tmB, &tmC, D, dlo, dhi, nsq, plane0, ppc, Mp, Np, KB, parts, raster,
                     norm_a, norm_b},
           pace, epoch, no_loads);
}

// The batched plan's grouped GEMM on CTA pairs (no pacing: the clusters work
// on different problems).
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(THREADS2, 1)
    diag_gemm_tc2_grouped_kernel(const mdgi::GroupedProblem *__restrict__ probs, int count,
                                 const int *__restrict__ starts, const int *__restrict__ order) {
  tc2_body(PairGrouped{{starts, order}, probs, count}, 0, 0, 0);
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  // looked up once per process; the initialisation of a function-local
  // static is serialised between threads
  static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    return static_cast<PFN_cuTensorMapEncodeTiled_v12000>(nullptr);
  }();
  return fn;
}

// 2-D map over `planes` planes of rows x Kp BF16 (row stride Kp), box
// 64 x box_rows, 128-byte swizzle.
int make_map(CUtensorMap *m, const void *base, int Kp, long long rows_total, int box_rows) {
  auto fn = encode_fn();
  if (!fn) return MDG_ERROR_NOT_SUPPORTED;
  cuuint64_t dims[2] = {(cuuint64_t)Kp, (cuuint64_t)rows_total};
  cuuint64_t strides[1] = {(cuuint64_t)Kp * 2};
  cuuint32_t box[2] = {(cuuint32_t)TK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? MDG_SUCCESS : MDG_ERROR_NOT_SUPPORTED;
}

// 2-D map over `planes` int32 output planes of rows x Np, box 32 x 32,
// 128-byte swizzle (store_rows).
int make_out_map(CUtensorMap *m, const void *base, int Np, long long rows_total) {
  auto fn = encode_fn();
  if (!fn) return MDG_ERROR_NOT_SUPPORTED;
  cuuint64_t dims[2] = {(cuuint64_t)Np, (cuuint64_t)rows_total};
  cuuint64_t strides[1] = {(cuuint64_t)Np * 4};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<void *>(base), dims, strides, box,
                  estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? MDG_SUCCESS : MDG_ERROR_NOT_SUPPORTED;
}

// How one launch of a pair kernel runs: work units, tile order, pacing.
// as_asked: the parts or a pacing window are the caller's (or MDG_TC_PACE's), so
// the units are taken in turn.
struct PairSchedule {
  int clusters, parts, raster, pace, no_loads;
  bool as_asked;
  uint32_t epoch;
};

// Parts of a problem whose tiles do not fill the workers: a run each where
// they all fit, else as many as fit (at least `parts`).
int few_tile_parts(int tiles, int runs, int workers, int parts) {
  const int fit = workers / tiles;
  return runs <= fit ? runs : std::max(parts, fit);
}

// Dealing of units of work to workers (clusters or CTAs) by cost.
struct Unit {
  long long cost;
  int id;
};

// The costs in k-steps of the `parts` parts that `all` is cut into: a part's own
// steps, about 6 per run for the drain and the store, about 10 to fill and empty
// the pipeline.  A run of size(run) belongs to the part whose 1/parts of `total`
// it starts in, as part_runs and cross_part cut; all in one walk, since a walk a
// part cost the host more than the rest of a call (hd 256^3 147 us a call).
// runs: how many each part has.
template <class Runs, class Size>
std::vector<long long> part_costs(Runs all, long long total, int parts, const Size &size,
                                  std::vector<int> *runs = nullptr) {
  std::vector<long long> cost(parts, 10);
  if (runs) runs->assign(parts, 0);
  long long at = 0;
  for (Run r; all.next(r); at += size(r)) {
    const int part = (int)(((at + 1) * parts - 1) / total);
    cost[part] += r.steps + 6;
    if (runs) ++(*runs)[part];
  }
  return cost;
}

// The same over digit planes (part_runs).
std::vector<long long> digit_part_costs(int s, int D, int KB, int cs, int stack, int parts) {
  const DigitRuns all = part_runs(s, D, KB, cs, stack, 0, 1);
  long long steps = 0, runs = 0;
  DigitRuns it = all;
  for (Run r; it.next(r); ++runs) steps += r.steps;
  if (parts == runs) return part_costs(all, runs, parts, [](const Run &) { return 1; });
  return part_costs(all, steps, parts, [](const Run &r) { return r.steps; });
}

// Each unit, in the order given, to the worker with the least so far; the
// largest sum.
long long deal_in_order(const std::vector<Unit> &units, int workers, std::vector<int> *starts,
                        std::vector<int> *order) {
  typedef std::pair<long long, int> Load;
  std::priority_queue<Load, std::vector<Load>, std::greater<Load>> least;
  for (int w = 0; w < workers; ++w) least.push(Load(0, w));
  std::vector<int> of(units.size());  // the unit's worker
  starts->assign(workers + 1, 0);
  long long most = 0;
  for (size_t i = 0; i < units.size(); ++i) {
    const Load l = least.top();
    least.pop();
    of[i] = l.second;
    ++(*starts)[l.second + 1];
    least.push(Load(l.first + units[i].cost, l.second));
    most = std::max(most, l.first + units[i].cost);
  }
  for (int w = 0; w < workers; ++w) (*starts)[w + 1] += (*starts)[w];
  std::vector<int> next(starts->begin(), starts->end() - 1);
  order->resize(units.size());
  for (size_t i = 0; i < units.size(); ++i) (*order)[next[of[i]]++] = units[i].id;
  return most;
}

// The units (tile, part) of a single problem, the dearest first, dealt, where
// that ends sooner than sc's parts taken in turn.  Clusters at work then have
// units of about equal length and few planes between them, so no pacing.
// us a call over digit pairs, in turn / a tile's runs in a row / the longest
// runs first: dd 16001 x 96 x 3001 1666 / 1584 / 1600, od 3000 x 64 x 1000 1106
// / 1100 / 991, dd 4000 x 64 x 300 102 / 102 / 89, qd 2000 x 300 x 450 316 / 317
// / 282, dd 3000 x 1000 x 500 375 / 376 / 344, qd 700 x 300 x 200 125 / 116 / 96.
// Over sum planes, in turn / 24 / 32 / 48 / 64 parts dealt: qd 1024^3 658 / 637 /
// 627 / 624 / 625 (64 of 76 clusters at work / all), 1000 x 777 x 1531 884 / 844
// / 843 / 831 / 833, od 1024^3 2060 / 1990 / 2000 / 1960 / 1954, hd 1024 x 1024 x
// 512 4584 / 4520 / 4368 / 4448 / 4480, qd 2048^3 (16 parts) 3620 / 3400.  But a
// product of more than about 3 ms runs at the power cap, where the idle clusters'
// share of the power drives the others, and the worse sharing of planes costs:
// od 2048^3 12.3 / 12.7 ms, qd 3000 x 2500 x 3000 8.95 / 9.2, od 1500^3 5.5 / 5.7,
// hd 2048 x 2048 x 512 14.37 / 14.39: in turn beyond kCrossDealSteps k-steps a
// cluster (qd 2048^3 6036, od 1500^3 9219).
constexpr int kCrossDealParts = 48;
constexpr long long kCrossDealSteps = 7000;

// costs(parts): of a tile's parts, 0 for one that has no runs; fine: the parts to
// deal.
template <class Costs>
bool deal_single(int tiles, int fine, const Costs &costs, int ncl, PairSchedule *sc,
                 UnitDeal *deal) {
  const long long all_units = (long long)tiles * fine;
  if (ncl > kDealtWorkers || all_units > kDealtUnits) return false;
  if (sc->parts == fine && all_units <= ncl) return false;  // a unit each already
  std::vector<long long> in_turn(ncl, 0);
  const std::vector<long long> coarse = costs(sc->parts), cost = costs(fine);
  for (int part = 0; part < sc->parts; ++part)
    for (int t = 0; t < tiles; ++t) in_turn[(part * tiles + t) % ncl] += coarse[part];
  std::vector<int> parts;
  for (int part = 0; part < fine; ++part)
    if (cost[part]) parts.push_back(part);
  std::stable_sort(parts.begin(), parts.end(), [&](int a, int b) { return cost[a] > cost[b]; });
  std::vector<Unit> units;
  units.reserve(parts.size() * tiles);
  for (int part : parts)
    for (int t = 0; t < tiles; ++t) units.push_back(Unit{cost[part], part * tiles + t});
  std::vector<int> starts, order;
  if (deal_in_order(units, ncl, &starts, &order) >=
      *std::max_element(in_turn.begin(), in_turn.end()))
    return false;
  std::copy(starts.begin(), starts.end(), deal->starts);
  std::copy(order.begin(), order.end(), deal->order);
  sc->parts = fine;
  sc->clusters = (int)std::min<long long>(ncl, (long long)units.size());
  sc->pace = 0;
  return true;
}

// runs: of a tile, what parts can separate.
PairSchedule pair_schedule(int mt, int nt, int runs, int sms, int parts_opt, int raster_opt,
                           int pace_opt) {
  PairSchedule sc;
  const int tiles = mt * nt;
  // split tiles into `parts` diagonal ranges when that shrinks the idle
  // part of the last wave of clusters by more than it costs: each extra
  // part makes the work about 4 % slower (fitted to quad-double 4096^3 and
  // 8192^3: 1024 tiles on 76 clusters run best unsplit, 256 tiles best in
  // two parts)
  const int ncl = sms / 2;
  sc.parts = 1;
  double best = 0.0;
  for (int u = 1; u <= 8 && u <= runs; ++u) {
    const long long units = (long long)tiles * u;
    const long long waves = (units + ncl - 1) / ncl;
    const double cost = (double)waves / u * (1.0 + 0.04 * (u - 1));
    if (u == 1 || cost < best) {
      best = cost;
      sc.parts = u;
    }
  }
  if ((long long)tiles * sc.parts <= ncl) sc.parts = few_tile_parts(tiles, runs, ncl, sc.parts);
  if (parts_opt > 0) sc.parts = std::min(8, parts_opt);
  // tile order: strips about sqrt(clusters) column blocks wide, so that
  // the tiles in work at one time span few row and column blocks (the
  // largest power of two not above sqrt(76) = 8.7 on 152 SMs)
  sc.raster = 1;
  while ((sc.raster * 2) * (sc.raster * 2) <= ncl) sc.raster *= 2;
  if (raster_opt > 0) sc.raster = raster_opt;
  sc.raster = std::min(nt, sc.raster);
  const long long units = (long long)tiles * sc.parts;
  sc.clusters = units < ncl ? (int)units : ncl;
  // pacing window in k-steps, 0 = off (MDG_TC_PACE overrides); every
  // launch gets its own epoch so that slots left by earlier launches read
  // as "not started"
  // With no more units than clusters every tile is in work at once and
  // the operands of the whole GEMM are read in one sweep: pacing has no
  // drift to correct there and only costs (qd 1024^3: 7 % slower paced), so
  // the default turns it off; an explicit window still applies.
  sc.pace = units <= ncl ? 0 : kDefaultPace;
  const char *e = std::getenv("MDG_TC_PACE");
  if (pace_opt == 0 && e) pace_opt = std::atoi(e) > 0 ? std::atoi(e) : -1;
  if (pace_opt > 0) sc.pace = pace_opt;
  if (pace_opt < 0) sc.pace = 0;
  sc.as_asked = parts_opt > 0 || pace_opt > 0;
  static std::atomic<uint32_t> epochs{0};
  sc.epoch = ++epochs;
  if (sc.epoch == 0) sc.epoch = ++epochs;
  // MDG_TC_SELFTEST_NO_LOADS=1: the producers issue no copies, the waits
  // for data run out after their 2 s limit and mdg_device_status then
  // reports MDG_ERROR_TIMEOUT (a test of the failure path; the result
  // planes are not written)
  const char *nl = std::getenv("MDG_TC_SELFTEST_NO_LOADS");
  sc.no_loads = (nl && *nl == '1') ? 1 : 0;
  return sc;
}

}  // namespace

namespace mdgi {

int launch_diag_gemm_cross(int s, int D, int dlo, int dhi, int squares, int sum_planes, int Mp,
                           int Np, int Kp, const void *dA, const void *dB, const unsigned *norm_a,
                           const unsigned *norm_b, int *out, int parts, int raster, int pace, cudaStream_t st) {
  if (Mp % 256 || Np % TN2 || Kp % TK) return MDG_ERROR_INVALID_SIZE;
  const int KB = Kp / TK;
  if (KB < 1 || KB > CROSS_CHUNK_STEPS) return MDG_ERROR_INVALID_SIZE;
  CUtensorMap ma, mb, mc;
  MDG_TRY(make_map(&ma, dA, Kp, (long long)(s + sum_planes) * Mp, TM));
  MDG_TRY(make_map(&mb, dB, Kp, (long long)(s + sum_planes) * Np, BH));
  MDG_TRY(make_out_map(&mc, out, Np, (long long)cross_outputs(D, KB) * Mp));
  int dev = 0, sms = 0;
  MDG_TRY_CUDA(cudaGetDevice(&dev));
  MDG_TRY_CUDA(cudaFuncSetAttribute(diag_gemm_cross_kernel,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM2_BYTES));
  MDG_TRY_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int tiles = (Mp / 256) * (Np / TN2), plane0 = s - cross_offset(dlo);
  const int ppc = cross_pairs_per_chunk(KB);
  PairSchedule sc = pair_schedule(Mp / 256, Np / TN2, squares + dhi - dlo, sms, parts, raster, pace);
  UnitDeal deal = {};
  bool dealt = false;
  const int products = squares + cross_offset(dhi) - cross_offset(dlo);
  if (!sc.as_asked &&
      (long long)tiles * products * KB <= kCrossDealSteps * (sms / 2)) {
    auto costs = [&](int of) {
      std::vector<int> runs;
      std::vector<long long> cost = part_costs(
          cross_part(D, dlo, dhi, squares, plane0, ppc, KB, cross_groups(KB), 0, 1), products, of,
          [KB](const Run &r) { return r.steps / KB; }, &runs);
      for (int part = 0; part < of; ++part)
        if (!runs[part]) cost[part] = 0;
      return cost;
    };
    const int fine = std::min(products, std::min(kCrossDealParts, kDealtUnits / tiles));
    dealt = fine > 0 && deal_single(tiles, fine, costs, sms / 2, &sc, &deal);
  }
  diag_gemm_cross_kernel<<<2 * sc.clusters, THREADS2, SMEM2_BYTES, st>>>(
      ma, mb, mc, D, dlo, dhi, squares, plane0, ppc, Mp, Np, KB, sc.parts, sc.raster, norm_a, norm_b,
      sc.pace, sc.epoch, sc.no_loads, dealt, deal);
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

int stacked_tiles(int s, int D, int m, int n, int KB) {
  if (D > s || (long long)(D + 1) * KB > CHUNK_STEPS) return kStackNone;
  long long pairs = 0, stacked = 0;
  for (int d = 0; d < D; ++d) pairs += diag_pairs(d, s);
  for (int d = -(D & 1); d < D; d += 2) stacked += d + 2;
  const long long m256 = (m + 255) / 256, n256 = (n + 255) / 256;
  const long long work[3] = {m256 * n256 * pairs, m256 * ((n + 127) / 128) * stacked,
                             (m + 127) / 128 * n256 * stacked};
  return (int)(std::min_element(work, work + 3) - work);
}

int launch_diag_gemm_tc(int s, int D, int Mp, int Np, int Kp, int m, int n, int k, const void *dA,
                        const void *dB, int ld, long long plane_a, long long plane_b, int *chunks,
                        long long plane_c, int cs, int engine, int parts_opt, int raster_opt,
                        cudaStream_t st, int pace_opt) {
  if (Mp % TM || Np % TN || Kp % TK || ld != Kp || k <= Kp - TK || k > Kp) return MDG_ERROR_INVALID_SIZE;
  if (plane_a != (long long)Mp * Kp || plane_b != (long long)Np * Kp) return MDG_ERROR_INVALID_SIZE;
  if ((reinterpret_cast<uintptr_t>(dA) | reinterpret_cast<uintptr_t>(dB)) & 15)
    return MDG_ERROR_INVALID_SIZE;
  if (plane_c != (long long)Mp * Np) return MDG_ERROR_INVALID_SIZE;
  // the CTA-pair kernel needs 256-row tiles
  const AutoTiles own = engine == 1 ? auto_tiles(s, D, m, n, Kp / TK, cs) : AutoTiles{};
  const bool pair = Mp % 256 == 0 && engine != 2 && !own.narrow;
  const int tn = own.narrow ? own.narrow : TN;
  const int runs = total_chunks(s, D, Kp / TK, cs);
  CUtensorMap ma, mb, mc;
  MDG_TRY(make_out_map(&mc, chunks, Np, (long long)runs * Mp));
  MDG_TRY(make_map(&ma, dA, Kp, (long long)s * Mp, TM));
  MDG_TRY(make_map(&mb, dB, Kp, (long long)s * Np, pair ? BH : tn));
  int dev = 0, sms = 0;
  MDG_TRY_CUDA(cudaGetDevice(&dev));
  // per-device attribute, set on every launch (no process-wide record that
  // a second device or a second host thread could find stale)
  if (pair)
    MDG_TRY_CUDA(cudaFuncSetAttribute(diag_gemm_tc2_kernel,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM2_BYTES));
  else
    MDG_TRY_CUDA(cudaFuncSetAttribute(diag_gemm_tc_kernel,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  MDG_TRY_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  if (pair) {
    const int stack = own.stack;
    const int mt = stack == kStackM ? (m + 127) / 128 : Mp / 256;
    const int nt = stack == kStackN ? (n + 127) / 128 : Np / TN2;
    const int separable = stack ? (D + 1) / 2 : runs;
    PairSchedule sc = pair_schedule(mt, nt, separable, sms, parts_opt, raster_opt, pace_opt);
    UnitDeal deal = {};
    auto costs = [&](int parts) { return digit_part_costs(s, D, Kp / TK, cs, stack, parts); };
    const bool dealt = !sc.as_asked &&
                       deal_single(mt * nt, separable, costs, sms / 2, &sc, &deal);
    diag_gemm_tc2_kernel<<<2 * sc.clusters, THREADS2, SMEM2_BYTES, st>>>(
        ma, mb, mc, s, D, Mp, Np, Kp / TK, cs, stack, (k - (Kp - TK) + 15) / 16, mt, nt, sc.parts,
        sc.raster, sc.pace, sc.epoch, sc.no_loads, dealt, deal);
  } else {
    const int mt = (m + TM - 1) / TM, nt = (n + tn - 1) / tn, tiles = mt * nt;
    const int parts = parts_opt > 0 ? std::min(8, parts_opt)
                      : tiles <= sms ? few_tile_parts(tiles, runs, sms, 1)
                                     : 1;
    const int grid = (int)std::min<long long>((long long)tiles * parts, sms);
    diag_gemm_tc_kernel<<<grid, THREADS, SMEM_BYTES, st>>>(ma, mb, mc, s, D, Mp, Np, Kp / TK, cs,
                                                           tn, mt, nt, parts);
  }
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

int encode_plane_map(void *map128, const void *base, int Kp, long long rows_total, int box_rows) {
  return make_map(reinterpret_cast<CUtensorMap *>(map128), base, Kp, rows_total, box_rows);
}

int encode_out_map(void *map128, const void *base, int Np, long long rows_total) {
  return make_out_map(reinterpret_cast<CUtensorMap *>(map128), base, Np, rows_total);
}

// The units of a table (numbered as the kernels number them) over the
// workers, in the table's order, each to the worker with the least so far.  The
// table's order, dear
// problems first and a problem's units in a row, keeps the workers on few
// problems at a time.  ms a call, units in turn / dearest unit first / in the
// table's order: 64 mixed problems of 32 .. 512 2.67 / 2.30 / 2.12, 256 of
// them - / 9.5 / 8.6, their octo-double ones on 128 x 256 tiles - / 11.6 / 7.5.
int deal_units(const std::vector<GroupedProblem> &probs, int workers, std::vector<int> *starts,
               std::vector<int> *order) {
  std::vector<Unit> units;
  for (const GroupedProblem &g : probs) {
    const std::vector<long long> cost =
        digit_part_costs(g.s, g.D, g.KB, CHUNK_STEPS, g.stack, g.parts);
    for (int part = 0; part < g.parts; ++part)
      for (int tile = 0; tile < g.mt * g.nt; ++tile)
        units.push_back(Unit{cost[part] * (g.tn == 128 && !g.stack ? 2 : 4),
                             g.unit_begin + part * g.mt * g.nt + tile});
  }
  deal_in_order(units, workers, starts, order);
  return MDG_SUCCESS;
}

int launch_diag_gemm_grouped(const GroupedProblem *dev_probs, int count, int workers,
                             const int *dev_starts, const int *dev_order, int pair,
                             cudaStream_t st) {
  if (pair) {
    MDG_TRY_CUDA(cudaFuncSetAttribute(diag_gemm_tc2_grouped_kernel,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM2_BYTES));
    diag_gemm_tc2_grouped_kernel<<<2 * workers, THREADS2, SMEM2_BYTES, st>>>(
        dev_probs, count, dev_starts, dev_order);
  } else {
    MDG_TRY_CUDA(cudaFuncSetAttribute(diag_gemm_tc_grouped_kernel,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
    diag_gemm_tc_grouped_kernel<<<workers, THREADS, SMEM_BYTES, st>>>(dev_probs, count, dev_starts,
                                                                     dev_order);
  }
  MDG_TRY_LAUNCH();
  return MDG_SUCCESS;
}

int tc_device_status() {
  MDG_TRY_CUDA(cudaDeviceSynchronize());
  int flag = 0, zero = 0;
  MDG_TRY_CUDA(cudaMemcpyFromSymbol(&flag, g_tc_error, sizeof(int)));
  if (flag) {
    MDG_TRY_CUDA(cudaMemcpyToSymbol(g_tc_error, &zero, sizeof(int)));
    return MDG_ERROR_TIMEOUT;
  }
  return MDG_SUCCESS;
}

}  // namespace mdgi
