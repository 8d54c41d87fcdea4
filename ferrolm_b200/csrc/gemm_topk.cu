// Tensor-core front end of exact search (flat.rs:40-53 at batch scale).
//
//   scores(q, b) = ||b||^2 - 2 <q, b>      (L2; the per-query constant ||q||^2 is left out)
//                = -<q, b>                 (inner product)
//
// computed as a 16-bit-input, fp32-accumulate GEMM on the 5th-generation tensor cores:
// tcgen05.mma issued by one thread, operands staged in shared memory by TMA with the 128-byte
// swizzle, accumulators in tensor memory.  The accumulator IS the score: the query operand is
// stored pre-multiplied by -2 (or -1), and for L2 one extra k step of 16 adds ||b||^2, split
// into three 16-bit pieces, inside the MMA.  The epilogue reads the accumulators back with
// tcgen05.ld (one query row per thread) and only compares.
//
// Two passes.  A sample pass over 1 base row in 8 to 128 leaves, per query, the smallest score of every few
// rows; about the fifth smallest of those is that query's bound.  The main pass appends every row scoring below
// the bound to a candidate list.  A third kernel recomputes the reference's exact fp32 distance
// chain (src/kernels.rs:200-231) for those candidates, picks the k best by (distance, id) and
// CERTIFIES the result: a query passes only if every row that was not a candidate is provably
// farther than its k-th result.  Queries that do not pass are re-run by the full-precision scan,
// so 16-bit scores never decide a result on their own.  L2 over whole numbers within 255 of each other is scored in 8-bit
// integers instead, exactly (convert8_rows_kernel): there the scores are the distances, and the re-rank reads no row.
//
// Work split: a unit is (query tile, 256 base rows); see make_tiling for how units become chunks
// and chunks are dealt to the persistent CTAs (one per SM) so that base tiles are shared in L2.
//
// Two tilings share the code:
//   MH = 2: 256 queries per tile, kept in shared memory for a whole chunk (K <= 128);
//           the two 128-row halves use the two accumulator slots, so each B tile is read once
//           from L2 for 256 queries.
//   MH = 1: 128 queries per tile (K <= 384); the two accumulator slots alternate between units.
// Batches with queries for more than one such tile are dealt to pairs of CTAs, two tiles at a time (gemm_topk_body, PAIR).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <numeric>

#include "internal.h"

namespace fv {

static constexpr int TILE_N = 256;     // base rows per unit
static constexpr int KBLK = 64;        // k elements per shared-memory block (128 bytes)
static constexpr int A_BLOCK_BYTES = 128 * 128;   // 128 rows x 128 B
static constexpr int B_STAGE_BYTES = TILE_N * 128;  // (of a pair of CTAs: half in each)
static constexpr int EXT_K = 16;                  // k elements of the norm step: one MMA
static constexpr int A_EXT_BYTES = 128 * EXT_K * 2;     // query side of the norm step
static constexpr int B_EXT_BYTES = TILE_N * EXT_K * 2;  // base side: one 8 KB tile per unit
static constexpr int NEPI = 16;        // epilogue warps: four per tensor-memory lane quadrant
static constexpr int NTHREADS = 64 + NEPI * 32;   // warp 0 TMA, warp 1 MMA, warps 2..17 epilogue
static constexpr long long WAIT_LIMIT_CYCLES = 4000000000ll;  // about 2 s; then the kernel gives up

// ------------------------------------------------------------------------------------------------
// PTX wrappers
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// What a waiting thread needs to give up: the CTA's abort flag (shared memory) and the launch's limit in cycles.
struct AbortCtl {
  volatile int* flag;
  long long limit;
};

// Bounded wait.  Returns false when the limit ran out or another thread already gave up.
// Every failed probe reads shared memory, and the tensor cores fetch their operands through the same port:
// sixteen warps probing back to back slow the MMAs measurably, so a waiting thread sleeps between probes.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, const AbortCtl& abort_flag, unsigned sleep_ns = 64) {
  if (mbar_try(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
    for (int i = 0; i < 64; ++i) {
      if (sleep_ns) __nanosleep(sleep_ns);
      if (mbar_try(bar, parity)) return true;
    }
    if (*abort_flag.flag) return false;
    if (clock64() - t0 > abort_flag.limit) {
      *abort_flag.flag = 1;
      return false;
    }
  }
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

// ---- two CTAs of a cluster working as a pair (cta_group::2): the first one's barriers are known to both by their
// cluster-wide addresses, a commit arrives on the barriers of both
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t in_first_cta(const void* p) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
// (at the scope of the CTA: what it hands over is tensor memory, not memory; a release at that of the cluster waits for the
// thread's stores: 2,376 us for 10,000 queries at 1M x 128, 1,478 without)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"(map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}

__device__ __forceinline__ void bulk_load_1d(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

template <bool PAIR>
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  if (PAIR) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                     smem_u32(bar)),
                 "h"(uint16_t(3))
                 : "memory");
    return;
  }
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

template <bool PAIR>
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                           uint32_t accumulate) {
  if (PAIR) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
    return;
  }
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// 8-bit signed operands, 32-bit integer accumulators: exact, and K = 32 in the time and bytes of a 16-bit K = 16.
template <bool PAIR>
__device__ __forceinline__ void tc_mma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                          uint32_t accumulate) {
  if (PAIR) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
    return;
  }
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// 32 lanes x 32 columns of 32-bit accumulators: thread l of the warp gets lane (base + l), columns c..c+31.
// The load is asynchronous: the registers are valid only after tc_ld_wait on the same array, which takes
// them as in/out operands so that no use can be scheduled ahead of the wait.
__device__ __forceinline__ void tc_ld32_issue(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_ld_wait(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]),
                 "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]),
                 "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]),
                 "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// The same for 64 columns.
__device__ __forceinline__ void tc_ld64_issue(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, "
      "%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, %48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]), "=r"(r[32]),
        "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]), "=r"(r[40]),
        "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]), "=r"(r[48]),
        "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]), "=r"(r[56]),
        "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_ld64_wait(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                 "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]),
                 "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
                 "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31]), "+r"(r[32]),
                 "+r"(r[33]), "+r"(r[34]), "+r"(r[35]), "+r"(r[36]), "+r"(r[37]), "+r"(r[38]), "+r"(r[39]), "+r"(r[40]),
                 "+r"(r[41]), "+r"(r[42]), "+r"(r[43]), "+r"(r[44]), "+r"(r[45]), "+r"(r[46]), "+r"(r[47]), "+r"(r[48]),
                 "+r"(r[49]), "+r"(r[50]), "+r"(r[51]), "+r"(r[52]), "+r"(r[53]), "+r"(r[54]), "+r"(r[55]), "+r"(r[56]),
                 "+r"(r[57]), "+r"(r[58]), "+r"(r[59]), "+r"(r[60]), "+r"(r[61]), "+r"(r[62]), "+r"(r[63])
               :
               : "memory");
}

__device__ __forceinline__ float min3(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Shared-memory matrix descriptors of K-major operands.  Low word: start address and leading byte offset (unused with
// swizzle: 1), both in 16-byte units; high word: stride byte offset, the descriptor version of this architecture (bit 46)
// and the swizzle (bits 61-63).  SW128: rows of 128 bytes, groups of 8 rows 1024 bytes apart; SW32 (a K of 32 bytes): rows
// of 32 bytes, groups 256 bytes apart.  Shared memory ends below 2^18, so an offset is added to the low word.
static constexpr uint32_t DESC_HI_SW128 = (1024u >> 4) | (1u << 14) | (2u << 29);
static constexpr uint32_t DESC_HI_SW32 = (256u >> 4) | (1u << 14) | (6u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return (saddr >> 4) | (1u << 16); }
__device__ __forceinline__ uint64_t make_desc(uint32_t lo, uint32_t hi) { return (uint64_t(hi) << 32) | lo; }

// true in one lane of the (converged) warp, always the same one
__device__ __forceinline__ bool elect_one() {
  uint32_t on;
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "elect.sync _|p, 0xFFFFFFFF;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(on));
  return on != 0;
}

// Instruction descriptor of kind::f16: fp32 accumulate, A and B both K-major, M x N tile.
__host__ __device__ constexpr uint32_t make_idesc(int m, int n, bool bf16) {
  return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) | (uint32_t(n >> 3) << 17) |
         (uint32_t(m >> 4) << 24);
}

// Instruction descriptor of kind::i8: 32-bit integer accumulate, A and B signed and K-major.
__host__ __device__ constexpr uint32_t make_idesc_i8(int m, int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(m >> 4) << 24);
}

// Ring position (stage index and phase bit), advanced without divisions: each role loop is a single thread on
// the critical path of the tensor pipe, and a 64-bit division per k block is a measurable bubble there.
struct StageCursor {
  int s, n;
  uint32_t phase;
  __device__ StageCursor(int n_) : s(0), n(n_), phase(0) {}
  __device__ __forceinline__ void next() {
    if (++s == n) {
      s = 0;
      phase ^= 1;
    }
  }
};

// ------------------------------------------------------------------------------------------------
struct GemmParams {
  int n, nq;
  int a_row0;      // operand row of the first query
  int grid;        // CTAs, or pairs of CTAs, that take work (task mode: all)
  int KB;          // k blocks of 128 bytes per row (64 16-bit or 128 8-bit elements)
  int last_steps;  // MMAs (32 bytes per row) of the last k block: 4 less the ones that would only meet padding
  int NT;          // base tiles of 256 rows
  int MT;          // query tiles of 128 * MH rows
  int cpn;         // base tiles per chunk
  int nchunks;     // MT * parts; chunk g = part * MT + query tile, taken by CTA g % grid as its (g / grid)-th segment
  int segmax;      // segments per CTA
  int nstage;
  int has_ext;        // L2: one more k step of 16 adds the row norms inside the MMA
  int ext_ring;       // norm-step tiles (8 KB each) kept in shared memory
  uint4 aext;         // the query side of the norm step: both 16-byte halves of every row
  const uint16_t* ext;  // base side of the norm step: 32 bytes per row, padded to whole tiles
  uint32_t idesc;
  // sample mode: the smallest score of every `group` (1, 8, 32 or 64) base rows, +inf beyond the last row
  float* smin;         // [MT * 128 * MH][smin_ld]
  int smin_ld, group;
  int* err;            // set to 1 when a bounded wait ran out
  long long wait_limit;  // cycles a thread waits on one barrier before the kernel gives up (WAIT_LIMIT_CYCLES)
  int fault_skip_unit;   // test hook, -1 = off: the producer of work item 0 leaves out the loads of this unit of it
  // threshold mode: per-query bounds from the sample pass, and the candidate buffers they fill
  const float* tau;      // [MT * 128 * MH]
  u64* cbuf;             // [grid * segmax][128 * MH][4][ccap] (score, row) keys: a list per query row, column quarter and segment
  unsigned int* ccnt;    // [grid * segmax][128 * MH][4] entries appended (may exceed ccap: overflow)
  int ccap;
  // task mode (TASKS): the work is a table of (A tile, run of B units) pairs instead of the tiling above
  // x: first operand row of the 256-row A tile; y: first B row of the task; z: its B units of 256 rows (low 16 bits)
  // and the number of the first one within the run of B rows the task is a segment of (high 16 bits: survivors and
  // the valid-row test count rows from the start of that run); w: valid B rows of the run
  const uint4* tasks;
  const uint32_t* ntasks;      // device word: number of tasks
  unsigned int* next_task;     // device word, zero at launch: the next task nobody has taken yet
  u64* pool;                   // [grid][pool_cap] survivors: (A row << 32) | B row relative to y
  unsigned int* pool_cnt;      // [grid] entries each CTA produced (may exceed pool_cap: overflow)
  unsigned int pool_cap;
  // A survivor that finds its CTA's pool full is dropped, and the owner of its operand row (row_owner[A row], a
  // query number) is marked in owner_dropped so that the caller can hand that query to another kernel.
  const uint32_t* row_owner;
  uint32_t* owner_dropped;
  // task mode, minima variant (minima != null): instead of survivors, the smallest score of every 32 B rows, for the
  // first task_rows[t] operand rows of task t: minima[task_moff[t] + (row in tile * units + unit) * 8 + column / 32];
  // B rows beyond the task's valid ones count as +inf.  Tasks with task_moff[t] == 0xFFFFFFFF write nothing.
  float* minima;
  const uint32_t* task_moff;
  const uint32_t* task_rows;
};

struct __align__(8) Barriers {
  uint64_t full[8], empty[8];
  uint64_t a_full, a_empty;
  uint64_t tfull[2], tempty[2];
  uint32_t tmem_base;
  int abort_flag;
  unsigned int pool_pos;  // task mode: survivors this CTA has appended
  // task mode: the tasks this CTA has drawn, handed from the producer to the MMA and epilogue warps.  Entry
  // i & 7 holds the i-th draw (a value >= the task count ends the work); tq_full[i & 7] completes once per draw.
  uint64_t tq_full[8];
  unsigned int tq[8];
};

// Sampling.  The sample pass scores 1 base row in E; a query's bound is its R-th best sampled score, so about R * E
// rows of the full set score below it (negative binomial) and the k nearest are among them unless R or more of the
// k - 1 nearest rows happen to be sampled: probability P(Binomial(k - 1, 1/E) >= R), kept below 2e-5 by the choice
// of R (5..13: k = 10 takes 5 to 7, k = 32 up to 13 -- with R capped at 7 a quarter of the queries of a k = 32
// search over 16384 rows failed their certificate and went to the full-precision scan).  E follows the base size
// (sqrt(n / 8000), up to twice that): the sample pass costs ~ n / E, hits and re-rank ~ R * E.  1M x 128, 10,000 queries over
// bytes, E 32 -> 16: sample and bound 66 -> 110 us, main pass and re-rank 1,539 -> 1,400; 200,003 x 384, 2,049 queries,
// E 16 -> 8: 34 -> 45 and 330 -> 301.
static constexpr int SAMPLE_R_MIN = 5, SAMPLE_R_MAX = 13;
static constexpr int TC_MAX_K = 128;  // results per query: what a warp of the re-rank still keeps sorted cheaply

static int pick_sample_every(size_t n) {
  int e = 8;
  while (e < 128 && double(e) * double(e) * 8000.0 < double(n)) e <<= 1;  // 512k -> 8, 2M -> 16, 8M -> 32
  return e;
}

// SAMPLE_R_MAX + 1: no R up to SAMPLE_R_MAX will do at this rate
static int pick_sample_r(int k, int every) {
  const double p = 1.0 / every;
  for (int r = SAMPLE_R_MIN; r <= SAMPLE_R_MAX; ++r) {
    // P(Binomial(k - 1, p) >= r) by summing the lower tail
    double tail = 1.0, term = std::pow(1.0 - p, k - 1);
    for (int i = 0; i < r; ++i) {
      tail -= term;
      term *= double(k - 1 - i) / double(i + 1) * p / (1.0 - p);
    }
    if (tail < 2e-5) return r;
  }
  return SAMPLE_R_MAX + 1;
}

// How a pass dealt out its work, for the kernels that read what it left; where a search may take the 8-bit operands, the
// device word q8_bad says which of the two passes ran.
struct PassShape {
  int MT, parts, grid, segmax, MH;
  int ctas;  // 2: pairs of CTAs
  int ccap;  // slots of a candidate list
};
struct PassShapes {
  PassShape s16, s8;
  const unsigned int* q8_bad;  // null: the base has no 8-bit operands
  __device__ __forceinline__ bool is8() const { return q8_bad && *q8_bad == 0u; }
  __device__ __forceinline__ const PassShape& taken() const { return is8() ? s8 : s16; }
};

// Accumulators as the epilogue compares them: scores in fp32, or whole numbers (I8), whose order is the same.
template <bool I8>
struct Score {
  typedef float T;
  __device__ static __forceinline__ T of(uint32_t r) { return __uint_as_float(r); }
  __device__ static __forceinline__ T bound(float f) { return f; }
  __device__ static __forceinline__ T min2(T a, T b) { return fminf(a, b); }
  __device__ static __forceinline__ T min3(T a, T b, T c) { return fv::min3(a, b, c); }
};
template <>
struct Score<true> {
  typedef int T;
  __device__ static __forceinline__ T of(uint32_t r) { return int(r); }
  // bounds are scores that this kernel wrote as floats (exact: below 2^24), or +inf
  __device__ static __forceinline__ T bound(float f) { return f < 2.0e9f ? int(f) : 0x7FFFFFFF; }
  __device__ static __forceinline__ T min2(T a, T b) { return min(a, b); }
  __device__ static __forceinline__ T min3(T a, T b, T c) { return min(min(a, b), c); }
};

// PAIR: the CTAs of a cluster of two work as one on tiles of twice as many queries (cta_group::2).  Each has its half of the
// queries and, of every 256 base rows, 128 in its shared memory; the first one issues the MMAs, which read both halves, so a
// base row is fetched into and read from shared memory once for twice the scores.  Each CTA's accumulators are its own
// queries' scores.
// 384 dimensions are bound by that traffic (209 cycles per 128 x 256 MMA with one CTA, 165 with pairs; 128 nominal): main
// pass of 2,049 queries over 200,003 x 384 274 -> 230 us; 5,000 over 500,000 x 128 in 16 bits 578 -> 499, in bytes, where the
// epilogue's hits bound it, 0.98 to 1.02 times.
template <int MH, bool SAMPLE, bool TASKS, bool I8, bool PAIR>
__device__ __forceinline__ void gemm_topk_body(const CUtensorMap& tmA, const CUtensorMap& tmB, const CUtensorMap& tmE,
                                               const GemmParams& p) {
  static_assert(!(TASKS && PAIR), "tasks are drawn by single CTAs");
  typedef Score<I8> S;
  typedef typename S::T T;
  constexpr int KE = I8 ? 2 * KBLK : KBLK;  // elements of a k block
  constexpr int CTAS = PAIR ? 2 : 1;
  constexpr int B_ROWS = TILE_N / CTAS;  // base rows of a unit in this CTA's shared memory
  constexpr int STAGE_BYTES = B_ROWS * 128, EXT_BYTES = B_ROWS * EXT_K * 2;
  const int rank = PAIR ? int(cluster_rank()) : 0, worker = int(blockIdx.x) / CTAS;
  if (!TASKS && worker >= p.grid) return;
  unsigned char* raw = dyn_smem();
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~uintptr_t(1023));
  unsigned char* sA = base;                                            // [MH][KB] blocks of 16 KB
  unsigned char* sAext = sA + size_t(MH) * p.KB * A_BLOCK_BYTES;       // 4 KB: the constant rows of the norm step
  unsigned char* sB = sAext + A_EXT_BYTES;                             // [nstage] stages of 32 KB (PAIR: 16)
  unsigned char* sE = sB + size_t(p.nstage) * STAGE_BYTES;             // [ext_ring] norm-step tiles of 8 KB (4)
  Barriers* bars = reinterpret_cast<Barriers*>(sE + size_t(p.ext_ring) * EXT_BYTES);
  const AbortCtl abort_flag{&bars->abort_flag, p.wait_limit};

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 8; ++i) {
      mbar_init(&bars->full[i], 1);
      mbar_init(&bars->empty[i], 1);
    }
    mbar_init(&bars->a_full, 1);
    mbar_init(&bars->a_empty, 1);
    for (int i = 0; i < 8; ++i) mbar_init(&bars->tq_full[i], 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->tfull[i], 1);
      mbar_init(&bars->tempty[i], NEPI * CTAS);
    }
    bars->abort_flag = 0;
    bars->pool_pos = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // Query side of the norm step.  Both 16-byte halves of a row are equal, so the 32-byte swizzle (which only exchanges
  // the halves of some rows) leaves the tile as written.
  if (threadIdx.x < A_EXT_BYTES / 16) reinterpret_cast<uint4*>(sAext)[threadIdx.x] = p.aext;
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  if (warp == 1) {  // the MMA warp owns the tensor memory: all 512 columns (one CTA per SM)
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&bars->tmem_base))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&bars->tmem_base))
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();  // the other CTA's barriers are set up
  tc_fence_after();
  const uint32_t tmem_base = bars->tmem_base;
  // Work items.  Plain and threshold mode: chunk g of the tiling, CTA b taking g = b, b + grid, ...
  // Task mode: tasks cost very different amounts (their length, and how many survivors the epilogue has to append),
  // so they are not dealt in advance: the producer draws the next task from a device-wide counter whenever the
  // operand tile is free again, and passes the number on to the MMA and epilogue warps through a small ring in shared
  // memory.  The ring has 8 entries; the producer is at most 3 draws ahead of the slowest reader, because it draws
  // task i + 1 only after every MMA of task i - 1 has completed, by when the epilogue is at work on task i - 2 at
  // the latest (two accumulator slots).  The caller sorts the tasks by decreasing length: longest first.
  const int nwork = TASKS ? int(*p.ntasks) : p.nchunks;
  auto work_of = [&](int seg) -> int {  // consumer side
    if (!TASKS) return worker + seg * p.grid;
    if (!mbar_wait(&bars->tq_full[seg & 7], uint32_t(seg >> 3) & 1, abort_flag)) return 0x7FFFFFFF;
    return int(*reinterpret_cast<volatile unsigned int*>(&bars->tq[seg & 7]));
  };
  auto draw = [&](int seg) -> int {  // producer side
    if (!TASKS) return worker + seg * p.grid;
    const unsigned int g = min(atomicAdd(p.next_task, 1u), 0x7FFFFFFEu);
    bars->tq[seg & 7] = g;
    mbar_arrive(&bars->tq_full[seg & 7]);  // release: the entry is visible to whoever sees this phase complete
    return int(g);
  };

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      bool ok = true;
      StageCursor st(p.nstage);
      int ring = 0, seg = 0;
      // (both CTAs of a pair fill their halves of a stage and count on the first one's barrier)
      auto load = [&](void* dst, const CUtensorMap& map, uint64_t* bar, int x, int y) {
        if (PAIR) tma_load_2d_pair(dst, &map, in_first_cta(bar), x, y);
        else tma_load_2d(dst, &map, bar, x, y);
      };
      for (int g = draw(0); g < nwork && ok; g = draw(++seg)) {
        int nt0, nt1, a_row0, b_row0 = 0;
        if (TASKS) {
          const uint4 t = p.tasks[g];
          a_row0 = int(t.x);
          b_row0 = int(t.y);
          nt0 = 0;
          nt1 = int(t.z & 0xFFFFu);
        } else {
          const int part = g / p.MT, mt = g - part * p.MT;
          nt0 = part * p.cpn;
          nt1 = min(p.NT, nt0 + p.cpn);
          a_row0 = p.a_row0 + (mt * CTAS + rank) * MH * 128;
        }
        ok = mbar_wait(&bars->a_empty, (seg & 1) ^ 1, abort_flag);
        if (!ok) break;
        if (rank == 0) mbar_expect_tx(&bars->a_full, uint32_t(CTAS * MH * p.KB * A_BLOCK_BYTES));
        for (int mh = 0; mh < MH; ++mh)
          for (int kb = 0; kb < p.KB; ++kb)
            load(sA + size_t(mh * p.KB + kb) * A_BLOCK_BYTES, tmA, &bars->a_full, kb * KE, a_row0 + mh * 128);
        for (int nt = nt0; nt < nt1 && ok; ++nt) {
          for (int kb = 0; kb < p.KB; ++kb, st.next()) {
            const int s = st.s;
            ok = mbar_wait(&bars->empty[s], st.phase ^ 1, abort_flag);
            if (!ok) break;
            // The unit's norm-step tile rides on the barrier of its first k block.  Its ring slot is reused
            // ext_ring units later; the stage acquired just above was last read by a unit at most
            // ceil(nstage / KB) back, and the commit that freed it also covers every norm step issued before it.
            const bool with_ext = kb == 0 && p.has_ext;
            // (test hook: the stage is never posted, its consumer waits until the limit and the kernel gives up)
            if (p.fault_skip_unit >= 0 && g == 0 && nt == nt0 + p.fault_skip_unit) continue;
            if (rank == 0) mbar_expect_tx(&bars->full[s], uint32_t(CTAS * (STAGE_BYTES + (with_ext ? EXT_BYTES : 0))));
            // first B row of the unit (task mode: a multiple of 8, which keeps the norm tile's swizzle image in step)
            const size_t brow = size_t(b_row0) + size_t(nt) * TILE_N + rank * B_ROWS;
            if (with_ext) {  // stored as the swizzled shared-memory image: one contiguous copy (PAIR: as rows of 128 bytes)
              if (PAIR) load(sE + size_t(ring) * EXT_BYTES, tmE, &bars->full[s], 0, int(brow / 4));
              else bulk_load_1d(sE + size_t(ring) * EXT_BYTES, p.ext + brow * EXT_K, EXT_BYTES, &bars->full[s]);
            }
            load(sB + size_t(s) * STAGE_BYTES, tmB, &bars->full[s], kb * KE, int(brow));
          }
          if (++ring == p.ext_ring) ring = 0;
        }
      }
      if (PAIR && ok && seg > 0) {  // nor while the first CTA's commits may still arrive here: the last ones of all stages and tiles
        for (int i = 0; i < p.nstage && ok; ++i, st.next()) ok = mbar_wait(&bars->empty[st.s], st.phase ^ 1, abort_flag);
        ok = ok && mbar_wait(&bars->a_empty, (seg & 1) ^ 1, abort_flag);
      }
      // Do not leave while copies may still land in this CTA's shared memory: wait (bounded) until the
      // MMA side has consumed everything that was issued, or until the abort flag says nobody will.
      if (!ok) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {
        }
      }
    }
  } else if (warp == 1 && rank == 0) {
    // ---------------------------------------------------------------- MMA issuer
    // The whole warp walks the loop, so that everything an MMA is issued with is uniform, and one elected lane issues.
    // Descriptors advance by adding to their low words.
    const bool leader = elect_one();
    int job = 0, ring = 0;
    bool ok = true;
    StageCursor st(p.nstage);
    const uint32_t a_lo0 = desc_lo(smem_u32(sA)), b_lo0 = desc_lo(smem_u32(sB)), e_lo0 = desc_lo(smem_u32(sE));
    const uint32_t aext_lo = desc_lo(smem_u32(sAext));
    auto mma = [&](uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
      if (I8) tc_mma_i8<PAIR>(d, a, b, p.idesc, accumulate);
      else tc_mma_f16<PAIR>(d, a, b, p.idesc, accumulate);
    };
    for (int seg = 0, g = work_of(0); g < nwork && ok; g = work_of(++seg)) {
      int nt0, nt1;
      if (TASKS) {
        nt0 = 0;
        nt1 = int(p.tasks[g].z & 0xFFFFu);
      } else {
        const int part = g / p.MT;
        nt0 = part * p.cpn;
        nt1 = min(p.NT, nt0 + p.cpn);
      }
      ok = __all_sync(FV_FULL, mbar_wait(&bars->a_full, seg & 1, abort_flag, 0));
      if (!ok) break;
      tc_fence_after();
      for (int nt = nt0; nt < nt1 && ok; ++nt) {
#pragma unroll
        for (int mh = 0; mh < MH; ++mh, ++job) {
          const int slot = job & 1;
          ok = ok && __all_sync(FV_FULL, mbar_wait(&bars->tempty[slot], (uint32_t(job >> 1) & 1) ^ 1, abort_flag, 0));
          if (!ok) break;
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + uint32_t(slot * TILE_N);
          StageCursor sk = st;  // both halves walk the same stages of this unit
          for (int kb = 0; kb < p.KB; ++kb, sk.next()) {
            const int s = sk.s;
            if (mh == 0) {
              ok = __all_sync(FV_FULL, mbar_wait(&bars->full[s], sk.phase, abort_flag, 0));
              if (!ok) break;
              tc_fence_after();
            }
            if (leader) {
              uint32_t acc = kb != 0 ? 1u : 0u;  // the first MMA of a job overwrites the accumulator
              if (kb == 0 && p.has_ext) {        // + ||b||^2: always the first step of a job
                mma(d_tmem, make_desc(aext_lo, DESC_HI_SW32), make_desc(e_lo0 + uint32_t(ring * (EXT_BYTES >> 4)), DESC_HI_SW32), 0u);
                acc = 1;
              }
              const uint32_t a_lo = a_lo0 + uint32_t((mh * p.KB + kb) * (A_BLOCK_BYTES >> 4));
              const uint32_t b_lo = b_lo0 + uint32_t(s * (STAGE_BYTES >> 4));
              mma(d_tmem, make_desc(a_lo, DESC_HI_SW128), make_desc(b_lo, DESC_HI_SW128), acc);
              if (kb + 1 < p.KB || p.last_steps == 4) {
#pragma unroll
                for (int k4 = 1; k4 < 4; ++k4)
                  mma(d_tmem, make_desc(a_lo + 2 * k4, DESC_HI_SW128), make_desc(b_lo + 2 * k4, DESC_HI_SW128), 1u);
              } else {
                for (int k4 = 1; k4 < p.last_steps; ++k4)
                  mma(d_tmem, make_desc(a_lo + 2 * k4, DESC_HI_SW128), make_desc(b_lo + 2 * k4, DESC_HI_SW128), 1u);
              }
              if (mh == MH - 1) tc_commit<PAIR>(&bars->empty[s]);  // the stage is free once these MMAs have read it
              if (kb + 1 == p.KB) tc_commit<PAIR>(&bars->tfull[slot]);
            }
            __syncwarp();
          }
          if (!ok) break;
        }
        for (int kb = 0; kb < p.KB; ++kb) st.next();
        if (++ring == p.ext_ring) ring = 0;
      }
      if (ok && leader) tc_commit<PAIR>(&bars->a_empty);  // the query tile may be replaced once every MMA above has read it
      __syncwarp();
    }
  } else if (warp > 1) {
    // ---------------------------------------------------------------- epilogue: 16 warps, one query row per thread
    // Every warp reads its 64 columns of every accumulator in one load and hands the slot back at once: what it then does
    // with them delays no MMA as long as it keeps up on average.  (With MH = 2 each half's accumulators used to belong to
    // half of the warps, 128 columns each in two loads: the slot then waited for the slowest warp's hits.  10,000 queries at
    // 1M x 128, main pass over bytes: 1,785 us, now 1,449.)
    const int ew = warp - 2;
    const int quad = warp & 3;   // tensor-memory lanes this warp may read: 32 * quad .. +31
    const int sub = ew >> 2;     // warp group 0..3: which quarter of the columns
    const int r0 = quad * 32 + lane;  // row within 128
    const uint32_t lane_addr = uint32_t(quad * 32) << 16;
    int job = 0;
    bool ok = true;
    constexpr int NCOL = TILE_N / 4;
    const int col0 = sub * NCOL;
    uint32_t n_rows = uint32_t(p.n);
    uint32_t unit0 = 0;  // task mode: number of the task's first unit within its B run
    struct Row {         // this thread's row of each 128-row half
      T thr;
      unsigned int ncand;
      u64* list;         // threshold mode: its candidates of the current segment
      float* sdst;       // sample mode: its row of smin
      uint32_t a_row;    // task mode: the operand row
      float* mdst;       // task mode, minima variant: where its minima of the current task go
    } rows[MH];
    for (int seg = 0, g = work_of(0); g < nwork && ok; g = work_of(++seg)) {
      int nt0, nt1, mt = 0;
      uint4 t = make_uint4(0, 0, 0, 0);
      if (TASKS) {
        t = p.tasks[g];
        nt0 = 0;
        nt1 = int(t.z & 0xFFFFu);
        unit0 = t.z >> 16;
        n_rows = t.w;  // rows of this task's B run; the rest of its last unit belongs to someone else
      } else {
        const int part = g / p.MT;
        mt = g - part * p.MT;
        nt0 = part * p.cpn;
        nt1 = min(p.NT, nt0 + p.cpn);
      }
      const size_t lists0 = (size_t(blockIdx.x) * p.segmax + seg) * (128 * MH * 4) + sub;
#pragma unroll
      for (int mh = 0; mh < MH; ++mh) {
        Row& w = rows[mh];
        const int r = mh * 128 + r0, q = (mt * CTAS + rank) * (128 * MH) + r;
        w.ncand = 0;
        if (SAMPLE) {
          w.sdst = p.smin + size_t(q) * p.smin_ld;
        } else if (TASKS) {
          w.a_row = t.x + uint32_t(r);
          w.thr = S::bound(p.minima ? 0.f : p.tau[w.a_row]);
          w.mdst = nullptr;
          if (p.minima) {
            const uint32_t moff = p.task_moff[g];
            if (moff != 0xFFFFFFFFu && uint32_t(r) < p.task_rows[g]) w.mdst = p.minima + size_t(moff) + size_t(r) * (t.z & 0xFFFFu) * 8;
          }
        } else {  // the bound is fixed: the sample pass's estimate for this query
          w.thr = S::bound(p.tau[q]);
          w.list = p.cbuf + (lists0 + size_t(r) * 4) * size_t(p.ccap);
        }
      }
      for (int nt = nt0; nt < nt1 && ok; ++nt) {
        const uint32_t row_base = (unit0 + uint32_t(nt)) * TILE_N + col0;
#pragma unroll
        for (int mh = 0; mh < MH; ++mh, ++job) {
          const int slot = job & 1;
          ok = ok && __all_sync(FV_FULL, mbar_wait(&bars->tfull[slot], uint32_t(job >> 1) & 1, abort_flag));
          if (!ok) break;
          tc_fence_after();
          Row& w = rows[mh];
          // Threshold mode.  The accumulator IS the score (the norm step and the scaled query side put
          // ||b||^2 - 2<q,b> there), so a chunk of 64 columns costs a minimum tree and one vote.  Every column
          // below the bound is appended to this thread's private list: a plain store and a register counter.
          // the runs of eight columns in which some row of the warp has a hit
          auto runs_with_hits = [&](const uint32_t* r) -> uint32_t {
            T g8[8];
#pragma unroll
            for (int gi = 0; gi < 8; ++gi) {
              const uint32_t* q = r + gi * 8;
              const T t0 = S::min3(S::of(q[0]), S::of(q[1]), S::of(q[2]));
              const T t1 = S::min3(S::of(q[3]), S::of(q[4]), S::of(q[5]));
              g8[gi] = S::min2(S::min3(t0, t1, S::of(q[6])), S::of(q[7]));
            }
            const T m = S::min2(S::min3(g8[0], g8[1], g8[2]), S::min3(S::min3(g8[3], g8[4], g8[5]), g8[6], g8[7]));
            if (!__any_sync(FV_FULL, m < w.thr)) return 0u;
            uint32_t runs = 0;
#pragma unroll
            for (int gi = 0; gi < 8; ++gi) runs |= g8[gi] < w.thr ? 1u << gi : 0u;
            return __reduce_or_sync(FV_FULL, runs);
          };
          auto chunk = [&](const uint32_t* r) {
            uint32_t groups = runs_with_hits(r);
            // One run at a time: its eight scores are moved to the same registers, so that there is one copy of the code
            // that looks at them (with eight the loop outgrew the instruction cache: 3 times the time at MH = 2).
            while (groups) {
              const int gi = __ffs(groups) - 1;
              groups &= groups - 1;
              T v[8];
              auto run = [&](int k) {
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = S::of(r[k * 8 + i]);
              };
              switch (gi) {
                case 0: run(0); break;
                case 1: run(1); break;
                case 2: run(2); break;
                case 3: run(3); break;
                case 4: run(4); break;
                case 5: run(5); break;
                case 6: run(6); break;
                default: run(7); break;
              }
              const uint32_t row0 = row_base + uint32_t(gi * 8);
              uint32_t hits = 0;
#pragma unroll
              for (int i = 0; i < 8; ++i) hits |= v[i] < w.thr ? 1u << i : 0u;
              if (row0 + 8 > n_rows) hits &= row0 < n_rows ? (1u << (n_rows - row0)) - 1u : 0u;
              while (hits) {
                const int i = __ffs(hits) - 1;
                hits &= hits - 1;
                const T a = i & 1 ? v[1] : v[0], b = i & 1 ? v[3] : v[2], c = i & 1 ? v[5] : v[4], d = i & 1 ? v[7] : v[6];
                const T x = i & 4 ? (i & 2 ? d : c) : (i & 2 ? b : a);
                if (w.ncand < unsigned(p.ccap)) w.list[w.ncand] = make_key(float(x), row0 + uint32_t(i));
                w.ncand++;
              }
              __syncwarp();
            }
          };
          // Task mode.  Survivors are dense where a query meets its own neighbourhood (one row in ten of a near list),
          // so the append must not cost a shared-memory atomic per hit: every thread collects its hits of the chunk
          // as two bit masks, the warp reserves room for all of them with ONE atomic on the CTA's counter, and each
          // thread stores its own.
          auto chunk_tasks = [&](const uint32_t* r) {
            const uint32_t runs = runs_with_hits(r);
            if (!runs) return;
            uint32_t mk[2] = {0u, 0u};
#pragma unroll
            for (int gi = 0; gi < 8; ++gi) {
              if (!(runs & (1u << gi))) continue;
#pragma unroll
              for (int i = gi * 8; i < gi * 8 + 8; ++i)
                if (S::of(r[i]) < w.thr) mk[i >> 5] |= 1u << (i & 31);
            }
            if (row_base + 64u > n_rows) {  // the run ends within these columns
              const uint32_t left = row_base < n_rows ? n_rows - row_base : 0u;
              mk[0] &= left >= 32u ? ~0u : (1u << left) - 1u;
              mk[1] &= left >= 64u ? ~0u : left > 32u ? (1u << (left - 32u)) - 1u : 0u;
            }
            const int mine = __popc(mk[0]) + __popc(mk[1]);
            int incl = mine;  // inclusive prefix sum over the warp
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const int t = __shfl_up_sync(FV_FULL, incl, o);
              if (lane >= o) incl += t;
            }
            const int total = __shfl_sync(FV_FULL, incl, 31);
            if (total == 0) return;
            unsigned int base = 0;
            if (lane == 31) base = atomicAdd(&bars->pool_pos, unsigned(total));
            base = __shfl_sync(FV_FULL, base, 31);
            unsigned int pos = base + unsigned(incl - mine);
            u64* dst = p.pool + size_t(blockIdx.x) * p.pool_cap;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint32_t mm = mk[h];
              while (mm) {
                const int i = __ffs(mm) - 1;
                mm &= mm - 1;
                if (pos < p.pool_cap) dst[pos] = (u64(w.a_row) << 32) | u64(row_base + uint32_t(h * 32 + i));
                ++pos;
              }
            }
            if (mine && pos > p.pool_cap) p.owner_dropped[p.row_owner[w.a_row]] = 1u;  // some of this row's did not fit
          };
          // Sample mode.  Minima of 8 columns, of 32 or of 64, or every score: 4 to 256 bytes of the query's own row.
          auto sample = [&](uint32_t* r) {
            const uint32_t row0 = row_base;
            const T inf = S::bound(INFINITY);
            if (row0 + 64 > n_rows) {
#pragma unroll
              for (int i = 0; i < 64; ++i)
                if (row0 + uint32_t(i) >= n_rows) r[i] = I8 ? 0x7FFFFFFFu : 0x7F800000u;
            }
            const auto f = [&](T v) { return I8 && v == inf ? INFINITY : float(v); };
            float4* d4 = reinterpret_cast<float4*>(w.sdst + row0 / uint32_t(p.group));
            if (p.group == 1) {
#pragma unroll
              for (int i = 0; i < 64; i += 4) d4[i / 4] = make_float4(f(S::of(r[i])), f(S::of(r[i + 1])), f(S::of(r[i + 2])), f(S::of(r[i + 3])));
              return;
            }
            T g8[8];
#pragma unroll
            for (int gi = 0; gi < 8; ++gi) {
              const uint32_t* q = r + gi * 8;
              g8[gi] = S::min2(S::min3(S::min3(S::of(q[0]), S::of(q[1]), S::of(q[2])), S::of(q[3]), S::of(q[4])),
                               S::min3(S::of(q[5]), S::of(q[6]), S::of(q[7])));
            }
            if (p.group == 8) {
              d4[0] = make_float4(f(g8[0]), f(g8[1]), f(g8[2]), f(g8[3]));
              d4[1] = make_float4(f(g8[4]), f(g8[5]), f(g8[6]), f(g8[7]));
              return;
            }
            const T a = S::min2(S::min3(g8[0], g8[1], g8[2]), g8[3]), b = S::min2(S::min3(g8[4], g8[5], g8[6]), g8[7]);
            if (p.group == 32) *reinterpret_cast<float2*>(d4) = make_float2(f(a), f(b));
            else *reinterpret_cast<float*>(d4) = f(S::min2(a, b));
          };
          uint32_t rbuf[64];
          tc_ld64_issue(tmem_base + lane_addr + uint32_t(slot * TILE_N + col0), rbuf);
          tc_ld64_wait(rbuf);
          tc_fence_before();  // the load has landed: the MMA may overwrite this accumulator slot
          __syncwarp();
          if (lane == 0) {
            if (PAIR) mbar_arrive_cluster(in_first_cta(&bars->tempty[slot]));
            else mbar_arrive(&bars->tempty[slot]);
          }
          if (SAMPLE) {
            sample(rbuf);
          } else if (!TASKS) {
            chunk(rbuf);
          } else if (!p.minima) {
            chunk_tasks(rbuf);
          } else if (w.mdst) {
            // minima variant: the smallest score of every 32 columns, rows beyond the task's as +inf
            float g2[2];
            const bool tail = row_base + 63u >= n_rows;
#pragma unroll
            for (int gi = 0; gi < 2; ++gi) {
              float m = INFINITY;
#pragma unroll
              for (int i = gi * 32; i < gi * 32 + 32; ++i) {
                const float v = __uint_as_float(rbuf[i]);
                m = fminf(m, (!tail || row_base + uint32_t(i) < n_rows) ? v : INFINITY);
              }
              g2[gi] = m;
            }
            *reinterpret_cast<float2*>(w.mdst + size_t(nt) * 8 + col0 / 32) = make_float2(g2[0], g2[1]);
          }
        }
      }
      if (!ok) break;
      if (!SAMPLE && !TASKS) {
#pragma unroll
        for (int mh = 0; mh < MH; ++mh) p.ccnt[lists0 + size_t(mh * 128 + r0) * 4] = rows[mh].ncand;
      }
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (PAIR) cluster_sync();  // nothing of the other CTA's is on its way here
  if (threadIdx.x == 0 && *abort_flag.flag) atomicExch(p.err, 1);
  if (TASKS && threadIdx.x == 0) p.pool_cnt[blockIdx.x] = bars->pool_pos;
  if (warp == 1) {
    tc_fence_after();
    if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
  }
}

// What a pass is launched with; the maps of the operands and, for pairs, of the norm step's tiles
struct GemmWay {
  CUtensorMap tmA, tmB, tmE;
  GemmParams p;
};
template <int MH, bool SAMPLE, bool TASKS, bool PAIR>
__global__ void __launch_bounds__(NTHREADS, 1) gemm_topk_kernel(const __grid_constant__ GemmWay w) {
  gemm_topk_body<MH, SAMPLE, TASKS, false, PAIR>(w.tmA, w.tmB, w.tmE, w.p);
}

// The pass over the 8-bit operands or, where a query of the batch does not fit them (q8_bad, known on the device only), over
// the 16-bit ones: one launch, since one that leaves at once costs a pass over 100,000 rows 3 us of 40.
template <int MH16, bool SAMPLE, bool PAIR>
__global__ void __launch_bounds__(NTHREADS, 1)
    gemm_topk_either_kernel(const __grid_constant__ GemmWay w16, const __grid_constant__ GemmWay w8, const unsigned int* q8_bad) {
  if (*q8_bad) gemm_topk_body<MH16, SAMPLE, false, false, PAIR>(w16.tmA, w16.tmB, w16.tmE, w16.p);
  else gemm_topk_body<2, SAMPLE, false, true, PAIR>(w8.tmA, w8.tmB, w8.tmE, w8.p);
}

// ------------------------------------------------------------------------------------------------
// fp32 rows -> 16-bit operand rows (zero padded to Kp), squared norms and range statistics
struct RangeStats {
  float min_v, max_v;      // over all values seen
  float max_norm2;         // largest squared row norm
  int not_integer;         // some value is not integer-valued
  int not_finite;
};

__device__ __forceinline__ void atomic_min_f(float* a, float v) {
  if (v >= 0) atomicMin(reinterpret_cast<int*>(a), __float_as_int(v));
  else atomicMax(reinterpret_cast<unsigned*>(a), __float_as_uint(v));
}
__device__ __forceinline__ void atomic_max_f(float* a, float v) {
  if (v >= 0) atomicMax(reinterpret_cast<int*>(a), __float_as_int(v));
  else atomicMin(reinterpret_cast<unsigned*>(a), __float_as_uint(v));
}

// ---- 8-bit operands, for L2 over whole numbers that lie within 255 of each other (bytes, as SIFT's components are).
// With b' = b - lo - 128 and a = 127 - (q - lo), both in [-128, 127], and t = sum (b' + 1)^2,
//   ||q - b||^2 = 2 (a . b' + floor(t / 2)) + (t & 1) + sum (q - lo - 128)^2 - pd
// in whole numbers, so the tensor cores' integer score a . b' + floor(t / 2) and the parity of t give the distance
// itself.  floor(t / 2) enters in one MMA of K = 32 like the norm of the 16-bit form: it is 127 times a number that 30
// bytes of at most 255 add up to (stored less 128, which takes I8_SHIFT off every score), plus a remainder that the
// query side multiplies by 1.  Scores stay below 2^22, distances and doubled scores below 2^24: exact as floats too.
// Half the MMAs per score, and the re-rank has no row left to read: 10,000 queries at 1M x 128, main pass 2,400 -> 1,837 us,
// re-rank 196 -> 57, the search 2,964 -> 2,181; 501 queries, 100 results of 50,001 x 100 211 -> 176.
static constexpr int I8_MAX_PD = 224;
static constexpr int I8_MAX_HALF = 30 * 255 * 127 + 126;  // the largest floor(t / 2) that fits
static constexpr int I8_SHIFT = 30 * 127 * 128;

// one warp per row: the operand row, the image of its 32 bytes of the norm step (rows from n on: a large one), the parity
// of t; `too_large` is set when a row's floor(t / 2) does not fit
__global__ void convert8_rows_kernel(const float* __restrict__ src, size_t first, size_t n, size_t n_pad, int pd, int Kp8, float lo,
                                     uint8_t* __restrict__ dst, uint8_t* __restrict__ ext, uint8_t* __restrict__ parity,
                                     unsigned int* __restrict__ too_large) {
  const int lane = threadIdx.x & 31;
  const size_t row = first + blockIdx.x * size_t(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n_pad) return;
  int t = 2 * I8_MAX_HALF;
  if (row < n) {
    t = 0;
    for (int c = lane; c < Kp8; c += 32) {
      int v = 0;
      if (c < pd) {
        v = int(src[row * size_t(pd) + c] - lo) - 128;
        t += (v + 1) * (v + 1);
      }
      dst[row * size_t(Kp8) + c] = uint8_t(int8_t(v));
    }
    t = __reduce_add_sync(FV_FULL, t);
    if (lane == 0) {
      parity[row] = uint8_t(t & 1);
      if (t / 2 > I8_MAX_HALF) *too_large = 1u;
    }
  }
  const int h = min(t / 2, I8_MAX_HALF);
  const int left = h / 127, j = lane < 16 ? lane - 1 : lane - 2;  // the lane's place among the 30
  const int x = lane == 0 ? h % 127 : lane == 16 ? 0 : min(255, max(0, left - 255 * j)) - 128;
  ext[row * 32 + (lane ^ ((int(row >> 2) & 1) << 4))] = uint8_t(int8_t(x));
}

// one warp per row.  dst8 (queries over a base with 8-bit operands): the 8-bit query row and the query's constant of the
// formula above as well; q8_bad is set when a component is not one of the base's 256 numbers.
template <bool BF16>
__global__ void convert_rows_kernel(const float* __restrict__ src, size_t n, int pd, int Kp, uint16_t* __restrict__ dst,
                                    float* __restrict__ norm2, int is_l2, float mul, RangeStats* __restrict__ st,
                                    uint8_t* __restrict__ dst8, int Kp8, float lo8, float* __restrict__ const8,
                                    unsigned int* __restrict__ q8_bad) {
  const int lane = threadIdx.x & 31;
  const size_t row = blockIdx.x * size_t(blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= n) return;
  float s = 0.f, mn = INFINITY, mx = -INFINITY;
  int bad_int = 0, bad_fin = 0;
  for (int c = lane; c < Kp; c += 32) {
    float x = c < pd ? src[row * size_t(pd) + c] : 0.f;
    if (c < pd) {
      s = __fmaf_rn(x, x, s);
      mn = fminf(mn, x);
      mx = fmaxf(mx, x);
      if (x != rintf(x)) bad_int = 1;
      if (!(fabsf(x) <= 3.0e38f)) bad_fin = 1;
    }
    uint16_t h;
    if (BF16) h = __bfloat16_as_ushort(__float2bfloat16_rn(x * mul));
    else h = __half_as_ushort(__float2half_rn(x * mul));
    dst[row * size_t(Kp) + c] = h;
  }
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(FV_FULL, s, o);
    mn = fminf(mn, __shfl_xor_sync(FV_FULL, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(FV_FULL, mx, o));
    bad_int |= __shfl_xor_sync(FV_FULL, bad_int, o);
    bad_fin |= __shfl_xor_sync(FV_FULL, bad_fin, o);
  }
  if (dst8) {
    int t = 0;
    bool bad = bad_int || bad_fin;
    for (int c = lane; c < Kp8; c += 32) {
      const float v = c < pd ? src[row * size_t(pd) + c] - lo8 : 127.f;
      bad = bad || !(v >= 0.f && v <= 255.f);
      const int w = bad ? 127 : int(v);
      if (c < pd) t += (w - 128) * (w - 128);
      dst8[row * size_t(Kp8) + c] = uint8_t(int8_t(127 - w));
    }
    t = __reduce_add_sync(FV_FULL, t);
    bad = __any_sync(FV_FULL, bad);
    if (lane == 0) {
      const8[row] = float(t - pd + 2 * I8_SHIFT);
      if (bad) *q8_bad = 1u;
    }
  }
  if (lane == 0) {
    if (norm2) norm2[row] = is_l2 ? s : 0.f;
    atomic_min_f(&st->min_v, mn);
    atomic_max_f(&st->max_v, mx);
    atomic_max_f(&st->max_norm2, s);
    if (bad_int) st->not_integer = 1;
    if (bad_fin) st->not_finite = 1;
  }
}

// Base side of the norm step: ||b||^2 / 2^e as three 16-bit pieces (p0 + p1 + p2, each the rounding of what the
// ones before left), then 13 zeros.  The query side holds 2^e three times, so the MMA adds the norm back exactly
// to 24 bits (fp16: 3 x 11 bits, bf16: 3 x 8).  Rows with a non-finite norm (the padding is +inf) get +inf.
// The array is kept as the shared-memory image of the 32-byte swizzle (the two 16-byte halves of a row trade
// places in rows 4..7 of every 8), so that a tile is one contiguous bulk copy instead of 256 narrow TMA rows.
template <bool BF16>
__global__ void split_norms_kernel(const float* __restrict__ norm2, size_t first, size_t count, float inv_scale,
                                   uint16_t* __restrict__ ext) {
  const size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x;
  if (i >= count) return;
  const size_t row = first + i;
  const float t = norm2[row] * inv_scale;
  uint16_t pc[3] = {0, 0, 0};
  if (!(fabsf(t) < INFINITY)) {
    pc[0] = BF16 ? 0x7F80 : 0x7C00;
  } else {
    float r = t;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      float back;
      if (BF16) {
        const __nv_bfloat16 h = __float2bfloat16_rn(r);
        pc[j] = __bfloat16_as_ushort(h);
        back = __bfloat162float(h);
      } else {
        const __half h = __float2half_rn(r);
        pc[j] = __half_as_ushort(h);
        back = __half2float(h);
      }
      if (!(fabsf(back) < INFINITY)) break;  // beyond the 16-bit range: the row scores +inf and is never a candidate
      r = __fsub_rn(r, back);
    }
  }
  uint4* dst = reinterpret_cast<uint4*>(ext + row * EXT_K);
  const int sw = int(row >> 2) & 1;
  dst[sw] = make_uint4(uint32_t(pc[0]) | (uint32_t(pc[1]) << 16), uint32_t(pc[2]), 0u, 0u);
  dst[sw ^ 1] = make_uint4(0u, 0u, 0u, 0u);
}

__global__ void fill_f32_kernel(float* p, size_t n, float v) {
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) p[i] = v;
}

__global__ void init_stats_kernel(RangeStats* st) {
  st->min_v = INFINITY;
  st->max_v = -INFINITY;
  st->max_norm2 = 0.f;
  st->not_integer = 0;
  st->not_finite = 0;
}

// what a search begins with: the queries' statistics, no query to re-run, no error, no query known to miss the 8-bit form
__global__ void init_search_kernel(RangeStats* qst, unsigned int* words) {
  qst->min_v = INFINITY;
  qst->max_v = -INFINITY;
  qst->max_norm2 = 0.f;
  qst->not_integer = 0;
  qst->not_finite = 0;
  for (int i = 0; i < 3; ++i) words[i] = 0u;
}

// ------------------------------------------------------------------------------------------------
// A query's bound and the error bound of its scores, by a warp per query.
//
// The bound is the R-th smallest of the group minima the sample pass left (+inf where there are fewer), which that many
// sampled rows do not exceed, plus the error bound: the re-rank's certificate asks for the k-th distance to lie below the
// bound by that much, and a query that misses it costs a scan of the base (2,049 queries of 200,003 x 384: without it one
// query in 2,000 did at a sample of 1 in 16, and several at 1 in 8).  Each lane keeps the four smallest of its share: where
// a lane holds more than four of the R smallest the bound is a little looser.  Bound by reading the minima from L2.
// With the R best scores of the sample kept in registers by the epilogue, as it was, every chunk of 32 columns had an
// insertion in some row: 251 us for 31,250 rows x 10,000 queries, 52 and 16 now; 1,000 queries at 100k x 128 38, 12 and 10.
struct TauParams {
  const float* smin;
  int ld, groups, nq, R;
  const float* queries;    // nq x pd; rows from `real` on are padding
  int real, pd, Kp, is_l2, bf16;
  const float* qnorm2;
  const RangeStats* bst;   // base statistics
  const RangeStats* qst;   // query statistics
  const unsigned int* q8_bad;
  float* tau;
  float* eps;
};
__global__ void __launch_bounds__(256) sample_tau_kernel(TauParams p) {
  const int q = blockIdx.x * int(blockDim.x >> 5) + int(threadIdx.x >> 5), lane = lane_id();
  if (q >= p.nq) return;
  const float* src = p.smin + size_t(q) * p.ld;
  float best[4] = {INFINITY, INFINITY, INFINITY, INFINITY};
#pragma unroll 4
  for (int i = lane; i < p.groups; i += 32) {
    float v = src[i];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const float lo = fminf(best[t], v);
      v = fmaxf(best[t], v);
      best[t] = lo;
    }
  }
  float eps = 0.f;
  if (q < p.real && !(p.q8_bad && *p.q8_bad == 0u)) {  // (8-bit scores are exact)
    const float* query = p.queries + size_t(q) * p.pd;
    float s = 0.f, qmax = 0.f;
    bool fin = true;
    for (int c = lane; c < p.pd; c += 32) {
      const float x = query[c];
      s = __fmaf_rn(x, x, s);
      qmax = fmaxf(qmax, fabsf(x));
      fin = fin && fabsf(x) <= 3.0e38f;  // false for inf and NaN
    }
    for (int o = 16; o > 0; o >>= 1) {
      s += __shfl_xor_sync(FV_FULL, s, o);
      qmax = fmaxf(qmax, __shfl_xor_sync(FV_FULL, qmax, o));
    }
    fin = __all_sync(FV_FULL, fin);
    // exact-arithmetic regime: integer-valued inputs small enough that every product, partial sum and
    // distance is an integer below 2^24 in both the tensor-core score and the reference's fp32 chain
    const float lo = fminf(p.bst->min_v, p.qst->min_v), hi = fmaxf(p.bst->max_v, p.qst->max_v);
    const float mabs = fmaxf(fabsf(lo), fabsf(hi)), range = hi - lo;
    // the accumulator starts at ||b||^2 <= Kp mabs^2 and then takes the terms -2 q_i b_i: it stays within
    // [-2 Kp mabs^2, Kp mabs^2 + 2 Kp |lo hi|], the upper end only when the values take both signs
    const float negprod = (lo < 0.f && hi > 0.f) ? -lo * hi : 0.f;
    const float kf = float(p.Kp);
    const bool exact_regime = !p.bst->not_integer && !p.qst->not_integer && !p.bst->not_finite && !p.qst->not_finite &&
                              mabs <= (p.bf16 ? 256.f : 2048.f) && kf * mabs * mabs <= 8388608.f &&
                              kf * (mabs * mabs + 2.f * negprod) <= 16777216.f && kf * range * range < 16777216.f;
    // error bound of a score against the reference distance (minus ||q||^2 for L2) outside that regime
    const float u16 = p.bf16 ? 0.00390625f : 0.00048828125f;
    const float qnorm = sqrtf(p.is_l2 ? p.qnorm2[q] : s), bn = sqrtf(p.bst->max_norm2);
    const float e_dot = (2.f * u16 * (1.f + u16) + kf * 4.7683716e-7f + kf * 1.1920929e-7f) * qnorm * bn +
                        5.9604645e-8f * sqrtf(kf) * (qnorm + bn);
    // L2: the norm is added inside the MMA (its split loses < 2^-24 of the largest norm, the accumulation
    // about 2^-21 per step of a partial sum that now includes it), then the reference chain's own rounding
    const float e_norm = (kf + 16.f) * 4.7683716e-7f * bn * bn + 1.1920929e-7f * bn * bn;
    eps = p.is_l2 ? 2.f * e_dot + e_norm + kf * 2.3841858e-7f * (qnorm * qnorm + bn * bn) * 2.f : e_dot;
    eps = exact_regime ? 0.f : eps * 1.01f + 1e-30f;
    // The query operand of the GEMM is this row times -2 (L2) or -1 in the 16-bit type.  A component that leaves that
    // type's range (fp16: 65504) turns every score of the query into +-inf or NaN, so no row is a candidate and the
    // reasoning of the certificate ("a row that is not a candidate scores above the bound") says nothing: such a query is
    // never certified and goes to the full-precision scan, which returns the reference's k finite neighbours.
    const bool in_range = fin && (p.bf16 ? qmax <= 1.0e38f : qmax * (p.is_l2 ? 2.f : 1.f) <= 65504.f);
    if (!in_range) eps = INFINITY;
  }
  uint32_t w = 0;
  for (int i = 0; i < p.R; ++i) {
    const uint32_t head = order_bits(best[0]);
    w = __reduce_min_sync(FV_FULL, head);
    const int owner = __ffs(__ballot_sync(FV_FULL, head == w)) - 1;
    if (lane == owner) {
#pragma unroll
      for (int t = 0; t < 3; ++t) best[t] = best[t + 1];
      best[3] = INFINITY;
    }
  }
  if (lane == 0) {
    const float t = order_bits_to_float(w);
    p.tau[q] = eps < INFINITY ? __fadd_ru(t, eps) : t;
    p.eps[q] = eps;
  }
}

// ------------------------------------------------------------------------------------------------
// Exact re-rank and certification: one warp per query.
struct RerankParams {
  const float* tau;       // the bound every candidate was tested against
  const u64* cbuf;        // candidates of the main pass: [grid * segmax][128 * MH][4][ccap]
  const unsigned int* ccnt;
  PassShapes shapes;      // main pass
  const float* const8;    // 8-bit operands: the queries' constants, the parity of every row's t
  const uint8_t* parity8;
  const float* rows;      // n x pd fp32
  const float* queries;   // nq x pd fp32
  const float* qnorm2;    // nq (0 for inner product)
  const float* eps;       // nq: error bound of a score
  int n, nq, pd, k;
  int wpq;                // warps per query: 1, 2, 4 or 8
  uint32_t id_base;
  u64* out_keys;          // nq x k
  uint32_t* retry_ids;    // queries that did not certify
  unsigned int* retry_count;
};

// Bound by gathering the candidates' rows (56 to 112 per query at k = 10, 420 at k = 100): eight rows at a time, four
// lanes to a row (group_distance), the result list in registers (32 * KR places).  With four rows of eight lanes staged
// through shared memory and the list there too 10,000 queries at 1M x 128 took 274 us (201 this way, with 160 candidates
// each).  Bytes have no rows to gather: 48 us.  A batch that leaves
// the SMs short of warps and has long results is given `wpq` warps per query, which share its candidates and merge
// their lists: 501 queries with k = 100 over 50,001 x 100, the whole search 455 us in the old form, 315 with a warp per
// query, 217 with eight.
template <bool IS_L2, int KR, bool MULTI>  // MULTI: several warps per query
__global__ void __launch_bounds__(256, KR == 1 ? 3 : 2) rerank_kernel(RerankParams p) {
  const int W = blockDim.x >> 5, w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = MULTI ? w % p.wpq : 0;  // which share of the query's candidates this warp takes
  const size_t q_own = MULTI ? size_t(blockIdx.x) * (W / p.wpq) + w / p.wpq : size_t(blockIdx.x) * W + w;
  if (!MULTI && q_own >= size_t(p.nq)) return;
  // (MULTI: a warp beyond the last query works on the last one and writes nothing: all warps meet at the barriers below)
  const size_t q = MULTI ? min(q_own, size_t(p.nq) - 1) : q_own;
  float* sq = reinterpret_cast<float*>(dyn_smem()) + size_t(w) * p.pd;
  for (int c = lane; c < p.pd; c += 32) sq[c] = p.queries[q * size_t(p.pd) + c];
  TopList<KR> top;
  top.init(p.k);
  __syncwarp();

  // how far a score can be from the reference distance (minus ||q||^2 for L2): 0 in the exact-arithmetic regime, inf for
  // a query that cannot be scored
  const float eps = p.eps[q];
  const bool exact_regime = eps == 0.f, q_in_range = eps < INFINITY;
  const float qn2 = p.qnorm2[q];

  const bool is8 = IS_L2 && p.shapes.is8();
  const PassShape& sh = p.shapes.taken();
  const int rows_per_tile = 128 * sh.MH;
  const int cta_tile = int(q / rows_per_tile), r = int(q % rows_per_tile);  // a CTA's share of a query tile
  const int mt = cta_tile / sh.ctas, rank = cta_tile % sh.ctas;
  const float const8 = is8 ? p.const8[q] : 0.f;
  // every row whose score is below tau is in the buffer; every other row scores >= tau
  const float tau = p.tau[q];
  bool overflow = false;
  bool mismatch = false;  // exact regime only: a score that is not the exact distance
  u64 bound = FV_EMPTY_KEY;
  const int ccap = sh.ccap;
  // The candidates of this query sit in four short lists per chunk.  32 chunks at a time: each lane looks up the four
  // counts of one, a prefix sum lines the entries up, and the warp walks them 32 per step (a lane finds the chunk of its
  // entry by bisection over the prefix sums), so every step computes 32 exact distances.
  int taken = 0;  // runs of eight candidates seen so far, the same in all warps of the query
  for (int l0 = 0; l0 < sh.parts; l0 += 32) {
    const int l = l0 + lane;
    unsigned int cnt = 0;
    u64 ends = 0;  // where the first three lists end, 16 bits each
    unsigned long long slot = 0;
    if (l < sh.parts) {
      const int g = l * sh.MT + mt;
      const int c = g % sh.grid * sh.ctas + rank, seg_local = g / sh.grid;
      slot = (size_t(c) * sh.segmax + seg_local) * rows_per_tile + r;
      const uint4 c4 = reinterpret_cast<const uint4*>(p.ccnt)[slot];
      if (max(max(c4.x, c4.y), max(c4.z, c4.w)) > unsigned(ccap)) overflow = true;
      const unsigned int e0 = min(c4.x, unsigned(ccap)), e1 = e0 + min(c4.y, unsigned(ccap)), e2 = e1 + min(c4.z, unsigned(ccap));
      cnt = e2 + min(c4.w, unsigned(ccap));
      ends = u64(e0) | (u64(e1) << 16) | (u64(e2) << 32);
    }
    unsigned int pre = cnt;  // inclusive prefix sum
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int v = __shfl_up_sync(FV_FULL, pre, o);
      if (lane >= o) pre += v;
    }
    const unsigned int total = __shfl_sync(FV_FULL, pre, 31);
    for (unsigned int t0 = 0; t0 < total; t0 += 32) {
      const unsigned int x = t0 + lane;
      int j = 0;  // chunks whose entries all come before entry x
#pragma unroll
      for (int step = 16; step > 0; step >>= 1) {
        const unsigned int pv = __shfl_sync(FV_FULL, pre, j + step - 1);
        if (pv <= x) j += step;
      }
      const unsigned int pj = __shfl_sync(FV_FULL, pre, j), cj = __shfl_sync(FV_FULL, cnt, j);
      const unsigned long long sj = __shfl_sync(FV_FULL, slot, j);
      const u64 ej = __shfl_sync(FV_FULL, ends, j);
      u64 ck = 0;
      uint32_t id = 0;
      bool have = false;
      if (x < total) {
        const unsigned int at = x - (pj - cj), e0 = unsigned(ej) & 0xFFFFu, e1 = unsigned(ej >> 16) & 0xFFFFu, e2 = unsigned(ej >> 32);
        const int li = (at >= e0) + (at >= e1) + (at >= e2);
        ck = p.cbuf[(sj * 4 + li) * size_t(ccap) + (at - (li == 0 ? 0u : li == 1 ? e0 : li == 2 ? e1 : e2))];
        id = key_id(ck);
        have = id < uint32_t(p.n);
        if (!have) mismatch = true;  // a padded row can only get here through a non-finite score
      }
      if (is8) {  // the score is the distance but for the query's constant and one bit
        if (MULTI && ((taken++) & (p.wpq - 1)) != sub) continue;
        const float d = have ? 2.f * key_distance(ck) + float(p.parity8[id]) + const8 : INFINITY;
        top.offer(have ? make_key(d, id + p.id_base) : FV_EMPTY_KEY, bound);
        continue;
      }
      for (int s = 0; s < 32 && t0 + s < total; s += 8) {
        if (MULTI && ((taken++) & (p.wpq - 1)) != sub) continue;  // runs of eight are dealt in turn
        const int from = s + (lane >> 2);
        const uint32_t rid = __shfl_sync(FV_FULL, id, from);
        const bool rhave = __shfl_sync(FV_FULL, int(have), from) != 0;
        const float score = __shfl_sync(FV_FULL, key_distance(ck), from);
        const float d = group_distance<IS_L2, 4>(sq, p.rows + size_t(rhave ? rid : 0u) * p.pd, p.pd);
        if (rhave && exact_regime && d != score + qn2) mismatch = true;
        const bool in = rhave && (lane & 3) == 0 && d < INFINITY;
        top.offer(in ? make_key(d, rid + p.id_base) : FV_EMPTY_KEY, bound);
      }
    }
  }
  mismatch = __any_sync(FV_FULL, mismatch);
  overflow = __any_sync(FV_FULL, overflow);
  if (MULTI) {
    u64* lists = reinterpret_cast<u64*>(reinterpret_cast<float*>(dyn_smem()) + size_t(W) * p.pd) + size_t(w) * 32 * KR;  // 16-byte aligned: pd is a multiple of 8
    __shared__ int bad[8];
    if (lane == 0) bad[w] = mismatch ? 1 : 0;
    for (int step = 1; step < p.wpq; step <<= 1) {
      __syncthreads();
      if ((sub & (2 * step - 1)) == step) top.store(lists, p.k);
      __syncthreads();
      if ((sub & (2 * step - 1)) == 0) {
        u64 c[KR];
        TopList<KR>::load(c, lists + size_t(step) * 32 * KR, p.k);
        top.merge(c);
      }
    }
    for (int i = 0; i < p.wpq; ++i) mismatch = mismatch || bad[w - sub + i];
  }
  if (sub != 0 || q_own >= size_t(p.nq)) return;
  const u64 kth = top.last();
  bool certified;
  if (overflow || mismatch || !(is8 || q_in_range) || !(tau == tau)) {
    certified = false;
  } else if (tau == INFINITY) {
    certified = true;  // every row with a finite score was a candidate
  } else if (is8) {
    certified = kth != FV_EMPTY_KEY && key_distance(kth) < 2.f * tau + const8;  // every other row's distance is at least that
  } else {
    // the k-th result must be provably nearer than anything that was not a candidate
    certified = kth != FV_EMPTY_KEY && (key_distance(kth) - qn2) + eps < tau;
  }
#pragma unroll
  for (int r = 0; r < KR; ++r) {
    const int e = r * 32 + lane - (32 * KR - p.k);
    if (e >= 0) p.out_keys[q * size_t(p.k) + e] = top.e[r];
  }
  if (!certified && lane == 0) {
    const unsigned int slot = atomicAdd(p.retry_count, 1u);
    p.retry_ids[slot] = uint32_t(q);
  }
}

// Rows of the strided sample: sample row i is base row floor(i * n / ns).  They are stored with the multiples of 16
// first, then the other multiples of 8, 4 and 2, then the odd ones: the first ceil(ns / 2^j) rows are the sample of
// every 2^j-th of them (j <= 4), for searches that want a coarser one.  Within each of these runs the order goes round by
// steps of about 0.618 of its length, so that rows side by side, whose minimum stands for them all, come from all over the
// base: in a base stored cluster by cluster neighbours in the base are neighbours in space.
static constexpr int SAMPLE_LEVELS = 4;
__host__ __device__ __forceinline__ size_t sample_prefix(size_t ns, int j) { return (ns + (size_t(1) << j) - 1) >> j; }
struct SampleOrder {
  size_t ns;
  size_t step[SAMPLE_LEVELS + 1];  // of the run of the multiples of 2^j that no coarser run holds
};
static SampleOrder sample_order(size_t ns) {
  SampleOrder o{ns, {}};
  for (int j = 0; j <= SAMPLE_LEVELS; ++j) {
    const size_t len = sample_prefix(ns, j) - (j < SAMPLE_LEVELS ? sample_prefix(ns, j + 1) : 0);
    size_t s = std::max<size_t>(1, size_t(double(len) * 0.6180339887));
    while (std::gcd(s, len) > 1) ++s;  // (len 0 has no rows; len 1: any step)
    o.step[j] = s;
  }
  return o;
}
__device__ __forceinline__ size_t sample_row_at(size_t slot, const SampleOrder& o) {  // the sample row stored in `slot`
  const size_t coarse = sample_prefix(o.ns, SAMPLE_LEVELS);
  if (slot < coarse) return (slot * o.step[SAMPLE_LEVELS] % coarse) << SAMPLE_LEVELS;
  int j = SAMPLE_LEVELS - 1;
  while (slot >= sample_prefix(o.ns, j)) --j;
  const size_t first = sample_prefix(o.ns, j + 1), len = sample_prefix(o.ns, j) - first;
  return (((slot - first) * o.step[j] % len) << (j + 1)) + (size_t(1) << j);
}

// base8 (bases with 8-bit operands): those and their norm bytes too, up to row nspad of the latter
__global__ void gather_sample_kernel(const uint16_t* __restrict__ half, const float* __restrict__ norm2, size_t n, int Kp,
                                     SampleOrder order, uint16_t* __restrict__ samp, float* __restrict__ snorm,
                                     const uint8_t* __restrict__ base8, const uint8_t* __restrict__ ext8, int Kp8, size_t nspad,
                                     uint8_t* __restrict__ samp8, uint8_t* __restrict__ samp_ext8) {
  const int lane = threadIdx.x & 31;
  const size_t i = blockIdx.x * size_t(blockDim.x >> 5) + (threadIdx.x >> 5);
  const auto swap8 = [](size_t row) { return (int(row >> 2) & 1) << 4; };  // the image's halves trade places in rows 4..7 of 8
  const size_t ns = order.ns;
  if (i >= ns) {
    if (base8 && i < nspad) samp_ext8[i * 32 + lane] = uint8_t((lane & 15) == 0 ? 0 : 127);  // beyond the sample: a large score
    return;
  }
  const size_t src = size_t((unsigned long long)sample_row_at(i, order) * n / ns);
  const uint4* a = reinterpret_cast<const uint4*>(half + src * size_t(Kp));
  uint4* b = reinterpret_cast<uint4*>(samp + i * size_t(Kp));
  for (int c = lane; c < Kp / 8; c += 32) b[c] = a[c];
  if (lane == 0) snorm[i] = norm2[src];
  if (base8) {
    const uint4* a8 = reinterpret_cast<const uint4*>(base8 + src * size_t(Kp8));
    uint4* b8 = reinterpret_cast<uint4*>(samp8 + i * size_t(Kp8));
    for (int c = lane; c < Kp8 / 16; c += 32) b8[c] = a8[c];
    samp_ext8[i * 32 + (lane ^ swap8(i))] = ext8[src * 32 + (lane ^ swap8(src))];
  }
}

__global__ void scatter_keys_kernel(const u64* __restrict__ src, const uint32_t* __restrict__ qids, size_t nsub, int L,
                                    u64* __restrict__ dst) {
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < nsub * L; i += size_t(gridDim.x) * blockDim.x) {
    const size_t s = i / L;
    dst[size_t(qids[s]) * L + (i - s * L)] = src[i];
  }
}

// ------------------------------------------------------------------------------------------------
// host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// rows x K matrix of operands, boxes of `box_rows` rows x 128 bytes, 128-byte swizzle
static CUtensorMapDataType type16(bool bf16) { return bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16; }
static int make_tmap(CUtensorMap* map, CUtensorMapDataType type, void* ptr, size_t rows, int K, int box_rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail(FV_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  const int size = type == CU_TENSOR_MAP_DATA_TYPE_UINT8 ? 1 : 2;
  cuuint64_t gdim[2] = {cuuint64_t(K), cuuint64_t(rows)};
  cuuint64_t gstride[1] = {cuuint64_t(K) * size};
  cuuint32_t box[2] = {cuuint32_t(128 / size), cuuint32_t(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, type, 2, ptr, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(FV_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string(int(r)));
  return FV_OK;
}

// the norm step's bytes as rows of 128, boxes of 32 rows: 128 rows' worth, as they lie in memory
static int make_norm_tmap(CUtensorMap* map, void* ptr, size_t rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return fail(FV_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t gdim[2] = {128, cuuint64_t(rows / 4)};
  cuuint64_t gstride[1] = {128};
  cuuint32_t box[2] = {128, 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, ptr, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(FV_ERR_CUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string(int(r)));
  return FV_OK;
}

struct TcSide {
  int pd = 0, Kp = 0;
  bool bf16 = false;
  size_t n = 0;            // rows converted
  DevBuf half;             // n_cap x Kp 16-bit
  DevBuf norm2;            // padded to 256, +inf beyond n
  DevBuf stats;            // RangeStats (base), RangeStats (queries), retry counter, error word
  size_t ns = 0;           // rows of the strided sample
  int every = 32;          // 1 row in `every` is sampled
  DevBuf samp, samp_norm2; // the sample's operand rows and norms (+inf padded)
  DevBuf ext, samp_ext;    // norm pieces of the base rows and of the sample (padded like the norms), 32 B per row
  bool i8 = false;         // the base has 8-bit operands too
  int Kp8 = 0;             // their row length: pd rounded up to 128
  float lo8 = 0.f;         // the value they store as -128
  float refused_lo8 = NAN; // above this value some row is too far from the middle: rows only come, so no add need look again
  DevBuf rows8, ext8, parity8, samp8, samp_ext8;
  int ext_e = 0;           // the pieces hold ||b||^2 / 2^ext_e
  bool ext_valid = false;
  RangeStats h_stats{};
  // The maps of the base, the sample and their norm steps, by operand form and by CTAs per tile: made by the first search
  // that needs them (3 us each; ten of them in every call were a sixth of 1,000 queries at 100k x 128).
  struct Maps {
    bool valid = false;
    CUtensorMap base, sample, base_norm, sample_norm;
  } maps[2][2];
};

void tc_free(TcSide* tc) { delete tc; }

// the words behind the two RangeStats in `stats`
enum { W_RETRY = 0, W_ERR = 1, W_Q8_BAD = 2, W_TOO_LARGE = 3 };
static unsigned int* side_words(TcSide* tc) { return reinterpret_cast<unsigned int*>(tc->stats.as<RangeStats>() + 2); }

static inline int round_up(int x, int m) { return (x + m - 1) / m * m; }

struct Queries8 {  // where convert puts the 8-bit form of queries
  uint8_t* dst = nullptr;
  int Kp8 = 0;
  float lo8 = 0.f;
  float* const8 = nullptr;
  unsigned int* bad = nullptr;
};

static int convert(fv_ctx* ctx, bool bf16, const float* d_src, size_t n, int pd, int Kp, uint16_t* dst, float* norm2,
                   bool is_l2, float mul, RangeStats* st, const Queries8& q8 = {}) {
  if (n == 0) return FV_OK;
  const int wpb = 8;
  const unsigned blocks = unsigned((n + wpb - 1) / wpb);
  if (bf16)
    convert_rows_kernel<true><<<blocks, wpb * 32, 0, ctx->stream>>>(d_src, n, pd, Kp, dst, norm2, is_l2 ? 1 : 0, mul, st, q8.dst,
                                            q8.Kp8, q8.lo8, q8.const8, q8.bad);
  else
    convert_rows_kernel<false><<<blocks, wpb * 32, 0, ctx->stream>>>(d_src, n, pd, Kp, dst, norm2, is_l2 ? 1 : 0, mul, st, q8.dst,
                                             q8.Kp8, q8.lo8, q8.const8, q8.bad);
  ctx->stats.launches++;
  FV_CUDA(cudaGetLastError());
  return FV_OK;
}

static int split_norms(fv_ctx* ctx, bool bf16, const float* norm2, size_t first, size_t count, int e, uint16_t* ext) {
  if (count == 0) return FV_OK;
  const float inv = std::ldexp(1.f, -e);
  const unsigned blocks = unsigned((count + 255) / 256);
  if (bf16) split_norms_kernel<true><<<blocks, 256, 0, ctx->stream>>>(norm2, first, count, inv, ext);
  else split_norms_kernel<false><<<blocks, 256, 0, ctx->stream>>>(norm2, first, count, inv, ext);
  ctx->stats.launches++;
  FV_CUDA(cudaGetLastError());
  return FV_OK;
}

// The 8-bit form of rows n_old .. total, or of all of them where the rows before have none or another `lo`, and room for the
// sample's; none for a base that does not qualify, nor where the device has no room for it: the 16-bit form does alone.
// Costs 128 ceil(pd / 128) + 33 bytes per row and the sample's, and time: 100,000 x 128 in one add from the device 1.6 -> 2.7 ms, mostly the allocations.
static int append8(fv_ctx* ctx, TcSide* tc, const float* all_rows, size_t n_old, size_t total, size_t npad, size_t nspad) {
  const RangeStats& st = tc->h_stats;
  const float lo = st.min_v >= 0.f && st.max_v <= 255.f ? 0.f : st.min_v >= -128.f && st.max_v <= 127.f ? -128.f : st.min_v;
  bool fits = !st.not_integer && !st.not_finite && tc->pd <= I8_MAX_PD && std::fabs(lo) <= 65536.f && st.max_v - lo <= 255.f &&
              lo != tc->refused_lo8;
  const size_t first = tc->i8 && tc->lo8 == lo ? n_old : 0;
  if (fits) {
    tc->Kp8 = round_up(tc->pd, 2 * KBLK);
    auto room = [&]() -> int {
      FV_TRY(tc->rows8.grow(total * size_t(tc->Kp8), first * size_t(tc->Kp8), ctx->stream));
      FV_TRY(tc->ext8.grow(npad * 32, first * 32, ctx->stream));
      FV_TRY(tc->parity8.grow(npad, first, ctx->stream));
      FV_TRY(tc->samp8.reserve(tc->ns * size_t(tc->Kp8)));
      return tc->samp_ext8.reserve(nspad * 32);
    };
    const int got = room();
    if (got != FV_OK && got != FV_ERR_NOMEM) return got;
    fits = got == FV_OK;
  }
  if (fits) {
    unsigned int* too_large = side_words(tc) + W_TOO_LARGE;
    FV_CUDA(cudaMemsetAsync(too_large, 0, sizeof(unsigned int), ctx->stream));
    convert8_rows_kernel<<<unsigned((npad - first + 7) / 8), 256, 0, ctx->stream>>>(
        all_rows, first, total, npad, tc->pd, tc->Kp8, lo, tc->rows8.as<uint8_t>(), tc->ext8.as<uint8_t>(),
        tc->parity8.as<uint8_t>(), too_large);
    ctx->stats.launches++;
    FV_CUDA(cudaGetLastError());
    unsigned int h_large = 0;
    FV_CUDA(cudaMemcpyAsync(&h_large, too_large, sizeof(h_large), cudaMemcpyDeviceToHost, ctx->stream));
    FV_CUDA(cudaStreamSynchronize(ctx->stream));
    fits = h_large == 0;
    if (!fits) tc->refused_lo8 = lo;
  }
  tc->i8 = fits;
  tc->lo8 = lo;
  if (!fits)
    for (DevBuf* b : {&tc->rows8, &tc->ext8, &tc->parity8, &tc->samp8, &tc->samp_ext8}) b->release();
  return FV_OK;
}

// Called by FlatIndex::add after the fp32 rows are in place.  d_rows_new points at the new rows.
int tc_append(fv_ctx* ctx, TcSide** ptc, int metric, const float* d_rows_new, size_t n_old, size_t n_new, int pd) {
  const int Kp = round_up(pd, KBLK);
  if (Kp > 384) return FV_OK;  // beyond the tilings of this kernel: such an index uses the scan only
  if (!*ptc) {
    *ptc = new TcSide();
    (*ptc)->pd = pd;
    (*ptc)->Kp = Kp;
  }
  TcSide* tc = *ptc;
  // before any buffer moves: should this call fail halfway, the rows of before are searched on, where they lie then
  for (auto& form : tc->maps)
    for (TcSide::Maps& m : form) m.valid = false;
  const size_t total = n_old + n_new;
  if (!tc->stats.p) {
    FV_TRY(tc->stats.reserve(256));
    init_stats_kernel<<<1, 1, 0, ctx->stream>>>(tc->stats.as<RangeStats>());
    FV_CUDA(cudaGetLastError());
  }
  FV_TRY(tc->half.grow(total * size_t(Kp) * 2 + 1024, n_old * size_t(Kp) * 2, ctx->stream));
  const size_t npad = (total + TILE_N - 1) / TILE_N * TILE_N + TILE_N;
  FV_TRY(tc->norm2.grow(npad * sizeof(float), n_old * sizeof(float), ctx->stream));
  // pick the operand type from the range of the NEW rows first (fp16 unless the values do not fit)
  DevBuf tmp_stats;
  FV_TRY(tmp_stats.reserve(sizeof(RangeStats)));
  init_stats_kernel<<<1, 1, 0, ctx->stream>>>(tmp_stats.as<RangeStats>());
  FV_CUDA(cudaGetLastError());
  uint16_t* dst = tc->half.as<uint16_t>() + n_old * size_t(Kp);
  float* nrm = tc->norm2.as<float>() + n_old;
  FV_TRY(convert(ctx, tc->bf16, d_rows_new, n_new, pd, Kp, dst, nrm, metric == FV_L2, 1.f, tmp_stats.as<RangeStats>()));
  RangeStats hs;
  FV_CUDA(cudaMemcpyAsync(&hs, tmp_stats.p, sizeof(hs), cudaMemcpyDeviceToHost, ctx->stream));
  FV_CUDA(cudaStreamSynchronize(ctx->stream));
  const float mabs = std::max(std::fabs(hs.min_v), std::fabs(hs.max_v));
  // fp16 also needs the largest squared norm within reach of the norm step: 2^15 (query side) x 2^15 (pieces)
  const float max_n2 = std::max(hs.max_norm2, tc->n ? tc->h_stats.max_norm2 : 0.f);
  const bool need_bf16 = !(mabs <= 32768.f) || !(max_n2 <= 1073741824.f);
  bool resplit = false;
  if (need_bf16 && !tc->bf16) {
    resplit = true;
    // values beyond the fp16 range: the whole operand copy becomes bf16.  The caller passes the new rows
    // only, so the old ones are re-read from the fp32 matrix that precedes them in the same allocation.
    tc->bf16 = true;
    const float* all_rows = d_rows_new - n_old * size_t(pd);
    init_stats_kernel<<<1, 1, 0, ctx->stream>>>(tc->stats.as<RangeStats>());
    FV_TRY(convert(ctx, true, all_rows, total, pd, Kp, tc->half.as<uint16_t>(), tc->norm2.as<float>(), metric == FV_L2,
                   1.f, tc->stats.as<RangeStats>()));
    FV_CUDA(cudaMemcpyAsync(&tc->h_stats, tc->stats.p, sizeof(RangeStats), cudaMemcpyDeviceToHost, ctx->stream));
    FV_CUDA(cudaStreamSynchronize(ctx->stream));
  } else {
    // fold the new rows' statistics into the running ones
    FV_CUDA(cudaMemcpyAsync(&tc->h_stats, tc->stats.p, sizeof(RangeStats), cudaMemcpyDeviceToHost, ctx->stream));
    FV_CUDA(cudaStreamSynchronize(ctx->stream));
    RangeStats m = tc->h_stats;
    m.min_v = std::min(m.min_v, hs.min_v);
    m.max_v = std::max(m.max_v, hs.max_v);
    m.max_norm2 = std::max(m.max_norm2, hs.max_norm2);
    m.not_integer |= hs.not_integer;
    m.not_finite |= hs.not_finite;
    FV_CUDA(cudaMemcpyAsync(tc->stats.p, &m, sizeof(m), cudaMemcpyHostToDevice, ctx->stream));
    FV_CUDA(cudaStreamSynchronize(ctx->stream));
    tc->h_stats = m;
  }
  fill_f32_kernel<<<8, 256, 0, ctx->stream>>>(tc->norm2.as<float>() + total, npad - total, INFINITY);
  ctx->stats.launches++;
  FV_CUDA(cudaGetLastError());
  tc->n = total;
  if (metric == FV_L2) {
    // norm pieces: ||b||^2 / 2^e with the largest quotient in (128, 256] when e was chosen, re-split when it outgrows 2^15
    FV_TRY(tc->ext.grow(npad * size_t(EXT_K) * 2, n_old * size_t(EXT_K) * 2, ctx->stream));
    int e = tc->ext_e;
    const float mx = tc->h_stats.max_norm2;
    if (tc->bf16) {
      e = 0;
      if (!tc->ext_valid || tc->ext_e != 0) resplit = true;
    } else if (!tc->ext_valid || !(std::ldexp(mx, -e) <= 32768.f)) {
      int ex = 0;
      if (mx > 0.f && mx < INFINITY) std::frexp(mx, &ex);  // mx in [2^(ex-1), 2^ex)
      e = std::min(15, std::max(-14, ex - 8));
      resplit = true;
    }
    tc->ext_e = e;
    tc->ext_valid = true;
    const size_t first = resplit ? 0 : n_old;
    FV_TRY(split_norms(ctx, tc->bf16, tc->norm2.as<float>(), first, npad - first, e, tc->ext.as<uint16_t>()));
  }
  // the strided sample the threshold of the main pass is estimated from
  tc->every = pick_sample_every(total);
  tc->ns = std::max<size_t>(SAMPLE_R_MAX, total / size_t(tc->every));
  const size_t nspad = (tc->ns + TILE_N - 1) / TILE_N * TILE_N + TILE_N;
  FV_TRY(tc->samp.reserve(tc->ns * size_t(Kp) * 2 + 1024));
  FV_TRY(tc->samp_norm2.reserve(nspad * sizeof(float)));
  if (metric == FV_L2) {
    FV_TRY(tc->samp_ext.reserve(nspad * size_t(EXT_K) * 2));
    FV_TRY(append8(ctx, tc, d_rows_new - n_old * size_t(pd), n_old, total, npad, nspad));  // (the last to ask for room)
  }
  gather_sample_kernel<<<unsigned((nspad + 7) / 8), 256, 0, ctx->stream>>>(
      tc->half.as<uint16_t>(), tc->norm2.as<float>(), total, Kp, sample_order(tc->ns), tc->samp.as<uint16_t>(), tc->samp_norm2.as<float>(),
      tc->i8 ? tc->rows8.as<uint8_t>() : nullptr, tc->ext8.as<uint8_t>(), tc->Kp8, nspad, tc->samp8.as<uint8_t>(),
      tc->samp_ext8.as<uint8_t>());
  fill_f32_kernel<<<8, 256, 0, ctx->stream>>>(tc->samp_norm2.as<float>() + tc->ns, nspad - tc->ns, INFINITY);
  ctx->stats.launches += 2;
  FV_CUDA(cudaGetLastError());
  if (metric == FV_L2)
    FV_TRY(split_norms(ctx, tc->bf16, tc->samp_norm2.as<float>(), 0, nspad, tc->ext_e, tc->samp_ext.as<uint16_t>()));
  return FV_OK;
}

// Results of more than 32 of 4,096 rows, which the scan of every key (exact_scan) serves too: both times in microseconds,
// fitted to calls at 32, 128 and 384 dimensions.  Here / there: 33 results of 65 queries x 128 136 / 112, of 300 152 / 166,
// of 2,000 207 / 607; 128 results 177 / 112, 202 / 166, 420 / 607; 33 of 300 x 384 147 / 240; 128 of 256 x 32 150 / 112.
static bool tc_beats_dense(size_t nq, int k, int Kp) {
  const double here = 115.0 + 0.45 * k + double(nq) * k * (0.0004 + 3e-6 * Kp), there = 65.0 + double(nq) * (0.2 + 0.001 * Kp);
  return here < there;
}

bool tc_usable(const TcSide* tc, size_t n, size_t nq, int k) {
  return tc && tc->n == n && k <= TC_MAX_K && n >= 4096 && n <= 0x7FFFFF00ull &&
         (k <= 32 || n > 4096 || tc_beats_dense(nq, k, tc->Kp));
}

// One launch of the GEMM kernel over `rows` operand rows.
//
// Work split.  A unit is (query tile, 256 base rows).  Each query tile's row of units is cut into `parts` chunks of
// `cpn` units; chunk g = part * MT + query tile goes to CTA g % grid as that CTA's (g / grid)-th segment.  The CTAs
// that run side by side therefore hold DIFFERENT query tiles but walk the SAME base tiles at about the same time:
// a base tile is fetched from HBM once and served to the other query tiles from L2 (with a contiguous split of the
// units the 16-bit copy of the base was streamed from HBM once per query tile).  `parts` is the value that minimises
// waves x (chunk length + a fixed cost per chunk).
struct Tiling {
  int KB, last_steps, MH, ctas, MT, NT, grid, segmax, nstage, cpn, parts, nchunks, ext_ring;
  size_t smem;
  size_t nlists;  // candidate lists of the pass, `ccap` slots each
  int ccap;
};

// `row_bytes`: bytes of an operand row that hold data
static int make_tiling(fv_ctx* ctx, int row_bytes, size_t nq, size_t rows, Tiling* t, int force_mh = 0, bool pairs = false) {
  t->KB = (row_bytes + 127) / 128;
  t->last_steps = (row_bytes - (t->KB - 1) * 128 + 31) / 32;
  t->MH = force_mh ? force_mh : (t->KB <= 2 ? 2 : 1);
  t->ctas = pairs ? 2 : 1;
  const int rows_per_tile = 128 * t->MH * t->ctas;
  t->MT = int((nq + rows_per_tile - 1) / rows_per_tile);
  t->NT = int((rows + TILE_N - 1) / TILE_N);
  t->grid = int(std::min<long long>(ctx->sm_count / t->ctas, (long long)t->MT * t->NT));
  // for a number of waves the most parts that fit are the best: shorter chunks at the same cost of each
  long long best = -1;
  const long long units = (long long)t->MT * t->NT;
  for (long long waves = (t->MT + t->grid - 1) / t->grid; best < 0 || units / t->grid + 3 * waves < best; ++waves) {
    const int P = int(std::max<long long>(1, std::min<long long>(std::min(t->NT, 4096), waves * t->grid / t->MT)));
    const int cpn = (t->NT + P - 1) / P;
    const int parts = (t->NT + cpn - 1) / cpn;
    const long long cost = ((long long)t->MT * parts + t->grid - 1) / t->grid * (cpn + 3);
    if (best < 0 || cost < best) {
      best = cost;
      t->cpn = cpn;
      t->parts = parts;
    }
  }
  const long long chunks = (long long)t->MT * t->parts;
  if (chunks > 0x7FFFFFFF) return fail(FV_ERR_UNSUPPORTED, "too many work chunks for the tensor-core tiling");
  t->nchunks = int(chunks);
  t->segmax = int((chunks + t->grid - 1) / t->grid);
  const size_t a_bytes = size_t(t->MH) * t->KB * A_BLOCK_BYTES + A_EXT_BYTES;
  const size_t tail = sizeof(Barriers) + 64;
  for (t->nstage = 6 + t->ctas; t->nstage >= 2; --t->nstage) {
    t->ext_ring = (t->nstage + t->KB - 1) / t->KB + 1;
    t->smem = 1024 + a_bytes + (size_t(t->nstage) * B_STAGE_BYTES + size_t(t->ext_ring) * B_EXT_BYTES) / t->ctas + tail;
    if (t->smem <= ctx->smem_optin) return FV_OK;
  }
  return fail(FV_ERR_UNSUPPORTED, "not enough shared memory for the tensor-core tiling");
}

static PassShape pass_shape(const Tiling& t) { return PassShape{t.MT, t.parts, t.grid, t.segmax, t.MH, t.ctas, t.ccap}; }

// One launch over one way's operands, or over whichever of two the queries allow (`w8` and its word).
template <bool SAMPLE>
static int launch_gemm(fv_ctx* ctx, const Tiling& t16, const GemmWay& w16, const Tiling& t8, const GemmWay* w8,
                       const unsigned int* q8_bad) {
  const bool pair = t16.ctas == 2;
  const size_t smem = w8 ? std::max(t16.smem, t8.smem) : t16.smem;
  cudaLaunchAttribute cluster{};
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim = {2, 1, 1};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = unsigned((w8 ? std::max(t16.grid, t8.grid) : t16.grid) * t16.ctas);
  cfg.blockDim = NTHREADS;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = ctx->stream;
  cfg.attrs = &cluster;
  cfg.numAttrs = pair ? 1 : 0;
  if (!w8) {
    auto kern = t16.MH == 2 ? (pair ? gemm_topk_kernel<2, SAMPLE, false, true> : gemm_topk_kernel<2, SAMPLE, false, false>)
                            : (pair ? gemm_topk_kernel<1, SAMPLE, false, true> : gemm_topk_kernel<1, SAMPLE, false, false>);
    FV_TRY(allow_smem(ctx, kern, smem));
    FV_CUDA(cudaLaunchKernelEx(&cfg, kern, w16));
  } else {
    auto kern = t16.MH == 2 ? (pair ? gemm_topk_either_kernel<2, SAMPLE, true> : gemm_topk_either_kernel<2, SAMPLE, false>)
                            : (pair ? gemm_topk_either_kernel<1, SAMPLE, true> : gemm_topk_either_kernel<1, SAMPLE, false>);
    FV_TRY(allow_smem(ctx, kern, smem));
    FV_CUDA(cudaLaunchKernelEx(&cfg, kern, w16, *w8, q8_bad));
  }
  ctx->stats.launches++;
  FV_CUDA(cudaGetLastError());
  return FV_OK;
}

// Test hook (fv_debug_tc_fault): the next launch of the kernel, once, runs with this wait limit and with one unit's
// loads left out, so that the give-up path of the bounded waits can be exercised without any fault on the device.
static std::atomic<long long> g_test_wait_limit{0};
static std::atomic<int> g_test_skip_unit{-1};

// The query side of the norm step, 16 bytes that a row holds twice: 2^ext_e for each of the three pieces of a norm (bf16:
// 1.0); in the 8-bit form 1 for the remainder and 127 for the rest.
static uint4 norm_step_queries(const TcSide* tc) {
  const uint32_t c = tc->bf16 ? 0x3F80u : uint32_t((tc->ext_e + 15) << 10);
  return make_uint4(c | (c << 16), c, 0u, 0u);
}
static uint4 norm_step_queries8() { return make_uint4(0x7F7F7F01u, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu); }

struct WaitLimit {
  long long cycles = WAIT_LIMIT_CYCLES;
  int skip_unit = -1;
};
static WaitLimit next_wait_limit() {  // of one launch
  WaitLimit l;
  const long long test_limit = g_test_wait_limit.exchange(0);
  if (test_limit > 0) l = WaitLimit{test_limit, g_test_skip_unit.exchange(-1)};
  return l;
}

static void fill_params(GemmParams* g, const Tiling& t, size_t rows, size_t nq, const WaitLimit& limit) {
  g->wait_limit = limit.cycles;
  g->fault_skip_unit = limit.skip_unit;
  g->grid = t.grid;
  g->n = int(rows);
  g->nq = int(nq);
  g->KB = t.KB;
  g->last_steps = t.last_steps;
  g->NT = t.NT;
  g->MT = t.MT;
  g->cpn = t.cpn;
  g->nchunks = t.nchunks;
  g->segmax = t.segmax;
  g->nstage = t.nstage;
  g->ext_ring = t.ext_ring;
}

// ------------------------------------------------------------------------------------------------
// Task mode for other callers (the IVF-PQ scan): operand rows they prepared, scored against runs of this side's rows.
void tc_info(const TcSide* tc, TcInfo* out) {
  out->Kp = tc->Kp;
  out->bf16 = tc->bf16;
  out->n = tc->n;
  out->max_norm2 = tc->h_stats.max_norm2;
  out->min_v = tc->h_stats.min_v;
  out->max_v = tc->h_stats.max_v;
  out->not_finite = tc->h_stats.not_finite != 0;
  out->bytes = tc->i8;
}

int* tc_error_word(TcSide* tc) {
  return reinterpret_cast<int*>(side_words(tc) + W_ERR);
}

int tc_list_pass(fv_ctx* ctx, TcSide* tc, int metric, const uint16_t* d_A, size_t a_rows, const float* d_thr,
                 const uint4* d_tasks, const uint32_t* d_ntasks, unsigned int* d_next_task, u64* d_pool, unsigned int* d_pool_cnt,
                 unsigned int pool_cap, const uint32_t* d_row_owner, uint32_t* d_dropped, int* grid_out, int tile_rows,
                 float* d_minima, const uint32_t* d_task_moff, const uint32_t* d_task_rows) {
  const int Kp = tc->Kp;
  if (Kp > 2 * KBLK) return fail(FV_ERR_UNSUPPORTED, "task mode of the tensor-core kernel covers padded dimensions up to 128");
  if (tile_rows != 128 && tile_rows != 256) return fail(FV_ERR_ARG, "operand tiles have 128 or 256 rows");
  Tiling t{};
  // stages and shared memory for operand tiles of that height; the tiling itself is unused
  FV_TRY(make_tiling(ctx, tc->pd * 2, 256, size_t(TILE_N) * 1024, &t, tile_rows == 128 ? 1 : 2));
  GemmParams gp{};
  fill_params(&gp, t, tc->n, a_rows, next_wait_limit());
  gp.nchunks = 0;
  gp.has_ext = metric == FV_L2 ? 1 : 0;
  gp.aext = norm_step_queries(tc);
  gp.idesc = make_idesc(128, TILE_N, tc->bf16);
  gp.err = tc_error_word(tc);
  gp.ext = tc->ext.as<uint16_t>();
  gp.tau = d_thr;
  gp.tasks = d_tasks;
  gp.ntasks = d_ntasks;
  gp.next_task = d_next_task;
  gp.pool = d_pool;
  gp.pool_cnt = d_pool_cnt;
  gp.pool_cap = pool_cap;
  gp.row_owner = d_row_owner;
  gp.owner_dropped = d_dropped;
  gp.minima = d_minima;
  gp.task_moff = d_task_moff;
  gp.task_rows = d_task_rows;
  GemmWay w{};
  w.p = gp;
  FV_TRY(make_tmap(&w.tmA, type16(tc->bf16), const_cast<uint16_t*>(d_A), a_rows, Kp, 128));
  FV_TRY(make_tmap(&w.tmB, type16(tc->bf16), tc->half.p, tc->n, Kp, TILE_N));
  FV_CUDA(cudaMemsetAsync(d_next_task, 0, sizeof(unsigned int), ctx->stream));
  auto kern = tile_rows == 128 ? gemm_topk_kernel<1, false, true, false> : gemm_topk_kernel<2, false, true, false>;
  FV_TRY(allow_smem(ctx, kern, t.smem));
  kern<<<ctx->sm_count, NTHREADS, t.smem, ctx->stream>>>(w);
  ctx->stats.launches++;
  FV_CUDA(cudaGetLastError());
  *grid_out = ctx->sm_count;
  return FV_OK;
}

// Stages (fv_stats.stage_ms): 0 query conversion, 1 sample pass, 2 main pass, 3 re-rank + certificate, 4 fallback.
// scratch slots: 2 scan partials (fallback), 3 A operands (16 bits, then bytes), 5 query norms + bounds + constants of the byte
// form + error bounds + candidate counters, 6 group minima of the sample, 7 retry ids, 8 fallback keys, 9 candidate buffers
int tc_search(fv_ctx* ctx, TcSide* tc, int metric, const float* d_rows, size_t n, int pd, const float* d_queries,
              size_t nq, int k, uint32_t id_base, u64* d_out_keys, bool mark_stages, bool prefilter_inf,
              const std::function<int()>& then) {
  FV_TRY(pin_ready(ctx));
  const int Kp = tc->Kp;
  const bool is_l2 = metric == FV_L2;
  // The rank R of the sampled bound is kept to SAMPLE_R_MAX: a long result takes a coarser sample (a
  // prefix of the stored one), where fewer of its rows are sampled.  k = 100 over 50,000 rows: 1 row in 32 instead of
  // 1 in 8, R = 13 (at 1 in 8 the bound would have to be about the 29th).  Results of up to 32 keep their own rate even
  // where R = 13 misses the aim by a factor of two (32 results at 1 in 8: one query in 25,000 is re-run): the coarser
  // sample's bound lets 40 % more rows into the re-rank (10,000 queries, 32 of 8,192 x 384: 829 us, 584 at 1 in 8).
  int level = 0;
  int R = pick_sample_r(k, tc->every);
  while (k > 32 && R > SAMPLE_R_MAX && level < SAMPLE_LEVELS) R = pick_sample_r(k, tc->every << ++level);
  R = std::min(R, SAMPLE_R_MAX);
  const size_t ns = sample_prefix(tc->ns, level);
  // One way through both passes, or two: over the 8-bit operands where the base has them and, should a query of the batch
  // not fit them (known on the device only), over the 16-bit ones: one launch that takes either (gemm_topk_either_kernel).
  const int ways = tc->i8 ? 2 : 1;
  // Pairs of CTAs where the batch has queries for both: more than one CTA's tile of the taller of the two ways.
  const bool pairs = nq > (Kp <= 2 * KBLK || tc->i8 ? 256u : 128u);
  struct Way {
    Tiling tm;               // main pass
    GemmWay main, sample;
    size_t nq_pad = 0;
  } way[2] = {};             // 0: 16-bit, 1: 8-bit
  size_t nq_pad = 0, nlists = 0, cand_slots = 0;
  for (int i = 0; i < ways; ++i) {
    const int row_bytes = i ? pd : pd * 2;
    FV_TRY(make_tiling(ctx, row_bytes, nq, n, &way[i].tm, 0, pairs));
    way[i].nq_pad = size_t(way[i].tm.MT) * 128 * way[i].tm.MH * way[i].tm.ctas;
    nq_pad = std::max(nq_pad, way[i].nq_pad);
    Tiling& t = way[i].tm;
    // Candidate slots per list, 4 lists per query and chunk: 256 (128 with the twice as many lists of MH = 2) unless the
    // buffers would pass 2 GB (they are written sparsely: 56 to 112 entries per query in all).  A base stored cluster by
    // cluster puts most of a query's candidates into one or two chunks, so the slots must hold more than the average.
    t.nlists = size_t(t.grid) * t.ctas * t.segmax * (128 * t.MH * 4);
    t.ccap = t.MH == 2 ? 128 : 256;
    while (t.ccap > 16 && t.nlists * size_t(t.ccap) * sizeof(u64) > (size_t(2) << 30)) t.ccap >>= 1;
    nlists = std::max(nlists, t.nlists);
    cand_slots = std::max(cand_slots, t.nlists * size_t(t.ccap));
  }

  // queries -> operand rows (16 bits: scaled by -2 for L2, -1 for inner product), padded to whole tiles with zeros; norms;
  // statistics
  const size_t a16_bytes = (nq_pad * size_t(Kp) * 2 + 255) & ~size_t(255);
  FV_TRY(ctx->scratch[3].reserve(a16_bytes + (tc->i8 ? nq_pad * size_t(tc->Kp8) : 0)));
  FV_TRY(ctx->scratch[5].reserve(4 * nq_pad * sizeof(float) + nlists * sizeof(unsigned int)));  // (nq_pad is a multiple of 128: the counts are aligned)
  // Sample pass: the minima of 1, 8, 32 or 64 sampled rows, so that there are hundreds of groups and two of a query's R best
  // seldom share one (their number times R (R - 1) / 2 is what the rank slips by), for at most 512 MB of queries at a time.
  const int group = ns <= 1024 ? 1 : ns <= 16384 ? 8 : ns <= 65536 ? 32 : 64;
  const size_t smin_ld = (ns + TILE_N - 1) / TILE_N * TILE_N / group;
  size_t slice = std::min(nq_pad, std::max<size_t>(512, ((size_t(512) << 20) / (smin_ld * sizeof(float))) & ~size_t(511)));
  for (;;) {  // (fewer at a time where the device has no room for those of so many)
    const int got = ctx->scratch[6].reserve(slice * smin_ld * sizeof(float));
    if (got == FV_OK) break;
    if (got != FV_ERR_NOMEM || slice <= 512) return got;
    slice = std::max<size_t>(512, slice / 2 & ~size_t(511));
  }
  FV_TRY(ctx->scratch[7].reserve(nq * sizeof(uint32_t)));
  FV_TRY(ctx->scratch[9].reserve(cand_slots * sizeof(u64)));
  uint16_t* dA = ctx->scratch[3].as<uint16_t>();
  uint8_t* dA8 = ctx->scratch[3].as<uint8_t>() + a16_bytes;
  float* qn2 = ctx->scratch[5].as<float>();
  float* tau = qn2 + nq_pad;
  float* const8 = tau + nq_pad;
  float* eps = const8 + nq_pad;
  unsigned int* ccnt = reinterpret_cast<unsigned int*>(eps + nq_pad);
  RangeStats* bst = tc->stats.as<RangeStats>();
  RangeStats* qst = bst + 1;
  unsigned int* words = side_words(tc);
  unsigned int* retry_count = words + W_RETRY;
  unsigned int* q8_bad = tc->i8 ? words + W_Q8_BAD : nullptr;
  for (int i = 0; i < ways; ++i) {
    Way& w = way[i];
    const CUtensorMapDataType type = i ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : type16(tc->bf16);
    const int K = i ? tc->Kp8 : Kp;
    TcSide::Maps& maps = tc->maps[i][pairs ? 1 : 0];
    if (!maps.valid) {
      const int box = TILE_N / w.tm.ctas;
      FV_TRY(make_tmap(&maps.base, type, (i ? tc->rows8 : tc->half).p, n, K, box));
      FV_TRY(make_tmap(&maps.sample, type, (i ? tc->samp8 : tc->samp).p, tc->ns, K, box));  // (a coarser sample: the kernel's n)
      if (is_l2 && pairs) {
        FV_TRY(make_norm_tmap(&maps.base_norm, (i ? tc->ext8 : tc->ext).p, (n + TILE_N - 1) / TILE_N * TILE_N));
        FV_TRY(make_norm_tmap(&maps.sample_norm, (i ? tc->samp_ext8 : tc->samp_ext).p, (tc->ns + TILE_N - 1) / TILE_N * TILE_N));
      }
      maps.valid = true;
    }
    FV_TRY(make_tmap(&w.main.tmA, type, i ? static_cast<void*>(dA8) : dA, nq_pad, K, 128));
    GemmParams& g = w.main.p;
    g = GemmParams{};
    g.has_ext = is_l2 ? 1 : 0;
    g.aext = i ? norm_step_queries8() : norm_step_queries(tc);
    g.idesc = i ? make_idesc_i8(128 * w.tm.ctas, TILE_N) : make_idesc(128 * w.tm.ctas, TILE_N, tc->bf16);
    g.err = tc_error_word(tc);
    w.sample = w.main;
    w.main.tmB = maps.base;
    w.main.tmE = maps.base_norm;
    w.sample.tmB = maps.sample;
    w.sample.tmE = maps.sample_norm;
    g.ext = (i ? tc->ext8 : tc->ext).as<uint16_t>();
    w.sample.p.ext = (i ? tc->samp_ext8 : tc->samp_ext).as<uint16_t>();
  }

  init_search_kernel<<<1, 1, 0, ctx->stream>>>(qst, words);
  if (nq_pad > nq) {
    FV_CUDA(cudaMemsetAsync(dA + nq * size_t(Kp), 0, (nq_pad - nq) * size_t(Kp) * 2, ctx->stream));
    if (tc->i8) FV_CUDA(cudaMemsetAsync(dA8 + nq * size_t(tc->Kp8), 0, (nq_pad - nq) * size_t(tc->Kp8), ctx->stream));
  }
  Queries8 q8;
  if (tc->i8) q8 = Queries8{dA8, tc->Kp8, tc->lo8, const8, q8_bad};
  FV_TRY(convert(ctx, tc->bf16, d_queries, nq, pd, Kp, dA, qn2, is_l2, is_l2 ? -2.f : -1.f, qst, q8));
  if (mark_stages) stage_mark(ctx);

  // sample pass: group minima of the sampled rows' scores, and from them the queries' bounds
  for (size_t q0 = 0; q0 < nq; q0 += slice) {
    const size_t nqs = std::min(slice, nq - q0);
    Tiling ts[2] = {};
    const WaitLimit limit = next_wait_limit();
    for (int i = 0; i < ways; ++i) {
      FV_TRY(make_tiling(ctx, i ? pd : pd * 2, nqs, ns, &ts[i], 0, pairs));
      GemmParams& g = way[i].sample.p;
      fill_params(&g, ts[i], ns, nqs, limit);
      g.a_row0 = int(q0);
      g.smin = ctx->scratch[6].as<float>();
      g.smin_ld = int(smin_ld);
      g.group = group;
    }
    FV_TRY(launch_gemm<true>(ctx, ts[0], way[0].sample, ts[1], tc->i8 ? &way[1].sample : nullptr, q8_bad));
    const size_t with_bound = std::min(slice, nq_pad - q0);
    TauParams tp{};
    tp.smin = ctx->scratch[6].as<float>();
    tp.ld = int(smin_ld);
    tp.groups = int((ns + group - 1) / group);
    tp.nq = int(with_bound);
    tp.R = R;
    tp.queries = d_queries + q0 * size_t(pd);
    tp.real = int(nqs);
    tp.pd = pd;
    tp.Kp = Kp;
    tp.is_l2 = is_l2 ? 1 : 0;
    tp.bf16 = tc->bf16 ? 1 : 0;
    tp.qnorm2 = qn2 + q0;
    tp.bst = bst;
    tp.qst = qst;
    tp.q8_bad = q8_bad;
    tp.tau = tau + q0;
    tp.eps = eps + q0;
    sample_tau_kernel<<<unsigned((with_bound + 7) / 8), 256, 0, ctx->stream>>>(tp);
    ctx->stats.launches++;
    FV_CUDA(cudaGetLastError());
  }
  if (mark_stages) stage_mark(ctx);

  // main pass: every row scoring below the query's sampled bound becomes a candidate
  const WaitLimit limit = next_wait_limit();
  for (int i = 0; i < ways; ++i) {
    GemmParams& g = way[i].main.p;
    fill_params(&g, way[i].tm, n, nq, limit);
    g.tau = tau;
    g.cbuf = ctx->scratch[9].as<u64>();
    g.ccnt = ccnt;
    g.ccap = way[i].tm.ccap;
  }
  FV_TRY(launch_gemm<false>(ctx, way[0].tm, way[0].main, way[1].tm, tc->i8 ? &way[1].main : nullptr, q8_bad));
  if (mark_stages) stage_mark(ctx);

  RerankParams rp{};
  rp.tau = tau;
  rp.cbuf = ctx->scratch[9].as<u64>();
  rp.ccnt = ccnt;
  rp.shapes = PassShapes{pass_shape(way[0].tm), pass_shape(way[1].tm), q8_bad};
  rp.const8 = const8;
  rp.parity8 = tc->parity8.as<uint8_t>();
  rp.rows = d_rows;
  rp.queries = d_queries;
  rp.qnorm2 = qn2;
  rp.eps = eps;
  rp.n = int(n);
  rp.nq = int(nq);
  rp.pd = pd;
  rp.k = k;
  rp.id_base = id_base;
  rp.out_keys = d_out_keys;
  rp.retry_ids = ctx->scratch[7].as<uint32_t>();
  rp.retry_count = retry_count;
  // long results: several warps per query while the batch fills the resident warps (16 to 24 per SM) at most one and a
  // half to two times (with 10 results, some 20 runs of eight rows, the merge takes what the shares save)
  const int wpb = 8;
  rp.wpq = 1;
  while (k > 32 && rp.wpq < 8 && nq * size_t(rp.wpq) * 2 <= size_t(ctx->sm_count) * 36) rp.wpq <<= 1;
  const size_t rsmem = size_t(wpb) * (pd * sizeof(float) + (rp.wpq > 1 ? 128 * sizeof(u64) : 0));
  auto pick = [&](auto l2) {
    constexpr bool IS_L2 = decltype(l2)::value;
    return k <= 32 ? rerank_kernel<IS_L2, 1, false> : rp.wpq > 1 ? rerank_kernel<IS_L2, 4, true> : rerank_kernel<IS_L2, 4, false>;
  };
  auto rk = is_l2 ? pick(std::true_type{}) : pick(std::false_type{});
  rk<<<unsigned((nq * size_t(rp.wpq) + wpb - 1) / wpb), wpb * 32, rsmem, ctx->stream>>>(rp);
  ctx->stats.launches++;
  FV_CUDA(cudaGetLastError());
  if (mark_stages) stage_mark(ctx);

  if (then) FV_TRY(then());
  const unsigned int* h_words = reinterpret_cast<const unsigned int*>(ctx->h_pin);  // retry count, error word
  FV_CUDA(cudaMemcpyAsync(ctx->h_pin, retry_count, 2 * sizeof(unsigned int), cudaMemcpyDeviceToHost, ctx->stream));
  FV_CUDA(cudaStreamSynchronize(ctx->stream));
  if (h_words[1]) return fail(FV_ERR_TIMEOUT, "a bounded wait inside the tensor-core kernel ran out");
  ctx->stats.uncertified = h_words[0];
  if (h_words[0]) {
    const size_t nsub = h_words[0];
    FV_TRY(ctx->scratch[8].reserve(nsub * size_t(k) * sizeof(u64)));
    u64* sub = ctx->scratch[8].as<u64>();
    FV_TRY(exact_scan(ctx, metric, d_rows, n, pd, d_queries, size_t(pd), rp.retry_ids, nsub, k, prefilter_inf, id_base, sub, 2));
    scatter_keys_kernel<<<ctx->sm_count, 256, 0, ctx->stream>>>(sub, rp.retry_ids, nsub, k, d_out_keys);
    ctx->stats.launches++;
    FV_CUDA(cudaGetLastError());
    if (then) FV_TRY(then());
  }
  if (mark_stages) stage_mark(ctx);
  return FV_OK;
}

}  // namespace fv

// Test hook: arms the next launch of the tensor-core kernel (once) with a short wait limit, in cycles, and makes the
// producer of work item 0 leave out the loads of unit `skip_unit` of it: the consumer of that stage waits until
// the limit, the kernel sets its error word, frees its tensor memory and returns, and the search that launched it
// fails with FV_ERR_TIMEOUT.  Nothing on the device faults or spins without bound.  (0, -1) disarms.
extern "C" int fv_debug_tc_fault(long long wait_limit_cycles, int skip_unit) {
  if (wait_limit_cycles < 0 || skip_unit < -1) return fv::fail(FV_ERR_ARG, "fv_debug_tc_fault: bad argument");
  fv::g_test_skip_unit.store(skip_unit);
  fv::g_test_wait_limit.store(wait_limit_cycles);
  return FV_OK;
}
