// batch_dev.cuh -- device side of the batch engine: many independent transforms of uneven sizes in one persistent,
// graph-launched work-queue kernel.
//
// Work items (16 bytes each) are tiles:
//   SMALL   TPC transforms of one size 2^n <= 1024, consecutive in the
//           size-sorted job descriptors (one sub-transform per job)
//   PASS p  TPC sub-transforms of HBM pass p of one large transform
//           (n > 10, passes from batch_split: strided passes of 5..7 stages
//           keep >= 8 adjacent columns; 2^16 = 6 + 10, 2^20 = 6 + 6 + 8)
// A CTA takes the next item with an atomic counter.  Queue order is: all
// first passes of large jobs, then small tiles from the largest size down, cut
// into one segment before each later pass group, then the smallest.  Pass p > 0 of a job reads what pass p-1 wrote, so its
// tiles first wait until the job's pass p-1 counter reaches that pass's tile
// count.  The wait cannot deadlock: every pass p-1 tile was handed out
// before any pass p tile (see the loop in k_batch).  The wait is
// still bounded; when it gives up it raises the error word, the tile is
// skipped, and bntt_batch_status() reports BNTT_ETIMEOUT.
//
// The control words (queue head, error word, per-job pass counters) live in a
// device workspace owned by the batch and are cleared by a memset node of the
// same CUDA graph before each launch.
#pragma once
#include "internal.h"
#include "ntt_core.cuh"

namespace bntt {

// Threads and resident CTAs per SM of the kernels.
//
// Long lists of a fast modulus: 128 threads, 7 CTAs (72 registers).  The rate of
// a tile does not change between 24 and 32 resident warps, and small CTAs overlap
// more of each other's item fetches, loads and barriers (818 us for the uneven
// batch with 4 CTAs of 256 threads, 804 with 6 of 128).  Uneven batch and ragged
// inverse batch, us, with 5, 6 and 7 CTAs: 813 and 533, 793 and 520, 791 and 513.
//
// Short lists: 256 threads, 4 CTAs (64 registers), 4 elements per thread
// throughout.  Their tiles do not fill the SMs, so a tile's own time counts, and
// with twice the threads it is shorter.  Lists of tiles, us, 128 and 256 threads:
// 1 x 2^10 12.0 and 10.3, 1,036 x 2^10 28.7 and 26.8, 8 x 2^16 43.1 and 28.7, 143
// of each of 2^4..2^10 16.3 and 12.3; but 8,288 x 2^10 166 and 170, 4 x 2^20 168
// and 190.  Short is what the long lists' kernel would hold in one wave
// (batch_launch): 1,500 x 2^10 are 37.0 and 37.5.
//
// The general multiply always takes 256 threads: 4,000 of each of 2^4..2^10 292
// us, with 128 (6 CTAs of 80 registers) 336.
constexpr int kBatchThreads = 128, kShortThreads = 256;
constexpr int batch_ctas(int threads) { return threads == kBatchThreads ? 7 : 4; }
// log2 of the elements per thread of a tile whose shape has 2^logr of them
constexpr int batch_logr(int logr, int threads) { return threads == kBatchThreads || logr < 2 ? logr : 2; }

// Object files of the fast kernels, forward and inverse: one layout and one number
// of threads each, so that a program loads what it runs (ntt_kernels.cuh; the
// first batch of a process took 12.4 ms forward and 6.1 to 8.2 inverse with all
// four in one module, 3.5 to 4.8 and 1.1 to 3.7 now).
constexpr int batch_part(int layout, int threads) {
  return (layout == LAYOUT_HILO ? 0 : 1) + (threads == kBatchThreads ? 0 : 2);
}
constexpr int part_layout(int part) { return part & 1 ? LAYOUT_U128 : LAYOUT_HILO; }
constexpr int part_threads(int part) { return part < 2 ? kBatchThreads : kShortThreads; }
template <int PART>
const void* batch_kernel_fast();
template <int PART>
const void* batch_kernel_inverse();

struct alignas(16) DevJob {  // two 16-byte loads
  const uint4* x;
  uint4* y;
  const uint4* tw;
  uint32_t log2n;
  uint32_t slot;  // counter slot for large jobs
};

// Device build of a new job list's descriptors (k_build_jobs): a plan's table
// and size, and a large job's counter slot.
struct PlanRef {
  const uint4* tw;
  uint32_t log2n;
  uint32_t pad;
};
struct LargeRef {
  uint32_t job;
  uint32_t slot;
};
// first position of each small size in the size-sorted order
struct SizeFirst {
  uint32_t first[11];
};

enum : uint32_t { ITEM_SMALL = 0, ITEM_PASS = 1 };

struct WorkItem {
  uint16_t shape;   // index into the shape table below
  uint16_t kind;    // ITEM_SMALL or ITEM_PASS
  uint32_t a;       // SMALL: first descriptor of the tile; PASS: the job's descriptor
  uint32_t b;       // SMALL: number of jobs in the tile; PASS: first sub-transform id
  uint16_t pass;    // PASS: pass index
  uint16_t wait;    // PASS: bit 0 the tile waits for the pass run before it,
                    // bit 1 the pass reads the job's input, bits 8.. its first stage
};
static_assert(sizeof(WorkItem) == 16, "work item layout");

// Tile shapes of the persistent kernel: X(id, M, LOGR, TPC, map), TPC
// sub-transforms per item, of which 128 threads hold 128 >> (M - LOGR) at a time
// (4-element shapes take two turns); 256 threads hold all of them, 4 elements
// each (batch_logr).  Interleaved
// (strided) tiles keep at least 8 adjacent columns (128 bytes of each row).
// 8 elements per thread run three stages per exchange, with about a fifth
// fewer index and exchange instructions, but twice the code: the strided
// passes (two tile passes each) and 2^10 gain from it (64 x 2^16: 1076 ->
// 1034 us), the contiguous tiles below do not, since the warps then wait for
// instructions (with 8 elements throughout the uneven batch takes 822 us).
// A tile engine with the size at run time (one body for all shapes) takes 84
// instructions per butterfly instead of 66 and 909 us.
#define BNTT_BATCH_SHAPES(X)               \
  X(0, 1, 1, 256, MAP_CONTIG)              \
  X(1, 2, 2, 256, MAP_CONTIG)              \
  X(2, 3, 2, 128, MAP_CONTIG)              \
  X(3, 4, 2, 64, MAP_CONTIG)               \
  X(4, 5, 2, 32, MAP_CONTIG)               \
  X(5, 6, 2, 16, MAP_CONTIG)               \
  X(6, 7, 2, 8, MAP_CONTIG)                \
  X(7, 8, 2, 4, MAP_CONTIG)                \
  X(8, 9, 2, 2, MAP_CONTIG)                \
  X(9, 10, 3, 1, MAP_CONTIG)               \
  X(10, 5, 3, 32, MAP_INTERLEAVED)         \
  X(11, 6, 3, 16, MAP_INTERLEAVED)         \
  X(12, 7, 3, 8, MAP_INTERLEAVED)

struct BatchShape {
  int m, logr, tpc, map;
};
inline constexpr BatchShape kShapes[] = {
#define BNTT_SHAPE_ROW(id, M, LOGR, TPC, MAP) {M, LOGR, TPC, MAP},
    BNTT_BATCH_SHAPES(BNTT_SHAPE_ROW)
#undef BNTT_SHAPE_ROW
};
constexpr int kNumShapes = sizeof(kShapes) / sizeof(kShapes[0]);

// control words: [0] queue head, [1] error word, [2 + 4*slot + p] pass counters
constexpr int kCtlHeader = 2;
constexpr int kMaxPasses = 4;
// bounded wait: default poll limit (polls x ~100 ns sleeps, a few seconds)
constexpr uint32_t kWaitPolls = 1u << 25;

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

struct BatchArgs {
  const WorkItem* items;
  uint32_t nitems;
  const DevJob* jobs;  // small jobs sorted by size, then the large jobs
  uint32_t* ctl;
  const uint32_t* pass_tiles;  // [slot * kMaxPasses + p] tile count of pass p
  uint32_t wait_polls;         // give up a dependency wait after this many polls
};

// A later-pass item waits until its job's earlier pass is complete; returns
// false when the wait gave up (the error word is set; the tile is skipped).
// INV: the passes of a large job run last to first (inverse transform), so a
// pass waits for the pass after it and the last pass is the one that reads the
// job's input.
template <bool INV>
__device__ __forceinline__ bool item_wait(const WorkItem& it, const BatchArgs& ba, int* s_flag) {
  if (it.kind != ITEM_PASS || !(it.wait & 1)) return true;
  const uint32_t slot = ba.jobs[it.a].slot;
  uint32_t* counters = ba.ctl + kCtlHeader + slot * kMaxPasses;
  const int pred = INV ? (int)it.pass + 1 : (int)it.pass - 1;
  if (threadIdx.x == 0) {
    const uint32_t want = ba.pass_tiles[slot * kMaxPasses + pred];
    uint32_t polls = 0;
    int ok = 1;
    while (ld_acquire(&counters[pred]) < want) {
      if (++polls > ba.wait_polls) {
        atomicOr(&ba.ctl[1], 1u);
        ok = 0;
        break;
      }
      __nanosleep(100);
    }
    *s_flag = ok;
  }
  __syncthreads();
  return *s_flag != 0;
}

// The sub-transform a work item hands to thread `sub` of the tile: a whole
// small job, or one sub-transform of an HBM pass of a large job (whose tiles
// are always full: batch_split's passes are whole numbers of tiles).
template <int M, int MAP>
__device__ __forceinline__ SubRef item_subref(const WorkItem& it, const BatchArgs& ba, int sub) {
  SubRef sr;
  if (MAP == MAP_CONTIG && it.kind == ITEM_SMALL) {
    sr.valid = (uint32_t)sub < it.b;
    const DevJob& j = ba.jobs[it.a + (sr.valid ? (uint32_t)sub : 0u)];
    sr.x = j.x;
    sr.y = j.y;
    sr.tw = j.tw;
    sr.trow = 1;
    sr.lshift = 0;
    return sr;
  }
  const DevJob& j = ba.jobs[it.a];
  const uint32_t s0 = it.wait >> 8;  // first stage of this pass
  const uint32_t l = MAP == MAP_CONTIG ? 0u : j.log2n - s0 - M;
  const uint32_t sid = it.b + (uint32_t)sub;  // (H << L) | c
  const uint32_t h = sid >> l;
  const uint32_t off = (h << (l + M)) + (sid & ((1u << l) - 1u));
  sr.valid = true;
  sr.x = ((it.wait & 2) ? j.x : j.y) + off;
  sr.y = j.y + off;
  sr.tw = j.tw;
  sr.trow = (1u << s0) + h;
  sr.lshift = l;
  return sr;
}

// A pass tile publishes its completion: every thread's stores, then one
// release increment of the job's pass counter.
__device__ __forceinline__ void item_publish(const WorkItem& it, const BatchArgs& ba) {
  if (it.kind != ITEM_PASS) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    const DevJob& j = ba.jobs[it.a];
    __threadfence();
    atomicAdd(&ba.ctl[kCtlHeader + j.slot * kMaxPasses + it.pass], 1u);
  }
}

// One item on the compile-time tile of the plan kernels.  Inlined into the
// kernel: as separate functions the items spilled around the call's fixed
// registers (848 -> 826 us for the uneven batch).  L2-coherent loads: a later
// pass reads what other CTAs wrote in this launch.
template <int M, int LOGR, int TPC, int MAP, class Arith, int LY, int THREADS>
__device__ __forceinline__ void run_item(const WorkItem& it, const BatchArgs& ba, uint4* smem,
                                      const ModParams& mp, int layout_arg, int* s_flag) {
  const int layout = LY >= 0 ? LY : layout_arg;
  constexpr int HELD = THREADS >> (M - LOGR);  // sub-transforms the threads hold at a time
  using T = NttTile<M, LOGR, HELD, MAP, Arith>;
  static_assert(T::THREADS == THREADS && TPC % HELD == 0, "tile shape");
  if (!item_wait<false>(it, ba, s_flag)) return;
#pragma unroll 1
  for (int turn = 0; turn < TPC / HELD; ++turn) {
    const int sub = T::sub_of(threadIdx.x), lane = T::lane_of(threadIdx.x);
    const SubRef sr = item_subref<M, MAP>(it, ba, turn * HELD + sub);
    if (turn > 0) T::sync();  // smem is reused
    T::template run<TW_CONST>(sr, sub, lane, smem, mp, layout);
  }
  item_publish(it, ba);
}

// LY: the element layout as a constant (LAYOUT_HILO or LAYOUT_U128), or -1
// for the `layout` argument.  A constant layout removes the runtime word
// select of every HBM load and store (measured +0.9 % on the uneven batch).
template <class Arith, int LY, int THREADS>
__global__ void __launch_bounds__(THREADS, batch_ctas(THREADS)) k_batch(BatchArgs ba, ModParams mp, int layout) {
  extern __shared__ uint4 smem[];
  __shared__ uint32_t s_item;
  __shared__ int s_flag;
  // (The next item is not taken while this one runs: with few items per CTA the
  // early CTAs then hold what late ones could run -- 296 x 2^10 22.3 instead of
  // 14.4 us, one 2^20 91 instead of 55 -- and long lists gain nothing, the uneven
  // batch 789 instead of 784.)
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(&ba.ctl[0], 1u);
    __syncthreads();
    const uint32_t i = s_item;
    if (i >= ba.nitems) break;
    const WorkItem it = ba.items[i];
    switch (it.shape) {
#define BNTT_RUN_SHAPE(id, M, LOGR, TPC, MAP)                                   \
  case id:                                                                      \
    run_item<M, batch_logr(LOGR, THREADS), TPC, MAP, Arith, LY, THREADS>(it, ba, smem, mp, layout, &s_flag);  \
    break;
      BNTT_BATCH_SHAPES(BNTT_RUN_SHAPE)
#undef BNTT_RUN_SHAPE
      default: break;
    }
    __syncthreads();  // smem and s_item are reused by the next item
  }
}

}  // namespace bntt
