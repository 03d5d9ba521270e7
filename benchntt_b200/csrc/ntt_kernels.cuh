// ntt_kernels.cuh -- kernel template over NttTile and its registry entries.
#pragma once
#include "internal.h"
#include "ntt_core.cuh"

namespace bntt {

// One CTA per tile of a geometry: CTA t transforms sub-transforms
// [t*TPC, t*TPC + TPC).  The hardware hands a CTA to an SM as soon as one of
// its resident CTAs ends, which balances what the warp schedulers do not:
// among the CTAs of an SM the oldest gets most of the issue slots, so with a
// fixed share of the tiles per CTA (a grid of the resident CTAs walking the
// tiles) the CTAs drifted apart and the SM ran its last third with fewer of
// them (39 % of the warp slots active on average, of the 50 % the registers
// allow).  65,536 x 1024: 1331 -> 1219 us; a grid of 2, 4 and 8 times the
// resident CTAs lies between (1282, 1247, 1229).  Without the walk's loop and its
// registers 1183 us.
// MINB > 0 asks for at least MINB resident CTAs per SM (fewer registers per
// thread, more warps to hide the latency of the carry chains).
template <int M, int LOGR, int TPC, int MAP, class Arith, int MINB, int SRC = SRC_GLOBAL>
__global__ void __launch_bounds__(NttTile<M, LOGR, TPC, MAP, Arith>::THREADS, MINB)
    k_ntt_sub(SubGeom g, ModParams mp, int layout) {
  using T = NttTile<M, LOGR, TPC, MAP, Arith>;
  extern __shared__ uint4 smem[];
  const int tid = threadIdx.x;
  const int sub = T::sub_of(tid), lane = T::lane_of(tid);
  stream_wait();
  const uint64_t sid = (uint64_t)blockIdx.x * TPC + (uint64_t)sub;
  const SubRef sr = MAP == MAP_CONTIG ? make_subref_contig<M>(g, sid) : make_subref(g, sid);
  // the element layout as a constant in each branch: no word select per
  // HBM load and store
  if (layout == LAYOUT_HILO) T::template run<SRC>(sr, sub, lane, smem, mp, LAYOUT_HILO, MulB{g.b, g.y, g.bmask});
  else T::template run<SRC>(sr, sub, lane, smem, mp, LAYOUT_U128, MulB{g.b, g.y, g.bmask});
}

// Contiguous sub-transforms (L = 0: tile t is the 16-byte elements
// [t*TPC*2^M, (t+1)*TPC*2^M) of g.x), each CTA walking tiles blockIdx.x,
// +gridDim.x, ..., with every tile's input copied into shared memory by
// cp.async one tile ahead: while a CTA transforms tile
// t, the copy of its next tile is in flight, so the load latency that bounds
// small transforms (little work per element, a few tiles per CTA) overlaps
// the arithmetic.  The copy lands in the tile's exchange slots, the first pass
// gathers from there and every pass exchanges in place (a thread writes back
// only the slots it read).  Two tile buffers per CTA.  With TW_SHARED the
// CTA first copies the table's 2^M entries into shared memory (only for
// whole transforms, S0 = 0, where a tile reads entries below 2^M).
template <int M, int LOGR, int TPC, class Arith, int MINB, int SRC>
__global__ void __launch_bounds__(NttTile<M, LOGR, TPC, MAP_CONTIG, Arith>::THREADS, MINB)
    k_ntt_sub_staged(SubGeom g, ModParams mp, int layout) {
  using T = NttTile<M, LOGR, TPC, MAP_CONTIG, Arith>;
  constexpr int N = 1 << M;
  constexpr int TILE = TPC * N;  // elements per tile
  static_assert(T::THREADS * T::R == TILE, "tile shape");
  extern __shared__ uint4 smem[];
  const int tid = threadIdx.x;
  const int sub = T::sub_of(tid), lane = T::lane_of(tid);
  const uint64_t ntiles = (g.nsub + TPC - 1) / TPC;
  stream_wait();
  // tile t's valid elements, copied into `dst` in slot order
  auto stage = [&](uint64_t t, uint4* dst) {
    const uint64_t first = t * TPC;
    const uint64_t left = g.nsub - first;
    const uint32_t elems = (uint32_t)(left < (uint64_t)TPC ? left : (uint64_t)TPC) << M;
    const uint4* src = g.x + (first << M);
#pragma unroll
    for (int k = 0; k < T::R; ++k) {
      const uint32_t e = (uint32_t)tid + (uint32_t)k * T::THREADS;
      if (e < elems) cp_async16(&dst[T::slot((int)(e >> M), (int)(e & (N - 1)))], src + e);
    }
  };
  const uint4* tw = g.tw;
  if constexpr ((SRC & TW_SHARED) != 0) {
    uint4* const tws = smem + 2 * TILE;
    for (int e = tid; e < N; e += T::THREADS) tws[e] = g.tw[e];
    tw = tws;  // made visible by the barrier before the first tile
  }
  uint64_t tile = blockIdx.x;
  if (tile < ntiles) stage(tile, smem);
  cp_async_commit();
  for (int b = 0; tile < ntiles; tile += gridDim.x, b ^= 1) {
    const uint64_t next = tile + gridDim.x;
    if (next < ntiles) stage(next, smem + (b ^ 1) * TILE);
    cp_async_commit();
    cp_async_wait<1>();  // every group but the newest: this tile's copies
    __syncthreads();
    SubRef sr = make_subref_contig<M>(g, tile * TPC + (uint64_t)sub);
    sr.tw = tw;
    if (layout == LAYOUT_HILO)
      T::template run<SRC | SRC_STAGED>(sr, sub, lane, smem + b * TILE, mp, LAYOUT_HILO,
                                               MulB{g.b, g.y, g.bmask});
    else
      T::template run<SRC | SRC_STAGED>(sr, sub, lane, smem + b * TILE, mp, LAYOUT_U128,
                                               MulB{g.b, g.y, g.bmask});
    __syncthreads();  // this buffer is refilled by the next iteration's copy
  }
  cp_async_wait<0>();
}

}  // namespace bntt

// Default shapes of the plan transforms with the fast multiply, forward and
// inverse: X(M, LOGR, TPC, map, resident CTAs per SM, SRC, use).  CTAs of 64 or
// 128 threads: with one CTA per tile, smaller ones keep an SM's warps in more
// different phases (2^24 elements of 2^8: 256 threads 250 us, 64 threads 234).
// Interleaved tiles keep at least 8 columns (128 bytes of a row).
//
// In parts, one object file each (forward and inverse): an object file's module is
// loaded by the first launch of one of its kernels, and that takes the longer the
// more kernels and line tables it holds.  First transform of a process, all shapes
// in one module and in parts, ms: one 2^10 forward 14.3 and 1.3, inverse 4.0 and
// 0.7; 64 x 2^16 forward 13.7 and 3.2.  Three to eight kernels to a part.
#define BNTT_PLAN_SHAPES_0(X)                                         \
  X(1, 1, 256, MAP_CONTIG, 4, SRC_GLOBAL, USE_ALL)                    \
  X(2, 2, 256, MAP_CONTIG, 4, SRC_GLOBAL, USE_ALL)                    \
  X(3, 2, 32, MAP_CONTIG, 16, SRC_GLOBAL, USE_ALL)                    \
  X(4, 2, 16, MAP_CONTIG, 8, TW_AHEAD, USE_LONE)                      \
  X(4, 2, 16, MAP_CONTIG, 16, SRC_GLOBAL, USE_FEW | USE_MANY)
#define BNTT_PLAN_SHAPES_1(X)                                         \
  X(5, 2, 8, MAP_CONTIG, 8, TW_AHEAD, USE_LONE)                       \
  X(5, 2, 8, MAP_CONTIG, 16, SRC_GLOBAL, USE_FEW)                     \
  X(5, 3, 16, MAP_CONTIG, 12, SRC_GLOBAL, USE_MANY)                   \
  X(6, 2, 4, MAP_CONTIG, 8, TW_AHEAD, USE_LONE)                       \
  X(6, 2, 4, MAP_CONTIG, 16, SRC_GLOBAL, USE_FEW)                     \
  X(6, 3, 8, MAP_CONTIG, 10, SRC_GLOBAL, USE_MANY)
#define BNTT_PLAN_SHAPES_2(X)                                         \
  X(7, 2, 2, MAP_CONTIG, 8, TW_AHEAD, USE_LONE)                       \
  X(7, 2, 2, MAP_CONTIG, 16, SRC_GLOBAL, USE_FEW)                     \
  X(7, 3, 4, MAP_CONTIG, 12, SRC_GLOBAL, USE_MANY)
#define BNTT_PLAN_SHAPES_3(X)                                         \
  X(8, 2, 1, MAP_CONTIG, 8, TW_AHEAD, USE_LONE)                       \
  X(8, 2, 1, MAP_CONTIG, 16, SRC_GLOBAL, USE_FEW)                     \
  X(8, 3, 2, MAP_CONTIG, 10, SRC_GLOBAL, USE_MANY)
#define BNTT_PLAN_SHAPES_4(X)                                         \
  X(9, 2, 1, MAP_CONTIG, 4, TW_AHEAD, USE_LONE)                       \
  X(9, 2, 1, MAP_CONTIG, 8, SRC_GLOBAL, USE_FEW)                      \
  X(9, 3, 1, MAP_CONTIG, 10, SRC_GLOBAL, USE_MANY)
#define BNTT_PLAN_SHAPES_5(X)                                         \
  X(10, 2, 1, MAP_CONTIG, 2, TW_AHEAD, USE_LONE)                      \
  X(10, 2, 1, MAP_CONTIG, 4, SRC_GLOBAL, USE_FEW)                     \
  X(10, 3, 1, MAP_CONTIG, 7, SRC_GLOBAL, USE_MANY)
#define BNTT_PLAN_SHAPES_6(X)                                         \
  X(5, 2, 16, MAP_INTERLEAVED, 8, SRC_GLOBAL, USE_LONE | USE_FEW)     \
  X(5, 3, 32, MAP_INTERLEAVED, 6, SRC_GLOBAL, USE_MANY)               \
  X(6, 2, 8, MAP_INTERLEAVED, 4, TW_AHEAD, USE_LONE)                  \
  X(6, 2, 8, MAP_INTERLEAVED, 8, SRC_GLOBAL, USE_FEW)                 \
  X(6, 3, 16, MAP_INTERLEAVED, 5, SRC_GLOBAL, USE_MANY)               \
  X(7, 2, 8, MAP_INTERLEAVED, 2, TW_AHEAD, USE_LONE)                  \
  X(7, 2, 8, MAP_INTERLEAVED, 4, SRC_GLOBAL, USE_FEW)                 \
  X(7, 3, 8, MAP_INTERLEAVED, 6, SRC_GLOBAL, USE_MANY)

#define BNTT_SUBK_FN(M, LOGR, TPC, MAP, ARITH, MINB, FN, USE)                             \
  ::bntt::SubKernel {                                                                     \
    M, LOGR, TPC, MAP, ARITH::kFast ? 1 : 0, ::bntt::NttTile<M, LOGR, TPC, MAP, ARITH>::THREADS, \
        (size_t)::bntt::NttTile<M, LOGR, TPC, MAP, ARITH>::SMEM_SLOTS * 16u,              \
        (const void*)&FN, 0, MINB, 0, USE                                                 \
  }
#define BNTT_SUBK_U(M, LOGR, TPC, MAP, ARITH, MINB, USE) \
  BNTT_SUBK_FN(M, LOGR, TPC, MAP, ARITH, MINB, (::bntt::k_ntt_sub<M, LOGR, TPC, MAP, ARITH, MINB>), USE)
#define BNTT_SUBK_B(M, LOGR, TPC, MAP, ARITH, MINB) \
  BNTT_SUBK_U(M, LOGR, TPC, MAP, ARITH, MINB, ::bntt::USE_TUNED)
#define BNTT_SUBK(M, LOGR, TPC, MAP, ARITH) BNTT_SUBK_B(M, LOGR, TPC, MAP, ARITH, 1)
// staged contiguous kernels: two tile buffers (+ the table with TW_SHARED)
#define BNTT_SUBK_STAGED(M, LOGR, TPC, ARITH, MINB, SRC)                                       \
  ::bntt::SubKernel {                                                                         \
    M, LOGR, TPC, ::bntt::MAP_CONTIG, ARITH::kFast ? 1 : 0,                                   \
        ::bntt::NttTile<M, LOGR, TPC, ::bntt::MAP_CONTIG, ARITH>::THREADS,                    \
        (size_t)(2 * (TPC << M) + (((SRC) & ::bntt::TW_SHARED) ? (1 << M) : 0)) * 16u,        \
        (const void*)&::bntt::k_ntt_sub_staged<M, LOGR, TPC, ARITH, MINB, SRC>, 0, MINB, SRC  \
  }
