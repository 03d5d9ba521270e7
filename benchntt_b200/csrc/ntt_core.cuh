// ntt_core.cuh -- the forward network of benchNTT on sm_100a.
//
// The reference transform (src/ntt_scalar.c:582-627) is a radix-2 network:
// with n = log2 N, stage s (0 <= s < n) pairs indices that differ in bit
// n-1-s and multiplies by the table entry T[2^s + (index >> (n - s))].  The
// reference evaluates it in constant-geometry order with ping-pong buffers;
// here it is evaluated in place, in natural order, which yields the same
// outputs (tests check both against the reference).
//
// Sub-transforms.  Stages [S0, S0 + M) of an n-point transform touch index
// bits [L, L + M) with L = n - S0 - M; every assignment of the other bits --
// the top S0 bits H and the low L bits c -- selects an independent 2^M-point
// sub-network on the elements
//     idx(j) = (H << (n - S0)) | (j << L) | c,     j in [0, 2^M)
// whose stage S0 + s multiplies by
//     T[((2^S0 + H) << s) + (j >> (M - s))].
// A small transform is one sub-transform (S0 = L = 0).  Large transforms run
// as passes over HBM: for 2^16, pass A has S0 = 0, M = 6, L = 10 (columns)
// and pass B has S0 = 6, M = 10, L = 0 (rows).  This holds for any table T
// because it only regroups the network's data flow.
//
// Inside a sub-transform each thread holds R = 2^LOGR elements in registers.
// The M stages are cut into passes of at most LOGR stages; in a pass a thread
// owns R / 2^r groups of 2^r elements that differ only in that pass's bits
// and runs the r stages on them without communication.  Passes exchange data
// through shared memory (XOR-swizzled 16-byte slots), the first pass reads
// HBM and the last writes HBM.
#pragma once
#include "u128.cuh"

namespace bntt {

enum : int { MAP_CONTIG = 0, MAP_INTERLEAVED = 1 };

// Where one sub-transform's elements and twiddles live, as a thread sees it.
struct SubRef {
  const uint4* x;    // element j at x[j << L]
  uint4* y;          // element j at y[j << L]
  const uint4* tw;   // table of the whole transform, limb order (LAYOUT_U128)
  uint32_t trow;     // 2^S0 + H
  uint32_t lshift;   // L
  bool valid;
};

// Data and tables are read with coherent loads, data through L2 only: a
// transform's input may have been written earlier in the same launch (later
// passes of the persistent kernel) or by the kernel before it, which a plan
// kernel overlaps (stream_wait).
__device__ __forceinline__ uint4 ld_data(const uint4* p) { return __ldcg(p); }

// Programmatic dependent launch: the plan and vector kernels are launched as
// soon as the kernel before them in the stream has started its last CTA, and
// wait here until that kernel has completed and its writes are visible;
// nothing is read or written before.  The wait comes first, so a kernel lets
// the next one in only after its own predecessor has completed.  Without it
// the end of one kernel and the start of the next cost a small launch about
// 2 us (2^15 elements of 2^9 points back to back: 6.2 -> 4.0 us).
__device__ __forceinline__ void stream_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Optional pointwise product fused into the store of a transform's last
// pass: element e of y becomes y[e] * b[e'] mod q (vector_mul,
// src/blas_scalar.c:594), e' = (e's offset from ybase) & bmask.  bmask = N - 1
// applies one vector to every transform of the batch; all ones pairs
// transform t with b's t-th vector.  b == nullptr: plain store.
struct MulB {
  const uint4* b = nullptr;
  const uint4* ybase = nullptr;
  uint64_t bmask = 0;
};

// Where a tile's first pass finds its inputs and every pass its twiddles.
//   SRC_STAGED  the inputs were copied into the tile's shared-memory slots
//               beforehand (cp.async, k_ntt_sub_staged); the first pass
//               gathers from there like the later passes
//   TW_SHARED   sr.tw points at a copy of the table in shared memory
//   TW_CONST    no kernel still running may write the table: read-only loads,
//               which the compiler may move over the exchanges (kernels
//               without stream_wait)
//   TW_AHEAD    the entries of every pass are loaded into registers together
//               with the input (launches that do not fill the SMs, where a
//               table load per pass is latency nothing hides)
enum : int { SRC_GLOBAL = 0, SRC_STAGED = 1, TW_SHARED = 2, TW_CONST = 4, TW_AHEAD = 8 };

// 16-byte asynchronous copy global -> shared (cp.async, L2 only), and the
// group commit / wait that order them.
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}
__device__ __forceinline__ uint4 lds128(const uint4* p) {
  uint4 v;
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}

// Table entry i (i < 2^24): the byte offset fits 32 bits, so the address is
// one shift and one 64-bit add.
__device__ __forceinline__ const uint4* tw_at(const uint4* tw, uint32_t i) {
  return reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(tw) + (i << 4));
}

template <int M, int LOGR, int TPC, int MAP, class Arith>
struct NttTile {
  static constexpr int R = 1 << LOGR;
  static constexpr int N = 1 << M;
  static constexpr int TPT = N / R;             // threads per sub-transform
  static constexpr int THREADS = TPC * TPT;
  static constexpr int NPASS = (M + LOGR - 1) / LOGR;
  static constexpr int PBASE = M / NPASS, PEXTRA = M % NPASS;
  static constexpr int SMEM_SLOTS = NPASS > 1 ? TPC * N : 0;
  // a sub-transform's threads sit in one warp
  static constexpr bool WARP_LOCAL = (MAP == MAP_CONTIG) && (TPT <= 32);
  static_assert(M >= 1 && LOGR >= 1 && LOGR <= M, "bad shape");

  __host__ __device__ static constexpr int bits(int p) { return PBASE + (p < PEXTRA ? 1 : 0); }
  __host__ __device__ static constexpr int start(int p) {
    return p * PBASE + (p < PEXTRA ? p : PEXTRA);
  }

  __device__ __forceinline__ static int sub_of(int tid) {
    return MAP == MAP_INTERLEAVED ? tid % TPC : tid / TPT;
  }
  __device__ __forceinline__ static int lane_of(int tid) {
    return MAP == MAP_INTERLEAVED ? tid / TPC : tid % TPT;
  }

  // shared-memory slot of element j of sub-transform `sub`
  __device__ __forceinline__ static int slot(int sub, int j) {
    if constexpr (MAP == MAP_INTERLEAVED) {
      return j * TPC + sub;
    } else {
      return swz((sub << M) | j);
    }
  }

  __device__ __forceinline__ static void sync() {
    if constexpr (WARP_LOCAL) __syncwarp();
    else __syncthreads();
  }

  // Contiguous tiles: linear index L of the tile -> slot.  The 8 lanes of one
  // quarter of a 16-byte access vary three bits of L, which ones depends on
  // the pass (bits lo.. of the group number skip the pass's own bits); adding
  // 3, 6 and 4 to the slot's low three bits for L's bits 3, 4 and 5 makes them
  // hit eight different banks for passes of 2 or 3 stages at every lo (with
  // L ^ ((L >> 3) & 7) the two-stage pass at lo = 2 hit four).
  __host__ __device__ static constexpr int swz(int l) {
    return M >= 3 ? l ^ (((l >> 3) ^ ((l >> 2) & 6)) & 7) : l;
  }
  // slot(sub, base | c) from sb = slot(sub, base) when base and c share no
  // bit and c is a constant (c = j << lo in a pass): the swizzle is linear
  // over XOR, so a contiguous tile's slot is sb ^ swz(c), with c above the
  // swizzled bits sb + c; for interleaved tiles the parts add.  One operation
  // per element at most, with the constant folded.
  __device__ __forceinline__ static int slot_at(int sb, int c) {
    if constexpr (MAP == MAP_INTERLEAVED) return sb + c * TPC;
    else return swz(c) == c && (c & 63) == 0 ? sb + c : sb ^ swz(c);
  }

  // Lowest local bit pass p touches.
  __host__ __device__ static constexpr int low(int p) { return M - start(p) - bits(p); }
  // Passes a and b exchange within each warp when both hold one group per
  // thread (r = LOGR) of a contiguous tile and both start at local bit 5 or
  // below: a warp's 32 consecutive groups then cover the indices whose bits
  // from 5 + LOGR up equal the warp's number, in both passes, so each warp
  // reads back only slots it wrote itself (the slot swizzle keeps indices in
  // their 8-aligned block).
  __host__ __device__ static constexpr bool warp_exchange(int a, int b) {
    return WARP_LOCAL || (MAP == MAP_CONTIG && bits(a) == LOGR && bits(b) == LOGR && low(a) <= 5 &&
                          low(b) <= 5);
  }
  template <int A, int B>
  __device__ __forceinline__ static void sync_between() {
    if constexpr (warp_exchange(A, B)) __syncwarp();
    else __syncthreads();
  }

  // The same, and whether `flag` is set in a thread that takes part.
  template <int A, int B>
  __device__ __forceinline__ static bool any_between(bool flag) {
    if constexpr (warp_exchange(A, B)) {
      __syncwarp();
      return __any_sync(0xFFFFFFFFu, flag);
    } else {
      return __syncthreads_or(flag) != 0;
    }
  }

  // Runs the whole sub-transform.  Every thread of the tile must call it
  // (it synchronises); threads whose sub-transform is not valid compute on
  // zeros and store nothing.
  template <int SRC = SRC_GLOBAL>
  __device__ __forceinline__ static void run(const SubRef& sr, int sub, int lane, uint4* smem,
                                             const ModParams& mp, int layout,
                                             const MulB& mb = MulB{}) {
    U128 v[R];
    if constexpr (Arith::kFast) {
      Table<SRC> tw;
      load_table<0, SRC>(tw, sr, lane);
      if constexpr (Table<SRC>::kAhead) pass_ahead<0, SRC>(v, sr, sub, lane, smem, mp, layout, mb, tw, false);
      else pass_lazy<0, SRC>(v, sr, sub, lane, smem, mp, layout, mb, tw, false);
    } else {
      pass<0>(v, sr, sub, lane, smem, mp, layout, mb);
    }
  }

  // The thread's table entries: with TW_AHEAD those of all passes in registers
  // (entry u of stage t of group i at (i << r) + 2^t - 1 + u), else none.
  template <int SRC>
  struct Table {
    static constexpr bool kAhead = (SRC & TW_AHEAD) != 0;
    uint4 at[kAhead ? NPASS : 1][kAhead ? R : 1];
  };
  __device__ __forceinline__ static uint32_t table_row(const SubRef& sr, int lane, int i, int s0, int lo) {
    return (sr.trow << s0) + (uint32_t)((lane + i * TPT) >> lo);
  }
  template <int P, int SRC>
  __device__ __forceinline__ static void load_table(Table<SRC>& a, const SubRef& sr, int lane) {
    if constexpr (Table<SRC>::kAhead) {
      constexpr int r = bits(P);
#pragma unroll
      for (int i = 0; i < (R >> r); ++i) {
        const uint32_t gt = table_row(sr, lane, i, start(P), low(P));
#pragma unroll
        for (int t = 0; t < r; ++t)
#pragma unroll
          for (int u = 0; u < (1 << t); ++u) a.at[P][(i << r) + (1 << t) - 1 + u] = tw_at(sr.tw, gt << t)[u];
      }
      if constexpr (P + 1 < NPASS) load_table<P + 1, SRC>(a, sr, lane);
    }
  }
  // entry u of stage t of group i in pass P; gt: the group's table_row
  template <int P, int SRC>
  __device__ __forceinline__ static U128 table_entry(const Table<SRC>& a, const SubRef& sr, uint32_t gt, int i, int t,
                                                     int u) {
    uint4 v;
    if constexpr (Table<SRC>::kAhead) {
      v = a.at[P][(i << bits(P)) + (1 << t) - 1 + u];
    } else {
      // tables are stored in limb order (LAYOUT_U128) by the plan
      const uint4* p = tw_at(sr.tw, gt << t) + u;  // u as an immediate offset
      if constexpr ((SRC & TW_SHARED) != 0) v = lds128(p);
      else if constexpr ((SRC & TW_CONST) != 0) v = __ldg(p);
      else v = *p;
    }
    return U128{{v.x, v.y, v.z, v.w}};
  }

  // Stages run on partly reduced values (u128.cuh) before pass p since they
  // were last brought back to 8q + [0, 2^124 + 2^32): by the first pass's
  // gather, or where one more pass would exceed kLazyStages.
  __host__ __device__ static constexpr int lazy_before(int p) {
    int a = 0;
    for (int i = 0; i < p; ++i) a = (a + bits(i) > kLazyStages ? 0 : a) + bits(i);
    return a;
  }
  __host__ __device__ static constexpr bool rebase(int p) { return lazy_before(p) + bits(p) > kLazyStages; }

  // Local index and slot of group i of pass P, and its elements before the pass.
  template <int P>
  __device__ __forceinline__ static int base_of(int lane, int i) {
    constexpr int lo = low(P);
    const int g = lane + i * TPT;
    return (g & ((1 << lo) - 1)) | ((g >> lo) << (lo + bits(P)));
  }
  template <int P, int SRC>
  __device__ __forceinline__ static U128 gather(const SubRef& sr, const uint4* smem, int layout, int base, int sb, int j) {
    if constexpr (P == 0 && (SRC & SRC_STAGED) != 0) {
      return from_mem(smem[slot_at(sb, j << low(P))], layout);  // staged in memory order
    } else if constexpr (P == 0) {
      if (!sr.valid) return U128{{0u, 0u, 0u, 0u}};
      const uint32_t lshift = MAP == MAP_CONTIG ? 0u : sr.lshift;  // L, 0 for contiguous tiles
      return from_mem(ld_data(sr.x + ((size_t)base << lshift) + (size_t)j * ((size_t)1 << (low(P) + lshift))), layout);
    } else {
      const uint4 t = smem[slot_at(sb, j << low(P))];
      return U128{{t.x, t.y, t.z, t.w}};
    }
  }
  // Element j of group i after the pass: to the next pass's slots, or to HBM
  // (times its element of b).
  template <int P>
  __device__ __forceinline__ static void scatter(const SubRef& sr, uint4* smem, int layout, const MulB& mb, uint32_t k,
                                                 int base, int sb, int j, const U128& e) {
    if constexpr (P == NPASS - 1) {
      if (!sr.valid) return;
      const uint32_t lshift = MAP == MAP_CONTIG ? 0u : sr.lshift;
      uint4* yp = sr.y + ((size_t)base << lshift) + (size_t)j * ((size_t)1 << (low(P) + lshift));
      U128 o = e;
      if (mb.b) {
        const uint4 bv = mb.b[(uint64_t)(yp - mb.ybase) & mb.bmask];
        o = reduce_once(mul_lazy(from_mem(bv, layout), o, k), k);
      }
      *yp = to_mem(o, layout);
    } else {
      smem[slot_at(sb, j << low(P))] = make_uint4(e.w[0], e.w[1], e.w[2], e.w[3]);
    }
  }

  // 0 where the first stage's sum of x and a product of y will be flagged because
  // both are zero, as their second limbs tell: 0 in the input, all ones in what an
  // exact pass left.
  template <int P>
  __device__ __forceinline__ static uint32_t zero_pair(const U128& x, const U128& y) {
    return P == 0 ? x.w[1] | y.w[1] : ~(x.w[1] & y.w[1]);
  }
  // Whether a lane of the warp holds such a pair among its elements of pass P.
  template <int P>
  __device__ __forceinline__ static bool warp_sees_zeros(const U128 (&v)[R], bool valid) {
    constexpr int G = 1 << bits(P);
    uint32_t seen = ~0u;
#pragma unroll
    for (int i = 0; i < R / G; ++i)
#pragma unroll
      for (int j = 0; j < G / 2; ++j) seen = min(seen, zero_pair<P>(v[i * G + j], v[i * G + j + G / 2]));
    return __any_sync(0xFFFFFFFFu, valid && seen == 0u);
  }

  // All of the thread's elements before pass P.
  template <int P, int SRC>
  __device__ __forceinline__ static void gather_pass(U128 (&v)[R], const SubRef& sr, int sub, int lane,
                                                     const uint4* smem, int layout) {
    constexpr int G = 1 << bits(P);
#pragma unroll
    for (int i = 0; i < R / G; ++i) {
      const int base = base_of<P>(lane, i), sb = slot(sub, base);
#pragma unroll
      for (int j = 0; j < G; ++j) v[i * G + j] = gather<P, SRC>(sr, smem, layout, base, sb, j);
    }
  }

  // The thread's part of pass P with the reference's butterflies, from its
  // gather to its scatter; with `look`, only if its warp holds a zero pair.
  // Returns whether it ran.  A function of its own, without register results, so
  // that the common path carries no registers for it (inlined in every pass it
  // cost 3 % of a plan transform and 6 % of the persistent kernel).
  template <int P, int SRC>
  __device__ __noinline__ static bool exact_pass(const SubRef sr, int sub, int lane, uint4* smem, uint32_t k, int layout,
                                                 const MulB mb, bool look) {
    constexpr int r = bits(P), G = 1 << r;
    if (look) {
      uint32_t seen = ~0u;
#pragma unroll 1
      for (int i = 0; i < R / G; ++i) {
        const int base = base_of<P>(lane, i), sb = slot(sub, base);
#pragma unroll
        for (int j = 0; j < G / 2; ++j)
          seen = min(seen, zero_pair<P>(gather<P, SRC>(sr, smem, layout, base, sb, j),
                                        gather<P, SRC>(sr, smem, layout, base, sb, j + G / 2)));
      }
      if (!__any_sync(0xFFFFFFFFu, sr.valid && seen == 0u)) return false;
    }
#pragma unroll 1
    for (int i = 0; i < R / G; ++i) {
      const int base = base_of<P>(lane, i), sb = slot(sub, base);
      const uint32_t gt = table_row(sr, lane, i, start(P), low(P));
      U128 e[G];
#pragma unroll
      for (int j = 0; j < G; ++j) {
        e[j] = gather<P, SRC>(sr, smem, layout, base, sb, j);
        if constexpr (P > 0) e[j] = lazy_value(e[j], k);
      }
      exact_stages<r, true>(e, [&](int t, int u) {
        const uint4 v = (tw_at(sr.tw, gt << t))[u];  // generic: the table may be in shared memory
        return U128{{v.x, v.y, v.z, v.w}};
      }, k);
#pragma unroll
      for (int j = 0; j < G; ++j)
        scatter<P>(sr, smem, layout, mb, k, base, sb, j, P == NPASS - 1 ? e[j] : add_8q(e[j], k));
    }
    return true;
  }

  // The stages of pass P on partly reduced values, in registers; whether the
  // pass has to be rerun with the reference's butterflies.  Only the elements
  // that the first stage adds to need a base of 8q; the ones it multiplies are
  // taken as they are.  STOP as in lazy_stages.
  template <int P, int SRC, bool STOP>
  __device__ __forceinline__ static bool lazy_pass(U128 (&v)[R], const SubRef& sr, int lane, uint32_t k,
                                                   const MulB& mb, const Table<SRC>& tw) {
    constexpr int r = bits(P), G = 1 << r;
    bool rerun = false;
#pragma unroll
    for (int i = 0; i < R / G; ++i) {
#pragma unroll
      for (int j = 0; j < G / 2; ++j) {
        U128& x = v[i * G + j];
        if constexpr (P == 0) x = add_8q(x, k);
        else if constexpr (rebase(P)) x = add_8q(fold_top(x, k), k);
      }
      const uint32_t gt = table_row(sr, lane, i, start(P), low(P));
      lazy_stages<r, STOP>(v, i * G, [&](int t, int u) { return table_entry<P, SRC>(tw, sr, gt, i, t, u); }, k, rerun,
                           sr.valid);
    }
    // the transform's outputs: below q unless the top limb says otherwise
    if constexpr (P == NPASS - 1) {
      if (!mb.b) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
          v[j] = fold_top(v[j], k);
          rerun |= v[j].w[3] >= 0x0FFFFFFFu;
        }
      }
    }
    return rerun && sr.valid;
  }

  // One pass of a fast modulus: lazy_pass, or the exact pass in its place.
  //
  // Where x and y of a butterfly are both zero, its sum looks like the corner
  // cases (all-zero, sparse and short-coefficient polynomials).  A warp that
  // finds such a pair takes the exact pass at once instead of running the stages
  // twice; after the first pass it looks only if a thread it exchanges with ran
  // an exact pass (`suspect`).  16,384 x 2^10, us: spread residues 281, their
  // upper half zero 281, ternary 338, 31 of 32 values zero 403, all zero 373 (334,
  // 343, 435 and 454 for the last four kinds when any zero multiplicand called for
  // the exact pass and zeros were multiplied; 431 for any values with the exact
  // butterflies throughout).  Testing whole groups for zeros takes all-zero inputs
  // to 157, and spread ones to 283.
  template <int P, int SRC>
  __device__ __forceinline__ static void pass_lazy(U128 (&v)[R], const SubRef& sr, int sub, int lane,
                                                   uint4* smem, const ModParams& mp, int layout,
                                                   const MulB& mb, const Table<SRC>& tw, bool suspect) {
    constexpr int r = bits(P);
    constexpr int G = 1 << r;             // elements per group
    constexpr int GPT = R / G;            // groups per thread
    static_assert(GPT >= 1, "pass wider than the register tile");
    static_assert(r <= kLazyStages, "pass wider than the partly reduced range");
    const uint32_t k = mp.k;

    bool ran = false;  // an exact pass
    if constexpr (P > 0) {
      if (__builtin_expect(suspect, 0)) ran = exact_pass<P, SRC>(sr, sub, lane, smem, k, layout, mb, true);
    }
    if (__builtin_expect(!ran, 1)) {
#pragma unroll
      for (int i = 0; i < GPT; ++i) {
        const int base = base_of<P>(lane, i), sb = slot(sub, base);
#pragma unroll
        for (int j = 0; j < G; ++j) v[i * G + j] = gather<P, SRC>(sr, smem, layout, base, sb, j);
      }
      bool exact = false;
      if constexpr (P == 0) exact = warp_sees_zeros<P>(v, sr.valid);
      if (__builtin_expect(!exact, 1)) exact = lazy_pass<P, SRC, false>(v, sr, lane, k, mb, tw);
      if (__builtin_expect(exact, 0)) {
        // the pass's inputs are still where they were gathered from
        ran = exact_pass<P, SRC>(sr, sub, lane, smem, k, layout, mb, false);
      } else {
#pragma unroll
        for (int i = 0; i < GPT; ++i) {
          const int base = base_of<P>(lane, i), sb = slot(sub, base);
#pragma unroll
          for (int j = 0; j < G; ++j) scatter<P>(sr, smem, layout, mb, k, base, sb, j, v[i * G + j]);
        }
      }
    }
    if constexpr (P + 1 < NPASS)
      pass_lazy<P + 1, SRC>(v, sr, sub, lane, smem, mp, layout, mb, tw, any_between<P, P + 1>(ran));
  }

  // The same for launches with TW_AHEAD, which wait for every load and have
  // registers to spare: the exact pass is inline, on the registers that hold the
  // table's entries.  Zeros are found where spread values do not pay for it: in
  // the first pass by the sums of its first stage (a look at the elements costs a
  // lone 2^10 transform 0.25 us, as the first butterflies then wait for every
  // load), later among the elements of a warp that ran an exact pass before.  One
  // transform of 2^10, us: spread 4.5, ternary 5.2, 31 of 32 values zero 6.4, all
  // zero 3.5 (4.4, 5.8, 8.6 and 10.6 when each pass was run twice, out of line;
  // 5.9 for any values with the exact butterflies throughout, which mostly zero
  // inputs do not quite reach: up to 1.13 of that for 4,096 x 2^5).
  template <int P, int SRC>
  __device__ __forceinline__ static void pass_ahead(U128 (&v)[R], const SubRef& sr, int sub, int lane,
                                                    uint4* smem, const ModParams& mp, int layout,
                                                    const MulB& mb, const Table<SRC>& tw, bool suspect) {
    constexpr int G = 1 << bits(P);
    static_assert(R >= G && bits(P) <= kLazyStages, "pass shape");
    const uint32_t k = mp.k;
    bool zeros = false, rerun = false;
    gather_pass<P, SRC>(v, sr, sub, lane, smem, layout);
    if constexpr (P > 0) zeros = suspect && warp_sees_zeros<P>(v, sr.valid);
    if (__builtin_expect(!zeros, 1)) rerun = lazy_pass<P, SRC, P == 0>(v, sr, lane, k, mb, tw);
    const bool ran = zeros || rerun;
    if (__builtin_expect(!ran, 1)) {
#pragma unroll
      for (int i = 0; i < R / G; ++i) {
        const int base = base_of<P>(lane, i), sb = slot(sub, base);
#pragma unroll
        for (int j = 0; j < G; ++j) scatter<P>(sr, smem, layout, mb, k, base, sb, j, v[i * G + j]);
      }
    } else {
      if (rerun) gather_pass<P, SRC>(v, sr, sub, lane, smem, layout);  // the inputs are still there
#pragma unroll
      for (int i = 0; i < R / G; ++i) {
        const int base = base_of<P>(lane, i), sb = slot(sub, base);
        U128 e[G];
#pragma unroll
        for (int j = 0; j < G; ++j) e[j] = P > 0 ? lazy_value(v[i * G + j], k) : v[i * G + j];
        uint32_t any = 0;
#pragma unroll
        for (int j = 0; j < G; ++j) any |= e[j].w[0] | e[j].w[1] | e[j].w[2] | e[j].w[3];
        if (any != 0u)  // a group of zeros stays one
          exact_stages<bits(P)>(e, [&](int t, int u) { return table_entry<P, SRC>(tw, sr, 0u, i, t, u); }, k);
#pragma unroll
        for (int j = 0; j < G; ++j)
          scatter<P>(sr, smem, layout, mb, k, base, sb, j, P == NPASS - 1 ? e[j] : add_8q(e[j], k));
      }
    }
    if constexpr (P + 1 < NPASS) {
      const bool next = __any_sync(0xFFFFFFFFu, ran);
      sync_between<P, P + 1>();
      pass_ahead<P + 1, SRC>(v, sr, sub, lane, smem, mp, layout, mb, tw, next);
    }
  }

  // One pass in the replica arithmetic (ArithRef).
  template <int P>
  __device__ __forceinline__ static void pass(U128 (&v)[R], const SubRef& sr, int sub, int lane,
                                              uint4* smem, const ModParams& mp, int layout,
                                              const MulB& mb) {
    constexpr int r = bits(P);
    constexpr int s0 = start(P);
    constexpr int lo = M - s0 - r;        // lowest local bit this pass touches
    constexpr int G = 1 << r;             // elements per group
    constexpr int GPT = R / G;            // groups per thread
    static_assert(GPT >= 1, "pass wider than the register tile");
    // element j of a group in HBM: the group's first element plus j * gstep
    const size_t gstep = (size_t)1 << (lo + sr.lshift);

    // ---- gather
#pragma unroll
    for (int i = 0; i < GPT; ++i) {
      const int g = lane + i * TPT;
      const int base = (g & ((1 << lo) - 1)) | ((g >> lo) << (lo + r));
      const int sb = slot(sub, base);
#pragma unroll
      for (int j = 0; j < G; ++j) {
        if constexpr (P == 0) {
          if (sr.valid) {
            v[i * G + j] = from_mem(ld_data(sr.x + ((size_t)base << sr.lshift) + (size_t)j * gstep), layout);
          } else {
#pragma unroll
            for (int w = 0; w < 4; ++w) v[i * G + j].w[w] = 0u;
          }
        } else {
          const uint4 t = smem[slot_at(sb, j << lo)];
          v[i * G + j] = U128{{t.x, t.y, t.z, t.w}};
        }
      }
    }

    // ---- r stages on each group
#pragma unroll
    for (int i = 0; i < GPT; ++i) {
      const int g = lane + i * TPT;
      const uint32_t gt = (sr.trow << s0) + (uint32_t)(g >> lo);
#pragma unroll
      for (int t = 0; t < r; ++t) {
        const int half = 1 << (r - 1 - t);
#pragma unroll
        for (int u = 0; u < (1 << t); ++u) {
          // tables are stored in limb order (LAYOUT_U128) by the plan
          const uint4* twt = sr.tw + (gt << t);  // u as an immediate offset
          const uint4 tv = twt[u];
          const U128 w = U128{{tv.x, tv.y, tv.z, tv.w}};
#pragma unroll
          for (int k = 0; k < half; ++k) {
            const int j = (u << (r - t)) | k;
            butterfly<Arith>(v[i * G + j], v[i * G + j + half], w, mp);
          }
        }
      }
    }

    // ---- scatter
#pragma unroll
    for (int i = 0; i < GPT; ++i) {
      const int g = lane + i * TPT;
      const int base = (g & ((1 << lo) - 1)) | ((g >> lo) << (lo + r));
      const int sb = slot(sub, base);
#pragma unroll
      for (int j = 0; j < G; ++j) {
        if constexpr (P == NPASS - 1) {
          if (sr.valid) {
            uint4* yp = sr.y + ((size_t)base << sr.lshift) + (size_t)j * gstep;
            U128 o = v[i * G + j];
            if (mb.b) {
              const uint4 bv = mb.b[(uint64_t)(yp - mb.ybase) & mb.bmask];
              o = Arith::mul(o, from_mem(bv, layout), mp);
            }
            *yp = to_mem(o, layout);
          }
        } else {
          const U128& e = v[i * G + j];
          smem[slot_at(sb, j << lo)] = make_uint4(e.w[0], e.w[1], e.w[2], e.w[3]);
        }
      }
    }
    if constexpr (P + 1 < NPASS) {
      sync_between<P, P + 1>();
      pass<P + 1>(v, sr, sub, lane, smem, mp, layout, mb);
    }
  }

  // The inverse network of the same passes: the last pass first, each pass's
  // stages in reverse order as Gentleman-Sande butterflies on the inverse
  // table, on partly reduced values (inverse_stages).  The store that finishes the transform (pass 0)
  // multiplies the lower half of each group -- the x outputs of stage 0 --
  // by *scale_at (N^-1) when scale_at is not null; the upper half gets N^-1
  // through the inverse table's entry 1.  Fast moduli only.
  template <int SRC = SRC_GLOBAL>
  __device__ __forceinline__ static void run_inv(const SubRef& sr, int sub, int lane, uint4* smem,
                                                 const ModParams& mp, int layout,
                                                 const uint4* scale_at) {
    U128 v[R];
    Table<SRC> tw;
    load_table<0, SRC>(tw, sr, lane);
    pass_inv<NPASS - 1, SRC>(v, sr, sub, lane, smem, mp, layout, scale_at, tw);
  }

  template <int P, int SRC>
  __device__ __forceinline__ static void pass_inv(U128 (&v)[R], const SubRef& sr, int sub, int lane,
                                                  uint4* smem, const ModParams& mp, int layout,
                                                  const uint4* scale_at, const Table<SRC>& tw) {
    constexpr int r = bits(P);
    constexpr int s0 = start(P);
    constexpr int lo = M - s0 - r;
    constexpr int G = 1 << r;
    constexpr int GPT = R / G;
    static_assert(GPT >= 1 && r <= 4, "pass shape");
    const uint32_t lshift = MAP == MAP_CONTIG ? 0u : sr.lshift;
    const size_t gstep = (size_t)1 << (lo + lshift);  // HBM distance of j and j + 1

    // ---- gather: the inverse reads its input in the last pass's order
#pragma unroll
    for (int i = 0; i < GPT; ++i) {
      const int g = lane + i * TPT;
      const int base = (g & ((1 << lo) - 1)) | ((g >> lo) << (lo + r));
      const int sb = slot(sub, base);
#pragma unroll
      for (int j = 0; j < G; ++j) {
        if constexpr (P == NPASS - 1) {
          if (sr.valid) {
            v[i * G + j] = from_mem(ld_data(sr.x + ((size_t)base << lshift) + (size_t)j * gstep), layout);
          } else {
#pragma unroll
            for (int w = 0; w < 4; ++w) v[i * G + j].w[w] = 0u;
          }
        } else {
          const uint4 t = smem[slot_at(sb, j << lo)];
          v[i * G + j] = U128{{t.x, t.y, t.z, t.w}};
        }
      }
    }

    // ---- r stages on each group, the last first
#pragma unroll
    for (int i = 0; i < GPT; ++i) {
      const uint32_t gt = table_row(sr, lane, i, s0, lo);
      inverse_stages<r, P == 0>(
          v, i * G, [&](int t, int u) { return table_entry<P, SRC>(tw, sr, gt, i, t, u); }, mp.k);
    }

    // ---- canonical results; N^-1 on the finishing store
    if constexpr (P == 0) {
      if (scale_at) {
        const uint4 f = *scale_at;
        const U128 fs = U128{{f.x, f.y, f.z, f.w}};
#pragma unroll
        for (int i = 0; i < GPT; ++i)
#pragma unroll
          for (int j = 0; j < G / 2; ++j) v[i * G + j] = mul_lazy(fs, v[i * G + j], mp.k);
      } else {
#pragma unroll
        for (int i = 0; i < GPT; ++i)
#pragma unroll
          for (int j = 0; j < G / 2; ++j) v[i * G + j] = fold_top(v[i * G + j], mp.k);
      }
#pragma unroll
      for (int j = 0; j < R; ++j) v[j] = reduce_once(v[j], mp.k);
    }

    // ---- scatter
#pragma unroll
    for (int i = 0; i < GPT; ++i) {
      const int g = lane + i * TPT;
      const int base = (g & ((1 << lo) - 1)) | ((g >> lo) << (lo + r));
      const int sb = slot(sub, base);
#pragma unroll
      for (int j = 0; j < G; ++j) {
        if constexpr (P == 0) {
          if (sr.valid) sr.y[((size_t)base << lshift) + (size_t)j * gstep] = to_mem(v[i * G + j], layout);
        } else {
          const U128& e = v[i * G + j];
          smem[slot_at(sb, j << lo)] = make_uint4(e.w[0], e.w[1], e.w[2], e.w[3]);
        }
      }
    }
    if constexpr (P > 0) {
      sync_between<P, P - 1>();
      pass_inv<P - 1, SRC>(v, sr, sub, lane, smem, mp, layout, scale_at, tw);
    }
  }
};

// Geometry of one launch over sub-transforms (see the header comment).
struct SubGeom {
  const uint4* x;
  uint4* y;
  const uint4* tw;
  uint32_t n;       // log2 of the whole transform
  uint32_t s0;      // first stage of this pass
  uint32_t m;       // stages in this pass
  uint32_t l;       // low bits below the pass bits
  uint64_t nsub;    // number of sub-transforms (all transforms of the batch)
  const uint4* b = nullptr;  // last pass only: fused pointwise product (MulB)
  uint64_t bmask = 0;
};

// Sub-transform `sid` of a geometry: sid = (transform << (S0 + L)) | (H << L) | c.
__device__ __forceinline__ SubRef make_subref(const SubGeom& g, uint64_t sid) {
  SubRef r;
  r.valid = sid < g.nsub;
  const uint64_t s = r.valid ? sid : 0;
  const uint64_t big = s >> (g.s0 + g.l);
  const uint64_t hbits = (s >> g.l) & ((1ull << g.s0) - 1);
  const uint64_t c = s & ((1ull << g.l) - 1);
  const uint64_t off = (big << g.n) + (hbits << (g.n - g.s0)) + c;
  r.x = g.x + off;
  r.y = g.y + off;
  r.tw = g.tw;
  r.trow = (1u << g.s0) + (uint32_t)hbits;
  r.lshift = g.l;
  return r;
}

// The same for contiguous sub-transforms (L = 0): sub-transform sid is the
// 2^M elements from sid << M on.
template <int M>
__device__ __forceinline__ SubRef make_subref_contig(const SubGeom& g, uint64_t sid) {
  SubRef r;
  r.valid = sid < g.nsub;
  const uint64_t s = r.valid ? sid : 0;
  r.x = g.x + (s << M);
  r.y = g.y + (s << M);
  r.tw = g.tw;
  r.trow = (1u << g.s0) + ((uint32_t)s & ((1u << g.s0) - 1u));
  r.lshift = 0;
  return r;
}

}  // namespace bntt
