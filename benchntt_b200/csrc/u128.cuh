// u128.cuh -- 128-bit modular arithmetic on sm_100a for the benchNTT hot path.
//
// A residue is four little-endian 32-bit limbs (w[0] least significant).
// In HBM an element is 16 bytes in one of two layouts:
//   HILO : the reference's u64 pair, high word first (src/config.c:29-30);
//          as u32 words: [hi.lo32, hi.hi32, lo.lo32, lo.hi32]
//   U128 : a native little-endian unsigned __int128 (the scalar API's
//          uint128_t arrays, src/ntt_scalar.c:582)
//
// Two multiply policies produce results bit-identical to the reference
// mulmod128 (src/ntt_scalar.c:173-199):
//   ArithFast -- q = 2^124 - k with k < 2^28 and mu = floor(2^251 / q) (both
//     reference primes and the NTT-friendly primes of roots.cu).  For such (q, mu) and operands below 2^124 the
//     reference's Barrett quotient is within one of the true quotient, so its
//     single conditional subtraction always lands in [0, q): the reference
//     returns exactly a*b mod q.  ArithFast computes that value with a
//     pseudo-Mersenne fold (2^128 == 16k, 2^124 == k mod q): 16 limb products
//     for a*b, 4 for the first fold, 1 for the second, one conditional
//     subtraction.  Its first operand must be below 2^124.
//   ArithRef  -- every other (q, mu): a replica of the reference's 64-bit word
//     data flow, including the points where it drops carries, so it matches
//     for arbitrary 128-bit inputs.
// add and sub are the reference's exact semantics in both policies,
// including addmod's two corner behaviours (see addmod_ref).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace bntt {

struct U128 {
  uint32_t w[4];
};

// Parameters of one modulus as the kernels see them.
struct ModParams {
  U128 q;        // modulus
  U128 mu;       // Barrett constant of the reference (used by ArithRef)
  uint32_t k;    // q = 2^124 - k (used by ArithFast)
  uint32_t pad[3];
};

enum Layout : int { LAYOUT_HILO = 0, LAYOUT_U128 = 1 };

__device__ __forceinline__ U128 from_mem(uint4 v, int layout) {
  U128 r;
  if (layout == LAYOUT_HILO) {
    r.w[0] = v.z; r.w[1] = v.w; r.w[2] = v.x; r.w[3] = v.y;
  } else {
    r.w[0] = v.x; r.w[1] = v.y; r.w[2] = v.z; r.w[3] = v.w;
  }
  return r;
}

__device__ __forceinline__ uint4 to_mem(const U128& a, int layout) {
  if (layout == LAYOUT_HILO) return make_uint4(a.w[2], a.w[3], a.w[0], a.w[1]);
  return make_uint4(a.w[0], a.w[1], a.w[2], a.w[3]);
}

// ---------------------------------------------------------------- add / sub

// Reference addmod128 (src/ntt_scalar.c:49-79).  s = a + b mod 2^128 and
// e = q - s mod 2^128; the borrow out of e is "s > q" (a strict test, so
// s == q is returned as q).  The reference assembles s - q from e's 64-bit
// words as (~e.hi, -e.lo): equal to s - q except when lo64(s) == lo64(q),
// where its high word comes out one lower.  This routine reproduces exactly
// that.
__device__ __forceinline__ U128 addmod_ref(const U128& a, const U128& b, const U128& q) {
  uint32_t s0, s1, s2, s3, e0, e1, e2, e3, gt;
  asm("add.cc.u32  %0, %9, %13;\n\t"
      "addc.cc.u32 %1, %10, %14;\n\t"
      "addc.cc.u32 %2, %11, %15;\n\t"
      "addc.u32    %3, %12, %16;\n\t"
      "sub.cc.u32  %4, %17, %0;\n\t"
      "subc.cc.u32 %5, %18, %1;\n\t"
      "subc.cc.u32 %6, %19, %2;\n\t"
      "subc.cc.u32 %7, %20, %3;\n\t"
      "subc.u32    %8, 0, 0;\n\t"
      : "=&r"(s0), "=&r"(s1), "=&r"(s2), "=&r"(s3), "=&r"(e0), "=&r"(e1), "=&r"(e2),
        "=&r"(e3), "=r"(gt)
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(b.w[0]), "r"(b.w[1]),
        "r"(b.w[2]), "r"(b.w[3]), "r"(q.w[0]), "r"(q.w[1]), "r"(q.w[2]), "r"(q.w[3]));
  uint32_t n0, n1;
  asm("sub.cc.u32 %0, 0, %2;\n\t"
      "subc.u32   %1, 0, %3;\n\t"
      : "=r"(n0), "=r"(n1)
      : "r"(e0), "r"(e1));
  U128 r;
  const bool sub = gt != 0u;
  r.w[0] = sub ? n0 : s0;
  r.w[1] = sub ? n1 : s1;
  r.w[2] = sub ? ~e2 : s2;
  r.w[3] = sub ? ~e3 : s3;
  return r;
}

// Reference submod128 (src/ntt_scalar.c:81-104): d = a - b, plus q on borrow.
__device__ __forceinline__ U128 submod_ref(const U128& a, const U128& b, const U128& q) {
  uint32_t d0, d1, d2, d3, bw;
  asm("sub.cc.u32  %0, %5, %9;\n\t"
      "subc.cc.u32 %1, %6, %10;\n\t"
      "subc.cc.u32 %2, %7, %11;\n\t"
      "subc.cc.u32 %3, %8, %12;\n\t"
      "subc.u32    %4, 0, 0;\n\t"
      : "=&r"(d0), "=&r"(d1), "=&r"(d2), "=&r"(d3), "=r"(bw)
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(b.w[0]), "r"(b.w[1]),
        "r"(b.w[2]), "r"(b.w[3]));
  // add (q & borrow-mask): one chain, no select
  uint32_t m0 = q.w[0] & bw, m1 = q.w[1] & bw, m2 = q.w[2] & bw, m3 = q.w[3] & bw;
  U128 r;
  asm("add.cc.u32  %0, %4, %8;\n\t"
      "addc.cc.u32 %1, %5, %9;\n\t"
      "addc.cc.u32 %2, %6, %10;\n\t"
      "addc.u32    %3, %7, %11;\n\t"
      : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3])
      : "r"(d0), "r"(d1), "r"(d2), "r"(d3), "r"(m0), "r"(m1), "r"(m2), "r"(m3));
  return r;
}

// The same two operations for q = 2^124 - k with k < 2^31, whose limbs are
// (2^32 - k, 0xFFFFFFFF, 0xFFFFFFFF, 0x0FFFFFFF): three of them become
// immediates, which frees registers in the butterfly loops.
__device__ __forceinline__ U128 addmod_pm(const U128& a, const U128& b, uint32_t q0) {
  uint32_t s0, s1, s2, s3, e0, e1, e2, e3, gt;
  asm("add.cc.u32  %0, %9, %13;\n\t"
      "addc.cc.u32 %1, %10, %14;\n\t"
      "addc.cc.u32 %2, %11, %15;\n\t"
      "addc.u32    %3, %12, %16;\n\t"
      "sub.cc.u32  %4, %17, %0;\n\t"
      "subc.cc.u32 %5, 0xFFFFFFFF, %1;\n\t"
      "subc.cc.u32 %6, 0xFFFFFFFF, %2;\n\t"
      "subc.cc.u32 %7, 0x0FFFFFFF, %3;\n\t"
      "subc.u32    %8, 0, 0;\n\t"
      : "=&r"(s0), "=&r"(s1), "=&r"(s2), "=&r"(s3), "=&r"(e0), "=&r"(e1), "=&r"(e2),
        "=&r"(e3), "=r"(gt)
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(b.w[0]), "r"(b.w[1]),
        "r"(b.w[2]), "r"(b.w[3]), "r"(q0));
  uint32_t n0, n1;
  asm("sub.cc.u32 %0, 0, %2;\n\t"
      "subc.u32   %1, 0, %3;\n\t"
      : "=r"(n0), "=r"(n1)
      : "r"(e0), "r"(e1));
  U128 r;
  const bool sub = gt != 0u;
  r.w[0] = sub ? n0 : s0;
  r.w[1] = sub ? n1 : s1;
  r.w[2] = sub ? ~e2 : s2;
  r.w[3] = sub ? ~e3 : s3;
  return r;
}

__device__ __forceinline__ U128 submod_pm(const U128& a, const U128& b, uint32_t q0) {
  uint32_t d0, d1, d2, d3, bw;
  asm("sub.cc.u32  %0, %5, %9;\n\t"
      "subc.cc.u32 %1, %6, %10;\n\t"
      "subc.cc.u32 %2, %7, %11;\n\t"
      "subc.cc.u32 %3, %8, %12;\n\t"
      "subc.u32    %4, 0, 0;\n\t"
      : "=&r"(d0), "=&r"(d1), "=&r"(d2), "=&r"(d3), "=r"(bw)
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(b.w[0]), "r"(b.w[1]),
        "r"(b.w[2]), "r"(b.w[3]));
  U128 r;
  asm("add.cc.u32  %0, %4, %8;\n\t"
      "addc.cc.u32 %1, %5, %9;\n\t"
      "addc.cc.u32 %2, %6, %9;\n\t"
      "addc.u32    %3, %7, %10;\n\t"
      : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3])
      : "r"(d0), "r"(d1), "r"(d2), "r"(d3), "r"(q0 & bw), "r"(bw), "r"(bw & 0x0FFFFFFFu));
  return r;
}

// ------------------------------------------------------------------ ArithFast

// a * b mod q up to a multiple of q, for q = 2^124 - k, k < 2^28: the result r
// is congruent to a * b and 0 <= r < 2^124 + 2^60.  a < 2^124; b is any value
// below 2^128 - 2^101 (a partly reduced one included).
//
// The product's 16 partial products are summed in two columns of 64-bit
// accumulators, E at the even limbs and O at the odd ones, so that every
// partial product is one 32 x 32 + 64-bit multiply-add whose carry runs into
// the next one of its column (each mad.lo.cc / madc.hi.cc pair on one pair of
// limbs).  P = E + O*2^32 is never put together: the upper parts are added,
// H = E / 2^128 + O / 2^96, and the two lower parts take the first fold
// separately, 2^128 = 16 * 2^124 == 16k (mod q):
//   t = E mod 2^128 + (O mod 2^96)*2^32 + H*16k      (< 2^156: 5 limbs)
//   r = t mod 2^124 + (t >> 124)*k
// What bounds it: the multiply-add pipe, on which a 32 x 32 + 64-bit
// multiply-add takes 4 cycles per warp and scheduler and other integer
// instructions there 2 (measured: 31 wide products per clock and SM against
// 64 mad.lo).  This form has 21 wide multiply-adds (16 + 4 + 1) and about 20
// other instructions; the product on 64-bit halves in C++ with the folds as
// separate lo and hi rows had 22 and about 50.  In the register-only
// butterfly probe with the exact add and sub: 233 -> 287 G butterflies/s.
// Carries out of a column (c5, c6, c7) are added to H at the end; as
// zero-extended accumulators of the next row they cost moves on the same pipe
// (349 against 354 G/s in the probe without exact add and sub).
__device__ __forceinline__ U128 mul_lazy(const U128& a, const U128& b, uint32_t k) {
  uint32_t e0, e1, e2, e3, e4, e5, e6, e7, o1, o2, o3, o4, o5, o6, c5, c6, c7;
  // limb 0 of a: E at 0 and 2, O at 1 and 3
  asm("mul.lo.u32 %0, %4, %5;\n\t"
      "mul.hi.u32 %1, %4, %5;\n\t"
      "mul.lo.u32 %2, %4, %6;\n\t"
      "mul.hi.u32 %3, %4, %6;\n\t"
      : "=&r"(e0), "=&r"(e1), "=&r"(e2), "=&r"(e3)
      : "r"(a.w[0]), "r"(b.w[0]), "r"(b.w[2]));
  asm("mul.lo.u32 %0, %4, %5;\n\t"
      "mul.hi.u32 %1, %4, %5;\n\t"
      "mul.lo.u32 %2, %4, %6;\n\t"
      "mul.hi.u32 %3, %4, %6;\n\t"
      : "=&r"(o1), "=&r"(o2), "=&r"(o3), "=&r"(o4)
      : "r"(a.w[0]), "r"(b.w[1]), "r"(b.w[3]));
  // limb 1: O at 1 and 3, E at 2 and 4
  asm("mad.lo.cc.u32  %0, %5, %6, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %5, %7, %3;\n\t"
      "addc.u32       %4, 0, 0;\n\t"
      : "+r"(o1), "+r"(o2), "+r"(o3), "+r"(o4), "=r"(c5)
      : "r"(a.w[1]), "r"(b.w[0]), "r"(b.w[2]));
  asm("mad.lo.cc.u32  %0, %4, %5, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %4, %6, 0;\n\t"
      "madc.hi.u32    %3, %4, %6, 0;\n\t"
      : "+r"(e2), "+r"(e3), "=&r"(e4), "=&r"(e5)
      : "r"(a.w[1]), "r"(b.w[1]), "r"(b.w[3]));
  // limb 2: E at 2 and 4, O at 3 and 5
  asm("mad.lo.cc.u32  %0, %5, %6, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %5, %7, %3;\n\t"
      "addc.u32       %4, 0, 0;\n\t"
      : "+r"(e2), "+r"(e3), "+r"(e4), "+r"(e5), "=r"(c6)
      : "r"(a.w[2]), "r"(b.w[0]), "r"(b.w[2]));
  asm("mad.lo.cc.u32  %0, %4, %5, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %4, %6, 0;\n\t"
      "madc.hi.u32    %3, %4, %6, 0;\n\t"
      : "+r"(o3), "+r"(o4), "=&r"(o5), "=&r"(o6)
      : "r"(a.w[2]), "r"(b.w[1]), "r"(b.w[3]));
  // limb 3: O at 3 and 5, E at 4 and 6
  asm("mad.lo.cc.u32  %0, %5, %6, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %5, %7, %3;\n\t"
      "addc.u32       %4, 0, 0;\n\t"
      : "+r"(o3), "+r"(o4), "+r"(o5), "+r"(o6), "=r"(c7)
      : "r"(a.w[3]), "r"(b.w[0]), "r"(b.w[2]));
  asm("mad.lo.cc.u32  %0, %4, %5, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %4, %6, 0;\n\t"
      "madc.hi.u32    %3, %4, %6, 0;\n\t"
      : "+r"(e4), "+r"(e5), "=&r"(e6), "=&r"(e7)
      : "r"(a.w[3]), "r"(b.w[1]), "r"(b.w[3]));
  // H = upper parts and the carries at limbs 5, 6 and 7 (H <= P / 2^128)
  uint32_t h0, h1, h2, h3;
  asm("add.cc.u32  %0, %4, %8;\n\t"
      "addc.cc.u32 %1, %5, %9;\n\t"
      "addc.cc.u32 %2, %6, %10;\n\t"
      "addc.u32    %3, %7, %11;\n\t"
      : "=&r"(h0), "=&r"(h1), "=&r"(h2), "=&r"(h3)
      : "r"(e4), "r"(e5), "r"(e6), "r"(e7), "r"(o4), "r"(o5), "r"(o6), "r"(c7));
  asm("add.cc.u32  %0, %0, %3;\n\t"
      "addc.cc.u32 %1, %1, %4;\n\t"
      "addc.u32    %2, %2, 0;\n\t"
      : "+r"(h1), "+r"(h2), "+r"(h3)
      : "r"(c5), "r"(c6));
  // first fold, by column, then the columns together
  const uint32_t c = k << 4;
  uint32_t t1, t2, t3, t4, u4;
  asm("mad.lo.cc.u32  %0, %5, %7, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %7, %1;\n\t"
      "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %6, %7, %3;\n\t"
      "addc.u32       %4, 0, 0;\n\t"
      : "+r"(e0), "+r"(e1), "+r"(e2), "+r"(e3), "=r"(t4)
      : "r"(h0), "r"(h2), "r"(c));
  asm("mad.lo.cc.u32  %0, %4, %6, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %6, %2;\n\t"
      "madc.hi.u32    %3, %5, %6, 0;\n\t"
      : "+r"(o1), "+r"(o2), "+r"(o3), "=&r"(u4)
      : "r"(h1), "r"(h3), "r"(c));
  asm("add.cc.u32  %0, %4, %7;\n\t"
      "addc.cc.u32 %1, %5, %8;\n\t"
      "addc.cc.u32 %2, %6, %9;\n\t"
      "addc.u32    %3, %10, %11;\n\t"
      : "=&r"(t1), "=&r"(t2), "=&r"(t3), "=&r"(t4)
      : "r"(e1), "r"(e2), "r"(e3), "r"(o1), "r"(o2), "r"(o3), "r"(t4), "r"(u4));
  // second fold
  const uint32_t h = __funnelshift_r(t3, t4, 28);  // t >> 124
  U128 r;
  asm("mad.lo.cc.u32  %0, %4, %5, %6;\n\t"
      "madc.hi.cc.u32 %1, %4, %5, %7;\n\t"
      "addc.cc.u32    %2, %8, 0;\n\t"
      "addc.u32       %3, %9, 0;\n\t"
      : "=&r"(r.w[0]), "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3])
      : "r"(h), "r"(k), "r"(e0), "r"(t1), "r"(t2), "r"(t3 & 0x0FFFFFFFu));
  return r;
}

// r < 2^124 + 2^60 -> [0, q): r less q when r >= q, tested as bit 124 of
// r + k.  r >= q needs r's top limb at least 0x0FFFFFFF, about one case in
// 2^28 for spread residues, so the exact test and the subtraction sit behind
// a branch.
__device__ __forceinline__ U128 reduce_once(U128 r, uint32_t k) {
  if (__builtin_expect(r.w[3] >= 0x0FFFFFFFu, 0)) {  // r >= q is possible only here
    uint32_t s0, s1, s2, s3;
    asm("add.cc.u32  %0, %4, %8;\n\t"
        "addc.cc.u32 %1, %5, 0;\n\t"
        "addc.cc.u32 %2, %6, 0;\n\t"
        "addc.u32    %3, %7, 0;\n\t"
        : "=&r"(s0), "=&r"(s1), "=&r"(s2), "=&r"(s3)
        : "r"(r.w[0]), "r"(r.w[1]), "r"(r.w[2]), "r"(r.w[3]), "r"(k));
    if (s3 >> 28) {  // r + k >= 2^124, i.e. r >= q
      r.w[0] = s0; r.w[1] = s1; r.w[2] = s2; r.w[3] = s3 & 0x0FFFFFFFu;
    }
  }
  return r;
}

struct ArithFast {
  static constexpr bool kFast = true;
  __device__ __forceinline__ static U128 mul(const U128& a, const U128& b, const ModParams& m) {
    return reduce_once(mul_lazy(a, b, m.k), m.k);
  }
};

// ------------------------------------------------------------------- ArithRef

struct W128 {
  uint64_t hi, lo;
};

__device__ __forceinline__ W128 w_add(W128 a, W128 b) {  // mod 2^128
  W128 r;
  r.lo = a.lo + b.lo;
  r.hi = a.hi + b.hi + (r.lo < a.lo ? 1ull : 0ull);
  return r;
}
__device__ __forceinline__ W128 w_mul64(uint64_t a, uint64_t b) {
  return W128{__umul64hi(a, b), a * b};
}
__device__ __forceinline__ W128 to_w(const U128& a) {
  return W128{((uint64_t)a.w[3] << 32) | a.w[2], ((uint64_t)a.w[1] << 32) | a.w[0]};
}
__device__ __forceinline__ U128 from_w(W128 a) {
  U128 r;
  r.w[0] = (uint32_t)a.lo; r.w[1] = (uint32_t)(a.lo >> 32);
  r.w[2] = (uint32_t)a.hi; r.w[3] = (uint32_t)(a.hi >> 32);
  return r;
}

// Reference mulmod128 with MBITS = 124, word for word: the 128x128 product
// keeps its middle sum to 128 bits (src/ntt_scalar.c:106-128), the high
// product of the quotient estimate likewise (:151-171), the low product keeps
// its cross terms to 64 bits (:130-149), and one conditional subtraction ends
// it (:194-196).
inline __device__ __noinline__ U128 mulmod_words(const U128 ua, const U128 ub, const U128 uq, const U128 umu) {
  const W128 a = to_w(ua), b = to_w(ub), q = to_w(uq), mu = to_w(umu);
  // product
  W128 p00 = w_mul64(a.lo, b.lo), p01 = w_mul64(a.lo, b.hi);
  W128 p10 = w_mul64(a.hi, b.lo), p11 = w_mul64(a.hi, b.hi);
  W128 mid = w_add(w_add(p01, p10), W128{0, p00.hi});
  W128 ph = w_add(p11, W128{0, mid.hi});
  W128 pl = W128{mid.lo, p00.lo};
  // quotient estimate from bits 122.. of the product
  // t = (P >> 122) mod 2^128 = (ph << 6) | (pl >> 122)
  W128 t = W128{(ph.hi << 6) | (ph.lo >> 58), (ph.lo << 6) | (pl.hi >> 58)};
  uint64_t top = ph.hi >> 58;
  W128 m01 = w_mul64(t.lo, mu.hi), m10 = w_mul64(t.hi, mu.lo), m11 = w_mul64(t.hi, mu.hi);
  W128 mm = w_add(w_add(m01, m10), W128{0, __umul64hi(t.lo, mu.lo)});
  W128 qm = w_add(w_add(m11, W128{0, mm.hi}), W128{0, top * mu.lo});
  W128 qq = W128{qm.hi >> 1, (qm.lo >> 1) | (qm.hi << 63)};
  // low product qq*q
  W128 l00 = w_mul64(qq.lo, q.lo);
  uint64_t cross = qq.lo * q.hi + qq.hi * q.lo + l00.hi;
  W128 qql = W128{cross, l00.lo};
  // r = pl - qql mod 2^128
  W128 r;
  r.lo = pl.lo - qql.lo;
  r.hi = pl.hi - qql.hi - (pl.lo < qql.lo ? 1ull : 0ull);
  const bool lt = (r.hi < q.hi) || (r.hi == q.hi && r.lo < q.lo);
  if (!lt) {
    uint64_t lo2 = r.lo - q.lo;
    r.hi = r.hi - q.hi - (r.lo < q.lo ? 1ull : 0ull);
    r.lo = lo2;
  }
  return from_w(r);
}

// The two columns of a 128 x 128-bit product (see mul_lazy): E at limbs 0..7
// in e, O at limbs 1..7 in o[1..7], P = E + O*2^32 with the carries out of the
// columns already in.
__device__ __forceinline__ void mul_columns(const U128& a, const U128& b, uint32_t (&e)[8], uint32_t (&o)[8]) {
  asm("mul.lo.u32 %0, %4, %5;\n\t"
      "mul.hi.u32 %1, %4, %5;\n\t"
      "mul.lo.u32 %2, %4, %6;\n\t"
      "mul.hi.u32 %3, %4, %6;\n\t"
      : "=&r"(e[0]), "=&r"(e[1]), "=&r"(e[2]), "=&r"(e[3])
      : "r"(a.w[0]), "r"(b.w[0]), "r"(b.w[2]));
  asm("mul.lo.u32 %0, %4, %5;\n\t"
      "mul.hi.u32 %1, %4, %5;\n\t"
      "mul.lo.u32 %2, %4, %6;\n\t"
      "mul.hi.u32 %3, %4, %6;\n\t"
      : "=&r"(o[1]), "=&r"(o[2]), "=&r"(o[3]), "=&r"(o[4])
      : "r"(a.w[0]), "r"(b.w[1]), "r"(b.w[3]));
  asm("mad.lo.cc.u32  %0, %5, %6, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %5, %7, %3;\n\t"
      "addc.u32       %4, 0, 0;\n\t"
      : "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "=r"(o[5])
      : "r"(a.w[1]), "r"(b.w[0]), "r"(b.w[2]));
  asm("mad.lo.cc.u32  %0, %4, %5, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %4, %6, 0;\n\t"
      "madc.hi.u32    %3, %4, %6, 0;\n\t"
      : "+r"(e[2]), "+r"(e[3]), "=&r"(e[4]), "=&r"(e[5])
      : "r"(a.w[1]), "r"(b.w[1]), "r"(b.w[3]));
  asm("mad.lo.cc.u32  %0, %5, %6, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %5, %7, %3;\n\t"
      "addc.u32       %4, 0, 0;\n\t"
      : "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "=r"(e[6])
      : "r"(a.w[2]), "r"(b.w[0]), "r"(b.w[2]));
  asm("mad.lo.cc.u32  %0, %4, %5, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %4, %6, %2;\n\t"
      "madc.hi.u32    %3, %4, %6, 0;\n\t"
      : "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "=&r"(o[6])
      : "r"(a.w[2]), "r"(b.w[1]), "r"(b.w[3]));
  asm("mad.lo.cc.u32  %0, %5, %6, %0;\n\t"
      "madc.hi.cc.u32 %1, %5, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %5, %7, %3;\n\t"
      "addc.u32       %4, 0, 0;\n\t"
      : "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "=r"(o[7])
      : "r"(a.w[3]), "r"(b.w[0]), "r"(b.w[2]));
  asm("mad.lo.cc.u32  %0, %4, %5, %0;\n\t"
      "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %4, %6, %2;\n\t"
      "madc.hi.u32    %3, %4, %6, 0;\n\t"
      : "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "=&r"(e[7])
      : "r"(a.w[3]), "r"(b.w[1]), "r"(b.w[3]));
}

// mulmod_words on 32-bit limbs with the carries inside the multiply-adds, for
// operands below 2^127 (their middle sum cannot leave 128 bits; larger ones
// take mulmod_words).  38 wide products and about 70 other instructions,
// where the 64-bit words' products (each a low and a high product of their
// own) cost about twice that.  The quotient estimate's middle sum M is kept
// to 128 bits as in the reference: the carry out of its top limb is dropped.
struct ArithRef {
  static constexpr bool kFast = false;
  __device__ __forceinline__ static U128 mul(const U128& a, const U128& b, const ModParams& m) {
    if (__builtin_expect((a.w[3] | b.w[3]) >> 31, 0)) return mulmod_words(a, b, m.q, m.mu);
    uint32_t p[8];  // the product
    {
      uint32_t e[8], o[8];
      mul_columns(a, b, e, o);
      p[0] = e[0];
      asm("add.cc.u32  %0, %7, %14;\n\t"
          "addc.cc.u32 %1, %8, %15;\n\t"
          "addc.cc.u32 %2, %9, %16;\n\t"
          "addc.cc.u32 %3, %10, %17;\n\t"
          "addc.cc.u32 %4, %11, %18;\n\t"
          "addc.cc.u32 %5, %12, %19;\n\t"
          "addc.u32    %6, %13, %20;\n\t"
          : "=&r"(p[1]), "=&r"(p[2]), "=&r"(p[3]), "=&r"(p[4]), "=&r"(p[5]), "=&r"(p[6]), "=&r"(p[7])
          : "r"(e[1]), "r"(e[2]), "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]), "r"(o[1]), "r"(o[2]),
            "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]));
    }
    // t = (P >> 122) mod 2^128; the 6 bits above it
    uint32_t t[4], top = p[7] >> 26;
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = __funnelshift_r(p[3 + i], p[4 + i], 26);
    const uint32_t* u = m.mu.w;
    // limbs 2 and 3 of t_lo * mu_lo
    uint32_t c1, c2, c3;
    {
      uint32_t e1, e2, e3, o1, o2, o3;
      asm("mul.hi.u32 %0, %1, %2;\n\t" : "=r"(e1) : "r"(t[0]), "r"(u[0]));
      asm("mul.lo.u32 %0, %4, %6;\n\t"
          "mul.hi.u32 %1, %4, %6;\n\t"
          "mul.lo.u32 %2, %5, %6;\n\t"
          "mul.hi.u32 %3, %5, %6;\n\t"
          : "=&r"(o1), "=&r"(o2), "=&r"(e2), "=&r"(e3)
          : "r"(t[0]), "r"(t[1]), "r"(u[1]));
      asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
          "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
          "addc.u32       %2, 0, 0;\n\t"
          : "+r"(o1), "+r"(o2), "=r"(o3)
          : "r"(t[1]), "r"(u[0]));
      asm("add.cc.u32  %0, %3, %6;\n\t"
          "addc.cc.u32 %1, %4, %7;\n\t"
          "addc.u32    %2, %5, %8;\n\t"
          : "=&r"(c1), "=&r"(c2), "=&r"(c3)
          : "r"(e1), "r"(e2), "r"(e3), "r"(o1), "r"(o2), "r"(o3));
    }
    // M = that + t_lo * mu_hi + t_hi * mu_lo at limbs 2..5, columns E (2, 4)
    // and O (3, 5); carries out of limb 5 are dropped
    uint32_t e4, e5, o3, o4, o5;
    asm("mad.lo.cc.u32  %0, %4, %5, %0;\n\t"
        "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
        "madc.lo.cc.u32 %2, %6, %7, 0;\n\t"
        "madc.hi.u32    %3, %6, %7, 0;\n\t"
        : "+r"(c2), "+r"(c3), "=&r"(e4), "=&r"(e5)
        : "r"(t[0]), "r"(u[2]), "r"(t[1]), "r"(u[3]));
    asm("mad.lo.cc.u32  %0, %4, %5, %0;\n\t"
        "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
        "madc.lo.cc.u32 %2, %6, %7, %2;\n\t"
        "madc.hi.u32    %3, %6, %7, %3;\n\t"
        : "+r"(c2), "+r"(c3), "+r"(e4), "+r"(e5)
        : "r"(t[2]), "r"(u[0]), "r"(t[3]), "r"(u[1]));
    asm("mul.lo.u32 %0, %2, %3;\n\t"
        "mul.hi.u32 %1, %2, %3;\n\t"
        : "=&r"(o3), "=&r"(o4)
        : "r"(t[0]), "r"(u[3]));
    asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32       %2, 0, 0;\n\t"
        : "+r"(o3), "+r"(o4), "=r"(o5)
        : "r"(t[1]), "r"(u[2]));
    asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32       %2, %2, 0;\n\t"
        : "+r"(o3), "+r"(o4), "+r"(o5)
        : "r"(t[2]), "r"(u[1]));
    asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32       %2, %2, 0;\n\t"
        : "+r"(o3), "+r"(o4), "+r"(o5)
        : "r"(t[3]), "r"(u[0]));
    uint32_t m4, m5;
    asm("{\n\t.reg .u32 lim3;\n\t"
        "add.cc.u32  lim3, %2, %5;\n\t"
        "addc.cc.u32 %0, %3, %6;\n\t"
        "addc.u32    %1, %4, %7;\n\t}"
        : "=&r"(m4), "=&r"(m5)
        : "r"(c3), "r"(e4), "r"(e5), "r"(o3), "r"(o4), "r"(o5));
    // Q = t_hi * mu_hi + M's high word + top * mu_lo, at limbs 4..7
    uint32_t q4, q5, q6, q7, r5, r6, r7;
    asm("mad.lo.cc.u32  %0, %4, %5, %8;\n\t"
        "madc.hi.cc.u32 %1, %4, %5, %9;\n\t"
        "madc.lo.cc.u32 %2, %6, %7, 0;\n\t"
        "madc.hi.u32    %3, %6, %7, 0;\n\t"
        : "=&r"(q4), "=&r"(q5), "=&r"(q6), "=&r"(q7)
        : "r"(t[2]), "r"(u[2]), "r"(t[3]), "r"(u[3]), "r"(m4), "r"(m5));
    asm("mul.lo.u32 %0, %2, %3;\n\t"
        "mul.hi.u32 %1, %2, %3;\n\t"
        : "=&r"(r5), "=&r"(r6)
        : "r"(t[2]), "r"(u[3]));
    asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32       %2, 0, 0;\n\t"
        : "+r"(r5), "+r"(r6), "=r"(r7)
        : "r"(t[3]), "r"(u[2]));
    asm("add.cc.u32  %0, %0, %3;\n\t"
        "addc.cc.u32 %1, %1, %4;\n\t"
        "addc.u32    %2, %2, %5;\n\t"
        : "+r"(q5), "+r"(q6), "+r"(q7)
        : "r"(r5), "r"(r6), "r"(r7));
    if (__builtin_expect(top != 0u, 0)) {  // P >= 2^250
      const uint64_t x = (uint64_t)top * (((uint64_t)u[1] << 32) | u[0]);
      asm("add.cc.u32  %0, %0, %4;\n\t"
          "addc.cc.u32 %1, %1, %5;\n\t"
          "addc.cc.u32 %2, %2, 0;\n\t"
          "addc.u32    %3, %3, 0;\n\t"
          : "+r"(q4), "+r"(q5), "+r"(q6), "+r"(q7)
          : "r"((uint32_t)x), "r"((uint32_t)(x >> 32)));
    }
    // (Q >> 1) * q mod 2^128
    const uint32_t h0 = __funnelshift_r(q4, q5, 1), h1 = __funnelshift_r(q5, q6, 1),
                   h2 = __funnelshift_r(q6, q7, 1), h3 = q7 >> 1;
    const uint32_t* q = m.q.w;
    uint32_t l0, l1, l2, l3, s1, s2, s3;
    asm("mul.lo.u32 %0, %4, %6;\n\t"
        "mul.hi.u32 %1, %4, %6;\n\t"
        "mul.lo.u32 %2, %5, %7;\n\t"
        "mul.hi.u32 %3, %5, %7;\n\t"
        : "=&r"(l0), "=&r"(l1), "=&r"(l2), "=&r"(l3)
        : "r"(h0), "r"(h1), "r"(q[0]), "r"(q[1]));
    asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\t"
        "madc.hi.u32   %1, %2, %3, %1;\n\t"
        : "+r"(l2), "+r"(l3)
        : "r"(h0), "r"(q[2]));
    asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\t"
        "madc.hi.u32   %1, %2, %3, %1;\n\t"
        : "+r"(l2), "+r"(l3)
        : "r"(h2), "r"(q[0]));
    asm("mul.lo.u32 %0, %2, %3;\n\t"
        "mul.hi.u32 %1, %2, %3;\n\t"
        : "=&r"(s1), "=&r"(s2)
        : "r"(h0), "r"(q[1]));
    asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32       %2, 0, 0;\n\t"
        : "+r"(s1), "+r"(s2), "=r"(s3)
        : "r"(h1), "r"(q[0]));
    s3 += h0 * q[3] + h1 * q[2] + h2 * q[1] + h3 * q[0];
    asm("add.cc.u32  %0, %0, %3;\n\t"
        "addc.cc.u32 %1, %1, %4;\n\t"
        "addc.u32    %2, %2, %5;\n\t"
        : "+r"(l1), "+r"(l2), "+r"(l3)
        : "r"(s1), "r"(s2), "r"(s3));
    // r = P - that mod 2^128, less q unless r < q
    U128 r;
    uint32_t d0, d1, d2, d3, lt;
    asm("sub.cc.u32  %0, %4, %8;\n\t"
        "subc.cc.u32 %1, %5, %9;\n\t"
        "subc.cc.u32 %2, %6, %10;\n\t"
        "subc.u32    %3, %7, %11;\n\t"
        : "=&r"(r.w[0]), "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3])
        : "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]), "r"(l0), "r"(l1), "r"(l2), "r"(l3));
    asm("sub.cc.u32  %0, %5, %9;\n\t"
        "subc.cc.u32 %1, %6, %10;\n\t"
        "subc.cc.u32 %2, %7, %11;\n\t"
        "subc.cc.u32 %3, %8, %12;\n\t"
        "subc.u32    %4, 0, 0;\n\t"
        : "=&r"(d0), "=&r"(d1), "=&r"(d2), "=&r"(d3), "=r"(lt)
        : "r"(r.w[0]), "r"(r.w[1]), "r"(r.w[2]), "r"(r.w[3]), "r"(q[0]), "r"(q[1]), "r"(q[2]), "r"(q[3]));
    r.w[0] = lt ? r.w[0] : d0;
    r.w[1] = lt ? r.w[1] : d1;
    r.w[2] = lt ? r.w[2] : d2;
    r.w[3] = lt ? r.w[3] : d3;
    return r;
  }
};

// One butterfly of the network: (x, y) <- (x + w*y, x - w*y) with the
// reference's addmod / submod (src/ntt_scalar.c:586-588).  The kernels with the
// general multiply run it; a fast modulus takes lazy_stages below.
template <class Arith>
__device__ __forceinline__ void butterfly(U128& x, U128& y, const U128& w, const ModParams& m) {
  const U128 p = Arith::mul(w, y, m);
  const U128 s = addmod_ref(x, p, m.q);
  y = submod_ref(x, p, m.q);
  x = s;
}

// ---------------------------------------------------- partly reduced values
//
// The forward network of a fast modulus keeps its values u partly reduced
// between the stages of a pass: u is congruent to the reference's value v
// and lies around 8q,
//     8q - s*(2^124 + 2^60) <= u <= 9q + s*(2^124 + 2^60) + 2^32
// after s stages (s <= kLazyStages keeps 0 < u < 2^128 - 2^101, the range
// mul_lazy takes), so a butterfly is one mul_lazy, one 128-bit add and one
// 128-bit subtract: 50 instructions instead of 70 with the exact add and sub
// (probe: 287 -> 354 G butterflies/s).
//
// The reference's addmod is not reduction mod q for two kinds of sum: it
// returns q for a sum of exactly q, and a value 2^64 short when a sum above
// q has q's low 64 bits.  Both leave a value whose low 64 bits are -j*k for
// some 1 <= j <= 16, whose second limb is therefore all ones; so is that of
// every u whose v is congruent to 0 or is at least q.  A thread that sees that limb in a
// sum, or in any value a pass leaves, reruns the pass on its elements with
// the reference's butterflies (exact_stages).  Spread residues do that once
// in 2^32 butterflies; for others it costs time only.  What a rerun leaves
// for the next pass is 8q + v, v exact, so lazy_value can tell 0 from q: a
// value with that limb always comes from a rerun.
constexpr int kLazyStages = 6;

__device__ __forceinline__ U128 add_nc(const U128& a, const U128& b) {  // mod 2^128
  U128 r;
  asm("add.cc.u32  %0, %4, %8;\n\t"
      "addc.cc.u32 %1, %5, %9;\n\t"
      "addc.cc.u32 %2, %6, %10;\n\t"
      "addc.u32    %3, %7, %11;\n\t"
      : "=&r"(r.w[0]), "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3])
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]), "r"(b.w[3]));
  return r;
}
__device__ __forceinline__ U128 sub_nc(const U128& a, const U128& b) {  // mod 2^128
  U128 r;
  asm("sub.cc.u32  %0, %4, %8;\n\t"
      "subc.cc.u32 %1, %5, %9;\n\t"
      "subc.cc.u32 %2, %6, %10;\n\t"
      "subc.u32    %3, %7, %11;\n\t"
      : "=&r"(r.w[0]), "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3])
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(b.w[0]), "r"(b.w[1]), "r"(b.w[2]), "r"(b.w[3]));
  return r;
}
// u + 8q, 8q = 2^127 - 8k
__device__ __forceinline__ U128 add_8q(const U128& a, uint32_t k) {
  U128 r;
  asm("add.cc.u32  %0, %4, %8;\n\t"
      "addc.cc.u32 %1, %5, 0xFFFFFFFF;\n\t"
      "addc.cc.u32 %2, %6, 0xFFFFFFFF;\n\t"
      "addc.u32    %3, %7, 0x7FFFFFFF;\n\t"
      : "=&r"(r.w[0]), "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3])
      : "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3]), "r"(0u - (k << 3)));
  return r;
}
// any u below 2^128 -> congruent, below 2^124 + 16k
__device__ __forceinline__ U128 fold_top(const U128& a, uint32_t k) {
  U128 r;
  asm("mad.lo.cc.u32  %0, %4, %5, %6;\n\t"
      "madc.hi.cc.u32 %1, %4, %5, %7;\n\t"
      "addc.cc.u32    %2, %8, 0;\n\t"
      "addc.u32       %3, %9, 0;\n\t"
      : "=&r"(r.w[0]), "=&r"(r.w[1]), "=&r"(r.w[2]), "=&r"(r.w[3])
      : "r"(a.w[3] >> 28), "r"(k), "r"(a.w[0]), "r"(a.w[1]), "r"(a.w[2]), "r"(a.w[3] & 0x0FFFFFFFu));
  return r;
}
// the reference's value of a u that a pass left
__device__ __forceinline__ U128 lazy_value(const U128& u, uint32_t k) {
  const U128 zero_based = add_8q(u, k);             // u + 8q = (u - 8q) + 16q, 16q = 2^128 - 16k
  if (u.w[1] == 0xFFFFFFFFu) {                      // left by a rerun: u - 8q
    const U128 c{{k << 4, 0u, 0u, 0u}};
    return add_nc(zero_based, c);
  }
  return reduce_once(fold_top(u, k), k);
}

// The r stages of a group of 2^r registers from e0 on partly reduced values;
// tw(t, u) is the twiddle of block u of stage t.  Sets `rerun` when a value
// has the limb described above.  STOP (every lane of the warp takes part): the
// warp's lanes end together after the first stage, all with `rerun` set, if one
// of those with `counts` has it set by then.
template <int r, bool STOP = false, int R, class Tw>
__device__ __forceinline__ void lazy_stages(U128 (&v)[R], int e0, const Tw& tw, uint32_t k, bool& rerun,
                                            bool counts = true) {
#pragma unroll
  for (int t = 0; t < r; ++t) {
    if (STOP && t == 1 && __builtin_expect(__any_sync(0xFFFFFFFFu, rerun && counts), 0)) {
      rerun = true;
      return;
    }
    const int half = 1 << (r - 1 - t);
#pragma unroll
    for (int u = 0; u < (1 << t); ++u) {
      const U128 w = tw(t, u);
#pragma unroll
      for (int i = 0; i < half; ++i) {
        U128 &x = v[e0 + ((u << (r - t)) | i)], &y = v[e0 + ((u << (r - t)) | i) + half];
        const U128 p = mul_lazy(w, y, k);
        y = sub_nc(x, p);
        x = add_nc(x, p);
        rerun |= x.w[1] == 0xFFFFFFFFu;
        if (t == r - 1) rerun |= y.w[1] == 0xFFFFFFFFu;
      }
    }
  }
}

// The same stages with the reference's butterflies, on exact values.  ZEROS: the
// first stage multiplies no zeros.
template <int r, bool ZEROS = false, int R, class Tw>
__device__ __forceinline__ void exact_stages(U128 (&v)[R], const Tw& tw, uint32_t k) {
#pragma unroll
  for (int t = 0; t < r; ++t) {
    const int half = 1 << (r - 1 - t);
#pragma unroll
    for (int u = 0; u < (1 << t); ++u) {
      const U128 w = tw(t, u);
#pragma unroll
      for (int i = 0; i < half; ++i) {
        U128 &x = v[(u << (r - t)) | i], &y = v[((u << (r - t)) | i) + half];
        U128 p = y;
        if (!ZEROS || t > 0 || (y.w[0] | y.w[1] | y.w[2] | y.w[3])) p = reduce_once(mul_lazy(w, y, k), k);
        y = submod_pm(x, p, 0u - k);
        x = addmod_pm(x, p, 0u - k);
      }
    }
  }
}

// ------------------------------------------- partly reduced inverse butterflies
//
// The inverse network (Gentleman-Sande: x + y and (x - y) * w) is exact mod q
// with canonical results and has no corner cases to keep, so its values stay
// partly reduced without a check.  Bounds in units of 2^124 + 2^61: a pass
// starts with at most 2; its first stage's sums reach 4, its differences, less
// than 5 with the multiple of q that keeps them positive, go through mul_lazy
// and come out below 1.  A sum of two unfolded sums (8 at most) is folded
// where it arises, so every later stage sees at most 4 and a pass leaves at
// most 2.  Per group of 4 butterflies that is one fold, against an exact sum
// and difference in each (70 -> 57 instructions per butterfly).
template <int C>
__device__ __forceinline__ U128 sub_plus_q(const U128& x, const U128& y, uint32_t k) {  // x - y + C*q
  const U128 cq{{0u - (uint32_t)C * k, 0xFFFFFFFFu, 0xFFFFFFFFu, ((uint32_t)C << 28) - 1u}};
  return sub_nc(add_nc(x, cq), y);
}

// Inverse of stage t of the group of 2^r registers from e0: butterflies of
// distance 2^(r-1-t), the stages running from t = r - 1 down.  KEEP leaves the
// sums of stage 0 unfolded (at most 8): the caller reduces them.
template <int r, int t, bool KEEP, int R, class Tw>
__device__ __forceinline__ void inverse_stage(U128 (&v)[R], int e0, const Tw& tw, uint32_t k) {
  constexpr int e = r - 1 - t, half = 1 << e;
#pragma unroll
  for (int u = 0; u < (1 << t); ++u) {
    const U128 w = tw(t, u);
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const int j = (u << (r - t)) | i;
      U128 &x = v[e0 + j], &y = v[e0 + j + half];
      const U128 d = sub_plus_q<e == 0 ? 3 : 5>(x, y, k);
      x = add_nc(x, y);
      // both operands are sums (of stage t + 1; of the pass's inputs if r = 1)
      const bool big = r == 1 || (e > 0 && ((j >> (e > 0 ? e - 1 : 0)) & 1) == 0);
      if (big && !(KEEP && t == 0)) x = fold_top(x, k);
      y = mul_lazy(w, d, k);
    }
  }
}
template <int r, bool KEEP, int R, class Tw>
__device__ __forceinline__ void inverse_stages(U128 (&v)[R], int e0, const Tw& tw, uint32_t k) {
  if constexpr (r > 3) inverse_stage<r, 3, KEEP>(v, e0, tw, k);
  if constexpr (r > 2) inverse_stage<r, 2, KEEP>(v, e0, tw, k);
  if constexpr (r > 1) inverse_stage<r, 1, KEEP>(v, e0, tw, k);
  inverse_stage<r, 0, KEEP>(v, e0, tw, k);
}

}  // namespace bntt
