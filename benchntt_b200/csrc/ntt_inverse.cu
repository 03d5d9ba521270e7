// ntt_inverse.cu -- the inverse transform of a plan.
//
// The reference has no inverse transform.  The forward network
// (src/ntt_scalar.c:582-627, in its in-place form: stage s pairs indices
// that differ in bit n-1-s with twiddle T[2^s + (index >> (n-s))]) is a
// product of butterflies (x, y) -> (x + w y, x - w y); each is invertible
// when w is, with inverse (u, v) -> ((u + v) / 2, (u - v) / (2 w)).  So
// running the stages from the last to the first with Gentleman-Sande
// butterflies (x, y) -> (x + y, (x - y) w^-1) and multiplying by N^-1 at the
// end returns the input, for every table whose entries are invertible mod a
// prime q.  With the root-power tables of roots.cu it is the inverse
// negacyclic NTT, and ntt^-1(ntt(a) o ntt(b)) = a * b mod (x^N + 1).
//
// Sums here are exact mod q (no reference quirk applies: the reference has
// no such code); results are canonical residues in [0, q).  The fast
// pseudo-Mersenne multiply is required (q = 2^124 - k, k < 2^28).
//
// Kernels: the compile-time tile in inverse mode (k_ntt_tile_inv, ntt_inst_inverse.cu), one
// launch for N up to 2^10 and above that one launch per HBM pass of the
// persistent kernel's split (tile_split), in reverse pass order (the pass
// over the low index bits first).
#include <vector>

#include "ntt_kernels.cuh"

namespace bntt {

#define BNTT_DECLARE(p) void append_inverse_##p(std::vector<SubKernel>& v);  // ntt_inst_inverse.cu
BNTT_PLAN_PARTS(BNTT_DECLARE)
#undef BNTT_DECLARE

namespace {

// The shape for a pass of m stages over `elems` elements.
const SubKernel* inverse_kernel(int m, int map, uint64_t elems) {
  static const std::vector<SubKernel> kernels = [] {
    std::vector<SubKernel> v;
#define BNTT_ADD(p) append_inverse_##p(v);
    BNTT_PLAN_PARTS(BNTT_ADD)
#undef BNTT_ADD
    return v;
  }();
  for (const SubKernel& k : kernels)
    if (k.m == m && k.map == map && (k.use & use_of(elems))) return &k;
  return nullptr;
}

// out[k] = tw[k]^-1 = tw[k]^(q-2) mod q for k >= 1, out[1] times ninv as well;
// out[0].x becomes nonzero if an entry is not a residue above 0 or its power is
// not its inverse.  One thread per entry: about 230 dependent products, so a
// 2^20 table takes under a millisecond, where the host took 40 ms (two
// sequential products per entry) and two copies of the table.
__global__ void __launch_bounds__(128) k_invert_table(uint4* out, const uint4* tw, uint32_t n, U128 ninv, ModParams mp) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k == 0 || k >= n) return;
  const uint4 v = tw[k];
  const U128 e{{v.x, v.y, v.z, v.w}};
  U128 x = e;  // e^(leading bit of q - 2, bit 123)
#pragma unroll 1
  for (int bit = 122; bit >= 0; --bit) {
    // q - 2 = 2^124 - (k + 2): bits 0..31 from the low limb, the borrow out of it below
    const uint32_t low = mp.q.w[0] - 2u;
    const uint32_t above = mp.q.w[0] >= 2u ? mp.q.w[1] : mp.q.w[1] - 1u;
    const uint32_t limb = bit < 32 ? low : bit < 64 ? above : mp.q.w[bit >> 5];
    x = ArithFast::mul(x, x, mp);
    if (limb >> (bit & 31) & 1u) x = ArithFast::mul(x, e, mp);
  }
  const U128 one = ArithFast::mul(x, e, mp);
  const bool residue = e.w[3] < 0x0FFFFFFFu || (e.w[3] == 0x0FFFFFFFu && (e.w[2] != 0xFFFFFFFFu || e.w[1] != 0xFFFFFFFFu ||
                                                                         e.w[0] < mp.q.w[0]));
  if (!residue || one.w[0] != 1u || (one.w[1] | one.w[2] | one.w[3])) atomicOr(&out[0].x, 1u);
  if (k == 1) x = ArithFast::mul(x, ninv, mp);
  out[k] = make_uint4(x.w[0], x.w[1], x.w[2], x.w[3]);
}

// Inverse table (T[k]^-1, limb order) and N^-1, built once per plan.  Entry 0,
// which no network stage reads, holds N^-1 (the inverse batch kernel takes
// each job's scale from its own table), and entry 1 holds T[1]^-1 * N^-1: every
// inverse kernel then scales only the first half of its outputs (the x outputs
// of the last stage).
//
// On the host, for small tables, for those the device build does not finish (an
// entry without an inverse, q not prime) and for their errors: one modular
// exponentiation and three multiplies per entry (batch inversion).
static u128 entry_of(const std::vector<uint32_t>& t, size_t k) {
  u128 v = 0;
  for (int l = 3; l >= 0; --l) v = (v << 32) | t[4 * k + l];
  return v;
}

int ensure_inverse_host(bntt_plan* p) {
  const u128 q = to_u128(p->mod.q), mu = to_u128(p->mod.mu);
  const size_t n = (size_t)1 << p->log2n;
  std::vector<uint32_t> t(4 * n);
  // copies on the context's stream (ordered after any work that wrote the
  // table, and finished before the first inverse launch reads the result)
  BNTT_CK(cudaMemcpyAsync(t.data(), p->tw, n * 16, cudaMemcpyDeviceToHost, p->ctx->stream));
  BNTT_CK(cudaStreamSynchronize(p->ctx->stream));
  auto entry = [&](size_t k) {
    u128 v = 0;
    for (int l = 3; l >= 0; --l) v = (v << 32) | t[4 * k + l];
    return v;
  };
  // prefix products, one inverse, then walk back
  std::vector<u128> pre(n, 1);
  u128 acc = 1;
  for (size_t k = 1; k < n; ++k) {
    const u128 e = entry(k);
    BNTT_REQUIRE(e != 0 && e < q, "twiddle %zu is 0 mod q (or not a residue): no inverse", k);
    pre[k] = acc;
    acc = host_mulmod(acc, e, q, mu);
  }
  u128 inv = host_powmod(acc, q - 2, q, mu);
  BNTT_REQUIRE(host_mulmod(inv, acc, q, mu) == 1,
               "the product of the twiddles has no inverse mod q (q is not prime)");
  std::vector<uint32_t> ti(4 * n, 0);
  for (size_t k = n - 1; k >= 1; --k) {
    const u128 ik = host_mulmod(inv, pre[k], q, mu);  // = T[k]^-1
    inv = host_mulmod(inv, entry(k), q, mu);
    for (int l = 0; l < 4; ++l) ti[4 * k + l] = (uint32_t)(ik >> (32 * l));
  }
  const u128 ninv = host_powmod((u128)n % q, q - 2, q, mu);
  BNTT_REQUIRE(host_mulmod(ninv, (u128)n % q, q, mu) == 1, "N has no inverse mod q");
  for (int l = 0; l < 4; ++l) ti[l] = (uint32_t)(ninv >> (32 * l));
  // entry 1 (the last inverse stage, which ends in y = (x - y) * T[1]^-1)
  // carries N^-1 too, so the final scaling multiplies the x half only
  const u128 t1 = host_mulmod(entry_of(ti, 1), ninv, q, mu);
  for (int l = 0; l < 4; ++l) ti[4 + l] = (uint32_t)(t1 >> (32 * l));
  void* d = nullptr;
  if (int rc = ctx_alloc(p->ctx, &d, n * 16)) return rc;
  cudaError_t e = cudaMemcpyAsync(d, ti.data(), n * 16, cudaMemcpyHostToDevice, p->ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(p->ctx->stream);
  if (e != cudaSuccess) {
    ctx_free(p->ctx, d);
    return cuda_error(e, "copy of the inverse twiddles");
  }
  p->tw_inv = d;
  return BNTT_OK;
}

int ensure_inverse(bntt_plan* p) {
  if (p->tw_inv) return BNTT_OK;
  // below 2^10 entries the host is quicker: the device build's chain of products
  // takes its time whatever the size (first inverse call, host and device, us:
  // 2^4 48 and 83, 2^9 79 and 84, 2^10 109 and 86, 2^14 723 and 88)
  if (p->log2n < 10) return ensure_inverse_host(p);
  const u128 q = to_u128(p->mod.q), mu = to_u128(p->mod.mu);
  const size_t n = (size_t)1 << p->log2n;
  const u128 ninv = host_powmod((u128)n % q, q - 2, q, mu);
  void* d = nullptr;
  if (host_mulmod(ninv, (u128)n % q, q, mu) != 1 || ctx_alloc(p->ctx, &d, n * 16)) return ensure_inverse_host(p);
  // on the context's stream, after any work that wrote the table; finished
  // before the first inverse launch
  cudaStream_t s = p->ctx->stream;
  const U128 scale = to_limbs(ninv);
  uint32_t flag[4] = {1, 0, 0, 0};
  cudaError_t e = cudaMemsetAsync(d, 0, 16, s);
  if (e == cudaSuccess) {
    k_invert_table<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(static_cast<uint4*>(d), static_cast<const uint4*>(p->tw),
                                                              (uint32_t)n, scale, p->mp);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpyAsync(flag, d, 16, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e == cudaSuccess && flag[0] == 0) e = cudaMemcpyAsync(d, scale.w, 16, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess || flag[0] != 0) {
    ctx_free(p->ctx, d);
    return e != cudaSuccess ? cuda_error(e, "inverse twiddles") : ensure_inverse_host(p);
  }
  p->tw_inv = d;
  return BNTT_OK;
}

int inverse_on(bntt_plan* p, void* x, const void* y, size_t batch, cudaStream_t s) {
  const int n = (int)p->log2n;
  // up to 2^10 points one tile pass; above, the persistent kernel's split
  // (strided passes of 5..7 stages, then a contiguous one), run last pass
  // first, the first run reading y and every run writing x
  const std::vector<int> split = n <= 10 ? std::vector<int>{n} : tile_split(n);
  const int np = (int)split.size();
  std::vector<int> starts(np, 0);
  for (int i = 1; i < np; ++i) starts[i] = starts[i - 1] + split[i - 1];
  for (int k = 0; k < np; ++k) {
    const int i = np - 1 - k;
    SubGeom g;
    g.x = static_cast<const uint4*>(k == 0 ? y : x);
    g.y = static_cast<uint4*>(x);
    g.tw = static_cast<const uint4*>(p->tw_inv);
    g.n = (uint32_t)n;
    g.s0 = (uint32_t)starts[i];
    g.m = (uint32_t)split[i];
    g.l = (uint32_t)(n - starts[i] - split[i]);
    g.nsub = (uint64_t)batch << (n - split[i]);
    const SubKernel* kern = inverse_kernel(split[i], g.l > 0 ? MAP_INTERLEAVED : MAP_CONTIG, (uint64_t)batch << n);
    if (!kern) return set_error(BNTT_EINVAL, "no inverse tile for a pass of %d stages", split[i]);
    if (int rc = launch_sub(p->ctx, kern, &g, p->mp, p->layout, s, i == 0 ? 1 : 0)) return rc;
  }
  return BNTT_OK;
}

}  // namespace

int plan_ensure_inverse(bntt_plan* p) {
  if (!p->fast) return set_error(BNTT_EINVAL, "the inverse transform needs q = 2^124 - k (k < 2^28), mu = floor(2^251/q)");
  return ensure_inverse(p);
}

}  // namespace bntt

using namespace bntt;

extern "C" int bntt_ntt_inverse_dev(bntt_plan* p, void* x, const void* y, size_t batch) {
  BNTT_REQUIRE(p, "plan is NULL");
  if (batch == 0) return BNTT_OK;
  BNTT_REQUIRE(x && y, "NULL buffer");
  BNTT_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)y & 15) == 0,
               "device buffers must be 16-byte aligned");
  BNTT_REQUIRE(p->fast, "the inverse transform needs q = 2^124 - k (k < 2^28), mu = floor(2^251/q)");
  if (int rc = ctx_use_device(p->ctx)) return rc;
  if (int rc = ensure_inverse(p)) return rc;
  return inverse_on(p, x, y, batch, p->ctx->stream);
}
