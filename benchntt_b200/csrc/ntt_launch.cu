// ntt_launch.cu -- registry of compiled sub-transform kernels, the HBM pass
// split, and the stream-ordered forward transform.
#include <algorithm>
#include <mutex>

#include "internal.h"
#include "ntt_core.cuh"

namespace bntt {

#define BNTT_DECLARE(p) void append_fast_plan_##p(std::vector<SubKernel>& v);
BNTT_PLAN_PARTS(BNTT_DECLARE)
#undef BNTT_DECLARE
#define BNTT_DECLARE(p) void append_ref_##p(std::vector<SubKernel>& v);
BNTT_REF_PARTS(BNTT_DECLARE)
#undef BNTT_DECLARE
void append_fast_contig(std::vector<SubKernel>& v);
void append_fast_contig_r4(std::vector<SubKernel>& v);
void append_fast_il(std::vector<SubKernel>& v);
void append_fast_occ(std::vector<SubKernel>& v);
void append_fast_small(std::vector<SubKernel>& v);
void append_fast_staged(std::vector<SubKernel>& v);
void append_fast_occ5(std::vector<SubKernel>& v);

const std::vector<SubKernel>& sub_kernels() {
  static std::vector<SubKernel> v = [] {
    std::vector<SubKernel> r;
    append_fast_contig(r);
    append_fast_contig_r4(r);
    append_fast_il(r);
#define BNTT_ADD(p) append_ref_##p(r);
    BNTT_REF_PARTS(BNTT_ADD)
#undef BNTT_ADD
    append_fast_occ(r);
    append_fast_small(r);
    append_fast_staged(r);
    append_fast_occ5(r);
#define BNTT_ADD(p) append_fast_plan_##p(r);
    BNTT_PLAN_PARTS(BNTT_ADD)
#undef BNTT_ADD
    return r;
  }();
  return v;
}

const SubKernel* default_sub_kernel(int m, int map, int fast, uint64_t elems) {
  struct Table {
    const SubKernel* at[11][2][2][8] = {};
  };
  static const Table table = [] {
    Table t;
    for (const SubKernel& k : sub_kernels())
      for (int use : {USE_LONE, USE_FEW, USE_MANY})
        if (k.use & use) t.at[k.m][k.map][k.fast][use] = &k;
    return t;
  }();
  return m >= 1 && m <= 10 ? table.at[m][map][fast][use_of(elems)] : nullptr;
}

int blocks_per_sm(const SubKernel* k) {
  static std::mutex mu;
  std::lock_guard<std::mutex> g(mu);
  SubKernel* mk = const_cast<SubKernel*>(k);
  if (mk->max_blocks_per_sm > 0) return mk->max_blocks_per_sm;
  if (k->smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k->fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)k->smem);
    if (e != cudaSuccess) return -cuda_error(e, "cudaFuncSetAttribute(smem)");
  }
  int b = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k->fn, k->threads, k->smem);
  if (e != cudaSuccess) return -cuda_error(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
  if (b < 1) return -set_error(BNTT_ECUDA, "kernel m=%d logr=%d tpc=%d does not fit on an SM", k->m,
                               k->logr, k->tpc);
  mk->max_blocks_per_sm = b;
  return b;
}

int launch_sub(bntt_ctx* ctx, const SubKernel* k, const void* geom, const ModParams& mp,
               int layout, cudaStream_t stream, int finishing) {
  const SubGeom& g = *static_cast<const SubGeom*>(geom);
  const uint64_t ntiles = (g.nsub + (uint64_t)k->tpc - 1) / (uint64_t)k->tpc;
  if (ntiles == 0) return BNTT_OK;
  BNTT_REQUIRE(ntiles <= 0x7fffffffu, "%llu tiles are more than one launch takes", (unsigned long long)ntiles);
  uint64_t grid = ntiles;  // one CTA per tile; the staged kernels are persistent
  if (k->smem > 48 * 1024 || k->src != 0) {
    const int bps = blocks_per_sm(k);
    if (bps < 0) return -bps;
    if (k->src != 0) grid = std::min<uint64_t>(grid, (uint64_t)bps * (uint64_t)ctx->sms);
  }
  SubGeom gg = g;
  ModParams mm = mp;
  int lay = layout;
  void* args[] = {&gg, &mm, &lay, &finishing};  // the forward kernels take the first three
  return launch_overlapped(ctx, k->fn, (unsigned)grid, (unsigned)k->threads, k->smem, args, stream);
}

int launch_overlapped(bntt_ctx* ctx, const void* fn, unsigned grid, unsigned threads, size_t smem, void** args,
                      cudaStream_t stream) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  BNTT_CK(cudaLaunchKernelExC(&cfg, fn, args));
  ctx->launches++;
  return BNTT_OK;
}

int plan_choose_kernels(bntt_plan* p) {
  const int n = (int)p->log2n;
  p->passes = n <= 10 ? std::vector<int>{n} : tile_split(n);
  p->created_fast = arith_fast(p->ctx, p->fast);
  p->tuned.clear();
  int s0 = 0;
  for (int m : p->passes) {
    const int l = n - s0 - m;
    const SubKernel* k = tuned_sub_kernel(m, l > 0 ? MAP_INTERLEAVED : MAP_CONTIG, p->created_fast ? 1 : 0, l);
    // a table copied into shared memory holds entries below 2^m only: whole
    // transforms
    if (k && (k->src & TW_SHARED) && s0 != 0) k = nullptr;
    p->tuned.push_back(k);
    s0 += m;
  }
  return BNTT_OK;
}

// The HBM passes of the transform in order: whole transforms of up to 2^10
// points in one, larger ones as strided passes of 5..7 stages over 2^(10-m)
// adjacent columns (128 B or more per row), then a contiguous pass.  Compiled
// tiles with 10-stage passes, whose strided passes touch 2 or 4 columns per
// row, were 2x slower.
int ntt_forward_on(bntt_plan* plan, void* y, const void* x, size_t batch, cudaStream_t s,
                   const void* b, uint64_t bmask) {
  if (batch == 0) return BNTT_OK;
  const int n = (int)plan->log2n;
  // above 2^10 points a plan takes the fast multiply as soon as its context does
  const bool fast = plan->created_fast || (n > 10 && arith_fast(plan->ctx, plan->fast));
  int s0 = 0;
  for (size_t i = 0; i < plan->passes.size(); ++i) {
    const int m = plan->passes[i];
    const int map = n - s0 - m > 0 ? MAP_INTERLEAVED : MAP_CONTIG;
    const uint64_t elems = (uint64_t)batch << n;
    const SubKernel* k = plan->tuned[i];
    if (!k || k->fast != (fast ? 1 : 0) || elems < tuned_from(m, map)) k = default_sub_kernel(m, map, fast ? 1 : 0, elems);
    if (!k) return set_error(BNTT_EINVAL, "no kernel compiled for pass m=%d map=%d", m, map);
    SubGeom g;
    g.x = static_cast<const uint4*>(i == 0 ? x : y);
    g.y = static_cast<uint4*>(y);
    g.tw = static_cast<const uint4*>(plan->tw);
    g.n = (uint32_t)n;
    g.s0 = (uint32_t)s0;
    g.m = (uint32_t)m;
    g.l = (uint32_t)(n - s0 - m);
    g.nsub = (uint64_t)batch << (n - m);
    if (i + 1 == plan->passes.size()) {
      g.b = static_cast<const uint4*>(b);
      g.bmask = bmask;
    }
    if (int rc = launch_sub(plan->ctx, k, &g, plan->mp, plan->layout, s)) return rc;
    s0 += m;
  }
  return BNTT_OK;
}

}  // namespace bntt
