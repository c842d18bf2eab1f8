// Host-side launcher of the SpMM core: picks the lane layout for the row
// width and walks column slabs of at most 128 16-byte vectors.
#pragma once
#include <cuda_runtime.h>

#include "lne_internal.h"
#include "spmm_core.cuh"

#include <algorithm>

namespace lne {

template <typename XT, int G, int VPL, bool VAL, class Epi>
static void spmm_launch(lne_ctx* ctx, const SpmmArgs<XT>& s, const Epi& epi, int* nl) {
  int64_t blocks = ((int64_t)s.n_items + kSpmmWarps - 1) / kSpmmWarps;
  const int64_t cap = (int64_t)ctx->num_sms * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  k_spmm<XT, G, VPL, VAL, false, Epi><<<(unsigned)blocks, kSpmmThreads, 0, ctx->stream>>>(s, epi);
  *nl += 1;
}

static constexpr int kSpmmPartsMax = HeavyTune<32, false>::kParts;
// Blocks of the light rows of the balanced form: persistent, four per SM.
static inline int64_t spmm_bal_blocks(const lne_ctx* ctx, const SpmmPlan& plan) {
  const int64_t want = (plan.n_items - plan.n_heavy + kSpmmWarps - 1) / kSpmmWarps;
  return std::max<int64_t>(1, std::min<int64_t>(want, (int64_t)ctx->num_sms * 4));
}

// The heavy rows, and the light rows beside them (programmatic dependent
// launch: the second kernel starts once the first one's blocks all have, and
// ends after it).  Adds the launches to *nl.
template <typename XT, int G, bool VAL, class Epi>
static void spmm_launch_bal(lne_ctx* ctx, const SpmmPlan& plan, const SpmmArgs<XT>& s, const Epi& epi, int* nl) {
  if (plan.n_heavy > 0) {
    const int64_t units = plan.n_heavy * HeavyTune<G, VAL>::kWarps;
    k_spmm_heavy<XT, G, VAL, Epi>
        <<<(unsigned)((units + kHeavyWarps - 1) / kHeavyWarps), kHeavyWarps * 32, 0, ctx->stream>>>(s, epi);
    *nl += 1;
  }
  if (plan.n_items == plan.n_heavy) return;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3((unsigned)spmm_bal_blocks(ctx, plan), 1, 1);
  cfg.blockDim = dim3(kSpmmThreads, 1, 1);
  cfg.stream = ctx->stream;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = plan.n_heavy > 0 ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k_spmm<XT, G, 1, VAL, true, Epi>, s, epi);
  *nl += 1;
}

// Scratch of the launches over a plan, owned by one call: partial sums of
// the chunks up to `width` floats wide and their arrival counters (launches
// on a stream follow one another and leave them at zero).
struct SpmmWork {
  float* partial = nullptr;
  unsigned* done = nullptr;
};
static inline int spmm_work_alloc(lne_ctx* ctx, const SpmmPlan& plan, int64_t width, SpmmWork* w) {
  *w = SpmmWork();
  if (plan.n_big == 0) return LNE_OK;
  const size_t pb = sizeof(float) * (size_t)plan.n_big * (size_t)width;  // width: a multiple of 4 floats
  const size_t zb = sizeof(unsigned) * kSpmmPartsMax * (size_t)plan.n_big;
  int rc = dalloc(ctx, (void**)&w->partial, pb + zb, "spmm partials");
  if (rc) return rc;
  w->done = reinterpret_cast<unsigned*>(reinterpret_cast<char*>(w->partial) + pb);
  LNE_CUDA_TRY(cudaMemsetAsync(w->done, 0, zb, ctx->stream));
  return LNE_OK;
}
static inline void spmm_work_free(lne_ctx* ctx, SpmmWork* w) {
  if (w->partial) dfree(ctx, w->partial);
  *w = SpmmWork();
}
// Floats per chunk that a product with d columns needs (slabs of at most 128
// vectors).
template <typename XT>
static inline int64_t spmm_work_width(int64_t d) {
  constexpr int E = Vec16<XT>::E;
  const int64_t vecs = (d + E - 1) / E;
  return (vecs < 128 ? vecs : 128) * E;
}

// Copies columns [v0, v0 + C) (16-byte vectors) of the x_rows rows of X
// into a dense x_rows x C array.
static __global__ void k_slab_copy(const uint4* __restrict__ X, int64_t ldv, int64_t v0, int64_t x_rows, int C,
                            uint4* __restrict__ out) {
  const int64_t total = x_rows * C;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = i / C;
    const int c = (int)(i - r * C);
    out[i] = __ldg(X + r * ldv + v0 + c);
  }
}

// A narrow slab after the first (the tail columns of a 144-wide operand)
// is gathered from a dense copy of its columns when that copy is at most
// this size: rows of the copy are 32-64 bytes instead of one 128-byte line
// per row of X, so the copy stays in L2 while the slab's gathers run.
static constexpr int64_t kSlabCopyMaxBytes = (int64_t)96 << 20;

// Runs Y-epilogue(A * X) over all rows.  A: the work list `plan` over the
// column ids `col` (and values, null: ones).  X rows: ldx elements, 16-byte
// aligned; d columns are produced (the epilogue sees element offsets).
// x_rows (the rows of X; 0 if unknown) enables the tail-slab copies.
template <typename XT, bool VAL, class Epi>
static int spmm_run(lne_ctx* ctx, const SpmmPlan& plan, const uint32_t* col, const float* val, const XT* X, int64_t ldx,
                    int64_t d, const Epi& epi, int* launches = nullptr, int64_t x_rows = 0,
                    const SpmmWork* work = nullptr) {
  constexpr int E = Vec16<XT>::E;
  const int64_t c_total = (d + E - 1) / E;
  int rc;
  int nl = 0;
  // graphs, and matrices so small that a warp walking a 2048-entry row (some
  // 250 us) would outlast the rest: below 4 GB of gathers (about 0.4 ms).
  // Above, the 16-byte gathers of a warp per row take fewer instructions.
  // The line follows the size alone, while what decides is also how long the
  // rows are.  Measured both ways on power-law matrices, us balanced / a warp
  // per row: 200,000 rows of 20, FP32, 32 columns (0.5 GB) 94 / 83, 128 (2 GB)
  // 189 / 356, 256 (4.1 GB) 380 / 734; 10,312 rows of 340, 64 columns (0.9 GB)
  // 83 / 100, 256 (3.6 GB) 301 / 314; 60,000 rows of 280, 32 columns (2.2 GB)
  // 167 / 163, 64 (4.4 GB) 298 / 260, 256 (17 GB) 1071 / 831; 10,312 rows of
  // 1,100, 64 columns (2.8 GB) 237 / 167, 256 (11 GB) 930 / 503.
  const bool bal = !VAL || (plan.warp_max < kChunkNnz && (double)plan.nnz * d * sizeof(XT) < 4e9);
  SpmmWork own;
  if (!work) {
    if ((rc = spmm_work_alloc(ctx, plan, spmm_work_width<XT>(d), &own))) return rc;
    work = &own;
  }
  // Column slabs of a power-of-two number of 16-byte vectors (at most 128),
  // largest first: each slab fills its lane layout exactly (a 144-wide FP32
  // row is a 32-vector slab and a 4-vector slab, not 36 vectors on 32 lanes).
  int64_t c_off = 0;
  while (c_off < c_total) {
    int64_t rem = c_total - c_off, C2 = 1;
    while (C2 * 2 <= rem && C2 * 2 <= 128) C2 *= 2;
    // a 144-element row is one slab of three groups of 9 lanes: 9 FP8
    // vectors (one per lane) or 18 BF16 / FP16 vectors (two per lane), so
    // its tail shares the gathers of the row instead of a second pass
    if (E == 16 && rem == 9) C2 = 9;
    if (E == 8 && rem == 18) C2 = 18;
    // from 32 vectors on a row is one strand: narrower slabs, same sums
    if (bal && C2 > 32) C2 = 32;
    const int C = (int)C2;
    const XT* Xs = X + c_off * E;
    int64_t ldxs = ldx;
    XT* slab = nullptr;
    if (c_off > 0 && C < 32 && x_rows > 0 && x_rows * C * 16 <= kSlabCopyMaxBytes) {
      if ((rc = dalloc(ctx, (void**)&slab, (size_t)(x_rows * C * 16), "spmm slab copy"))) {
        spmm_work_free(ctx, &own);
        return rc;
      }
      const int64_t nv = x_rows * C;
      int64_t blocks = (nv + 255) / 256;
      if (blocks > (int64_t)ctx->num_sms * 16) blocks = (int64_t)ctx->num_sms * 16;
      k_slab_copy<<<(unsigned)blocks, 256, 0, ctx->stream>>>(reinterpret_cast<const uint4*>(X), ldx / E, c_off, x_rows,
                                                             C, reinterpret_cast<uint4*>(slab));
      ++nl;
      Xs = slab;
      ldxs = (int64_t)C * E;
    }
    SpmmArgs<XT> s;
    s.items = plan.items;
    s.n_items = (uint32_t)plan.n_items;
    s.n_big = (uint32_t)plan.n_big;
    s.n_heavy = (uint32_t)plan.n_heavy;
    s.span = plan.span;
    s.col = col;
    s.val = val;
    s.X = Xs;
    s.ldx = ldxs;
    s.C = C;
    s.partial = work->partial;
    s.ldp = (int64_t)C * E;
    s.done = work->done;
    s.e_base = (int)(c_off * E);
    const bool nine = (E == 8 && C == 18) || (E == 16 && C == 9);
    if (bal && !nine && !(E == 16 && C == 1)) {
      if (C <= 2)
        spmm_launch_bal<XT, 2, VAL>(ctx, plan, s, epi, &nl);
      else if (C <= 4)
        spmm_launch_bal<XT, 4, VAL>(ctx, plan, s, epi, &nl);
      else if (C <= 8)
        spmm_launch_bal<XT, 8, VAL>(ctx, plan, s, epi, &nl);
      else if (C <= 16)
        spmm_launch_bal<XT, 16, VAL>(ctx, plan, s, epi, &nl);
      else
        spmm_launch_bal<XT, 32, VAL>(ctx, plan, s, epi, &nl);
    } else if (nine) {
      // E == 4 rows have no 9-lane layout
      if constexpr (E == 8) spmm_launch<XT, 9, 2, VAL>(ctx, s, epi, &nl);
      if constexpr (E == 16) spmm_launch<XT, 9, 1, VAL>(ctx, s, epi, &nl);
    } else if (E == 16 && C == 1) {
      // FP8: one lane per nonzero for one vector
      if constexpr (E == 16) spmm_launch<XT, 1, 1, VAL>(ctx, s, epi, &nl);
    } else if constexpr (VAL) {
      if (C <= 2)
        spmm_launch<XT, 2, 1, VAL>(ctx, s, epi, &nl);
      else if (C <= 4)
        spmm_launch<XT, 4, 1, VAL>(ctx, s, epi, &nl);
      else if (C <= 8)
        spmm_launch<XT, 8, 1, VAL>(ctx, s, epi, &nl);
      else if (C <= 16)
        spmm_launch<XT, 16, 1, VAL>(ctx, s, epi, &nl);
      else if (C <= 32)
        spmm_launch<XT, 32, 1, VAL>(ctx, s, epi, &nl);
      else if (C <= 64)
        spmm_launch<XT, 32, 2, VAL>(ctx, s, epi, &nl);
      else
        spmm_launch<XT, 32, 4, VAL>(ctx, s, epi, &nl);
    }
    if (slab) dfree(ctx, slab);
    c_off += C;
  }
  spmm_work_free(ctx, &own);
  if (launches) *launches += nl;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    set_error(std::string("spmm launch: ") + cudaGetErrorString(e));
    return LNE_ERR_CUDA;
  }
  return LNE_OK;
}

// Cache-blocked SpMM over a CSR: when the dense operand is larger than the
// context's panel budget, the columns are cut into panels whose slice of X
// fits in L2 and one pass per panel gathers only from that slice (panels of
// at most the budget each, or, with a negative budget, two panels: the
// lowest ids up to the budget, which on graphs whose hubs have low ids
// take most of the gathers, then the rest).  The epilogue is called with
// add = false on the first panel and add = true on the later ones (fixed
// panel order: reproducible sums).
template <typename XT, class EpiT>
static int spmm_csr_panels(lne_ctx* ctx, lne_csr* A, const XT* X, int64_t ldx, int64_t d, EpiT epi,
                           int* launches = nullptr, int64_t panel_bytes = 0) {
  const int64_t row_bytes = ldx * (int64_t)sizeof(XT);
  const int64_t xbytes = A->n * row_bytes;
  // the context's setting wins; otherwise the caller's suggestion
  const int64_t want = ctx->spmm_panel_bytes != 0 ? ctx->spmm_panel_bytes : panel_bytes;
  int64_t budget = want < 0 ? -want : want;
  int rc;
  if (want < 0 && budget > 0 && xbytes > budget) {
    // a two-panel split pays only when the first panel takes most entries
    const int64_t pw = std::max<int64_t>(1, budget / row_bytes);
    if (launches && !(A->hub_share >= 0.0 && A->hub_cols == pw)) *launches += 1;
    if ((rc = hub_share(ctx, A, pw))) return rc;
    if (A->hub_share < 0.5) budget = 0;
  }
  if (budget == 0 || xbytes <= budget) {
    if (!A->plan_ready && launches) *launches += plan_launches(A->n);
    if ((rc = build_plan_csr(ctx, A))) return rc;
    epi.add = false;
    return spmm_run<XT, true>(ctx, A->plan, reinterpret_cast<const uint32_t*>(A->col), A->val, X, ldx, d, epi, launches,
                              A->n);
  }
  const int64_t pw = std::max<int64_t>(1, budget / row_bytes);
  std::vector<int64_t> bounds{0};
  if (want < 0) {
    bounds.push_back(pw);
  } else {
    for (int64_t b = pw; b < A->n; b += pw) bounds.push_back(b);
  }
  bounds.push_back(A->n);
  if (A->panel_bounds != bounds && launches) *launches += 1 + (int)(bounds.size() - 1) * plan_launches(A->n);
  if ((rc = build_panels(ctx, A, bounds))) return rc;
  for (int p = 0; p < A->npanels; ++p) {
    epi.add = p > 0;
    if ((rc = spmm_run<XT, true>(ctx, A->panel_plans[p], reinterpret_cast<const uint32_t*>(A->col), A->val, X, ldx, d,
                                 epi, launches)))
      return rc;
  }
  return LNE_OK;
}

}  // namespace lne
