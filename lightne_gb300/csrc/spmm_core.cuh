// Row-parallel SpMM core: Y[i,:] = epi(i, sum_j v_ij * X[c_ij, :]).
//
// Work is split into items (SpmmItem: first nonzero, row, length) of at most
// kChunkNnz nonzeros; the partial sums of a longer row's chunks go to a
// scratch buffer, and whoever finishes the row's last chunk adds them in
// chunk order.  Every output is a sum in a fixed order, whichever kernel
// takes the item: P = 32/G strands, strand g adding the nonzeros t with
// t % P == g of the item one after the other in FP32, then the strands in a
// balanced tree.  Results are bitwise reproducible run to run.
//
// In a warp, lane gl of group g owns the 16-byte column vectors gl, gl+G, ...
// of the rows of strand g.  Column ids (and values) are loaded up to 32 at a
// time, one per lane, and broadcast with shuffles; the gathers of several
// nonzeros are issued before their FMAs so that every lane keeps several
// 16-byte loads in flight (SpmmTune).
//
// On a sparse graph an item is a handful of gathers, and a warp that loads
// the item, then its ids, then the rows, then the epilogue's operands waits
// out four dependent latencies per row.  So the items run as a pipeline: while
// one is gathered, the ids of the next are in flight, and the epilogue's
// operands (Epi::load) are issued before the gathers.
//
// On graphs, and on matrices too small to hide a warp that walks a 2048-entry
// row, the longer rows are taken first, by several warps each (balanced form).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "dense_common.cuh"
#include "lne_internal.h"

namespace lne {

static constexpr unsigned kFull = 0xffffffffu;

// An epilogue without operands to load ahead.
struct NoPre {};

// Row ranges of a sparse operator, from which a work list is built.
struct CsrRows {  // explicit CSR: int64 row_ptr
  const int64_t* __restrict__ row_ptr;
  __device__ __forceinline__ int64_t begin(int64_t r) const { return __ldg(row_ptr + r); }
  __device__ __forceinline__ int64_t end(int64_t r) const { return __ldg(row_ptr + r + 1); }
};

// The entries of a CSR row whose columns fall in one column panel.
struct PanelRows {
  const int64_t* __restrict__ row_ptr;
  const int32_t* __restrict__ seg;  // n x (np1) relative panel starts
  int np1;                          // panels + 1
  int p;                            // this panel
  __device__ __forceinline__ int64_t begin(int64_t r) const {
    return __ldg(row_ptr + r) + __ldg(seg + r * np1 + p);
  }
  __device__ __forceinline__ int64_t end(int64_t r) const {
    return __ldg(row_ptr + r) + __ldg(seg + r * np1 + p + 1);
  }
};

struct GraphRows {  // graph adjacency: {offset, degree} per vertex
  const Vertex* __restrict__ vdata;
  __device__ __forceinline__ int64_t begin(int64_t r) const { return (int64_t)__ldg(&vdata[r].off); }
  __device__ __forceinline__ int64_t end(int64_t r) const {
    return (int64_t)__ldg(&vdata[r].off) + (int64_t)__ldg(&vdata[r].deg);
  }
};

// Gather depth: each lane issues the gathers of kU nonzeros before their
// FMAs, kept as raw 16-byte words (4 registers each).  Column ids are loaded
// in batches of kBatch <= 32, a multiple of the P kU nonzeros a warp takes
// per step, so that no step of a batch runs part-empty, and a step whose
// nonzeros are all in the batch loads without predicates.  Measured at
// n = 1.14M, nnz = 351M (`B = A Q`, the sketch product, the 19 SpMMs of the
// propagation), unpredicated full steps included: a 144-element FP16 row at
// kU = 2 (batch 30) 11.1 ms against 11.6 at 3 and 12.8 at 4; 144-element FP8
// rows at kU = 5 (batch 30) 8.0 against 8.4 at 4 and 9.2 at 6.  Deeper
// staging spills (64 registers a thread at 4 CTAs of 256 per SM); compiled
// for 3 CTAs per SM it lost more warps than it gained in flight.
template <typename XT, int G, int VPL>
struct SpmmTune {
  static constexpr int E = Vec16<XT>::E;
  static constexpr int P = 32 / G;
  static constexpr int kWant = VPL == 1 ? (G == 9 ? 5 : 4) : (VPL == 2 ? (E == 8 && G == 32 ? 1 : 2) : 1);
  static constexpr int kU = kWant * P <= 32 ? kWant : 32 / P;
  static constexpr int kBatch = (32 / (P * kU)) * (P * kU);
  static_assert(kBatch >= 1 && kBatch <= 32, "a batch of column ids is one per lane");
  // 16-bit vectors of one per lane: two groups share the epilogue, four
  // elements of a vector each
  static constexpr bool kSplit = E == 8 && VPL == 1 && G <= 16 && (G & (G - 1)) == 0;
  static constexpr int kEpi = kSplit ? 4 : E;  // elements per epilogue call
};

// What one SpMM launch reads besides the epilogue.
template <typename XT>
struct SpmmArgs {
  const SpmmItem* __restrict__ items;
  uint32_t n_items, n_big, n_heavy;    // see SpmmPlan
  const uint2* __restrict__ span;      // [n_big] {first item of its row, items of its row}
  const uint32_t* __restrict__ col;
  const float* __restrict__ val;       // null: unit values
  const XT* __restrict__ X;
  int64_t ldx;
  int C;                               // 16-byte vectors of the slab
  float* partial;                      // [n_big][ldp]
  int64_t ldp;
  unsigned* done;                      // arrivals per long row (and part), zero between launches
  int e_base;                          // first column of the slab
};

__device__ __forceinline__ int64_t item_begin(const uint4& it) {
  return (int64_t)(((uint64_t)it.y << 32) | it.x);
}

static constexpr int kSpmmThreads = 256;
static constexpr int kSpmmWarps = kSpmmThreads / 32;

// ---------------------------------------------------------------------------
// Balanced form (one 16-byte vector per lane, G a power of two): the rows
// above warp_max go to k_spmm_heavy, with one 32-bit column word per lane
// instead of one 16-byte vector, so that a 512-byte row is the work of four
// warps and each lane has 64 rows in flight instead of four; a lane adds its
// strands' rows in order, so the sums are those of k_spmm.  The rest go
// to k_spmm (BAL), which starts beside it.  On a graph of 10,312 vertices
// and 668K entries (128 FP32 columns) one product took 200 us with a warp
// per row: a 2048-entry row is a chain of gathers that four rows in flight
// leave waiting.  Passing the rows through shared memory to adding threads
// took 110 us (51 instructions per entry), 32 rows in flight in registers
// 110 us (about 1 us per 32 rows).
// ---------------------------------------------------------------------------
static constexpr int kHeavyWarps = 4;
template <int G, bool VAL>
struct HeavyTune {
  static constexpr int P = 32 / G;
  static constexpr int W = G * 4 < 32 ? G * 4 : 32;  // lanes of one row
  static constexpr int LG = 32 / W;                  // rows side by side in a warp
  static constexpr int kParts = G * 4 / W;           // warps side by side on one row
  // warps on strands of their own: an item of a graph, whose products wait
  // for their longest rows, has the block, an item of a matrix kParts warps
  // (one of either measured, see k_spmm_heavy; the number of heavy items was
  // not tried as the rule)
  static constexpr int NS = VAL ? 1 : kHeavyWarps / kParts;
  static constexpr int A = P / (LG * NS);            // strands per lane
  static constexpr int kWarps = kParts * NS;         // warps of one item
  static constexpr int kSets = 2;                    // sets of 32 rows in flight per lane
  static_assert(A >= 1 && A * LG * NS == P && (A == 1 || NS == 1), "strands of the lanes, groups and warps");
};

// Elements of one 32-bit word of a dense row, widened.
template <typename XT>
struct Word32;
template <>
struct Word32<float> {
  static constexpr int E = 1;
  __device__ __forceinline__ static void unpack(uint32_t w, float (&o)[1]) { o[0] = __uint_as_float(w); }
};
template <>
struct Word32<__nv_bfloat16> {
  static constexpr int E = 2;
  __device__ __forceinline__ static void unpack(uint32_t w, float (&o)[2]) {
    o[0] = __uint_as_float(w << 16);
    o[1] = __uint_as_float(w & 0xffff0000u);
  }
};
template <>
struct Word32<__half> {
  static constexpr int E = 2;
  __device__ __forceinline__ static void unpack(uint32_t w, float (&o)[2]) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w));
    o[0] = f.x;
    o[1] = f.y;
  }
};
template <>
struct Word32<__nv_fp8_e4m3> {
  static constexpr int E = 4;
  __device__ __forceinline__ static void unpack(uint32_t w, float (&o)[4]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const __half2_raw r = __nv_cvt_fp8x2_to_halfraw2((__nv_fp8x2_storage_t)(w >> (16 * h)), __NV_E4M3);
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&r));
      o[2 * h] = f.x;
      o[2 * h + 1] = f.y;
    }
  }
};

// kWarps warps per heavy item: warp (part, ws) has the words 32 part .. of
// the rows, its lane group lg the strands lg + LG ws, and A - 1 more.  The
// hardware hands out the blocks in order, so the longest class of items starts
// first.
// Spreading the strands of rows narrower than 512 bytes over a block's warps
// took 19 products of a 2,001-vertex graph at 33 columns from 513 to 348 us;
// on a matrix (12K rows of 250, 42 columns) it made a randomized SVD of
// 1454 us 55 us longer, so its items have kParts warps.
template <typename XT, int G, bool VAL, class Epi>
__global__ void __launch_bounds__(kHeavyWarps * 32, 4) k_spmm_heavy(const SpmmArgs<XT> s, const Epi epi) {
  using Tune = HeavyTune<G, VAL>;
  constexpr int W = Tune::W, LG = Tune::LG, A = Tune::A, NS = Tune::NS, kSets = Tune::kSets, EW = Word32<XT>::E;
  constexpr int kGap = LG * NS;     // from a lane's nonzero to its next
  constexpr int kStep = 32 * kGap;  // nonzeros of a set
  // the light rows' kernel may start: it does not read what this one writes
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // the item from the warp's number, not the block's: 32.4 us per product of
  // that graph against 35.8 us with the item in uniform registers
  const uint32_t unit = blockIdx.x * kHeavyWarps + (threadIdx.x >> 5);
  if (unit >= s.n_heavy * Tune::kWarps) return;  // (an item's warps in one block, all or none)
  const uint32_t it = unit / Tune::kWarps;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lg = lane / W;
  const int part = (int)(unit % Tune::kParts), ws = NS == 1 ? 0 : warp / Tune::kParts;
  const int q = part * 32 + lane % W;
  const bool on = q < s.C * 4;
  const uint4 rec = __ldg(reinterpret_cast<const uint4*>(s.items) + it);
  const uint32_t r = rec.z;
  const int len = (int)rec.w;
  const uint32_t* col = s.col + item_begin(rec);
  const float* val = VAL ? s.val + item_begin(rec) : nullptr;
  const uint32_t* X = reinterpret_cast<const uint32_t*>(s.X) + (on ? q : 0);
  const uint32_t ldw = (uint32_t)(s.ldx * (int64_t)sizeof(XT) / 4);
  float acc[A][EW];
#pragma unroll
  for (int a = 0; a < A; ++a)
#pragma unroll
    for (int e = 0; e < EW; ++e) acc[a][e] = 0.0f;
  // Ids and values pass through shared memory, each lane group's together,
  // so that one 16-byte broadcast serves four rows (a shuffle per row made
  // a chain of 30 cycles each); 36 words apart the groups meet no bank twice.
  __shared__ __align__(16) uint32_t sid[kHeavyWarps][LG * 36];
  __shared__ __align__(16) float sva[VAL ? kHeavyWarps : 1][VAL ? kSets : 1][VAL ? LG * 36 : 1];
  uint32_t* my_id = sid[warp];
  uint32_t w[kSets][32];  // words in flight
  uint32_t c[LG];         // ids (and values) of the set after those
  float v[LG];
  // entry `at` of this warp's 32 LG ids of a set: group at % LG, its at / LG-th
  auto nz = [&](int base, int at) { return NS == 1 ? base + at : base + kGap * (at / LG) + LG * ws + at % LG; };
  auto load_ids = [&](int base) {
#pragma unroll
    for (int i = 0; i < LG; ++i) {
      const int j = nz(base, 32 * i + lane);
      c[i] = j < len ? __ldg(col + j) : 0u;
      if (VAL) v[i] = j < len ? __ldg(val + j) : 0.0f;
    }
  };
  // the ids in c to shared memory, the next ones on their way, the gathers
  auto gather = [&](int base, int set, uint32_t (&o)[32]) {
    __syncwarp();
#pragma unroll
    for (int i = 0; i < LG; ++i) {
      const int at = 32 * i + lane;
      my_id[(at % LG) * 36 + at / LG] = c[i];
      if (VAL) sva[warp][set][(at % LG) * 36 + at / LG] = v[i];
    }
    __syncwarp();
    load_ids(base + kStep);
    const uint4* ids = reinterpret_cast<const uint4*>(my_id + lg * 36);
    if (base + kStep <= len) {
#pragma unroll
      for (int u = 0; u < 32; u += 4) {
        const uint4 cc = ids[u / 4];
        o[u] = __ldg(X + (uint64_t)cc.x * ldw);
        o[u + 1] = __ldg(X + (uint64_t)cc.y * ldw);
        o[u + 2] = __ldg(X + (uint64_t)cc.z * ldw);
        o[u + 3] = __ldg(X + (uint64_t)cc.w * ldw);
      }
    } else if (base < len) {
#pragma unroll
      for (int u = 0; u < 32; u += 4) {
        const uint4 cc = ids[u / 4];
        const uint32_t id[4] = {cc.x, cc.y, cc.z, cc.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
          o[u + i] = base + (u + i) * kGap + LG * ws + lg < len ? __ldg(X + (uint64_t)id[i] * ldw) : 0u;
      }
    }
  };
  auto add = [&](int base, int set, const uint32_t (&o)[32]) {
    const float4* vs = reinterpret_cast<const float4*>(sva[VAL ? warp : 0][VAL ? set : 0] + (VAL ? lg * 36 : 0));
    auto four = [&](int u, auto whole) {
      const float4 m4 = VAL ? vs[u / 4] : make_float4(1.0f, 1.0f, 1.0f, 1.0f);
      const float m[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float x[EW];
        Word32<XT>::unpack(o[u + i], x);
        if (decltype(whole)::value || base + (u + i) * kGap + LG * ws + lg < len) {
#pragma unroll
          for (int e = 0; e < EW; ++e) acc[(u + i) % A][e] = fmaf(m[i], x[e], acc[(u + i) % A][e]);
        }
      }
    };
    if (base + kStep <= len) {
#pragma unroll
      for (int u = 0; u < 32; u += 4) four(u, std::true_type{});
    } else if (base < len) {
#pragma unroll
      for (int u = 0; u < 32; u += 4) four(u, std::false_type{});
    }
  };
  load_ids(0);
#pragma unroll
  for (int k = 0; k < kSets; ++k) gather(k * kStep, k, w[k]);
  for (int base = 0; base < len; base += kSets * kStep) {
#pragma unroll
    for (int k = 0; k < kSets; ++k) {
      add(base + k * kStep, k, w[k]);
      __syncwarp();
      gather(base + (k + kSets) * kStep, k, w[k]);
    }
  }
  // the strands in a balanced tree: the lane groups', then the lane's own or
  // the warps'
#pragma unroll
  for (int o = W; o < 32; o <<= 1)
#pragma unroll
    for (int a = 0; a < A; ++a)
#pragma unroll
      for (int e = 0; e < EW; ++e) acc[a][e] += __shfl_xor_sync(kFull, acc[a][e], o);
#pragma unroll
  for (int o = 1; o < A; o <<= 1)
#pragma unroll
    for (int a = 0; a + o < A; a += 2 * o)
#pragma unroll
      for (int e = 0; e < EW; ++e) acc[a][e] += acc[a + o][e];
  if constexpr (NS > 1) {
    __shared__ float red[kHeavyWarps][32][EW];
    if (ws > 0) {
#pragma unroll
      for (int e = 0; e < EW; ++e) red[warp][lane][e] = acc[0][e];
    }
    __syncthreads();
    if (ws > 0) return;
#pragma unroll
    for (int e = 0; e < EW; ++e) {
      if constexpr (NS == 2)
        acc[0][e] += red[warp + Tune::kParts][lane][e];
      else
        acc[0][e] = (acc[0][e] + red[1][lane][e]) + (red[2][lane][e] + red[3][lane][e]);
    }
  }
  const bool out = on && lane < W;
  const int e0 = q * EW;
  const uint2 sp = it < s.n_big ? __ldg(s.span + it) : make_uint2(it, 1);
  if (sp.y > 1) {
    // a chunk: the warp that completes its row's last one adds them, in order
    if (out) {
#pragma unroll
      for (int e = 0; e < EW; ++e) __stcg(s.partial + (int64_t)it * s.ldp + e0 + e, acc[0][e]);
    }
    __threadfence();
    __syncwarp();
    unsigned* done = s.done + (int64_t)sp.x * Tune::kParts + part;
    unsigned before = 0;
    if (lane == 0) before = atomicAdd(done, 1u);
    before = __shfl_sync(kFull, before, 0);
    if (before + 1 != sp.y) return;
    __threadfence();
    if (lane == 0) *done = 0;  // ready for the next launch
    if (out) {
      const float* p = s.partial + (int64_t)sp.x * s.ldp + e0;
#pragma unroll
      for (int e = 0; e < EW; ++e) acc[0][e] = 0.0f;
      constexpr int kD = 8;  // chunks in flight
      for (unsigned i = 0; i < sp.y; i += kD) {
        float t[kD][EW];
#pragma unroll
        for (int d = 0; d < kD; ++d)
#pragma unroll
          for (int e = 0; e < EW; ++e) t[d][e] = i + d < sp.y ? __ldcg(p + (int64_t)(i + d) * s.ldp + e) : 0.0f;
#pragma unroll
        for (int d = 0; d < kD; ++d)
          if (i + d < sp.y)
#pragma unroll
            for (int e = 0; e < EW; ++e) acc[0][e] += t[d][e];
      }
    }
  }
  if (out) {
    const auto pre = epi.template load<EW>(r, s.e_base + e0);
    epi.template store<EW>(r, s.e_base + e0, acc[0], pre);
  }
}

// Every item to a warp, or (BAL) the rows of at most warp_max entries.
template <typename XT, int G, int VPL, bool VAL, bool BAL, class Epi>
__global__ void __launch_bounds__(kSpmmThreads, 4) k_spmm(const SpmmArgs<XT> s, const Epi epi) {
  using Tune = SpmmTune<XT, G, VPL>;
  constexpr int E = Tune::E, P = Tune::P, kU = Tune::kU, kB = Tune::kBatch, N = Tune::kEpi;
  constexpr bool kSplit = Tune::kSplit;
  // The operands of wider epilogues would not fit the registers beside the
  // gathers, nor would the next ids beside 16 sums per lane (whose matrices,
  // the sparsifier's, have hundreds of entries per row).
  constexpr bool kHoist = VPL == 1 && N == 4;
  constexpr bool kPipe = !VAL || VPL * E < 16;
  const int lane = threadIdx.x & 31;
  const int grp = lane / G, gl = lane % G;
  // G = 9: three groups of 9 lanes, lanes 27..31 idle
  const bool in_grp = grp < P;
  const bool epi_lane = lane < (kSplit ? 2 * G : G);
  const int e_lane = kSplit ? 4 * (grp & 1) : 0;
  // a step whose P kU nonzeros are all in the batch, on a slab that fills
  // the lane layout, loads without predicates: lanes past the groups
  // (27..31) read rows of valid columns too and their sums are not used
  const bool full_cols = s.C == G * VPL;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  uint32_t it = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if constexpr (BAL) {
    static_assert(VPL == 1 && (G & (G - 1)) == 0, "the balanced form has one vector per lane");
    it += s.n_heavy;
  }
  const uint4* items = reinterpret_cast<const uint4*>(s.items);
  const uint4 none = make_uint4(0, 0, 0, 0);
  uint4 nxt = it < s.n_items ? __ldg(items + it) : none;
  uint32_t c = 0;
  float v = 1.0f;
  if constexpr (kPipe) {
    const int cnt = (int)nxt.w < kB ? (int)nxt.w : kB;
    if (lane < cnt) c = __ldg(s.col + item_begin(nxt) + lane);
    if (VAL) v = lane < cnt ? __ldg(s.val + item_begin(nxt) + lane) : 0.0f;
  }
  for (; it < s.n_items; it += nwarps) {
    const uint2 sp = !BAL && it < s.n_big ? __ldg(s.span + it) : make_uint2(it, 1);
    const bool chunk = !BAL && sp.y > 1;
    const uint32_t r = nxt.z;
    int left = (int)nxt.w;               // nonzeros from jb on
    int64_t jb = item_begin(nxt);
    if constexpr (kPipe) nxt = it + nwarps < s.n_items ? __ldg(items + it + nwarps) : none;
    typename Epi::template Pre<N> pre[VPL];
    if (kHoist && !chunk && epi_lane) {
#pragma unroll
      for (int k = 0; k < VPL; ++k) {
        const int ch = gl + G * k;
        if (ch < s.C) pre[k] = epi.template load<N>(r, s.e_base + ch * E + e_lane);
      }
    }
    float acc[VPL][E];
#pragma unroll
    for (int k = 0; k < VPL; ++k)
#pragma unroll
      for (int e = 0; e < E; ++e) acc[k][e] = 0.f;
    do {
      const int cnt = left < kB ? left : kB;
      if constexpr (!kPipe) {
        c = lane < cnt ? __ldg(s.col + jb + lane) : 0u;
        if (VAL) v = lane < cnt ? __ldg(s.val + jb + lane) : 0.0f;
      }
      uint32_t c2 = 0;
      float v2 = 1.0f;
      bool fetched = !kPipe;
      // the ids after these: the item's next batch, or the next item's first
      auto fetch = [&]() {
        fetched = true;
        const bool last = left <= kB;
        const int64_t j2 = last ? item_begin(nxt) : jb + kB;
        int cnt2 = last ? (int)nxt.w : left - kB;
        cnt2 = cnt2 < kB ? cnt2 : kB;
        if (lane < cnt2) c2 = __ldg(s.col + j2 + lane);
        if (VAL) v2 = lane < cnt2 ? __ldg(s.val + j2 + lane) : 0.0f;
      };
      auto step = [&](int t0, auto checked) {
        constexpr bool kChecked = decltype(checked)::value;
        uint4 raw[kU][VPL];
        float vv[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          if (kChecked && u > 0 && t0 + u * P >= cnt) {  // the same for the whole warp
            vv[u] = 0.0f;
#pragma unroll
            for (int k = 0; k < VPL; ++k) raw[u][k] = make_uint4(0, 0, 0, 0);
            continue;
          }
          const int t = t0 + u * P + grp;
          const uint32_t cc = __shfl_sync(kFull, c, t & 31);
          vv[u] = VAL ? __shfl_sync(kFull, v, t & 31) : 1.f;
          const XT* xr = s.X + (int64_t)cc * s.ldx;
#pragma unroll
          for (int k = 0; k < VPL; ++k) {
            const int ch = gl + G * k;
            if constexpr (kChecked)
              raw[u][k] = (in_grp && t < cnt && ch < s.C) ? __ldg(reinterpret_cast<const uint4*>(xr + ch * E))
                                                          : make_uint4(0, 0, 0, 0);
            else
              raw[u][k] = __ldg(reinterpret_cast<const uint4*>(xr + ch * E));
          }
        }
        if (!fetched) fetch();  // behind the first gathers, ahead of their FMAs
#pragma unroll
        for (int u = 0; u < kU; ++u) {
          if (kChecked && u > 0 && t0 + u * P >= cnt) break;
#pragma unroll
          for (int k = 0; k < VPL; ++k) {
            float x[E];
            Vec16<XT>::unpack(raw[u][k], x);
            // paired FP32 FMAs: each element rounded as by fmaf
#pragma unroll
            for (int e = 0; e < E; e += 2) {
              const float2 q = __ffma2_rn(make_float2(vv[u], vv[u]), make_float2(x[e], x[e + 1]),
                                          make_float2(acc[k][e], acc[k][e + 1]));
              acc[k][e] = q.x;
              acc[k][e + 1] = q.y;
            }
          }
        }
      };
      for (int t0 = 0; t0 < cnt; t0 += P * kU) {
        if (full_cols && t0 + P * kU <= cnt)
          step(t0, std::false_type{});
        else
          step(t0, std::true_type{});
      }
      if (kPipe && !fetched) fetch();  // an empty row
      left -= kB;
      jb += kB;
      if constexpr (kPipe) {
        c = c2;
        v = v2;
      }
    } while (left > 0);
    if constexpr (!kPipe) nxt = it + nwarps < s.n_items ? __ldg(items + it + nwarps) : none;

    // add the groups' sums: in sum[k], the elements of this lane's epilogue
    float sum[VPL][N];
    if constexpr (kSplit) {
      // the two halves of a vector change places between neighbouring groups
      const bool hi = grp & 1;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float give = hi ? acc[0][e] : acc[0][4 + e];
        const float keep = hi ? acc[0][4 + e] : acc[0][e];
        sum[0][e] = keep + __shfl_xor_sync(kFull, give, G);
      }
#pragma unroll
      for (int o = 2 * G; o < 32; o <<= 1)
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[0][e] += __shfl_xor_sync(kFull, sum[0][e], o);
    } else {
      if constexpr ((G & (G - 1)) == 0) {
#pragma unroll
        for (int o = G; o < 32; o <<= 1)
#pragma unroll
          for (int k = 0; k < VPL; ++k)
#pragma unroll
            for (int e = 0; e < E; ++e) acc[k][e] += __shfl_xor_sync(kFull, acc[k][e], o);
      } else {
        static_assert(P == 3, "non-power-of-two groups: three groups per warp");
#pragma unroll
        for (int k = 0; k < VPL; ++k)
#pragma unroll
          for (int e = 0; e < E; ++e) {
            const float g1 = __shfl_down_sync(kFull, acc[k][e], G);
            const float g2 = __shfl_down_sync(kFull, acc[k][e], 2 * G);
            acc[k][e] = (acc[k][e] + g1) + g2;
          }
      }
#pragma unroll
      for (int k = 0; k < VPL; ++k)
#pragma unroll
        for (int e = 0; e < N; ++e) sum[k][e] = acc[k][e];
    }

    if (!chunk) {
      if (epi_lane) {
#pragma unroll
        for (int k = 0; k < VPL; ++k) {
          const int ch = gl + G * k;
          if (ch >= s.C) continue;
          if (!kHoist) pre[k] = epi.template load<N>(r, s.e_base + ch * E + e_lane);
          epi.template store<N>(r, s.e_base + ch * E + e_lane, sum[k], pre[k]);
        }
      }
    } else {
      if (epi_lane) {
#pragma unroll
        for (int k = 0; k < VPL; ++k) {
          const int ch = gl + G * k;
          if (ch < s.C) {
            float* p = s.partial + (int64_t)it * s.ldp + ch * E + e_lane;
#pragma unroll
            for (int q = 0; q < N; q += 4)
              __stcg(reinterpret_cast<float4*>(p + q), make_float4(sum[k][q], sum[k][q + 1], sum[k][q + 2], sum[k][q + 3]));
          }
        }
      }
      // the warp that completes the row's last chunk adds them all, in order
      __threadfence();
      __syncwarp();
      unsigned before = 0;
      if (lane == 0) before = atomicAdd(s.done + sp.x, 1u);
      before = __shfl_sync(kFull, before, 0);
      if (before + 1 == sp.y) {
        __threadfence();
        if (lane == 0) s.done[sp.x] = 0;  // ready for the next launch
        const int cols = s.C * E;
        for (int q = lane * 4; q < cols; q += 128) {
          const auto fin = epi.template load<4>(r, s.e_base + q);
          const float* p = s.partial + (int64_t)sp.x * s.ldp + q;
          float t[4] = {0.f, 0.f, 0.f, 0.f};
          constexpr int kD = 4;  // chunks in flight
          for (unsigned i = 0; i < sp.y; i += kD) {
            float4 w[kD];
#pragma unroll
            for (int d = 0; d < kD; ++d)
              w[d] = i + d < sp.y ? __ldcg(reinterpret_cast<const float4*>(p + (int64_t)(i + d) * s.ldp))
                                  : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int d = 0; d < kD; ++d) {
              if (i + d < sp.y) {
                t[0] += w[d].x;
                t[1] += w[d].y;
                t[2] += w[d].z;
                t[3] += w[d].w;
              }
            }
          }
          epi.template store<4>(r, s.e_base + q, t, fin);
        }
        __syncwarp();
      }
    }
  }
  // Launched beside k_spmm_heavy, whose blocks have all started by then:
  // this launch ends after that one, so that what follows it on the stream
  // sees the rows of both.
  if constexpr (BAL) asm volatile("griddepcontrol.wait;" ::: "memory");
}

}  // namespace lne
