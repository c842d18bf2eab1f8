// Spectral propagation: the Bessel-weighted Chebyshev filter on
// M = I - D~^-1 A~ - mu I (A~ = A + I, D~ = D + I), then (A + I) a.
//
// Reference: spectral_propagation::chebyshev_expansion
// (LightNE/SpectralPropagation.h:45-221):
//   Lx0 = a;  tmp = M a;  Lx1 = 0.5 M tmp - a;  conv = I0(s) Lx0 - 2 I1(s) Lx1
//   for k = 2 .. order-1:  tmp = M Lx1;  Lx2 = M tmp - Lx0 - 2 Lx1;
//                          conv += (k odd ? -2 : 2) I_k(s) Lx2;  rotate
//   a -= conv;  y = (A + I) a
// M is applied as an implicit operator: row i has the value
// (float)(1 - mu - 1/d~_i) on the diagonal and (float)(-1/d~_i) on each
// neighbour (the reference stores these floats in a CSR, :59-75), so
// (M x)_i = m_i x_i + o_i * sum_{j in N(i)} x_j with the neighbour sum
// gathered by the SpMM core.  Every half-step is one product whose epilogue
// applies the recursion's axpbys while the row is in registers (one kernel,
// and a second beside it for the long rows of a graph that has some).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <type_traits>
#include <vector>

#include "dense.h"
#include "dense_common.cuh"
#include "lne_internal.h"
#include "spmm_core.cuh"
#include "spmm_dispatch.cuh"

namespace lne {

// Modified Bessel function of the first kind I_k(x) by its power series
// sum_m (x/2)^(2m+k) / (m! (m+k)!), summed in long double until the terms
// vanish (x = 0.5 in LightNE; the series converges for every x).
double bessel_i(int k, double x) {
  long double h = (long double)x / 2.0L, term = 1.0L;
  for (int i = 1; i <= k; ++i) term *= h / (long double)i;
  long double sum = term;
  for (int m = 1; m < 500; ++m) {
    term *= h * h / ((long double)m * (long double)(m + k));
    sum += term;
    if (term < sum * 1e-21L) break;
  }
  return (double)sum;
}

void chebyshev_coeffs(int order, double s, std::vector<float>& c) {
  // the reference evaluates iv(k, s) with s a float and narrows each axpy
  // coefficient to float (SpectralPropagation.h:129-197)
  const double sf = (double)(float)s;
  c.assign(order > 2 ? order : 2, 0.0f);
  c[0] = (float)bessel_i(0, sf);
  c[1] = (float)(-2.0 * bessel_i(1, sf));
  for (int k = 2; k < order; ++k) c[k] = (float)(((k & 1) ? -2.0 : 2.0) * bessel_i(k, sf));
}

namespace {

// Type of the 16-bit shadow copies of the propagation vectors that the
// SpMM gathers: the operand type itself in the 16-bit forms (the FP32 form
// keeps no shadows; its shadow pointers stay null).
template <typename XT>
struct ShadowOf {
  using type = __nv_bfloat16;
};
template <>
struct ShadowOf<__half> {
  using type = __half;
};

// Per-row operator data: x = diagonal m_i, y = off-diagonal o_i (the floats
// the reference stores), z = d~_i = deg + 1, w = 1 / d~_i.
__global__ void k_op_coef(const Vertex* __restrict__ vd, int64_t n, float mu, float4* __restrict__ coef) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float dt = (float)(vd[i].deg + 1u);
  const double inv = 1.0 / (double)dt;
  coef[i] = make_float4((float)(1.0 - (double)mu - inv), (float)(-inv), dt, (float)inv);
}

// W 32-bit words at p (16-, 8- or 4-byte accesses; p aligned to them).
template <int W>
__device__ __forceinline__ void load_words(const uint32_t* __restrict__ p, uint32_t (&w)[W]) {
  if constexpr (W % 4 == 0) {
#pragma unroll
    for (int i = 0; i < W; i += 4) {
      const uint4 v = *reinterpret_cast<const uint4*>(p + i);
      w[i] = v.x; w[i + 1] = v.y; w[i + 2] = v.z; w[i + 3] = v.w;
    }
  } else if constexpr (W == 2) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    w[0] = v.x; w[1] = v.y;
  } else {
    static_assert(W == 1, "one, two or a multiple of four words");
    w[0] = *p;
  }
}
template <int W>
__device__ __forceinline__ void store_words(uint32_t* __restrict__ p, const uint32_t (&w)[W]) {
  if constexpr (W % 4 == 0) {
#pragma unroll
    for (int i = 0; i < W; i += 4) *reinterpret_cast<uint4*>(p + i) = make_uint4(w[i], w[i + 1], w[i + 2], w[i + 3]);
  } else if constexpr (W == 2) {
    *reinterpret_cast<uint2*>(p) = make_uint2(w[0], w[1]);
  } else {
    static_assert(W == 1, "one, two or a multiple of four words");
    *p = w[0];
  }
}

// N elements of a dense row as loaded (16-bit types: not yet widened); an
// epilogue sees 4 or 8 of them, or one 32-bit word's.
template <typename T, int N>
struct RawRow {
  static constexpr int W = N * (int)sizeof(T) / 4;
  uint32_t w[W];
  __device__ __forceinline__ void load(const T* __restrict__ X, int64_t ld, int64_t r, int e0) {
    load_words<W>(reinterpret_cast<const uint32_t*>(X + r * ld + e0), w);
  }
  __device__ __forceinline__ float at(int i) const {
    if constexpr (sizeof(T) == 4) {
      return __uint_as_float(w[i]);
    } else if constexpr (std::is_same<T, __half>::value) {
      const __half2 h = *reinterpret_cast<const __half2*>(&w[i >> 1]);
      return (i & 1) ? __high2float(h) : __low2float(h);
    } else {
      return __uint_as_float((i & 1) ? (w[i >> 1] & 0xffff0000u) : (w[i >> 1] << 16));
    }
  }
};
// FP32 state of the recursion: read and written once per product, with the
// streaming policy, so that it does not push the gathered operand out of L2.
template <int N>
__device__ __forceinline__ void load_f32(const float* __restrict__ X, int64_t ld, int64_t r, int e0, float (&o)[N]) {
  const float* p = X + r * ld + e0;
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      const float4 v = __ldcs(reinterpret_cast<const float4*>(p + i));
      o[i] = v.x; o[i + 1] = v.y; o[i + 2] = v.z; o[i + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) o[i] = __ldcs(p + i);
  }
}
template <int N>
__device__ __forceinline__ void store_f32(float* __restrict__ X, int64_t ld, int64_t r, int e0, const float (&o)[N]) {
  uint32_t w[N];
#pragma unroll
  for (int i = 0; i < N; ++i) w[i] = __float_as_uint(o[i]);
  store_words<N>(reinterpret_cast<uint32_t*>(X + r * ld + e0), w);
}
template <int N>
__device__ __forceinline__ void store_f32_cs(float* __restrict__ X, int64_t ld, int64_t r, int e0,
                                             const float (&o)[N]) {
  float* p = X + r * ld + e0;
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int i = 0; i < N; i += 4)
      __stcs(reinterpret_cast<float4*>(p + i), make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]));
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) __stcs(p + i, o[i]);
  }
}
// A Chebyshev vector's FP32 copy: gathered by the next product in the FP32
// form only.
template <typename XT, int N>
__device__ __forceinline__ void store_state(float* __restrict__ X, int64_t ld, int64_t r, int e0,
                                            const float (&o)[N]) {
  if constexpr (sizeof(XT) == 4)
    store_f32<N>(X, ld, r, e0, o);
  else
    store_f32_cs<N>(X, ld, r, e0, o);
}
template <typename HT, int N>
__device__ __forceinline__ void store_16(HT* __restrict__ X, int64_t ld, int64_t r, int e0, const float (&o)[N]) {
  if constexpr (N % 2 == 0) {  // (an FP32 form keeps no 16-bit copies)
    uint32_t w[N / 2];
#pragma unroll
    for (int i = 0; i < N; i += 2) w[i / 2] = pack2_16<HT>(o[i], o[i + 1]);
    store_words<N / 2>(reinterpret_cast<uint32_t*>(X + r * ld + e0), w);
  }
}

// The coefficients of row r that an epilogue needs: {m_i, o_i}, or d~_i.
__device__ __forceinline__ float2 coef_mo(const float4* __restrict__ coef, int64_t r) {
  return __ldg(reinterpret_cast<const float2*>(coef + r));
}
__device__ __forceinline__ float coef_dt(const float4* __restrict__ coef, int64_t r) {
  return __ldg(reinterpret_cast<const float*>(coef + r) + 2);
}

// Epilogues of the SpMM (spmm_core.cuh): load() fetches the row's operands
// ahead of the gathers, store() applies the recursion to the finished sums.

// tmp = M x: out = m_i x_i + o_i acc (operand x of type XT); FP32 and/or
// 16-bit outputs.
template <typename XT>
struct EpiApplyM {
  using HT = typename ShadowOf<XT>::type;
  const float4* __restrict__ coef;
  const XT* __restrict__ X;  // the operand (diagonal term)
  int64_t ld;
  float* __restrict__ out_f;
  HT* __restrict__ out_b;
  template <int N>
  struct Pre {
    float2 c;
    RawRow<XT, N> x;
  };
  template <int N>
  __device__ __forceinline__ Pre<N> load(int64_t r, int e0) const {
    Pre<N> q;
    q.c = coef_mo(coef, r);
    q.x.load(X, ld, r, e0);
    return q;
  }
  template <int N>
  __device__ __forceinline__ void store(int64_t r, int e0, const float (&a)[N], const Pre<N>& q) const {
    float y[N];
#pragma unroll
    for (int i = 0; i < N; ++i) y[i] = fmaf(q.c.x, q.x.at(i), q.c.y * a[i]);
    if (out_f) store_f32<N>(out_f, ld, r, e0, y);
    if (out_b) store_16<HT, N>(out_b, ld, r, e0, y);
  }
};

// Final vector of a filter: fin = base_scale base - (scale_dt ? d~_i : 1)
// conv, written as out_scale fin (FP32) and fin (16-bit); either may be null.
template <typename HT>
struct FinalOut {
  const float* __restrict__ base = nullptr;  // null: not the final step
  bool scale_dt = false;
  float* __restrict__ out = nullptr;
  HT* __restrict__ outb = nullptr;
  float base_scale = 1.0f, out_scale = 1.0f;
  template <int N>
  __device__ __forceinline__ void apply(int64_t r, int e0, int64_t ld, const float4* __restrict__ coef,
                                        const float (&cv)[N]) const {
    float b[N], f[N];
    load_f32<N>(base, ld, r, e0, b);
    const float sc = scale_dt ? coef_dt(coef, r) : 1.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) f[i] = fmaf(-sc, cv[i], base_scale * b[i]);
    if (outb) store_16<HT, N>(outb, ld, r, e0, f);
    if (out) {
#pragma unroll
      for (int i = 0; i < N; ++i) f[i] *= out_scale;
      store_f32<N>(out, ld, r, e0, f);
    }
  }
};

// First order: Lx1 = 0.5 M tmp - x;  conv = c0 x + c1 Lx1 (conv may be null:
// the tangent pass keeps no sum);  or the final vector when order <= 2.
// x = x_scale A.
template <typename XT>
struct EpiFirst {
  using HT = typename ShadowOf<XT>::type;
  const float4* __restrict__ coef;
  const XT* __restrict__ T;        // tmp (operand)
  const float* __restrict__ A;     // x (FP32)
  float* __restrict__ L1;          // Lx1 FP32
  HT* __restrict__ L1b;            // Lx1 16-bit copy (16-bit forms) or null
  float* __restrict__ conv;
  FinalOut<HT> fin;
  int64_t ld;
  float c0, c1;
  float x_scale;
  template <int N>
  struct Pre {
    float2 c;
    RawRow<XT, N> t;
    float a[N];
  };
  template <int N>
  __device__ __forceinline__ Pre<N> load(int64_t r, int e0) const {
    Pre<N> q;
    q.c = coef_mo(coef, r);
    q.t.load(T, ld, r, e0);
    load_f32<N>(A, ld, r, e0, q.a);
    return q;
  }
  template <int N>
  __device__ __forceinline__ void store(int64_t r, int e0, const float (&acc)[N], const Pre<N>& q) const {
    float l1[N], cv[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float a = x_scale * q.a[i];
      const float mt = fmaf(q.c.x, q.t.at(i), q.c.y * acc[i]);
      l1[i] = fmaf(0.5f, mt, -a);
      cv[i] = fmaf(c1, l1[i], c0 * a);
    }
    if (L1) store_state<XT, N>(L1, ld, r, e0, l1);
    if (L1b) store_16<HT, N>(L1b, ld, r, e0, l1);
    if (fin.base)
      fin.template apply<N>(r, e0, ld, coef, cv);
    else if (conv)
      store_f32_cs<N>(conv, ld, r, e0, cv);
  }
};

// Order k >= 2: Lx2 = M tmp - Lx0 - 2 Lx1;  conv += ck Lx2 (conv may be
// null);  or the final vector on the last order.  Lx0 = l0_scale L0.
// The sum is read and written every second order: `skip` leaves conv alone
// and the next order adds ck_prev Lx1 (the skipped order's vector) as well.
// TAN (the tangent pass): Lx2 = M tmp - Lx0 - 2 Lx1 - 2 extra, where L0 ==
// null means a zero Lx0.
template <typename XT, bool TAN = false>
struct EpiStep {
  using HT = typename ShadowOf<XT>::type;
  const float4* __restrict__ coef;
  const XT* __restrict__ T;
  const float* __restrict__ L0;
  const float* __restrict__ L1;
  float* __restrict__ L2;          // null: not stored (the last order)
  HT* __restrict__ L2b;
  float* __restrict__ conv;
  FinalOut<HT> fin;
  int64_t ld;
  float ck;
  float ck_prev = 0.0f;
  bool skip = false;
  float l0_scale = 1.0f;
  const float* __restrict__ extra = nullptr;
  template <int N>
  struct Pre {
    float2 c;
    RawRow<XT, N> t;
    float l0[N], l1[N], cv[N], ex[TAN ? N : 1];
  };
  template <int N>
  __device__ __forceinline__ Pre<N> load(int64_t r, int e0) const {
    Pre<N> q;
    q.c = coef_mo(coef, r);
    q.t.load(T, ld, r, e0);
    if (!TAN || L0) {
      load_f32<N>(L0, ld, r, e0, q.l0);
    } else {
#pragma unroll
      for (int i = 0; i < N; ++i) q.l0[i] = 0.0f;
    }
    load_f32<N>(L1, ld, r, e0, q.l1);
    if constexpr (TAN) load_f32<N>(extra, ld, r, e0, q.ex);
    if (conv && !skip) load_f32<N>(conv, ld, r, e0, q.cv);
    return q;
  }
  template <int N>
  __device__ __forceinline__ void store(int64_t r, int e0, const float (&acc)[N], const Pre<N>& q) const {
    float l2[N], cv[N];
    const bool sum = conv && !skip;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const float mt = fmaf(q.c.x, q.t.at(i), q.c.y * acc[i]);
      l2[i] = fmaf(-2.0f, q.l1[i], fmaf(-l0_scale, q.l0[i], mt));
      if constexpr (TAN) l2[i] = fmaf(-2.0f, q.ex[i], l2[i]);
      cv[i] = fmaf(ck, l2[i], sum ? fmaf(ck_prev, q.l1[i], q.cv[i]) : 0.0f);
    }
    if (fin.base) {
      fin.template apply<N>(r, e0, ld, coef, cv);
    } else {
      if (L2) store_state<XT, N>(L2, ld, r, e0, l2);
      if (L2b) store_16<HT, N>(L2b, ld, r, e0, l2);
      if (sum) store_f32_cs<N>(conv, ld, r, e0, cv);
    }
  }
};

// y = (A + I) x: out = out_scale * (x_i + acc), written with leading
// dimension ldy for columns < d (out_scale undoes the input scaling of the
// FP16 form; 1 otherwise); vec: Y's rows are whole 16-byte vectors.
template <typename XT>
struct EpiAPlusI {
  const XT* __restrict__ X;
  int64_t ld;
  float* __restrict__ Y;
  int64_t ldy;
  int d;
  float out_scale;
  bool vec;
  template <int N>
  struct Pre {
    RawRow<XT, N> x;
  };
  template <int N>
  __device__ __forceinline__ Pre<N> load(int64_t r, int e0) const {
    Pre<N> q;
    q.x.load(X, ld, r, e0);
    return q;
  }
  template <int N>
  __device__ __forceinline__ void store(int64_t r, int e0, const float (&acc)[N], const Pre<N>& q) const {
    float o[N];
#pragma unroll
    for (int i = 0; i < N; ++i) o[i] = out_scale * (q.x.at(i) + acc[i]);
    if (vec) {
      store_f32<N>(Y, ldy, r, e0, o);
      return;
    }
    float* y = Y + r * ldy + e0;
#pragma unroll
    for (int i = 0; i < N; ++i)
      if (e0 + i < d) y[i] = o[i];
  }
};

// Adjoint start: h = (A + I) g;  b = h / d~_i (FP32, may be null, and 16-bit
// copy).
template <typename XT>
struct EpiAdjInit {
  using HT = typename ShadowOf<XT>::type;
  const float4* __restrict__ coef;
  const XT* __restrict__ G;
  int64_t ld;
  float* __restrict__ H;
  float* __restrict__ Bf;
  HT* __restrict__ Bb;
  template <int N>
  struct Pre {
    float inv_dt;
    RawRow<XT, N> g;
  };
  template <int N>
  __device__ __forceinline__ Pre<N> load(int64_t r, int e0) const {
    Pre<N> q;
    q.inv_dt = __ldg(reinterpret_cast<const float*>(coef + r) + 3);
    q.g.load(G, ld, r, e0);
    return q;
  }
  template <int N>
  __device__ __forceinline__ void store(int64_t r, int e0, const float (&acc)[N], const Pre<N>& q) const {
    float h[N], b[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
      h[i] = q.g.at(i) + acc[i];
      b[i] = h[i] * q.inv_dt;
    }
    store_f32<N>(H, ld, r, e0, h);
    if (Bf) store_f32<N>(Bf, ld, r, e0, b);
    if (Bb) store_16<HT, N>(Bb, ld, r, e0, b);
  }
};

// dst (n x ld, zero padding; may be null) = scale * src (n x d) and its
// 16-bit copy (may be null).
template <typename HT>
__global__ void k_pad_copy(const float* __restrict__ src, int64_t n, int d, float scale, float* __restrict__ dst,
                           int64_t ld, HT* __restrict__ dstb) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n * ld; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / ld;
    const int j = (int)(t - i * ld);
    const float v = j < d ? scale * src[i * d + j] : 0.0f;
    if (dst) dst[t] = v;
    if (dstb) {
      if constexpr (std::is_same<HT, __half>::value)
        dstb[t] = __float2half_rn(v);
      else
        dstb[t] = __float2bfloat16_rn(v);
    }
  }
}

// dst = the 16-bit copy of scale * src, total a multiple of 8 values, both
// 16-byte aligned.
template <typename HT>
__global__ void k_shadow_copy(const float4* __restrict__ src, int64_t total8, float scale, uint4* __restrict__ dst) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total8; t += (int64_t)gridDim.x * blockDim.x) {
    const float4 a = __ldcs(src + 2 * t), b = __ldcs(src + 2 * t + 1);
    dst[t] = make_uint4(pack2_16<HT>(scale * a.x, scale * a.y), pack2_16<HT>(scale * a.z, scale * a.w),
                        pack2_16<HT>(scale * b.x, scale * b.y), pack2_16<HT>(scale * b.z, scale * b.w));
  }
}

// dst (n x d) = scale * src (n x ld).
__global__ void k_unpad_copy(const float* __restrict__ src, int64_t ld, int64_t n, int d, float scale,
                             float* __restrict__ dst) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < n * d; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = t / d;
    dst[t] = scale * src[i * ld + (t - i * d)];
  }
}

// Largest |x| over an n x d FP32 matrix (row stride d): one float per
// block; non-finite values count as +inf.
static constexpr int kAmaxBlocks = 1216;
__global__ void k_amax_partial(const float* __restrict__ x, int64_t total, float* __restrict__ out) {
  float m = 0.0f;
  auto take = [&](float v) {
    const float a = fabsf(v);
    m = (a <= m) ? m : (isfinite(a) ? a : INFINITY);
  };
  // 16-byte loads where x allows, two in flight; then the rest
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nth = (int64_t)gridDim.x * blockDim.x;
  const int64_t n4 = (reinterpret_cast<uintptr_t>(x) & 15) == 0 ? total / 4 : 0;
  const float4* x4 = reinterpret_cast<const float4*>(x);
  for (int64_t t = tid; t < n4; t += 2 * nth) {
    const float4 a = x4[t], b = t + nth < n4 ? x4[t + nth] : make_float4(0.f, 0.f, 0.f, 0.f);
    take(a.x); take(a.y); take(a.z); take(a.w);
    take(b.x); take(b.y); take(b.z); take(b.w);
  }
  for (int64_t t = 4 * n4 + tid; t < total; t += nth) take(x[t]);
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, o));
  __shared__ float ws[32];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.0f;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t = fmaxf(t, ws[i]);
    out[blockIdx.x] = t;
  }
}

// y = alpha x.
__global__ void k_scale_copy(const float* __restrict__ x, int64_t total, float alpha, float* __restrict__ y) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x)
    y[t] = alpha * x[t];
}

// <h, x> partial sums: FP32 within a thread, FP64 across threads, one
// value per block (summed in block order on the host).
static constexpr int kDotBlocks = 1024;
__global__ void k_dot_partial(const float* __restrict__ h, const float* __restrict__ x, int64_t total,
                              double* __restrict__ out) {
  float s = 0.0f;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x)
    s = fmaf(h[t], x[t], s);
  double d = (double)s;
  for (int o = 16; o > 0; o >>= 1) d += __shfl_down_sync(kFull, d, o);
  __shared__ double ws[32];
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = d;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += ws[i];
    out[blockIdx.x] = t;
  }
}

struct Bufs {
  lne_ctx* ctx;
  std::vector<void*> ptrs;
  explicit Bufs(lne_ctx* c) : ctx(c) {}
  template <typename T>
  int get(T** out, size_t count, const char* what) {
    void* p = nullptr;
    int rc = dalloc(ctx, &p, sizeof(T) * (count > 0 ? count : 1), what);
    if (rc == LNE_OK) ptrs.push_back(p);
    *out = (T*)p;
    return rc;
  }
  ~Bufs() {
    for (void* p : ptrs) dfree(ctx, p);
  }
};

// Shared state of one filter evaluation.
template <typename XT>
struct Filter {
  static constexpr bool k16 = sizeof(XT) == 2;
  using HT = typename ShadowOf<XT>::type;
  lne_ctx* ctx;
  lne_graph* g;
  int64_t n, ld;
  const float4* coef;
  int* launches;
  Bufs* B;
  const SpmmWork* work;
  size_t sz() const { return (size_t)n * ld; }

  // operand view of an FP32 vector with an optional 16-bit copy
  const XT* op(const float* f, const HT* b) const { return k16 ? (const XT*)b : (const XT*)f; }

  template <class Epi>
  int spmm(const XT* X, const Epi& epi) {
    return spmm_run<XT, false>(ctx, g->plan, g->nbrs, nullptr, X, ld, ld, epi, launches, 0, work);
  }

  int apply_m(const XT* X, float* out_f, HT* out_b) {
    return spmm(X, EpiApplyM<XT>{coef, X, ld, out_f, out_b});
  }

  // The Chebyshev filter on x = x_scale xf (operand copy xb):
  // fin.base_scale fin.base - scale * sum_k c_k T_k(X) x written as `fin`
  // says.
  int run(const float* xf, const HT* xb, float x_scale, int order, const std::vector<float>& c,
          const FinalOut<HT>& fin) {
    int rc;
    float *conv = nullptr, *Tf = nullptr;
    HT* Tb = nullptr;
    float* ring[3] = {nullptr, nullptr, nullptr};
    HT* ringb[3] = {nullptr, nullptr, nullptr};
    const int nring = order > 2 ? 3 : 0;
    if (order > 2 && (rc = B->get(&conv, sz(), "conv"))) return rc;
    for (int i = 0; i < nring; ++i) {
      if ((rc = B->get(&ring[i], sz(), "Chebyshev vector"))) return rc;
      if (k16 && (rc = B->get(&ringb[i], sz(), "Chebyshev vector 16-bit"))) return rc;
    }
    if (k16) {
      if ((rc = B->get(&Tb, sz(), "tmp 16-bit"))) return rc;
    } else if ((rc = B->get(&Tf, sz(), "tmp"))) {
      return rc;
    }
    const XT* X0 = op(xf, xb);
    const XT* Tx = k16 ? (const XT*)Tb : (const XT*)Tf;
    if ((rc = apply_m(X0, k16 ? nullptr : Tf, k16 ? Tb : nullptr))) return rc;  // tmp = M x
    {
      const FinalOut<HT> fo = order <= 2 ? fin : FinalOut<HT>();
      EpiFirst<XT> epi{coef, Tx, xf, ring[0], ringb[0], conv, fo, ld, c[0], c[1], x_scale};
      if ((rc = spmm(Tx, epi))) return rc;
    }
    const float* l0 = xf;
    float l0_scale = x_scale;
    int j1 = 0;
    for (int k = 2; k < order; ++k) {
      const int j2 = (j1 + 1) % 3;
      if ((rc = apply_m(op(ring[j1], ringb[j1]), k16 ? nullptr : Tf, k16 ? Tb : nullptr))) return rc;
      const bool last = k == order - 1;
      const FinalOut<HT> fo = last ? fin : FinalOut<HT>();
      // conv is updated on odd orders (and on the last): even orders are
      // added with the next one
      const bool skip = !last && (k % 2 == 0);
      const float ck_prev = (k % 2 == 1) ? c[k - 1] : 0.0f;
      float* out = last ? nullptr : ring[j2];
      HT* outb = last ? nullptr : ringb[j2];
      EpiStep<XT> epi{coef, Tx, l0, ring[j1], out, outb, conv, fo, ld, c[k], ck_prev, skip, l0_scale};
      if ((rc = spmm(Tx, epi))) return rc;
      l0 = ring[j1];
      l0_scale = 1.0f;
      j1 = j2;
    }
    return LNE_OK;
  }
};

template <typename XT>
int setup_filter(lne_ctx* ctx, lne_graph* g, const lne_propagate_params* p, Bufs& B, SpmmWork* work, int* launches,
                 Filter<XT>& F) {
  const int64_t n = g->n, ld = pad_ld(p->dim);
  float4* coef = nullptr;
  int rc;
  if ((rc = B.get(&coef, n, "operator coefficients"))) return rc;
  // the partial sums of the long rows, as wide as the FP32 form needs them
  if ((rc = spmm_work_alloc(ctx, g->plan, std::max(spmm_work_width<XT>(ld), spmm_work_width<float>(ld)), work))) return rc;
  B.ptrs.push_back(work->partial);
  k_op_coef<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(g->vdata, n, (float)p->mu, coef);
  *launches += 1;
  F = Filter<XT>{ctx, g, n, ld, coef, launches, &B, work};
  return LNE_OK;
}

// An n x ld FP32 matrix the kernels can read and write in 16-byte vectors.
bool rows_direct(const void* p, int64_t d, int64_t ld) { return d == ld && ((uintptr_t)p & 15) == 0; }
bool ranges_overlap(const void* a, const void* b, size_t bytes) {
  return (uintptr_t)a < (uintptr_t)b + bytes && (uintptr_t)b < (uintptr_t)a + bytes;
}

// Power-of-two input scale of the FP16 form.  The propagation is linear in
// its input, and scaling FP32 values by a power of two is exact, so the
// filter runs on scale * x and the outputs are multiplied by 1 / scale.
// The scale puts the input's largest |value| in [2^6, 2^7): the Chebyshev
// vectors keep 2^9 of headroom below FP16's largest finite value (65504),
// and entries down to 2^-18 of the largest stay in FP16's normal range.
// The FP32 and BF16 forms (BF16 has FP32's exponent range) use 1.
template <typename XT>
int input_scale(lne_ctx* ctx, const float* x, int64_t total, Bufs& B, int* launches, float* scale) {
  *scale = 1.0f;
  if constexpr (!std::is_same<XT, __half>::value) {
    return LNE_OK;
  } else {
    float* part = nullptr;
    int rc;
    if ((rc = B.get(&part, kAmaxBlocks, "amax partials"))) return rc;
    k_amax_partial<<<kAmaxBlocks, 256, 0, ctx->stream>>>(x, total, part);
    *launches += 1;
    std::vector<float> h(kAmaxBlocks);
    LNE_CUDA_TRY(cudaMemcpyAsync(h.data(), part, sizeof(float) * kAmaxBlocks, cudaMemcpyDeviceToHost, ctx->stream));
    LNE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    float m = 0.0f;
    for (float v : h) m = v > m ? v : m;
    if (!(m > 0.0f) || !std::isfinite(m)) return LNE_OK;
    int e = 0;
    frexpf(m, &e);  // m in [2^(e-1), 2^e)
    int k = 7 - e;
    k = k < -126 ? -126 : (k > 126 ? 126 : k);
    *scale = ldexpf(1.0f, k);
    return LNE_OK;
  }
}

struct TimedEvents {
  cudaEvent_t e[2] = {};
  TimedEvents() {
    for (auto& x : e) cudaEventCreate(&x);
  }
  ~TimedEvents() {
    for (auto& x : e) cudaEventDestroy(x);
  }
};

template <typename XT>
int propagate_impl(lne_ctx* ctx, lne_graph* g, const lne_propagate_params* p, const float* d_a, float* d_y,
                   float* d_a_out, lne_propagate_stats* stats) {
  constexpr bool k16 = sizeof(XT) == 2;
  using HT = typename ShadowOf<XT>::type;
  const int64_t n = g->n;
  const int d = (int)p->dim;
  const int64_t ld = pad_ld(d);
  cudaStream_t st = ctx->stream;
  int launches = 0;
  std::vector<float> c;
  chebyshev_coeffs(p->order, p->s, c);
  Bufs B(ctx);
  Filter<XT> F;
  SpmmWork work;
  int rc;
  TimedEvents ev;
  cudaEventRecord(ev.e[0], st);
  if ((rc = setup_filter<XT>(ctx, g, p, B, &work, &launches, F))) return rc;
  float sc = 1.0f;
  if ((rc = input_scale<XT>(ctx, d_a, n * d, B, &launches, &sc))) return rc;
  const size_t sz = (size_t)n * ld;
  // The caller's rows are read in place where they are whole 16-byte
  // vectors, else a zero-padded copy; the 16-bit forms gather a scaled copy.
  const bool direct = rows_direct(d_a, d, ld);
  float* Acopy = nullptr;
  HT *Ab = nullptr, *Afb = nullptr;
  if (!direct && (rc = B.get(&Acopy, sz, "a"))) return rc;
  if (k16 && ((rc = B.get(&Ab, sz, "a 16-bit")) || (rc = B.get(&Afb, sz, "a - conv 16-bit")))) return rc;
  const unsigned pg = (unsigned)std::min<int64_t>((n * ld + 255) / 256, (int64_t)ctx->num_sms * 32);
  if (direct && k16) {
    k_shadow_copy<HT><<<pg, 256, 0, st>>>(reinterpret_cast<const float4*>(d_a), (int64_t)sz / 8, sc,
                                          reinterpret_cast<uint4*>(Ab));
    launches += 1;
  } else if (!direct) {
    k_pad_copy<HT><<<pg, 256, 0, st>>>(d_a, n, d, sc, Acopy, ld, Ab);
    launches += 1;
  }
  const float* A = direct ? d_a : Acopy;
  const float a_scale = direct ? sc : 1.0f;
  // a - conv: to the caller's buffer where it can be written in place.  The
  // (A + I) product gathers it in the FP32 form, so it must not be y; and rows
  // are written while other rows of a are still read, so it must not be a.
  const size_t bytes = sizeof(float) * (size_t)n * d;
  const bool out_direct = d_a_out && rows_direct(d_a_out, d, ld) && !ranges_overlap(d_a_out, d_y, bytes) &&
                          !ranges_overlap(d_a_out, d_a, bytes);
  float* Af = nullptr;
  if (!out_direct && (!k16 || d_a_out) && (rc = B.get(&Af, sz, "a - conv"))) return rc;
  FinalOut<HT> fin;
  fin.base = A;
  fin.base_scale = a_scale;
  fin.out = out_direct ? d_a_out : Af;
  fin.out_scale = out_direct ? 1.0f / sc : 1.0f;
  fin.outb = Afb;
  // a - conv, then y = (A + I)(a - conv)
  if ((rc = F.run(A, Ab, a_scale, p->order, c, fin))) return rc;
  {
    const XT* Xf = F.op(fin.out, Afb);
    EpiAPlusI<XT> epi{Xf, ld, d_y, d, d, 1.0f / sc, rows_direct(d_y, d, ld)};
    if ((rc = F.spmm(Xf, epi))) return rc;
  }
  if (d_a_out && !out_direct) {
    k_unpad_copy<<<pg, 256, 0, st>>>(Af, ld, n, d, 1.0f / sc, d_a_out);
    launches += 1;
  }
  cudaEventRecord(ev.e[1], st);
  LNE_CUDA_TRY(cudaEventSynchronize(ev.e[1]));
  LNE_CUDA_TRY(cudaGetLastError());
  if (stats) {
    memset(stats, 0, sizeof(*stats));
    cudaEventElapsedTime(&stats->ms_total, ev.e[0], ev.e[1]);
    stats->kernel_launches = launches;
    stats->spmm_calls = 2 * (p->order > 2 ? p->order - 1 : 1) + 1;
  }
  ctx->launch_count += launches;
  return LNE_OK;
}

// Derivatives of the reference's weights with respect to s:
// c_0 = I0(s), c_k = 2 (-1)^k I_k(s);  I0' = I1, I_k' = (I_{k-1} + I_{k+1}) / 2.
void chebyshev_coeffs_ds(int order, double s, std::vector<double>& dc) {
  const double sf = (double)(float)s;
  dc.assign(order > 2 ? order : 2, 0.0);
  dc[0] = bessel_i(1, sf);
  for (int k = 1; k < (int)dc.size(); ++k)
    dc[k] = ((k & 1) ? -1.0 : 1.0) * (bessel_i(k - 1, sf) + bessel_i(k + 1, sf));
}

// dL/dmu and dL/ds in FP32 (P3): the forward pass on a with the mu-tangent
// T'_1 = -M a, T'_{k+1} = M(M T'_k) - 2 T'_k - T'_{k-1} - 2 M T_k, and the
// dots <h, T_k a>, <h, T'_k> (h = hscale^-1 H): dL/ds = -sum_k c_k'(s)
// <h, T_k a>, dL/dmu = -sum_k c_k <h, T'_k>.
//
// The same gradients as sums over the vectors V_k = T_k(X) D~^-1 h that
// dL/da's recursion forms anyway (<V_k, D~ a>, <M V_j, D~ a>) take none of
// these products, but are less exact: the row of a hub is an FP32 sum over its
// neighbours, weighted by its d~.  At 6,000 vertices with a hub of 5,500
// neighbours and 128 columns that form was off by 7.1e-7 (mu) and 6.0e-7 (s)
// of |h a|, root mean square of 8 draws, this one by 1.3e-7 and 2.7e-7; at
// 1.14M vertices and 128 columns that form's relative errors were up to 40
// times this one's (1.7e-7 against 4.8e-9 in dL/dmu of one draw).
int param_grads(lne_ctx* ctx, Filter<float>& F, const lne_propagate_params* p, const std::vector<float>& c,
                const float* H, const float* d_a, double hscale, double* h_dmu, double* h_ds) {
  const int64_t n = F.n, ld = F.ld;
  const int d = (int)p->dim;
  const int order = p->order;
  const size_t sz = (size_t)n * ld;
  const int64_t total = (int64_t)sz;
  cudaStream_t st = ctx->stream;
  Bufs& B = *F.B;
  int& launches = *F.launches;
  int rc;
  const int K = order > 2 ? order : 2;
  double* partial = nullptr;
  if ((rc = B.get(&partial, (size_t)2 * K * kDotBlocks, "dot partials"))) return rc;
  LNE_CUDA_TRY(cudaMemsetAsync(partial, 0, sizeof(double) * 2 * K * kDotBlocks, st));
  auto dot = [&](int slot, const float* x) {
    k_dot_partial<<<kDotBlocks, 256, 0, st>>>(H, x, total, partial + (int64_t)slot * kDotBlocks);
    launches += 1;
  };
  float *Tm = nullptr, *Tpm = nullptr;  // M T_k, M T'_k
  float* T[3];
  float* Tp[3];
  if ((rc = B.get(&Tm, sz, "M T")) || (rc = B.get(&Tpm, sz, "M T'"))) return rc;
  for (int i = 0; i < 3; ++i)
    if ((rc = B.get(&T[i], sz, "T")) || (rc = B.get(&Tp[i], sz, "T'"))) return rc;
  const unsigned pg = (unsigned)std::min<int64_t>((total + 255) / 256, (int64_t)ctx->num_sms * 32);
  const float* A = d_a;
  if (!rows_direct(d_a, d, ld)) {
    float* Acopy = nullptr;
    if ((rc = B.get(&Acopy, sz, "a"))) return rc;
    k_pad_copy<__nv_bfloat16><<<pg, 256, 0, st>>>(d_a, n, d, 1.0f, Acopy, ld, nullptr);
    launches += 1;
    A = Acopy;
  }
  dot(0, A);  // <h, T_0>
  // tmp = M a;  T_1 = 0.5 M tmp - a;  T'_1 = -tmp
  const FinalOut<__nv_bfloat16> none;
  if ((rc = F.apply_m(A, Tm, nullptr))) return rc;
  if ((rc = F.spmm(Tm, EpiFirst<float>{F.coef, Tm, A, T[0], nullptr, nullptr, none, ld, 0.0f, 0.0f, 1.0f}))) return rc;
  k_scale_copy<<<pg, 256, 0, st>>>(Tm, total, -1.0f, Tp[0]);
  launches += 1;
  dot(1, T[0]);
  dot(K + 1, Tp[0]);
  const float* t0 = A;         // T_{k-1}
  const float* tp0 = nullptr;  // T'_{k-1} (T'_0 = 0)
  int j1 = 0;
  for (int k = 1; k + 1 < order; ++k) {
    const int j2 = (j1 + 1) % 3;
    // tmp = M T_k; T_{k+1} = M tmp - 2 T_k - T_{k-1}
    if ((rc = F.apply_m(T[j1], Tm, nullptr))) return rc;
    if ((rc = F.spmm(Tm, EpiStep<float>{F.coef, Tm, t0, T[j1], T[j2], nullptr, nullptr, none, ld, 0.0f}))) return rc;
    // tmp' = M T'_k; T'_{k+1} = M tmp' - 2 T'_k - T'_{k-1} - 2 M T_k
    if ((rc = F.apply_m(Tp[j1], Tpm, nullptr))) return rc;
    if ((rc = F.spmm(Tpm, EpiStep<float, true>{F.coef, Tpm, tp0, Tp[j1], Tp[j2], nullptr, nullptr, none, ld, 0.0f, 0.0f,
                                               false, 1.0f, Tm})))
      return rc;
    dot(k + 1, T[j2]);
    dot(K + k + 1, Tp[j2]);
    t0 = T[j1];
    tp0 = Tp[j1];
    j1 = j2;
  }
  std::vector<double> hp((size_t)2 * K * kDotBlocks);
  LNE_CUDA_TRY(cudaMemcpyAsync(hp.data(), partial, sizeof(double) * hp.size(), cudaMemcpyDeviceToHost, st));
  LNE_CUDA_TRY(cudaStreamSynchronize(st));
  std::vector<double> dots(2 * K, 0.0);
  for (int sidx = 0; sidx < 2 * K; ++sidx) {
    for (int b = 0; b < kDotBlocks; ++b) dots[sidx] += hp[(size_t)sidx * kDotBlocks + b];
    dots[sidx] *= hscale;
  }
  std::vector<double> dc;
  chebyshev_coeffs_ds(order, p->s, dc);
  // only the terms the forward filter uses: k < max(order, 2)
  double gs = 0.0, gmu = 0.0;
  for (int k = 0; k < K; ++k) gs -= dc[k] * dots[k];
  for (int k = 1; k < K; ++k) gmu -= (double)c[k] * dots[K + k];
  if (h_ds) *h_ds = gs;
  if (h_dmu) *h_dmu = gmu;
  return LNE_OK;
}

template <typename XT>
int adjoint_impl(lne_ctx* ctx, lne_graph* g, const lne_propagate_params* p, const float* d_a, const float* d_gy,
                 float* d_ga, double* h_dmu, double* h_ds, lne_propagate_stats* stats) {
  constexpr bool k16 = sizeof(XT) == 2;
  using HT = typename ShadowOf<XT>::type;
  const int64_t n = g->n;
  const int d = (int)p->dim;
  const int64_t ld = pad_ld(d);
  const int order = p->order;
  cudaStream_t st = ctx->stream;
  int launches = 0;
  std::vector<float> c;
  chebyshev_coeffs(order, p->s, c);
  Bufs B(ctx);
  Filter<XT> F;
  SpmmWork work;
  int rc;
  TimedEvents ev;
  cudaEventRecord(ev.e[0], st);
  if ((rc = setup_filter<XT>(ctx, g, p, B, &work, &launches, F))) return rc;
  const size_t sz = (size_t)n * ld;
  const bool params = h_dmu || h_ds;
  // the FP16 form runs on a scaled output gradient sg * g (dL/da is linear
  // in g; the FP32 parameter-gradient pass unscales its dots by 1 / sg)
  float sg = 1.0f;
  if ((rc = input_scale<XT>(ctx, d_gy, n * d, B, &launches, &sg))) return rc;
  // g is read in place where its rows are whole 16-byte vectors; the FP32
  // pass of the FP16 form takes a scaled copy (sums of g itself may overflow)
  const bool g_direct = rows_direct(d_gy, d, ld) && !(params && sg != 1.0f);
  float *Gcopy = nullptr, *H = nullptr, *Bf = nullptr;
  HT *Gb = nullptr, *Bb = nullptr;
  if ((!g_direct && (!k16 || params) && (rc = B.get(&Gcopy, sz, "g"))) || (rc = B.get(&H, sz, "h")) ||
      (rc = B.get(&Bf, sz, "b")))
    return rc;
  if (k16 && ((rc = B.get(&Gb, sz, "g 16-bit")) || (rc = B.get(&Bb, sz, "b 16-bit")))) return rc;
  const unsigned pg = (unsigned)std::min<int64_t>(((int64_t)sz + 255) / 256, (int64_t)ctx->num_sms * 32);
  if (g_direct && k16) {
    k_shadow_copy<HT><<<pg, 256, 0, st>>>(reinterpret_cast<const float4*>(d_gy), (int64_t)sz / 8, sg,
                                          reinterpret_cast<uint4*>(Gb));
    launches += 1;
  } else if (!g_direct) {
    k_pad_copy<HT><<<pg, 256, 0, st>>>(d_gy, n, d, sg, Gcopy, ld, Gb);
    launches += 1;
  }
  const float* G = g_direct ? d_gy : Gcopy;  // (Gcopy holds sg * g)
  // h = (A + I) g, b = D~^-1 h
  {
    const XT* Gx = F.op(G, Gb);
    EpiAdjInit<XT> epi{F.coef, Gx, ld, H, Bf, Bb};
    if ((rc = F.spmm(Gx, epi))) return rc;
  }
  if (params) {
    // The parameter gradients run in FP32 in every form: they are sums over
    // the orders whose terms cancel, so 16-bit gathers would cost them far
    // more relative accuracy than they cost dL/da.  The 16-bit forms first
    // form an FP32 h = (A + I) g from the FP32 (scaled) g.  They read a, so
    // they come before dL/da is written.
    Filter<float> F32{ctx, g, n, ld, F.coef, &launches, &B, &work};
    const float* H32 = H;
    if (k16) {
      float* H2 = nullptr;
      if ((rc = B.get(&H2, sz, "h fp32"))) return rc;
      if ((rc = F32.spmm(G, EpiAdjInit<float>{F.coef, G, ld, H2, nullptr, nullptr}))) return rc;
      H32 = H2;
    }
    if ((rc = param_grads(ctx, F32, p, c, H32, d_a, 1.0 / (double)sg, h_dmu, h_ds))) return rc;
  }
  // grad a = h - D~ sum_k c_k T_k(X) b      (M^T = D~ M D~^-1)
  const bool out_direct = d_ga && rows_direct(d_ga, d, ld);
  float* GA = nullptr;
  if (!out_direct && (rc = B.get(&GA, sz, "grad a"))) return rc;
  FinalOut<HT> fin;
  fin.base = H;
  fin.scale_dt = true;
  fin.out = out_direct ? d_ga : GA;
  fin.out_scale = out_direct ? 1.0f / sg : 1.0f;
  if ((rc = F.run(Bf, Bb, 1.0f, order, c, fin))) return rc;
  if (d_ga && !out_direct) {
    k_unpad_copy<<<pg, 256, 0, st>>>(GA, ld, n, d, 1.0f / sg, d_ga);
    launches += 1;
  }
  cudaEventRecord(ev.e[1], st);
  LNE_CUDA_TRY(cudaEventSynchronize(ev.e[1]));
  LNE_CUDA_TRY(cudaGetLastError());
  if (stats) {
    memset(stats, 0, sizeof(*stats));
    cudaEventElapsedTime(&stats->ms_total, ev.e[0], ev.e[1]);
    stats->kernel_launches = launches;
  }
  ctx->launch_count += launches;
  return LNE_OK;
}

}  // namespace

}  // namespace lne

using namespace lne;

extern "C" int lne_propagate(lne_ctx* ctx, const lne_graph* g, const lne_propagate_params* p, const float* d_a,
                             float* d_y, float* d_a_out, lne_propagate_stats* stats) {
  LNE_CHECK_ARG(ctx && g && p && d_a && d_y, "lne_propagate: NULL argument");
  LNE_CHECK_ARG(p->dim >= 1 && p->order >= 0, "lne_propagate: bad dim/order");
  LNE_CHECK_ARG(p->precision == LNE_PREC_FP32 || p->precision == LNE_PREC_BF16 || p->precision == LNE_PREC_FP16,
                "lne_propagate: bad precision");
  LNE_CUDA_TRY(cudaSetDevice(ctx->device));
  lne_graph* gm = const_cast<lne_graph*>(g);
  if (!gm->plan_ready) ctx->launch_count += plan_launches(gm->n);
  int rc = build_plan_graph(ctx, gm);
  if (rc) return rc;
  if (p->precision == LNE_PREC_BF16) return propagate_impl<__nv_bfloat16>(ctx, gm, p, d_a, d_y, d_a_out, stats);
  if (p->precision == LNE_PREC_FP16) return propagate_impl<__half>(ctx, gm, p, d_a, d_y, d_a_out, stats);
  return propagate_impl<float>(ctx, gm, p, d_a, d_y, d_a_out, stats);
}

extern "C" int lne_propagate_adjoint(lne_ctx* ctx, const lne_graph* g, const lne_propagate_params* p,
                                     const float* d_a, const float* d_gy, float* d_ga, double* h_dmu, double* h_ds,
                                     lne_propagate_stats* stats) {
  LNE_CHECK_ARG(ctx && g && p && d_gy, "lne_propagate_adjoint: NULL argument");
  LNE_CHECK_ARG(d_a || (!h_dmu && !h_ds), "lne_propagate_adjoint: the parameter gradients need a");
  LNE_CHECK_ARG(p->dim >= 1 && p->order >= 0, "lne_propagate_adjoint: bad dim/order");
  LNE_CHECK_ARG(p->precision == LNE_PREC_FP32 || p->precision == LNE_PREC_BF16 || p->precision == LNE_PREC_FP16,
                "lne_propagate_adjoint: bad precision");
  LNE_CUDA_TRY(cudaSetDevice(ctx->device));
  lne_graph* gm = const_cast<lne_graph*>(g);
  if (!gm->plan_ready) ctx->launch_count += plan_launches(gm->n);
  int rc = build_plan_graph(ctx, gm);
  if (rc) return rc;
  if (p->precision == LNE_PREC_BF16)
    return adjoint_impl<__nv_bfloat16>(ctx, gm, p, d_a, d_gy, d_ga, h_dmu, h_ds, stats);
  if (p->precision == LNE_PREC_FP16) return adjoint_impl<__half>(ctx, gm, p, d_a, d_gy, d_ga, h_dmu, h_ds, stats);
  return adjoint_impl<float>(ctx, gm, p, d_a, d_gy, d_ga, h_dmu, h_ds, stats);
}

extern "C" int lne_chebyshev_coefficients(int32_t order, double s, float* out) {
  LNE_CHECK_ARG(out && order >= 0, "lne_chebyshev_coefficients: bad argument");
  std::vector<float> c;
  chebyshev_coeffs(order, s, c);
  for (size_t i = 0; i < c.size(); ++i) out[i] = c[i];
  return LNE_OK;
}
