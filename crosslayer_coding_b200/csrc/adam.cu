// Backward + optimizer in one pass over the parameters (sm_100a).
//
// The reference materialises dense gradients for every decoder and encoder matrix with autograd GEMMs and
// then runs torch.optim.Adam/AdamW over them (clt/training/trainer.py:751-783).  With a (Batch)TopK or
// JumpReLU code the gradients are row-sparse sums over the active (token, feature) entries, so this file
// never writes a gradient tensor: one warp per parameter row gathers the few rows of the gradient seed
// (decoder) or of the layer input (encoder) that touch its feature, forms the row gradient in registers,
// and applies the Adam update to (w, m, v) in the same pass.  The decoder pass also produces
//   * dL/da for every entry (dot of the seed row with the *old* weight row), consumed by the encoder pass,
//   * the squared decoder norm of every feature after the update (used by the sparsity penalty next step).
//
// Row layout: decoder tensor s is [F, R_s, d] (feature-major), encoder is [L, F, d]; bf16 weights with
// fp32 moments (or fp32 weights).  d must be a multiple of 8.
#include <climits>

#include "common.cuh"

#include <type_traits>

namespace clt {

constexpr int kMaxLayersA = 32;

struct AdamHyper {
  float lr, beta1, beta2, eps, weight_decay;
  float bc1, bc2;        // 1 - beta^step
  int decoupled;         // 1: AdamW, 0: Adam (decay folded into the gradient)
  float grad_scale;      // multiplies the gathered gradient (e.g. 2/(B*d), 1/loss_scale, clip factor)
  unsigned int sr_seed;  // stochastic rounding seed; 0 = round to nearest
  unsigned int moment_seed;  // seed for the stochastic rounding of bf16 moments (changes every step)
};

__device__ __forceinline__ uint32_t hash32(uint32_t x) {
  x ^= x >> 16; x *= 0x7feb352dU; x ^= x >> 15; x *= 0x846ca68bU; x ^= x >> 16;
  return x;
}
// fp32 -> 16-bit weight; a non-zero seed asks for stochastic rounding (bf16 builds; fp16 rounds to nearest)
__device__ __forceinline__ t16 to_bf16(float v, unsigned int seed, unsigned long long idx) {
#if CLT_T16_IS_HALF
  return float_to_t16(v);
#else
  if (seed == 0) return float_to_t16(v);
  const uint32_t u = __float_as_uint(v);
  if ((u & 0x7F800000u) == 0x7F800000u) return float_to_t16(v);
  const uint32_t r = hash32(uint32_t(idx) ^ hash32(seed + uint32_t(idx >> 32))) & 0xFFFFu;
  const uint32_t t = (u + r) & 0xFFFF0000u;
  return float_to_t16(__uint_as_float(t));
#endif
}

// Hyper-parameters pre-combined once per thread so the per-element update is 11 instructions.
struct HyperRegs {
  float decay;   // 1 - lr * wd (AdamW) or 1
  float wd_l2;   // wd folded into the gradient (Adam) or 0
  float omb1, omb2;
  float step;    // lr / (1 - beta1^t)
  float isb2;    // 1 / sqrt(1 - beta2^t)
  float eps;
  float gscale;
};
__device__ __forceinline__ HyperRegs make_regs(const AdamHyper& h) {
  HyperRegs r;
  r.decay = h.decoupled ? 1.f - h.lr * h.weight_decay : 1.f;
  r.wd_l2 = h.decoupled ? 0.f : h.weight_decay;
  r.omb1 = 1.f - h.beta1;
  r.omb2 = 1.f - h.beta2;
  r.step = h.lr / h.bc1;
  r.isb2 = rsqrtf(h.bc2);
  r.eps = h.eps;
  r.gscale = h.grad_scale;
  return r;
}
// m <- m + (1-b1)(g - m);  v <- v + (1-b2)(g^2 - v);  w <- decay*w - step * m / (sqrt(v)/sqrt(bc2) + eps)
__device__ __forceinline__ void adam1(float& w, float& m, float& v, float g, const HyperRegs& r) {
  g = fmaf(r.wd_l2, w, g);
  w *= r.decay;
  m = fmaf(r.omb1, g - m, m);
  v = fmaf(r.omb2, fmaf(g, g, -v), v);
  const float denom = fmaf(sqrtf(v), r.isb2, r.eps);
  w = fmaf(-r.step, __fdividef(m, denom), w);
}
// The same for two elements (every operation rounds as in adam1).
__device__ __forceinline__ void adam2(float2& w, float2& m, float2& v, float2 g, const HyperRegs& r) {
  g = f2_fma(f2_all(r.wd_l2), w, g);
  w = f2_mul(w, f2_all(r.decay));
  m = f2_fma(f2_all(r.omb1), f2_sub(g, m), m);
  v = f2_fma(f2_all(r.omb2), f2_fma(g, g, make_float2(-v.x, -v.y)), v);
  const float2 denom = f2_fma(make_float2(sqrtf(v.x), sqrtf(v.y)), f2_all(r.isb2), f2_all(r.eps));
  w = f2_fma(f2_all(-r.step), make_float2(__fdividef(m.x, denom.x), __fdividef(m.y, denom.y)), w);
}
__device__ __forceinline__ void adam_update8(float (&w)[8], float (&m)[8], float (&v)[8], const float (&g)[8], const AdamHyper& h) {
  const HyperRegs r = make_regs(h);
#pragma unroll
  for (int i = 0; i < 8; ++i) adam1(w[i], m[i], v[i], g[i], r);
}
// 8 fp32 -> 8 bf16 (one 16-byte vector); SR selects stochastic rounding with a counter-based hash.
template <bool SR>
__device__ __forceinline__ uint4 pack8_bf16(const float (&o)[8], unsigned int seed, unsigned int idx) {
  uint4 q;
  if (!SR || CLT_T16_IS_HALF) {
    q.x = pack_t16x2(o[0], o[1]); q.y = pack_t16x2(o[2], o[3]);
    q.z = pack_t16x2(o[4], o[5]); q.w = pack_t16x2(o[6], o[7]);
  } else {
    uint32_t h[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const uint32_t u = __float_as_uint(o[k]);
      const uint32_t rnd = hash32((idx + k) ^ seed) & 0xFFFFu;
      h[k] = ((u & 0x7F800000u) == 0x7F800000u) ? (u >> 16) : ((u + rnd) >> 16);
    }
    q.x = h[0] | (h[1] << 16); q.y = h[2] | (h[3] << 16); q.z = h[4] | (h[5] << 16); q.w = h[6] | (h[7] << 16);
  }
  return q;
}

__device__ __forceinline__ void unpack8(const uint4& q, float (&o)[8]) {
  const uint32_t u[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) { o[2 * j] = t16_lo(u[j]); o[2 * j + 1] = t16_hi(u[j]); }
}
__device__ __forceinline__ void load8f(const float* p, float (&o)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
}
__device__ __forceinline__ void store8f(float* p, const float (&o)[8]) {
  *reinterpret_cast<float4*>(p) = make_float4(o[0], o[1], o[2], o[3]);
  *reinterpret_cast<float4*>(p + 4) = make_float4(o[4], o[5], o[6], o[7]);
}

template <typename WT>
__device__ __forceinline__ void load_w8(const WT* p, float (&o)[8]);
template <>
__device__ __forceinline__ void load_w8<t16>(const t16* p, float (&o)[8]) {
  unpack8(*reinterpret_cast<const uint4*>(p), o);
}
template <>
__device__ __forceinline__ void load_w8<float>(const float* p, float (&o)[8]) { load8f(p, o); }

template <typename WT>
__device__ __forceinline__ void store_w8(WT* p, const float (&o)[8], unsigned int seed, unsigned long long idx);
template <>
__device__ __forceinline__ void store_w8<t16>(t16* p, const float (&o)[8], unsigned int seed, unsigned long long idx) {
  t16 b[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) b[i] = to_bf16(o[i], seed, idx + i);
  *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(b);
}
template <>
__device__ __forceinline__ void store_w8<float>(float* p, const float (&o)[8], unsigned int, unsigned long long) { store8f(p, o); }

// ------------------------------------------------------------------ decoder rows
struct DecAdamParams {
  void* w[kMaxLayersA];        // tensor i: [F_pitch, rows_i, d]
  float* m[kMaxLayersA];
  float* v[kMaxLayersA];
  long long row_start[kMaxLayersA + 1];  // prefix of F_pitch * rows_i over tensors
  int rows[kMaxLayersA];
  int ntensors;
  int L, B, d, F_pitch, tying;
  const int* feat_off;         // [L * F_pitch + 1] feature-major CSR
  const int* fcsr_tok;
  const float* fcsr_val;
  const t16* gs;     // [L, B, d] gradient seed
  float* grad_a;               // [nnz] dL/da per CSR slot (atomicAdd; zeroed by the caller); may be null
  const float* pen_coef;       // optional [L * F_pitch]: coefficient of w in the row gradient (sparsity penalty via norms)
  float* norm2_out;            // optional [L * F_pitch]: sum of squares of the updated rows (atomicAdd; zeroed by caller)
  const float* feat_offset;    // tied decoders: optional [L, F_pitch] affine applied to the activation
  const float* feat_scale;
  float* d_feat_offset;        // optional [L, F_pitch] gradient accumulators of the affine terms (zeroed by the caller); filled in
  float* d_feat_scale;         // the pass that also writes grad_a
  int moments_bf16;            // bulk pipeline only: m / v hold bf16 (stochastically rounded) instead of fp32
  const float* dgrad_row0;     // optional [ntensors, F_pitch, d] fp32: extra gradient of every feature's first row
  // optional compact extras (auxiliary loss on dead features): extra_idx[col] = row of extra_rows, or -1
  const int* extra_idx;
  const float* extra_rows;     // [n_extra, d] fp32, added to the feature's first row
  const float* ctl;            // optional step control block (skip flag, 1 / loss scale, clip coefficient)
  int use_inv_scale;           // the "gradient seed" operand carries the loss scale (decoder: yes; encoder inputs: no)
  float* norm_sq_out;          // norm-only pass: squared norm of all row gradients is added here
  int* status;                 // for the index checks of the debug build; may be null
  AdamHyper h;
};

// The debug build reports a token (from the feature-major lists) outside the batch; row 0 with activation 0 is taken in its place.
__device__ __forceinline__ void check_token(int& tok, float& a, int B, int* status, int site) {
  if (!clt_in_bounds(tok, B, status, site)) { tok = 0; a = 0.f; }
}

// Extra gradient of a feature's first row (dense buffer or compact rows through an index), or null.
__device__ __forceinline__ const float* extra_row_ptr(const DecAdamParams& p, int col) {
  if (p.dgrad_row0 != nullptr) return p.dgrad_row0 + 1LL * col * p.d;
  if (p.extra_idx != nullptr) {
    const int i = __ldg(p.extra_idx + col);
    if (i >= 0) return p.extra_rows + 1LL * i * p.d;
  }
  return nullptr;
}
// Block-wide sum of `v` added to *out (one atomic per CTA); every thread of the CTA calls it.
__device__ __forceinline__ void block_add(float v, float* out) {
  __shared__ float red_s[32];
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red_s[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
    for (int w = 0; w < int((blockDim.x + 31) >> 5); ++w) tot += red_s[w];
    if (tot != 0.f && out != nullptr) atomicAdd(out, tot);
  }
}

__device__ __forceinline__ void f4x2_to8(const float4& a, const float4& b, float (&o)[8]) {
  o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
}
__device__ __forceinline__ void stream_store8f(float* p, const float (&o)[8]) {
  __stcs(reinterpret_cast<float4*>(p), make_float4(o[0], o[1], o[2], o[3]));
  __stcs(reinterpret_cast<float4*>(p) + 1, make_float4(o[4], o[5], o[6], o[7]));
}
template <typename WT>
struct WVec;
template <>
struct WVec<t16> {
  uint4 q;
  __device__ __forceinline__ void load(const t16* p) { q = __ldcs(reinterpret_cast<const uint4*>(p)); }
  __device__ __forceinline__ void get(float (&o)[8]) const { unpack8(q, o); }
};
template <>
struct WVec<float> {
  float4 a, b;
  __device__ __forceinline__ void load(const float* p) {
    a = __ldcs(reinterpret_cast<const float4*>(p));
    b = __ldcs(reinterpret_cast<const float4*>(p) + 1);
  }
  __device__ __forceinline__ void get(float (&o)[8]) const { f4x2_to8(a, b, o); }
};

template <typename WT>
struct RowRegs {
  WVec<WT> w;
  float4 m0, m1, v0, v1;
  __device__ __forceinline__ void load(const WT* wp, const float* mp, const float* vp) {
    w.load(wp);
    m0 = __ldcs(reinterpret_cast<const float4*>(mp)); m1 = __ldcs(reinterpret_cast<const float4*>(mp) + 1);
    v0 = __ldcs(reinterpret_cast<const float4*>(vp)); v1 = __ldcs(reinterpret_cast<const float4*>(vp) + 1);
  }
};

// Untied decoders, the flagship path.  Work item = (source feature, 256-element segment): one warp, 8
// elements per lane, walking the feature's R = L - s target rows with the next row's (w, m, v) already in
// flight.  The first four entries of the feature stay in registers: their activation, token and the
// partial dot products for dL/da, which are reduced once per item instead of once per row.
template <typename WT, bool SR>
__global__ void __launch_bounds__(256, 2) decoder_rows_adam_untied_kernel(const DecAdamParams p) {
  const int lane = threadIdx.x & 31;
  const int warp_global = int((blockIdx.x * 1LL * blockDim.x + threadIdx.x) >> 5);
  const int nwarps = int((gridDim.x * 1LL * blockDim.x) >> 5);
  const HyperRegs hr = make_regs(p.h);
  const StepScales sc = read_step_ctl(p.ctl);
  if (sc.skip) return;
  const float gsc = hr.gscale * (p.use_inv_scale ? sc.inv_scale : 1.f);
  const int d = p.d, B = p.B, Fp = p.F_pitch;
  const int nseg = (d + 255) / 256;
  const int per_tensor = Fp * nseg;
  const int total_items = per_tensor * p.ntensors;
  const t16* __restrict__ gs = p.gs;
  for (int item = warp_global; item < total_items; item += nwarps) {
    const int ti = item / per_tensor;
    const int rem = item - ti * per_tensor;
    const int f = rem / nseg;
    const int seg = rem - f * nseg;
    const int R = p.rows[ti];
    const int e0 = seg * 256 + lane * 8;
    const bool act = e0 < d;
    const long long row0 = 1LL * f * R;
    WT* wbase = static_cast<WT*>(p.w[ti]) + row0 * d + e0;
    float* mbase = p.m[ti] + row0 * d + e0;
    float* vbase = p.v[ti] + row0 * d + e0;
    const int col = ti * Fp + f;
    const int b = __ldg(p.feat_off + col), e = __ldg(p.feat_off + col + 1);
    const int ne = e - b;
    const float* xrow = extra_row_ptr(p, col);
    RowRegs<WT> cur, nxt;
    if (act) cur.load(wbase, mbase, vbase);
    int tok4[4];
    float a4[4], dacc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      tok4[j] = j < ne ? __ldg(p.fcsr_tok + b + j) : 0;
      a4[j] = j < ne ? __ldg(p.fcsr_val + b + j) : 0.f;
      dacc[j] = 0.f;
      check_token(tok4[j], a4[j], B, p.status, 203);
    }
    const float pc = p.pen_coef ? p.pen_coef[col] : 0.f;
    float norm2 = 0.f;
    const unsigned int idx_base = (unsigned int)((p.row_start[ti] + row0) * d + e0);
    for (int r = 0; r < R; ++r) {
      const long long roff = 1LL * r * d;
      if (act && r + 1 < R) nxt.load(wbase + roff + d, mbase + roff + d, vbase + roff + d);
      float w[8], g[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) { g[i] = 0.f; w[i] = 0.f; }
      if (act) {
        cur.w.get(w);
        const t16* gs_t = gs + 1LL * (ti + r) * B * d + e0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (j < ne) {
            float gv[8];
            unpack8(__ldg(reinterpret_cast<const uint4*>(gs_t + 1LL * tok4[j] * d)), gv);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              g[k] = fmaf(a4[j], gv[k], g[k]);
              dacc[j] = fmaf(gv[k], w[k], dacc[j]);
            }
          }
        }
      }
      for (int i = b + 4; i < e; ++i) {  // rare: features with more than four entries
        float dot = 0.f;
        if (act) {
          int tok = __ldg(p.fcsr_tok + i);
          float a = __ldg(p.fcsr_val + i), gv[8];
          check_token(tok, a, B, p.status, 204);
          unpack8(__ldg(reinterpret_cast<const uint4*>(gs + (1LL * (ti + r) * B + tok) * d + e0)), gv);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            g[k] = fmaf(a, gv[k], g[k]);
            dot = fmaf(gv[k], w[k], dot);
          }
        }
        if (p.grad_a != nullptr) {
          dot = warp_sum(dot);
          if (lane == 0 && dot != 0.f) atomicAdd(&p.grad_a[i], dot * gsc);
        }
      }
      if (act) {
        float dg0[8];
        const bool extra = r == 0 && xrow != nullptr;
        if (extra) load8f(xrow + e0, dg0);
        float m[8], v[8];
        f4x2_to8(cur.m0, cur.m1, m);
        f4x2_to8(cur.v0, cur.v1, v);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          float gk = fmaf(pc, w[k], g[k] * gsc);
          if (extra) gk += dg0[k];
          adam1(w[k], m[k], v[k], gk * sc.clip, hr);
          norm2 = fmaf(w[k], w[k], norm2);
        }
        stream_store8f(mbase + roff, m);
        stream_store8f(vbase + roff, v);
        if (sizeof(WT) == 2) __stcs(reinterpret_cast<uint4*>(wbase + roff), pack8_bf16<SR>(w, p.h.sr_seed, idx_base + (unsigned int)roff));
        else stream_store8f(reinterpret_cast<float*>(wbase + roff), w);
      }
      cur = nxt;
    }
    if (p.grad_a != nullptr) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j < ne) {
          const float sdot = warp_sum(dacc[j]);
          if (lane == 0 && sdot != 0.f) atomicAdd(&p.grad_a[b + j], sdot * gsc);
        }
      }
    }
    if (p.norm2_out != nullptr) {
      norm2 = warp_sum(norm2);
      if (lane == 0) atomicAdd(&p.norm2_out[col], norm2);
    }
  }
}

// ---------------------------------------------------------------- gradient norms (clipping)
// The pre-pass of gradient clipping: squared norms of all row gradients into p.norm_sq_out and, with DOTS (decoders), dL/da into p.grad_a.  Nothing
// is updated, so features without entries (and without an extra row) are skipped and neither moments nor, without DOTS, weights are read.
// A gather of every entry's seed row for every target, which L2 could deliver three times as fast as the one-segment form read it: instructions bound
// that one (a warp per 256 elements of a feature's rows: divisions, list and reductions for each).  Here a warp takes up to 1024 elements of the rows
// (NV vectors of eight per lane), kEntries entries at a time, with the list of the next feature and the offsets of the one after it on the way.
// us before and now, decoder + encoder: 12 x 768, 24576 features, 4096 tokens, k = 200 3243 + 321 / 1638 + 196; 3072 features, k = 25 498 + 48 / 262 + 33;
// 5 x 520, 2056 features, 776 tokens 62 + 15 / 41 + 11; 12 x 352 tied 114 + 50 / 68 + 37; 6 x 136 145 + 37 / 118 + 35; 4 x 2048 102 + 36 / 76 + 26.
template <typename WT, bool DOTS, int NV>
__global__ void __launch_bounds__(256, 2) rows_norm_kernel(const DecAdamParams p) {
  constexpr int kEntries = NV <= 2 ? 4 : 2;
  const int lane = threadIdx.x & 31;
  const int warp_global = int((blockIdx.x * 1LL * blockDim.x + threadIdx.x) >> 5);
  const int nwarps = int((gridDim.x * 1LL * blockDim.x) >> 5);
  const StepScales sc = read_step_ctl(p.ctl);
  if (sc.skip) return;
  const float gsc = p.h.grad_scale * (p.use_inv_scale ? sc.inv_scale : 1.f);
  float nsq = 0.f;
  const int d = p.d, Fp = p.F_pitch;
  const int nseg = (d + 256 * NV - 1) / (256 * NV), seg_width = (d / 8 + nseg - 1) / nseg * 8;  // even segments
  const int total_cols = Fp * p.ntensors;
  const long long total_items = 1LL * total_cols * nseg;
  struct List {
    int b, e;
    int tok[4];
    float a[4];
  };
  const auto load_range = [&](long long item, List& m) {
    m.b = m.e = 0;
    if (item >= total_items) return;
    const int col = nseg == 1 ? int(item) : int(item / nseg);
    m.b = __ldg(p.feat_off + col);
    m.e = __ldg(p.feat_off + col + 1);
  };
  const auto load_entries = [&](List& m) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool in = m.b + j < m.e;
      m.tok[j] = in ? __ldg(p.fcsr_tok + m.b + j) : 0;
      m.a[j] = in ? __ldg(p.fcsr_val + m.b + j) : 0.f;
      check_token(m.tok[j], m.a[j], p.B, p.status, 205);
    }
  };
  List cur, nxt;
  load_range(warp_global, cur);
  load_entries(cur);
  load_range(1LL * warp_global + nwarps, nxt);
  for (long long item = warp_global; item < total_items; item += nwarps) {
    List after;
    load_range(item + 2LL * nwarps, after);
    load_entries(nxt);
    const int col = nseg == 1 ? int(item) : int(item / nseg);
    const int seg0 = nseg == 1 ? 0 : int(item - 1LL * col * nseg) * seg_width, end = min(d, seg0 + seg_width);
    const int b = cur.b, ne = cur.e - b;
    const float* xrow = extra_row_ptr(p, col);
    if (ne > 0 || xrow != nullptr) {
      const int ti = col / Fp, f = col - ti * Fp;
      const int R = p.rows[ti];
      const int e0 = seg0 + lane * 8;
      const WT* wrow = static_cast<const WT*>(p.w[ti]) + 1LL * f * R * d + e0;
      const t16* gs_t = p.gs + 1LL * ti * p.B * d + e0;
      const float pc = DOTS && p.pen_coef ? p.pen_coef[col] : 0.f;
      float dacc[4] = {0.f, 0.f, 0.f, 0.f};
      float dx = 0.f;  // dL/da of entry 4 + lane
#pragma unroll 1
      for (int r = 0; r < R; ++r, wrow += d, gs_t += 1LL * p.B * d) {
        WVec<WT> wv[NV];
        float g[NV][8];
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          if (DOTS && e0 + 256 * n < end) wv[n].load(wrow + 256 * n);
#pragma unroll
          for (int k = 0; k < 8; ++k) g[n][k] = 0.f;
        }
#pragma unroll
        for (int j0 = 0; j0 < 4; j0 += kEntries) {  // the first four entries, whose list is in registers
          if (j0 >= ne) break;
          uint4 v[kEntries][NV];
#pragma unroll
          for (int j = 0; j < kEntries; ++j)
            if (j0 + j < ne) {
#pragma unroll
              for (int n = 0; n < NV; ++n)
                if (e0 + 256 * n < end) v[j][n] = __ldg(reinterpret_cast<const uint4*>(gs_t + 1LL * cur.tok[j0 + j] * d + 256 * n));
            }
#pragma unroll
          for (int j = 0; j < kEntries; ++j)
            if (j0 + j < ne) {
#pragma unroll
              for (int n = 0; n < NV; ++n)
                if (e0 + 256 * n < end) {
                  float gv[8], w[8];
                  unpack8(v[j][n], gv);
                  if (DOTS) wv[n].get(w);
#pragma unroll
                  for (int k = 0; k < 8; ++k) {
                    g[n][k] = fmaf(cur.a[j0 + j], gv[k], g[n][k]);
                    if (DOTS) dacc[j0 + j] = fmaf(gv[k], w[k], dacc[j0 + j]);
                  }
                }
            }
        }
#pragma unroll 1
        for (int i = 4; i < ne; ++i) {
          float a = __ldg(p.fcsr_val + b + i);
          int tok = __ldg(p.fcsr_tok + b + i);
          check_token(tok, a, p.B, p.status, 206);
          const t16* src = gs_t + 1LL * tok * d;
          uint4 v[NV];
          float dot = 0.f;
#pragma unroll
          for (int n = 0; n < NV; ++n)
            if (e0 + 256 * n < end) v[n] = __ldg(reinterpret_cast<const uint4*>(src + 256 * n));
#pragma unroll
          for (int n = 0; n < NV; ++n)
            if (e0 + 256 * n < end) {
              float gv[8], w[8];
              unpack8(v[n], gv);
              if (DOTS) wv[n].get(w);
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                g[n][k] = fmaf(a, gv[k], g[n][k]);
                if (DOTS) dot = fmaf(gv[k], w[k], dot);
              }
            }
          if (DOTS && p.grad_a != nullptr) {
            dot = warp_sum(dot);
            if (i < 36) dx += lane == i - 4 ? dot : 0.f;
            else if (lane == 0 && dot != 0.f) atomicAdd(&p.grad_a[b + i], dot * gsc);
          }
        }
#pragma unroll
        for (int n = 0; n < NV; ++n) {
          if (e0 + 256 * n < end) {
            float w[8], dg0[8];
            if (DOTS) wv[n].get(w);
            const bool extra = r == 0 && xrow != nullptr;
            if (extra) load8f(xrow + e0 + 256 * n, dg0);
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              float gk = g[n][k] * gsc;
              if (DOTS) gk = fmaf(pc, w[k], gk);  // without a penalty too, as in the update: a weight that is not finite shows in the norm
              if (extra) gk += dg0[k];
              nsq = fmaf(gk, gk, nsq);
            }
          }
        }
      }
      if (DOTS && p.grad_a != nullptr) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (j < ne) {
            const float sdot = warp_sum(dacc[j]);
            if (lane == 0 && sdot != 0.f) atomicAdd(&p.grad_a[b + j], sdot * gsc);
          }
        }
        if (4 + lane < ne && dx != 0.f) atomicAdd(&p.grad_a[b + 4 + lane], dx * gsc);
      }
    }
    cur = nxt;
    nxt = after;
  }
  block_add(nsq, p.norm_sq_out);
}
template <typename WT, bool DOTS>
static void launch_rows_norm(const DecAdamParams& p, int num_sms, cudaStream_t st) {
  const int vecs = (p.d + 255) / 256;  // a warp per row up to 1024 elements, even segments of longer ones
  if (vecs <= 1) launch_alone(rows_norm_kernel<WT, DOTS, 1>, 2 * num_sms, 256, 0, st, p);
  else if (vecs == 2) launch_alone(rows_norm_kernel<WT, DOTS, 2>, 2 * num_sms, 256, 0, st, p);
  else if (vecs == 3 || vecs == 5 || vecs == 6) launch_alone(rows_norm_kernel<WT, DOTS, 3>, 2 * num_sms, 256, 0, st, p);
  else launch_alone(rows_norm_kernel<WT, DOTS, 4>, 2 * num_sms, 256, 0, st, p);
}

// ---------------------------------------------------------------- untied decoders, bulk-copy pipeline
// The update streams every decoder row once: (w, m, v) in, (w, m, v) out, 20 bytes per element with bf16
// weights, so the kernel is a copy with some arithmetic in the middle.  A producer thread per CTA moves
// whole rows between global and shared memory with 1-D bulk copies (cp.async.bulk, no multicast): row in
// (w, m, v and the gradient-seed rows of the feature's first four entries) -> consumers update the row in
// place in shared memory -> row out.  The ring keeps several rows per CTA in flight in both directions and
// the consumers only wait on global loads for features with more than four entries.
// Entries beyond the staged ones are gathered by the consumers in batches, see add_entries.
// Every mbarrier wait is bounded; a timeout sets the status word and drains the copies in flight.
constexpr int kAdamStages = 4;  // at most; rows above 24 KB per stage run with three so that two CTAs fit an SM
constexpr int kAdamSlots = 4;  // gradient-seed rows per stage

struct AdamStageHdr {  // 64 bytes in front of every stage, written by the producer before it arms the barrier
  int ne;      // entries of the feature
  int b;       // start of the feature in the CSR arrays
  int col;     // ti * F_pitch + f
  int ti;
  int r;       // row inside the feature
  int R;
  long long elem_off;  // element offset of the row inside its tensor
  float a[kAdamSlots];
  int pad[4];
};
static_assert(sizeof(AdamStageHdr) == 64, "stage header is 64 bytes");

struct AdamBulkShared {
  uint64_t full[kAdamStages];
  uint64_t done[kAdamStages];
  int abort_flag;
};

struct FeatMeta {
  int b, e;
  int tok[kAdamSlots];
  float a[kAdamSlots];
};

// Vector access to EPT (4 or 8) consecutive elements of a row held in shared memory.
template <int EPT>
__device__ __forceinline__ void ldf(const float* p, float (&o)[EPT]) {
#pragma unroll
  for (int i = 0; i < EPT; i += 4) {
    const float4 a = *reinterpret_cast<const float4*>(p + i);
    o[i] = a.x; o[i + 1] = a.y; o[i + 2] = a.z; o[i + 3] = a.w;
  }
}
template <int EPT>
__device__ __forceinline__ void stf(float* p, const float (&o)[EPT]) {
#pragma unroll
  for (int i = 0; i < EPT; i += 4) *reinterpret_cast<float4*>(p + i) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
}
template <int EPT>
__device__ __forceinline__ void ldbf(const t16* p, float (&o)[EPT]) {
#pragma unroll
  for (int i = 0; i < EPT; i += 4) {
    const uint2 q = *reinterpret_cast<const uint2*>(p + i);
    o[i] = t16_lo(q.x); o[i + 1] = t16_hi(q.x); o[i + 2] = t16_lo(q.y); o[i + 3] = t16_hi(q.y);
  }
}
template <int EPT, bool SR>
__device__ __forceinline__ void stbf(t16* p, const float (&o)[EPT], unsigned int seed, unsigned int idx) {
#pragma unroll
  for (int i = 0; i < EPT; i += 4) {
    uint2 q;
    if (!SR || CLT_T16_IS_HALF) {
      q.x = pack_t16x2(o[i], o[i + 1]); q.y = pack_t16x2(o[i + 2], o[i + 3]);
    } else {
      uint32_t h[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t u = __float_as_uint(o[i + k]);
        const uint32_t rnd = hash32((idx + i + k) ^ seed) & 0xFFFFu;
        h[k] = ((u & 0x7F800000u) == 0x7F800000u) ? (u >> 16) : ((u + rnd) >> 16);
      }
      q.x = h[0] | (h[1] << 16); q.y = h[2] | (h[3] << 16);
    }
    *reinterpret_cast<uint2*>(p + i) = q;
  }
}

// Elements i and i + 1 of a register array.
template <int N>
__device__ __forceinline__ float2 f2_get(const float (&x)[N], int i) { return make_float2(x[i], x[i + 1]); }
template <int N>
__device__ __forceinline__ void f2_put(float (&x)[N], int i, float2 v) { x[i] = v.x; x[i + 1] = v.y; }

// Warp sums of N values at once (N a power of two up to 32): every exchange halves the number of values a lane still carries,
// N - 1 + 5 - log2(N) shuffles instead of 5 N.  Returns the total of value warp_sum_slot<N>(lane); the tree is warp_sum's.
template <int N>
__device__ __forceinline__ float warp_sum_many(float (&v)[N], int lane) {
  int o = 16;
#pragma unroll
  for (int half = N / 2; half >= 1; half >>= 1, o >>= 1) {
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < half; ++i) {
      const float send = upper ? v[i] : v[i + half];
      const float keep = upper ? v[i + half] : v[i];
      v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, o);
    }
  }
  float r = v[0];
#pragma unroll
  for (int q = 16 / N; q >= 1; q >>= 1) r += __shfl_xor_sync(0xFFFFFFFFu, r, q);
  return r;
}
template <int N>
__device__ __forceinline__ int warp_sum_slot(int lane) { return lane / (32 / N); }

// g += a_j * seed_j and dL/da of the entries of one batch: lane j of the warp holds entry j (its slot in the CSR arrays, token and
// activation), cnt of them.  The seed rows come kBatch at a time, so a feature with many entries waits for L2 once per
// kBatch of them and not twice per entry (eight entries per feature on average, tied Pythia-70m shape: both sweeps of a step
// 1.81 -> 1.60 ms).  It takes 72 registers; a cap of 64 spills and cost 0.4 ms at the GPT-2 shape.
template <int EPT, int kBatch, bool kPairs>
__device__ __forceinline__ void add_entries(int cnt, int my_x, int my_tok, float my_a, const t16* gs_t, int d, bool act, int lane, const float (&w)[EPT],
                                            float (&g)[EPT], float* grad_a, float gsc) {
  for (int j0 = 0; j0 < cnt; j0 += kBatch) {
    uint2 q2[kBatch][EPT / 4];
    float dot[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int tok = __shfl_sync(0xFFFFFFFFu, my_tok, j0 + k);
      if (act && j0 + k < cnt) {
#pragma unroll
        for (int z = 0; z < EPT / 4; ++z) q2[k][z] = __ldg(reinterpret_cast<const uint2*>(gs_t + 1LL * tok * d) + z);
      }
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const float a = __shfl_sync(0xFFFFFFFFu, my_a, j0 + k);
      float2 dot2 = f2_all(0.f);
      if (act && j0 + k < cnt) {
#pragma unroll
        for (int z = 0; z < EPT / 4; ++z) {
          const float2 gv[2] = {make_float2(t16_lo(q2[k][z].x), t16_hi(q2[k][z].x)), make_float2(t16_lo(q2[k][z].y), t16_hi(q2[k][z].y))};
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            const int e = 4 * z + 2 * c;
            if constexpr (kPairs) {
              f2_put(g, e, f2_fma(f2_all(a), gv[c], f2_get(g, e)));
              dot2 = f2_fma(gv[c], f2_get(w, e), dot2);
            } else {
              g[e] = fmaf(a, gv[c].x, g[e]); g[e + 1] = fmaf(a, gv[c].y, g[e + 1]);
              dot2.x = fmaf(gv[c].y, w[e + 1], fmaf(gv[c].x, w[e], dot2.x));
            }
          }
        }
      }
      dot[k] = dot2.x + dot2.y;
    }
    if (grad_a != nullptr) {
      const float sdot = warp_sum_many<kBatch>(dot, lane);
      const int k = j0 + warp_sum_slot<kBatch>(lane);
      const int x = __shfl_sync(0xFFFFFFFFu, my_x, k);
      if (lane % (32 / kBatch) == 0 && k < cnt && sdot != 0.f) atomicAdd(&grad_a[x], sdot * gsc);
    }
  }
}

// PT: per-target tied decoders (one row per feature and target layer, shared by the source layers below): the entries of a row
// come from several CSR segments, so none are staged in slots.
// NB: entries beyond the staged ones that are loaded together.  NARROW: 64 registers instead of 72 (d <= 640), 80 instead of 96 with
// eight elements per thread (d <= 1792).
template <typename WT, bool SR, int EPT, typename MT, bool PT = false, int NB = 4, bool NARROW = false>
__global__ void __launch_bounds__(NARROW ? (EPT == 4 ? 192 : 256) : 288, NARROW ? (EPT == 4 ? 5 : 3) : (EPT == 4 ? 3 : 2)) decoder_rows_adam_bulk_kernel(const DecAdamParams p, int gthreads, int stage_bytes, int ns, int* status) {
  // Two-wide arithmetic (12 x 768, 24576 features: both sweeps 5987 -> 5932 us, 3072 features 820 -> 794; 4 x 640, 25 entries per feature 1335 -> 1276),
  // except in the form whose registers it overflows (6 x 2048: 861 us without, 869 with it).
  constexpr bool kPairs = EPT == 4 || NB != 4 || PT;
  extern __shared__ __align__(128) uint8_t smem_raw_adam[];  // bulk copies need 16-byte alignment only
  uint8_t* ring = smem_raw_adam;
  AdamBulkShared* sh = reinterpret_cast<AdamBulkShared*>(ring + size_t(ns) * stage_bytes);
  const int d = p.d, B = p.B, Fp = p.F_pitch;
  const int nconsumer = gthreads;
  const int tid = threadIdx.x;
  const StepScales sc = read_step_ctl(p.ctl);
  if (sc.skip) return;  // the whole grid sees the same flag: a skipped step touches nothing
  // Features b, b + grid, ... of every tensor.  PT: rows b, b + grid, ... of all tensors taken as one list, so that the rows of a
  // feature with many entries (one per target, gathered by the consumers) fall to different CTAs: 90 entries in eight of 1128
  // features, 8 targets, d = 512: 285 us when one CTA had all rows of a feature, 62 us now.
  const int nf = (Fp - int(blockIdx.x) + int(gridDim.x) - 1) / int(gridDim.x);  // features of this CTA per tensor
  long long n_rows = 0;
  for (int ti = 0; ti < p.ntensors; ++ti) n_rows += 1LL * (nf > 0 ? nf : 0) * p.rows[ti];
  if (PT) n_rows = (1LL * p.ntensors * Fp - blockIdx.x + gridDim.x - 1) / gridDim.x;
  const int n = int(n_rows);
  const uint32_t w_bytes = uint32_t(d) * sizeof(WT), mv_bytes = uint32_t(d) * sizeof(MT), gs_bytes = uint32_t(d) * 2u;
  const uint32_t off_w = 64, off_m = off_w + w_bytes, off_v = off_m + mv_bytes, off_gs = off_v + mv_bytes;
  if (tid == 0) {
    for (int s = 0; s < ns; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->done[s], nconsumer / 32);
    }
    sh->abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();
  volatile int* abort_flag = &sh->abort_flag;

  if (tid == nconsumer) {
    // ------------------------------------------------------------------ producer / store issuer
    const int n_feat = PT ? n : nf * p.ntensors;
    auto col_of = [&](int k) { const int ti = k / nf; return ti * Fp + int(blockIdx.x) + (k - ti * nf) * int(gridDim.x); };
    auto load_offsets = [&](int k, FeatMeta& mt) {
      if (k < n_feat) { const int c = col_of(k); mt.b = __ldg(p.feat_off + c); mt.e = __ldg(p.feat_off + c + 1); }
      else { mt.b = 0; mt.e = 0; }
    };
    auto load_entries = [&](FeatMeta& mt) {
#pragma unroll
      for (int j = 0; j < kAdamSlots; ++j) {
        const bool in = mt.b + j < mt.e;
        mt.tok[j] = in ? __ldg(p.fcsr_tok + mt.b + j) : 0;
        mt.a[j] = in ? __ldg(p.fcsr_val + mt.b + j) : 0.f;
        if (!clt_in_bounds(mt.tok[j], B, status, 201)) { mt.tok[j] = 0; mt.a[j] = 0.f; }  // debug build: token index from the CSR
      }
    };
    // rows are touched once per step, the gradient seed is re-read by every feature: keep the latter in L2
    const uint64_t pol_stream = l2_policy_evict_first();
    const uint64_t pol_keep = l2_policy_evict_last();
    FeatMeta cur, nxt, nn;
    if (PT) {
      cur.b = cur.e = 0;
#pragma unroll
      for (int j = 0; j < kAdamSlots; ++j) { cur.tok[j] = 0; cur.a[j] = 0.f; }
    } else {
      load_offsets(0, cur); load_entries(cur);
      load_offsets(1, nxt);
    }
    int k = 0, r = 0;             // feature / row whose loads are issued next
    int ti = 0, R = n_feat > 0 ? p.rows[0] : 0;
    int f = int(blockIdx.x);
    if (PT) { ti = f / Fp; f -= ti * Fp; R = 1; }
    bool fresh = true;            // first row of a feature: start the prefetch of the following ones
    auto issue_loads = [&](int i) {
      if (!PT && fresh) {
        load_entries(nxt);        // offsets of k + 1 were requested one feature ago
        load_offsets(k + 2, nn);
        fresh = false;
      }
      const int st = i % ns;
      uint8_t* stage = ring + size_t(st) * stage_bytes;
      AdamStageHdr* h = reinterpret_cast<AdamStageHdr*>(stage);
      const int ne = PT ? 0 : cur.e - cur.b;
      const long long elem_off = (1LL * f * R + r) * d;
      h->ne = ne; h->b = cur.b; h->col = ti * Fp + f; h->ti = ti; h->r = r; h->R = R; h->elem_off = elem_off;
#pragma unroll
      for (int j = 0; j < kAdamSlots; ++j) h->a[j] = cur.a[j];
      const int nslot = ne < kAdamSlots ? ne : kAdamSlots;
      mbar_expect_tx(&sh->full[st], w_bytes + 2u * mv_bytes + uint32_t(nslot) * gs_bytes);
      bulk_load_1d_hint(stage + off_w, static_cast<const WT*>(p.w[ti]) + elem_off, w_bytes, &sh->full[st], pol_stream);
      bulk_load_1d_hint(stage + off_m, reinterpret_cast<const MT*>(p.m[ti]) + elem_off, mv_bytes, &sh->full[st], pol_stream);
      bulk_load_1d_hint(stage + off_v, reinterpret_cast<const MT*>(p.v[ti]) + elem_off, mv_bytes, &sh->full[st], pol_stream);
      const t16* gs_t = p.gs + 1LL * (ti + r) * B * d;
#pragma unroll
      for (int j = 0; j < kAdamSlots; ++j)
        if (j < nslot) bulk_load_1d_hint(stage + off_gs + j * gs_bytes, gs_t + 1LL * cur.tok[j] * d, gs_bytes, &sh->full[st], pol_keep);
      // advance to the next row
      if (PT) {
        for (f += int(gridDim.x); f >= Fp; f -= Fp) ++ti;
      } else if (++r == R) {
        r = 0; ++k;
        cur = nxt; nxt.b = nn.b; nxt.e = nn.e;
        fresh = true;
        if (k < n_feat) {
          const int nti = k / nf;
          if (nti != ti) { ti = nti; R = p.rows[ti]; }
          f = int(blockIdx.x) + (k - ti * nf) * int(gridDim.x);
        }
      }
    };
    int issued = 0;
    for (; issued < n && issued < ns; ++issued) issue_loads(issued);
    int i = 0;
    for (; i < n; ++i) {
      const int st = i % ns;
      if (!mbar_wait(&sh->done[st], (i / ns) & 1, abort_flag)) break;
      uint8_t* stage = ring + size_t(st) * stage_bytes;
      const AdamStageHdr* h = reinterpret_cast<const AdamStageHdr*>(stage);
      const int sti = h->ti;
      const long long eo = h->elem_off;
      bulk_store_1d_hint(static_cast<WT*>(p.w[sti]) + eo, stage + off_w, w_bytes, pol_stream);
      bulk_store_1d_hint(reinterpret_cast<MT*>(p.m[sti]) + eo, stage + off_m, mv_bytes, pol_stream);
      bulk_store_1d_hint(reinterpret_cast<MT*>(p.v[sti]) + eo, stage + off_v, mv_bytes, pol_stream);
      bulk_commit();
      if (i >= 1 && issued < n) {
        bulk_wait_read<1>();  // the stores of row i - 1 have read their stage: it can be refilled
        issue_loads(issued);
        ++issued;
      }
    }
    bulk_wait_all();
    if (*abort_flag) {
      // rows whose loads were issued but never consumed: give them a bounded chance to land
      for (int j = i; j < issued; ++j) {
        const long long start = clock64();
        while (!mbar_try_wait(&sh->full[j % ns], (j / ns) & 1))
          if (clock64() - start > kWaitTimeoutCycles) break;
      }
    }
  } else if (tid < nconsumer) {
// ------------------------------------------------------------------ consumers: one row per stage
    const int lane = tid & 31;
    const int e0 = tid * EPT;
    const bool act = e0 < d;
    const HyperRegs hr = make_regs(p.h);
    const float gsc = hr.gscale * (p.use_inv_scale ? sc.inv_scale : 1.f);
    float dacc[kAdamSlots] = {0.f, 0.f, 0.f, 0.f};
    float norm2 = 0.f, pc = 0.f;
    for (int i = 0; i < n; ++i) {
      const int st = i % ns;
      if (!mbar_wait_warp(&sh->full[st], (i / ns) & 1, abort_flag)) break;
      uint8_t* stage = ring + size_t(st) * stage_bytes;
      const AdamStageHdr* h = reinterpret_cast<const AdamStageHdr*>(stage);
      const int ne = h->ne, r = h->r, R = h->R, col = h->col, ti = h->ti, b = h->b;
      if (r == 0) {
#pragma unroll
        for (int j = 0; j < kAdamSlots; ++j) dacc[j] = 0.f;
        norm2 = 0.f;
        pc = p.pen_coef ? __ldg(p.pen_coef + col) : 0.f;
        if (PT && p.pen_coef) pc = warp_sum(lane <= ti ? __ldg(p.pen_coef + lane * Fp + col - ti * Fp) : 0.f);  // the row is part of the norms of all sources
      }
      float w[EPT], m[EPT], v[EPT], g[EPT];
#pragma unroll
      for (int q = 0; q < EPT; ++q) { g[q] = 0.f; w[q] = 0.f; }
      WT* w_s = reinterpret_cast<WT*>(stage + off_w) + e0;
      MT* m_s = reinterpret_cast<MT*>(stage + off_m) + e0;
      MT* v_s = reinterpret_cast<MT*>(stage + off_v) + e0;
      if (act) {
        if (sizeof(WT) == 2) ldbf<EPT>(reinterpret_cast<const t16*>(w_s), w);
        else ldf<EPT>(reinterpret_cast<const float*>(w_s), w);
        if (sizeof(MT) == 2) {
          ldbf<EPT>(reinterpret_cast<const t16*>(m_s), m);
          ldbf<EPT>(reinterpret_cast<const t16*>(v_s), v);
        } else {
          ldf<EPT>(reinterpret_cast<const float*>(m_s), m);
          ldf<EPT>(reinterpret_cast<const float*>(v_s), v);
        }
        const t16* gs_s = reinterpret_cast<const t16*>(stage + off_gs) + e0;
#pragma unroll
        for (int j = 0; j < kAdamSlots; ++j) {
          if (j < ne) {
            const float a = h->a[j];
            float gv[EPT];
            ldbf<EPT>(gs_s + j * d, gv);
#pragma unroll
            for (int q = 0; q < EPT; q += 2) {
              if constexpr (kPairs) {
                f2_put(g, q, f2_fma(f2_all(a), f2_get(gv, q), f2_get(g, q)));
              } else {
                g[q] = fmaf(a, gv[q], g[q]); g[q + 1] = fmaf(a, gv[q + 1], g[q + 1]);
                dacc[j] = fmaf(gv[q + 1], w[q + 1], fmaf(gv[q], w[q], dacc[j]));
              }
            }
            if constexpr (kPairs) {
              float2 dot = f2_mul(f2_get(gv, 0), f2_get(w, 0));
#pragma unroll
              for (int q = 2; q < EPT; q += 2) dot = f2_fma(f2_get(gv, q), f2_get(w, q), dot);
              dacc[j] += dot.x + dot.y;
            }
          }
        }
      }
      if (PT) {
        // the entries of feature f in all source layers s <= ti, one CSR segment per layer: the lanes hold the segments, and
        // entry j of their concatenation lies in the segment whose inclusive count is the first above j
        const int f = col - ti * Fp;
        int seg_b = 0, seg_n = 0;
        if (lane <= ti) {
          seg_b = __ldg(p.feat_off + lane * Fp + f);
          seg_n = __ldg(p.feat_off + lane * Fp + f + 1) - seg_b;
        }
        int incl = seg_n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
          if (lane >= o) incl += up;
        }
        const int total = __shfl_sync(0xFFFFFFFFu, incl, 31);
        for (int j0 = 0; j0 < total; j0 += 32) {
          const int j = j0 + lane;
          int seg = 0;
          for (int s = 0; s < ti; ++s) seg += __shfl_sync(0xFFFFFFFFu, incl, s) <= j ? 1 : 0;
          const int x = __shfl_sync(0xFFFFFFFFu, seg_b, seg) + j - (__shfl_sync(0xFFFFFFFFu, incl, seg) - __shfl_sync(0xFFFFFFFFu, seg_n, seg));
          int my_tok = j < total ? __ldg(p.fcsr_tok + x) : 0;
          float my_a = j < total ? __ldg(p.fcsr_val + x) : 0.f;
          check_token(my_tok, my_a, B, status, 207);
          add_entries<EPT, NB, kPairs>(min(32, total - j0), x, my_tok, my_a, p.gs + 1LL * ti * B * d + e0, d, act, lane, w, g, p.grad_a, gsc);
        }
      } else {
        for (int x0 = b + kAdamSlots; x0 < b + ne; x0 += 32) {  // entries beyond the slots
          const int cnt = min(32, b + ne - x0);
          int my_tok = lane < cnt ? __ldg(p.fcsr_tok + x0 + lane) : 0;
          float my_a = lane < cnt ? __ldg(p.fcsr_val + x0 + lane) : 0.f;
          check_token(my_tok, my_a, B, status, 208);
          add_entries<EPT, NB, kPairs>(cnt, x0 + lane, my_tok, my_a, p.gs + 1LL * (ti + r) * B * d + e0, d, act, lane, w, g, p.grad_a, gsc);
        }
      }
      if (act) {
        float dg0[EPT];
        const float* xrow = r == 0 ? extra_row_ptr(p, col) : nullptr;
        const bool extra = xrow != nullptr;
        if (extra) {
#pragma unroll
          for (int q = 0; q < EPT; q += 4) {
            const float4 t4 = __ldg(reinterpret_cast<const float4*>(xrow + e0 + q));
            dg0[q] = t4.x; dg0[q + 1] = t4.y; dg0[q + 2] = t4.z; dg0[q + 3] = t4.w;
          }
        }
        float2 row2 = f2_all(0.f);
#pragma unroll
        for (int q = 0; q < EPT; q += 2) {
          if constexpr (kPairs) {
            float2 w2 = f2_get(w, q), m2 = f2_get(m, q), v2 = f2_get(v, q);
            float2 gq = f2_fma(f2_all(pc), w2, f2_mul(f2_get(g, q), f2_all(gsc)));
            if (extra) gq = f2_add(gq, f2_get(dg0, q));
            adam2(w2, m2, v2, f2_mul(gq, f2_all(sc.clip)), hr);
            f2_put(w, q, w2); f2_put(m, q, m2); f2_put(v, q, v2);
            if (!PT) row2 = f2_fma(w2, w2, row2);
          } else {
#pragma unroll
            for (int z = q; z < q + 2; ++z) {
              float gq = fmaf(pc, w[z], g[z] * gsc);
              if (extra) gq += dg0[z];
              adam1(w[z], m[z], v[z], gq * sc.clip, hr);
              if (!PT) row2.x = fmaf(w[z], w[z], row2.x);
            }
          }
        }
        const unsigned long long gidx = (unsigned long long)(p.row_start[ti] * d + h->elem_off + e0);
        if (sizeof(WT) == 2) stbf<EPT, SR>(reinterpret_cast<t16*>(w_s), w, p.h.sr_seed, (unsigned int)gidx);
        else stf<EPT>(reinterpret_cast<float*>(w_s), w);
        if (PT) {  // norms of the stored (rounded) weights
          ldbf<EPT>(reinterpret_cast<const t16*>(w_s), w);
#pragma unroll
          for (int q = 0; q < EPT; q += 2) row2 = f2_fma(f2_get(w, q), f2_get(w, q), row2);
        }
        norm2 += row2.x + row2.y;
        if (sizeof(MT) == 2) {
          // bf16 moments are always rounded stochastically: with beta2 = 0.999 a nearest rounding would freeze v
          // one hash per thread and row seeds a linear congruential stream: two 16-bit dither values per element
          uint32_t rng = hash32((unsigned int)gidx ^ p.h.moment_seed);
          t16* mo = reinterpret_cast<t16*>(m_s);
          t16* vo = reinterpret_cast<t16*>(v_s);
#pragma unroll
          for (int q = 0; q < EPT; q += 2) {
            uint32_t hm[2], hv[2];
#pragma unroll
            for (int z = 0; z < 2; ++z) {
              rng = rng * 1664525u + 1013904223u;
              const uint32_t um = __float_as_uint(m[q + z]), uv = __float_as_uint(v[q + z]);
              hm[z] = ((um & 0x7F800000u) == 0x7F800000u) ? (um >> 16) : ((um + (rng >> 16)) >> 16);
              hv[z] = ((uv & 0x7F800000u) == 0x7F800000u) ? (uv >> 16) : ((uv + ((rng * 0x9E3779B1u) >> 16)) >> 16);
            }
            *reinterpret_cast<uint32_t*>(mo + q) = hm[0] | (hm[1] << 16);
            *reinterpret_cast<uint32_t*>(vo + q) = hv[0] | (hv[1] << 16);
          }
        } else {
          stf<EPT>(reinterpret_cast<float*>(m_s), m);
          stf<EPT>(reinterpret_cast<float*>(v_s), v);
        }
      }
      if (r == R - 1) {
        if (!PT && p.grad_a != nullptr) {
          const float sdot = warp_sum_many<kAdamSlots>(dacc, lane);  // the sums of slots without an entry are zero
          const int j = warp_sum_slot<kAdamSlots>(lane);
          if (lane % (32 / kAdamSlots) == 0 && j < ne && sdot != 0.f) atomicAdd(&p.grad_a[b + j], sdot * gsc);
        }
        if (p.norm2_out != nullptr) {
          const float sn = warp_sum(norm2);
          if (lane == 0) atomicAdd(&p.norm2_out[col], sn);
        }
      }
      fence_proxy_async();  // the row written above is read next by the bulk store (async proxy)
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh->done[st]);
    }
  }
  __syncthreads();
  if (tid == 0 && sh->abort_flag && status != nullptr) atomicCAS(status, STATUS_OK, STATUS_WAIT_TIMEOUT);
}

// ------------------------------------------------------------------ row update, one warp per row
// Rows of up to 512 elements (16-bit weights, fp32 moments): the row is one warp's alone, NC blocks of 128 elements, four per lane.  A
// warp has its own ring of kNarrowStages rows in shared memory, filled and drained by bulk copies that its first lane issues, and gathers the
// seed (input) rows of the row's entries itself, kNarrowBatch at a time; offsets are requested two rows ahead, the first 32 entries one row
// ahead, the first batch of seed rows before the row itself is waited for.
// Against the row pipeline above (a CTA per row): that one has five or six rows per SM at its consumers, each of which waits
// for the lists and seed rows beyond the four staged ones, twice per row and one row after the other; here 16 to 24 rows per SM do so at the
// same time, and the dot products of a row (dL/da) and its norm need no sum across warps.
// With sixteen warps per SM what counts is the instructions of a row (issue slots 60 % full, DRAM at 45 %), so the arithmetic is two-wide: tied
// Pythia-70m shape, both sweeps 933 -> 860 us; per-target decoders of 6 x 16384 x 512, 9 entries per row, 284 -> 254; rows with three entries unchanged.
// A row's stage is refilled in the next row's turn, behind the requests for its seed rows, when the store has long read it: waiting for
// the store at the end of the row, and a test per block of 128 although only the last can be short, cost 3 to 7 % (6 x 32768 x 512 with 4 entries
// per row 677 -> 655 us, per-target decoders 230 -> 213, 8 x 8192 x 256 untied 358 -> 344).  Rows of up to 128 elements are over too
// soon for that (277 us, refilled late 283): they wait for the store.  With few entries wide rows of this form ask for more than DRAM takes; the
// launcher then lets fewer CTAs work.
template <int NC>
__device__ __forceinline__ void load_seed_row(const t16* row, int lane, int d, uint2 (&q)[NC]) {
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int e = c * 128 + lane * 4;
    if (c + 1 < NC || e < d) q[c] = __ldg(reinterpret_cast<const uint2*>(row + e));
  }
}

constexpr int kNarrowStages = 2;
constexpr int kNarrowWarps = 4;
constexpr int kNarrowBatch = 4;

// Resident CTAs per SM: 128 registers for rows above 256, 96 for 129 to 256, 80 below.  Five CTAs of 96 registers spill at 512 (1069 us
// against 925 for both sweeps of the tied Pythia-70m shape), and three stages with 14 warps are slower than two with 16 (1063).
__host__ __device__ constexpr int narrow_ctas(int nc) { return nc >= 3 ? 4 : (nc == 2 ? 5 : 6); }

struct RowAt {
  long long idx;  // position in the list of all rows
  int ti, f, r;
};

template <bool SR, int NC, bool PT>
__global__ void __launch_bounds__(32 * kNarrowWarps, narrow_ctas(NC))
narrow_rows_adam_kernel(const DecAdamParams p, long long total_rows, float ctas_empty, float ctas_per_entry, int* status) {
  static_assert(kNarrowStages == 2, "the late refill is for the next row");
  constexpr bool kRefillLate = NC > 1;
  extern __shared__ __align__(128) uint8_t smem_narrow[];
  __shared__ uint64_t full_s[kNarrowWarps][kNarrowStages];
  __shared__ int abort_s;
  const int n_entries = NC >= 3 ? __ldg(p.feat_off + p.L * p.F_pitch) : 0;
  const StepScales sc = read_step_ctl(p.ctl);
  if (sc.skip) return;  // the whole grid sees the same flag: a skipped step touches nothing
  int grid = int(gridDim.x);
  if (NC >= 3) {  // of the resident CTAs, as many as keep DRAM busy with these lists
    float per_row = float(n_entries) / float(p.L * p.F_pitch);
    if (PT) per_row *= 0.5f * float(p.L + 1);  // an entry is in the rows of all later targets
    const float enough = ctas_empty + ctas_per_entry * per_row;
    if (enough < 0.93f * float(grid)) grid = int(enough);
    if (int(blockIdx.x) >= grid) return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int d = p.d, Fp = p.F_pitch;
  const uint32_t w_bytes = uint32_t(d) * 2u, mv_bytes = uint32_t(d) * 4u, stage_bytes = w_bytes + 2u * mv_bytes;
  uint8_t* ring = smem_narrow + size_t(warp) * kNarrowStages * stage_bytes;
  uint64_t* full = full_s[warp];
  if (threadIdx.x == 0) abort_s = 0;
  if (lane == 0) {
    for (int s = 0; s < kNarrowStages; ++s) mbar_init(&full[s], 1);
    fence_barrier_init();
  }
  __syncthreads();
  volatile int* abort_flag = &abort_s;
  const HyperRegs hr = make_regs(p.h);
  const float gsc = hr.gscale * (p.use_inv_scale ? sc.inv_scale : 1.f);
  const uint64_t pol_stream = l2_policy_evict_first();  // rows are touched once per step

  const int stride = grid * kNarrowWarps;
  const auto place = [&](RowAt& at) {  // tensor, feature and row of at.idx (at.ti: at or before the right one)
    if (at.idx >= total_rows) return;
    while (at.idx >= p.row_start[at.ti + 1]) ++at.ti;
    const long long rem = at.idx - p.row_start[at.ti];
    const int R = p.rows[at.ti];
    at.f = R == 1 ? int(rem) : int(rem / R);
    at.r = R == 1 ? 0 : int(rem - 1LL * at.f * R);
  };
  const auto elem_of = [&](const RowAt& at) { return (at.idx - p.row_start[at.ti]) * d; };
  // entries: PT: lane s holds the segment of source layer s <= ti; else all lanes hold the feature's one segment
  const auto load_offsets = [&](const RowAt& at, int& b, int& n) {
    b = n = 0;
    if (at.idx >= total_rows) return;
    if (PT ? lane <= at.ti : true) {
      const int* o = p.feat_off + (PT ? lane : at.ti) * Fp + at.f;
      b = __ldg(o);
      n = __ldg(o + 1) - b;
    }
  };
  // entry j0 + lane of the row: its place in the CSR arrays, token and activation; returns the number of entries
  const auto load_list = [&](const RowAt& at, int b, int n, int j0, int& x, int& tok, float& a) -> int {
    const int j = j0 + lane;
    int total = n;
    if (PT) {
      int incl = n;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += up;
      }
      total = __shfl_sync(0xFFFFFFFFu, incl, 31);
      int seg = 0;
      if (total > 0)
        for (int s = 0; s < at.ti; ++s) seg += __shfl_sync(0xFFFFFFFFu, incl, s) <= j ? 1 : 0;
      x = __shfl_sync(0xFFFFFFFFu, b, seg) + j - (__shfl_sync(0xFFFFFFFFu, incl, seg) - __shfl_sync(0xFFFFFFFFu, n, seg));
    } else {
      x = b + j;
    }
    tok = j < total ? __ldg(p.fcsr_tok + x) : 0;
    a = j < total ? __ldg(p.fcsr_val + x) : 0.f;
    if (!clt_in_bounds(tok, p.B, status, 202)) { tok = 0; a = 0.f; }
    return total;
  };
  const auto issue_row = [&](const RowAt& at, int st) {
    if (lane != 0 || at.idx >= total_rows) return;
    uint8_t* stage = ring + size_t(st) * stage_bytes;
    const long long eo = elem_of(at);
    mbar_expect_tx(&full[st], stage_bytes);
    bulk_load_1d_hint(stage, static_cast<const t16*>(p.w[at.ti]) + eo, w_bytes, &full[st], pol_stream);
    bulk_load_1d_hint(stage + w_bytes, p.m[at.ti] + eo, mv_bytes, &full[st], pol_stream);
    bulk_load_1d_hint(stage + w_bytes + mv_bytes, p.v[at.ti] + eo, mv_bytes, &full[st], pol_stream);
  };

  RowAt cur{1LL * blockIdx.x * kNarrowWarps + warp, 0, 0, 0};
  place(cur);
  RowAt nxt{cur.idx + stride, cur.ti, 0, 0};
  place(nxt);
  for (int k = 0; k < kNarrowStages; ++k) {
    RowAt at{cur.idx + k * stride, cur.ti, 0, 0};
    place(at);
    issue_row(at, k);
  }
  int b = 0, n = 0, b1 = 0, n1 = 0;  // offsets of the current and the next row
  load_offsets(cur, b, n);
  load_offsets(nxt, b1, n1);
  int x, tok;
  float a;
  int total = load_list(cur, b, n, 0, x, tok, a);
  bool ok = true;
  uint32_t i = 0;
  for (; cur.idx < total_rows; ++i) {
    const int st = int(i % kNarrowStages);
    RowAt nn{nxt.idx + stride, nxt.ti, 0, 0};
    place(nn);
    int b2, n2;
    load_offsets(nn, b2, n2);
    const t16* gs_t = p.gs + 1LL * (cur.ti + cur.r) * p.B * d;
    uint2 q[kNarrowBatch][NC];
#pragma unroll
    for (int k = 0; k < kNarrowBatch; ++k) {
      const int tk = __shfl_sync(0xFFFFFFFFu, tok, k);
      if (k < total) load_seed_row<NC>(gs_t + 1LL * tk * d, lane, d, q[k]);
    }
    int x1, tok1;
    float a1;
    const int total1 = load_list(nxt, b1, n1, 0, x1, tok1, a1);
    if (kRefillLate && i > 0) {  // the stage of the row before; its store has read it by now
      if (lane == 0) bulk_wait_read<0>();
      issue_row(nxt, int((i + 1) % kNarrowStages));
    }
    const int col = cur.ti * Fp + cur.f;
    float pc = p.pen_coef ? __ldg(p.pen_coef + col) : 0.f;
    if (PT && p.pen_coef) pc = warp_sum(lane <= cur.ti ? __ldg(p.pen_coef + lane * Fp + cur.f) : 0.f);  // the row is part of the norms of all sources
    if (!mbar_wait_warp(&full[st], (i / kNarrowStages) & 1, abort_flag)) { ok = false; break; }
    uint8_t* stage = ring + size_t(st) * stage_bytes;
    t16* w_s = reinterpret_cast<t16*>(stage);
    float* m_s = reinterpret_cast<float*>(stage + w_bytes);
    float* v_s = reinterpret_cast<float*>(stage + w_bytes + mv_bytes);
    float2 w[NC][2], g[NC][2];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
#pragma unroll
      for (int k = 0; k < 2; ++k) w[c][k] = g[c][k] = f2_all(0.f);
      if (c + 1 < NC || c * 128 + lane * 4 < d) {
        const uint2 u = *reinterpret_cast<const uint2*>(w_s + c * 128 + lane * 4);
        w[c][0] = make_float2(t16_lo(u.x), t16_hi(u.x));
        w[c][1] = make_float2(t16_lo(u.y), t16_hi(u.y));
      }
    }
    for (int j0 = 0; j0 < total; j0 += 32) {
      if (j0 > 0) load_list(cur, b, n, j0, x, tok, a);
      const int cnt = min(32, total - j0);
      for (int k0 = 0; k0 < cnt; k0 += kNarrowBatch) {
        if (j0 + k0 > 0) {
#pragma unroll
          for (int k = 0; k < kNarrowBatch; ++k) {
            const int tk = __shfl_sync(0xFFFFFFFFu, tok, (k0 + k) & 31);
            if (k0 + k < cnt) load_seed_row<NC>(gs_t + 1LL * tk * d, lane, d, q[k]);
          }
        }
        float dot[kNarrowBatch];
#pragma unroll
        for (int k = 0; k < kNarrowBatch; ++k) {
          const float2 ak = f2_all(__shfl_sync(0xFFFFFFFFu, a, (k0 + k) & 31));
          float2 dot2 = f2_all(0.f);
          if (k0 + k < cnt) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              if (c + 1 < NC || c * 128 + lane * 4 < d) {
                const float2 gv[2] = {make_float2(t16_lo(q[k][c].x), t16_hi(q[k][c].x)), make_float2(t16_lo(q[k][c].y), t16_hi(q[k][c].y))};
#pragma unroll
                for (int z = 0; z < 2; ++z) {
                  g[c][z] = f2_fma(ak, gv[z], g[c][z]);
                  dot2 = f2_fma(gv[z], w[c][z], dot2);
                }
              }
            }
          }
          dot[k] = dot2.x + dot2.y;
        }
        if (p.grad_a != nullptr) {
          const float sdot = warp_sum_many<kNarrowBatch>(dot, lane);
          const int k = k0 + warp_sum_slot<kNarrowBatch>(lane);
          const int xk = __shfl_sync(0xFFFFFFFFu, x, k & 31);
          if (lane % (32 / kNarrowBatch) == 0 && k < cnt && sdot != 0.f) atomicAdd(&p.grad_a[xk], sdot * gsc);
        }
      }
    }
    const float* xrow = cur.r == 0 ? extra_row_ptr(p, col) : nullptr;
    const long long eo = elem_of(cur);
    float2 norm2 = f2_all(0.f);
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int e = c * 128 + lane * 4;
      if (c + 1 < NC || e < d) {
        const float4 m4 = *reinterpret_cast<const float4*>(m_s + e), v4 = *reinterpret_cast<const float4*>(v_s + e);
        float2 m[2] = {make_float2(m4.x, m4.y), make_float2(m4.z, m4.w)}, v[2] = {make_float2(v4.x, v4.y), make_float2(v4.z, v4.w)};
        float4 extra = make_float4(0.f, 0.f, 0.f, 0.f);
        if (xrow != nullptr) extra = __ldg(reinterpret_cast<const float4*>(xrow + e));
#pragma unroll
        for (int z = 0; z < 2; ++z) {
          float2 gq = f2_fma(f2_all(pc), w[c][z], f2_mul(g[c][z], f2_all(gsc)));
          if (xrow != nullptr) gq = f2_add(gq, z == 0 ? make_float2(extra.x, extra.y) : make_float2(extra.z, extra.w));
          adam2(w[c][z], m[z], v[z], f2_mul(gq, f2_all(sc.clip)), hr);
          if (!PT) norm2 = f2_fma(w[c][z], w[c][z], norm2);
        }
        const float wn[4] = {w[c][0].x, w[c][0].y, w[c][1].x, w[c][1].y};
        stbf<4, SR>(w_s + e, wn, p.h.sr_seed, (unsigned int)(unsigned long long)(p.row_start[cur.ti] * d + eo + e));
        if (PT) {  // norms of the stored (rounded) weights
          float wr[4];
          ldbf<4>(w_s + e, wr);
#pragma unroll
          for (int z = 0; z < 2; ++z) norm2 = f2_fma(make_float2(wr[2 * z], wr[2 * z + 1]), make_float2(wr[2 * z], wr[2 * z + 1]), norm2);
        }
        *reinterpret_cast<float4*>(m_s + e) = make_float4(m[0].x, m[0].y, m[1].x, m[1].y);
        *reinterpret_cast<float4*>(v_s + e) = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
      }
    }
    if (p.norm2_out != nullptr) {
      const float sn = warp_sum(norm2.x + norm2.y);
      if (lane == 0) atomicAdd(&p.norm2_out[col], sn);
    }
    fence_proxy_async();  // the row written above is read next by the bulk stores (async proxy)
    __syncwarp();
    if (lane == 0) {
      bulk_store_1d_hint(static_cast<t16*>(p.w[cur.ti]) + eo, stage, w_bytes, pol_stream);
      bulk_store_1d_hint(p.m[cur.ti] + eo, stage + w_bytes, mv_bytes, pol_stream);
      bulk_store_1d_hint(p.v[cur.ti] + eo, stage + w_bytes + mv_bytes, mv_bytes, pol_stream);
      bulk_commit();
      if (!kRefillLate) bulk_wait_read<0>();  // the stage is refilled
    }
    if (!kRefillLate) {
      RowAt far{cur.idx + kNarrowStages * stride, nxt.ti, 0, 0};
      place(far);
      issue_row(far, st);
    }
    cur = nxt; nxt = nn;
    b = b1; n = n1; b1 = b2; n1 = n2;
    x = x1; tok = tok1; a = a1; total = total1;
  }
  if (lane == 0) {
    bulk_wait_all();
    if (!ok) {
      // rows whose loads were issued but never consumed: give them a bounded chance to land
      for (uint32_t j = i; j < i + kNarrowStages && cur.idx + 1LL * (j - i) * stride < total_rows; ++j) {
        const long long start = clock64();
        while (!mbar_try_wait(&full[j % kNarrowStages], (j / kNarrowStages) & 1))
          if (clock64() - start > kWaitTimeoutCycles) break;
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && abort_s && status != nullptr) atomicCAS(status, STATUS_OK, STATUS_WAIT_TIMEOUT);
}

// Tied decoders (per_source / per_target): same structure without the register-resident entries.
// Work item = (feature of one decoder tensor, 256-element segment): one warp, 8 elements per lane, walking
// the feature's R rows with the next row's (w, m, v) already in flight while the current row is updated.
// Row r of tensor i (source layer i, or target layer i with per_target tying); its gradient is
//   grad_scale * sum over contributing (entry, target) pairs of  a' * gs[target][tok, :]  (+ pen_coef * w).
template <typename WT, bool NORM_ONLY>
__global__ void __launch_bounds__(256) decoder_rows_adam_kernel(const DecAdamParams p) {
  const int lane = threadIdx.x & 31;
  const long long warp_global = (blockIdx.x * 1LL * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = (gridDim.x * 1LL * blockDim.x) >> 5;
  const StepScales sc = read_step_ctl(p.ctl);
  if (sc.skip) return;
  const float gsc = p.h.grad_scale * (p.use_inv_scale ? sc.inv_scale : 1.f);
  float nsq = 0.f;
  const int nseg = (p.d + 255) / 256;
  const long long per_tensor = 1LL * p.F_pitch * nseg;
  const long long total_items = per_tensor * p.ntensors;
  const bool affine_grads = p.tying != 0 && p.grad_a != nullptr && (p.d_feat_offset != nullptr || p.d_feat_scale != nullptr);
  for (long long item = warp_global; item < total_items; item += nwarps) {
    const int ti = int(item / per_tensor);
    const long long rem = item - ti * per_tensor;
    const int f = int(rem / nseg);
    const int seg = int(rem - 1LL * f * nseg);
    const int R = p.rows[ti];
    const int e0 = seg * 256 + lane * 8;
    const bool act = e0 < p.d;
    const long long row0 = 1LL * f * R;
    WT* wbase = static_cast<WT*>(p.w[ti]) + row0 * p.d + e0;
    float* mbase = p.m[ti] + row0 * p.d + e0;
    float* vbase = p.v[ti] + row0 * p.d + e0;
    // contributing source layers of this tensor's rows
    const int s_lo = p.tying == 2 ? 0 : ti;
    const int s_hi = ti;
    // d/dw of the norm-weighted sparsity penalty: coefficient of feature (ti, f); with per-target tying
    // the row belongs to the norm of every source feature (s <= ti, f).
    float pc = 0.f;
    if (p.pen_coef) {
      if (p.tying == 2) { for (int s = 0; s <= ti; ++s) pc += p.pen_coef[s * p.F_pitch + f]; }
      else pc = p.pen_coef[ti * p.F_pitch + f];
    }
    const float* xrow = extra_row_ptr(p, ti * p.F_pitch + f);
    if (NORM_ONLY && xrow == nullptr) {
      bool any = false;
      for (int s = s_lo; s <= s_hi; ++s) any |= __ldg(p.feat_off + s * p.F_pitch + f + 1) > __ldg(p.feat_off + s * p.F_pitch + f);
      if (!any) continue;
    }
    RowRegs<WT> cur, nxt;
    if (act) { if (NORM_ONLY) cur.w.load(wbase); else cur.load(wbase, mbase, vbase); }
    float norm2 = 0.f;
    for (int r = 0; r < R; ++r) {
      if (act && r + 1 < R) {
        if (NORM_ONLY) nxt.w.load(wbase + 1LL * (r + 1) * p.d);
        else nxt.load(wbase + 1LL * (r + 1) * p.d, mbase + 1LL * (r + 1) * p.d, vbase + 1LL * (r + 1) * p.d);
      }
      const int t_fixed = p.tying == 0 ? ti + r : (p.tying == 2 ? ti : -1);
      float w[8], g[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) { g[i] = 0.f; w[i] = 0.f; }
      if (act) cur.w.get(w);
      for (int s = s_lo; s <= s_hi; ++s) {
        const int col = s * p.F_pitch + f;
        const int b = __ldg(p.feat_off + col), e = __ldg(p.feat_off + col + 1);
        for (int i = b; i < e; ++i) {
          int tok = __ldg(p.fcsr_tok + i);
          float a = __ldg(p.fcsr_val + i);
          check_token(tok, a, p.B, p.status, 209);
          const int t_begin = t_fixed >= 0 ? t_fixed : s;
          const int t_end = t_fixed >= 0 ? t_fixed : p.L - 1;
          float dot = 0.f;
          for (int t = t_begin; t <= t_end; ++t) {
            float av = a, dscale = 1.f, shifted = a;
            if (p.tying != 0 && a != 0.f) {
              if (p.feat_offset) av += p.feat_offset[1LL * t * p.F_pitch + f];
              shifted = av;
              if (p.feat_scale) { const float fsc = p.feat_scale[1LL * t * p.F_pitch + f]; av *= fsc; dscale = fsc; }
            }
            float dot_t = 0.f;
            if (act) {
              float gv[8];
              unpack8(__ldg(reinterpret_cast<const uint4*>(p.gs + (1LL * t * p.B + tok) * p.d + e0)), gv);
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                g[k] = fmaf(av, gv[k], g[k]);
                dot_t = fmaf(gv[k], w[k], dot_t);
              }
            }
            dot = fmaf(dot_t, dscale, dot);
            // gradients of the affine terms of target t: d/d offset = scale * (gs_t . w), d/d scale = (a + offset) * (gs_t . w)
            if (affine_grads && a != 0.f) {
              const float ds = warp_sum(dot_t) * gsc;
              if (lane == 0 && ds != 0.f) {
                if (p.d_feat_offset != nullptr) atomicAdd(&p.d_feat_offset[1LL * t * p.F_pitch + f], ds * dscale);
                if (p.d_feat_scale != nullptr) atomicAdd(&p.d_feat_scale[1LL * t * p.F_pitch + f], ds * shifted);
              }
            }
          }
          if (p.grad_a != nullptr) {
            dot = warp_sum(dot);
            if (lane == 0 && dot != 0.f) atomicAdd(&p.grad_a[i], dot * gsc);
          }
        }
      }
      if (act) {
#pragma unroll
        for (int k = 0; k < 8; ++k) g[k] = fmaf(pc, w[k], g[k] * gsc);
        if (r == 0 && xrow != nullptr) {
          float dg0[8];
          load8f(xrow + e0, dg0);
#pragma unroll
          for (int k = 0; k < 8; ++k) g[k] += dg0[k];
        }
        if (NORM_ONLY) {
#pragma unroll
          for (int k = 0; k < 8; ++k) nsq = fmaf(g[k], g[k], nsq);
          cur = nxt;
          continue;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) g[k] *= sc.clip;
        float m[8], v[8];
        f4x2_to8(cur.m0, cur.m1, m);
        f4x2_to8(cur.v0, cur.v1, v);
        adam_update8(w, m, v, g, p.h);
        WT* wrow = wbase + 1LL * r * p.d;
        stream_store8f(mbase + 1LL * r * p.d, m);
        stream_store8f(vbase + 1LL * r * p.d, v);
        if (sizeof(WT) == 2) {
          t16 bq[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            bq[k] = to_bf16(w[k], p.h.sr_seed, (unsigned long long)((p.row_start[ti] + row0 + r) * p.d + e0 + k));
            const float wr = t16_to_float(bq[k]);  // norms are taken of the stored (rounded) weights
            norm2 = fmaf(wr, wr, norm2);
          }
          __stcs(reinterpret_cast<uint4*>(wrow), *reinterpret_cast<const uint4*>(bq));
        } else {
          stream_store8f(reinterpret_cast<float*>(wrow), w);
#pragma unroll
          for (int k = 0; k < 8; ++k) norm2 = fmaf(w[k], w[k], norm2);
        }
      }
      cur = nxt;
    }
    if (!NORM_ONLY && p.norm2_out != nullptr) {
      norm2 = warp_sum(norm2);
      if (lane == 0) atomicAdd(&p.norm2_out[ti * p.F_pitch + f], norm2);
    }
  }
  if (NORM_ONLY) block_add(nsq, p.norm_sq_out);
}

// ------------------------------------------------------------------ encoder rows
struct EncAdamParams {
  void* w;            // [L, F_pitch, d]
  float* m;
  float* v;
  void* bias;         // [L, F_pitch] (same dtype as w), updated here too
  float* bias_m;
  float* bias_v;
  int L, B, d, F_pitch;
  const int* feat_off;
  const int* fcsr_tok;
  const float* delta;           // [nnz] dL/d(pre-activation) per CSR slot (already scaled)
  const t16* x;       // [L, B, d] layer inputs
  const float* dense_grad;      // optional [L, F_pitch, d] fp32 gradient added to the sparse one (e.g. pre-activation loss)
  const float* dense_bias_grad; // optional [L, F_pitch]
  const int* extra_idx;         // optional compact extras (auxiliary loss): extra_idx[row] = row of extra_rows / extra_bias, or -1
  const float* extra_rows;      // [n_extra, d]
  const float* extra_bias;      // [n_extra]
  const float* ctl;             // optional step control block
  float* norm_sq_out;           // norm-only pass
  int norm_only;                // bias kernel: 1 = only add the squared bias gradients to norm_sq_out
  int* status;                  // see DecAdamParams
  AdamHyper h;                  // grad_scale applies to the sparse part
};
__device__ __forceinline__ int enc_extra_index(const EncAdamParams& p, long long row) {
  return p.extra_idx != nullptr ? __ldg(p.extra_idx + row) : -1;
}

template <typename WT, bool NORM_ONLY>
__global__ void __launch_bounds__(256) encoder_rows_adam_kernel(const EncAdamParams p) {
  const int lane = threadIdx.x & 31;
  const long long warp_global = (blockIdx.x * 1LL * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = (gridDim.x * 1LL * blockDim.x) >> 5;
  const StepScales sc = read_step_ctl(p.ctl);
  if (sc.skip) return;
  float nsq = 0.f;
  const int nseg = (p.d + 255) / 256;
  const long long total_items = 1LL * p.L * p.F_pitch * nseg;
  for (long long item = warp_global; item < total_items; item += nwarps) {
    const long long row = item / nseg;
    const int seg = int(item - row * nseg);
    const int l = int(row / p.F_pitch);
    const int e0 = seg * 256 + lane * 8;
    const bool act = e0 < p.d;
    const int b = __ldg(p.feat_off + row), e = __ldg(p.feat_off + row + 1);
    const int xi = enc_extra_index(p, row);
    if (NORM_ONLY && e == b && xi < 0 && p.dense_grad == nullptr) continue;
    WT* wrow = static_cast<WT*>(p.w) + row * p.d + e0;
    float* mrow = p.m + row * p.d + e0;
    float* vrow = p.v + row * p.d + e0;
    WVec<WT> wq;
    float4 m0, m1, v0, v1;
    if (act && !NORM_ONLY) {
      wq.load(wrow);
      m0 = __ldcs(reinterpret_cast<const float4*>(mrow)); m1 = __ldcs(reinterpret_cast<const float4*>(mrow) + 1);
      v0 = __ldcs(reinterpret_cast<const float4*>(vrow)); v1 = __ldcs(reinterpret_cast<const float4*>(vrow) + 1);
    }
    if (act) {
      float w[8], g[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) g[i] = 0.f;
      for (int i = b; i < e; ++i) {
        int tok = __ldg(p.fcsr_tok + i);
        float dl = __ldg(p.delta + i), xv[8];
        check_token(tok, dl, p.B, p.status, 210);
        unpack8(__ldg(reinterpret_cast<const uint4*>(p.x + (1LL * l * p.B + tok) * p.d + e0)), xv);
#pragma unroll
        for (int k = 0; k < 8; ++k) g[k] = fmaf(dl, xv[k], g[k]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) g[k] *= p.h.grad_scale;
      if (p.dense_grad) {
        float dg[8];
        load8f(p.dense_grad + row * p.d + e0, dg);
#pragma unroll
        for (int k = 0; k < 8; ++k) g[k] += dg[k];
      }
      if (xi >= 0) {
        float dg[8];
        load8f(p.extra_rows + 1LL * xi * p.d + e0, dg);
#pragma unroll
        for (int k = 0; k < 8; ++k) g[k] += dg[k];
      }
      if (NORM_ONLY) {
#pragma unroll
        for (int k = 0; k < 8; ++k) nsq = fmaf(g[k], g[k], nsq);
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) g[k] *= sc.clip;
        float m[8], v[8];
        wq.get(w);
        f4x2_to8(m0, m1, m);
        f4x2_to8(v0, v1, v);
        adam_update8(w, m, v, g, p.h);
        stream_store8f(mrow, m);
        stream_store8f(vrow, v);
        store_w8<WT>(wrow, w, p.h.sr_seed, (unsigned long long)(row * p.d + e0));
      }
    }
    if (seg == 0 && lane == 0 && p.bias != nullptr) {
      float gb = 0.f;
      for (int i = b; i < e; ++i) gb += p.delta[i];
      gb *= p.h.grad_scale;
      if (p.dense_bias_grad) gb += p.dense_bias_grad[row];
      if (xi >= 0 && p.extra_bias != nullptr) gb += p.extra_bias[xi];
      if (NORM_ONLY) { nsq = fmaf(gb, gb, nsq); continue; }
      gb *= sc.clip;
      WT* bp = static_cast<WT*>(p.bias) + row;
      float wv = sizeof(WT) == 2 ? t16_to_float(*reinterpret_cast<t16*>(bp)) : *reinterpret_cast<float*>(bp);
      float mm = p.bias_m[row], vv = p.bias_v[row];
      if (p.h.decoupled) wv *= (1.f - p.h.lr * p.h.weight_decay);
      else gb = fmaf(p.h.weight_decay, wv, gb);
      mm = fmaf(p.h.beta1, mm, (1.f - p.h.beta1) * gb);
      vv = fmaf(p.h.beta2, vv, (1.f - p.h.beta2) * gb * gb);
      wv -= (p.h.lr / p.h.bc1) * (mm / (sqrtf(vv) * rsqrtf(p.h.bc2) + p.h.eps));
      p.bias_m[row] = mm; p.bias_v[row] = vv;
      if (sizeof(WT) == 2) *reinterpret_cast<t16*>(bp) = to_bf16(wv, p.h.sr_seed, 0x9000000000ULL + row);
      else *reinterpret_cast<float*>(bp) = wv;
    }
  }
  if (NORM_ONLY) block_add(nsq, p.norm_sq_out);
}

// Encoder bias update on its own (used with the bulk-copy row pipeline, which handles the weight rows).
template <typename WT>
__global__ void __launch_bounds__(256) encoder_bias_adam_kernel(const EncAdamParams p) {
  if (chain_wait()) return;
  chain_release();
  const long long rows = 1LL * p.L * p.F_pitch;
  const StepScales sc = read_step_ctl(p.ctl);
  if (sc.skip) return;
  float nsq = 0.f;
  for (long long row = blockIdx.x * 1LL * blockDim.x + threadIdx.x; row < rows; row += 1LL * gridDim.x * blockDim.x) {
    const int b = __ldg(p.feat_off + row), e = __ldg(p.feat_off + row + 1);
    float gb = 0.f;
    for (int i = b; i < e; ++i) gb += p.delta[i];
    gb *= p.h.grad_scale;
    if (p.dense_bias_grad) gb += p.dense_bias_grad[row];
    const int xi = enc_extra_index(p, row);
    if (xi >= 0 && p.extra_bias != nullptr) gb += p.extra_bias[xi];
    if (p.norm_only) { nsq = fmaf(gb, gb, nsq); continue; }
    gb *= sc.clip;
    WT* bp = static_cast<WT*>(p.bias) + row;
    float wv = sizeof(WT) == 2 ? t16_to_float(*reinterpret_cast<t16*>(bp)) : *reinterpret_cast<float*>(bp);
    float mm = p.bias_m[row], vv = p.bias_v[row];
    if (p.h.decoupled) wv *= (1.f - p.h.lr * p.h.weight_decay);
    else gb = fmaf(p.h.weight_decay, wv, gb);
    mm = fmaf(p.h.beta1, mm, (1.f - p.h.beta1) * gb);
    vv = fmaf(p.h.beta2, vv, (1.f - p.h.beta2) * gb * gb);
    wv -= (p.h.lr / p.h.bc1) * (mm / (sqrtf(vv) * rsqrtf(p.h.bc2) + p.h.eps));
    p.bias_m[row] = mm; p.bias_v[row] = vv;
    if (sizeof(WT) == 2) *reinterpret_cast<t16*>(bp) = to_bf16(wv, p.h.sr_seed, 0x9000000000ULL + row);
    else *reinterpret_cast<float*>(bp) = wv;
  }
  if (p.norm_only) block_add(nsq, p.norm_sq_out);
}

// ------------------------------------------------------------------ dense Adam for the small tensors
// `ctl` (optional): skip flag and clip coefficient; `seed_scaled`: the gradient carries the loss scale (times 1 / scale);
// `norm_weight` > 0: norm-only pass, norm_weight * sum g^2 is added to ctl[SC_GRAD_NORM_SQ] and nothing is updated.
template <typename WT>
__global__ void __launch_bounds__(256) dense_adam_kernel(WT* __restrict__ w, float* __restrict__ m, float* __restrict__ v,
                                                           const float* __restrict__ grad, long long n, AdamHyper h,
                                                           float* __restrict__ ctl, int seed_scaled, float norm_weight) {
  if (chain_wait()) return;
  chain_release();
  const StepScales sc = read_step_ctl(ctl);
  if (sc.skip) return;
  const float gmul = h.grad_scale * (seed_scaled ? sc.inv_scale : 1.f);
  if (norm_weight > 0.f) {
    float nsq = 0.f;
    for (long long i = blockIdx.x * 1LL * blockDim.x + threadIdx.x; i < n; i += 1LL * gridDim.x * blockDim.x) {
      const float g = grad[i] * gmul;
      nsq = fmaf(g, g, nsq);
    }
    block_add(nsq * norm_weight, ctl != nullptr ? ctl + SC_GRAD_NORM_SQ : nullptr);
    return;
  }
  for (long long i = blockIdx.x * 1LL * blockDim.x + threadIdx.x; i < n; i += 1LL * gridDim.x * blockDim.x) {
    float wv = sizeof(WT) == 2 ? t16_to_float(*reinterpret_cast<const t16*>(w + i)) : *reinterpret_cast<const float*>(w + i);
    float g = grad[i] * gmul * sc.clip;
    if (h.decoupled) wv *= (1.f - h.lr * h.weight_decay);
    else g = fmaf(h.weight_decay, wv, g);
    const float mm = fmaf(h.beta1, m[i], (1.f - h.beta1) * g);
    const float vv = fmaf(h.beta2, v[i], (1.f - h.beta2) * g * g);
    wv -= (h.lr / h.bc1) * (mm / (sqrtf(vv) * rsqrtf(h.bc2) + h.eps));
    m[i] = mm; v[i] = vv;
    if (sizeof(WT) == 2) *reinterpret_cast<t16*>(w + i) = to_bf16(wv, h.sr_seed, 0xA000000000ULL + i);
    else *reinterpret_cast<float*>(w + i) = wv;
  }
}

// Squared decoder norms per feature: out[ti * F_pitch + f] = sum over the feature's rows and d of w^2.
template <typename WT>
__global__ void __launch_bounds__(256) decoder_norm2_kernel(const WT* __restrict__ w, float* __restrict__ out, int F, int R, int d) {
  if (chain_wait()) return;
  chain_release();
  const int lane = threadIdx.x & 31;
  const int warp_global = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const long long per_feat = 1LL * R * d;
  for (int f = warp_global; f < F; f += nwarps) {
    const WT* base = w + per_feat * f;
    float s = 0.f;
    for (long long i = lane * 8; i < per_feat; i += 256) {
      float x[8];
      load_w8<WT>(base + i, x);
#pragma unroll
      for (int k = 0; k < 8; ++k) s = fmaf(x[k], x[k], s);
    }
    s = warp_sum(s);
    if (lane == 0) out[f] = s;
  }
}

// Norm-weighted tanh sparsity penalty on the active entries (reference clt/training/losses.py:143-195):
//   penalty = lambda * sum tanh(c * n_f * a),  n_f = decoder norm of the entry's feature.
// One thread per feature column walks its CSR segment and writes
//   grad_a[i]   = lambda * c * n * sech^2(c n a)                (assignment: runs before the decoder pass)
//   pen_coef[f] = lambda * c * sum_i a_i sech^2(c n a_i) / n    (coefficient of w in dL/dw through the norm)
// and adds the penalty value to *penalty_out.
__global__ void __launch_bounds__(256) sparsity_penalty_kernel(const int* __restrict__ feat_off, const float* __restrict__ fcsr_val,
                                                                 const float* __restrict__ norm2, int ncols, float lambda, float c,
                                                                 float* __restrict__ grad_a, float* __restrict__ pen_coef,
                                                                 double* __restrict__ penalty_out) {
  if (chain_wait()) return;
  chain_release();
  float local = 0.f;
  for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < ncols; col += gridDim.x * blockDim.x) {
    const int b = feat_off[col], e = feat_off[col + 1];
    float coef = 0.f;
    if (e > b) {
      const float n = sqrtf(norm2[col]);
      float acc = 0.f;
      for (int i = b; i < e; ++i) {
        const float a = fcsr_val[i];
        const float th = tanhf(c * n * a);
        const float sech2 = 1.f - th * th;
        local += th;
        grad_a[i] = lambda * c * n * sech2;
        acc = fmaf(a, sech2, acc);
      }
      coef = n > 0.f ? lambda * c * acc / n : 0.f;
    }
    pen_coef[col] = coef;
  }
  __shared__ float red[8];
  local = warp_sum(local);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = local;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
    for (int w = 0; w < 8; ++w) tot += red[w];
    if (tot != 0.f) atomicAdd(penalty_out, double(tot) * double(lambda));
  }
}

}  // namespace clt

using namespace clt;

struct CltAdamHyper {
  float lr, beta1, beta2, eps, weight_decay, bc1, bc2;
  int decoupled;
  float grad_scale;
  unsigned int sr_seed;
  unsigned int moment_seed;
};
static AdamHyper to_hyper(const CltAdamHyper& c) {
  AdamHyper h;
  h.lr = c.lr; h.beta1 = c.beta1; h.beta2 = c.beta2; h.eps = c.eps; h.weight_decay = c.weight_decay;
  h.bc1 = c.bc1; h.bc2 = c.bc2; h.decoupled = c.decoupled; h.grad_scale = c.grad_scale; h.sr_seed = c.sr_seed; h.moment_seed = c.moment_seed;
  return h;
}

struct CltDecAdamArgs {
  void* w[32]; float* m[32]; float* v[32]; int rows[32];
  int ntensors, L, B, d, F_pitch, tying, weights_bf16;
  const int* feat_off; const int* fcsr_tok; const float* fcsr_val;
  const void* gs; float* grad_a; const float* pen_coef; float* norm2_out;
  const float* feat_offset; const float* feat_scale;
  const float* dgrad_row0;
  CltAdamHyper h;
  int* status;  // when given, untied decoders use the bulk-copy pipeline (its bounded waits report here)
  int moments_bf16;  // m / v are bf16 tensors (bulk pipeline with bf16 weights only)
  const int* extra_idx; const float* extra_rows;  // compact extra gradient rows (auxiliary loss), see DecAdamParams
  float* ctl;        // step control block (skip flag, 1 / loss scale, clip coefficient); may be null
  int norm_only;     // 1: gradient-norm pre-pass (adds to ctl[SC_GRAD_NORM_SQ], writes grad_a, updates nothing)
  float* d_feat_offset; float* d_feat_scale;  // tied decoders: gradient accumulators of the affine terms, see DecAdamParams
  long long n_entries;  // length of fcsr_tok / fcsr_val
};

// Launch geometry of the bulk-copy row pipeline (shared by the decoder and the encoder update).
static int bulk_rows_adam_geometry(int d, bool weights_bf16, bool moments_bf16, int* ept_out, int* gthreads_out, int* stage_bytes_out, size_t* smem_out,
                                   int* nstages_out = nullptr) {
  const int ept = d <= 1024 ? 4 : 8;  // elements per consumer thread: more, shorter threads where the row allows
  const int gthreads = ((d / ept + 31) / 32) * 32;
  const size_t wsz = weights_bf16 ? 2 : 4;
  const size_t msz = moments_bf16 ? 2 : 4;
  const int stage_bytes = int(((64 + size_t(d) * (wsz + 2 * msz + 2 * kAdamSlots)) + 127) / 128 * 128);
  const int nstages = stage_bytes > 24 * 1024 ? 3 : kAdamStages;
  if (nstages_out) *nstages_out = nstages;
  const size_t smem = size_t(nstages) * stage_bytes + sizeof(AdamBulkShared) + 256;
  *ept_out = ept; *gthreads_out = gthreads; *stage_bytes_out = stage_bytes; *smem_out = smem;
  return (d % 8 == 0 && gthreads <= 256 && smem <= 200 * 1024) ? 1 : 0;
}
static bool bulk_rows_adam_fits(int d, int weights_bf16) {
  int ept, gthreads, stage_bytes;
  size_t smem;
  return bulk_rows_adam_geometry(d, weights_bf16 != 0, false, &ept, &gthreads, &stage_bytes, &smem) != 0;
}
// Rows of up to 512 elements, one warp per row.
constexpr int kNarrowMaxWidth = 512;
static int launch_narrow_rows(const DecAdamParams& p, bool sr, int num_sms, int* status, cudaStream_t st, bool per_target) {
  const long long total = p.row_start[p.ntensors];
  const size_t smem = size_t(kNarrowWarps) * kNarrowStages * p.d * 10;
  // Rows above 256 elements with few entries leave more requests in flight than DRAM takes, and then it falls behind its own rate (one row of 512 per
  // feature, 0.6 entries each: 530 us with 16 warps per SM, 457 with 12; 2.6 entries: 476 and 506).  So many warps run as 6.55 TB/s need and 5 %
  // more, or all when that is nearly all of them: a warp takes 2.3 us for a row of up to 384 elements, 1.35 + 0.00258 d for a longer one, and 0.23 for
  // each of its entries (2.17 + 0.00125 d and 0.25 with the lists of several layers); a row moves 20 d bytes.  The kernel knows how many entries
  // there are, the host often only a bound.  us with all warps / with the rule (and of the form before two-wide arithmetic and late refills), rows of
  // 512, one per feature, by entries: 0.6 535 / 499 (548), 1 543 / 486 (542), 1.6 530 / 481 (471), 2 524 / 475 (474), 2.6 482 / 476 (492); of 448, 1
  // entry: 525 / 484 (484); of 384, six to one per feature, 0.6: 498 / 469 (472); per target, 0.1 per row: of 512 538 / 478 (538).
  const float ctas_per_us = 1.05f * 6.55e6f / float(20 * p.d * kNarrowWarps);
  const float row_us = per_target ? 2.17f + 0.00125f * float(p.d) : p.d <= 384 ? 2.3f : 1.35f + 0.00258f * float(p.d);
  const float ctas_empty = ctas_per_us * row_us, ctas_per_entry = ctas_per_us * (per_target ? 0.25f : 0.23f);
  auto launch = [&](auto kern) -> int {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return -4;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kNarrowWarps, smem) != cudaSuccess || per_sm < 1) return -4;
    long long grid = 1LL * num_sms * per_sm;
    const long long ctas = (total + kNarrowWarps - 1) / kNarrowWarps;
    if (grid > ctas) grid = ctas;
    launch_alone(kern, int(grid), 32 * kNarrowWarps, smem, st, p, total, ctas_empty, ctas_per_entry, status);
    return 0;
  };
  auto pick = [&](auto srv, auto ptv) -> int {
    constexpr bool S = decltype(srv)::value, T = decltype(ptv)::value;
    if (p.d <= 128) return launch(narrow_rows_adam_kernel<S, 1, T>);
    if (p.d <= 256) return launch(narrow_rows_adam_kernel<S, 2, T>);
    if (p.d <= 384) return launch(narrow_rows_adam_kernel<S, 3, T>);
    return launch(narrow_rows_adam_kernel<S, 4, T>);
  };
  using yes = std::true_type;
  using no = std::false_type;
  if (per_target) return sr ? pick(yes{}, yes{}) : pick(no{}, yes{});
  return sr ? pick(yes{}, no{}) : pick(no{}, no{});
}

// n_entries: length of the entry list (an upper bound where the number of active entries is not known to the host).
static int launch_rows_adam_bulk(const DecAdamParams& p, bool weights_bf16, bool sr, int num_sms, int* status, cudaStream_t st, long long n_entries,
                                 bool per_target = false) {
  int ept, gthreads, stage_bytes;
  size_t smem;
  const bool mb = p.moments_bf16 != 0;
  if (mb && !weights_bf16) return -1;  // bf16 moments go with bf16 weights
  int nstages = kAdamStages;
  if (!bulk_rows_adam_geometry(p.d, weights_bf16, mb, &ept, &gthreads, &stage_bytes, &smem, &nstages)) return -1;
  bool single_rows = true;
  for (int i = 0; i < p.ntensors; ++i) single_rows = single_rows && p.rows[i] == 1;
  // One warp per row up to 512 elements.  Both sweeps of a step, row pipeline -> one warp per row, us: tied Pythia-70m shape (one row of 512,
  // eight entries per feature) 1557 -> 925; per-target 6 x 16384 rows of 512, nine entries per row 565 -> 284, of 256 (12 per row, general
  // sweep) 484 -> 231; untied 6 x 12288 features of 512, 3.5 entries 760 -> 590, of 384 608 -> 501, 8 x 12288 of 256 774 -> 597, 8 x 16384 of
  // 128, six entries 1451 -> 777, one entry in sixteen 694 -> 472.  Where almost no feature has an entry, wide rows are a plain stream and
  // the deeper ring of the pipeline is ahead by 2 to 3 % (one entry in nine, rows of 512: 569 against 586; one in eight, tied: 348, 353).  With
  // several rows per feature that holds up to one entry per feature for the widest of them (6 x 5576 features of 512, six to one row each,
  // entries per feature: 0.5 208 / 221 us, 0.8 211 / 219, 1 215 / 215; of 480: 0.5 220 / 223, 0.7 225 / 222; of 448: 0.5 223 / 216).
  const long long features = 1LL * p.F_pitch * p.L;
  const bool idle_lists = !per_target && ((p.d > 384 && 2 * n_entries < features) || (p.d > 480 && !single_rows && n_entries < features));
  if (weights_bf16 && !mb && p.d <= kNarrowMaxWidth && !idle_lists) return launch_narrow_rows(p, sr, num_sms, status, st, per_target);
  auto launch = [&](auto kern) -> int {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return -4;
    // resident CTAs per SM from the runtime (shared memory, threads and registers together): a grid beyond them would run a
    // second wave of CTAs over features that were dealt out evenly
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, gthreads + 32, smem) != cudaSuccess || per_sm < 1) return -4;
    int bgrid = num_sms * (per_sm > 6 ? 6 : per_sm);
    int best = bgrid;
    if (per_target) {
      // one list of all rows: any grid splits it evenly.  The rows of a feature are F_pitch apart; take the grid, among a few at the
      // upper end, that sends the most of them to CTAs of their own
      const long long rows = 1LL * p.ntensors * p.F_pitch;
      if (bgrid > rows) bgrid = int(rows);
      int best_distinct = 0;
      for (int g = bgrid; g > bgrid - 8 && g >= 1 && best_distinct < p.ntensors; --g) {
        int distinct = 0;
        for (int i = 0; i < p.ntensors; ++i) {
          bool seen = false;
          for (int j = 0; j < i && !seen; ++j) seen = (1LL * (i - j) * p.F_pitch) % g == 0;
          distinct += seen ? 0 : 1;
        }
        if (distinct > best_distinct) { best_distinct = distinct; best = g; }
      }
    } else {
      // CTA b owns the features b, b + grid, ... of every tensor.  With one row per feature all resident slots run, also where they do
      // not divide the features: fewer CTAs keep fewer rows in flight (6 x 6144 rows of 592: 104 us on 683 CTAs, 88 on 740; 6 x 3072
      // of 768: 64 us on 512, 59 on 592).
      if (bgrid > p.F_pitch) bgrid = p.F_pitch;
      best = bgrid;
      // With several rows a feature is a longer piece of work: pick the grid (between three quarters of the resident slots and all of
      // them) that splits the features most evenly, so that no CTA still streams rows when the others are done.  2864 features of
      // 6 to 1 rows of 512, 888 slots: 111 us on the 716 CTAs that have four each, 118 on all.
      double best_waste = double((p.F_pitch + bgrid - 1) / bgrid) * bgrid / double(p.F_pitch) - 0.03;  // a few per cent do not pay for fewer CTAs
      for (int g = bgrid - 1; !single_rows && g >= (3 * bgrid) / 4 && g >= 1; --g) {
        const int per = (p.F_pitch + g - 1) / g;
        const double waste = double(per) * g / double(p.F_pitch);
        if (waste < best_waste - 1e-9) { best_waste = waste; best = g; }
      }
    }
    launch_alone(kern, best, gthreads + 32, smem, st, p, gthreads, stage_bytes, nstages, status);
    return 0;
  };
  // Registers against batches.  Four entries per batch take 72 registers, which costs rows of 392 to 608 elements a resident CTA per SM
  // (five for six up to 512, four for five above), and a list of a few entries beyond the staged ones fills no batch.  So the 64-register
  // form with batches of two runs where it has more resident CTAs and
  //  * there is one row per feature (encoder; tied decoders): 6 x 10520 rows of 440, one entry in four features 123 -> 119 us (152 with
  //    72 registers), eight per feature 246 -> 233 (274); 4 x 11312 rows of 592, one in four 112 -> 105 (133), eight 215 -> 203 (233).
  //    With sixteen per feature the batches of four are ahead again (6 x 1504 rows of 576: 119 -> 99 us against 88);
  //  * or untied decoders have at most three entries per feature on average: 6 x 2864 features 576 wide, one entry in four 126 -> 126
  //    us (129 with 72 registers), 2.7 per feature 162 -> 154 (162).
  // Above 1024 (eight elements per thread) one row per feature takes its entries one by one: 6 x 10520 rows of 1432, five per feature
  // 478 -> 469 us (488 with batches of four).  Between 1288 and 1408 three CTAs fit an SM with 80 registers and two with 96, and the
  // 80-register form without batches runs whatever the lists hold: 6 x 10520 rows of 1400, one entry in four features 298 -> 298 us
  // (355 with 96), untied rows of 6 x 4672 features 458 -> 460 (542), with eight entries per feature 1080 -> 1025 (1062).
  // The first figure of a pair is the sweep that waited twice per entry.  Encoder rows of 1032 to 1280 elements with fewer than three
  // entries stay 3 to 5 % above it (6 x 10520 rows of 1152: 295 -> 306 us), with five and more they are below.
  auto per_sm_of = [&](auto kern) -> int {
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return -1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, gthreads + 32, smem) != cudaSuccess) return -1;
    return n > 6 ? 6 : n;
  };
  const bool short_lists = gthreads <= 160 && (single_rows || n_entries <= 3LL * p.F_pitch * p.L);
  auto pick = [&](auto srv, auto wt, auto mt) -> int {
    constexpr bool S = decltype(srv)::value;
    using W = decltype(wt);
    using M = decltype(mt);
    if (ept == 8 && gthreads <= 224 && per_sm_of(decoder_rows_adam_bulk_kernel<W, S, 8, M, false, 1, true>) > per_sm_of(decoder_rows_adam_bulk_kernel<W, S, 8, M>))
      return launch(decoder_rows_adam_bulk_kernel<W, S, 8, M, false, 1, true>);
    if (ept == 8) return single_rows ? launch(decoder_rows_adam_bulk_kernel<W, S, 8, M, false, 1>) : launch(decoder_rows_adam_bulk_kernel<W, S, 8, M>);
    if (short_lists && per_sm_of(decoder_rows_adam_bulk_kernel<W, S, 4, M, false, 2, true>) > per_sm_of(decoder_rows_adam_bulk_kernel<W, S, 4, M>))
      return launch(decoder_rows_adam_bulk_kernel<W, S, 4, M, false, 2, true>);
    return launch(decoder_rows_adam_bulk_kernel<W, S, 4, M>);
  };
  using yes = std::true_type;
  using no = std::false_type;
  using bf = t16;
  if (per_target) {
    if (ept == 4) return sr ? launch(decoder_rows_adam_bulk_kernel<bf, true, 4, float, true>) : launch(decoder_rows_adam_bulk_kernel<bf, false, 4, float, true>);
    return sr ? launch(decoder_rows_adam_bulk_kernel<bf, true, 8, float, true>) : launch(decoder_rows_adam_bulk_kernel<bf, false, 8, float, true>);
  }
  if (mb) {
#if CLT_T16_IS_HALF
    return -6;  // bf16 moments go with bf16 weights
#else
    return sr ? pick(yes{}, bf{}, bf{}) : pick(no{}, bf{}, bf{});
#endif
  }
  if (!weights_bf16) return pick(no{}, float{}, float{});
  return sr ? pick(yes{}, bf{}, float{}) : pick(no{}, bf{}, float{});
}

extern "C" int CLT_FN(clt_decoder_rows_adam)(const CltDecAdamArgs* a, int num_sms, cudaStream_t st) {
  if (a->d % 8 != 0 || a->ntensors > kMaxLayersA) return -1;
  DecAdamParams p;
  long long acc = 0;
  for (int i = 0; i < kMaxLayersA; ++i) {
    p.w[i] = a->w[i]; p.m[i] = a->m[i]; p.v[i] = a->v[i]; p.rows[i] = a->rows[i];
    p.row_start[i] = acc;
    if (i < a->ntensors) acc += 1LL * a->F_pitch * a->rows[i];
  }
  p.row_start[kMaxLayersA] = acc;
  for (int i = a->ntensors; i <= kMaxLayersA; ++i) p.row_start[i] = acc;
  p.ntensors = a->ntensors; p.L = a->L; p.B = a->B; p.d = a->d; p.F_pitch = a->F_pitch; p.tying = a->tying;
  p.feat_off = a->feat_off; p.fcsr_tok = a->fcsr_tok; p.fcsr_val = a->fcsr_val;
  p.gs = static_cast<const t16*>(a->gs); p.grad_a = a->grad_a; p.pen_coef = a->pen_coef; p.norm2_out = a->norm2_out;
  p.feat_offset = a->feat_offset; p.feat_scale = a->feat_scale; p.dgrad_row0 = a->dgrad_row0; p.h = to_hyper(a->h);
  p.d_feat_offset = a->d_feat_offset; p.d_feat_scale = a->d_feat_scale;
  p.moments_bf16 = a->moments_bf16;
  p.extra_idx = a->extra_idx; p.extra_rows = a->extra_rows; p.ctl = a->ctl; p.use_inv_scale = 1;
  p.norm_sq_out = a->ctl != nullptr ? a->ctl + SC_GRAD_NORM_SQ : nullptr;
  p.status = a->status;
  if (a->moments_bf16 && !(a->tying == 0 && a->status != nullptr && a->weights_bf16)) return -6;  // only the bulk pipeline handles bf16 moments
  if (acc == 0) return 0;
  bool single_rows = true;
  for (int i = 0; i < a->ntensors; ++i) single_rows = single_rows && a->rows[i] == 1;
  const int grid = num_sms * 8;
  if (a->norm_only) {
    if (a->ctl == nullptr) return -1;
    if (a->tying == 0) {
      if (a->weights_bf16) launch_rows_norm<t16, true>(p, num_sms, st);
      else launch_rows_norm<float, true>(p, num_sms, st);
    } else if (a->weights_bf16) {
      launch_alone(decoder_rows_adam_kernel<t16, true>, grid, 256, 0, st, p);
    } else {
      launch_alone(decoder_rows_adam_kernel<float, true>, grid, 256, 0, st, p);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
  }
  if (a->tying == 0 && a->status != nullptr && bulk_rows_adam_fits(a->d, a->weights_bf16) && acc * a->d < (1LL << 62)) {
    const int rc = launch_rows_adam_bulk(p, a->weights_bf16 != 0, a->h.sr_seed != 0, num_sms, a->status, st, a->n_entries);
    if (rc != 0) return rc;
  } else if (a->tying == 2 && a->status != nullptr && a->weights_bf16 && a->L <= 32 && a->ntensors == a->L && single_rows &&
             a->feat_offset == nullptr && a->feat_scale == nullptr && a->d_feat_offset == nullptr && a->d_feat_scale == nullptr &&
             bulk_rows_adam_fits(a->d, a->weights_bf16)) {
    // Per-target tied rows without affine terms and without gradients of such terms, which neither form of the row update forms: one
    // warp per row up to 512 elements, the row pipeline above, whose consumers gather the entries.
    const int rc = launch_rows_adam_bulk(p, true, a->h.sr_seed != 0, num_sms, a->status, st, a->n_entries, true);
    if (rc != 0) return rc;
  } else if (a->tying == 0) {
    const bool sr = a->h.sr_seed != 0;
    if (a->weights_bf16) {
      if (sr) launch_alone(decoder_rows_adam_untied_kernel<t16, true>, grid, 256, 0, st, p);
      else launch_alone(decoder_rows_adam_untied_kernel<t16, false>, grid, 256, 0, st, p);
    } else {
      launch_alone(decoder_rows_adam_untied_kernel<float, false>, grid, 256, 0, st, p);
    }
  } else if (a->weights_bf16) {
    launch_alone(decoder_rows_adam_kernel<t16, false>, grid, 256, 0, st, p);
  } else {
    launch_alone(decoder_rows_adam_kernel<float, false>, grid, 256, 0, st, p);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

struct CltEncAdamArgs {
  void* w; float* m; float* v; void* bias; float* bias_m; float* bias_v;
  int L, B, d, F_pitch, weights_bf16;
  const int* feat_off; const int* fcsr_tok; const float* delta; const void* x;
  const float* dense_grad; const float* dense_bias_grad;
  CltAdamHyper h;
  int* status;  // when given, the weight rows go through the bulk-copy pipeline
  int moments_bf16;
  const int* extra_idx; const float* extra_rows; const float* extra_bias;  // compact extras, see EncAdamParams
  float* ctl;
  int norm_only;
  long long n_entries;  // length of fcsr_tok / delta
};

extern "C" int CLT_FN(clt_encoder_rows_adam)(const CltEncAdamArgs* a, int num_sms, cudaStream_t st) {
  if (a->d % 8 != 0) return -1;
  EncAdamParams p;
  p.w = a->w; p.m = a->m; p.v = a->v; p.bias = a->bias; p.bias_m = a->bias_m; p.bias_v = a->bias_v;
  p.L = a->L; p.B = a->B; p.d = a->d; p.F_pitch = a->F_pitch;
  p.feat_off = a->feat_off; p.fcsr_tok = a->fcsr_tok; p.delta = a->delta; p.x = static_cast<const t16*>(a->x);
  p.dense_grad = a->dense_grad; p.dense_bias_grad = a->dense_bias_grad; p.h = to_hyper(a->h);
  p.extra_idx = a->extra_idx; p.extra_rows = a->extra_rows; p.extra_bias = a->extra_bias; p.ctl = a->ctl;
  p.norm_sq_out = a->ctl != nullptr ? a->ctl + SC_GRAD_NORM_SQ : nullptr; p.norm_only = a->norm_only;
  p.status = a->status;
  const int grid = num_sms * 8, bgrid = int((1LL * a->L * a->F_pitch + 255) / 256);
  // the encoder as the one-row-per-feature case of the decoder's kernels: layer l is "tensor" l with R = 1, the layer inputs play the gradient
  // seed and delta the activation
  DecAdamParams q;
  const size_t wsz = a->weights_bf16 ? 2 : 4;
  const long long per_layer = 1LL * a->F_pitch * a->d;
  for (int i = 0; i < kMaxLayersA; ++i) {
    const int l = i < a->L ? i : 0;
    q.w[i] = static_cast<char*>(a->w) + size_t(l) * per_layer * wsz;
    const size_t msz = a->moments_bf16 ? 2 : 4;
    q.m[i] = reinterpret_cast<float*>(reinterpret_cast<char*>(a->m) + size_t(l) * per_layer * msz);
    q.v[i] = reinterpret_cast<float*>(reinterpret_cast<char*>(a->v) + size_t(l) * per_layer * msz);
    q.rows[i] = 1;
    q.row_start[i] = 1LL * (i < a->L ? i : a->L) * a->F_pitch;
  }
  q.row_start[kMaxLayersA] = 1LL * a->L * a->F_pitch;
  q.ntensors = a->L; q.L = a->L; q.B = a->B; q.d = a->d; q.F_pitch = a->F_pitch; q.tying = 0;
  q.feat_off = a->feat_off; q.fcsr_tok = a->fcsr_tok; q.fcsr_val = a->delta; q.gs = p.x;
  q.grad_a = nullptr; q.pen_coef = nullptr; q.norm2_out = nullptr; q.feat_offset = nullptr; q.feat_scale = nullptr;
  q.d_feat_offset = nullptr; q.d_feat_scale = nullptr;
  q.dgrad_row0 = a->dense_grad; q.h = p.h;
  q.moments_bf16 = a->moments_bf16;
  q.extra_idx = a->dense_grad == nullptr ? a->extra_idx : nullptr; q.extra_rows = a->extra_rows;
  q.ctl = a->ctl; q.use_inv_scale = 0; q.norm_sq_out = p.norm_sq_out;
  q.status = a->status;
  if (a->norm_only) {
    if (a->ctl == nullptr) return -1;
    if (a->L <= kMaxLayersA && (a->dense_grad == nullptr || a->extra_idx == nullptr) && 1LL * a->L * a->F_pitch < INT_MAX) {
      launch_rows_norm<t16, false>(q, num_sms, st);  // the weights' type does not matter: they are not read
      if (p.bias != nullptr) launch_chained(encoder_bias_adam_kernel<t16>, bgrid, 256, 0, st, p);
    } else if (a->weights_bf16) {  // two kinds of extra rows
      launch_alone(encoder_rows_adam_kernel<t16, true>, grid, 256, 0, st, p);
    } else {
      launch_alone(encoder_rows_adam_kernel<float, true>, grid, 256, 0, st, p);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
  }
  if (a->status != nullptr && a->L <= kMaxLayersA && bulk_rows_adam_fits(a->d, a->weights_bf16)) {
    if (a->dense_grad != nullptr && a->extra_idx != nullptr) return -7;  // the row pipeline takes one kind of extra rows
    const int rc = launch_rows_adam_bulk(q, a->weights_bf16 != 0, a->h.sr_seed != 0, num_sms, a->status, st, a->n_entries);
    if (rc != 0) return rc;
    if (p.bias != nullptr) {
      if (a->weights_bf16) launch_chained(encoder_bias_adam_kernel<t16>, bgrid, 256, 0, st, p);
      else launch_chained(encoder_bias_adam_kernel<float>, bgrid, 256, 0, st, p);
    }
  } else if (a->moments_bf16) {
    return -6;  // only the bulk pipeline handles bf16 moments
  } else if (a->weights_bf16) launch_alone(encoder_rows_adam_kernel<t16, false>, grid, 256, 0, st, p);
  else launch_alone(encoder_rows_adam_kernel<float, false>, grid, 256, 0, st, p);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

extern "C" int CLT_FN(clt_dense_adam)(void* w, float* m, float* v, const float* grad, long long n, int weights_bf16, const CltAdamHyper* h,
                                      float* ctl, int seed_scaled, float norm_weight, cudaStream_t st) {
  if (n <= 0) return 0;
  const int grid = int((n + 255) / 256 < 1184 ? (n + 255) / 256 : 1184);
  if (weights_bf16) launch_chained(dense_adam_kernel<t16>, grid, 256, 0, st, static_cast<t16*>(w), m, v, grad, n, to_hyper(*h), ctl, seed_scaled, norm_weight);
  else launch_chained(dense_adam_kernel<float>, grid, 256, 0, st, static_cast<float*>(w), m, v, grad, n, to_hyper(*h), ctl, seed_scaled, norm_weight);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

extern "C" int CLT_FN(clt_decoder_norm2)(const void* w, float* out, int F, int R, int d, int weights_bf16, cudaStream_t st) {
  if ((1LL * R * d) % 8 != 0) return -1;
  const int grid = (F + 7) / 8 < 1184 ? (F + 7) / 8 : 1184;
  if (grid == 0) return 0;
  if (weights_bf16) launch_chained(decoder_norm2_kernel<t16>, grid, 256, 0, st, static_cast<const t16*>(w), out, F, R, d);
  else launch_chained(decoder_norm2_kernel<float>, grid, 256, 0, st, static_cast<const float*>(w), out, F, R, d);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

#if !CLT_T16_IS_HALF
extern "C" int clt_sparsity_penalty(const int* feat_off, const float* fcsr_val, const float* norm2, int ncols, float lambda, float c,
                                    float* grad_a, float* pen_coef, double* penalty_out, cudaStream_t st) {
  if (ncols <= 0) return 0;
  const int grid = (ncols + 255) / 256 < 1184 ? (ncols + 255) / 256 : 1184;
  launch_chained(sparsity_penalty_kernel, grid, 256, 0, st, feat_off, fcsr_val, norm2, ncols, lambda, c, grad_a, pen_coef, penalty_out);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
#endif
