// Sparse cross-layer decode and the reconstruction loss (sm_100a).
//
// The reference decodes with one dense GEMM per (source, target) pair over activations that are more
// than 99 % zeros, each followed by an all-reduce (clt/models/decoder.py:289-295, clt/models/parallel.py:363-383),
// and then computes the MSE in separate passes (clt/training/losses.py:76-90).  Here a warp takes one token and one target
// layer, walks the token's active (layer, feature, value) entries, reads the decoder row of each (feature-major layout
// [F, R, d]) and accumulates the reconstruction in registers.
// The epilogue either writes the fp32 partial reconstruction (tensor parallel: summed across ranks before
// the loss) or, single rank, finishes in place: bias, optional dense addend (skip connection), residual,
// per-layer squared-error sum in de-normalised units and the bf16 gradient seed  gs = (y_hat - y) * sigma^2.
#include "common.cuh"

namespace clt {

constexpr int kMaxLayers = 32;

struct DecodeParams {
  const t16* w[kMaxLayers];  // decoder tensor i: [F_pitch, rows_i, d]
  int rows[kMaxLayers];                // rows per feature of tensor i
  int L, B, d;
  int col_pitch;                       // entries encode column = layer * col_pitch + feature
  int tying;                           // 0 untied, 1 per_source, 2 per_target
  const int* tok_off;                  // [B+1]
  const int* tcsr_col;                 // (layer << 24) | feature
  const float* tcsr_val;
  const float* feat_offset;            // optional [L, col_pitch]  (tied decoders)
  const float* feat_scale;             // optional [L, col_pitch]
  // outputs / epilogue
  float* yhat_partial;                 // mode 0: [L, B, d] fp32 partial sums
  const float* bias_sum;               // mode 1: [L, d] summed decoder biases per target
  const float* addend;                 // mode 1: optional [L, B, d] fp32 (skip term)
  const t16* target;         // mode 1: [L, B, d]
  const float* sigma;                  // mode 1: optional [L, d] de-normalisation scale of the targets
  t16* gs;                   // mode 1: [L, B, d] (y_hat - y) * sigma^2
  float* yhat_out;                     // mode 1: optional [L, B, d] fp32 reconstruction
  double* sq_err;                      // mode 1: [L] sum of ((y_hat - y) * sigma)^2
  // mode 2 (tensor parallel): partial sums are pushed into the staging area of the rank that owns the token.
  // stage_peers[o] = rank o's staging area [world][L][rows_per_rank][d] fp32; this rank writes slot `rank`.
  float* stage_peers[8];
  int rows_per_rank, rank, world;
  int mode;
  // optional step control block: the gradient seed is multiplied by ctl[SC_LOSS_SCALE] (fp16 loss scaling) and a
  // seed that leaves the 16-bit range or is NaN raises ctl[SC_FOUND_INF] (the step is then skipped)
  float* ctl;
  int rows_limit;  // > 0: only the first rows_limit target rows of a feature are decoded (auxiliary loss: same layer only)
  int* dbg_status; // status words for the index checks of the debug build (may be null)
};

__device__ __forceinline__ void fma8(float (&acc)[8], float a, const uint4& v) {
  const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    acc[2 * j] = fmaf(a, t16_lo(u[j]), acc[2 * j]);
    acc[2 * j + 1] = fmaf(a, t16_hi(u[j]), acc[2 * j + 1]);
  }
}

// Output of one (token, target, 8-element slice): partial sums (mode 0), peer push (mode 2) or the finished
// loss epilogue (mode 1).  Returns the slice's squared error (mode 1, else 0); the callers sum it in registers and
// across the warp: a shared-memory atomic per thread on the L per-target sums costs tens of thousands of cycles
// per token (32 lanes on one address, floating-point add as a compare-and-swap loop).
__device__ __forceinline__ float decode_epilogue(const DecodeParams& p, int tok, int t, int e0, const float (&a)[8], float loss_scale) {
  const long long off = (1LL * t * p.B + tok) * p.d + e0;
  if (p.mode == 0) {
    float4* dst = reinterpret_cast<float4*>(p.yhat_partial + off);
    dst[0] = make_float4(a[0], a[1], a[2], a[3]);
    dst[1] = make_float4(a[4], a[5], a[6], a[7]);
    return 0.f;
  } else if (p.mode == 2) {
    // reduce-scatter by push: peer store into the owner's slot for this rank (NVLink posted writes)
    const int owner = tok / p.rows_per_rank;
    const int lrow = tok - owner * p.rows_per_rank;
    if (!clt_in_bounds(owner, p.world, p.dbg_status, 105)) return 0.f;  // peer rank derived from the token index
    float4* dst = reinterpret_cast<float4*>(p.stage_peers[owner] + ((1LL * p.rank * p.L + t) * p.rows_per_rank + lrow) * p.d + e0);
    dst[0] = make_float4(a[0], a[1], a[2], a[3]);
    dst[1] = make_float4(a[4], a[5], a[6], a[7]);
    return 0.f;
  } else {
    if (p.target == nullptr) {  // inference: the reconstruction is all there is to write
      float v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[i] = a[i] + p.bias_sum[1LL * t * p.d + e0 + i];
        if (p.addend) v[i] += p.addend[off + i];
      }
      float4* dst = reinterpret_cast<float4*>(p.yhat_out + off);
      dst[0] = make_float4(v[0], v[1], v[2], v[3]);
      dst[1] = make_float4(v[4], v[5], v[6], v[7]);
      return 0.f;
    }
    float y[8], out[8];
    const uint4 tv = *reinterpret_cast<const uint4*>(p.target + off);
    const uint32_t u[4] = {tv.x, tv.y, tv.z, tv.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { y[2 * i] = t16_lo(u[i]); y[2 * i + 1] = t16_hi(u[i]); }
    float sq = 0.f;
    bool bad = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float v = a[i] + p.bias_sum[1LL * t * p.d + e0 + i];
      if (p.addend) v += p.addend[off + i];
      const float sg = p.sigma ? p.sigma[1LL * t * p.d + e0 + i] : 1.f;
      out[i] = v;
      const float r = (v - y[i]) * sg;
      sq = fmaf(r, r, sq);
      y[i] = r * sg * loss_scale;  // gradient seed
      bad |= !(fabsf(y[i]) <= kT16Max);
    }
    if (bad && p.ctl != nullptr) atomicOr(reinterpret_cast<int*>(p.ctl) + SC_FOUND_INF, 1);
    uint4 gv;
    gv.x = pack_t16x2(y[0], y[1]); gv.y = pack_t16x2(y[2], y[3]);
    gv.z = pack_t16x2(y[4], y[5]); gv.w = pack_t16x2(y[6], y[7]);
    *reinterpret_cast<uint4*>(p.gs + off) = gv;
    if (p.yhat_out) {
      float4* dst = reinterpret_cast<float4*>(p.yhat_out + off);
      dst[0] = make_float4(out[0], out[1], out[2], out[3]);
      dst[1] = make_float4(out[4], out[5], out[6], out[7]);
    }
    return sq;
  }
}

// ------------------------------------------------------------------ gather kernels
// Both kernels below give a warp one token and one slice of d_model and let it walk the token's active entries with
// plain 16-byte loads, a few decoder rows at a time; the sums stay in registers.  The work is a read of n_entries * targets
// decoder rows, several times the size of the touched weights, by chains of dependent loads (list, row): bound by how many warps
// are in a chain at any moment, and with thousands of tokens by DRAM (GPT-2 shape, 4096 tokens, k = 200: 7.0 GB in 1.39 ms, 5.2 TB/s,
// where 2.9 GB are touched; all warps are at the same target and the entries of a token are sorted by (layer, feature), so that L2
// serves the rest).
//
// Lists differ in length (a global selection gives the tokens between none and six times the average), and warps that share a CTA
// wait for the longest of their lists, so a walk of three or four vectors per lane is a CTA of one warp.  GPT-2 shape, 4096
// tokens, BatchTopK k = 200: 1977 us with seven tokens per CTA, 1400 with one; k = 32: 555 and 379 (a CTA per token behind a ring of
// bulk copies, the form before: 2013 and 475).  With equally long lists it is 268 and 238 us (2048 tokens, top-k of 64).  Narrow
// rows are over sooner, and what a CTA costs by itself (its launch, its addition to the error sum, 1.5 ns together) shows: 12 x 6208
// (token, target) pairs of 136 elements without an entry 116 us with one warp per CTA, 46 with eight, although 8000 tokens of 64 entries
// (6 x 256) take 289 with one, 305 with two, 322 with four and 348 with eight.  So two vectors per lane go two warps to a CTA, one
// vector four.
// Two walk configurations, by rows in flight against warps per SM: four rows and 16 warps (three or four vectors per lane) finish a
// short list soonest, two rows and 28 (three vectors: 72 registers) or 20 (four) keep more tokens on the chip.  GPT-2 shape, k = 32: 1024 tokens
// 155 us with four rows against 186 with two, 2048 252 against 264, 3072 324 against 315, 4096 402 against 375; k = 200: 2048 870
// against 895, 4096 1503 against 1399; equal lists of 64, 2048 tokens: 262 against 238.  So the line is at 2048 tokens.
// The entries of a token are split over the eight warps of a CTA while there are few (token, target) warps: long lists then
// decide.  340 tokens, k = 32: 70 us split, 122 not; 512 tokens (6144 warps): 102 and 127; 1024: 181 and 155.  Equal lists gain less
// from it: top-k of 32, 128 tokens 31 us split against 25 not, 340 tokens 67 against 38; of 200, 128 tokens 76 against 86.
constexpr int kSplitWarps = 8;
__host__ __device__ constexpr int walk_warps(int nv) { return nv == 1 ? 4 : (nv == 2 ? 2 : 1); }
constexpr long long kRunningMinWarps = 1024;   // below: too few warps, the (token, target) split has L times as many
constexpr int kFullMinTokens = 2048;
constexpr long long kSplitBelowWarps = 4096;

__device__ __forceinline__ int decode_token(const DecodeParams& p, int i) {
  // Tensor-parallel push: rank r starts with the tokens owned by rank r + 1, so that at any moment the ranks
  // store into different owners instead of all into the same one.
  return p.mode == 2 ? int((i + 1LL * ((p.rank + 1) % p.world) * p.rows_per_rank) % p.B) : i;
}

// acc += a_j * row_j over the entries whose bits are set in `mask` (lane i of the warp holds entry i of the batch: its
// activation and the address of its decoder row).  The order of the additions is the order of the entries.
template <int NV, int R>
__device__ __forceinline__ void gather_rows(uint32_t mask, float a, const t16* row, const int (&e0)[NV], const bool (&act)[NV], float (&acc)[NV][8]) {
  const uint32_t row_lo = uint32_t(reinterpret_cast<uintptr_t>(row)), row_hi = uint32_t(reinterpret_cast<uintptr_t>(row) >> 32);
  while (mask != 0u) {
    uint4 q[R][NV];
    float w[R];
    bool have[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      have[k] = mask != 0u;
      const int src = have[k] ? __ffs(mask) - 1 : 0;
      mask &= mask - 1u;
      w[k] = __shfl_sync(0xFFFFFFFFu, a, src);
      const uintptr_t r = (uintptr_t(__shfl_sync(0xFFFFFFFFu, row_hi, src)) << 32) | uintptr_t(__shfl_sync(0xFFFFFFFFu, row_lo, src));
#pragma unroll
      for (int v = 0; v < NV; ++v)
        if (have[k] && act[v]) q[k][v] = __ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const t16*>(r) + e0[v]));
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
      if (have[k]) {
#pragma unroll
        for (int v = 0; v < NV; ++v)
          if (act[v]) fma8(acc[v], w[k], q[k][v]);
      }
    }
  }
}

// One warp (SPLIT = 1) or one CTA of kSplitWarps warps (few tokens, the entries of a token are dealt to the warps and the
// partial sums meet in shared memory) per (token, target, column chunk of NV * 256).  Every tying mode: `tying` only decides which
// row an entry reads.  blockIdx.y counts the targets from the last one down: the longest lists come first, so that the short ones
// fill the tail.
template <int NV, int SPLIT, bool FULL = false>
__global__ void __launch_bounds__(32 * (SPLIT > 1 ? SPLIT : walk_warps(NV)), SPLIT > 1 ? (NV >= 3 ? 2 : (NV == 2 ? 3 : 4))
                                                                                        : (FULL ? (NV == 4 ? 20 : 28) : (NV >= 3 ? 16 : (NV == 2 ? 24 : 32))) / walk_warps(NV))
    decode_walk_kernel(const DecodeParams p) {
  constexpr int kWarps = SPLIT > 1 ? SPLIT : walk_warps(NV);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = p.L - 1 - int(blockIdx.y);
  const int slot = SPLIT > 1 ? int(blockIdx.x) : int(blockIdx.x) * kWarps + warp;
  const int d = p.d;
  const float loss_scale = p.ctl != nullptr ? p.ctl[SC_LOSS_SCALE] : 1.f;
  float sq = 0.f;
  if (slot < p.B) {
    const int tok = decode_token(p, slot);
    int e0[NV];
    bool act[NV];
    float acc[NV][8];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      e0[v] = ((int(blockIdx.z) * NV + v) * 32 + lane) * 8;
      act[v] = e0[v] < d;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[v][i] = 0.f;
    }
    const int span = p.rows_limit > 0 ? p.rows_limit : kMaxLayers;  // targets s .. s + span - 1 of a source layer s
    const int b = __ldg(p.tok_off + tok), e = __ldg(p.tok_off + tok + 1);
    int seen = 0;  // SPLIT: entries dealt so far
    for (int i0 = b; i0 < e; i0 += 32) {
      const int i = i0 + lane;
      const int col = i < e ? __ldg(p.tcsr_col + i) : 0;  // packed by the CSR build: (layer << 24) | feature
      float a = i < e ? __ldg(p.tcsr_val + i) : 0.f;
      const int s = col >> 24, f = col & 0xFFFFFF;
      bool use = a != 0.f;
      if (use && (!clt_in_bounds(s, p.L, p.dbg_status, 101) || !clt_in_bounds(f, p.col_pitch, p.dbg_status, 102))) use = false;
      use = use && s <= t && t - s < span;
      const t16* row = nullptr;
      if (use) {
        const int wi = p.tying == 2 ? t : s;
        row = p.w[wi] + (p.tying == 0 ? 1LL * f * p.rows[s] + (t - s) : 1LL * f) * d;
        if (p.tying != 0) {
          if (p.feat_offset) a += p.feat_offset[1LL * t * p.col_pitch + f];
          if (p.feat_scale) a *= p.feat_scale[1LL * t * p.col_pitch + f];
        }
      }
      uint32_t mask = __ballot_sync(0xFFFFFFFFu, use);
      if (SPLIT > 1) {
        const int rank = seen + __popc(mask & ((1u << lane) - 1u));
        seen += __popc(mask);
        mask = __ballot_sync(0xFFFFFFFFu, use && rank % SPLIT == warp);
      }
      gather_rows<NV, FULL ? 2 : 4>(mask, a, row, e0, act, acc);
    }
    if (SPLIT == 1) {
#pragma unroll
      for (int v = 0; v < NV; ++v)
        if (act[v]) sq += decode_epilogue(p, tok, t, e0[v], acc[v], loss_scale);
    } else {
      __shared__ __align__(16) float part[SPLIT > 1 ? SPLIT : 1][SPLIT > 1 ? NV * 256 : 4];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        float4* dst = reinterpret_cast<float4*>(&part[warp][(v * 32 + lane) * 8]);
        dst[0] = make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
        dst[1] = make_float4(acc[v][4], acc[v][5], acc[v][6], acc[v][7]);
      }
      __syncthreads();
      for (int c = threadIdx.x; c < NV * 32; c += blockDim.x) {  // one 8-element slice per thread
        const int ec = (int(blockIdx.z) * NV * 32 + c) * 8;
        if (ec >= d) continue;
        float out[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) out[i] = 0.f;
#pragma unroll
        for (int w = 0; w < SPLIT; ++w) {
#pragma unroll
          for (int i = 0; i < 8; ++i) out[i] += part[w][c * 8 + i];
        }
        sq += decode_epilogue(p, tok, t, ec, out, loss_scale);
      }
    }
  }
  if (p.mode == 1) {
    // one global atomic per CTA: all warps of the CTA work on the same target
    sq = warp_sum(sq);
    if (kWarps > 1) {
      __shared__ float red_s[kWarps];
      if (lane == 0) red_s[warp] = sq;
      __syncthreads();
      sq = 0.f;
      for (int w = 0; w < kWarps; ++w) sq += red_s[w];
    }
    if (threadIdx.x == 0 && sq != 0.f && p.sq_err != nullptr) atomicAdd(&p.sq_err[t], double(sq));
  }
}

// Per-source tied decoders without affine terms: the row of feature (s, f) serves every target t >= s with the same weight,
// so the reconstruction of target t is the one of t - 1 plus the entries of layer t.  One warp per (token, column chunk)
// reads every row once and finishes a target whenever a layer's entries are in.  The list is scanned once per layer
// (coalesced, a few hundred bytes), so the entries of a token may come in any order (within a layer they are added in the
// order of the list: bit for bit the same sums take a sorted list).  One warp per CTA, as in the walk: tied Pythia-70m shape, 4096
// tokens, k = 200: 571 us with eight, 518 with one.
template <int NV>
__global__ void __launch_bounds__(32, NV >= 2 ? 16 : 24) decode_running_kernel(const DecodeParams p) {
  const int lane = threadIdx.x & 31;
  const int d = p.d;
  const float loss_scale = p.ctl != nullptr ? p.ctl[SC_LOSS_SCALE] : 1.f;
  const int tok = decode_token(p, int(blockIdx.x));
  int e0[NV];
  bool act[NV];
  float acc[NV][8];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    e0[v] = ((int(blockIdx.y) * NV + v) * 32 + lane) * 8;
    act[v] = e0[v] < d;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[v][i] = 0.f;
  }
  const int b = __ldg(p.tok_off + tok), e = __ldg(p.tok_off + tok + 1);
  float sq_t = 0.f;  // lane t: the sum of target t (at most 32 layers), one addition per CTA and target at the end
  for (int t = 0; t < p.L; ++t) {
    for (int i0 = b; i0 < e; i0 += 32) {
      const int i = i0 + lane;
      const int col = i < e ? __ldg(p.tcsr_col + i) : 0;
      const float a = i < e ? __ldg(p.tcsr_val + i) : 0.f;
      const int f = col & 0xFFFFFF;
      bool use = a != 0.f;
      if (use && (!clt_in_bounds(col >> 24, p.L, p.dbg_status, 103) || !clt_in_bounds(f, p.col_pitch, p.dbg_status, 104))) use = false;
      use = use && (col >> 24) == t;
      const uint32_t mask = __ballot_sync(0xFFFFFFFFu, use);
      if (mask != 0u) gather_rows<NV, 4>(mask, a, p.w[t] + 1LL * f * d, e0, act, acc);
    }
    float sq = 0.f;
#pragma unroll
    for (int v = 0; v < NV; ++v)
      if (act[v]) sq += decode_epilogue(p, tok, t, e0[v], acc[v], loss_scale);
    if (p.mode == 1) {
      sq = warp_sum(sq);
      if (lane == t) sq_t = sq;
    }
  }
  if (p.mode == 1 && sq_t != 0.f && p.sq_err != nullptr) atomicAdd(&p.sq_err[lane], double(sq_t));
}

// Epilogue for the tensor-parallel path, run after the partial reconstructions were summed across ranks:
// bias, addend, residual, loss sum and gradient seed for rows [row0, row0 + nrows) of every layer.
__global__ void __launch_bounds__(256) recon_epilogue_kernel(const float* __restrict__ yhat_sum, const float* __restrict__ bias_sum,
                                                               const float* __restrict__ addend, const t16* __restrict__ target,
                                                               const float* __restrict__ sigma, t16* __restrict__ gs,
                                                               float* __restrict__ yhat_out, double* __restrict__ sq_err, int L, int B,
                                                               int d, int row0, int nrows, float* __restrict__ ctl) {
  const int t = blockIdx.y;
  const float loss_scale = ctl != nullptr ? ctl[SC_LOSS_SCALE] : 1.f;
  bool bad = false;
  const int vec_per_row = d / 8;
  const long long nvec = 1LL * nrows * vec_per_row;
  float sq = 0.f;
  for (long long i = blockIdx.x * 1LL * blockDim.x + threadIdx.x; i < nvec; i += 1LL * gridDim.x * blockDim.x) {
    const int row = row0 + int(i / vec_per_row);
    const int e0 = int(i % vec_per_row) * 8;
    const long long off = (1LL * t * B + row) * d + e0;
    const float4 a0 = *reinterpret_cast<const float4*>(yhat_sum + off), a1 = *reinterpret_cast<const float4*>(yhat_sum + off + 4);
    float v[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
    const uint4 tv = *reinterpret_cast<const uint4*>(target + off);
    const uint32_t u[4] = {tv.x, tv.y, tv.z, tv.w};
    float g[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] += bias_sum[1LL * t * d + e0 + j];
      if (addend) v[j] += addend[off + j];
      const float y = (j & 1) ? t16_hi(u[j >> 1]) : t16_lo(u[j >> 1]);
      const float sg = sigma ? sigma[1LL * t * d + e0 + j] : 1.f;
      const float r = (v[j] - y) * sg;
      sq = fmaf(r, r, sq);
      g[j] = r * sg * loss_scale;
      bad |= !(fabsf(g[j]) <= kT16Max);
    }
    uint4 gv;
    gv.x = pack_t16x2(g[0], g[1]); gv.y = pack_t16x2(g[2], g[3]); gv.z = pack_t16x2(g[4], g[5]); gv.w = pack_t16x2(g[6], g[7]);
    *reinterpret_cast<uint4*>(gs + off) = gv;
    if (yhat_out) {
      float4* dst = reinterpret_cast<float4*>(yhat_out + off);
      dst[0] = make_float4(v[0], v[1], v[2], v[3]);
      dst[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
  }
  __shared__ float red[8];
  sq = warp_sum(sq);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
    for (int w = 0; w < (blockDim.x >> 5); ++w) tot += red[w];
    atomicAdd(&sq_err[t], double(tot));
  }
  if (bad && ctl != nullptr) atomicOr(reinterpret_cast<int*>(ctl) + SC_FOUND_INF, 1);
}

// Column sums of the gradient seed: out[t, :] += sum_b gs[t, b, :]  (decoder-bias gradient up to a constant).
// blockDim = (d / 8 rounded up to 32, up to 8 row lanes): a thread owns 8 adjacent columns (one 16-byte load per row), the
// threadIdx.y lanes of a block walk the block's row range, shared memory folds them, one atomic per column and block.
__global__ void __launch_bounds__(1024) gs_colsum_kernel(const t16* __restrict__ gs, float* __restrict__ out, int B, int d,
                                                          int rows_per_block) {
  const int t = blockIdx.z;
  const int c0 = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  const int r0 = blockIdx.y * rows_per_block, r1 = min(B, r0 + rows_per_block);
  float s[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) s[j] = 0.f;
  if (c0 < d) {
    for (int r = r0 + threadIdx.y; r < r1; r += blockDim.y) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(gs + (1LL * t * B + r) * d + c0));
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) { s[2 * j] += t16_lo(u[j]); s[2 * j + 1] += t16_hi(u[j]); }
    }
  }
  __shared__ float red[1024][9];
  const int lin = threadIdx.y * blockDim.x + threadIdx.x;
#pragma unroll
  for (int j = 0; j < 8; ++j) red[lin][j] = s[j];
  __syncthreads();
  if (threadIdx.y == 0 && c0 < d) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float tot = 0.f;
      for (int y = 0; y < int(blockDim.y); ++y) tot += red[y * blockDim.x + threadIdx.x][j];
      atomicAdd(&out[1LL * t * d + c0 + j], tot);
    }
  }
}

// Suffix sums of the gradient seed over the layers: out[s] = sum over t >= s of gs[t]  (per_source tied decoders:
// the threshold-gradient GEMM of source layer s needs the seed of all its targets added up).  fp32 accumulation.
__global__ void __launch_bounds__(256) gs_suffix_sum_kernel(const t16* __restrict__ gs, t16* __restrict__ out, int L, long long per_layer) {
  for (long long i = (blockIdx.x * 1LL * blockDim.x + threadIdx.x) * 8; i < per_layer; i += 1LL * gridDim.x * blockDim.x * 8) {
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (int t = L - 1; t >= 0; --t) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(gs + t * per_layer + i));
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) { acc[2 * j] += t16_lo(u[j]); acc[2 * j + 1] += t16_hi(u[j]); }
      uint4 o;
      o.x = pack_t16x2(acc[0], acc[1]); o.y = pack_t16x2(acc[2], acc[3]); o.z = pack_t16x2(acc[4], acc[5]); o.w = pack_t16x2(acc[6], acc[7]);
      *reinterpret_cast<uint4*>(out + t * per_layer + i) = o;
    }
  }
}

}  // namespace clt

using namespace clt;

struct CltDecodeArgs {
  const void* w[32];
  int rows[32];
  int L, B, d, col_pitch, tying;
  const int* tok_off; const int* tcsr_col; const float* tcsr_val;
  const float* feat_offset; const float* feat_scale;
  float* yhat_partial;
  const float* bias_sum; const float* addend; const void* target; const float* sigma;
  void* gs; float* yhat_out; double* sq_err;
  void* stage_peers[8];
  int rows_per_rank, rank, world;
  int mode;
  int* status;  // may be null; the index checks of the debug build report here
  float* ctl;   // optional step control block (loss scale in, found-inf flag out)
  int rows_limit;
};

extern "C" int CLT_FN(clt_sparse_decode)(const CltDecodeArgs* a, cudaStream_t st) {
  if (a->d % 8 != 0 || a->L > kMaxLayers || a->d > 2048) return -1;
  DecodeParams p;
  for (int i = 0; i < kMaxLayers; ++i) { p.w[i] = static_cast<const t16*>(a->w[i]); p.rows[i] = a->rows[i]; }
  p.L = a->L; p.B = a->B; p.d = a->d; p.col_pitch = a->col_pitch; p.tying = a->tying;
  p.tok_off = a->tok_off; p.tcsr_col = a->tcsr_col; p.tcsr_val = a->tcsr_val;
  p.feat_offset = a->feat_offset; p.feat_scale = a->feat_scale;
  p.yhat_partial = a->yhat_partial; p.bias_sum = a->bias_sum; p.addend = a->addend;
  p.target = static_cast<const t16*>(a->target); p.sigma = a->sigma;
  p.gs = static_cast<t16*>(a->gs); p.yhat_out = a->yhat_out; p.sq_err = a->sq_err; p.mode = a->mode;
  for (int i = 0; i < 8; ++i) p.stage_peers[i] = static_cast<float*>(a->stage_peers[i]);
  p.rows_per_rank = a->rows_per_rank; p.rank = a->rank; p.world = a->world;
  p.ctl = a->ctl; p.rows_limit = a->rows_limit; p.dbg_status = a->status;
  if (a->B <= 0 || a->L <= 0) return 0;
  // 16-byte vectors per lane: the whole row up to d_model 1024 (a warp then reads an entry's row in one go), half of it above
  const int chunks = a->d > 1024 ? 2 : 1;
  const int nv = (a->d / 8 + 32 * chunks - 1) / (32 * chunks);
  const bool plain_tied = a->tying == 1 && a->feat_offset == nullptr && a->feat_scale == nullptr && a->rows_limit <= 0;
  auto pick = [&](auto k1, auto k2, auto k3, auto k4, bool split) {
    auto go = [&](auto kern, int warps) { kern<<<dim3(split ? a->B : (a->B + warps - 1) / warps, a->L, chunks), 32 * (split ? kSplitWarps : warps), 0, st>>>(p); };
    if (nv <= 1) go(k1, walk_warps(1));
    else if (nv == 2) go(k2, walk_warps(2));
    else if (nv == 3) go(k3, walk_warps(3));
    else go(k4, walk_warps(4));
  };
  const int run_chunks = (a->d + 511) / 512;  // at most two vectors per lane: the sums stay live across the epilogues of all targets
  if (plain_tied && 1LL * a->B * run_chunks >= kRunningMinWarps) {
    const dim3 grid(a->B, run_chunks);
    if (a->d <= 256) decode_running_kernel<1><<<grid, 32, 0, st>>>(p);
    else decode_running_kernel<2><<<grid, 32, 0, st>>>(p);
  } else if (1LL * a->B * a->L * chunks < kSplitBelowWarps) {
    pick(decode_walk_kernel<1, kSplitWarps>, decode_walk_kernel<2, kSplitWarps>, decode_walk_kernel<3, kSplitWarps>, decode_walk_kernel<4, kSplitWarps>, true);
  } else if (nv >= 3 && a->B >= kFullMinTokens) {
    const dim3 grid(a->B, a->L, chunks);
    if (nv == 3) decode_walk_kernel<3, 1, true><<<grid, 32, 0, st>>>(p);
    else decode_walk_kernel<4, 1, true><<<grid, 32, 0, st>>>(p);
  } else {
    pick(decode_walk_kernel<1, 1>, decode_walk_kernel<2, 1>, decode_walk_kernel<3, 1>, decode_walk_kernel<4, 1>, false);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

extern "C" int CLT_FN(clt_recon_epilogue)(const float* yhat_sum, const float* bias_sum, const float* addend, const void* target,
                                  const float* sigma, void* gs, float* yhat_out, double* sq_err, int L, int B, int d, int row0,
                                  int nrows, float* ctl, cudaStream_t st) {
  if (d % 8 != 0) return -1;
  if (nrows <= 0) return 0;
  dim3 grid(148, L);
  recon_epilogue_kernel<<<grid, 256, 0, st>>>(yhat_sum, bias_sum, addend, static_cast<const t16*>(target), sigma,
                                              static_cast<t16*>(gs), yhat_out, sq_err, L, B, d, row0, nrows, ctl);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

extern "C" int CLT_FN(clt_gs_colsum)(const void* gs, float* out, int L, int B, int d, cudaStream_t st) {
  if (d % 8 != 0) return -1;
  const int tx = d / 8 >= 128 ? 128 : ((d / 8 + 31) / 32) * 32;
  const int ty = 1024 / tx < 8 ? 1024 / tx : 8;
  const int rpb = 128;
  dim3 grid((d / 8 + tx - 1) / tx, (B + rpb - 1) / rpb, L), block(tx, ty);
  gs_colsum_kernel<<<grid, block, 0, st>>>(static_cast<const t16*>(gs), out, B, d, rpb);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

extern "C" int CLT_FN(clt_gs_suffix_sum)(const void* gs, void* out, int L, int B, int d, cudaStream_t st) {
  const long long per_layer = 1LL * B * d;
  if (per_layer % 8 != 0) return -1;
  const long long nvec = per_layer / 8;
  const int grid = int(nvec / 256 + 1 < 1184 ? nvec / 256 + 1 : 1184);
  gs_suffix_sum_kernel<<<grid, 256, 0, st>>>(static_cast<const t16*>(gs), static_cast<t16*>(out), L, per_layer);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
