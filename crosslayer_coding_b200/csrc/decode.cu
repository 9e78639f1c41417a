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
  const int* order; // optional [B]: the token of slot i (modes 0 and 1)
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
// Both kernels below give a CTA one token and one slice of d_model; its warps share the token's active entries and gather the
// decoder rows with plain 16-byte loads, a few rows at a time; the sums stay in registers and meet in shared memory.  The work is a
// read of n_entries * targets decoder rows, several times the size of the touched weights, by chains of dependent loads (list, row).
//
// What bounds it: lists differ in length (a global selection gives the tokens between none and six times the average), so a warp
// per token leaves the chip to the longest lists of every target, and warps that start together drift apart in the feature order, so that
// L2 serves less.  Four warps per token: GPT-2 shape, 4096 tokens, BatchTopK k = 200, 1435 us with one warp and 1081 with four (8.2 GB of
// rows at 7.6 TB/s, of which DRAM gives about 6); 512 tokens, k = 32: 124 and 62; 1000 tokens of 16 x 2048, 242 entries: 1138 and 963; 4096
// tokens of 6 x 512, per-target tied, k = 64: 172 and 132.  Eight warps pay where there are too few CTAs to fill the chip
// (16 tokens 36 us with four, 22 with eight; 128 tokens of 200 entries 72 and 67; 256: 102 and 109).
// With so few that their slices of 256 columns are all on the chip at once (four CTAs of eight warps per SM), a CTA takes a slice and its warps eight
// rows at a time: three or four times the loads in flight, and the chain of a warp is half as long.  16 tokens of 12 x 768, 200 entries, 29.2 -> 21.5 us
// (lists of 100: 22.1 -> 15.4), 8 of 12 x 1024 14.4 -> 10.4, 140 of 1 x 1024 21.7 -> 14.9; near-empty lists 4.0 -> 4.3 and 5.2 -> 4.6.  Beyond one round of
// CTAs it wins only with long lists (64 tokens of 12 x 768, 200 entries 70 -> 59, six entries 12 -> 14; 64 of 12 x 1024 32 and 33); short equal lists (8 to
// 24 entries 0.4 us), rows of up to 512 (12 x 24 tokens, 50 entries: 6.2 and 6.7) and above 1024 (60 tokens of 16 x 2048: 64 and 76) stay whole.
// Rows in flight against warps per SM: four rows and 20 warps (three vectors per lane) or 16 (four) are best up to some thousands of CTAs
// (2048 tokens, k = 200: 588 us against 605 with two rows and 28 warps), two rows and more warps beyond (4096 tokens 1164 and 1081; 1000 tokens
// of 16 x 2048 1003 and 963).  There the tokens are also taken in the order of their list lengths, longest first: warps that
// run together then end together and stay closer in the feature order (1081 -> 1032 us, 963 -> 913).
// Short lists over many tokens: the latency of a CTA by itself (offsets, list, rows, sums, targets) is what counts, and two warps keep
// twice the tokens on the chip.  4096 tokens, entries per token on average: 8 139 us with two and 174 with four, 16 182 and 213, 25 (one
// eighth of the features) 191 and 224, 32 266 and 287, 66 436 and 437, 100 629 and 606.  Only the caller knows the average without a
// host synchronisation (its k); a threshold selection does not, and counts as long.
// Equally long lists (a per-token selection) gain nothing from four warps while they are short: 2048 tokens of 6 x 768, k = 64, 82 us with one warp
// and 100 with four, 3536 of 4 x 856, k = 24, 71 and 104, 776 of 5 x 520, k = 24, 19 and 28.  Long ones (k = 200) do not either where the chip is full of
// wide rows: 12 x 768, 1024 tokens 227 and 223, 2048 305 and 404, 8192 1128 and 1327; 16 x 2048, 128 tokens 125 and 127, 512 313 and 350; 8 x
// 512, 4096 tokens of 8192 features 312 and 313, of 32768 385 and 444 (k = 400: 555 and 516, 665 and 722).  Running sums, k = 200: 1024 tokens of 6 x 512 76 and 57,
// 4096 141 and 159, of 8 x 256 74 and 122; k = 400, 4096 tokens of 12 x 768 509 and 482, of 8 x 256 117 and 165.  Their order by length
// says nothing: it is not formed.
// Near-empty lists of a length that the caller does not know take four warps too: 12 x 768, 4096 tokens without an entry 114 us, where two warps take 92
// and one 84.  Whoever knows that lists are short says so (the expected length).
// Narrow rows: what a CTA costs by itself shows, above all its addition to the error sum (1.5 ns, all CTAs of a target on one
// address): 12 x 6208 (token, target) pairs of 136 elements without an entry take 116 us with one token per CTA, 60 with two.  So with many
// tokens one vector per lane goes two tokens and two warps each to a CTA (4096 tokens of 6 x 256, k = 64: 93 us either way).
// Per-source tied, running sums: 4 warps 340 us, 1 warp 610 (8192 tokens of 6 x 512, k = 200), sorted by length 295; short or equally long
// lists are the other way round (5809 tokens of 4 x 600, k = 19: 122 us with four, 77 with one; 2048 of 6 x 512, equal lists of 64: 37, 33).  Lists
// of a length that the caller does not know: many tokens keep the chip busy with two warps each, whatever the length (four / two warps: 8192
// tokens of 6 x 512 without an entry 122 / 83 us, of 12 entries 140 / 97, of 200 288 / 235; 4096 of 12 x 768 198 / 126, 216 / 138, 349 / 259;
// below the line 4096 of 6 x 512, 48 entries on average but few in most lists, 99 / 130).
constexpr long long kRunningMinWarps = 1024;   // tokens x chunks; below, the (token, target) split has L times as many CTAs
constexpr long long kEightWarpsBelow = 2048;   // CTAs
constexpr long long kSliceCtasPerSm = 4;       // CTAs of 256 columns
constexpr long long kManyCtas = 28672;         // CTAs
constexpr long long kPairNarrowFrom = 24576;   // (token, target) pairs
constexpr int kRunningOrderFrom = 4096;        // tokens
constexpr int kShortBelow = 64;                // entries per token on average
constexpr long long kShortFrom = 16384;        // CTAs
constexpr int kRunningOneWarpBelow = 32;         // entries per token on average
constexpr long long kRunningTwoWarpsFrom = 8192; // tokens x chunks
constexpr int kOneWarpBelow = 128;               // entries of every token; above, by one_warp_lists
constexpr int kOneWarpMediumBelow = 256;        // entries of every token
constexpr int kOneWarpRunningFrom = 2048;        // tokens
constexpr long long kOneWarpWalkFrom = 16384, kOneWarpWideWalkFrom = 8192;  // CTAs; the second: four vectors per lane

__device__ __forceinline__ int decode_token(const DecodeParams& p, int i) {
  // Tensor-parallel push: rank r starts with the tokens owned by rank r + 1, so that at any moment the ranks
  // store into different owners instead of all into the same one.
  if (p.mode != 2) return p.order != nullptr ? __ldg(p.order + i) : i;
  return int((i + 1LL * ((p.rank + 1) % p.world) * p.rows_per_rank) % p.B);
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

// A warp's sums in shared memory, and the total of the SPLIT warps of a token for one 8-element slice (added in the order of
// the warps: equal lists give equal bits).  A slice is two 16-byte vectors that lie a row of 16-byte vectors apart, so that the lanes of a
// warp touch consecutive vectors.
template <int NV>
__device__ __forceinline__ void put_partial(float* sums, const float (&acc)[NV][8], int lane) {
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    float4* dst = reinterpret_cast<float4*>(sums) + v * 32 + lane;
    dst[0] = make_float4(acc[v][0], acc[v][1], acc[v][2], acc[v][3]);
    dst[NV * 32] = make_float4(acc[v][4], acc[v][5], acc[v][6], acc[v][7]);
  }
}
template <int NV, int SPLIT>
__device__ __forceinline__ void sum_partials(const float (*sums)[NV * 256], int slice, float (&out)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) out[i] = 0.f;
#pragma unroll
  for (int w = 0; w < SPLIT; ++w) {
    const float4* src = reinterpret_cast<const float4*>(sums[w]) + slice;
    const float4 lo = src[0], hi = src[NV * 32];
    out[0] += lo.x; out[1] += lo.y; out[2] += lo.z; out[3] += lo.w;
    out[4] += hi.x; out[5] += hi.y; out[6] += hi.z; out[7] += hi.w;
  }
}

// acc += the entries first, first + stride, first + 2 * stride, ... below `end` of a token's list for target t, 32 at a time (a lane
// holds one; the next 32 are loaded while the rows of these are gathered).
template <int NV, int R>
__device__ __forceinline__ void walk_list(const DecodeParams& p, int t, int first, int stride, int end, int lane, const int (&e0)[NV], const bool (&act)[NV],
                                          float (&acc)[NV][8]) {
  const int span = p.rows_limit > 0 ? p.rows_limit : kMaxLayers;  // targets s .. s + span - 1 of a source layer s
  int i = first + lane * stride;
  int col = i < end ? __ldg(p.tcsr_col + i) : 0;  // packed by the CSR build: (layer << 24) | feature
  float a = i < end ? __ldg(p.tcsr_val + i) : 0.f;
  for (int i0 = first; i0 < end; i0 += 32 * stride) {
    i += 32 * stride;
    const int col_next = i < end ? __ldg(p.tcsr_col + i) : 0;
    const float a_next = i < end ? __ldg(p.tcsr_val + i) : 0.f;
    const int s = col >> 24, f = col & 0xFFFFFF;
    bool use = a != 0.f;
    if (use && (!clt_in_bounds(s, p.L, p.dbg_status, 101) || !clt_in_bounds(f, p.col_pitch, p.dbg_status, 102))) use = false;
    use = use && s <= t && t - s < span;
    const t16* row = nullptr;
    if (use) {
      const int wi = p.tying == 2 ? t : s;
      row = p.w[wi] + (p.tying == 0 ? 1LL * f * p.rows[s] + (t - s) : 1LL * f) * p.d;
      if (p.tying != 0) {
        if (p.feat_offset) a += p.feat_offset[1LL * t * p.col_pitch + f];
        if (p.feat_scale) a *= p.feat_scale[1LL * t * p.col_pitch + f];
      }
    }
    gather_rows<NV, R>(__ballot_sync(0xFFFFFFFFu, use), a, row, e0, act, acc);
    col = col_next;
    a = a_next;
  }
}

// One CTA works on TOK tokens of one target layer and one column chunk of NV * 256, SPLIT warps to a token: the token's entries are
// dealt to them one by one and the partial sums meet in shared memory.  Every tying mode: `tying` only decides which row an entry reads.
// blockIdx.y counts the targets from the last one down: the longest lists come first, so that the short ones fill the tail.
template <int NV, int TOK, int SPLIT, int R, int WARPS_PER_SM>
__global__ void __launch_bounds__(32 * TOK * SPLIT, WARPS_PER_SM / (TOK * SPLIT)) decode_walk_kernel(const DecodeParams p) {
  if (chain_wait()) return;
  chain_release();
  constexpr int kWarps = TOK * SPLIT;
  __shared__ __align__(16) float sums[kWarps][NV * 256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = p.L - 1 - int(blockIdx.y);
  const int slot = int(blockIdx.x) * TOK + warp / SPLIT, part = warp % SPLIT;
  const int d = p.d;
  const float loss_scale = p.ctl != nullptr ? p.ctl[SC_LOSS_SCALE] : 1.f;
  int b = 0, e = 0;
  if (slot < p.B) {
    const int tok = decode_token(p, slot);
    b = __ldg(p.tok_off + tok);
    e = __ldg(p.tok_off + tok + 1);
    if (p.target != nullptr) {  // the epilogue's row on its way while the entries are gathered
      const int e0 = (int(blockIdx.z) * NV * 32 + part * 32 + lane) * 8;
      if (e0 < d && part < NV) asm volatile("prefetch.global.L1 [%0];" ::"l"(p.target + (1LL * t * p.B + tok) * d + e0));
    }
    int off[NV];
    bool act[NV];
    float acc[NV][8];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      off[v] = ((int(blockIdx.z) * NV + v) * 32 + lane) * 8;
      act[v] = off[v] < d;
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[v][i] = 0.f;
    }
    walk_list<NV, R>(p, t, b + part, SPLIT, e, lane, off, act, acc);
    if (TOK > 1 || e > b) put_partial<NV>(sums[warp], acc, lane);
  }
  const bool empty = TOK == 1 && e == b;  // nothing was gathered: no sums to wait for
  if (!empty) __syncthreads();
  float sq = 0.f;
  for (int c = threadIdx.x; c < TOK * NV * 32; c += 32 * kWarps) {  // one 8-element slice per thread
    const int g = TOK > 1 ? c / (NV * 32) : 0, cv = TOK > 1 ? c % (NV * 32) : c;
    const int ec = (int(blockIdx.z) * NV * 32 + cv) * 8, slot_c = int(blockIdx.x) * TOK + g;
    if (ec >= d || slot_c >= p.B) continue;
    float out[8];
    if (empty) {
#pragma unroll
      for (int i = 0; i < 8; ++i) out[i] = 0.f;
    } else {
      sum_partials<NV, SPLIT>(&sums[g * SPLIT], cv, out);
    }
    sq += decode_epilogue(p, decode_token(p, slot_c), t, ec, out, loss_scale);
  }
  if (p.mode == 1 && p.sq_err != nullptr) {
    // one global atomic per CTA: all warps of the CTA work on the same target
    __shared__ float red_s[kWarps];
    sq = warp_sum(sq);
    if (lane == 0) red_s[warp] = sq;
    __syncthreads();
    sq = 0.f;
    for (int w = 0; w < kWarps; ++w) sq += red_s[w];
    if (threadIdx.x == 0 && sq != 0.f) atomicAdd(&p.sq_err[t], double(sq));
  }
}

// Per-source tied decoders without affine terms: the row of feature (s, f) serves every target t >= s with the same weight,
// so the reconstruction of target t is the one of t - 1 plus the entries of layer t.  The SPLIT warps of a CTA read every row of a
// (token, column chunk) once and finish a target whenever a layer's entries are in: their running sums meet in shared memory at every target.
// A warp holds 32 of its entries at a time and moves on when a layer has used them up, which takes a list whose layers ascend; any other
// list (the entries of a token may come in any order) is scanned once per layer.
template <int NV, int SPLIT, int R, int WARPS_PER_SM>
__global__ void __launch_bounds__(32 * SPLIT, WARPS_PER_SM / SPLIT) decode_running_kernel(const DecodeParams p) {
  if (chain_wait()) return;
  chain_release();
  __shared__ __align__(16) float sums[2][SPLIT][NV * 256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int d = p.d;
  const float loss_scale = p.ctl != nullptr ? p.ctl[SC_LOSS_SCALE] : 1.f;
  const int tok = decode_token(p, int(blockIdx.x));
  const int b = __ldg(p.tok_off + tok), e = __ldg(p.tok_off + tok + 1);
  int off[NV];
  bool act[NV];
  float acc[NV][8];
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    off[v] = ((int(blockIdx.y) * NV + v) * 32 + lane) * 8;
    act[v] = off[v] < d;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[v][i] = 0.f;
  }
  bool in_order = true;
  for (int i = b + 1 + int(threadIdx.x); i < e; i += 32 * SPLIT) in_order &= (__ldg(p.tcsr_col + i) >> 24) >= (__ldg(p.tcsr_col + i - 1) >> 24);
  const bool ascending = __syncthreads_and(in_order);
  float sq_t = 0.f;  // lane t: this warp's share of the sum of target t (at most 32 layers), one addition per CTA and target at the end
  int base = b + warp;  // position of lane 0's entry
  int col = 0;
  float a = 0.f;
  const auto fetch = [&]() {
    const int i = base + lane * SPLIT;
    col = i < e ? __ldg(p.tcsr_col + i) : 0;
    a = i < e ? __ldg(p.tcsr_val + i) : 0.f;
    if (a != 0.f && (!clt_in_bounds(col >> 24, p.L, p.dbg_status, 103) || !clt_in_bounds(col & 0xFFFFFF, p.col_pitch, p.dbg_status, 104))) a = 0.f;
  };
  fetch();
#pragma unroll 1
  for (int t = 0; t < p.L; ++t) {
    if (!ascending) {
      base = b + warp;
      fetch();
    }
    for (;;) {
      const uint32_t mask = __ballot_sync(0xFFFFFFFFu, a != 0.f && (col >> 24) == t);
      if (mask != 0u) gather_rows<NV, R>(mask, a, p.w[t] + 1LL * (col & 0xFFFFFF) * d, off, act, acc);
      if (base + 32 * SPLIT >= e) break;                                               // no entries behind these
      if (ascending && (__shfl_sync(0xFFFFFFFFu, col, 31) >> 24) > t) break;           // the last of these is a later layer's
      base += 32 * SPLIT;
      fetch();
    }
    // two buffers in turn: a warp that is already at the next target writes the other one, and it cannot be two targets
    // ahead, because the barrier of the next target needs every warp
    float(*buf)[NV * 256] = sums[t & 1];
    put_partial<NV>(buf[warp], acc, lane);
    __syncthreads();
    float sq = 0.f;
    for (int c = threadIdx.x; c < NV * 32; c += 32 * SPLIT) {
      const int ec = (int(blockIdx.y) * NV * 32 + c) * 8;
      if (ec >= d) continue;
      float out[8];
      sum_partials<NV, SPLIT>(buf, c, out);
      sq += decode_epilogue(p, tok, t, ec, out, loss_scale);
    }
    sq = warp_sum(sq);
    if (lane == t) sq_t = sq;
  }
  if (p.mode == 1 && p.sq_err != nullptr) {
    __shared__ float red_s[SPLIT][kMaxLayers];
    red_s[warp][lane] = sq_t;
    __syncthreads();
    sq_t = 0.f;
    if (warp == 0)
      for (int w = 0; w < SPLIT; ++w) sq_t += red_s[w][lane];
    if (warp == 0 && sq_t != 0.f) atomicAdd(&p.sq_err[lane], double(sq_t));
  }
}

// order[0 .. B): the tokens by the length of their lists, longest first (in classes of four; the order inside a class is open).
// One CTA: a counting sort of a few thousand lengths, 4 us.
constexpr int kLenClasses = 1024;
__global__ void __launch_bounds__(kLenClasses) decode_order_kernel(const int* __restrict__ tok_off, int B, int* __restrict__ order) {
  if (chain_wait()) return;
  chain_release();
  __shared__ int place[kLenClasses];
  __shared__ int warp_sums[32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  place[tid] = 0;
  __syncthreads();
  const auto class_of = [&](int i) { return kLenClasses - 1 - min((tok_off[i + 1] - tok_off[i]) >> 2, kLenClasses - 1); };
  // one addition per class and warp: lists of equal length would otherwise queue up at one counter
  const auto take = [&](int i, bool valid) {
    const int c = valid ? class_of(i) : kLenClasses;
    const uint32_t same = __match_any_sync(0xFFFFFFFFu, c);
    const int leader = __ffs(same) - 1;
    int first = 0;
    if (valid && lane == leader) first = atomicAdd(&place[c], __popc(same));
    return __shfl_sync(0xFFFFFFFFu, first, leader) + __popc(same & ((1u << lane) - 1u));
  };
  const int rounds = (B + kLenClasses - 1) / kLenClasses;
  for (int r = 0; r < rounds; ++r) take(r * kLenClasses + tid, r * kLenClasses + tid < B);
  __syncthreads();
  const int mine = place[tid];
  int x = mine;  // inclusive prefix sum over the warp, then over the warps
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xFFFFFFFFu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[warp] = x;
  __syncthreads();
  if (warp == 0) {
    int s = warp_sums[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xFFFFFFFFu, s, o);
      if (lane >= o) s += y;
    }
    warp_sums[lane] = s;
  }
  __syncthreads();
  place[tid] = x - mine + (warp > 0 ? warp_sums[warp - 1] : 0);
  __syncthreads();
  for (int r = 0; r < rounds; ++r) {
    const int i = r * kLenClasses + tid;
    const int at = take(i, i < B);
    if (i < B) order[at] = i;
  }
}

// Epilogue for the tensor-parallel path, run after the partial reconstructions were summed across ranks:
// bias, addend, residual, loss sum and gradient seed for rows [row0, row0 + nrows) of every layer.
__global__ void __launch_bounds__(256) recon_epilogue_kernel(const float* __restrict__ yhat_sum, const float* __restrict__ bias_sum,
                                                               const float* __restrict__ addend, const t16* __restrict__ target,
                                                               const float* __restrict__ sigma, t16* __restrict__ gs,
                                                               float* __restrict__ yhat_out, double* __restrict__ sq_err, int L, int B,
                                                               int d, int row0, int nrows, float* __restrict__ ctl) {
  if (chain_wait()) return;
  chain_release();
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
  if (chain_wait()) return;
  chain_release();
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
  if (chain_wait()) return;
  chain_release();
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
  int expected; // entries per token that the caller expects (its k), 0: not known
  int equal;    // every token has that many
  int* order;   // scratch of clt_sparse_decode_scratch(args) ints, null where that is 0
};

// 16-byte vectors per lane: the whole row up to d_model 1024 (a warp then reads an entry's row in one go), half of it above
static int walk_chunks(const CltDecodeArgs* a) { return a->d > 1024 ? 2 : 1; }
// at most two vectors per lane: the sums stay live across the epilogues of all targets
static int running_chunks(const CltDecodeArgs* a) { return (a->d + 511) / 512; }
static bool takes_running(const CltDecodeArgs* a) {
  return a->tying == 1 && a->feat_offset == nullptr && a->feat_scale == nullptr && a->rows_limit <= 0 && 1LL * a->B * running_chunks(a) >= kRunningMinWarps;
}

static long long walk_ctas(const CltDecodeArgs* a) { return 1LL * a->B * a->L * walk_chunks(a); }
static int walk_vectors(const CltDecodeArgs* a) { return (a->d / 8 + 32 * walk_chunks(a) - 1) / (32 * walk_chunks(a)); }
static bool short_lists(const CltDecodeArgs* a) { return a->expected > 0 && a->expected < kShortBelow; }
static int slices(const CltDecodeArgs* a) { return (a->d + 255) / 256; }
static bool takes_slices(const CltDecodeArgs* a) {
  return a->d > 512 && a->d <= 1024 && !short_lists(a) && 1LL * a->B * a->L * slices(a) <= kSliceCtasPerSm * device_sms();
}
// Lists of one length that a warp takes alone.
static bool one_warp_lists(const CltDecodeArgs* a) {
  if (a->equal == 0 || a->expected <= 0) return false;
  if (a->expected < kOneWarpBelow) return true;
  if (takes_running(a)) return a->B >= kOneWarpRunningFrom && (a->expected < kOneWarpMediumBelow || a->d <= 256);
  const int nv = walk_vectors(a);
  if (nv == 2) return walk_ctas(a) >= kOneWarpWalkFrom && a->expected < kOneWarpMediumBelow;
  return nv >= 3 && walk_ctas(a) >= (nv == 3 ? kOneWarpWalkFrom : kOneWarpWideWalkFrom);
}

// Number of ints the call wants in `order`: the tokens are sorted by length where there are so many CTAs that it pays.
extern "C" long long CLT_FN(clt_sparse_decode_scratch)(const CltDecodeArgs* a) {
  if (a->mode == 2 || a->B <= 0 || a->equal != 0 || short_lists(a)) return 0;
  if (takes_running(a)) return a->B >= kRunningOrderFrom ? a->B : 0;
  return a->d > 512 && walk_ctas(a) >= kManyCtas ? a->B : 0;
}

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
  if (a->order != nullptr && CLT_FN(clt_sparse_decode_scratch)(a) > 0) {
    p.order = a->order;
    launch_chained(decode_order_kernel, 1, kLenClasses, 0, st, a->tok_off, a->B, a->order);
  } else {
    p.order = nullptr;
  }
  if (takes_running(a)) {
    const dim3 grid(a->B, running_chunks(a));
    if (one_warp_lists(a) || (a->equal == 0 && a->expected > 0 && a->expected < kRunningOneWarpBelow)) {
      if (a->d <= 256) launch_chained(decode_running_kernel<1, 1, 4, 28>, grid, 32, 0, st, p);
      else launch_chained(decode_running_kernel<2, 1, 4, 16>, grid, 32, 0, st, p);
    } else if (short_lists(a) || (a->expected <= 0 && 1LL * a->B * running_chunks(a) >= kRunningTwoWarpsFrom)) {
      if (a->d <= 256) launch_chained(decode_running_kernel<1, 2, 4, 24>, grid, 64, 0, st, p);
      else launch_chained(decode_running_kernel<2, 2, 4, 20>, grid, 64, 0, st, p);
    } else {
      if (a->d <= 256) launch_chained(decode_running_kernel<1, 4, 4, 24>, grid, 128, 0, st, p);
      else launch_chained(decode_running_kernel<2, 4, 4, 20>, grid, 128, 0, st, p);
    }
    return cudaGetLastError() == cudaSuccess ? 0 : -5;
  }
  const int chunks = walk_chunks(a), nv = walk_vectors(a);
  const long long ctas = walk_ctas(a);
  const dim3 grid(a->B, a->L, chunks);
  if (takes_slices(a)) {
    launch_chained(decode_walk_kernel<1, 1, 8, 8, 32>, dim3(a->B, a->L, slices(a)), 256, 0, st, p);
  } else if (ctas < kEightWarpsBelow) {
    if (nv <= 1) launch_chained(decode_walk_kernel<1, 1, 8, 4, 32>, grid, 256, 0, st, p);
    else if (nv == 2) launch_chained(decode_walk_kernel<2, 1, 8, 4, 24>, grid, 256, 0, st, p);
    else if (nv == 3) launch_chained(decode_walk_kernel<3, 1, 8, 4, 16>, grid, 256, 0, st, p);
    else launch_chained(decode_walk_kernel<4, 1, 8, 4, 16>, grid, 256, 0, st, p);
  } else if (one_warp_lists(a)) {
    if (nv <= 1) launch_chained(decode_walk_kernel<1, 4, 1, 4, 32>, dim3((a->B + 3) / 4, a->L), 128, 0, st, p);
    else if (nv == 2) launch_chained(decode_walk_kernel<2, 2, 1, 4, 24>, dim3((a->B + 1) / 2, a->L), 64, 0, st, p);
    else if (nv == 3) launch_chained(decode_walk_kernel<3, 1, 1, 2, 28>, grid, 32, 0, st, p);
    else launch_chained(decode_walk_kernel<4, 1, 1, 2, 20>, grid, 32, 0, st, p);
  } else if (nv <= 1) {
    if (ctas >= kPairNarrowFrom) launch_chained(decode_walk_kernel<1, 2, 2, 4, 40>, dim3((a->B + 1) / 2, a->L), 128, 0, st, p);
    else launch_chained(decode_walk_kernel<1, 1, 4, 4, 40>, grid, 128, 0, st, p);
  } else if (short_lists(a) && ctas >= kShortFrom) {
    if (nv == 2) launch_chained(decode_walk_kernel<2, 1, 2, 4, 24>, grid, 64, 0, st, p);
    else if (nv == 3) launch_chained(decode_walk_kernel<3, 1, 2, 2, 28>, grid, 64, 0, st, p);
    else launch_chained(decode_walk_kernel<4, 1, 2, 2, 20>, grid, 64, 0, st, p);
  } else if (nv == 2) {
    launch_chained(decode_walk_kernel<2, 1, 4, 4, 24>, grid, 128, 0, st, p);
  } else if (ctas >= kManyCtas) {
    if (nv == 3) launch_chained(decode_walk_kernel<3, 1, 4, 2, 28>, grid, 128, 0, st, p);
    else launch_chained(decode_walk_kernel<4, 1, 4, 2, 20>, grid, 128, 0, st, p);
  } else {
    if (nv == 3) launch_chained(decode_walk_kernel<3, 1, 4, 4, 20>, grid, 128, 0, st, p);
    else launch_chained(decode_walk_kernel<4, 1, 4, 4, 16>, grid, 128, 0, st, p);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

extern "C" int CLT_FN(clt_recon_epilogue)(const float* yhat_sum, const float* bias_sum, const float* addend, const void* target,
                                  const float* sigma, void* gs, float* yhat_out, double* sq_err, int L, int B, int d, int row0,
                                  int nrows, float* ctl, cudaStream_t st) {
  if (d % 8 != 0) return -1;
  if (nrows <= 0) return 0;
  dim3 grid(148, L);
  launch_chained(recon_epilogue_kernel, grid, 256, 0, st, yhat_sum, bias_sum, addend, static_cast<const t16*>(target), sigma,
                                              static_cast<t16*>(gs), yhat_out, sq_err, L, B, d, row0, nrows, ctl);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

extern "C" int CLT_FN(clt_gs_colsum)(const void* gs, float* out, int L, int B, int d, cudaStream_t st) {
  if (d % 8 != 0) return -1;
  const int tx = d / 8 >= 128 ? 128 : ((d / 8 + 31) / 32) * 32;
  const int ty = 1024 / tx < 8 ? 1024 / tx : 8;
  const int rpb = 128;
  dim3 grid((d / 8 + tx - 1) / tx, (B + rpb - 1) / rpb, L), block(tx, ty);
  launch_chained(gs_colsum_kernel, grid, block, 0, st, static_cast<const t16*>(gs), out, B, d, rpb);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

extern "C" int CLT_FN(clt_gs_suffix_sum)(const void* gs, void* out, int L, int B, int d, cudaStream_t st) {
  const long long per_layer = 1LL * B * d;
  if (per_layer % 8 != 0) return -1;
  const long long nvec = per_layer / 8;
  const int grid = int(nvec / 256 + 1 < 1184 ? nvec / 256 + 1 : 1184);
  launch_chained(gs_suffix_sum_kernel, grid, 256, 0, st, static_cast<const t16*>(gs), static_cast<t16*>(out), L, per_layer);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
