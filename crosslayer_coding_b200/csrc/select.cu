// Global BatchTopK without a dense [B, L*F] ranking tensor (sm_100a).
//
// The reference concatenates every layer's batch-z-scored pre-activations and calls torch.topk on the
// flattened tensor (clt/models/activations.py:27-32, 281-357).  Here the same selection is a threshold
// search over the bf16 pre-activations written by the encoder GEMM:
//
//   1. colstats      per-feature batch mean and 1/(std+1e-6) (unbiased std, shifted sums)
//   2. zhist         8192-bin histogram of the order-preserving key of z = (x-mean)*rstd, keys >= key_lo
//   3. find_bin      bin that contains the k_total-th largest key (after the ranks' histograms were summed)
//   4. compact       entries above the bin go to the output list, entries inside it to a candidate list
//   5. refine        exact key cut inside the bin by radix passes; ties resolved by lowest flat index
//                    b*(L*F) + l*F + f so the result does not depend on the tensor-parallel world size
//   6. finalize      candidates on the keep side of the cut are appended to the output list
//   7. csr           token-major and feature-major CSR views of the list for the decoder / backward
//
// Under tensor parallelism every rank runs 1-2 and 4-7 on its feature shard; only histograms cross GPUs
// (the 8192-bin one and the 512-bin refinement rounds), written straight into the peers' exchange
// buffers by the kernels below with bounded flag waits.
#include "common.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace clt {

constexpr int kHistBins = 8192;
constexpr int kRefineBins = 512;

// Control block shared by the selection kernels (device memory, int64 slots).
enum SelCtl : int {
  CTL_BIN = 0,          // threshold bin
  CTL_ABOVE = 1,        // number of keys in bins above it (global over ranks)
  CTL_NEED = 2,         // how many the threshold bin has to contribute (global)
  CTL_NUM_ENTRIES = 3,  // length of the output list (this rank)
  CTL_NUM_CAND = 4,     // length of the candidate list (this rank)
  CTL_CUT_KEY = 5,      // exact key cut T
  CTL_TIE_MODE = 6,     // 0: keep every key == T; 1: keep ties with flat index <= CTL_CUT_FLAT
  CTL_CUT_FLAT = 7,
  CTL_KEY_LO = 8,       // histogram range actually used: keys >= key_lo, bin = (key - key_lo) >> shift
  CTL_SHIFT = 9,
  CTL_RETRY = 10,       // 1: the narrow histogram did not contain the cut, the full-range pass runs
  CTL_SIZE = 16,
};

// Sum `n` uint32 counters over all ranks, in place in shared memory `vals` (one CTA).  Every rank stores
// its vector into slot [round][rank] of every peer, raises flag [round][rank] there, then waits (bounded)
// for the flags of all peers in its own area and adds the slots up.  Returns false on a timeout.
__device__ bool exchange_sum(const Exchange& ex, int round, uint32_t* vals, int n, int* timeout_flag_smem) {
  if (ex.world <= 1) return true;
  if (!exchange_gather(ex, round, vals, n, timeout_flag_smem)) return false;
  const uint32_t* mine = exchange_slot(ex, round, 0);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    uint32_t s = 0;
    for (int p = 0; p < ex.world; ++p) s += mine[size_t(p) * ex.slot_elems + i];
    vals[i] = s;
  }
  __syncthreads();
  return true;
}

// ------------------------------------------------------------------ 1. column statistics
// x: [L, B, ld] bf16.  Each thread owns VEC adjacent columns; blockDim = (32, 8): 8 row groups.
// With gridDim.z > 1 (narrow shards, where one CTA per column block would leave SMs idle) the rows are split
// over blockIdx.z: the shifted sums are additive because every chunk shifts by the column's first row, so the
// chunks add them into mean / rstd (zeroed by the launcher) and colstats_finalize_kernel converts in place.
// blockIdx.x counts blocks of 32 * VEC columns over strips of 256 columns over all layers, from strip `first_strip` on: the encoder GEMM computes the
// statistics of the strips before it, with the same sums in the same order (eight per column, rows r = y mod 8, added in the order of y).
// VEC = 8: 64 bytes in flight per thread, for many strips.  VEC = 2: four times the threads with 128 bytes each, for the few strips that the GEMM
// leaves, where the chip would wait for 8 x 256 chains (28 strips of 8192 rows: 25 us).
template <int VEC>
struct ColstatsLoad;
template <>
struct ColstatsLoad<8> {
  using T = uint4;
  static constexpr int kDepth = 4;
  __device__ static uint32_t word(const uint4& v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; }
};
template <>
struct ColstatsLoad<2> {
  using T = uint32_t;
  static constexpr int kDepth = 32;
  __device__ static uint32_t word(const uint32_t& v, int) { return v; }
};
template <int VEC>
__global__ void __launch_bounds__(256) colstats_kernel(const t16* __restrict__ x, float* __restrict__ mean,
                                                         float* __restrict__ rstd, int B, int F, long long ld,
                                                         long long layer_stride, long long first_strip) {
  if (chain_wait()) return;
  chain_release();
  using Ld = ColstatsLoad<VEC>;
  constexpr int kBlocks = 8 / VEC;  // of 32 * VEC columns in a strip
  constexpr int kDepth = Ld::kDepth;
  const int strips = (F + 255) / 256;
  const long long strip = first_strip + blockIdx.x / kBlocks;
  const int l = int(strip / strips);
  const int rows_per_z = (((B + int(gridDim.z) - 1) / int(gridDim.z)) + 31) / 32 * 32;
  const int row_lo = int(blockIdx.z) * rows_per_z;
  const int row_hi = min(B, row_lo + rows_per_z);
  const int c0 = int(strip % strips) * 256 + (int(blockIdx.x % kBlocks) * 32 + int(threadIdx.x)) * VEC;
  __shared__ float red[8][32][2 * VEC + 1];
  float s[VEC], q[VEC], shift[VEC];
#pragma unroll
  for (int j = 0; j < VEC; ++j) s[j] = q[j] = shift[j] = 0.f;
  const bool active = c0 < F;
  const t16* base = x + 1LL * l * layer_stride + c0;
  if (active) {
    const typename Ld::T v0 = *reinterpret_cast<const typename Ld::T*>(base);
#pragma unroll
    for (int j = 0; j < VEC / 2; ++j) { shift[2 * j] = t16_lo(Ld::word(v0, j)); shift[2 * j + 1] = t16_hi(Ld::word(v0, j)); }
    // kDepth independent loads in flight.  With eight columns only the last batch tests its rows (6 x 2048 x 32768: 176 us with a test of each, 164); with
    // two, full batches of 32 loads would be split up (14 strips of 4096 rows behind a GEMM: 30 us without tests, 20 with).
    const auto batch = [&](int r0, auto last) {
      constexpr bool kLast = decltype(last)::value;
      typename Ld::T v[kDepth];
#pragma unroll
      for (int k = 0; k < kDepth; ++k)
        v[k] = !kLast || r0 + 8 * k < row_hi ? __ldcs(reinterpret_cast<const typename Ld::T*>(base + 1LL * (r0 + 8 * k) * ld)) : v0;
#pragma unroll
      for (int k = 0; k < kDepth; ++k) {
        if (kLast && r0 + 8 * k >= row_hi) break;
#pragma unroll
        for (int j = 0; j < VEC / 2; ++j) {
          const uint32_t u = Ld::word(v[k], j);
          const float a = t16_lo(u) - shift[2 * j], b = t16_hi(u) - shift[2 * j + 1];
          s[2 * j] += a; q[2 * j] += a * a;
          s[2 * j + 1] += b; q[2 * j + 1] += b * b;
        }
      }
    };
    int r0 = row_lo + threadIdx.y;
    if constexpr (VEC == 8)
      for (; r0 + 8 * (kDepth - 1) < row_hi; r0 += 8 * kDepth) batch(r0, std::false_type{});
    for (; r0 < row_hi; r0 += 8 * kDepth) batch(r0, std::true_type{});
  }
#pragma unroll
  for (int j = 0; j < VEC; ++j) { red[threadIdx.y][threadIdx.x][j] = s[j]; red[threadIdx.y][threadIdx.x][VEC + j] = q[j]; }
  __syncthreads();
  if (threadIdx.y == 0 && active) {
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
      float ss = 0.f, qq = 0.f;
      for (int y = 0; y < 8; ++y) { ss += red[y][threadIdx.x][j]; qq += red[y][threadIdx.x][VEC + j]; }
      if (c0 + j < F && gridDim.z > 1) {
        atomicAdd(&mean[1LL * l * F + c0 + j], ss);
        atomicAdd(&rstd[1LL * l * F + c0 + j], qq);
      } else if (c0 + j < F) {
        colstats_finish(ss, qq, shift[j], B, &mean[1LL * l * F + c0 + j], &rstd[1LL * l * F + c0 + j]);
      }
    }
  }
}

// Column statistics from the per-block sums that the encoder GEMM's epilogue leaves behind:
// tile_stats [L][row_blocks][F][2] = (sum, sum of squares) over the rows of one 128-row block.  The blocks are merged
// with the pairwise update of Chan et al. (block means first), which keeps the variance accurate when the mean is
// large against the spread.
__global__ void __launch_bounds__(256) colstats_from_tiles_kernel(const float* __restrict__ tile_stats, float* __restrict__ mean,
                                                                    float* __restrict__ rstd, int B, int F, int row_blocks, long long n) {
  if (chain_wait()) return;
  chain_release();
  const long long i = blockIdx.x * 1LL * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int l = int(i / F), c = int(i - 1LL * l * F);
  const float2* src = reinterpret_cast<const float2*>(tile_stats) + (1LL * l * row_blocks) * F + c;
  float cnt = 0.f, mu = 0.f, m2 = 0.f;
  for (int rb = 0; rb < row_blocks; ++rb) {
    const float2 sq = src[1LL * rb * F];
    const float nb = float(min(128, B - rb * 128));
    const float mb = sq.x / nb;
    const float m2b = fmaxf(sq.y - sq.x * mb, 0.f);
    const float tot = cnt + nb;
    const float delta = mb - mu;
    m2 += m2b + delta * delta * (cnt * nb / tot);
    mu += delta * (nb / tot);
    cnt = tot;
  }
  const float var = B > 1 ? fmaxf(m2 / float(B - 1), 0.f) : 0.f;
  mean[i] = mu;
  rstd[i] = 1.f / (sqrtf(var) + 1e-6f);
}

// mean / rstd hold the shifted sum and sum of squares (shift = the column's first row); convert in place.
__global__ void __launch_bounds__(256) colstats_finalize_kernel(const t16* __restrict__ x, float* __restrict__ mean,
                                                                  float* __restrict__ rstd, int B, int F, long long layer_stride,
                                                                  long long first, long long n) {
  if (chain_wait()) return;
  chain_release();
  const long long i = first + blockIdx.x * 1LL * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int l = int(i / F), c = int(i - 1LL * l * F);
  const float shift = t16_to_float(x[1LL * l * layer_stride + c]);
  colstats_finish(mean[i], rstd[i], shift, B, &mean[i], &rstd[i]);
}

// ------------------------------------------------------------------ 2. histogram of z keys
struct ScanGeom {
  int B, F, L;           // F = valid local columns per layer
  int sp;                // pitch of the mean / rstd rows (>= F)
  long long ld;          // row pitch of x (elements)
  long long layer_stride;
  int rows_per_block;
};

__device__ __forceinline__ void load_cols8(const float* p, float (&o)[8]) {
  const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
  o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
}

// `only_if_retry`: the full-range pass; it runs only when the narrow pass asked for it.
__global__ void __launch_bounds__(256) zhist_kernel(const t16* __restrict__ x, const float* __restrict__ mean,
                                                      const float* __restrict__ rstd, ScanGeom g, uint32_t key_lo, int shift,
                                                      unsigned int* __restrict__ hist, const long long* __restrict__ ctl,
                                                      int only_if_retry) {
  if (chain_wait()) return;
  chain_release();
  if (only_if_retry && ctl[CTL_RETRY] == 0) return;
  const float z_lo = key_lo == 0u ? -INFINITY : key_to_float(key_lo);
  __shared__ unsigned int sh[kHistBins];
  for (int i = threadIdx.x; i < kHistBins; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const int l = blockIdx.z;
  const int c0 = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  if (c0 < g.F) {
    float mu[8], rs[8];
    if (c0 + 8 <= g.F) {
      load_cols8(mean + 1LL * l * g.sp + c0, mu);
      load_cols8(rstd + 1LL * l * g.sp + c0, rs);
    } else {
      for (int j = 0; j < 8; ++j) {
        const bool in = c0 + j < g.F;
        mu[j] = in ? mean[1LL * l * g.sp + c0 + j] : 0.f;
        rs[j] = in ? rstd[1LL * l * g.sp + c0 + j] : 0.f;
      }
    }
    const int nvalid = min(8, g.F - c0);
    const int r0 = blockIdx.y * g.rows_per_block;
    const int r1 = min(g.B, r0 + g.rows_per_block);
    const t16* base = x + 1LL * l * g.layer_stride + c0;
    for (int rb = r0; rb < r1; rb += 4) {
      uint4 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        v[k] = (rb + k < r1) ? __ldg(reinterpret_cast<const uint4*>(base + 1LL * (rb + k) * g.ld)) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (rb + k >= r1) break;
        const uint32_t u[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xv = (j & 1) ? t16_hi(u[j >> 1]) : t16_lo(u[j >> 1]);
          const float z = (xv - mu[j]) * rs[j];
          if (z >= z_lo && j < nvalid) {  // one float compare for the bulk; keys only for the tail that counts
            const uint32_t key = float_to_key(z);
            atomicAdd(&sh[min((key - key_lo) >> shift, uint32_t(kHistBins - 1))], 1u);
          }
        }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kHistBins; i += blockDim.x) {
    const unsigned int c = sh[i];
    if (c) atomicAdd(&hist[i], c);
  }
}

// ------------------------------------------------------------------ 2b. histogram + pool in one pass
// The range of the narrow histogram lives in device memory (`sel_state`: key_lo, shift) and follows the
// cut from step to step (find_bin_kernel moves it).  Every element inside the range is also appended to a
// pool (key, token, column, value), so that the later stages read a list of a few k_total elements instead
// of the whole pre-activation matrix a second time.
struct Pool {
  uint32_t* key;
  int* tok;
  int* col;
  float* val;
  long long cap;
  unsigned int* count;  // zeroed by the caller together with the histograms
};
constexpr int kPoolStage = 512;   // histogram + queue + staging stay inside the 48 KB of static shared memory
constexpr int kHitQueue = 1024;   // 16-byte groups per CTA that passed the coarse filter (threshold scan: four times that)
constexpr int kCollectQueue = 2 * kHitQueue;  // in the histogram scan, whose tile (64 rows, 256 threads) takes 16 bits to number
constexpr int kHistExtra = 32;    // words after the two histograms: [0] = pool counter

// Phase A streams the matrix with a coarse filter in the input's own format (one packed compare per two
// elements) and only queues the 16-byte groups that may hold an element of the range; phase B runs the exact
// test on the queued groups, one element per thread.  The hot loop stays a few instructions per group.
__global__ void __launch_bounds__(256) zhist_collect_kernel(const t16* __restrict__ x, const float* __restrict__ mean,
                                                              const float* __restrict__ rstd, ScanGeom g, int col_pitch,
                                                              const long long* __restrict__ sel_state,
                                                              unsigned int* __restrict__ hist, Pool pool) {
  if (chain_wait()) return;
  chain_release();
  const uint32_t key_lo = uint32_t(sel_state[0]);
  const int shift = int(sel_state[1]);
  const float z_lo = key_to_float(key_lo);
  __shared__ unsigned int sh[kHistBins];
  __shared__ uint16_t s_queue[kCollectQueue];
  __shared__ uint32_t s_key[kPoolStage];
  __shared__ int s_tok[kPoolStage];
  __shared__ int s_col[kPoolStage];
  __shared__ float s_val[kPoolStage];
  __shared__ int s_q, s_n;
  __shared__ unsigned int s_base;
  for (int i = threadIdx.x; i < kHistBins; i += blockDim.x) sh[i] = 0;
  if (threadIdx.x == 0) { s_q = 0; s_n = 0; }
  __syncthreads();
  const int l = blockIdx.z;
  const int c0 = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  const int r0 = blockIdx.y * g.rows_per_block;
  const int r1 = min(g.B, r0 + g.rows_per_block);
  if (c0 < g.F) {
    // thr_j = mean_j + z_lo / rstd_j, lowered by a margin for the fp32 rounding of the exact test and rounded
    // down to bf16: x >= thr_j is implied by z_j >= z_lo
    uint32_t thr2[4];
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      float t[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const bool in = c0 + j + q < g.F;
        const float mu = in ? __ldg(mean + 1LL * l * g.sp + c0 + j + q) : 0.f;
        const float rs = in ? __ldg(rstd + 1LL * l * g.sp + c0 + j + q) : 0.f;
        const float span = z_lo / rs;
        t[q] = (in && rs > 0.f) ? mu + span - 1e-5f * (fabsf(mu) + fabsf(span)) - 1e-30f : INFINITY;
      }
      const t16x2 pk = make_t16x2(float_to_t16_rd(t[0]), float_to_t16_rd(t[1]));
      thr2[j >> 1] = *reinterpret_cast<const uint32_t*>(&pk);
    }
    const t16* base = x + 1LL * l * g.layer_stride + c0;
    for (int rb = r0; rb < r1; rb += 8) {
      uint4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int r = min(rb + k, r1 - 1);
        v[k] = __ldcs(reinterpret_cast<const uint4*>(base + 1LL * r * g.ld));
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t hit = t16x2_ge_mask(v[k].x, thr2[0]) | t16x2_ge_mask(v[k].y, thr2[1]) |
                             t16x2_ge_mask(v[k].z, thr2[2]) | t16x2_ge_mask(v[k].w, thr2[3]);
        if (hit != 0 && rb + k < r1) {
          const int slot = atomicAdd(&s_q, 1);
          if (slot < kCollectQueue) s_queue[slot] = uint16_t((uint32_t(rb + k - r0) << 8) | threadIdx.x);
        }
      }
    }
  }
  __syncthreads();
  // ---- phase B: exact test, histogram and pool staging, one element per thread
  const int nq_all = s_q;
  if (nq_all > kCollectQueue && threadIdx.x == 0) atomicOr(pool.count, 0x80000000u);  // lost groups: force the full-range pass
  const int nq = nq_all > kCollectQueue ? 0 : nq_all;  // lost groups: nothing of this pass will be used
  // (four elements per thread and round: the loads of one after the other were a seventh of the kernel)
  for (int e0 = threadIdx.x; e0 < nq * 8; e0 += 4 * 256) {
    int r[4], c[4];
    bool in[4];
    float xv[4], mu[4], rs[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + 256 * u;
      const uint32_t item = e < nq * 8 ? s_queue[e >> 3] : 0u;
      r[u] = r0 + int(item >> 8);
      c[u] = (blockIdx.x * 256 + int(item & 255u)) * 8 + (e & 7);
      in[u] = e < nq * 8 && c[u] < g.F;
      xv[u] = in[u] ? t16_to_float(x[1LL * l * g.layer_stride + 1LL * r[u] * g.ld + c[u]]) : 0.f;
      mu[u] = in[u] ? __ldg(mean + 1LL * l * g.sp + c[u]) : 0.f;
      rs[u] = in[u] ? __ldg(rstd + 1LL * l * g.sp + c[u]) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float z = (xv[u] - mu[u]) * rs[u];
      if (!in[u] || !(z >= z_lo)) continue;
      const uint32_t key = float_to_key(z);
      atomicAdd(&sh[min((key - key_lo) >> shift, uint32_t(kHistBins - 1))], 1u);
      const int slot = atomicAdd(&s_n, 1);
      if (slot < kPoolStage) {
        s_key[slot] = key; s_tok[slot] = r[u]; s_col[slot] = l * col_pitch + c[u]; s_val[slot] = xv[u];
      } else {  // staging full: append directly
        const unsigned int q = atomicAdd(pool.count, 1u);
        if ((long long)q < pool.cap) { pool.key[q] = key; pool.tok[q] = r[u]; pool.col[q] = l * col_pitch + c[u]; pool.val[q] = xv[u]; }
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kHistBins; i += blockDim.x) {
    const unsigned int c = sh[i];
    if (c) atomicAdd(&hist[i], c);
  }
  const int staged = min(s_n, kPoolStage);
  if (staged == 0) return;
  if (threadIdx.x == 0) s_base = atomicAdd(pool.count, (unsigned int)staged);
  __syncthreads();
  for (int i = threadIdx.x; i < staged; i += blockDim.x) {
    const long long q = (long long)s_base + i;
    if (q < pool.cap) { pool.key[q] = s_key[i]; pool.tok[q] = s_tok[i]; pool.col[q] = s_col[i]; pool.val[q] = s_val[i]; }
  }
}

// ------------------------------------------------------------------ 3. threshold bin (one CTA, 1024 threads)
// pass 0: narrow histogram; when it does not contain the cut it only raises CTL_RETRY.
// pass 1: full-range histogram, runs only on retry; a miss there is a real error.
struct Lists {
  int* ent_tok;    // token index
  int* ent_col;    // l * F_local_pitch + f_local
  float* ent_val;  // original pre-activation
  long long ent_cap;
  uint32_t* cand_key;
  int* cand_tok;
  int* cand_col;
  float* cand_val;
  long long cand_cap;
};

// `sel_state` (optional): the tracked range.  Pass 0 reads the range from it; the pass that finds the cut
// moves the range for the next step so that about kPoolFactor * k_total elements fall inside it.
constexpr double kPoolFactor = 1.75;

// Bin width for a tracked range that starts at key_lo: the bins resolve z in [z_lo, max(2 z_lo, z_lo + 4)];
// everything above lands in the top bin (kernels clamp the bin index), which is therefore never accepted as
// the threshold bin.  Finer bins leave fewer candidates for the exact cut.
__device__ __forceinline__ int shift_for(uint32_t key_lo) {
  const float z_lo = key_to_float(key_lo);
  const uint32_t key_hi = float_to_key(fmaxf(2.f * z_lo, z_lo + 4.f));
  const uint32_t span = key_hi > key_lo ? key_hi - key_lo : 0xFFFFFFFFu - key_lo;
  int sh = 0;
  while ((span >> sh) >= uint32_t(kHistBins - 1)) ++sh;
  return sh;
}

__global__ void __launch_bounds__(1024) find_bin_kernel(const unsigned int* __restrict__ hist, long long k_total,
                                                          long long* __restrict__ ctl, Exchange ex, uint32_t key_lo_arg,
                                                          int shift_arg, int pass, int exchange_round,
                                                          long long* __restrict__ sel_state,
                                                          const unsigned int* __restrict__ pool_count, long long pool_cap,
                                                          int* __restrict__ status) {
  if (chain_wait()) return;
  if (ex.world <= 1) chain_release();  // else it waits for the other ranks below
  __shared__ uint32_t vals[kHistBins + kHistExtra];
  __shared__ unsigned long long part[1024];
  __shared__ int timeout;
  __shared__ int found;
  const int tid = threadIdx.x;
  if (pass == 1 && ctl[CTL_RETRY] == 0) return;
  const bool tracked = sel_state != nullptr;
  const uint32_t key_lo = (pass == 0 && tracked) ? uint32_t(sel_state[0]) : key_lo_arg;
  const int shift = (pass == 0 && tracked) ? int(sel_state[1]) : shift_arg;
  if (tid == 0) { timeout = 0; found = 0; }
  for (int i = tid; i < kHistBins; i += 1024) vals[i] = hist[i];
  if (tid < kHistExtra) vals[kHistBins + tid] = 0;
  __syncthreads();
  // a rank whose pool overflowed makes every rank take the full-range path
  if (tid == 0 && pass == 0 && pool_count != nullptr && (long long)(*pool_count) > pool_cap) vals[kHistBins] = 1;
  __syncthreads();
  if (!exchange_sum(ex, exchange_round, vals, kHistBins + 1, &timeout)) {
    if (tid == 0) atomicCAS(status, STATUS_OK, STATUS_WAIT_TIMEOUT);
    return;
  }
  const bool overflow = vals[kHistBins] != 0;
  // thread t owns bins [8t, 8t+8); part[t] = number of keys in the bins of all threads above t (suffix scan:
  // shuffles inside a warp, then over the 32 warp totals)
  unsigned long long mine = 0;
  for (int j = 0; j < 8; ++j) mine += vals[tid * 8 + j];
  {
    __shared__ unsigned long long warp_tot[32], warp_above[32];
    const int lane = tid & 31, warp = tid >> 5;
    unsigned long long incl = mine;  // sum over lanes >= this lane
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_down_sync(0xFFFFFFFFu, incl, o);
      if (lane + o < 32) incl += t;
    }
    if (lane == 0) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      unsigned long long w = warp_tot[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_down_sync(0xFFFFFFFFu, w, o);
        if (lane + o < 32) w += t;
      }
      warp_above[lane] = w - warp_tot[lane];
    }
    __syncthreads();
    part[tid] = (incl - mine) + warp_above[warp];
  }
  __syncthreads();
  unsigned long long total = 0;
  if (tid == 0) {
    const unsigned long long run = part[0] + mine;
    total = run;
    // tracked ranges clamp large keys into the top bin: a cut inside it cannot be refined, take the full pass
    const bool top_bin_cut = tracked && pass == 0 && (unsigned long long)vals[kHistBins - 1] >= (unsigned long long)k_total;
    const bool in_range = run >= (unsigned long long)k_total;
    found = (in_range && !overflow && !top_bin_cut) ? 1 : 0;
    if (!found) {
      if (pass == 0) ctl[CTL_RETRY] = 1;
      else atomicCAS(status, STATUS_OK, STATUS_SELECT_RANGE);
    } else if (pass == 0) {
      ctl[CTL_RETRY] = 0;
    }
    if (pass == 0 || found) {
      ctl[CTL_NUM_ENTRIES] = 0;
      ctl[CTL_NUM_CAND] = 0;
    }
    if (tracked && pass == 0 && !in_range) {
      // the range starts above the cut: lower it (the full-range pass of this step refines the guess)
      const float z = fmaxf(key_to_float(key_lo) - 0.1f, 0.f);
      const uint32_t nk = float_to_key(z);
      sel_state[0] = (long long)nk;
      sel_state[1] = shift_for(nk);
    }
  }
  __syncthreads();
  const unsigned long long target = (unsigned long long)(kPoolFactor * double(k_total));
  unsigned long long above = part[tid];  // keys in bins above this thread's group
  for (int j = 7; j >= 0; --j) {
    const unsigned long long c = vals[tid * 8 + j];
    if (found && above < (unsigned long long)k_total && above + c >= (unsigned long long)k_total) {
      ctl[CTL_BIN] = tid * 8 + j;
      ctl[CTL_ABOVE] = (long long)above;
      ctl[CTL_NEED] = k_total - (long long)above;
      ctl[CTL_KEY_LO] = (long long)key_lo;
      ctl[CTL_SHIFT] = shift;
    }
    if (tracked && above < target && above + c >= target) {
      // next step's range starts at the bin that holds the target-th largest key (never below z = 0)
      const unsigned long long nk64 = (unsigned long long)key_lo + ((unsigned long long)(tid * 8 + j) << shift);
      uint32_t nk = nk64 > 0xFFFFFFFFULL ? 0xFFFFFFFFu : uint32_t(nk64);
      if (nk < 0x80000000u) nk = 0x80000000u;
      sel_state[0] = (long long)nk;
      sel_state[1] = shift_for(nk);
    }
    above += c;
  }
  if (tracked && tid == 0 && found && total < target) {
    // fewer elements in range than wanted: widen a little for the next step
    const float z = fmaxf(key_to_float(key_lo) - 0.1f, 0.f);
    const uint32_t nk = float_to_key(z);
    sel_state[0] = (long long)nk;
    sel_state[1] = shift_for(nk);
  }
}

// ------------------------------------------------------------------ 2c. per-feature threshold selection
// JumpReLU (x >= theta_f) and ReLU (theta = smallest positive bf16) as a sparse selection: the same two-phase
// scan as above with the feature's own threshold as the filter; emits the (token, column, value) list that the
// CSR build and the sparse decode consume.  Meant for sparse activations: when a CTA queues more groups than
// its queue holds, or the list does not fit, the status word reports STATUS_CAPACITY and the caller falls back
// to the dense path.
__global__ void __launch_bounds__(256) threshold_collect_kernel(const t16* __restrict__ x, const float* __restrict__ theta,
                                                                  ScanGeom g, int col_pitch, long long* __restrict__ ctl,
                                                                  Lists o, int* __restrict__ status) {
  if (chain_wait()) return;
  chain_release();
  __shared__ uint32_t s_queue[4 * kHitQueue];
  __shared__ int s_tok[2 * kPoolStage];
  __shared__ int s_col[2 * kPoolStage];
  __shared__ float s_val[2 * kPoolStage];
  __shared__ int s_q, s_n;
  __shared__ unsigned long long s_base;
  constexpr int kQueue = 4 * kHitQueue, kStage = 2 * kPoolStage;
  if (threadIdx.x == 0) { s_q = 0; s_n = 0; }
  __syncthreads();
  const int l = blockIdx.z;
  const int c0 = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  const int r0 = blockIdx.y * g.rows_per_block;
  const int r1 = min(g.B, r0 + g.rows_per_block);
  unsigned long long* n_ent = reinterpret_cast<unsigned long long*>(ctl + CTL_NUM_ENTRIES);
  if (c0 < g.F) {
    uint32_t thr2[4];
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      float t[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) t[q] = c0 + j + q < g.F ? __ldg(theta + 1LL * l * g.sp + c0 + j + q) : INFINITY;
      const t16x2 pk = make_t16x2(float_to_t16_rd(t[0]), float_to_t16_rd(t[1]));
      thr2[j >> 1] = *reinterpret_cast<const uint32_t*>(&pk);
    }
    const t16* base = x + 1LL * l * g.layer_stride + c0;
    for (int rb = r0; rb < r1; rb += 8) {
      uint4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int r = min(rb + k, r1 - 1);
        v[k] = __ldcs(reinterpret_cast<const uint4*>(base + 1LL * r * g.ld));
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t hit = t16x2_ge_mask(v[k].x, thr2[0]) | t16x2_ge_mask(v[k].y, thr2[1]) |
                             t16x2_ge_mask(v[k].z, thr2[2]) | t16x2_ge_mask(v[k].w, thr2[3]);
        if (hit != 0 && rb + k < r1) {
          const int slot = atomicAdd(&s_q, 1);
          if (slot < kQueue) s_queue[slot] = (uint32_t(rb + k - r0) << 8) | threadIdx.x;
        }
      }
    }
  }
  __syncthreads();
  const int nq_all = s_q;
  if (nq_all > kQueue && threadIdx.x == 0) atomicCAS(status, STATUS_OK, STATUS_CAPACITY);  // too dense for this path
  const int nq = min(nq_all, kQueue);
  for (int e0 = 0; e0 < nq * 8; e0 += kStage) {
    // exact test, staged in rounds so that any number of queued groups fits the staging arrays
    const int e1 = min(nq * 8, e0 + kStage);
    for (int e = e0 + threadIdx.x; e < e1; e += blockDim.x) {
      const uint32_t item = s_queue[e >> 3];
      const int r = r0 + int(item >> 8);
      const int c = (blockIdx.x * blockDim.x + int(item & 255u)) * 8 + (e & 7);
      if (c >= g.F) continue;
      const float xv = t16_to_float(x[1LL * l * g.layer_stride + 1LL * r * g.ld + c]);
      if (!(xv >= __ldg(theta + 1LL * l * g.sp + c))) continue;
      const int slot = atomicAdd(&s_n, 1);
      s_tok[slot] = r; s_col[slot] = l * col_pitch + c; s_val[slot] = xv;
    }
    __syncthreads();
    const int staged = s_n;
    if (threadIdx.x == 0) s_base = staged ? atomicAdd(n_ent, (unsigned long long)staged) : 0ULL;
    __syncthreads();
    for (int i = threadIdx.x; i < staged; i += blockDim.x) {
      const long long q = (long long)s_base + i;
      if (q < o.ent_cap) { o.ent_tok[q] = s_tok[i]; o.ent_col[q] = s_col[i]; o.ent_val[q] = s_val[i]; }
      else atomicCAS(status, STATUS_OK, STATUS_CAPACITY);
    }
    __syncthreads();
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
  }
}

// ------------------------------------------------------------------ 2d. per-token top-k (TokenTopK)
// Every token keeps its k largest z-scores over all layers' features (reference: torch.topk(dim=-1) + scatter_,
// clt/models/activations.py:121-124, ranking on the per-feature batch z-scores).  One CTA handles four tokens (so
// that the per-column statistics are loaded once for four rows) and finds each token's k-th largest key exactly
// with a three-round radix select over the 32-bit keys (11 + 11 + 10 bits, histograms in shared memory), then
// emits the entries above the cut and the lowest-index ties at the cut.  Output: exactly k entries per token at
// [token * k, token * k + k) of the entry list.
constexpr int kTokPerCta = 4;
constexpr int kTokBins = 2048;
constexpr int kTieCap = 256;

struct TokenTopkShared {
  uint32_t hist[kTokPerCta][kTokBins];
  uint32_t prefix[kTokPerCta], mask[kTokPerCta];
  unsigned int need[kTokPerCta];
  int emitted[kTokPerCta];
  int nties[kTokPerCta];
  int tie_col[kTokPerCta][kTieCap];
  float tie_val[kTokPerCta][kTieCap];
};

template <typename Fn>
__device__ __forceinline__ void token_rows_scan(const t16* __restrict__ x, const float* __restrict__ mean,
                                                const float* __restrict__ rstd, const ScanGeom& g, int tok0, int ntok, Fn fn) {
  for (int l = 0; l < g.L; ++l) {
    for (int c0 = threadIdx.x * 8; c0 < g.F; c0 += blockDim.x * 8) {
      float mu[8], rs[8];
      load_cols8(mean + 1LL * l * g.sp + c0, mu);
      load_cols8(rstd + 1LL * l * g.sp + c0, rs);
      uint4 v[kTokPerCta];
#pragma unroll
      for (int t = 0; t < kTokPerCta; ++t)
        v[t] = t < ntok ? __ldg(reinterpret_cast<const uint4*>(x + 1LL * l * g.layer_stride + 1LL * (tok0 + t) * g.ld + c0)) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int t = 0; t < kTokPerCta; ++t) {
        if (t >= ntok) break;
        const uint32_t u[4] = {v[t].x, v[t].y, v[t].z, v[t].w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xv = (j & 1) ? t16_hi(u[j >> 1]) : t16_lo(u[j >> 1]);
          fn(t, l, c0 + j, xv, float_to_key((xv - mu[j]) * rs[j]));
        }
      }
    }
  }
}

__global__ void __launch_bounds__(256) token_topk_kernel(const t16* __restrict__ x, const float* __restrict__ mean,
                                                           const float* __restrict__ rstd, ScanGeom g, int col_pitch, int f_valid, int k,
                                                           long long* __restrict__ ctl, Lists o, int* __restrict__ status, int only_marked) {
  if (chain_wait()) return;
  chain_release();
  extern __shared__ uint8_t tk_smem[];
  TokenTopkShared* sh = reinterpret_cast<TokenTopkShared*>(tk_smem);
  const int tok0 = blockIdx.x * kTokPerCta;
  const int ntok = min(kTokPerCta, g.B - tok0);
  const int tid = threadIdx.x;
  if (only_marked) {  // every thread reads the marks before any of them is overwritten
    bool any = false;
    for (int t = 0; t < ntok; ++t) any |= o.ent_tok[1LL * (tok0 + t) * k] < 0;
    if (!__syncthreads_or(any)) return;
  }
  if (tid < kTokPerCta) { sh->prefix[tid] = 0; sh->mask[tid] = 0; sh->need[tid] = (unsigned int)k; sh->emitted[tid] = 0; sh->nties[tid] = 0; }
  if (blockIdx.x == 0 && tid == 0) ctl[CTL_NUM_ENTRIES] = 1LL * g.B * k;
  // ---- exact k-th largest key per token: radix select, most significant digits first
  const int shifts[3] = {21, 10, 0};
  const int widths[3] = {11, 11, 10};
  for (int round = 0; round < 3; ++round) {
    const int shift = shifts[round];
    const uint32_t nb = 1u << widths[round];
    for (int i = tid; i < kTokPerCta * kTokBins; i += blockDim.x) (&sh->hist[0][0])[i] = 0;
    __syncthreads();
    token_rows_scan(x, mean, rstd, g, tok0, ntok, [&](int t, int, int c, float, uint32_t key) {
      if (c < f_valid && (key & sh->mask[t]) == sh->prefix[t]) atomicAdd(&sh->hist[t][(key >> shift) & (nb - 1u)], 1u);
    });
    __syncthreads();
    if (tid < ntok) {
      // digit that holds the need-th largest remaining key (counting from the top)
      unsigned int run = 0, need = sh->need[tid];
      int digit = 0;
      for (int b = int(nb) - 1; b >= 0; --b) {
        const unsigned int c = sh->hist[tid][b];
        if (run + c >= need) { digit = b; break; }
        run += c;
      }
      sh->need[tid] = need - run;
      sh->prefix[tid] |= uint32_t(digit) << shift;
      sh->mask[tid] |= (nb - 1u) << shift;
    }
    __syncthreads();
  }
  // prefix[t] is now the cut key T of token t, need[t] the number of keys equal to T that are kept
  token_rows_scan(x, mean, rstd, g, tok0, ntok, [&](int t, int l, int c, float xv, uint32_t key) {
    const uint32_t T = sh->prefix[t];
    if (c >= f_valid) return;  // padding columns of a shard take no part
    if (key > T) {
      const int slot = atomicAdd(&sh->emitted[t], 1);
      if (slot < k) {
        const long long q = 1LL * (tok0 + t) * k + slot;
        o.ent_tok[q] = tok0 + t; o.ent_col[q] = l * col_pitch + c; o.ent_val[q] = xv;
      }
    } else if (key == T) {
      const int i = atomicAdd(&sh->nties[t], 1);
      if (i < kTieCap) { sh->tie_col[t][i] = l * col_pitch + c; sh->tie_val[t][i] = xv; }
    }
  });
  __syncthreads();
  // ---- ties at the cut: the lowest flat indices first (l * col_pitch + c grows with the reference's column order)
  for (int t = 0; t < ntok; ++t) {
    const int n = sh->nties[t];
    const int need = int(sh->need[t]);
    const int above = sh->emitted[t];
    if (n > kTieCap && need < n) {
      if (tid == 0) atomicCAS(status, STATUS_OK, STATUS_TIE_OVERFLOW);
      continue;
    }
    if (tid == 0 && above + need != k) atomicCAS(status, STATUS_OK, STATUS_SELECT_RANGE);
    for (int i = tid; i < min(n, kTieCap); i += blockDim.x) {
      const int ci = sh->tie_col[t][i];
      int rank = 0;
      for (int j = 0; j < min(n, kTieCap); ++j) rank += sh->tie_col[t][j] < ci;
      if (rank < need && above + rank < k) {
        const long long q = 1LL * (tok0 + t) * k + above + rank;
        o.ent_tok[q] = tok0 + t; o.ent_col[q] = ci; o.ent_val[q] = sh->tie_val[t][i];
      }
    }
  }
}

// The same selection with one scan of the rows instead of four.  A bound from below for a token's k-th largest key comes from
// a sample of its columns (every step-th block of 2048): every thread keeps the largest key of kTkSlots interleaved parts of
// the sample, and the k-th largest of those kTkMaxima maxima is reached by at least k elements.  One scan then collects what
// is at or above the bound (about step * k elements) and the exact cut is searched in that short list, whose 64-bit words
// (key, inverted column) are distinct and order ties by the lowest index.  A token whose list overflows is marked by a token
// index of -1 in its first entry, and the radix kernel above takes it.  TPC tokens per CTA share the loads of the column
// statistics.
constexpr int kTkSlots = 4;
constexpr int kTkThreads = 256;
constexpr int kTkMaxima = kTkSlots * kTkThreads;
constexpr int kTkList = 2048;

template <int TPC>
struct TokenListShared {
  union {
    uint32_t maxima[TPC][kTkMaxima];
    unsigned long long list[TPC][kTkList];
  } u;
  uint32_t bound[TPC];
  int n[TPC];
  unsigned long long cut[TPC];
  int out[TPC];
};

template <int TPC, typename Fn>
__device__ __forceinline__ void token_keys_scan(const t16* __restrict__ x, const float* __restrict__ mean, const float* __restrict__ rstd, const ScanGeom& g,
                                                int tok0, int ntok, int groups, int step, Fn fn) {
  // groups of 8 columns, counted over all layers; 8 elements of TPC tokens per thread and step
  const int per_layer = g.F / 8;
  int it = 0;
  for (int q = int(threadIdx.x); q < groups; q += kTkThreads * step, ++it) {
    const int l = q / per_layer, c0 = (q - l * per_layer) * 8;
    float mu[8], rs[8];
    load_cols8(mean + 1LL * l * g.sp + c0, mu);
    load_cols8(rstd + 1LL * l * g.sp + c0, rs);
    uint4 v[TPC];
#pragma unroll
    for (int t = 0; t < TPC; ++t)
      v[t] = t < ntok ? __ldg(reinterpret_cast<const uint4*>(x + 1LL * l * g.layer_stride + 1LL * (tok0 + t) * g.ld + c0)) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int t = 0; t < TPC; ++t) {
      if (t < ntok) {
        const uint32_t u[4] = {v[t].x, v[t].y, v[t].z, v[t].w};
        uint32_t key[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) key[j] = float_to_key((((j & 1) ? t16_hi(u[j >> 1]) : t16_lo(u[j >> 1])) - mu[j]) * rs[j]);
        fn(t, l, c0, it, key);
      }
    }
  }
}

template <int TPC>
__global__ void __launch_bounds__(kTkThreads) token_topk_list_kernel(const t16* __restrict__ x, const float* __restrict__ mean, const float* __restrict__ rstd,
                                                                     ScanGeom g, int col_pitch, int f_valid, int k, int step, long long* __restrict__ ctl, Lists o) {
  if (chain_wait()) return;
  chain_release();
  extern __shared__ __align__(16) uint8_t tl_smem[];
  TokenListShared<TPC>* sh = reinterpret_cast<TokenListShared<TPC>*>(tl_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tok0 = blockIdx.x * TPC;
  const int ntok = min(TPC, g.B - tok0);
  if (blockIdx.x == 0 && tid == 0) ctl[CTL_NUM_ENTRIES] = 1LL * g.B * k;
  const int groups = g.L * (g.F / 8);
  // ---- bound from the sample
  uint32_t best[TPC][kTkSlots];
#pragma unroll
  for (int t = 0; t < TPC; ++t)
#pragma unroll
    for (int i = 0; i < kTkSlots; ++i) best[t][i] = 0;
  token_keys_scan<TPC>(x, mean, rstd, g, tok0, ntok, groups, step, [&](int t, int, int c0, int it, const uint32_t (&key)[8]) {
    uint32_t m = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) m = max(m, c0 + j < f_valid ? key[j] : 0u);
    const int slot = it % kTkSlots;
#pragma unroll
    for (int i = 0; i < kTkSlots; ++i)
      if (i == slot) best[t][i] = max(best[t][i], m);
  });
#pragma unroll
  for (int t = 0; t < TPC; ++t)
#pragma unroll
    for (int i = 0; i < kTkSlots; ++i) sh->u.maxima[t][i * kTkThreads + tid] = best[t][i];
  __syncthreads();
  if (warp < ntok) {
    // largest key with zero low bits that at least k maxima reach
    uint32_t bound = 0;
    for (int bit = 31; bit >= 12; --bit) {
      const uint32_t trial = bound | (1u << bit);
      int cnt = 0;
      for (int i = lane; i < kTkMaxima; i += 32) cnt += sh->u.maxima[warp][i] >= trial ? 1 : 0;
      if (__reduce_add_sync(0xFFFFFFFFu, cnt) >= k) bound = trial;
    }
    if (lane == 0) { sh->bound[warp] = bound; sh->n[warp] = 0; sh->out[warp] = 0; }
  }
  __syncthreads();
  uint32_t bound[TPC];
#pragma unroll
  for (int t = 0; t < TPC; ++t) bound[t] = t < ntok ? sh->bound[t] : 0xFFFFFFFFu;
  __syncthreads();
  // ---- one scan: everything at or above the bound
  token_keys_scan<TPC>(x, mean, rstd, g, tok0, ntok, groups, 1, [&](int t, int l, int c0, int, const uint32_t (&key)[8]) {
    uint32_t m = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) m = max(m, key[j]);
    if (m < bound[t]) return;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (key[j] >= bound[t] && c0 + j < f_valid) {  // padding columns of a shard take no part
        const int slot = atomicAdd(&sh->n[t], 1);
        if (slot < kTkList) sh->u.list[t][slot] = ((unsigned long long)key[j] << 32) | (0xFFFFFFFFu - (unsigned int)(l * col_pitch + c0 + j));
      }
    }
  });
  __syncthreads();
  // ---- exact cut of the list: the largest word that exactly k words reach (one warp per token)
  if (warp < ntok) {
    const int n = sh->n[warp];
    const bool lost = n > kTkList || n < k;
    if (lost && lane == 0) o.ent_tok[1LL * (tok0 + warp) * k] = -1;
    if (!lost) {
      unsigned long long cut = 0;
      for (int bit = 63; bit >= 0; --bit) {
        const unsigned long long trial = cut | (1ULL << bit);
        int cnt = 0;
        for (int i = lane; i < n; i += 32) cnt += sh->u.list[warp][i] >= trial ? 1 : 0;
        cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
        if (cnt >= k) cut = trial;
        if (cnt == k) break;
      }
      const long long base = 1LL * (tok0 + warp) * k;
      int done = 0;
      for (int i0 = 0; i0 < n; i0 += 32) {
        const int i = i0 + lane;
        const bool keep = i < n && sh->u.list[warp][i] >= cut;
        const unsigned ball = __ballot_sync(0xFFFFFFFFu, keep);
        if (keep) {
          const int slot = done + __popc(ball & ((1u << lane) - 1u));
          const int col = int(0xFFFFFFFFu - (unsigned int)(sh->u.list[warp][i] & 0xFFFFFFFFULL));
          const int l = col / col_pitch, c = col - l * col_pitch;
          if (slot < k) {
            o.ent_tok[base + slot] = tok0 + warp;
            o.ent_col[base + slot] = col;
            o.ent_val[base + slot] = t16_to_float(x[1LL * l * g.layer_stride + 1LL * (tok0 + warp) * g.ld + c]);
          }
        }
        done += __popc(ball);
      }
    }
  }
}

// The list form for large matrices, in four passes.  The kernel above gives a CTA one to four tokens and reads the column statistics once
// per such group: 64 bytes of statistics per 16 bytes of a token, a chain of a hundred dependent loads, 350 us at 6 x 2048 x 32768, k = 64;
// the four passes take 302 (sample 46, bound 29, collect 206, cut 22).  Here a thread owns eight columns and walks 64 tokens, as the histogram scan does:
//   sample   maxima of groups of eight columns, every eighth run of 32 groups, one word per group and token
//   bound    per token: a key that at least k of its maxima reach
//   collect  one scan: what reaches the bound goes to the token's list (about 8 k words)
//   cut      per token (one warp): the exact cut of the list, as above; a token whose list overflows goes to the radix kernel
constexpr int kWideRows = 64;
constexpr int kWideMaxima = 4096;   // per token
constexpr int kWideQueue = 2048;    // groups of a tile that pass the coarse test, numbered with 16 bits
constexpr int kWideStep = 8;        // one run of groups in kWideStep is sampled: a list has about kWideStep * k words
struct WideTopk {
  int* n;                        // [B] list lengths (zeroed by the caller)
  uint32_t* bound;               // [B]
  uint32_t* maxima;              // [B][ng]
  unsigned long long* list;      // [B][cap] (key << 32 | inverted column)
  int ng, cap, groups;  // maxima per token (0: another form), room of a list, groups of eight columns
};

__device__ __forceinline__ float t16_of(const uint4& v, int j) {
  const uint32_t u = j < 2 ? v.x : (j < 4 ? v.y : (j < 6 ? v.z : v.w));
  return (j & 1) ? t16_hi(u) : t16_lo(u);
}

__global__ void __launch_bounds__(256) token_sample_kernel(const t16* __restrict__ x, const float* __restrict__ mean, const float* __restrict__ rstd, ScanGeom g,
                                                             int f_valid, WideTopk wt) {
  if (chain_wait()) return;
  chain_release();
  const int sg = blockIdx.x * 256 + threadIdx.x;  // < ng, a multiple of 256
  const int q = (sg >> 5) * 32 * kWideStep + (sg & 31);  // runs of 32 groups: short enough that a sample meets every layer
  const int r0 = blockIdx.y * kWideRows, r1 = min(g.B, r0 + kWideRows);
  if (q >= wt.groups) {
    for (int r = r0; r < r1; ++r) wt.maxima[1LL * r * wt.ng + sg] = 0u;
    return;
  }
  const int per_layer = g.F / 8;
  const int l = q / per_layer, c0 = (q - l * per_layer) * 8;
  float mu[8], rs[8];
  load_cols8(mean + 1LL * l * g.sp + c0, mu);
  load_cols8(rstd + 1LL * l * g.sp + c0, rs);
  const int nvalid = f_valid - c0;
  const t16* base = x + 1LL * l * g.layer_stride + c0;
  for (int rb = r0; rb < r1; rb += 8) {
    uint4 v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __ldg(reinterpret_cast<const uint4*>(base + 1LL * min(rb + k, r1 - 1) * g.ld));
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if (rb + k >= r1) break;
      float m = -INFINITY;  // a NaN, which sorts above everything, only makes the bound smaller here
#pragma unroll
      for (int j = 0; j < 8; ++j) m = fmaxf(m, j < nvalid ? (t16_of(v[k], j) - mu[j]) * rs[j] : -INFINITY);
      wt.maxima[1LL * (rb + k) * wt.ng + sg] = m == -INFINITY ? 0u : float_to_key(m);
    }
  }
}

__global__ void __launch_bounds__(256) token_bound_kernel(WideTopk wt, int k, long long* __restrict__ ctl, long long n_entries) {
  if (chain_wait()) return;
  chain_release();
  __shared__ int total[2];
  const int tok = blockIdx.x;
  if (tok == 0 && threadIdx.x == 0) ctl[CTL_NUM_ENTRIES] = n_entries;
  uint32_t mine[kWideMaxima / 256];
#pragma unroll
  for (int i = 0; i < kWideMaxima / 256; ++i) {
    const int at = i * 256 + threadIdx.x;
    mine[i] = at < wt.ng ? wt.maxima[1LL * tok * wt.ng + at] : 0u;
  }
  if (threadIdx.x < 2) total[threadIdx.x] = 0;
  __syncthreads();
  uint32_t bound = 0;  // largest key with zero low bits that at least k maxima reach
  int turn = 0;
#pragma unroll 1
  for (int bit = 31; bit >= 12; --bit, turn ^= 1) {
    const uint32_t trial = bound | (1u << bit);
    int cnt = 0;
#pragma unroll
    for (int i = 0; i < kWideMaxima / 256; ++i) cnt += mine[i] >= trial ? 1 : 0;
    cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
    if ((threadIdx.x & 31) == 0 && cnt != 0) atomicAdd(&total[turn], cnt);
    __syncthreads();
    if (total[turn] >= k) bound = trial;
    if (threadIdx.x == 0) total[turn ^ 1] = 0;
    __syncthreads();
  }
  if (threadIdx.x == 0) wt.bound[tok] = bound;
}

__global__ void __launch_bounds__(256, 4) token_collect_kernel(const t16* __restrict__ x, const float* __restrict__ mean, const float* __restrict__ rstd, ScanGeom g,
                                                              int col_pitch, int f_valid, WideTopk wt) {
  if (chain_wait()) return;
  chain_release();
  __shared__ uint16_t queue[kWideQueue];
  __shared__ float z_scaled[kWideRows];
  __shared__ uint32_t bound[kWideRows];
  __shared__ int s_q;
  const int l = blockIdx.z, c0 = (blockIdx.x * 256 + int(threadIdx.x)) * 8;
  const int r0 = blockIdx.y * kWideRows, r1 = min(g.B, r0 + kWideRows);
  constexpr float kSlack = 1.f / 256.f;
  if (threadIdx.x < kWideRows) {
    const uint32_t b = r0 + int(threadIdx.x) < r1 ? wt.bound[r0 + threadIdx.x] : 0xFFFFFFFFu;
    const float z = key_to_float(b);  // NaN for a bound of 0: everything passes
    bound[threadIdx.x] = b;
    z_scaled[threadIdx.x] = z - kSlack * fabsf(z);
  }
  if (threadIdx.x == 0) s_q = 0;
  __syncthreads();
  if (c0 < g.F) {
    // A coarse test in the input's own format (one packed compare per two elements, one FMA per column) lets through what the exact test may
    // accept: z >= z_b needs x >= mean + z_b / rstd, and the right side, lowered by 2^-8 of its terms, stays below that after
    // rounding to 16 bits.  "Not below" rather than "at or above": a NaN, in the element or in a column's statistics, is left to the
    // exact test, where it sorts above everything.
    float low[8], spread[8];
    {
      float mu[8], rs[8];
      load_cols8(mean + 1LL * l * g.sp + c0, mu);
      load_cols8(rstd + 1LL * l * g.sp + c0, rs);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        low[j] = mu[j] - fmaf(kSlack, fabsf(mu[j]), kT16Max < 1e5f ? 1e-7f : 1e-30f);  // fp16: below its smallest step
        spread[j] = __fdividef(1.f, rs[j]);
      }
    }
    const t16* base = x + 1LL * l * g.layer_stride + c0;
    for (int rb = r0; rb < r1; rb += 8) {
      uint4 v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = __ldcs(reinterpret_cast<const uint4*>(base + 1LL * min(rb + k, r1 - 1) * g.ld));
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float z = z_scaled[min(rb + k, r1 - 1) - r0];
        uint32_t thr[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) thr[j] = pack_t16x2(fmaf(z, spread[2 * j], low[2 * j]), fmaf(z, spread[2 * j + 1], low[2 * j + 1]));
        const uint32_t hit = t16x2_not_below_mask(v[k].x, thr[0]) | t16x2_not_below_mask(v[k].y, thr[1]) | t16x2_not_below_mask(v[k].z, thr[2]) |
                             t16x2_not_below_mask(v[k].w, thr[3]);
        if (hit != 0u && rb + k < r1) {
          const int slot = atomicAdd(&s_q, 1);
          if (slot < kWideQueue) queue[slot] = uint16_t((uint32_t(rb + k - r0) << 8) | threadIdx.x);
        }
      }
    }
  }
  __syncthreads();
  const int nq = s_q;
  if (nq > kWideQueue) {  // lost groups: the tokens of this tile go to the radix kernel
    if (int(threadIdx.x) < r1 - r0) atomicMax(&wt.n[r0 + threadIdx.x], 1 << 28);
    return;
  }
  // Four elements per thread and round: each is a load of the element, a test and a trip to its token's counter, one after the other.  One at a time
  // took longer than reading the tile (6 x 2048 x 32768, k = 64: 207 us, DRAM at 54 %).
  for (int e0 = threadIdx.x; e0 < nq * 8; e0 += 4 * 256) {
    int r[4], c[4], slot[4];
    uint32_t key[4];
    bool in[4];
    float xv[4], mu[4], rs[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + 256 * u;
      const uint32_t item = e < nq * 8 ? queue[e >> 3] : 0u;
      r[u] = int(item >> 8);
      c[u] = (blockIdx.x * 256 + int(item & 255u)) * 8 + (e & 7);
      in[u] = e < nq * 8 && c[u] < f_valid && c[u] < g.F;  // padding columns of a shard take no part
      xv[u] = in[u] ? t16_to_float(x[1LL * l * g.layer_stride + 1LL * (r0 + r[u]) * g.ld + c[u]]) : 0.f;
      mu[u] = in[u] ? __ldg(mean + 1LL * l * g.sp + c[u]) : 0.f;
      rs[u] = in[u] ? __ldg(rstd + 1LL * l * g.sp + c[u]) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      key[u] = float_to_key((xv[u] - mu[u]) * rs[u]);
      in[u] = in[u] && key[u] >= bound[r[u]];
      slot[u] = in[u] ? atomicAdd(&wt.n[r0 + r[u]], 1) : 0;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (in[u] && slot[u] >= 0 && slot[u] < wt.cap)
        wt.list[1LL * (r0 + r[u]) * wt.cap + slot[u]] = ((unsigned long long)key[u] << 32) | (0xFFFFFFFFu - (unsigned int)(l * col_pitch + c[u]));
  }
}

// W: words per lane (cap <= 32 W).
template <int W>
__global__ void __launch_bounds__(128) token_cut_kernel(const t16* __restrict__ x, ScanGeom g, int col_pitch, int k, WideTopk wt, Lists o) {
  if (chain_wait()) return;
  chain_release();
  const int tok = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (tok >= g.B) return;
  const int n = wt.n[tok];
  if (n > wt.cap || n < k) {
    if (lane == 0) o.ent_tok[1LL * tok * k] = -1;  // for the radix kernel
    return;
  }
  unsigned long long w[W];
#pragma unroll
  for (int i = 0; i < W; ++i) w[i] = i * 32 + lane < n ? wt.list[1LL * tok * wt.cap + i * 32 + lane] : 0ULL;
  unsigned long long cut = 0;  // the largest word that exactly k words reach
#pragma unroll 1
  for (int bit = 63; bit >= 0; --bit) {
    const unsigned long long trial = cut | (1ULL << bit);
    int cnt = 0;
#pragma unroll
    for (int i = 0; i < W; ++i) cnt += w[i] >= trial ? 1 : 0;
    cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
    if (cnt >= k) cut = trial;
    if (cnt == k) break;
  }
  const long long out = 1LL * tok * k;
  int done = 0;
#pragma unroll
  for (int i = 0; i < W; ++i) {
    const bool keep = i * 32 + lane < n && w[i] >= cut;
    const unsigned ball = __ballot_sync(0xFFFFFFFFu, keep);
    const int slot = done + __popc(ball & ((1u << lane) - 1u));
    if (keep && slot < k) {
      const int col = int(0xFFFFFFFFu - (unsigned int)(w[i] & 0xFFFFFFFFULL));
      const int l = col / col_pitch, c = col - l * col_pitch;
      o.ent_tok[out + slot] = tok;
      o.ent_col[out + slot] = col;
      o.ent_val[out + slot] = t16_to_float(x[1LL * l * g.layer_stride + 1LL * tok * g.ld + c]);
    }
    done += __popc(ball);
  }
}

// ------------------------------------------------------------------ 3b. split the pool at the threshold bin
// Runs instead of the full compaction pass when the tracked range contained the cut.
// Four elements per thread in flight, and the warp, not the element, takes places at the two shared counters: 47 -> 24 us for the 1.6
// million entries of 8192 tokens x 196608 columns, 29 -> 20 for 0.8 million of 4096 x 294912.
constexpr int kClassifyInFlight = 4;
__global__ void __launch_bounds__(256) classify_pool_kernel(Pool pool, long long* __restrict__ ctl, Lists o,
                                                              int* __restrict__ status) {
  if (chain_wait()) return;
  chain_release();
  if (ctl[CTL_RETRY] != 0) return;
  const uint32_t tbin = uint32_t(ctl[CTL_BIN]);
  const uint32_t key_lo = uint32_t(ctl[CTL_KEY_LO]);
  const int shift = int(ctl[CTL_SHIFT]);
  unsigned long long* n_ent = reinterpret_cast<unsigned long long*>(ctl + CTL_NUM_ENTRIES);
  unsigned long long* n_cand = reinterpret_cast<unsigned long long*>(ctl + CTL_NUM_CAND);
  const long long n = min((long long)(*pool.count), pool.cap);
  // every CTA owns one contiguous slice of the pool: count, reserve once per list, then place
  const long long per_cta = (n + gridDim.x - 1) / gridDim.x;
  const long long lo = blockIdx.x * per_cta, hi = min(n, lo + per_cta);
  __shared__ int cnt[2];
  __shared__ unsigned long long base[2];
  if (threadIdx.x < 2) cnt[threadIdx.x] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const auto bin_of = [&](long long i) { return min((pool.key[i] - key_lo) >> shift, uint32_t(kHistBins - 1)); };
  int my_ent = 0, my_cand = 0;
#pragma unroll 4
  for (long long i = lo + threadIdx.x; i < hi; i += blockDim.x) {
    const uint32_t bin = bin_of(i);
    my_ent += bin > tbin;
    my_cand += bin == tbin;
  }
  my_ent = __reduce_add_sync(0xFFFFFFFFu, my_ent);
  my_cand = __reduce_add_sync(0xFFFFFFFFu, my_cand);
  if (lane == 0 && my_ent) atomicAdd(&cnt[0], my_ent);
  if (lane == 0 && my_cand) atomicAdd(&cnt[1], my_cand);
  __syncthreads();
  if (threadIdx.x == 0) {
    base[0] = cnt[0] ? atomicAdd(n_ent, (unsigned long long)cnt[0]) : 0ULL;
    base[1] = cnt[1] ? atomicAdd(n_cand, (unsigned long long)cnt[1]) : 0ULL;
    cnt[0] = 0; cnt[1] = 0;
  }
  __syncthreads();
  for (long long i0 = lo; i0 < hi; i0 += kClassifyInFlight * blockDim.x) {
    uint32_t key[kClassifyInFlight], bin[kClassifyInFlight], ent[kClassifyInFlight], cand[kClassifyInFlight];
    int tok[kClassifyInFlight], col[kClassifyInFlight];
    float val[kClassifyInFlight];
#pragma unroll
    for (int u = 0; u < kClassifyInFlight; ++u) {
      const long long i = i0 + u * blockDim.x + threadIdx.x;
      const bool in = i < hi;
      key[u] = in ? pool.key[i] : 0u;
      bin[u] = in ? min((key[u] - key_lo) >> shift, uint32_t(kHistBins - 1)) : 0u;
      ent[u] = __ballot_sync(0xFFFFFFFFu, in && bin[u] > tbin);
      cand[u] = __ballot_sync(0xFFFFFFFFu, in && bin[u] == tbin);
      if ((ent[u] | cand[u]) >> lane & 1u) { tok[u] = pool.tok[i]; col[u] = pool.col[i]; val[u] = pool.val[i]; }
    }
    // one reservation per warp and list for all of them
    int ents = 0, cands = 0;
#pragma unroll
    for (int u = 0; u < kClassifyInFlight; ++u) { ents += __popc(ent[u]); cands += __popc(cand[u]); }
    int at = 0;
    if (lane < 2 && (lane == 0 ? ents : cands) > 0) at = atomicAdd(&cnt[lane], lane == 0 ? ents : cands);
    long long q_ent = (long long)base[0] + __shfl_sync(0xFFFFFFFFu, at, 0), q_cand = (long long)base[1] + __shfl_sync(0xFFFFFFFFu, at, 1);
#pragma unroll
    for (int u = 0; u < kClassifyInFlight; ++u) {
      const uint32_t below = (1u << lane) - 1u;
      if (ent[u] >> lane & 1u) {
        const long long q = q_ent + __popc(ent[u] & below);
        if (q < o.ent_cap) { o.ent_tok[q] = tok[u]; o.ent_col[q] = col[u]; o.ent_val[q] = val[u]; }
        else atomicCAS(status, STATUS_OK, STATUS_CAPACITY);
      } else if (cand[u] >> lane & 1u) {
        const long long q = q_cand + __popc(cand[u] & below);
        if (q < o.cand_cap) { o.cand_key[q] = key[u]; o.cand_tok[q] = tok[u]; o.cand_col[q] = col[u]; o.cand_val[q] = val[u]; }
        else atomicCAS(status, STATUS_OK, STATUS_CAPACITY);
      }
      q_ent += __popc(ent[u]);
      q_cand += __popc(cand[u]);
    }
  }
}

// ------------------------------------------------------------------ 4. compaction

// Selected elements are staged in shared memory and appended with one global reservation per CTA and
// list: a single counter cannot absorb one atomic per selected element (hundreds of thousands per step).
constexpr int kStageCap = 1024;

__global__ void __launch_bounds__(256) compact_kernel(const t16* __restrict__ x, const float* __restrict__ mean,
                                                        const float* __restrict__ rstd, ScanGeom g, int col_pitch,
                                                        long long* __restrict__ ctl, Lists o, int* __restrict__ status,
                                                        int only_if_retry) {
  if (chain_wait()) return;
  chain_release();
  if (only_if_retry && ctl[CTL_RETRY] == 0) return;
  __shared__ int s_tok[kStageCap];
  __shared__ int s_col[kStageCap];
  __shared__ float s_val[kStageCap];
  __shared__ uint32_t s_key[kStageCap];  // 0 marks a definite entry, otherwise the candidate's key (never 0 here)
  __shared__ int s_n;
  __shared__ unsigned long long s_base_ent, s_base_cand;
  __shared__ int s_cnt_ent, s_cnt_cand;
  if (threadIdx.x == 0) { s_n = 0; s_cnt_ent = 0; s_cnt_cand = 0; }
  __syncthreads();
  const int l = blockIdx.z;
  const int c0 = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
  const uint32_t tbin = uint32_t(ctl[CTL_BIN]);
  const uint32_t key_lo = uint32_t(ctl[CTL_KEY_LO]);
  const int shift = int(ctl[CTL_SHIFT]);
  // smallest key that can matter: everything below the threshold bin is dropped with one compare
  const unsigned long long lo64 = (unsigned long long)key_lo + ((unsigned long long)tbin << shift);
  const uint32_t key_min = lo64 > 0xFFFFFFFFULL ? 0xFFFFFFFFu : uint32_t(lo64);
  const float z_min = key_min == 0u ? -INFINITY : key_to_float(key_min);
  unsigned long long* n_ent = reinterpret_cast<unsigned long long*>(ctl + CTL_NUM_ENTRIES);
  unsigned long long* n_cand = reinterpret_cast<unsigned long long*>(ctl + CTL_NUM_CAND);
  if (c0 < g.F) {
    float mu[8], rs[8];
    if (c0 + 8 <= g.F) {
      load_cols8(mean + 1LL * l * g.sp + c0, mu);
      load_cols8(rstd + 1LL * l * g.sp + c0, rs);
    } else {
      for (int j = 0; j < 8; ++j) {
        const bool in = c0 + j < g.F;
        mu[j] = in ? mean[1LL * l * g.sp + c0 + j] : 0.f;
        rs[j] = in ? rstd[1LL * l * g.sp + c0 + j] : 0.f;
      }
    }
    const int nvalid = min(8, g.F - c0);
    const int r0 = blockIdx.y * g.rows_per_block;
    const int r1 = min(g.B, r0 + g.rows_per_block);
    const t16* base = x + 1LL * l * g.layer_stride + c0;
    for (int rb = r0; rb < r1; rb += 4) {
      uint4 v[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int r = min(rb + k, r1 - 1);
        v[k] = __ldcs(reinterpret_cast<const uint4*>(base + 1LL * r * g.ld));
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int r = rb + k;
        const uint32_t u[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float xv = (j & 1) ? t16_hi(u[j >> 1]) : t16_lo(u[j >> 1]);
          const float z = (xv - mu[j]) * rs[j];
          if (!(z >= z_min) || j >= nvalid || r >= r1) continue;
          const uint32_t key = float_to_key(z);
          const uint32_t bin = min((key - key_lo) >> shift, uint32_t(kHistBins - 1));
          if (bin < tbin) continue;
          const bool is_ent = bin > tbin;
          const int slot = atomicAdd(&s_n, 1);
          if (slot < kStageCap) {
            s_tok[slot] = r; s_col[slot] = l * col_pitch + c0 + j; s_val[slot] = xv; s_key[slot] = is_ent ? 0u : key;
            atomicAdd(is_ent ? &s_cnt_ent : &s_cnt_cand, 1);
          } else if (is_ent) {  // staging full: append directly
            const unsigned long long p = atomicAdd(n_ent, 1ULL);
            if ((long long)p < o.ent_cap) { o.ent_tok[p] = r; o.ent_col[p] = l * col_pitch + c0 + j; o.ent_val[p] = xv; }
            else atomicCAS(status, STATUS_OK, STATUS_CAPACITY);
          } else {
            const unsigned long long p = atomicAdd(n_cand, 1ULL);
            if ((long long)p < o.cand_cap) { o.cand_key[p] = key; o.cand_tok[p] = r; o.cand_col[p] = l * col_pitch + c0 + j; o.cand_val[p] = xv; }
            else atomicCAS(status, STATUS_OK, STATUS_CAPACITY);
          }
        }
      }
    }
  }
  __syncthreads();
  const int staged = min(s_n, kStageCap);
  if (staged == 0) return;
  if (threadIdx.x == 0) {
    s_base_ent = s_cnt_ent ? atomicAdd(n_ent, (unsigned long long)s_cnt_ent) : 0ULL;
    s_base_cand = s_cnt_cand ? atomicAdd(n_cand, (unsigned long long)s_cnt_cand) : 0ULL;
    s_cnt_ent = 0; s_cnt_cand = 0;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < staged; i += blockDim.x) {
    const uint32_t key = s_key[i];
    if (key == 0u) {
      const unsigned long long p = s_base_ent + (unsigned long long)atomicAdd(&s_cnt_ent, 1);
      if ((long long)p < o.ent_cap) { o.ent_tok[p] = s_tok[i]; o.ent_col[p] = s_col[i]; o.ent_val[p] = s_val[i]; }
      else atomicCAS(status, STATUS_OK, STATUS_CAPACITY);
    } else {
      const unsigned long long p = s_base_cand + (unsigned long long)atomicAdd(&s_cnt_cand, 1);
      if ((long long)p < o.cand_cap) { o.cand_key[p] = key; o.cand_tok[p] = s_tok[i]; o.cand_col[p] = s_col[i]; o.cand_val[p] = s_val[i]; }
      else atomicCAS(status, STATUS_OK, STATUS_CAPACITY);
    }
  }
}

// ------------------------------------------------------------------ 5. exact cut inside the bin (one CTA)
constexpr int kGatherCap = 4096;   // candidates (all ranks together) that the one-round exact cut handles
constexpr int kGatherSlot = 4096;  // ... and per rank: 2 + 2 * 4096 words fit one exchange slot (8224 words)
struct FlatGeom {
  int col_pitch;        // local column pitch used in ent_col / cand_col
  int feat_offset;      // first global feature of this shard
  long long full_F;     // un-sharded features per layer
  long long row_width;  // L * full_F
};
__device__ __forceinline__ unsigned long long flat_index(const FlatGeom& fg, int tok, int col) {
  const int l = col / fg.col_pitch, f = col - l * fg.col_pitch;
  return (unsigned long long)tok * (unsigned long long)fg.row_width + (unsigned long long)l * fg.full_F + (unsigned long long)(fg.feat_offset + f);
}

// Picks the digit whose bucket contains the `need`-th element counting from the top (descending=true)
// or from the bottom (descending=false).  Writes the digit and the remaining need.
__device__ void pick_digit(const uint32_t* hist, int nb, bool descending, unsigned long long need, int* digit_out,
                           unsigned long long* need_out) {
  if (threadIdx.x == 0) {
    unsigned long long run = 0;
    int d = descending ? nb - 1 : 0;
    for (int i = 0; i < nb; ++i) {
      const int b = descending ? nb - 1 - i : i;
      const unsigned long long c = hist[b];
      if (run + c >= need) { d = b; break; }
      run += c;
      d = b;
    }
    *digit_out = d;
    *need_out = need - run;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(1024) refine_kernel(const uint32_t* __restrict__ cand_key, const int* __restrict__ cand_tok,
                                                        const int* __restrict__ cand_col, long long cand_cap,
                                                        FlatGeom fg, long long* __restrict__ ctl, Exchange ex,
                                                        int* __restrict__ status) {
  if (chain_wait()) return;
  if (ex.world <= 1) chain_release();  // else it waits for the other ranks below
  const int shift = int(ctl[CTL_SHIFT]);
  const uint32_t key_lo = uint32_t(ctl[CTL_KEY_LO]);  // bins are over (key - key_lo): refine on the same offset
  __shared__ uint32_t hist[kRefineBins];
  __shared__ int digit;
  __shared__ unsigned long long need;
  __shared__ int timeout;
  const int tid = threadIdx.x;
  long long n = ctl[CTL_NUM_CAND];
  if (n > cand_cap) n = cand_cap;
  if (tid == 0) { timeout = 0; need = (unsigned long long)ctl[CTL_NEED]; }
  __syncthreads();
  const uint32_t low_mask = shift >= 32 ? 0xFFFFFFFFu : ((1u << shift) - 1u);
  // ---- fast path: one all-gather of the candidates of the threshold bin, exact cut found locally.
  // A candidate travels as one 64-bit word: (low key bits << 45) | (2^45 - 1 - flat index), so that a larger word
  // ranks first and, among equal keys, the lowest flat index does.  Every rank sorts out the same cut from the
  // same words.  Bins with more candidates than the gather holds (heavy ties) take the radix rounds below.
  {
    __shared__ unsigned long long comp[kGatherCap];
    __shared__ int total_s, fits_s;
    constexpr unsigned long long kFlatMask = (1ULL << 45) - 1ULL;
    const bool local_fits = n <= kGatherSlot && shift <= 19;
    const int world = ex.world <= 1 ? 1 : ex.world;
    // own candidates -> comp[0 .. n) (single rank) or through the exchange area
    if (world == 1) {
      if (tid == 0) { total_s = int(n); fits_s = (local_fits && n <= kGatherCap) ? 1 : 0; }
      __syncthreads();
      if (fits_s)
        for (long long i = tid; i < n; i += 1024)
          comp[i] = ((unsigned long long)((cand_key[i] - key_lo) & low_mask) << 45) | (kFlatMask - flat_index(fg, cand_tok[i], cand_col[i]));
    } else {
      // message: word 0 = count (0xFFFFFFFF: does not fit), then the 64-bit words
      uint32_t* msg = reinterpret_cast<uint32_t*>(comp);
      if (tid == 0) { msg[0] = local_fits ? uint32_t(n) : 0xFFFFFFFFu; msg[1] = 0; }
      if (local_fits)
        for (long long i = tid; i < n; i += 1024)
          comp[1 + i] = ((unsigned long long)((cand_key[i] - key_lo) & low_mask) << 45) | (kFlatMask - flat_index(fg, cand_tok[i], cand_col[i]));
      __syncthreads();
      if (!exchange_gather(ex, 2, msg, local_fits ? 2 + 2 * int(n) : 2, &timeout)) {
        if (tid == 0) atomicCAS(status, STATUS_OK, STATUS_WAIT_TIMEOUT);
        return;
      }
      if (tid == 0) {
        long long tot = 0;
        bool ok = true;
        for (int q = 0; q < world; ++q) {
          const uint32_t c = exchange_slot(ex, 2, q)[0];
          if (c == 0xFFFFFFFFu) ok = false; else tot += c;
        }
        fits_s = (ok && tot <= kGatherCap) ? 1 : 0;
        total_s = int(tot < kGatherCap ? tot : kGatherCap);
      }
      __syncthreads();
      if (fits_s) {
        int base = 0;
        for (int q = 0; q < world; ++q) {
          const uint32_t* slot = exchange_slot(ex, 2, q);
          const int c = int(slot[0]);
          const unsigned long long* src = reinterpret_cast<const unsigned long long*>(slot) + 1;
          for (int i = tid; i < c; i += 1024) comp[base + i] = src[i];
          base += c;
        }
      }
    }
    __syncthreads();
    if (fits_s) {
      const int G = total_s;
      const unsigned long long want = need;  // the want-th largest word is the cut
      // bitonic sort of the words in shared memory, descending (the words are distinct; zero pads the power of two)
      int P = 1;
      while (P < G) P <<= 1;
      for (int i = G + tid; i < P; i += 1024) comp[i] = 0ULL;
      __syncthreads();
      for (int size = 2; size <= P; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
          for (int t = tid; t < P / 2; t += 1024) {
            const int lo = 2 * t - (t & (stride - 1)), hi = lo + stride;
            const unsigned long long a = comp[lo], b = comp[hi];
            const bool descending = (lo & size) == 0;
            if (descending ? a < b : a > b) { comp[lo] = b; comp[hi] = a; }
          }
          __syncthreads();
        }
      }
      if (tid == 0) {
        if (want == 0 || want > (unsigned long long)G) {
          atomicCAS(status, STATUS_OK, STATUS_SELECT_RANGE);
        } else {
          const unsigned long long cutw = comp[want - 1];
          ctl[CTL_CUT_KEY] = (long long)(cutw >> 45);
          ctl[CTL_TIE_MODE] = 1;
          ctl[CTL_CUT_FLAT] = (long long)(kFlatMask - (cutw & kFlatMask));
        }
      }
      return;
    }
  }
  // ---- key cut: radix passes over the low `shift` bits, 9 bits at a time, most significant first.
  uint32_t prefix = 0, prefix_mask = 0;
  int round = 3;  // rounds 0 and 1 belong to the two histogram passes, round 2 to the candidate gather

  for (int hi = shift; hi > 0; hi -= 9, ++round) {
    const int lo = max(hi - 9, 0);
    const int nb = 1 << (hi - lo);
    for (int i = tid; i < kRefineBins; i += 1024) hist[i] = 0;
    __syncthreads();
    for (long long i = tid; i < n; i += 1024) {
      const uint32_t k = (cand_key[i] - key_lo) & low_mask;
      if ((k & prefix_mask) == prefix) atomicAdd(&hist[(k >> lo) & (nb - 1)], 1u);
    }
    __syncthreads();
    if (!exchange_sum(ex, round, hist, kRefineBins, &timeout)) {
      if (tid == 0) atomicCAS(status, STATUS_OK, STATUS_WAIT_TIMEOUT);
      return;
    }
    unsigned long long cur = need;
    __syncthreads();
    pick_digit(hist, nb, true, cur, &digit, &need);
    prefix |= uint32_t(digit) << lo;
    prefix_mask |= uint32_t(nb - 1) << lo;
    __syncthreads();
  }
  // All candidates share the bits above `shift`; recover them from the bin.  `prefix` now holds the low
  // bits of the cut key T and `need` how many keys equal to T must be kept.
  // ---- ties: count keys == T (global), then cut by flat index if only part of them is kept.
  for (int i = tid; i < kRefineBins; i += 1024) hist[i] = 0;
  __syncthreads();
  unsigned int local_ties = 0;
  for (long long i = tid; i < n; i += 1024) local_ties += (((cand_key[i] - key_lo) & low_mask) == prefix) ? 1u : 0u;
  if (local_ties) atomicAdd(&hist[0], local_ties);
  __syncthreads();
  if (!exchange_sum(ex, round++, hist, kRefineBins, &timeout)) {
    if (tid == 0) atomicCAS(status, STATUS_OK, STATUS_WAIT_TIMEOUT);
    return;
  }
  const unsigned long long ties = hist[0];
  __syncthreads();
  unsigned long long flat_prefix = 0, flat_mask = 0;
  const bool partial = need < ties;
  if (partial) {
    // the `need` smallest flat indices among the ties: radix passes over 45 bits, 9 at a time
    for (int hi = 45; hi > 0; hi -= 9, ++round) {
      const int lo = hi - 9;
      for (int i = tid; i < kRefineBins; i += 1024) hist[i] = 0;
      __syncthreads();
      for (long long i = tid; i < n; i += 1024) {
        if (((cand_key[i] - key_lo) & low_mask) != prefix) continue;
        const unsigned long long fl = flat_index(fg, cand_tok[i], cand_col[i]);
        if ((fl & flat_mask) == flat_prefix) atomicAdd(&hist[(fl >> lo) & 511ULL], 1u);
      }
      __syncthreads();
      if (!exchange_sum(ex, round, hist, kRefineBins, &timeout)) {
        if (tid == 0) atomicCAS(status, STATUS_OK, STATUS_WAIT_TIMEOUT);
        return;
      }
      unsigned long long cur = need;
      __syncthreads();
      pick_digit(hist, 512, false, cur, &digit, &need);
      flat_prefix |= (unsigned long long)digit << lo;
      flat_mask |= 511ULL << lo;
      __syncthreads();
    }
  }
  if (tid == 0) {
    ctl[CTL_CUT_KEY] = (long long)prefix;  // low bits; compared under low_mask
    ctl[CTL_TIE_MODE] = partial ? 1 : 0;
    ctl[CTL_CUT_FLAT] = (long long)flat_prefix;
  }
}

// ------------------------------------------------------------------ 6. append the kept candidates
__global__ void __launch_bounds__(256) finalize_kernel(Lists o, FlatGeom fg, long long* __restrict__ ctl,
                                                         int* __restrict__ status) {
  if (chain_wait()) return;
  chain_release();
  const int shift = int(ctl[CTL_SHIFT]);
  const uint32_t key_lo = uint32_t(ctl[CTL_KEY_LO]);
  long long n = ctl[CTL_NUM_CAND];
  if (n > o.cand_cap) n = o.cand_cap;
  const uint32_t low_mask = shift >= 32 ? 0xFFFFFFFFu : ((1u << shift) - 1u);
  const uint32_t cut = uint32_t(ctl[CTL_CUT_KEY]);
  const bool tie_cut = ctl[CTL_TIE_MODE] != 0;
  const unsigned long long cut_flat = (unsigned long long)ctl[CTL_CUT_FLAT];
  unsigned long long* n_ent = reinterpret_cast<unsigned long long*>(ctl + CTL_NUM_ENTRIES);
  for (long long i = blockIdx.x * 1LL * blockDim.x + threadIdx.x; i < n; i += 1LL * gridDim.x * blockDim.x) {
    const uint32_t k = (o.cand_key[i] - key_lo) & low_mask;
    bool keep = k > cut;
    if (k == cut) keep = !tie_cut || flat_index(fg, o.cand_tok[i], o.cand_col[i]) <= cut_flat;
    if (keep) {
      const unsigned long long p = atomicAdd(n_ent, 1ULL);
      if ((long long)p < o.ent_cap) {
        o.ent_tok[p] = o.cand_tok[i]; o.ent_col[p] = o.cand_col[i]; o.ent_val[p] = o.cand_val[i];
      } else {
        atomicCAS(status, STATUS_OK, STATUS_CAPACITY);
      }
    }
  }
}

// ------------------------------------------------------------------ 7. CSR views
__global__ void __launch_bounds__(256) csr_count_kernel(const int* __restrict__ ent_tok, const int* __restrict__ ent_col,
                                                          const float* __restrict__ ent_val, long long cap,
                                                          const long long* __restrict__ ctl, int* __restrict__ tok_cnt,
                                                          int* __restrict__ feat_cnt, unsigned char* __restrict__ fired,
                                                          int num_tokens, int num_cols) {
  if (chain_wait()) return;
  chain_release();
  long long n = ctl[CTL_NUM_ENTRIES];
  if (n > cap) n = cap;
  for (long long i = blockIdx.x * 1LL * blockDim.x + threadIdx.x; i < n; i += 1LL * gridDim.x * blockDim.x) {
    const int t = ent_tok[i];
    const int c = ent_col[i];
    // an entry outside the problem (a stale count, a wrong pitch on the caller's side) is left out of both views
    // instead of being counted into a neighbouring region
    if (t < 0 || t >= num_tokens || c < 0 || c >= num_cols) continue;
    atomicAdd(&tok_cnt[t], 1);
    atomicAdd(&feat_cnt[c], 1);
    if (fired != nullptr && ent_val[i] > 1e-6f) fired[c] = 1;  // c was range-checked above
  }
}

// Exclusive scan of `n` ints by one CTA (1024 threads) over coalesced tiles of 4096 elements; out has n+1
// entries.  cursor (optional) gets a copy of the offsets for the scatter pass.
__global__ void __launch_bounds__(1024) exclusive_scan_kernel(const int* __restrict__ in, int* __restrict__ out,
                                                                int* __restrict__ cursor, int n) {
  if (chain_wait()) return;
  chain_release();
  __shared__ int warp_tot[32];
  __shared__ int carry_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) carry_s = 0;
  __syncthreads();
  for (int base = 0; base < n; base += 4096) {
    const int i0 = base + tid * 4;
    int v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = (i0 + k < n) ? in[i0 + k] : 0;
    const int mine = v[0] + v[1] + v[2] + v[3];
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) warp_tot[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      int w = warp_tot[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xFFFFFFFFu, w, o);
        if (lane >= o) w += t;
      }
      warp_tot[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    const int carry = carry_s;
    int run = carry + (warp > 0 ? warp_tot[warp - 1] : 0) + incl - mine;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i0 + k < n) {
        out[i0 + k] = run;
        if (cursor != nullptr) cursor[i0 + k] = run;
      }
      run += v[k];
    }
    __syncthreads();
    if (tid == 1023) carry_s = carry + warp_tot[31];
    __syncthreads();
  }
  if (tid == 0) out[n] = carry_s;
}

// Multi-CTA variant without scratch memory: CTA t owns elements [4096 t, 4096 (t + 1)).  It first adds up
// everything in front of its tile (the counts are small and stay in L2, so the repeated reads are cheaper
// than a second launch or a look-back protocol), then scans its own tile.
// Both arrays of the CSR build go in one launch: the first `tiles_a` CTAs scan a, the rest b.
struct ScanJob {
  const int* in;
  int* out;
  int* cursor;  // optional copy of the offsets for the scatter pass
  int n;
};
__global__ void __launch_bounds__(1024) exclusive_scan_tiles_kernel(ScanJob ja, ScanJob jb, int tiles_a) {
  if (chain_wait()) return;
  chain_release();
  __shared__ int warp_tot[32];
  __shared__ int carry_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool second = int(blockIdx.x) >= tiles_a;
  const ScanJob& job = second ? jb : ja;
  const int tile = second ? int(blockIdx.x) - tiles_a : int(blockIdx.x);
  const int n = job.n;
  const int* __restrict__ in = job.in;
  int* __restrict__ out = job.out;
  int* __restrict__ cursor = job.cursor;
  const int base = tile * 4096;
  int front = 0;
  {
    const int4* in4 = reinterpret_cast<const int4*>(in);  // base is a multiple of 4
    for (int i = tid; i < base / 4; i += 1024) {
      const int4 q = __ldg(in4 + i);
      front += q.x + q.y + q.z + q.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) front += __shfl_xor_sync(0xFFFFFFFFu, front, o);
    if (lane == 0) warp_tot[warp] = front;
    __syncthreads();
    if (tid == 0) {
      int c = 0;
      for (int w = 0; w < 32; ++w) c += warp_tot[w];
      carry_s = c;
    }
    __syncthreads();
  }
  const int carry = carry_s;
  __syncthreads();
  const int i0 = base + tid * 4;
  int v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = (i0 + k < n) ? in[i0 + k] : 0;
  const int mine = v[0] + v[1] + v[2] + v[3];
  int incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = warp_tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xFFFFFFFFu, w, o);
      if (lane >= o) w += t;
    }
    warp_tot[lane] = w;
  }
  __syncthreads();
  int run = carry + (warp > 0 ? warp_tot[warp - 1] : 0) + incl - mine;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (i0 + k < n) {
      out[i0 + k] = run;
      if (cursor != nullptr) cursor[i0 + k] = run;
    }
    run += v[k];
  }
  if (base + 4096 >= n && tid == 1023) out[n] = carry + warp_tot[31];
}

static void launch_exclusive_scans(const ScanJob& a, const ScanJob& b, cudaStream_t st) {
  const int ta = (a.n + 4095) / 4096, tb = (b.n + 4095) / 4096;
  const bool aligned = ((reinterpret_cast<uintptr_t>(a.in) | reinterpret_cast<uintptr_t>(b.in)) & 15) == 0;
  if (a.n > 0 && b.n > 0 && ta <= 512 && tb <= 512 && aligned) {
    launch_chained(exclusive_scan_tiles_kernel, ta + tb, 1024, 0, st, a, b, ta);
  } else {
    launch_chained(exclusive_scan_kernel, 1, 1024, 0, st, a.in, a.out, a.cursor, a.n);
    launch_chained(exclusive_scan_kernel, 1, 1024, 0, st, b.in, b.out, b.cursor, b.n);
  }
}

__global__ void __launch_bounds__(256) csr_scatter_kernel(const int* __restrict__ ent_tok, const int* __restrict__ ent_col,
                                                            const float* __restrict__ ent_val, long long cap,
                                                            const long long* __restrict__ ctl, int* __restrict__ tok_cursor,
                                                            int* __restrict__ feat_cursor, int* __restrict__ tcsr_col,
                                                            float* __restrict__ tcsr_val, int* __restrict__ fcsr_tok,
                                                            float* __restrict__ fcsr_val, int col_pitch, int num_tokens, int num_cols,
                                                            const int* __restrict__ feat_off, int* __restrict__ layer_cnt) {
  if (chain_wait()) return;
  chain_release();
  if (layer_cnt != nullptr && blockIdx.x == 0) {  // entries per layer: the offsets are complete
    for (int l = threadIdx.x; 1LL * l * col_pitch < num_cols; l += blockDim.x)
      layer_cnt[l] = feat_off[min(1LL * (l + 1) * col_pitch, 1LL * num_cols)] - feat_off[1LL * l * col_pitch];
  }
  long long n = ctl[CTL_NUM_ENTRIES];
  if (n > cap) n = cap;
  for (long long i = blockIdx.x * 1LL * blockDim.x + threadIdx.x; i < n; i += 1LL * gridDim.x * blockDim.x) {
    const int t = ent_tok[i], c = ent_col[i];
    if (t < 0 || t >= num_tokens || c < 0 || c >= num_cols) continue;  // the same entries that the count pass left out
    const float v = ent_val[i];
    const int p = atomicAdd(&tok_cursor[t], 1);
    const int layer = c / col_pitch;  // token-major view stores (layer << 24) | feature for the decoder
    if (p >= 0 && p < cap) { tcsr_col[p] = (layer << 24) | (c - layer * col_pitch); tcsr_val[p] = v; }
    const int q = atomicAdd(&feat_cursor[c], 1);
    if (q >= 0 && q < cap) { fcsr_tok[q] = t; fcsr_val[q] = v; }
  }
}

// The token-major view alone, for callers that decode and update nothing: no counters, scan and scatter over the columns.
// layer_cnt [number of layers, at most 32]: entries per layer.
__global__ void __launch_bounds__(256) csr_token_count_kernel(const int* __restrict__ ent_tok, const int* __restrict__ ent_col, long long cap,
                                                                const long long* __restrict__ ctl, int* __restrict__ tok_cnt, int* __restrict__ layer_cnt,
                                                                int col_pitch, int num_tokens, int num_cols) {
  if (chain_wait()) return;
  chain_release();
  __shared__ int per_layer[32];
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) per_layer[threadIdx.x] = 0;
  __syncthreads();
  long long n = ctl[CTL_NUM_ENTRIES];
  if (n > cap) n = cap;
  const long long stride = 1LL * gridDim.x * blockDim.x;
  for (long long i0 = blockIdx.x * 1LL * blockDim.x; i0 < n; i0 += stride) {
    const long long i = i0 + threadIdx.x;
    const int t = i < n ? ent_tok[i] : -1, c = i < n ? ent_col[i] : -1;
    const bool in = t >= 0 && t < num_tokens && c >= 0 && c < num_cols;  // as in csr_count_kernel
    if (in) atomicAdd(&tok_cnt[t], 1);
    const int layer = in ? c / col_pitch : 32;
    const uint32_t same = __match_any_sync(0xFFFFFFFFu, layer);
    if (layer < 32 && lane == __ffs(same) - 1) atomicAdd(&per_layer[layer], __popc(same));
  }
  __syncthreads();
  if (threadIdx.x < 32 && per_layer[threadIdx.x] != 0) atomicAdd(&layer_cnt[threadIdx.x], per_layer[threadIdx.x]);
}
__global__ void __launch_bounds__(256) csr_token_scatter_kernel(const int* __restrict__ ent_tok, const int* __restrict__ ent_col,
                                                                  const float* __restrict__ ent_val, long long cap, const long long* __restrict__ ctl,
                                                                  int* __restrict__ tok_cursor, int* __restrict__ tcsr_col, float* __restrict__ tcsr_val,
                                                                  int col_pitch, int num_tokens, int num_cols) {
  if (chain_wait()) return;
  chain_release();
  long long n = ctl[CTL_NUM_ENTRIES];
  if (n > cap) n = cap;
  for (long long i = blockIdx.x * 1LL * blockDim.x + threadIdx.x; i < n; i += 1LL * gridDim.x * blockDim.x) {
    const int t = ent_tok[i], c = ent_col[i];
    if (t < 0 || t >= num_tokens || c < 0 || c >= num_cols) continue;
    const int p = atomicAdd(&tok_cursor[t], 1);
    const int layer = c / col_pitch;
    if (p >= 0 && p < cap) { tcsr_col[p] = (layer << 24) | (c - layer * col_pitch); tcsr_val[p] = ent_val[i]; }
  }
}

// Bitonic network on n 64-bit words in shared memory or on (key, value) pairs in global memory, by all threads of the CTA.  Every
// comparator puts the smaller key at the lower index (the first step of a merge pairs mirrored positions), so the virtual
// padding to a power of two, which stands for +infinity at the end of the array, never has to move.
template <typename CmpSwap>
__device__ __forceinline__ void bitonic_cta(int n, CmpSwap cmp_swap) {
  int p2 = 1;
  while (p2 < n) p2 <<= 1;
  for (int size = 2; size <= p2; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      __syncthreads();
      for (int i = threadIdx.x; i < p2 / 2; i += blockDim.x) {
        const int j = i & (stride - 1);
        const int lo = 2 * i - j;
        const int hi = stride == (size >> 1) ? lo + size - 1 - 2 * j : lo + stride;
        if (hi < n) cmp_swap(lo, hi);
      }
    }
  }
  __syncthreads();
}
__device__ __forceinline__ void sort_words_cta(unsigned long long* w, int n) {
  bitonic_cta(n, [&](int lo, int hi) {
    const unsigned long long x = w[lo], y = w[hi];
    if (x > y) { w[lo] = y; w[hi] = x; }
  });
}
__device__ __forceinline__ void sort_pairs_cta(int* k, float* v, int n) {
  bitonic_cta(n, [&](int lo, int hi) {
    const int ka = k[lo], kb = k[hi];
    if (ka > kb) {
      k[lo] = kb; k[hi] = ka;
      const float t = v[lo]; v[lo] = v[hi]; v[hi] = t;
    }
  });
}
__device__ __forceinline__ unsigned long long pack_entry(int key, float val) { return ((unsigned long long)(unsigned int)key << 32) | __float_as_uint(val); }

// Feature segments (sorted by token, so that every floating-point sum over a segment has one order).  A feature holds a few
// entries, so a CTA takes up to 256 adjacent features, whose entries are one contiguous range: it comes into shared memory with
// coalesced loads, one thread sorts one short segment there, and the CTA sorts the long ones together.  Ranges that do not
// fit (features that fire on most tokens) are sorted in place in global memory.
constexpr int kShortSegment = 32;
constexpr int kFeatSortCap = 4096;
__global__ void __launch_bounds__(256) csr_sort_feature_segments_kernel(const int* __restrict__ off, int nseg, int per_cta,
                                                                          int* __restrict__ key, float* __restrict__ val) {
  if (chain_wait()) return;
  chain_release();
  __shared__ unsigned long long w[kFeatSortCap];
  __shared__ int long_list[256];
  __shared__ int long_count;
  const int s0 = blockIdx.x * per_cta, s1 = min(nseg, s0 + per_cta);
  const int lo = off[s0], range = off[s1] - lo;
  if (range <= 1) return;
  const int mine = s0 + threadIdx.x;  // threads beyond per_cta own no segment
  const int b = mine < s1 ? off[mine] : 0, n = mine < s1 ? off[mine + 1] - b : 0;
  if (threadIdx.x == 0) long_count = 0;
  const bool in_smem = range <= kFeatSortCap;
  if (in_smem)
    for (int i = threadIdx.x; i < range; i += 256) w[i] = pack_entry(key[lo + i], val[lo + i]);
  __syncthreads();
  if (n > kShortSegment) {
    long_list[atomicAdd(&long_count, 1)] = mine;
  } else if (in_smem) {
    unsigned long long* q = w + (b - lo);
    for (int i = 1; i < n; ++i) {
      const unsigned long long x = q[i];
      int j = i - 1;
      while (j >= 0 && q[j] > x) { q[j + 1] = q[j]; --j; }
      q[j + 1] = x;
    }
  } else {
    for (int i = b + 1; i < b + n; ++i) {
      const int k = key[i];
      const float v = val[i];
      int j = i - 1;
      while (j >= b && key[j] > k) { key[j + 1] = key[j]; val[j + 1] = val[j]; --j; }
      key[j + 1] = k; val[j + 1] = v;
    }
  }
  __syncthreads();
  for (int q = 0; q < long_count; ++q) {
    const int sb = off[long_list[q]], sn = off[long_list[q] + 1] - sb;
    if (in_smem) sort_words_cta(w + (sb - lo), sn);
    else sort_pairs_cta(key + sb, val + sb, sn);
  }
  if (in_smem)
    for (int i = threadIdx.x; i < range; i += 256) { key[lo + i] = int(w[i] >> 32); val[lo + i] = __uint_as_float((unsigned int)(w[i] & 0xFFFFFFFFULL)); }
}

// Token segments: one CTA per token sorts its entries by (layer, feature).  Short lists: every thread counts how many keys are below
// its own (broadcast reads of shared memory, no barrier in between: 1 us where the 36 barriers of a network on 256 entries take ten)
// and stores its entry at that rank.  Longer ones: the entries are dealt into buckets by layer first, and an entry's place is the number of
// entries in lower layers plus the number of smaller keys in its own bucket.  Long buckets (kTokenBucketCap), or equal keys, go through the
// network in shared memory, and lists beyond its buffer through the one in global memory.  The order lets the decode's tokens pass over
// the decoder rows together (L2) and fixes the order of its sums.
// The buckets take a few more barriers and do n * n / layers instead of n * n comparisons: few tokens, where the latency of one CTA counts,
// rank up to 512 entries (512 tokens of at most 352: 5.3 us against 10.0 with buckets; 16 tokens of up to 605: 16.4 us with the
// network above 512, 9.1 with buckets); with many tokens the comparisons count (4096 tokens, 200 entries on average: 60 us with ranks up to
// 512, 48 with buckets; 8192 tokens: 86 and 77; 4096 tokens of 25: 8.7 and 9.7).  Lists that must have a bucket above the cap, because there are
// not layers enough, go to the network directly (1024 tokens of 800 entries in two layers: 47 us, 49 behind a count of the buckets), and
// with one layer there is one bucket: ranks up to 256 entries (4096 tokens of 200: 29 us, 38 as a bucket).
// The bucket of layer l starts at bank l: the lanes of a warp read the buckets of their layers side by side, and where those lie by the lengths before
// them they meet at few banks (1024 tokens of 2000 entries, up to 256 in each of eight layers: 594 us, with a bank for every layer 104).
constexpr int kTokenSortCap = 2048;
constexpr int kTokenBucketCap = 256;
constexpr int kTokenBuckets = 128;  // layers, as the packed key can number them
constexpr int kTokenBucketRoom = kTokenSortCap + 32 * 31 + kTokenBuckets;  // every bucket of 32 layers with room to the next layer's bank
constexpr int kFewTokens = 768;

// Ranks over the whole list, M entries per thread; false when two keys are equal.
template <int M>
__device__ __forceinline__ bool rank_sort_segment(int* __restrict__ key, float* __restrict__ val, int n, int* keys, int* taken) {
  int mine[M], rank[M];
  float v[M];
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int i = threadIdx.x + 256 * m;
    mine[m] = i < n ? key[i] : 0x7FFFFFFF;
    v[m] = i < n ? val[i] : 0.f;
    rank[m] = 0;
    keys[i] = mine[m];
    taken[i] = 0;
  }
  __syncthreads();
  const int4* k4 = reinterpret_cast<const int4*>(keys);
  for (int j = 0; j < (n + 3) / 4; ++j) {
    const int4 q = k4[j];
#pragma unroll
    for (int m = 0; m < M; ++m) rank[m] += (q.x < mine[m]) + (q.y < mine[m]) + (q.z < mine[m]) + (q.w < mine[m]);
  }
  bool clash = false;  // equal keys share a rank
#pragma unroll
  for (int m = 0; m < M; ++m)
    if (threadIdx.x + 256 * m < n) clash |= atomicExch(&taken[rank[m]], 1) != 0;
  if (__syncthreads_or(clash)) return false;
#pragma unroll
  for (int m = 0; m < M; ++m)
    if (threadIdx.x + 256 * m < n) { key[rank[m]] = mine[m]; val[rank[m]] = v[m]; }
  return true;
}

// M entries per thread (n <= 256 M); false when the network has to sort them.
template <int M>
__device__ __forceinline__ bool bucket_sort_segment(int* __restrict__ key, float* __restrict__ val, int n, int* bucket, int* taken, int* count, int* base, int* start) {
  int mine[M], slot[M];
  float v[M];
  if (threadIdx.x < kTokenBuckets) count[threadIdx.x] = 0;
  __syncthreads();
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const int i = threadIdx.x + 256 * m;
    if (i < n) {
      mine[m] = key[i];
      v[m] = val[i];
      slot[m] = atomicAdd(&count[(mine[m] >> 24) & (kTokenBuckets - 1)], 1);
      taken[i] = 0;
    }
  }
  __syncthreads();
  bool network = false;
  if (threadIdx.x < 32) {
    int c[4], sum = 0, room = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      c[k] = count[4 * threadIdx.x + k];
      network |= c[k] > kTokenBucketCap;
      sum += c[k];
      room += c[k] + ((1 - c[k]) & 31);
    }
    int incl = sum, incl_room = room;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xFFFFFFFFu, incl, o), up_room = __shfl_up_sync(0xFFFFFFFFu, incl_room, o);
      if (int(threadIdx.x) >= o) { incl += up; incl_room += up_room; }
    }
    network |= incl_room > kTokenBucketRoom;
    int run = incl - sum, at = incl_room - room;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      start[4 * threadIdx.x + k] = run;
      base[4 * threadIdx.x + k] = at;
      run += c[k];
      at += c[k] + ((1 - c[k]) & 31);
    }
  }
  if (__syncthreads_or(network)) return false;
#pragma unroll
  for (int m = 0; m < M; ++m)
    if (threadIdx.x + 256 * m < n) bucket[base[(mine[m] >> 24) & (kTokenBuckets - 1)] + slot[m]] = mine[m];
  __syncthreads();
  bool clash = false;  // equal keys share a place
#pragma unroll
  for (int m = 0; m < M; ++m) {
    if (threadIdx.x + 256 * m < n) {
      const int l = (mine[m] >> 24) & (kTokenBuckets - 1);
      const int b = base[l], e = b + count[l];
      int at = start[l];
      for (int j = b; j < e; ++j) at += bucket[j] < mine[m] ? 1 : 0;
      slot[m] = at;
      clash |= atomicExch(&taken[at], 1) != 0;
    }
  }
  if (__syncthreads_or(clash)) return false;
#pragma unroll
  for (int m = 0; m < M; ++m)
    if (threadIdx.x + 256 * m < n) { key[slot[m]] = mine[m]; val[slot[m]] = v[m]; }
  return true;
}

__global__ void __launch_bounds__(256) csr_sort_token_segments_kernel(const int* __restrict__ off, int* __restrict__ key, float* __restrict__ val, int rank_up_to,
                                                                         int bucket_up_to) {
  if (chain_wait()) return;
  chain_release();
  __shared__ __align__(16) unsigned long long w[(kTokenBucketRoom + kTokenSortCap) / 2];
  __shared__ int count[kTokenBuckets], base[kTokenBuckets], start[kTokenBuckets];
  const int b = off[blockIdx.x], n = off[blockIdx.x + 1] - b;
  if (n <= 1) return;
  if (n > kTokenSortCap) {
    sort_pairs_cta(key + b, val + b, n);
    return;
  }
  int* bucket = reinterpret_cast<int*>(w);  // the buckets share the network's buffer: keys first, marks behind them
  int* taken = bucket + kTokenBucketRoom;
  const bool done = n <= rank_up_to
                        ? (n <= 256 ? rank_sort_segment<1>(key + b, val + b, n, bucket, taken) : rank_sort_segment<2>(key + b, val + b, n, bucket, taken))
                    : n > bucket_up_to ? false
                    : n <= 256         ? bucket_sort_segment<1>(key + b, val + b, n, bucket, taken, count, base, start)
                    : n <= 512         ? bucket_sort_segment<2>(key + b, val + b, n, bucket, taken, count, base, start)
                    : n <= 1024        ? bucket_sort_segment<4>(key + b, val + b, n, bucket, taken, count, base, start)
                                       : bucket_sort_segment<8>(key + b, val + b, n, bucket, taken, count, base, start);
  if (done) return;
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += blockDim.x) w[i] = pack_entry(key[b + i], val[b + i]);
  sort_words_cta(w, n);
  for (int i = threadIdx.x; i < n; i += blockDim.x) { key[b + i] = int(w[i] >> 32); val[b + i] = __uint_as_float((unsigned int)(w[i] & 0xFFFFFFFFULL)); }
}

static void launch_token_sort(const int* off, int* key, float* val, int num_tokens, int num_cols, int col_pitch, cudaStream_t st) {
  if (num_tokens <= 0) return;
  const int layers = (num_cols + col_pitch - 1) / col_pitch;
  const int rank_up_to = num_tokens < kFewTokens ? 512 : (layers <= 1 ? 256 : 128);
  launch_chained(csr_sort_token_segments_kernel, num_tokens, 256, 0, st, off, key, val, rank_up_to, layers < 8 ? layers * kTokenBucketCap : kTokenSortCap);
}

// Dead-feature counters: +1 per step, reset where the feature fired (reference trainer.py:693-712).
__global__ void __launch_bounds__(256) dead_counter_kernel(long long* __restrict__ counter, unsigned char* __restrict__ fired, int n) {
  if (chain_wait()) return;
  chain_release();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    counter[i] = fired[i] ? 0 : counter[i] + 1;
    fired[i] = 0;
  }
}

}  // namespace clt

// ====================================================================== C launchers
using namespace clt;

// Chunks of rows in the statistics of L layers of F columns: one, or as many as fill the chip where the columns alone do not.
#if !CLT_T16_IS_HALF
extern "C" int clt_colstats_splits(int L, int B, int F) {
  const int col_blocks = (F / 8 + 31) / 32;
  int zsplit = 1;
  while (1LL * col_blocks * L * zsplit < 592 && zsplit < 16 && B / (zsplit * 2) >= 128) zsplit *= 2;
  return zsplit;
}
#else
extern "C" int clt_colstats_splits(int L, int B, int F);
#endif

// The statistics of the strips of 256 columns (counted over all layers) from `first_strip` on.
extern "C" int CLT_FN(clt_colstats_strips)(const void* x, float* mean, float* rstd, int L, int B, int F, long long ld, long long layer_stride,
                                           long long first_strip, int* kernels, cudaStream_t st) {
  *kernels = 0;
  if (F % 8 != 0 || ld % 8 != 0 || layer_stride % 8 != 0) return -1;
  const int strips = (F + 255) / 256;
  const long long todo = 1LL * L * strips - first_strip;
  if (todo <= 0) return 0;
  const int zsplit = clt_colstats_splits(L, B, F);
  const dim3 block(32, 8);
  const t16* xp = static_cast<const t16*>(x);
  const long long first = first_strip / strips * F + first_strip % strips * 256, n = 1LL * L * F;  // in mean / rstd
  if (zsplit > 1) {
    if (cudaMemsetAsync(mean + first, 0, sizeof(float) * size_t(n - first), st) != cudaSuccess) return -5;
    if (cudaMemsetAsync(rstd + first, 0, sizeof(float) * size_t(n - first), st) != cudaSuccess) return -5;
  }
  if (first_strip > 0)  // the rest of a GEMM: less than one strip for each pair of SMs
    launch_chained(colstats_kernel<2>, dim3(unsigned(4 * todo), 1, zsplit), block, 0, st, xp, mean, rstd, B, F, ld, layer_stride, first_strip);
  else
    launch_chained(colstats_kernel<8>, dim3(unsigned(todo), 1, zsplit), block, 0, st, xp, mean, rstd, B, F, ld, layer_stride, 0);
  if (zsplit > 1) launch_chained(colstats_finalize_kernel, int((n - first + 255) / 256), 256, 0, st, xp, mean, rstd, B, F, layer_stride, first, n);
  *kernels = zsplit > 1 ? 2 : 1;
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
extern "C" int CLT_FN(clt_colstats)(const void* x, float* mean, float* rstd, int L, int B, int F, long long ld, long long layer_stride,
                            cudaStream_t st) {
  int kernels;
  return CLT_FN(clt_colstats_strips)(x, mean, rstd, L, B, F, ld, layer_stride, 0, &kernels, st);
}

#if !CLT_T16_IS_HALF
extern "C" int clt_colstats_from_tiles(const float* tile_stats, float* mean, float* rstd, int L, int B, int F, cudaStream_t st) {
  const long long n = 1LL * L * F;
  if (n == 0) return 0;
  launch_chained(colstats_from_tiles_kernel, int((n + 255) / 256), 256, 0, st, tile_stats, mean, rstd, B, F, (B + 127) / 128, n);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

#endif

struct CltExchangeArgs {
  int world;
  int rank;
  void* data[8];
  void* flags[8];
  int slot_elems;
  unsigned int seq;
};

static Exchange to_exchange(const CltExchangeArgs* a) {
  Exchange ex;
  ex.world = a ? a->world : 1;
  ex.rank = a ? a->rank : 0;
  ex.slot_elems = a ? a->slot_elems : 0;
  ex.seq = a ? a->seq : 0;
  for (int i = 0; i < kMaxPeers; ++i) {
    ex.peers[i] = a ? static_cast<uint32_t*>(a->data[i]) : nullptr;
    ex.flags[i] = a ? static_cast<uint32_t*>(a->flags[i]) : nullptr;
  }
  return ex;
}

struct CltSelectArgs {
  const void* x;  // [L, B, ld] bf16 pre-activations
  const float* mean;
  const float* rstd;
  int L, B, F;  // F: valid local features per layer
  int stat_pitch;  // row pitch of mean / rstd
  long long ld, layer_stride;
  int col_pitch;       // pitch used to encode columns (l * col_pitch + f)
  int feat_offset;     // first global feature of the shard
  long long full_F;    // un-sharded feature count
  long long k_total;   // global number of entries to keep
  unsigned int key_lo; // histogram covers keys >= key_lo
  int shift;           // bin = (key - key_lo) >> shift
  unsigned int* hist;  // [2 * 8192 + 32], zeroed by the caller
  long long* ctl;      // [CTL_SIZE]
  int* ent_tok; int* ent_col; float* ent_val; long long ent_cap;
  unsigned int* cand_key; int* cand_tok; int* cand_col; float* cand_val; long long cand_cap;
  int* status;
  // Optional tracked range: sel_state = {key_lo, shift} in device memory, moved by the kernels every step,
  // and the pool that the single pass over the matrix fills.  Null sel_state: fixed range from key_lo / shift.
  long long* sel_state;
  unsigned int* pool_key; int* pool_tok; int* pool_col; float* pool_val; long long pool_cap;
};

static ScanGeom scan_geom(const CltSelectArgs* a) {
  ScanGeom g;
  g.B = a->B; g.F = a->F; g.L = a->L; g.sp = a->stat_pitch; g.ld = a->ld; g.layer_stride = a->layer_stride;
  g.rows_per_block = 64;
  return g;
}
static Lists lists_of(const CltSelectArgs* a) {
  Lists o;
  o.ent_tok = a->ent_tok; o.ent_col = a->ent_col; o.ent_val = a->ent_val; o.ent_cap = a->ent_cap;
  o.cand_key = a->cand_key; o.cand_tok = a->cand_tok; o.cand_col = a->cand_col; o.cand_val = a->cand_val; o.cand_cap = a->cand_cap;
  return o;
}
static FlatGeom flat_geom(const CltSelectArgs* a) {
  FlatGeom fg;
  fg.col_pitch = a->col_pitch; fg.feat_offset = a->feat_offset; fg.full_F = a->full_F; fg.row_width = a->full_F * a->L;
  return fg;
}

// Rows per CTA, 64 to begin with.  With more than one kept element in 256 half as many in the passes without a tracked range (one in five: 1041 us, 1312 with
// 64 of 100000 tokens x 264; 16 x 300 x 1024: 281, 493).
static int rows_halved(const CltSelectArgs* a, int rows) {  // the grid's second dimension has its limit
  return rows > 8 && (a->B + rows / 2 - 1) / (rows / 2) <= 65535 ? rows / 2 : rows;
}
static bool densely_kept(const CltSelectArgs* a) { return 256 * a->k_total > 1LL * a->B * a->L * a->full_F; }

// The collecting pass: its queue holds 2048 pieces of eight elements, of 16384 in 64 rows of 2048 columns, and must not overflow while the cut moves: every
// overflow costs the full-range passes (evaluation of 13 x 2536 features, 1504 tokens, k = 245: 677 us with them, 354 without).  A tracked range
// holds 1.75 k elements; rows are halved until, spread evenly, the pieces with one of them fill at most 0.35 of the queue (eight rows cannot overflow
// it), and once for densely kept elements where 64 rows make fewer than eight CTAs per SM.  us by rows per CTA (64, 32, 16, 8; + with full-range
// passes), 6 x 4096 tokens x 2048: one in 400 69 71 72 82; 250 91 81 80 87; 150 317+ 101 92 98; 90 484+ 157 111 113; 60 642+ 799+ 174 131; 30 836+ 726+
// 1119+ 252; 8 1801+ 1494+ 1814+ 882.
static int collect_rows(const CltSelectArgs* a) {
  const double q = kPoolFactor * double(a->k_total) / (double(a->B) * a->L * a->full_F);  // share of the elements
  const int pieces = (a->F + 7) / 8;
  const double per_row = (1.0 - std::pow(1.0 - std::min(q, 1.0), 8.0)) * std::min(pieces, 256);
  int rows = 64;
  if (densely_kept(a) && 1LL * ((pieces + 255) / 256) * ((a->B + 63) / 64) * a->L < 8LL * device_sms()) rows = rows_halved(a, rows);
  while (rows * per_row > 0.35 * kCollectQueue && rows_halved(a, rows) < rows) rows = rows_halved(a, rows);
  return rows;
}

// Steps 2-6.  `exa` may be null (single rank).  The histogram first covers keys >= key_lo only (the
// caller's guess of where the cut lies); if the cut is not inside, a full-range pass repeats it.
// `hist` holds two histograms of 8192 counters, zeroed by the caller.
extern "C" int CLT_FN(clt_batchtopk_select)(const CltSelectArgs* a, const CltExchangeArgs* exa, cudaStream_t st) {
  if (a->ld % 8 != 0 || a->layer_stride % 8 != 0 || a->stat_pitch % 4 != 0 || a->F > a->ld) return -1;
  ScanGeom g = scan_geom(a);
  const bool tracked = a->sel_state != nullptr && a->key_lo != 0;
  if (!tracked && densely_kept(a)) g.rows_per_block = rows_halved(a, g.rows_per_block);
  const Exchange ex = to_exchange(exa);
  const auto grid_of = [&](const ScanGeom& s) { return dim3(((a->F + 7) / 8 + 255) / 256, (a->B + s.rows_per_block - 1) / s.rows_per_block, a->L); };
  const dim3 grid = grid_of(g);
  const t16* x = static_cast<const t16*>(a->x);
  if (tracked) {
    Pool pool;
    pool.key = a->pool_key; pool.tok = a->pool_tok; pool.col = a->pool_col; pool.val = a->pool_val; pool.cap = a->pool_cap;
    pool.count = a->hist + 2 * kHistBins;
    ScanGeom gc = g;
    gc.rows_per_block = collect_rows(a);
    launch_chained(zhist_collect_kernel, grid_of(gc), 256, 0, st, x, a->mean, a->rstd, gc, a->col_pitch, a->sel_state, a->hist, pool);
    launch_chained(find_bin_kernel, 1, 1024, 0, st, a->hist, a->k_total, a->ctl, ex, 0u, 0, 0, 0, a->sel_state, pool.count, pool.cap, a->status);
    launch_chained(classify_pool_kernel, 592, 256, 0, st, pool, a->ctl, lists_of(a), a->status);
    // fallback, skipped inside the kernels unless the tracked range missed the cut or the pool overflowed
    launch_chained(zhist_kernel, grid, 256, 0, st, x, a->mean, a->rstd, g, 0u, 19, a->hist + kHistBins, a->ctl, 1);
    launch_chained(find_bin_kernel, 1, 1024, 0, st, a->hist + kHistBins, a->k_total, a->ctl, ex, 0u, 19, 1, 1, a->sel_state, nullptr, 0, a->status);
    launch_chained(compact_kernel, grid, 256, 0, st, x, a->mean, a->rstd, g, a->col_pitch, a->ctl, lists_of(a), a->status, 1);
  } else {
    launch_chained(zhist_kernel, grid, 256, 0, st, x, a->mean, a->rstd, g, a->key_lo, a->shift, a->hist, a->ctl, 0);
    launch_chained(find_bin_kernel, 1, 1024, 0, st, a->hist, a->k_total, a->ctl, ex, a->key_lo, a->shift, 0, 0, nullptr, nullptr, 0, a->status);
    if (a->key_lo != 0) {
      launch_chained(zhist_kernel, grid, 256, 0, st, x, a->mean, a->rstd, g, 0u, 19, a->hist + kHistBins, a->ctl, 1);
      launch_chained(find_bin_kernel, 1, 1024, 0, st, a->hist + kHistBins, a->k_total, a->ctl, ex, 0u, 19, 1, 1, nullptr, nullptr, 0, a->status);
    }
    launch_chained(compact_kernel, grid, 256, 0, st, x, a->mean, a->rstd, g, a->col_pitch, a->ctl, lists_of(a), a->status, 0);
  }
  launch_chained(refine_kernel, 1, 1024, 0, st, a->cand_key, a->cand_tok, a->cand_col, a->cand_cap, flat_geom(a), a->ctl, ex, a->status);
  launch_chained(finalize_kernel, 256, 256, 0, st, lists_of(a), flat_geom(a), a->ctl, a->status);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// Per-feature threshold selection (JumpReLU / ReLU as a sparse list).  theta: [L, stat_pitch] fp32.  Uses of the
// argument block: x, rstd (= theta), L, B, F, stat_pitch, ld, layer_stride, col_pitch, ctl, ent_*, status.
extern "C" int CLT_FN(clt_threshold_select)(const CltSelectArgs* a, cudaStream_t st) {
  if (a->ld % 8 != 0 || a->layer_stride % 8 != 0 || a->F > a->ld) return -1;
  const ScanGeom g = scan_geom(a);
  dim3 grid(((a->F + 7) / 8 + 255) / 256, (a->B + g.rows_per_block - 1) / g.rows_per_block, a->L);
  if (cudaMemsetAsync(a->ctl + CTL_NUM_ENTRIES, 0, sizeof(long long), st) != cudaSuccess) return -5;
  launch_chained(threshold_collect_kernel, grid, 256, 0, st, static_cast<const t16*>(a->x), a->rstd, g, a->col_pitch, a->ctl, lists_of(a), a->status);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

template <int TPC>
static int launch_token_list(const CltSelectArgs* a, const ScanGeom& g, int f_valid, int k, cudaStream_t st) {
  // per call, not once per process: the attribute belongs to the current device, and four tokens take more than the default limit
  if (cudaFuncSetAttribute(token_topk_list_kernel<TPC>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(TokenListShared<TPC>))) != cudaSuccess) return -4;
  // sample: at most every eighth block, at least enough groups for all maxima, and an expected list (step * k) of half its room
  const int groups = g.L * (g.F / 8);
  int step = kTkList / 2 / k;
  step = step > 8 ? 8 : step;
  if (step > groups / (2 * kTkMaxima)) step = groups / (2 * kTkMaxima);
  if (step < 1) step = 1;
  launch_chained(token_topk_list_kernel<TPC>, (a->B + TPC - 1) / TPC, kTkThreads, sizeof(TokenListShared<TPC>), st, 
      static_cast<const t16*>(a->x), a->mean, a->rstd, g, a->col_pitch, f_valid, k, step, a->ctl, lists_of(a));
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// The wide form: 131072 to 262144 columns over all layers, at most one column in 2048 kept (so k <= 128), 2^28 elements or more.
// One kernel / four passes, us:
//   elements: 6 x 32768 columns, k = 16 and 64, 900 tokens (1.8e8) 167 / 155 and 204 / 199, 1100 (2.2e8) 170 / 167 and 210 / 214, 1400 (2.8e8)
//     226 / 194 and 288 / 249, 2048 302 / 249 and 370 / 327, 8192 (k = 64) 1183 / 1114.  Below the line k = 90 is slower (1100 tokens 226 / 247,
//     1300 263 / 276), above it is not (1400 314 / 292).
//   columns: the passes over the tokens (bound, cut) do not shrink with them.  k = 24: 4 x 16384 x 4200 tokens 255 / 298, 12 x 8192 x 4096 321 / 331,
//     4 x 32768 x 2100 239 / 224, 12 x 16384 x 2048 325 / 265, 12 x 20480 x 2048 380 / 298; 1 x 4096 x 65600, k = 1: 654 / 1189.  Above 262144 the
//     maxima of a token (one in 64 columns) have no room in the bound pass.
//   k: 6 x 32768 x 2048, k = 96: 411 / 414; 8 x 32768 x 2048, k = 128: 539 / 507.  A tile (64 tokens, 2048 columns) has room for four times the
//     groups that are expected in it at the line; beyond it tokens would be lost to the radix kernel.
constexpr long long kWideElements = 1LL << 28;
constexpr long long kWideMinColumns = 1LL << 17, kWideMaxColumns = 1LL * kWideMaxima * 8 * kWideStep;
static_assert(1LL * kWideRows * kWideStep * 4 <= kWideQueue, "a tile of 2048 columns at the line: one kept column in 2048, kWideStep candidates for each");
static WideTopk wide_topk(const CltSelectArgs* a, long long k) {
  WideTopk w = {};
  const long long columns = 1LL * a->L * a->F;
  if (k <= 0 || columns < kWideMinColumns || columns > kWideMaxColumns || 2048 * k > columns || a->B * columns < kWideElements) return w;
  w.groups = int(columns / 8);
  w.cap = k <= 64 ? 1024 : 2048;  // twice the expected list
  w.ng = ((w.groups + 32 * kWideStep - 1) / (32 * kWideStep) * 32 + 255) / 256 * 256;
  return w;
}
// Bytes of scratch that clt_token_topk_select uses in its wide form (0: none).
extern "C" long long CLT_FN(clt_token_topk_scratch)(const CltSelectArgs* a) {
  const WideTopk w = wide_topk(a, a->k_total);
  if (w.ng == 0) return 0;
  return 1LL * a->B * (8LL * w.cap + 4LL * w.ng + 8);
}

// Per-token top-k of the batch z-scores (TokenTopK).  Uses x, mean, rstd, L, B, F, stat_pitch, ld, layer_stride,
// col_pitch, ctl, ent_* (capacity >= B * k), status of the argument block; k_total carries the per-token k and feat_offset
// (when positive) the number of valid columns per layer (the rest of F is shard padding).  *kernels: how many kernels were launched.
extern "C" int CLT_FN(clt_token_topk_select)(const CltSelectArgs* a, void* scratch, int* kernels, cudaStream_t st) {
  if (a->ld % 8 != 0 || a->layer_stride % 8 != 0 || a->F % 8 != 0 || a->stat_pitch % 4 != 0 || a->F > a->ld) return -1;
  const long long k = a->k_total;
  const int f_valid = a->feat_offset > 0 && a->feat_offset <= a->F ? a->feat_offset : a->F;  // feat_offset carries the valid column count here
  if (k <= 0 || k > 1LL * a->L * f_valid || 1LL * a->B * k > a->ent_cap) return -1;
  const ScanGeom g = scan_geom(a);
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(token_topk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(TokenTopkShared))) != cudaSuccess) return -4;
    attr_set = true;
  }
  const int grid = (a->B + kTokPerCta - 1) / kTokPerCta;
  const WideTopk shape = wide_topk(a, k);
  const bool wide = shape.ng > 0 && scratch != nullptr;
  const bool list = wide || k <= kTkMaxima / 2;
  *kernels = wide ? 5 : (list ? 2 : 1);
  if (wide) {
    WideTopk w = shape;
    w.list = static_cast<unsigned long long*>(scratch);
    w.maxima = reinterpret_cast<uint32_t*>(w.list + 1LL * a->B * w.cap);
    w.bound = w.maxima + 1LL * a->B * w.ng;
    w.n = reinterpret_cast<int*>(w.bound + a->B);
    const t16* x = static_cast<const t16*>(a->x);
    const int row_blocks = (a->B + kWideRows - 1) / kWideRows;
    if (cudaMemsetAsync(w.n, 0, sizeof(int) * size_t(a->B), st) != cudaSuccess) return -5;
    launch_chained(token_sample_kernel, dim3(w.ng / 256, row_blocks), 256, 0, st, x, a->mean, a->rstd, g, f_valid, w);
    launch_chained(token_bound_kernel, a->B, 256, 0, st, w, int(k), a->ctl, 1LL * a->B * k);
    launch_chained(token_collect_kernel, dim3((a->F / 8 + 255) / 256, row_blocks, a->L), 256, 0, st, x, a->mean, a->rstd, g, a->col_pitch, f_valid, w);
    if (w.cap <= 1024) launch_chained(token_cut_kernel<32>, (a->B + 3) / 4, 128, 0, st, x, g, a->col_pitch, int(k), w, lists_of(a));
    else launch_chained(token_cut_kernel<64>, (a->B + 3) / 4, 128, 0, st, x, g, a->col_pitch, int(k), w, lists_of(a));
  } else if (list) {
    // Tokens per CTA: what finishes in one wave of 148 SMs with four CTAs each (three of four tokens, whose lists are 64 KB).  More
    // tokens per CTA share the loads of the column statistics but take longer each, so one token while all fit that way, then
    // two, then four (from 1332: a second wave of a few CTAs of two costs less than four tokens in a row); beyond that, in several
    // waves, two.  6 x 32768 columns, k = 64, in us with one / two / four tokens per CTA: 592 tokens 155 / 175 / 224, 1184 288 / 222 /
    // 257, 1240 - / 255 / 290, 1500 320 / 339 / 298, 1776 355 / 365 / 302, 2368 466 / 427 / 509, 4096 750 / 667 / 765.
    constexpr int kOneWave = 148 * 4;
    const int rc = a->B <= kOneWave ? launch_token_list<1>(a, g, f_valid, int(k), st)
                   : a->B > kOneWave * 9 / 4 && a->B <= kOneWave * 3 ? launch_token_list<4>(a, g, f_valid, int(k), st)
                                                                   : launch_token_list<2>(a, g, f_valid, int(k), st);
    if (rc != 0) return rc;
  }
  launch_chained(token_topk_kernel, grid, 256, sizeof(TokenTopkShared), st, static_cast<const t16*>(a->x), a->mean, a->rstd, g, a->col_pitch,
                                                                 f_valid, int(k), a->ctl, lists_of(a), a->status, list ? 1 : 0);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

#if !CLT_T16_IS_HALF
// ------------------------------------------------------------------ TokenTopK across feature shards
// Every rank holds a slice of the columns; a token keeps its k largest z-scores over all ranks' columns (reference:
// clt/models/activations.py:360-491, where the full pre-activations are gathered and the mask is broadcast).  Here each
// rank first takes the exact top k of its own columns (token_topk_kernel: a superset of what survives), then
//   1. token_topk_push:   composite keys (z key << 32 | inverted global flat index) of the local candidates go to the
//                         owner of the token (tokens are dealt to the ranks in blocks of rows_per_rank) by peer stores;
//   2. token_topk_cut:    the owner ranks the W * k keys of each of its tokens, takes the k-th largest as the cut and stores
//                         it into every rank's cut array;
//   3. token_topk_filter: every rank keeps its candidates at or above the cut and appends them to its entry list.
// The composite keys are distinct and their order does not depend on the number of ranks (larger z first, lower flat index
// first among equal z), so the selection equals the single-GPU one entry for entry.  Phase barriers (peer_barrier) separate
// the three kernels; nothing here waits.
struct CltTopkTpArgs {
  const int* cand_col; const float* cand_val;   // [B * k] local candidates (token t at t * k ...), from token_topk_select
  unsigned long long* cand_key;                 // [B * k] composite keys (written by push, read by filter)
  const float* mean; const float* rstd; int stat_pitch;
  int col_pitch, feat_offset; long long full_F;
  int B, k, world, rank, rows_per_rank;
  void* stage[8];                               // every rank's key staging [world][rows_per_rank][k] u64
  void* cut[8];                                 // every rank's cut array [B] u64
  long long* ctl;
  int* ent_tok; int* ent_col; float* ent_val; long long ent_cap;
  int* status;
};

__global__ void __launch_bounds__(256) token_topk_push_kernel(CltTopkTpArgs a) {
  if (chain_wait()) return;
  chain_release();
  if (blockIdx.x == 0 && threadIdx.x == 0) a.ctl[CTL_NUM_ENTRIES] = 0;  // refilled by the filter pass
  const long long n = 1LL * a.B * a.k;
  for (long long i = blockIdx.x * 1LL * blockDim.x + threadIdx.x; i < n; i += 1LL * gridDim.x * blockDim.x) {
    const int t = int(i / a.k), j = int(i - 1LL * t * a.k);
    const int col = a.cand_col[i];
    const int l = col / a.col_pitch, c = col - l * a.col_pitch;
    const float z = (a.cand_val[i] - a.mean[1LL * l * a.stat_pitch + c]) * a.rstd[1LL * l * a.stat_pitch + c];
    const unsigned long long flat = (unsigned long long)l * (unsigned long long)a.full_F + (unsigned long long)(a.feat_offset + c);
    const unsigned long long key = ((unsigned long long)float_to_key(z) << 32) | (0xFFFFFFFFULL - flat);
    a.cand_key[i] = key;
    const int owner = t / a.rows_per_rank, lt = t - owner * a.rows_per_rank;
    static_cast<unsigned long long*>(a.stage[owner])[(1LL * a.rank * a.rows_per_rank + lt) * a.k + j] = key;
  }
}

// One CTA per owned token; dynamic shared memory world * k keys.
__global__ void __launch_bounds__(256) token_topk_cut_kernel(CltTopkTpArgs a) {
  if (chain_wait()) return;
  chain_release();
  extern __shared__ unsigned long long tk_keys[];
  const int lt = blockIdx.x;
  const int t = a.rank * a.rows_per_rank + lt;
  if (t >= a.B) return;
  const int n = a.world * a.k;
  const unsigned long long* mine = static_cast<const unsigned long long*>(a.stage[a.rank]);
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const int w = i / a.k, j = i - w * a.k;
    tk_keys[i] = mine[(1LL * w * a.rows_per_rank + lt) * a.k + j];
  }
  __syncthreads();
  // the key that exactly k - 1 keys exceed (the keys are distinct)
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    const unsigned long long ki = tk_keys[i];
    int above = 0;
    for (int j = 0; j < n; ++j) above += tk_keys[j] > ki;
    if (above == a.k - 1) {
      for (int w = 0; w < a.world; ++w) static_cast<unsigned long long*>(a.cut[w])[t] = ki;
    }
  }
}

// One warp per token: candidates at or above the cut are appended to the entry list.
__global__ void __launch_bounds__(256) token_topk_filter_kernel(CltTopkTpArgs a) {
  if (chain_wait()) return;
  chain_release();
  const int lane = threadIdx.x & 31;
  const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (t >= a.B) return;
  const unsigned long long cut = static_cast<const unsigned long long*>(a.cut[a.rank])[t];
  unsigned long long* n_ent = reinterpret_cast<unsigned long long*>(a.ctl + CTL_NUM_ENTRIES);
  for (int j0 = 0; j0 < a.k; j0 += 32) {
    const int j = j0 + lane;
    const long long i = 1LL * t * a.k + j;
    const bool keep = j < a.k && a.cand_key[i] >= cut;
    const unsigned ball = __ballot_sync(0xFFFFFFFFu, keep);
    if (ball == 0u) continue;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(n_ent, (unsigned long long)__popc(ball));
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (keep) {
      const long long q = (long long)base + __popc(ball & ((1u << lane) - 1u));
      if (q < a.ent_cap) { a.ent_tok[q] = t; a.ent_col[q] = a.cand_col[i]; a.ent_val[q] = a.cand_val[i]; }
      else atomicCAS(a.status, STATUS_OK, STATUS_CAPACITY);
    }
  }
}

// phase: 0 push, 1 cut, 2 filter (the caller puts a phase barrier between them)
extern "C" int clt_token_topk_tp(const CltTopkTpArgs* a, int phase, cudaStream_t st) {
  if (a->world < 1 || a->world > 8 || a->k <= 0 || a->B <= 0 || a->rows_per_rank <= 0) return -1;
  if (1LL * a->world * a->rows_per_rank < a->B) return -1;
  const size_t smem = sizeof(unsigned long long) * size_t(a->world) * size_t(a->k);
  if (smem > 200 * 1024) return -2;
  if (phase == 0) {
    const long long n = 1LL * a->B * a->k;
    const int grid = int((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16);
    launch_chained(token_topk_push_kernel, grid, 256, 0, st, *a);
  } else if (phase == 1) {
    static size_t attr_smem = 0;
    if (smem > 48 * 1024 && smem > attr_smem) {
      if (cudaFuncSetAttribute(token_topk_cut_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) return -4;
      attr_smem = smem;
    }
    launch_chained(token_topk_cut_kernel, a->rows_per_rank, 256, smem, st, *a);
  } else {
    launch_chained(token_topk_filter_kernel, (a->B + 7) / 8, 256, 0, st, *a);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

struct CltCsrArgs {
  const int* ent_tok; const int* ent_col; const float* ent_val; long long ent_cap;
  const long long* ctl;
  int num_tokens; int num_cols;
  int* tok_cnt; int* feat_cnt;        // zeroed by the caller
  int* tok_off; int* feat_off;        // [num_tokens+1], [num_cols+1]
  int* tok_cursor; int* feat_cursor;  // scratch
  int* tcsr_col; float* tcsr_val; int* fcsr_tok; float* fcsr_val;
  unsigned char* fired;               // optional [num_cols]
  int sort_segments;                  // bit 0: token segments, bit 1: feature segments
  int col_pitch;                      // columns are layer * col_pitch + feature (feature < 2^24)
  int* layer_cnt;                     // optional: entries per layer
};

// Features per CTA: as many as fill half of the shared buffer when the list is full, so that small dictionaries with long
// segments get a CTA per feature instead of a few CTAs that sort hundreds of long segments one after the other.
static void launch_feature_sort(const int* off, int num_cols, long long ent_cap, int* key, float* val, cudaStream_t st) {
  if (num_cols <= 0) return;
  int per_cta = 256;
  while (per_cta > 1 && double(ent_cap) / num_cols * per_cta > kFeatSortCap / 2) per_cta /= 2;
  launch_chained(csr_sort_feature_segments_kernel, (num_cols + per_cta - 1) / per_cta, 256, 0, st, off, num_cols, per_cta, key, val);
}

extern "C" int clt_build_csr(const CltCsrArgs* a, cudaStream_t st) {
  const int blocks = 592;
  launch_chained(csr_count_kernel, blocks, 256, 0, st, a->ent_tok, a->ent_col, a->ent_val, a->ent_cap, a->ctl, a->tok_cnt, a->feat_cnt, a->fired,
                                           a->num_tokens, a->num_cols);
  launch_exclusive_scans({a->tok_cnt, a->tok_off, a->tok_cursor, a->num_tokens}, {a->feat_cnt, a->feat_off, a->feat_cursor, a->num_cols}, st);
  launch_chained(csr_scatter_kernel, blocks, 256, 0, st, a->ent_tok, a->ent_col, a->ent_val, a->ent_cap, a->ctl, a->tok_cursor, a->feat_cursor,
                                             a->tcsr_col, a->tcsr_val, a->fcsr_tok, a->fcsr_val, a->col_pitch, a->num_tokens, a->num_cols, a->feat_off, a->layer_cnt);
  if (a->sort_segments & 1) launch_token_sort(a->tok_off, a->tcsr_col, a->tcsr_val, a->num_tokens, a->num_cols, a->col_pitch, st);
  if (a->sort_segments & 2) launch_feature_sort(a->feat_off, a->num_cols, a->ent_cap, a->fcsr_tok, a->fcsr_val, st);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// tok_cnt and layer_cnt are zeroed by the caller, as the counters of clt_build_csr are.
extern "C" int clt_build_token_csr(const CltCsrArgs* a, cudaStream_t st) {
  if (a->num_tokens <= 0) return 0;
  if ((a->num_cols + a->col_pitch - 1) / a->col_pitch > 32) return -1;
  const int blocks = int((a->ent_cap + 255) / 256 < 592 ? (a->ent_cap + 255) / 256 : 592);
  launch_chained(csr_token_count_kernel, blocks, 256, 0, st, a->ent_tok, a->ent_col, a->ent_cap, a->ctl, a->tok_cnt, a->layer_cnt, a->col_pitch, a->num_tokens, a->num_cols);
  const ScanJob job{a->tok_cnt, a->tok_off, a->tok_cursor, a->num_tokens}, none{nullptr, nullptr, nullptr, 0};
  const int tiles = (a->num_tokens + 4095) / 4096;
  if (tiles <= 512 && (reinterpret_cast<uintptr_t>(a->tok_cnt) & 15) == 0) launch_chained(exclusive_scan_tiles_kernel, tiles, 1024, 0, st, job, none, tiles);
  else launch_chained(exclusive_scan_kernel, 1, 1024, 0, st, job.in, job.out, job.cursor, job.n);
  launch_chained(csr_token_scatter_kernel, blocks, 256, 0, st, a->ent_tok, a->ent_col, a->ent_val, a->ent_cap, a->ctl, a->tok_cursor, a->tcsr_col, a->tcsr_val,
                                                   a->col_pitch, a->num_tokens, a->num_cols);
  launch_token_sort(a->tok_off, a->tcsr_col, a->tcsr_val, a->num_tokens, a->num_cols, a->col_pitch, st);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

extern "C" int clt_dead_counter_update(long long* counter, unsigned char* fired, int n, cudaStream_t st) {
  launch_chained(dead_counter_kernel, (n + 255) / 256, 256, 0, st, counter, fired, n);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

// ====================================================================== allocation-free CSR build
#include <cstdio>
#include <mutex>

#include "csr_static.h"

// Scratch of clt_build_csr_static: [tok_cnt | feat_cnt | tok_cursor | feat_cursor], each region sized for the
// maximum problem.  One copy per GPU that loads this library; host code must not pass this name to a kernel
// (on the host it is only a stand-in) - the device address comes from cudaGetSymbolAddress below.
static __device__ __align__(256) int csr_static_scratch[2 * (CLT_CSR_STATIC_MAX_TOKENS + CLT_CSR_STATIC_MAX_COLS)];

namespace {
constexpr int kMaxDevicesStatic = 64;
int* g_static_scratch_ptr[kMaxDevicesStatic] = {nullptr};
std::mutex g_static_scratch_mu;

// Device address of the scratch array on the current device; looked up once per device.
int* csr_static_scratch_address() {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevicesStatic) return nullptr;
  std::lock_guard<std::mutex> lock(g_static_scratch_mu);
  if (g_static_scratch_ptr[dev] == nullptr) {
    int* p = nullptr;
    const cudaError_t rc = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), csr_static_scratch);
    if (rc != cudaSuccess || p == nullptr) {
      fprintf(stderr, "clt_build_csr_static: cudaGetSymbolAddress failed on device %d: %s\n", dev, cudaGetErrorString(rc));
      return nullptr;
    }
    g_static_scratch_ptr[dev] = p;
  }
  return g_static_scratch_ptr[dev];
}
}  // namespace

extern "C" int clt_build_csr_static(const int* ent_tok, const int* ent_col, const float* ent_val, long long ent_cap,
                                    const long long* ctl, int num_tokens, int num_cols, int col_pitch, int* tok_off, int* feat_off,
                                    int* tcsr_col, float* tcsr_val, int* fcsr_tok, float* fcsr_val, int sort_segments,
                                    cudaStream_t stream) {
  if (!ent_tok || !ent_col || !ent_val || !ctl || !tok_off || !feat_off || !tcsr_col || !tcsr_val || !fcsr_tok || !fcsr_val ||
      ent_cap <= 0 || num_tokens <= 0 || num_cols <= 0 || col_pitch <= 0 || col_pitch >= (1 << 24)) {
    fprintf(stderr, "clt_build_csr_static: bad argument (null pointer, non-positive size or col_pitch outside (0, 2^24))\n");
    return -1;
  }
  if (num_tokens > CLT_CSR_STATIC_MAX_TOKENS || num_cols > CLT_CSR_STATIC_MAX_COLS) {
    fprintf(stderr, "clt_build_csr_static: num_tokens=%d / num_cols=%d exceed the built-in scratch (max %d tokens, %d columns); "
                    "use clt_build_csr with caller-provided scratch\n",
            num_tokens, num_cols, CLT_CSR_STATIC_MAX_TOKENS, CLT_CSR_STATIC_MAX_COLS);
    return -2;
  }
  int* scratch = csr_static_scratch_address();
  if (scratch == nullptr) return -3;
  int* tok_cnt = scratch;
  int* feat_cnt = tok_cnt + CLT_CSR_STATIC_MAX_TOKENS;
  int* tok_cursor = feat_cnt + CLT_CSR_STATIC_MAX_COLS;
  int* feat_cursor = tok_cursor + CLT_CSR_STATIC_MAX_TOKENS;
  // the array still holds the previous call's counters: clear the parts that must start at zero
  if (cudaMemsetAsync(tok_cnt, 0, sizeof(int) * size_t(num_tokens), stream) != cudaSuccess) return -5;
  if (cudaMemsetAsync(feat_cnt, 0, sizeof(int) * size_t(num_cols), stream) != cudaSuccess) return -5;
  const int blocks = 592;
  launch_chained(csr_count_kernel, blocks, 256, 0, stream, ent_tok, ent_col, ent_val, ent_cap, ctl, tok_cnt, feat_cnt, nullptr, num_tokens, num_cols);
  launch_chained(exclusive_scan_kernel, 1, 1024, 0, stream, tok_cnt, tok_off, tok_cursor, num_tokens);
  launch_chained(exclusive_scan_kernel, 1, 1024, 0, stream, feat_cnt, feat_off, feat_cursor, num_cols);
  launch_chained(csr_scatter_kernel, blocks, 256, 0, stream, ent_tok, ent_col, ent_val, ent_cap, ctl, tok_cursor, feat_cursor, tcsr_col, tcsr_val,
                                                 fcsr_tok, fcsr_val, col_pitch, num_tokens, num_cols, feat_off, nullptr);
  if (sort_segments & 1) launch_token_sort(tok_off, tcsr_col, tcsr_val, num_tokens, num_cols, col_pitch, stream);
  if (sort_segments & 2) launch_feature_sort(feat_off, num_cols, ent_cap, fcsr_tok, fcsr_val, stream);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}
#endif  // !CLT_T16_IS_HALF
