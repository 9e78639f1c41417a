// Column-parallel encoder GEMM for all layers in one persistent launch (sm_100a).
//
//   C[l][m, n] = sum_k A[l][m, k] * B[l][n, k] + bias[l][n]          (bf16 in, fp32 accumulate, bf16 out)
//
// A = token activations [L, M, K], B = encoder weights [L, N, K] (both K-major), C = pre-activations.
// Counterpart of the reference's per-layer F.linear calls (clt/models/parallel.py:286 through
// clt/models/encoder.py:101).
//
// Two kernels: CTA pairs on transposed tiles (below; from 256 tokens on), and the one here, one CTA per tile, for fewer tokens or few tiles.
//
// Structure of both: one CTA per SM.  Warp 0 feeds a shared-memory ring (here four stages) with TMA tile loads (no cluster
// multicast: every CTA fetches its own tiles), warp 1 issues tcgen05.mma into one of two 256-column TMEM accumulators, eight warps drain the
// other one with tcgen05.ld, add the bias, convert to 16 bit and hand staging tiles to TMA stores (which two more warps issue in the pairs).
// Every mbarrier wait is bounded; on a timeout the CTA records STATUS_WAIT_TIMEOUT, drains its copies,
// frees its TMEM and returns.
#include <climits>
#include <cstdlib>

#include "common.cuh"

namespace clt {

namespace gemm {
constexpr int BM = 128;
constexpr int BN = 256;
constexpr int BK = 64;  // 64 bf16 = one 128-byte swizzled row
constexpr int UMMA_K = 16;
constexpr uint32_t A_BYTES = BM * BK * 2;
constexpr uint32_t B_BYTES = BN * BK * 2;
constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int STAGES = 4;  // as many as fit beside the staging tiles
constexpr int NUM_THREADS = 320;
constexpr uint32_t TMEM_COLS = 512;
}  // namespace gemm

// Epilogue of 32 rows x 128 columns (one warp, lane = row): TMEM -> registers -> + bias -> 16 bit -> shared staging
// tile of 32 rows x 64 columns in the 128-byte-swizzled layout -> one TMA store per 64 columns.  Writing
// full rows through TMA instead of 16 bytes per lane and row keeps the L1/shared data pipe, which the tensor
// core's operand reads share, almost free.
//
// Eight warps drain a tile (two per TMEM lane quarter), and a warp takes all of its 128 columns into registers before it
// converts the first: the accumulator goes back to the MMA warp after the TMEM reads, not after the stores.  With four warps,
// 64 columns at a time, one chain of TMEM read, conversion, staging and store per 64 columns took about 2400 cycles, 9900 a tile,
// where the MMAs of a tile take 4096 at K = 512 (and 6144 at K = 768): the epilogue was what bounded every K below about 900.
constexpr int kEpiCols = 64;
constexpr int kEpiWarps = 8;
constexpr int kEpiWarpCols = 128;
constexpr uint32_t kEpiStageBytes = 32 * kEpiCols * 2;

// `tile`: this warp's staging tile (1024-byte aligned); `chunks` of the two 64-column chunks are inside the matrix; `release` hands the
// accumulator back.
template <typename Release>
__device__ __forceinline__ void epilogue_warp(uint32_t taddr, const CUtensorMap* map_c, uint8_t* tile, const t16* bias_s,
                                              int chunks, int n_base, int m_base, int l, int lane, Release release) {
  uint32_t r[4][32];
#pragma unroll
  for (int j = 0; j < 4; ++j) tmem_ld_32x32(taddr + j * 32, r[j]);
  tmem_ld_wait();
  release();
#pragma unroll
  for (int c = 0; c < kEpiWarpCols / kEpiCols; ++c) {
    if (c >= chunks) break;
    if (lane == 0) bulk_wait_read<0>();  // the store that used the staging tile before has read it
    __syncwarp();
    const uint4* b8 = reinterpret_cast<const uint4*>(bias_s + c * kEpiCols);
#pragma unroll
    for (int j = 0; j < 8; ++j) {  // 16-byte chunk j of this lane's row: columns [8j, 8j + 8)
      const uint32_t* v = &r[2 * c + (j >> 2)][8 * (j & 3)];
      const uint4 b = b8[j];  // the same address in every lane: one broadcast
      uint4 q;
      q.x = pack_t16x2(__uint_as_float(v[0]) + t16_lo(b.x), __uint_as_float(v[1]) + t16_hi(b.x));
      q.y = pack_t16x2(__uint_as_float(v[2]) + t16_lo(b.y), __uint_as_float(v[3]) + t16_hi(b.y));
      q.z = pack_t16x2(__uint_as_float(v[4]) + t16_lo(b.z), __uint_as_float(v[5]) + t16_hi(b.z));
      q.w = pack_t16x2(__uint_as_float(v[6]) + t16_lo(b.w), __uint_as_float(v[7]) + t16_hi(b.w));
      *reinterpret_cast<uint4*>(tile + lane * 128 + ((j ^ (lane & 7)) << 4)) = q;
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) {
      tma_store_3d(map_c, tile, n_base + c * kEpiCols, m_base, l);
      bulk_commit();
    }
  }
}

// This warp's 128 bias values in shared memory (four per lane, 16-bit as they are stored); columns beyond N read 0.
__device__ __forceinline__ void load_bias(t16* bias_s, const t16* bias, long long row, int n_base, int N, int lane) {
  t16 v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int n = n_base + 4 * lane + i;
    v[i] = (bias != nullptr && n < N) ? bias[row + n] : float_to_t16(0.f);
  }
  __syncwarp();  // the previous tile's reads are done
#pragma unroll
  for (int i = 0; i < 2; ++i) reinterpret_cast<t16x2*>(bias_s)[2 * lane + i] = make_t16x2(v[2 * i], v[2 * i + 1]);
  __syncwarp();
}

struct GemmShared {
  uint64_t full[gemm::STAGES];
  uint64_t empty[gemm::STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  alignas(16) t16 bias[kEpiWarps][kEpiWarpCols];  // per epilogue warp: no barrier between the warps of a tile
};
// ring + epilogue staging + barriers and bias
constexpr size_t kGemmSmem = size_t(gemm::STAGES) * gemm::STAGE_BYTES + size_t(kEpiWarps) * kEpiStageBytes + sizeof(GemmShared);
constexpr size_t kMaxDynamicSmem = 227 * 1024;
static_assert(kGemmSmem <= kMaxDynamicSmem, "shared memory of one CTA");

__global__ void __launch_bounds__(gemm::NUM_THREADS, 1)
encoder_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    const __grid_constant__ CUtensorMap map_c, const t16* __restrict__ bias,
                    int L, int M, int N, int K, int* __restrict__ status) {
  using namespace gemm;
  extern __shared__ __align__(1024) uint8_t tiles[];  // 128-byte-swizzled tiles need 1024-byte alignment
  uint8_t* epi_stage = tiles + size_t(STAGES) * STAGE_BYTES;  // 4 KB staging tiles, 1024-byte aligned
  GemmShared* sh = reinterpret_cast<GemmShared*>(epi_stage + kEpiWarps * kEpiStageBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int tiles_m = (M + BM - 1) / BM;
  const int tiles_n = (N + BN - 1) / BN;
  const int num_kb = (K + BK - 1) / BK;
  const long long total_tiles = 1LL * L * tiles_m * tiles_n;
  volatile int* abort_flag = &sh->abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sh->tmem_full[b], 1);
      mbar_init(&sh->tmem_empty[b], kEpiWarps);
    }
    sh->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&sh->tmem_base, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&map_a);
      tma_prefetch_desc(&map_b);
      uint32_t it = 0;
      bool ok = true;
      for (long long t = blockIdx.x; t < total_tiles && ok; t += gridDim.x) {
        const int mt = int(t % tiles_m);
        const int nt = int((t / tiles_m) % tiles_n);
        const int l = int(t / (1LL * tiles_m * tiles_n));
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&sh->empty[s], ph ^ 1, abort_flag)) { ok = false; break; }
          mbar_expect_tx(&sh->full[s], STAGE_BYTES);
          uint8_t* a_dst = tiles + size_t(s) * STAGE_BYTES;
          tma_load_3d(a_dst, &map_a, &sh->full[s], kb * BK, mt * BM, l);
          tma_load_3d(a_dst + A_BYTES, &map_b, &sh->full[s], kb * BK, nt * BN, l);
        }
      }
      if (!ok) {
        // Give the copies already issued a bounded chance to land before the CTA retires.
        const uint32_t issued = it;
        const uint32_t first = issued > STAGES ? issued - STAGES : 0;
        for (uint32_t j = first; j < issued; ++j) {
          const long long start = clock64();
          while (!mbar_try_wait(&sh->full[j % STAGES], (j / STAGES) & 1)) {
            if (clock64() - start > kWaitTimeoutCycles) break;
          }
        }
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer
    if (lane == 0) {
      constexpr uint32_t idesc = umma_idesc_bf16(BM, BN);
      uint32_t it = 0;
      uint32_t local_tile = 0;
      bool ok = true;
      for (long long t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++local_tile) {
        const uint32_t buf = local_tile & 1;
        const uint32_t tph = (local_tile >> 1) & 1;
        if (!mbar_wait(&sh->tmem_empty[buf], tph ^ 1, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * BN;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&sh->full[s], ph, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(tiles + size_t(s) * STAGE_BYTES);
          const uint32_t b_addr = a_addr + A_BYTES;
          const uint64_t a_desc = umma_desc_kmajor_sw128(a_addr);
          const uint64_t b_desc = umma_desc_kmajor_sw128(b_addr);
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            // advance 16 elements (32 bytes) along K inside the swizzled row: +2 in 16-byte units
            umma_bf16_ss(d_tmem, a_desc + uint64_t(k * 2), b_desc + uint64_t(k * 2), idesc, (kb | k) != 0);
          }
          tc_commit(&sh->empty[s]);  // frees the stage when these MMAs have read it
        }
        if (ok) tc_commit(&sh->tmem_full[buf]);
      }
    }
  } else {
    // ---------------------------------------------------------------- epilogue
    const int quarter = warp & 3;  // TMEM lanes [32*quarter, 32*quarter+32) belong to this warp
    const int ew = warp - 2;
    const int col0 = (ew >> 2) * kEpiWarpCols;
    uint8_t* stage = epi_stage + ew * kEpiStageBytes;
    uint32_t local_tile = 0;
    bool ok = true;
    for (long long t = blockIdx.x; t < total_tiles && ok; t += gridDim.x, ++local_tile) {
      const int mt = int(t % tiles_m);
      const int nt = int((t / tiles_m) % tiles_n);
      const int l = int(t / (1LL * tiles_m * tiles_n));
      const uint32_t buf = local_tile & 1;
      const uint32_t tph = (local_tile >> 1) & 1;
      const int n_base = nt * BN + col0;
      load_bias(sh->bias[ew], bias, 1LL * l * N, n_base, N, lane);
      ok = mbar_wait_leader(&sh->tmem_full[buf], tph, abort_flag, lane);
      if (!ok) break;
      tc_fence_after();
      const int m_base = (mt) * BM + quarter * 32;
      const uint32_t taddr = tmem_base + buf * BN + col0 + (uint32_t(quarter * 32) << 16);
      const int chunks = m_base < M ? (N - n_base + kEpiCols - 1) / kEpiCols : 0;
      const auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sh->tmem_empty[buf]);
      };
      if (chunks > 0)
        epilogue_warp(taddr, &map_c, stage, sh->bias[ew], chunks, n_base, m_base, l, lane, release);
      else
        release();
    }
  }

  if (warp >= 2 && lane == 0) bulk_wait_all();  // output stores of this warp are complete
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, TMEM_COLS);
  }
  if (threadIdx.x == 0 && sh->abort_flag && status != nullptr) atomicCAS(status, STATUS_OK, STATUS_WAIT_TIMEOUT);
}

// ------------------------------------------------------------------ CTA-pair variant (cta_group::2)
// Two CTAs of a cluster work on one tile of 256 features x 256 tokens, transposed: the weights are the A operand (128 features per CTA,
// one per TMEM lane) and the tokens the B operand (each CTA loads one half of the tile's tokens), so a CTA's accumulator holds
// all tokens of the tile for its own 128 features.  The leader CTA issues tcgen05.mma with cta_group::2 (M = 256), which
// reads the operand halves from both CTAs' shared memory.  Per CTA and k-step this moves 32 KB from L2 instead of the 48 KB of one CTA per
// tile for the same number of MMA cycles, and the ring holds six stages instead of four.  No multicast loads: tcgen05.commit is the only
// multicast (barrier arrivals).
//
//   full[s]        leader only: armed by the leader's producer for the bytes of both CTAs
//   empty[s]       both CTAs: commit (multicast) after the MMAs of the stage
//   tmem_full[b]   both CTAs: commit (multicast) after the tile's last MMA
//   tmem_empty[b]  leader only: 16 arrivals, eight epilogue warps of each CTA
//
// Column statistics (STATS).  The batch mean and deviation of a feature are sums over all tokens, which took a second pass over the
// output (2.4 GB and 395 us at 12 x 4096 x 24576, 3.2 GB and 620 us at 6 x 8192 x 32768).  With the features on the lanes
// and tcgen05.ld.16x256b, whose thread holds tokens 2q and 2q + 1 of every eight for two features, each of the eight sums per feature that
// colstats_kernel keeps (rows r = y mod 8, in order) lies in one register of one thread.  A pair takes the token tiles of a strip of 256
// features one after the other and carries the sums along: no shuffle, no shared memory and no partial sums per tile, and the same
// additions in the same order as in the separate pass, so that the statistics are the same bit for bit (where that pass takes the rows in at most two
// chunks; the sums of more chunks it adds by atomics, in no fixed order).  (Sums per tile, in another
// order, were tried before: +0.15 ms at K = 768, and a last bit that moves single entries across the cut of the selection.)
// Strips that do not fill a round of all pairs are taken tile by tile, and their statistics by colstats_kernel.
namespace gemm2 {
constexpr int BF = 128;       // features per CTA; the pair covers 256
constexpr int BT = 256;       // tokens per tile
constexpr int BT_HALF = 128;  // token rows loaded per CTA
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr uint32_t A_BYTES = BF * BK * 2;
constexpr uint32_t B_BYTES = BT_HALF * BK * 2;
constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int STAGES = 6;
constexpr int NUM_THREADS = 384;  // producer, MMA, eight epilogue warps, two store warps
constexpr uint32_t TMEM_COLS = 512;
constexpr int kChunk = 64;                                 // tokens per output store
constexpr uint32_t kChunkBytes = kChunk * 128;             // 64 tokens x 64 features, 128-byte swizzle
constexpr uint32_t kStagingBytes = 4 * kChunkBytes;        // two buffers for each half of the CTA's features

// The staging buffers go back and forth between four epilogue warps and a store warp by named barriers: a hop takes some 30 cycles, by mbarrier
// (a suspended waiter that has to wake up) several hundred, and 64 tokens of 64 features are written in about 300.
constexpr int kOutThreads = 32 * (kEpiWarps / 2 + 1);
__device__ __forceinline__ int bar_full(int group, int out) { return 1 + 2 * group + out; }
__device__ __forceinline__ int bar_free(int group, int out) { return 5 + 2 * group + out; }

struct Shared {
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
};
constexpr size_t kSmem = size_t(STAGES) * STAGE_BYTES + kStagingBytes + sizeof(Shared);
static_assert(kSmem <= kMaxDynamicSmem, "shared memory of one CTA");

// The tiles of one pair in order: its share of the strips below `main_strips`, all token tiles of one after the other, then its share of the
// tiles of the other strips.  Steps without a division: the MMA thread takes one between two tiles, and what it takes longer there the tensor
// cores stand still (with two 64-bit divisions 8 % at K = 512, 5 % at K = 768).
struct TileWalk {
  int tiles_m, tiles_n;
  int main_left, left;      // tiles of whole strips, all tiles
  int l, nt, mt;
  int step_l, step_n;       // whole strips: npairs strips on
  int tail_l, tail_n, tail_m;                  // first of the other tiles
  int tail_step_l, tail_step_n, tail_step_m;   // npairs tiles on
  __device__ TileWalk(int pair, int npairs, int tiles_m_, int tiles_n_, int L, long long main_strips) : tiles_m(tiles_m_), tiles_n(tiles_n_) {
    const long long tail = (1LL * L * tiles_n - main_strips) * tiles_m;
    main_left = main_strips > pair ? int((main_strips - pair + npairs - 1) / npairs) * tiles_m : 0;
    left = main_left + (tail > pair ? int((tail - pair + npairs - 1) / npairs) : 0);
    step_l = npairs / tiles_n; step_n = npairs % tiles_n;
    const long long first = main_strips + pair / tiles_m;
    tail_l = int(first / tiles_n); tail_n = int(first % tiles_n); tail_m = pair % tiles_m;
    const int q = npairs / tiles_m;
    tail_step_l = q / tiles_n; tail_step_n = q % tiles_n; tail_step_m = npairs % tiles_m;
    l = pair / tiles_n; nt = pair % tiles_n; mt = 0;
    if (main_left == 0) { l = tail_l; nt = tail_n; mt = tail_m; }
  }
  __device__ bool done() const { return left == 0; }
  __device__ bool whole_strip() const { return main_left > 0; }
  __device__ void strips_on(int dl, int dn) {
    l += dl; nt += dn;
    if (nt >= tiles_n) { nt -= tiles_n; ++l; }
  }
  __device__ void next() {
    --left;
    if (main_left > 0) {
      if (--main_left == 0) { l = tail_l; nt = tail_n; mt = tail_m; return; }
      if (++mt == tiles_m) { mt = 0; strips_on(step_l, step_n); }
    } else {
      mt += tail_step_m;
      const int carry = mt >= tiles_m ? 1 : 0;
      if (carry) mt -= tiles_m;
      strips_on(tail_step_l, tail_step_n + carry);
    }
  }
};
// Tokens of the tile that starts at m_base, as the N of its MMAs: no work for a ragged end beyond the next multiple of 32.
__device__ __forceinline__ int tile_tokens(int M, int m_base) { return min(BT, (M - m_base + 31) & ~31); }

// The sums of one thread: features a and b (rows lane / 4 and lane / 4 + 8 of its warp's 16), each as two sums (tokens 2q and 2q + 1 of every
// eight, q = lane % 4) and two sums of squares, packed for the two-wide fp32 instructions.
struct StripSums {
  float2 sa, qa, sb, qb;    // of the current chunk of rows
  float ta, ua, tb, ub;     // over the chunks before it (see colstats_kernel: rows split over blockIdx.z)
  float shift_a, shift_b;   // the first token's value
};
// Two stored values (tokens t and t + 1 of a feature); `valid` of them are rows of the matrix, the others add nothing.
template <bool MASKED>
__device__ __forceinline__ void add_pair(float2& s, float2& q, uint32_t u, float shift, int valid) {
  float2 a = f2_add(make_float2(t16_lo(u), t16_hi(u)), make_float2(-shift, -shift));
  if constexpr (MASKED) {
    a.x = valid > 0 ? a.x : 0.f;
    a.y = valid > 1 ? a.y : 0.f;
  }
  s = f2_add(s, a);
  q = f2_fma(a, a, q);
}
// The eight sums of a feature lie in four lanes; added in the order y = 0..7 of colstats_kernel.
__device__ __forceinline__ float fold8(float2 v, int lane) {
  float t = 0.f;
#pragma unroll
  for (int y = 0; y < 8; ++y) t += __shfl_sync(0xFFFFFFFFu, (y & 1) ? v.y : v.x, (lane & ~3) + (y >> 1));
  return t;
}
__device__ __forceinline__ void fold_sums(StripSums& S, int lane) {
  S.ta += fold8(S.sa, lane); S.ua += fold8(S.qa, lane);
  S.tb += fold8(S.sb, lane); S.ub += fold8(S.qb, lane);
  S.sa = S.qa = S.sb = S.qb = make_float2(0.f, 0.f);
}

// 64 tokens of this warp's 16 features: + bias -> 16 bit -> staging buffer (token rows of 64 features; stmatrix with transposition), and the
// sums.  v: eight groups of eight tokens, four registers each (feature a tokens 2q, 2q + 1, feature b the same).  `row`: this lane's row address
// in the buffer.
template <bool STATS, bool MASKED>
__device__ __forceinline__ void chunk_out(const uint32_t (&v)[32], uint32_t row, float bias_a, float bias_b, StripSums& S, int tok0, int M, int next_fold,
                                          int lane) {
  const float2 ba = make_float2(bias_a, bias_a), bb = make_float2(bias_b, bias_b);
#pragma unroll
  for (int j = 0; j < 4; ++j) {  // 16 tokens
    uint32_t p[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      const float2 x = f2_add(make_float2(__uint_as_float(v[8 * j + 2 * h]), __uint_as_float(v[8 * j + 2 * h + 1])), (h & 1) ? bb : ba);
      p[h] = pack_t16x2(x.x, x.y);
    }
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};"
                 ::"r"(row + j * 16 * 128), "r"(p[0]), "r"(p[1]), "r"(p[2]), "r"(p[3]) : "memory");
    if constexpr (STATS) {
      if (j == 0 && tok0 == 0) {  // the matrix' first row
        S.shift_a = __shfl_sync(0xFFFFFFFFu, t16_lo(p[0]), lane & ~3);
        S.shift_b = __shfl_sync(0xFFFFFFFFu, t16_lo(p[1]), lane & ~3);
      }
      if (MASKED && (j & 1) == 0 && tok0 + 16 * j == next_fold) fold_sums(S, lane);
      const int left = M - (tok0 + 16 * j + 2 * (lane & 3));
      add_pair<MASKED>(S.sa, S.qa, p[0], S.shift_a, left);
      add_pair<MASKED>(S.sb, S.qb, p[1], S.shift_b, left);
      add_pair<MASKED>(S.sa, S.qa, p[2], S.shift_a, left - 8);
      add_pair<MASKED>(S.sb, S.qb, p[3], S.shift_b, left - 8);
    }
  }
}

// 16 lanes x 64 fp32 columns: thread t receives, per eight columns, columns 2 (t % 4) + {0, 1} of rows t / 4 and t / 4 + 8.
__device__ __forceinline__ void tmem_ld_16x256b_x8(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x8.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
}  // namespace gemm2

template <bool STATS>
__global__ void __launch_bounds__(gemm2::NUM_THREADS, 1)
encoder_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                         const __grid_constant__ CUtensorMap map_c, const t16* __restrict__ bias, int L, int M, int N, int K,
                         int* __restrict__ status, long long main_strips, int rows_per_fold, float* __restrict__ mean, float* __restrict__ rstd) {
  using namespace gemm2;
  extern __shared__ __align__(1024) uint8_t tiles[];
  uint8_t* staging = tiles + size_t(STAGES) * STAGE_BYTES;
  Shared* sh = reinterpret_cast<Shared*>(staging + kStagingBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();
  const bool leader = cta_rank == 0;
  const int tiles_m = (M + BT - 1) / BT;
  const int tiles_n = (N + 2 * BF - 1) / (2 * BF);
  const int num_kb = (K + BK - 1) / BK;
  volatile int* abort_flag = &sh->abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sh->tmem_full[b], 1);
      mbar_init(&sh->tmem_empty[b], 2 * kEpiWarps);
    }
    sh->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&sh->tmem_base, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;
  TileWalk walk(int(blockIdx.x >> 1), int(gridDim.x >> 1), tiles_m, tiles_n, L, main_strips);

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (lane == 0) {
      tma_prefetch_desc(&map_w);
      tma_prefetch_desc(&map_x);
      int s = 0;
      uint32_t ph = 1;
      bool ok = true;
      for (; ok && !walk.done(); walk.next()) {
        const int feat = (walk.nt * 2 + int(cta_rank)) * BF;
        const int tok = walk.mt * BT + int(cta_rank) * (tile_tokens(M, walk.mt * BT) / 2);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&sh->empty[s], ph, abort_flag)) { ok = false; break; }
          if (leader) mbar_expect_tx(&sh->full[s], 2 * STAGE_BYTES);
          const uint32_t full_leader = mapa_shared(smem_u32(&sh->full[s]), 0);
          uint8_t* a_dst = tiles + size_t(s) * STAGE_BYTES;
          tma_load_3d_pair(a_dst, &map_w, full_leader, kb * BK, feat, walk.l);
          tma_load_3d_pair(a_dst + A_BYTES, &map_x, full_leader, kb * BK, tok, walk.l);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
      }
      // Copies still in flight are counted on the leader's barriers, which the MMA thread consumes; a CTA
      // that gave up waits below (cluster barrier) until its partner is done as well.
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer (leader CTA only)
    if (lane == 0 && leader) {
      const uint64_t a_desc0 = umma_desc_kmajor_sw128(smem_u32(tiles));
      const uint64_t b_desc0 = umma_desc_kmajor_sw128(smem_u32(tiles) + A_BYTES);
      constexpr uint32_t kFullTile = umma_idesc_bf16(2 * BF, BT);
      int s = 0;
      uint32_t ph = 0, buf = 0, tph = 1;
      bool ok = true;
      for (; ok && !walk.done(); walk.next()) {
        if (!mbar_wait(&sh->tmem_empty[buf], tph, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t idesc = walk.mt == tiles_m - 1 ? umma_idesc_bf16(2 * BF, tile_tokens(M, walk.mt * BT)) : kFullTile;
        const uint32_t d_tmem = tmem_base + buf * BT;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&sh->full[s], ph, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint64_t a_desc = a_desc0 + uint64_t(s * int(STAGE_BYTES >> 4));
          const uint64_t b_desc = b_desc0 + uint64_t(s * int(STAGE_BYTES >> 4));
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k)
            umma_bf16_ss_pair(d_tmem, a_desc + uint64_t(k * 2), b_desc + uint64_t(k * 2), idesc, (kb | k) != 0);
          tc_commit_pair(&sh->empty[s], 3);  // frees the stage in both CTAs
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (ok) tc_commit_pair(&sh->tmem_full[buf], 3);
        buf ^= 1;
        if (buf == 0) tph ^= 1;
      }
    }
  } else if (warp < 2 + kEpiWarps) {
    // ---------------------------------------------------------------- epilogue (both CTAs)
    // TMEM lanes [32 quarter, +32) are open to a warp, it takes 16 of them; four warps fill the staging buffers of 64 features.
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    const int group = quarter >> 1;
    const int lane16 = 32 * quarter + 16 * half;
    // stmatrix: lane i gives row i % 8 (a token) of matrix i / 8: features 0-7, 8-15, then the same for the next eight tokens
    const uint32_t piece = uint32_t((quarter & 1) * 4 + half * 2 + ((lane >> 3) & 1));  // 16-byte piece of the 128-byte row
    const uint32_t rows = smem_u32(staging + group * 2 * kChunkBytes) + uint32_t(8 * (lane >> 4) + (lane & 7)) * 128 + ((piece ^ uint32_t(lane & 7)) << 4);
    uint32_t buf = 0, tph = 0, chunk_no = 0;
    StripSums S = {};
    float bias_a = 0.f, bias_b = 0.f;
    int next_fold = 0;
    // After a wait that ran out the warp goes on through its tiles without touching memory, so that nobody is left alone at a named barrier.
    bool new_strip = true, ok = true;
    for (; !walk.done(); walk.next()) {
      const int fa = (walk.nt * 2 + int(cta_rank)) * BF + lane16 + (lane >> 2), fb = fa + 8;
      const bool stats = STATS && walk.whole_strip();
      if (new_strip) {
        bias_a = (bias != nullptr && fa < N) ? t16_to_float(bias[1LL * walk.l * N + fa]) : 0.f;
        bias_b = (bias != nullptr && fb < N) ? t16_to_float(bias[1LL * walk.l * N + fb]) : 0.f;
        S = StripSums{};
        next_fold = rows_per_fold;
      }
      const int m_base = walk.mt * BT;
      new_strip = !walk.whole_strip() || walk.mt == tiles_m - 1;
      if (ok) ok = mbar_wait_leader(&sh->tmem_full[buf], tph, abort_flag, lane);
      tc_fence_after();
      const uint32_t taddr = tmem_base + buf * BT + (uint32_t(lane16) << 16);
      const int chunks = min(BT / kChunk, (M - m_base + kChunk - 1) / kChunk);
      uint32_t r[2][32];
      if (ok) tmem_ld_16x256b_x8(taddr, r[0]);
#pragma unroll  // two copies of the body instead of four: 605 against 563 thousand cycles at K = 512, with the sums behind the store: 623
      for (int c = 0; c < BT / kChunk; ++c) {
        if (c < chunks) {
          const int tok0 = m_base + c * kChunk;
          tmem_ld_wait();
          if (c + 1 < chunks) {
            if (ok) tmem_ld_16x256b_x8(taddr + (c + 1) * kChunk, r[(c + 1) & 1]);  // in flight while this chunk is converted
          } else {  // the accumulator goes back (leader's barrier)
            tc_fence_before();
            __syncwarp();
            if (ok && lane == 0) mbar_arrive_cluster(mapa_shared(smem_u32(&sh->tmem_empty[buf]), 0));
          }
          const int out = chunk_no & 1;
          if (chunk_no >= 2) named_barrier_sync(bar_free(group, out), kOutThreads);
          ++chunk_no;
          if (ok) {
            const uint32_t row = rows + out * kChunkBytes;
            if (!stats)
              chunk_out<false, false>(r[c & 1], row, bias_a, bias_b, S, tok0, M, -1, lane);
            else if (tok0 + kChunk <= min(M, next_fold))
              chunk_out<STATS, false>(r[c & 1], row, bias_a, bias_b, S, tok0, M, -1, lane);
            else
              chunk_out<STATS, true>(r[c & 1], row, bias_a, bias_b, S, tok0, M, next_fold, lane);
          }
          if (STATS && next_fold < tok0 + kChunk) next_fold += rows_per_fold;
          named_barrier_arrive(bar_full(group, out), kOutThreads);
        }
      }
      if constexpr (STATS) {
        if (ok && stats && new_strip) {
          fold_sums(S, lane);
          if ((lane & 3) == 0) {
            if (fa < N) colstats_finish(S.ta, S.ua, S.shift_a, M, &mean[1LL * walk.l * N + fa], &rstd[1LL * walk.l * N + fa]);
            if (fb < N) colstats_finish(S.tb, S.ub, S.shift_b, M, &mean[1LL * walk.l * N + fb], &rstd[1LL * walk.l * N + fb]);
          }
        }
      }
      buf ^= 1;
      if (buf == 0) tph ^= 1;
    }
    for (int i = 0; i < 2; ++i)  // the last two buffers come back
      if (chunk_no >= 2 - i) named_barrier_sync(bar_free(group, (chunk_no + i) & 1), kOutThreads);
  } else {
    // ---------------------------------------------------------------- output stores, one warp for each half of the features
    const int group = warp - 2 - kEpiWarps;
    int chunk_no = 0;
    for (; !walk.done(); walk.next()) {
      const int feat = (walk.nt * 2 + int(cta_rank)) * BF + group * 64;
      const int end = min(M, (walk.mt + 1) * BT);
      for (int tok = walk.mt * BT; tok < end; tok += kChunk, ++chunk_no) {
        const int out = chunk_no & 1;
        named_barrier_sync(bar_full(group, out), kOutThreads);
        if (lane == 0) {
          fence_proxy_async();  // here and not in the warps that wrote: it stands some 500 cycles while loads are in flight
          if (feat < N && *abort_flag == 0) tma_store_3d(&map_c, staging + (group * 2 + out) * kChunkBytes, feat, tok, walk.l);
          bulk_commit();  // also without a store: the wait counts groups
          bulk_wait_read<1>();
        }
        __syncwarp();
        if (chunk_no > 0) named_barrier_arrive(bar_free(group, out ^ 1), kOutThreads);  // the buffer of the chunk before has been read
      }
    }
    if (lane == 0) bulk_wait_all();  // the output stores are complete
    __syncwarp();
    if (chunk_no > 0) named_barrier_arrive(bar_free(group, (chunk_no - 1) & 1), kOutThreads);
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // neither CTA retires (or frees TMEM) while the other may still use its memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
  if (threadIdx.x == 0 && sh->abort_flag && status != nullptr) atomicCAS(status, STATUS_OK, STATUS_WAIT_TIMEOUT);
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// [layers, rows, K] bf16, K contiguous; box = [1, box_rows, 64] with the 128-byte swizzle.
static bool make_kmajor_map(CUtensorMap* map, const void* base, int layers, int rows, int K, long long row_stride_elems,
                            long long layer_stride_elems, int box_rows) {
  EncodeTiledFn enc = get_encode_fn();
  if (enc == nullptr) return false;
  cuuint64_t dims[3] = {cuuint64_t(K), cuuint64_t(rows), cuuint64_t(layers)};
  cuuint64_t strides[2] = {cuuint64_t(row_stride_elems) * 2, cuuint64_t(layer_stride_elems) * 2};
  cuuint32_t box[3] = {cuuint32_t(gemm::BK), cuuint32_t(box_rows), 1};
  cuuint32_t elem[3] = {1, 1, 1};
  CUresult r = enc(map, (CLT_T16_IS_HALF ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16), 3, const_cast<void*>(base), dims, strides, box, elem,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// Rows that colstats_kernel puts into one chunk of its sums (one chunk unless the columns alone leave SMs idle).
extern "C" int clt_colstats_splits(int L, int B, int F);
static int rows_per_chunk(int L, int B, int F) {
  const int z = clt_colstats_splits(L, B, F);
  return ((B + z - 1) / z + 31) / 32 * 32;
}

// How many strips of 256 features the pairs take whole, with the statistics: all of them, in ceil(strips / pairs) rounds, the last of which
// may leave pairs idle; full rounds only, the rest tile by tile over all pairs with a separate pass for its statistics; or none, with a pass over
// everything.  Estimates in us, fitted to 4 to 600 strips of 256 to 8192 rows with K = 64 to 2048, taken all three ways (the choice is
// within 5 % of the best for all but 16 of 1150 shapes, and 2 to 9 % behind the third for four, with K = 2048):
//  * a tile of a whole strip takes a pair 1.2 + 0.0057 K, 0.0048 K in a round that is not full (clocks are higher then), at least the 3.4 of its
//    epilogue; a tile without sums 1.2 + 0.005 K, at least 2.5;
//  * a pass takes 10 (clears, sums, conversion) and 0.024 per tile, or 0.047 with two columns per thread, as behind whole strips, and 0.003 or
//    0.007 for each row of a chunk, which one thread waits for in turn.
// 16 strips of 8192 rows, K = 64: whole 100 us, none 46; 32, K = 768: 146 and 106; 64 of 4096, K = 768: 84 and 104; 130, K = 2048: whole 383, full
// rounds only 452, none 415; 80 of 8192, K = 2048: 739, 484 and 508; 96: 793, 669 and 636.
static long long whole_strips(long long strips, int npairs, int tiles_m, int K, int rows_per_fold) {
  const long long full = strips / npairs * npairs, tail = (strips - full) * tiles_m;
  if (tail == 0) return strips;
  const auto at_least = [](double least, double t) { return t < least ? least : t; };
  const double rounds = at_least(3.4, 1.2 + 0.0057 * K) * double(full / npairs) * tiles_m;
  const double plain_tile = at_least(2.5, 1.2 + 0.005 * K);
  const auto plain = [&](long long tiles) { return plain_tile * double((tiles + npairs - 1) / npairs); };
  const double all = rounds + at_least(3.4, 1.2 + 0.0048 * K) * tiles_m;
  const double split = rounds + plain(tail) + 10.0 + 0.047 * double(tail) + 0.007 * rows_per_fold;
  const double none = plain(strips * tiles_m) + 10.0 + 0.024 * double(strips * tiles_m) + 0.003 * rows_per_fold;
  const double other = split < none ? split : none;
  return all <= 1.01 * other ? strips : split < none ? full : 0;
}

template <bool STATS>
static int launch_pair(const CUtensorMap& map_w, const CUtensorMap& map_x, const CUtensorMap& map_c, const t16* bias, int L, int M, int N, int K,
                       int* status, float* mean, float* rstd, long long* whole, int num_sms, cudaStream_t stream) {
  auto* kernel = encoder_gemm_pair_kernel<STATS>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * num_sms);
  cfg.blockDim = dim3(gemm2::NUM_THREADS);
  cfg.dynamicSmemBytes = gemm2::kSmem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // co-resident clusters of two, probed once per device (the kernel's shared memory limit belongs to the device as well)
  constexpr int kDevices = 64;
  static int probed[kDevices] = {};  // clusters + 1, 0: not yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return -5;
  int n = dev < kDevices ? probed[dev] : 0;
  if (n == 0) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(gemm2::kSmem)) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
      n = 0;
      (void)cudaGetLastError();
    }
    ++n;
    if (dev < kDevices) probed[dev] = n;
  }
  const int pair_clusters = n - 1;
  if (pair_clusters <= 0) return 1;
  const int tiles_m = (M + gemm2::BT - 1) / gemm2::BT;
  const long long strips = 1LL * L * ((N + 2 * gemm2::BF - 1) / (2 * gemm2::BF));
  const int npairs = int(strips * tiles_m < pair_clusters ? strips * tiles_m : pair_clusters);
  const int rows_per_fold = STATS ? rows_per_chunk(L, M, N) : 0;
  *whole = STATS ? whole_strips(strips, npairs, tiles_m, K, rows_per_fold) : 0;
  if constexpr (STATS) {
    if (*whole == 0) return launch_pair<false>(map_w, map_x, map_c, bias, L, M, N, K, status, nullptr, nullptr, whole, num_sms, stream);
  }
  cfg.gridDim = dim3(unsigned(2 * npairs));
  if (cudaLaunchKernelEx(&cfg, kernel, map_w, map_x, map_c, bias, L, M, N, K, status, *whole, rows_per_fold, mean, rstd) != cudaSuccess) return -5;
  return 0;
}

static int launch_single(const CUtensorMap& map_a, const CUtensorMap& map_b, const CUtensorMap& map_c, const t16* bias, int L, int M, int N, int K, int* status,
                         int num_sms, cudaStream_t stream) {
  static bool attr_set = false;
  if (!attr_set) {
    if (cudaFuncSetAttribute(encoder_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kGemmSmem)) != cudaSuccess) return -4;
    attr_set = true;
  }
  const long long tiles = 1LL * L * ((M + gemm::BM - 1) / gemm::BM) * ((N + gemm::BN - 1) / gemm::BN);
  const int grid = int(tiles < num_sms ? tiles : num_sms);
  launch_alone(encoder_gemm_kernel, grid, gemm::NUM_THREADS, kGemmSmem, stream, map_a, map_b, map_c, bias, L, M, N, K, status);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

static int encoder_gemm(const void* A, const void* B, const void* bias, void* C, int L, int M, int N, int K, long long ldc, long long layer_stride_c,
                        int* status, float* mean, float* rstd, long long* whole, int num_sms, cudaStream_t stream) {
  *whole = 0;
  if (K % 8 != 0 || ldc % 8 != 0 || layer_stride_c % 8 != 0) return -1;  // 16-byte TMA strides / vector stores
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15) return -2;
  CUtensorMap map_a, map_b, map_c;
  if (!make_kmajor_map(&map_a, A, L, M, K, K, 1LL * M * K, gemm::BM)) return -3;
  // CLT_GEMM_SINGLE_CTA=1 keeps the single-CTA 128x256 kernel for every shape (for comparisons)
  static const bool force_single = [] { const char* e = getenv("CLT_GEMM_SINGLE_CTA"); return e != nullptr && e[0] == '1'; }();
  if (1LL * L * M * N == 0) return 0;
  const t16* bias_p = static_cast<const t16*>(bias);
  // CTA pairs when the problem has full tiles of 256 tokens, and without statistics more tiles than one round of the single CTAs, which start
  // and end sooner (us in pairs / alone: 1 x 256 x 2048, K = 64 8.3 / 6.5; 1 x 256 x 8192, K = 256 10.3 / 8.3; 9 x 256 x 2048, K = 1024 14.4 / 12.4, K = 2048
  // 20.6 / 20.6); with two to three rounds they are level up to K = 512 and pairs ahead beyond it (9 x 600 x 2048, K = 2048 45 / 53).
  const long long singles = 1LL * L * ((M + gemm::BM - 1) / gemm::BM) * ((N + gemm::BN - 1) / gemm::BN);
  if (M >= gemm2::BT && !force_single && (mean != nullptr || singles > num_sms)) {
    if (!make_kmajor_map(&map_b, B, L, N, K, K, 1LL * N * K, gemm2::BF)) return -3;
    // output map: [L, M, N] with boxes of 64 features x 64 tokens (one store), clipped at M and N
    if (!make_kmajor_map(&map_c, C, L, M, N, ldc, layer_stride_c, gemm2::kChunk)) return -3;
    static_assert(gemm::BM == gemm2::BT_HALF, "one map of the tokens serves both kernels");
    const int r = mean != nullptr ? launch_pair<true>(map_b, map_a, map_c, bias_p, L, M, N, K, status, mean, rstd, whole, num_sms, stream)
                                  : launch_pair<false>(map_b, map_a, map_c, bias_p, L, M, N, K, status, nullptr, nullptr, whole, num_sms, stream);
    if (r <= 0) return r;  // 1: the device cannot co-schedule clusters of two
  }
  if (!make_kmajor_map(&map_b, B, L, N, K, K, 1LL * N * K, gemm::BN)) return -3;
  // output map: boxes of 64 columns x 32 rows (one epilogue slab store)
  if (!make_kmajor_map(&map_c, C, L, M, N, ldc, layer_stride_c, 32)) return -3;
  return launch_single(map_a, map_b, map_c, bias_p, L, M, N, K, status, num_sms, stream);
}

// Sums and sums of squares of the stored outputs per block of 128 rows: one CTA for a block of 256 columns, 16 rows per thread, eight columns each.
__global__ void __launch_bounds__(256) block_sums_kernel(const t16* __restrict__ C, float2* __restrict__ sums, int M, int N, long long ldc, long long layer_stride_c) {
  if (chain_wait()) return;
  chain_release();
  const int col_blocks = (N + 255) / 256, row_blocks = (M + 127) / 128;
  const int cb = int(blockIdx.x % col_blocks), rest = int(blockIdx.x / col_blocks), rb = rest % row_blocks, l = rest / row_blocks;
  const int c0 = (cb * 32 + int(threadIdx.x)) * 8, r1 = min(M, (rb + 1) * 128);
  __shared__ float red[8][32][17];
  float s[8], q[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) s[j] = q[j] = 0.f;
  if (c0 < N) {
    const t16* base = C + 1LL * l * layer_stride_c + c0;
#pragma unroll 8
    for (int r = rb * 128 + int(threadIdx.y); r < r1; r += 8) {
      const uint4 v = __ldcs(reinterpret_cast<const uint4*>(base + 1LL * r * ldc));
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float a = t16_lo(u[j]), b = t16_hi(u[j]);
        s[2 * j] += a; q[2 * j] = fmaf(a, a, q[2 * j]);
        s[2 * j + 1] += b; q[2 * j + 1] = fmaf(b, b, q[2 * j + 1]);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) { red[threadIdx.y][threadIdx.x][j] = s[j]; red[threadIdx.y][threadIdx.x][8 + j] = q[j]; }
  __syncthreads();
  const int col = int(threadIdx.y) * 32 + int(threadIdx.x), n = cb * 256 + col;
  if (n >= N) return;
  float ss = 0.f, qq = 0.f;
#pragma unroll
  for (int y = 0; y < 8; ++y) { ss += red[y][col >> 3][col & 7]; qq += red[y][col >> 3][8 + (col & 7)]; }
  sums[(1LL * l * row_blocks + rb) * N + n] = make_float2(ss, qq);
}

}  // namespace clt

// Returns 0 on success, a negative value when the arguments cannot be handled (the caller raises).
// tile_stats (optional): [L][ceil(M / 128)][N][2] fp32, receives per 128-row block and column the sum and the sum of
// squares of the stored (16-bit-rounded) outputs; every element is written, nothing has to be cleared.
extern "C" int CLT_FN(clt_encoder_gemm)(const void* A, const void* B, const void* bias, void* C, int L, int M, int N, int K,
                                long long ldc, long long layer_stride_c, int* status, float* tile_stats, int num_sms, cudaStream_t stream) {
  using namespace clt;
  long long whole;
  const int r = encoder_gemm(A, B, bias, C, L, M, N, K, ldc, layer_stride_c, status, nullptr, nullptr, &whole, num_sms, stream);
  if (r != 0 || tile_stats == nullptr || 1LL * L * M * N == 0) return r;
  const long long ctas = 1LL * L * ((M + 127) / 128) * ((N + 255) / 256);
  if (ctas > INT_MAX) return -1;
  launch_chained(block_sums_kernel, dim3(unsigned(ctas)), dim3(32, 8), 0, stream, static_cast<const t16*>(C), reinterpret_cast<float2*>(tile_stats), M, N,
                 ldc, layer_stride_c);
  return cudaGetLastError() == cudaSuccess ? 0 : -5;
}

extern "C" int CLT_FN(clt_colstats_strips)(const void* x, float* mean, float* rstd, int L, int B, int F, long long ld, long long layer_stride,
                                           long long first_strip, int* kernels, cudaStream_t st);

// The GEMM and the batch statistics mean / rstd [L, N] of its stored outputs (C contiguous), equal bit for bit to clt_colstats on C where
// that takes the rows in at most two chunks.
// *kernels: how many kernels were launched.
extern "C" int CLT_FN(clt_encoder_gemm_stats)(const void* A, const void* B, const void* bias, void* C, int L, int M, int N, int K,
                                      int* status, float* mean, float* rstd, int* kernels, int num_sms, cudaStream_t stream) {
  long long whole;
  *kernels = 0;
  const int r = clt::encoder_gemm(A, B, bias, C, L, M, N, K, N, 1LL * M * N, status, mean, rstd, &whole, num_sms, stream);
  if (r != 0 || 1LL * L * M * N == 0) return r;
  const int rs = CLT_FN(clt_colstats_strips)(C, mean, rstd, L, M, N, N, 1LL * M * N, whole, kernels, stream);
  *kernels += 1;
  return rs;
}
