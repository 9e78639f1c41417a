// Threshold gradient of JumpReLU as one tcgen05 GEMM per source layer with a reducing epilogue (sm_100a).
//
// The straight-through estimator of the reference gives every feature's threshold the gradient
//     d loss / d theta[f] = -(1 / bw) * sum_b  1[|x[b,f] - theta[f]| <= bw / 2] * x[b,f] * G[b,f]
// (clt/models/activations.py:196-220), where G = d loss / d activation is needed at every position inside the
// window, active or not.  With bw = 1 the window holds most positions, so G is a dense quantity:
//     G[b, f] = sum over targets t >= s of  gs[t][b, :] . W_dec[s -> t][f, :]   (+ the sparsity-penalty term)
// For source layer s this is a GEMM  [B, (L - s) d] x [(L - s) d, F]  whose K dimension runs over the target
// layers: A = the gradient seed of layers s..L-1 side by side, B = the packed decoder tensor of layer s,
// which is already K-major ([F, (L - s), d]).  The [B, F] product is never written: the epilogue multiplies it
// with window * x and reduces over the 128 token rows of the tile,
//     S1[s, f] += sum_b window * x * G_recon        S2[s, f] += sum_b window * x
// (S2 carries the penalty term, whose G is a per-feature constant outside the active entries).
// The autograd path computes the same through P dense GEMM pairs and a dense [B, F] backward per layer.
//
// Structure: a persistent pipeline (TMA ring, one MMA thread, two TMEM accumulators, eight epilogue warps), one CTA on a tile of 128 tokens or
// a pair of CTAs (cta_group::2) on 256.  One CTA loads 48 KB for 512 MMA cycles, more than L2 hands an SM, and stood still for operands; a CTA
// of a pair loads 32 KB (its own tokens, half of the decoder rows).  With one row per feature the epilogue comes as often as every 12 k-steps, which
// eight warps keep up with.  12 x 4096 x 4096 x 768: untied 1450 -> 1300 us (2.0 TFLOP, 1.57 PFLOP/s: the rate of the tensor cores
// under the power cap bounds it now), one row per feature 463 -> 360; 2 x 8192 x 16384 x 136 603 -> 427.
// No multicast loads.  Every mbarrier wait is bounded.
#include <climits>

#include "common.cuh"

namespace clt {

namespace tg {
constexpr int BM = 128;
constexpr int BN = 256;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr uint32_t A_BYTES = BM * BK * 2;
constexpr int EPI_WARPS = 8;  // two per 32 token rows, each with half of the columns (four: 463 us against 360 at 12 x 4096 x 4096, K = 768)
constexpr int EPI_THREADS = 32 * EPI_WARPS;
constexpr int NUM_THREADS = 64 + EPI_THREADS;
constexpr uint32_t TMEM_COLS = 512;
constexpr int kMaxLayers = 32;
template <bool PAIR>
struct Ring {
  static constexpr int STAGES = PAIR ? 6 : 4;
  static constexpr int B_ROWS = PAIR ? BN / 2 : BN;  // decoder rows that a CTA loads
  static constexpr uint32_t B_BYTES = B_ROWS * BK * 2;
  static constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr size_t SMEM_BYTES = size_t(STAGES) * STAGE_BYTES + 4096;  // barriers, thresholds and sums behind the ring
};
}  // namespace tg

struct ThetaGradMaps {
  CUtensorMap b[tg::kMaxLayers];  // decoder tensor of source layer s viewed as [F, (L - s) * d]
};

template <bool PAIR>
struct ThetaGradShared {
  uint64_t full[tg::Ring<PAIR>::STAGES];   // pairs: the leader's counts the bytes of both CTAs
  uint64_t empty[tg::Ring<PAIR>::STAGES];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  int epi_ok;
  alignas(16) float theta[tg::BN];
  float acc1[tg::BN];
  float acc2[tg::BN];
};

// v[0..31] of every lane -> lane j holds the sum over the warp's lanes of v[j].
__device__ __forceinline__ float warp_transpose_sum(float (&v)[32], int lane) {
#pragma unroll
  for (int off = 16, n = 32; off >= 1; off >>= 1, n >>= 1) {
    const bool upper = (lane & off) != 0;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const float send = upper ? v[i] : v[i + n / 2];
      const float keep = upper ? v[i + n / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, off);
    }
  }
  return v[0];
}

template <bool PAIR>
__global__ void __launch_bounds__(tg::NUM_THREADS, 1)
theta_grad_gemm_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_a_cum,
                       const __grid_constant__ ThetaGradMaps maps_b, int tying,
                       const t16* __restrict__ preact, long long ldx, long long layer_stride_x,
                       const float* __restrict__ theta, int stat_pitch, float half_bw, float* __restrict__ S1,
                       float* __restrict__ S2, int L, int M, int N, int d, int* __restrict__ status) {
  using namespace tg;
  using R = Ring<PAIR>;
  using Shared = ThetaGradShared<PAIR>;
  constexpr int STAGES = R::STAGES;
  static_assert(sizeof(Shared) <= 4096 && R::SMEM_BYTES <= 227 * 1024, "shared memory of one CTA");
  extern __shared__ __align__(1024) uint8_t tiles[];  // 128-byte-swizzled tiles need 1024-byte alignment
  Shared* sh = reinterpret_cast<Shared*>(tiles + size_t(STAGES) * R::STAGE_BYTES);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int cta_rank = PAIR ? int(cluster_ctarank()) : 0;
  const bool leader = cta_rank == 0;
  const int worker = PAIR ? int(blockIdx.x >> 1) : int(blockIdx.x), workers = PAIR ? int(gridDim.x >> 1) : int(gridDim.x);
  constexpr int kTileRows = PAIR ? 2 * BM : BM;
  const int tiles_m = (M + kTileRows - 1) / kTileRows;
  const int tiles_n = (N + BN - 1) / BN;
  const int kb_per_layer = (d + BK - 1) / BK;
  const int tiles_per_layer = tiles_m * tiles_n;
  const int total_tiles = L * tiles_per_layer;  // source layers in ascending order: longest K first
  volatile int* abort_flag = &sh->abort_flag;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&sh->full[s], 1);
      mbar_init(&sh->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sh->tmem_full[b], 1);
      mbar_init(&sh->tmem_empty[b], (PAIR ? 2 : 1) * EPI_WARPS);
    }
    sh->abort_flag = 0;
    fence_barrier_init();
  }
  for (int j = threadIdx.x; j < BN; j += NUM_THREADS) { sh->acc1[j] = 0.f; sh->acc2[j] = 0.f; }
  if (warp == 1) {
    if constexpr (PAIR) {
      tmem_alloc_pair(&sh->tmem_base, TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(&sh->tmem_base, TMEM_COLS);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();  // the peer's barriers exist before anything arrives on them
  tc_fence_after();
  const uint32_t tmem_base = sh->tmem_base;

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs of a pair)
    if (lane == 0) {
      tma_prefetch_desc(&map_a);
      uint32_t it = 0;
      bool ok = true;
      for (int t = worker; t < total_tiles && ok; t += workers) {
        const int src = t / tiles_per_layer;
        const int rem = t - src * tiles_per_layer;
        const int row = (rem % tiles_m) * kTileRows + cta_rank * BM;
        const int col = (rem / tiles_m) * BN + cta_rank * R::B_ROWS;
        // K runs over the target layers t >= src (untied: rows of the packed tensor of layer src; per_target: the
        // tensors of the layers t); per_source has one decoder row per feature, its A operand is the seed summed over t
        const int num_kb = (tying == 1 ? 1 : L - src) * kb_per_layer;
        int tl = 0, kk = 0;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&sh->empty[s], ph ^ 1, abort_flag)) { ok = false; break; }
          uint8_t* a_dst = tiles + size_t(s) * R::STAGE_BYTES;
          const CUtensorMap* a_map = tying == 1 ? &map_a_cum : &map_a;
          const CUtensorMap* b_map = tying == 2 ? &maps_b.b[src + tl] : &maps_b.b[src];
          const int a_layer = tying == 1 ? src : src + tl, b_k = tying == 0 ? tl * d + kk * BK : kk * BK;
          if constexpr (PAIR) {
            if (leader) mbar_expect_tx(&sh->full[s], 2 * R::STAGE_BYTES);
            const uint32_t full_leader = mapa_shared(smem_u32(&sh->full[s]), 0);
            tma_load_3d_pair(a_dst, a_map, full_leader, kk * BK, row, a_layer);
            tma_load_3d_pair(a_dst + A_BYTES, b_map, full_leader, b_k, col, 0);
          } else {
            mbar_expect_tx(&sh->full[s], R::STAGE_BYTES);
            tma_load_3d(a_dst, a_map, &sh->full[s], kk * BK, row, a_layer);
            tma_load_3d(a_dst + A_BYTES, b_map, &sh->full[s], b_k, col, 0);
          }
          if (++kk == kb_per_layer) { kk = 0; ++tl; }
        }
      }
      // (A CTA of a pair that gave up waits at the cluster barrier below until its partner, whose barriers count the copies, is done.)
      if (!ok && !PAIR) {
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
    // -------------------------------------------------------------- MMA issuer (leader CTA of a pair)
    if (lane == 0 && leader) {
      constexpr uint32_t idesc = umma_idesc_bf16(kTileRows, BN);
      const uint64_t a_desc0 = umma_desc_kmajor_sw128(smem_u32(tiles));
      const uint64_t b_desc0 = umma_desc_kmajor_sw128(smem_u32(tiles) + A_BYTES);
      int s = 0;
      uint32_t ph = 0, buf = 0, tph = 1;
      bool ok = true;
      for (int t = worker; t < total_tiles && ok; t += workers) {
        const int num_kb = (tying == 1 ? 1 : L - t / tiles_per_layer) * kb_per_layer;
        if (!mbar_wait(&sh->tmem_empty[buf], tph, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + buf * BN;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(&sh->full[s], ph, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint64_t a_desc = a_desc0 + uint64_t(s * int(R::STAGE_BYTES >> 4));
          const uint64_t b_desc = b_desc0 + uint64_t(s * int(R::STAGE_BYTES >> 4));
#pragma unroll
          for (int k = 0; k < BK / UMMA_K; ++k) {
            if constexpr (PAIR) umma_bf16_ss_pair(d_tmem, a_desc + uint64_t(k * 2), b_desc + uint64_t(k * 2), idesc, (kb | k) != 0);
            else umma_bf16_ss(d_tmem, a_desc + uint64_t(k * 2), b_desc + uint64_t(k * 2), idesc, (kb | k) != 0);
          }
          if constexpr (PAIR) tc_commit_pair(&sh->empty[s], 3);
          else tc_commit(&sh->empty[s]);
          if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (ok) {
          if constexpr (PAIR) tc_commit_pair(&sh->tmem_full[buf], 3);
          else tc_commit(&sh->tmem_full[buf]);
        }
        buf ^= 1;
        if (buf == 0) tph ^= 1;
      }
    }
  } else {
    // ---------------------------------------------------------------- reducing epilogue
    const int quarter = warp & 3;
    const int half = (warp - 2) >> 2;
    const int etid = (warp - 2) * 32 + lane;
    uint32_t local_tile = 0;
    bool ok = true;
    for (int t = worker; t < total_tiles && ok; t += workers, ++local_tile) {
      const int src = t / tiles_per_layer;
      const int rem = t - src * tiles_per_layer;
      const int mt = rem % tiles_m;
      const int nt = rem / tiles_m;
      const uint32_t buf = local_tile & 1;
      const uint32_t tph = (local_tile >> 1) & 1;
      named_barrier_sync(1, EPI_THREADS);  // accumulators of the previous tile were flushed and cleared
      for (int j = etid; j < BN; j += EPI_THREADS) {
        const int n = nt * BN + j;
        sh->theta[j] = n < N ? theta[1LL * src * stat_pitch + n] : INFINITY;
      }
      if (etid == 0) sh->epi_ok = mbar_wait(&sh->tmem_full[buf], tph, abort_flag) ? 1 : 0;
      named_barrier_sync(1, EPI_THREADS);
      if (!sh->epi_ok) { ok = false; break; }
      tc_fence_after();
      const int m = mt * kTileRows + cta_rank * BM + quarter * 32 + lane;
      const bool row_ok = m < M;
      const t16* xrow = preact + 1LL * src * layer_stride_x + 1LL * (row_ok ? m : 0) * ldx + 1LL * nt * BN;
      const uint32_t taddr = tmem_base + buf * BN + (uint32_t(quarter * 32) << 16);
#pragma unroll 1
      for (int c = half * (BN / 64); c < (half + 1) * (BN / 64); ++c) {
        uint32_t r[32];
        tmem_ld_32x32(taddr + c * 32, r);
        float wx[32];
        const int n0 = nt * BN + c * 32;
        if (row_ok && n0 + 32 <= N) {
          const uint4* xp = reinterpret_cast<const uint4*>(xrow + c * 32);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint4 u = __ldg(xp + q);
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) { wx[q * 8 + 2 * j] = t16_lo(w[j]); wx[q * 8 + 2 * j + 1] = t16_hi(w[j]); }
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) wx[j] = (row_ok && n0 + j < N) ? t16_to_float(xrow[c * 32 + j]) : INFINITY;
        }
        tmem_ld_wait();
        float p[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const bool in = fabsf(wx[j] - sh->theta[c * 32 + j]) <= half_bw;  // false for the INFINITY fillers
          wx[j] = in ? wx[j] : 0.f;
          p[j] = wx[j] * __uint_as_float(r[j]);
        }
        const float s1 = warp_transpose_sum(p, lane);
        const float s2 = warp_transpose_sum(wx, lane);
        if (s1 != 0.f) atomicAdd(&sh->acc1[c * 32 + lane], s1);
        if (s2 != 0.f) atomicAdd(&sh->acc2[c * 32 + lane], s2);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) mbar_arrive_cluster(mapa_shared(smem_u32(&sh->tmem_empty[buf]), 0));  // the leader's barrier
        else mbar_arrive(&sh->tmem_empty[buf]);
      }
      named_barrier_sync(1, EPI_THREADS);  // all warps added their rows
      for (int j = etid; j < BN; j += EPI_THREADS) {
        const int n = nt * BN + j;
        const float a1 = sh->acc1[j], a2 = sh->acc2[j];
        if (n < N) {
          if (a1 != 0.f) atomicAdd(&S1[1LL * src * stat_pitch + n], a1);
          if (a2 != 0.f) atomicAdd(&S2[1LL * src * stat_pitch + n], a2);
        }
        sh->acc1[j] = 0.f;
        sh->acc2[j] = 0.f;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();  // neither CTA retires (or frees TMEM) while the other may still use its memory
  if (warp == 1) {
    tc_fence_after();
    if constexpr (PAIR) tmem_dealloc_pair(tmem_base, TMEM_COLS);
    else tmem_dealloc(tmem_base, TMEM_COLS);
  }
  if (threadIdx.x == 0 && sh->abort_flag && status != nullptr) atomicCAS(status, STATUS_OK, STATUS_WAIT_TIMEOUT);
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFnT)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFnT tg_encode_fn() {
  static EncodeTiledFnT fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFnT>(p);
  }
  return fn;
}

static bool tg_make_map(CUtensorMap* map, const void* base, int layers, int rows, long long K, long long row_stride_elems,
                        long long layer_stride_elems, int box_rows) {
  EncodeTiledFnT enc = tg_encode_fn();
  if (enc == nullptr) return false;
  cuuint64_t dims[3] = {cuuint64_t(K), cuuint64_t(rows), cuuint64_t(layers)};
  cuuint64_t strides[2] = {cuuint64_t(row_stride_elems) * 2, cuuint64_t(layer_stride_elems) * 2};
  cuuint32_t box[3] = {cuuint32_t(tg::BK), cuuint32_t(box_rows), 1};
  cuuint32_t elem[3] = {1, 1, 1};
  return enc(map, (CLT_T16_IS_HALF ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16), 3, const_cast<void*>(base), dims, strides, box, elem,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace clt

struct CltThetaGradArgs {
  const void* gs;          // [L, B, d] bf16 gradient seed
  const void* w[32];       // untied decoder tensors, layer s: [F, L - s, d] bf16
  const void* preact;      // [L, B, ldx] bf16
  long long ldx, layer_stride_x;
  const float* theta;      // [L, stat_pitch]
  int stat_pitch;
  float bandwidth;
  float* S1;               // [L, stat_pitch], zeroed by the caller
  float* S2;
  int L, B, F, d;
  int* status;
  int tying;               // 0 untied ([F, L - s, d]), 1 per_source, 2 per_target (tensors [F, 1, d])
  const void* gs_cum;      // per_source: [L, B, d] suffix sums of gs over the layers
};

namespace clt {

// 1: the device cannot co-schedule clusters of two
template <bool PAIR>
static int tg_launch(const CltThetaGradArgs* a, int num_sms, cudaStream_t stream) {
  using R = tg::Ring<PAIR>;
  CUtensorMap map_a, map_a_cum;
  ThetaGradMaps maps;
  if (!tg_make_map(&map_a, a->gs, a->L, a->B, a->d, a->d, 1LL * a->B * a->d, tg::BM)) return -3;
  if (!tg_make_map(&map_a_cum, a->tying == 1 ? a->gs_cum : a->gs, a->L, a->B, a->d, a->d, 1LL * a->B * a->d, tg::BM)) return -3;
  for (int s = 0; s < tg::kMaxLayers; ++s) {
    const int src = s < a->L ? s : a->L - 1;
    const long long K = a->tying == 0 ? 1LL * (a->L - src) * a->d : a->d;
    if ((reinterpret_cast<uintptr_t>(a->w[src]) & 15) != 0) return -2;
    if (!tg_make_map(&maps.b[s], a->w[src], 1, a->F, K, K, 1LL * a->F * K, R::B_ROWS)) return -3;
  }
  constexpr int kTileRows = PAIR ? 2 * tg::BM : tg::BM;
  const long long tiles = 1LL * a->L * ((a->B + kTileRows - 1) / kTileRows) * ((a->F + tg::BN - 1) / tg::BN);
  if (tiles == 0) return 0;
  if (tiles > INT_MAX / 2) return -1;
  auto* kernel = theta_grad_gemm_kernel<PAIR>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(PAIR ? 2 * num_sms : num_sms));
  cfg.blockDim = dim3(tg::NUM_THREADS);
  cfg.dynamicSmemBytes = R::SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = PAIR ? 1 : 0;
  // co-resident clusters, probed once per device (the kernel's shared memory limit belongs to the device as well)
  constexpr int kDevices = 64;
  static int probed[kDevices] = {};  // count + 1, 0: not yet
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return -5;
  int n = dev < kDevices ? probed[dev] : 0;
  if (n == 0) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(R::SMEM_BYTES)) != cudaSuccess) return -4;
    n = num_sms;
    if (PAIR && cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
      n = 0;
      (void)cudaGetLastError();
    }
    ++n;
    if (dev < kDevices) probed[dev] = n;
  }
  const int workers = n - 1;
  if (workers <= 0) return 1;
  cfg.gridDim = dim3(unsigned((PAIR ? 2 : 1) * (tiles < workers ? tiles : workers)));
  if (cudaLaunchKernelEx(&cfg, kernel, map_a, map_a_cum, maps, a->tying, static_cast<const t16*>(a->preact), a->ldx, a->layer_stride_x, a->theta,
                         a->stat_pitch, 0.5f * a->bandwidth, a->S1, a->S2, a->L, a->B, a->F, a->d, a->status) != cudaSuccess) return -5;
  return 0;
}

}  // namespace clt

// Returns 0 on success, a negative value when the arguments cannot be handled (the caller raises).
extern "C" int CLT_FN(clt_theta_grad_gemm)(const CltThetaGradArgs* a, int num_sms, cudaStream_t stream) {
  using namespace clt;
  if (a->d % 8 != 0 || a->ldx % 8 != 0 || a->layer_stride_x % 8 != 0 || a->L > tg::kMaxLayers || a->L < 1) return -1;
  if (a->tying < 0 || a->tying > 2 || (a->tying == 1 && a->gs_cum == nullptr)) return -1;
  // a pair multiplies 256 token rows whether they exist or not: with 640 (five times 128) the sixth of it that is for nothing costs more than
  // pairs gain (7 % slower, where 1024 and 2000 rows are 7 to 25 % faster)
  const int halves = (a->B + tg::BM - 1) / tg::BM;
  if (halves % 2 == 0 || halves > 8) {
    const int r = tg_launch<true>(a, num_sms, stream);
    if (r <= 0) return r;
  }
  return tg_launch<false>(a, num_sms, stream);
}
