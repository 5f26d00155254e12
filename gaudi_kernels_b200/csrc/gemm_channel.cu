// Token/channel-scaled E4M3 GEMM for sm_100a: one fp32 scale per activation row and one per output
// channel, so the whole K range accumulates in TMEM and the scales are applied once per tile.
//
//   out[i, j] = (sum_k a(i, k) * w(j, k)) * a_scale[i] * w_scale[j] + bias[j]
//
// This is the per-token / per-channel FP8 variant of the reference (gk_fp8_token_quant_bf16_v1 feeding an
// MME GEMM, finished by gk_fp8_channel_finish_bf16_v1: csrc/tpc/block_fp8_framework/activation_token.c:4-26,
// channel_finish.c:2-18).  Same tile machinery as the block-scaled kernel - TMA (SWIZZLE_128B) -> shared
// memory -> tcgen05.mma kind::f8f6f4 -> TMEM - but without the per-K-block read-back: a 128 x 256 tile's
// MMAs accumulate over all of K into one of two 256-column TMEM buffers, and the epilogue warps drain the
// other buffer (scale, bias, bf16, TMA store) while the next tile's MMAs run.
//
// Large calls run as CTA pairs on 256 x 256 tiles, calls with few tiles as clusters that split K (see the kernel).
//
// Warp roles (384 threads): warps 0-7 epilogue (two warpgroups of 128 columns each), warp 8 TMA producer,
// warp 9 TMEM owner + MMA issuer, warps 10-11 idle (setmaxnreg hands their registers to the epilogue).
// Persistent, one CTA per SM; every barrier wait is bounded and raises BFP8_STATUS_WAIT_TIMEOUT.
#include <cuda.h>

#include "common.cuh"
#include "ptx.cuh"
#include "split_exchange.cuh"

namespace bfp8 {

int split_cluster_size(int64_t tiles, int64_t groups, int sms);

namespace {

constexpr int BM = 128;
constexpr int BN = 256;
constexpr int BK = 128;
constexpr int kEpiWarps = 8;
constexpr int kThreads = (kEpiWarps + 4) * 32;
constexpr int kTmemCols = 512;
// The forms of the kernel: one CTA per tile; a cluster of CTAs that share the K range of a tile; two CTAs that share the
// MMAs of a 256 x 256 tile.
enum Form { kOne, kSplitK, kPair };

template <Form F>
struct Cfg {
  static constexpr int kABytes = BM * BK;                            // this CTA's A rows
  static constexpr int kBBytes = (F == kPair ? BN / 2 : BN) * BK;    // W rows, or half of the pair's
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kStages = F == kPair ? 6 : 4;                 // 192 KB either way
  static constexpr int kTileRows = F == kPair ? 2 * BM : BM;
};
constexpr int kOutWarpBytes = 32 * 64 * 2;
constexpr int kOutStageBytes = kEpiWarps * kOutWarpBytes;

struct SmemTail {
  uint64_t full[6];                // of the pair's first CTA in the pair form
  uint64_t empty[6];
  uint64_t tmem_full[2];
  uint64_t tmem_empty[2];
  uint32_t tmem_base;
  uint32_t abort_flag;
};

constexpr int kSmemBytes = 1024 + Cfg<kOne>::kStages * Cfg<kOne>::kStageBytes + kOutStageBytes + sizeof(SmemTail);
static_assert(Cfg<kPair>::kStages * Cfg<kPair>::kStageBytes == Cfg<kOne>::kStages * Cfg<kOne>::kStageBytes, "one layout");

struct Params {
  const float* a_scales;   // [M]
  const float* w_scales;   // [N]
  const float* bias;       // [N] or null
  void* out;
  int64_t ldo;
  int m, n, groups;
  int tiles_m, tiles_n;
  int split;               // CTAs (one cluster) that share a tile's K range in the split form, else 1
  long long wait_limit;
  uint32_t* status;
};

__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int& tm, int& tn) {
  constexpr int kBand = 8;
  const int per_band = kBand * tiles_n;
  const int band = t / per_band;
  const int first = band * kBand;
  const int rows = min(kBand, tiles_m - first);
  const int r = t - band * per_band;
  tm = first + r % rows;
  tn = r / rows;
}

// kSplit: few tiles and a long K range, so p.split CTAs form a cluster, each accumulates an equal slice of the tile's K
// blocks and the partial tiles are exchanged and added as split_exchange.cuh describes.  One tile per cluster.
//
// kPair: two CTAs of a cluster on one 256 x 256 tile.  What bounds the one-CTA form is the feed of its shared memory: 48 KB
// per K block arrive at about 62 B/clk per SM (785 cycles per K block, the MMAs take 512).  A cta_group::2 MMA reads its
// own A rows and half of the W rows from each CTA, 32 KB per CTA and K block.  The first CTA issues the MMAs, its `full`
// barriers collect the TMA bytes of both CTAs and its `tmem_empty` barriers the epilogue warps of both; the commits are
// multicast to both CTAs' `empty` and `tmem_full` barriers.
template <bool kOutBf16, Form F>
__global__ void __launch_bounds__(kThreads, 1)
gemm_channel_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w,
                    const __grid_constant__ CUtensorMap tmap_out, const Params p) {
  using C = Cfg<F>;
  constexpr bool kSplit = F == kSplitK;
  constexpr int kStages = C::kStages, kStageBytes = C::kStageBytes, kABytes = C::kABytes, kTileRows = C::kTileRows;
  extern __shared__ uint8_t smem_raw[];
  const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
  uint8_t* out_stage = smem + kStages * kStageBytes;
  SmemTail* tail = reinterpret_cast<SmemTail*>(out_stage + kOutStageBytes);
  volatile uint32_t* abort_flag = &tail->abort_flag;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int num_tiles = p.tiles_m * p.tiles_n;
  // this CTA's first tile, the distance to its next, and its K blocks [g_first, g_first + G) of each
  const int cs = kSplit ? p.split : F == kPair ? 2 : 1;
  const int crank = F == kOne ? 0 : static_cast<int>(blockIdx.x % cs);
  const int tile0 = F == kOne ? static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x / cs);
  const int tile_step = kSplit ? num_tiles : static_cast<int>(F == kPair ? gridDim.x >> 1 : gridDim.x);
  const int g_first = kSplit ? static_cast<int>(static_cast<long long>(crank) * p.groups / cs) : 0;
  const int G = kSplit ? static_cast<int>(static_cast<long long>(crank + 1) * p.groups / cs) - g_first : p.groups;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      ptx::mbar_init(ptx::smem_u32(&tail->full[s]), 1);
      ptx::mbar_init(ptx::smem_u32(&tail->empty[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(ptx::smem_u32(&tail->tmem_full[b]), 1);
      ptx::mbar_init(ptx::smem_u32(&tail->tmem_empty[b]), (F == kPair ? 2 : 1) * kEpiWarps);
    }
    tail->abort_flag = 0;
    ptx::fence_mbar_init();
  }
  if (warp == kEpiWarps + 1) {
    if (F == kPair) {
      ptx::tmem_alloc_pair(ptx::smem_u32(&tail->tmem_base), kTmemCols);
      ptx::tmem_relinquish_pair();
    } else {
      ptx::tmem_alloc(ptx::smem_u32(&tail->tmem_base), kTmemCols);
      ptx::tmem_relinquish();
    }
  }
  if (warp == kEpiWarps && lane == 0) {
    ptx::prefetch_tensormap(&tmap_a);
    ptx::prefetch_tensormap(&tmap_w);
    if (kOutBf16) ptx::prefetch_tensormap(&tmap_out);
  }
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (F == kPair) ptx::cluster_sync_all();          // both CTAs' barriers exist before any remote arrival
  ptx::tc_fence_after_sync();
  const uint32_t tmem_base = tail->tmem_base;
  // the set-up above touches no global memory and may overlap the previous kernel of the stream.  Unlike in the block-scaled
  // kernel this costs calls of several waves nothing: with its quantizer, M=4096, K=4096, N=14336 191.4 us against 192.3 in
  // ordinary launches, M=8192 and K=14336 equal within the spread of the runs
  ptx::griddep_launch_dependents();
  ptx::griddep_wait();

  if (warp >= kEpiWarps) {
    ptx::setmaxnreg_dec<40>();
    if (warp == kEpiWarps) {
      // ------------------------------------------------------------------ TMA producer
      if (lane == 0) {
        uint32_t stage = 0, phase = 0;
        bool ok = true;
        for (int t = tile0; t < num_tiles && ok; t += tile_step) {
          int tm, tn;
          tile_coords(t, p.tiles_m, p.tiles_n, tm, tn);
          for (int g = 0; g < G; ++g) {
            ok = ptx::mbar_wait(ptx::smem_u32(&tail->empty[stage]), phase ^ 1u, abort_flag, p.wait_limit);
            if (!ok) break;
            const uint32_t full = ptx::smem_u32(&tail->full[stage]);
            const uint32_t a_dst = smem_base + stage * kStageBytes;
            if (F == kPair) {
              const uint32_t full0 = ptx::cluster_map(full, 0);
              if (crank == 0) ptx::mbar_arrive_expect_tx(full, 2 * kStageBytes);
              ptx::tma_load_2d_pair(a_dst, &tmap_a, full0, g * BK, tm * kTileRows + crank * BM);
              ptx::tma_load_2d_pair(a_dst + kABytes, &tmap_w, full0, g * BK, tn * BN + crank * (BN / 2));
            } else {
              ptx::mbar_arrive_expect_tx(full, kStageBytes);
              ptx::tma_load_2d(a_dst, &tmap_a, full, (g_first + g) * BK, tm * BM);
              ptx::tma_load_2d(a_dst + kABytes, &tmap_w, full, (g_first + g) * BK, tn * BN);
            }
            if (++stage == kStages) { stage = 0; phase ^= 1u; }
          }
        }
      }
    } else if (warp == kEpiWarps + 1) {
      // ------------------------------------------------------------------ MMA issuer (of the pair's first CTA)
      if (lane == 0 && (F != kPair || crank == 0)) {
        constexpr uint32_t idesc = ptx::umma_idesc_e4m3(kTileRows, BN);
        uint32_t stage = 0, phase = 0, it = 0;
        bool ok = true;
        for (int t = tile0; t < num_tiles && ok; t += tile_step, ++it) {
          const uint32_t buf = it & 1u, acc_phase = (it >> 1) & 1u;
          ok = ptx::mbar_wait(ptx::smem_u32(&tail->tmem_empty[buf]), acc_phase ^ 1u, abort_flag, p.wait_limit);
          if (!ok) break;
          ptx::tc_fence_after_sync();
          const uint32_t d = tmem_base + buf * BN;
          for (int g = 0; g < G; ++g) {
            ok = ptx::mbar_wait(ptx::smem_u32(&tail->full[stage]), phase, abort_flag, p.wait_limit);
            if (!ok) break;
            ptx::tc_fence_after_sync();
            const uint32_t a_addr = smem_base + stage * kStageBytes;
            const uint64_t a_desc = ptx::umma_desc_k128(a_addr);
            const uint64_t b_desc = ptx::umma_desc_k128(a_addr + kABytes);
#pragma unroll
            for (int k4 = 0; k4 < BK / 32; ++k4) {
              if (F == kPair) ptx::umma_f8_pair(d, a_desc + 2u * k4, b_desc + 2u * k4, idesc, (g | k4) != 0);
              else ptx::umma_f8(d, a_desc + 2u * k4, b_desc + 2u * k4, idesc, (g | k4) != 0);
            }
            if (F == kPair) ptx::umma_commit_pair(ptx::smem_u32(&tail->empty[stage]));
            else ptx::umma_commit(ptx::smem_u32(&tail->empty[stage]));
            if (++stage == kStages) { stage = 0; phase ^= 1u; }
          }
          if (!ok) break;
          if (F == kPair) ptx::umma_commit_pair(ptx::smem_u32(&tail->tmem_full[buf]));
          else ptx::umma_commit(ptx::smem_u32(&tail->tmem_full[buf]));
        }
      }
    }
  } else {
    ptx::setmaxnreg_inc<232>();
    // ------------------------------------------------------------------ epilogue: once per tile
    const int wg = warp >> 2;
    const int quad = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    uint8_t* my_stage = out_stage + warp * kOutWarpBytes;
    uint32_t it = 0;
    bool ok = true;
    for (int t = tile0; t < num_tiles && ok; t += tile_step, ++it) {
      int tm, tn;
      tile_coords(t, p.tiles_m, p.tiles_n, tm, tn);
      const int row0 = tm * kTileRows + (F == kPair ? crank * BM : 0) + quad * 32;
      const int row = row0 + lane;
      const int col0 = tn * BN + wg * 128;
      const bool row_ok = row < p.m;
      const float act = row_ok ? __ldg(p.a_scales + row) : 0.0f;
      const uint32_t buf = it & 1u, acc_phase = (it >> 1) & 1u;
      // uniform across the warp: warp-collective TMEM loads follow
      ok = __all_sync(0xffffffffu, ptx::mbar_wait(ptx::smem_u32(&tail->tmem_full[buf]), acc_phase, abort_flag, p.wait_limit));
      if (!ok) break;
      ptx::tc_fence_after_sync();
      const uint32_t taddr = tmem_base + lane_addr + buf * BN + wg * 128;
      if (kSplit) {
        ptx::cluster_sync_all();                       // every CTA's pipeline buffers are idle
        const int trow = quad * 32 + lane;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t r[32];
          ptx::tmem_ld32(taddr + c * 32, r);
          ptx::tmem_wait_ld32(r);
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[8 * u + j]);
            split::send(smem_base, cs, crank, wg * 16 + c * 4 + u, trow, v);
          }
        }
        ptx::cluster_sync_all();                       // every partial sum has arrived
        split::finish<kOutBf16>(smem, cs, crank, threadIdx.x, kEpiWarps * 32, p.out, p.ldo, tm * BM, tn * BN, p.m, p.n,
                                [&](int r, int c, float x) {
                                  return fmaf(x * __ldg(p.a_scales + r), __ldg(p.w_scales + c),
                                              p.bias != nullptr ? __ldg(p.bias + c) : 0.0f);
                                });
        continue;
      }
      uint32_t ra[32], rb[32];
      ptx::tmem_ld32(taddr, ra);
      ptx::tmem_ld32(taddr + 32, rb);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        // chunk c = columns col0 + 32 c .. + 31, held in ra (even c) or rb (odd c)
        uint32_t (&r)[32] = (c & 1) ? rb : ra;
        if ((c & 1) == 0) {
          ptx::tmem_wait_ld32(ra);
          ptx::tmem_regs_ready32(rb);
        }
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const int col = col0 + c * 32 + j;
          const float ws = col < p.n ? __ldg(p.w_scales + col) : 0.0f;
          const float b = (p.bias != nullptr && col < p.n) ? __ldg(p.bias + col) : 0.0f;
          // (partial * act_scale) * w_scale + bias, the order of channel_finish.c:12-14
          v[j] = fmaf(__uint_as_float(r[j]) * act, ws, b);
        }
        if (c == 1) {
          // second half of the buffer: fetch it into the registers just consumed
          ptx::tmem_ld32(taddr + 64, ra);
          ptx::tmem_ld32(taddr + 96, rb);
        }
        if (c == 3) {
          // every column of the buffer has been read: release it to the MMA warp
          ptx::tc_fence_before_sync();
          __syncwarp();
          const uint32_t bar = ptx::smem_u32(&tail->tmem_empty[buf]);
          if (F == kPair) ptx::mbar_arrive_remote_lane0(ptx::cluster_map(bar, 0), lane);
          else ptx::mbar_arrive_lane0(bar, lane);
        }
        if (kOutBf16) {
          const int box = c >> 1;                        // one TMA box = 64 columns = two chunks
          const bool ragged = (p.n & 7) != 0 && col0 + box * 64 + 64 > p.n;
          if (ragged) {
            if (row_ok) {
              uint16_t* o = reinterpret_cast<uint16_t*>(p.out) + static_cast<int64_t>(row) * p.ldo + col0 + c * 32;
#pragma unroll
              for (int j = 0; j < 32; ++j)
                if (col0 + c * 32 + j < p.n) o[j] = static_cast<uint16_t>(float_to_bf16_bits(v[j]));
            }
          } else {
            if ((c & 1) == 0) {
              // the previous TMA store must have finished reading this warp's staging buffer
              if (lane == 0) ptx::tma_store_wait_read_all();
              __syncwarp();
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              uint4 q;
              q.x = pack_bf16x2(v[8 * j + 0], v[8 * j + 1]);
              q.y = pack_bf16x2(v[8 * j + 2], v[8 * j + 3]);
              q.z = pack_bf16x2(v[8 * j + 4], v[8 * j + 5]);
              q.w = pack_bf16x2(v[8 * j + 6], v[8 * j + 7]);
              const int chunk = (c & 1) * 4 + j;           // 16-byte chunk inside the 128-byte row
              *reinterpret_cast<uint4*>(my_stage + lane * 128 + ((chunk ^ (lane & 7)) << 4)) = q;
            }
            if (c & 1) {
              ptx::fence_proxy_async_smem();
              __syncwarp();
              if (lane == 0) {
                if (row0 < p.m && col0 + box * 64 < p.n)
                  ptx::tma_store_2d(&tmap_out, ptx::smem_u32(my_stage), col0 + box * 64, row0);
                ptx::tma_store_commit();
              }
            }
          }
        } else {
          store_box_f32(reinterpret_cast<float*>(my_stage), lane, v,
                        reinterpret_cast<float*>(p.out) + static_cast<int64_t>(row0) * p.ldo + col0 + c * 32, p.ldo,
                        p.m - row0, p.n - (col0 + c * 32));
        }
      }
    }
    if (kSplit && !ok) {
      // gave up inside the slice: keep the two appointments of the exchange
      ptx::cluster_sync_all();
      ptx::cluster_sync_all();
    }
    if (kOutBf16 && !kSplit && lane == 0) ptx::tma_store_wait_all();
  }
  if (kSplit && warp >= kEpiWarps) {
    // the other roles take part in the two cluster barriers of the exchange
    __syncwarp();
    ptx::cluster_sync_all();
    ptx::cluster_sync_all();
  }

  // ------------------------------------------------------------------ teardown
  ptx::tc_fence_before_sync();
  __syncthreads();
  if (F == kPair) ptx::cluster_sync_all();          // the peer may still use this CTA's shared memory or barriers
  ptx::tc_fence_after_sync();
  ptx::idle_after_abort(abort_flag);
  if (warp == kEpiWarps + 1) {
    if (F == kPair) ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
    else ptx::tmem_dealloc(tmem_base, kTmemCols);
  }
  if (threadIdx.x == 0 && tail->abort_flag != 0) atomicOr(p.status, BFP8_STATUS_WAIT_TIMEOUT);
}

}  // namespace

namespace {
// Whether the pair form is the faster one: a wave of pairs takes 0.92 of a wave of single CTAs (M=4096, K=4096, N=14336:
// 181 against 196 us, both 13 waves; M=8192, K=14336, N=4096: 326 / 355), but its tiles are twice as tall, so an odd number
// of 128-row tiles, or few of them, can cost it a wave.  Where the K range is worth splitting the one-CTA form has that -
// except that up to 128 rows a pair, half of it on padding rows, also gives a tile two CTAs to stream W, without the
// exchange (M=128, K=4096, N=14336: 20.4 us; split in two 23.7, one CTA 22.7; with N=8192, K=8192 four slices 24.1, pairs 28.0).
bool pair_is_faster(int64_t m, int64_t cols, int64_t groups, int sms) {
  const int64_t one = (m + BM - 1) / BM * cols, two = (m + 2 * BM - 1) / (2 * BM) * cols;
  const int64_t one_waves = (one + sms - 1) / sms, two_waves = (two + sms / 2 - 1) / (sms / 2);
  return split_cluster_size(one, groups, sms) <= (m <= BM ? 2 : 1) && two_waves * 92 <= one_waves * 100;
}
}  // namespace

// CTAs that share a tile's K range (1 in the pair form, whose CTAs share the MMAs).
int channel_k_split(int64_t m, int64_t n, int64_t groups, int sms) {
  const int64_t cols = (n + BN - 1) / BN;
  return pair_is_faster(m, cols, groups, sms) ? 1 : split_cluster_size((m + BM - 1) / BM * cols, groups, sms);
}

int launch_gemm_channel(const uint8_t* a_codes, int64_t lda, const float* a_scales, const uint8_t* w_codes,
                        int64_t ldw, const float* w_scales, const float* bias, void* out, int out_dtype, int64_t ldo,
                        int64_t m, int64_t n, int64_t k, uint32_t* status_dev, long long wait_limit, int max_ctas,
                        cudaStream_t st) {
  alignas(64) CUtensorMap tmap_a, tmap_w, tmap_out;
  int rc = make_tensor_map_2d(&tmap_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, a_codes, k, m, lda, BK, BM);
  if (rc != BFP8_OK) return rc;
  const int sms = sm_count();
  const bool pair = max_ctas <= 0 && pair_is_faster(m, (n + BN - 1) / BN, (k + BK - 1) / BK, sms);
  const int tile_rows = pair ? Cfg<kPair>::kTileRows : BM;
  rc = make_tensor_map_2d(&tmap_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, w_codes, k, n, ldw, BK, pair ? BN / 2 : BN);
  if (rc != BFP8_OK) return rc;
  const bool bf16 = out_dtype == BFP8_OUT_BF16;
  if (bf16) {
    rc = make_tensor_map_2d(&tmap_out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, out, n, m, ldo * 2, 64, 32);
    if (rc != BFP8_OK) return rc;
  } else {
    tmap_out = tmap_a;   // unused on the fp32 path
  }
  Params p;
  p.a_scales = a_scales;
  p.w_scales = w_scales;
  p.bias = bias;
  p.out = out;
  p.ldo = ldo;
  p.m = static_cast<int>(m);
  p.n = static_cast<int>(n);
  p.groups = static_cast<int>((k + BK - 1) / BK);
  p.tiles_m = static_cast<int>((m + tile_rows - 1) / tile_rows);
  p.tiles_n = static_cast<int>((n + BN - 1) / BN);
  p.wait_limit = wait_limit;
  p.status = status_dev;
  const int tiles = p.tiles_m * p.tiles_n;
  int grid = pair ? sms / 2 : sms;                       // pairs, or CTAs
  if (max_ctas > 0 && max_ctas < grid) grid = max_ctas;
  if (tiles < grid) grid = tiles;
  cudaLaunchAttribute attr[2];
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  p.split = 1;
  if (pair) {
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
    cfg.gridDim = dim3(static_cast<unsigned>(grid * 2), 1, 1);
    auto kern = bf16 ? gemm_channel_kernel<true, kPair> : gemm_channel_kernel<false, kPair>;
    static DeviceFlags done[2];
    rc = ensure_smem_limit(kern, kSmemBytes, done[bf16 ? 1 : 0]);
    if (rc != BFP8_OK) return rc;
    BFP8_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tmap_a, tmap_w, tmap_out, p));
    return BFP8_OK;
  }
  const int want = max_ctas <= 0 ? split_cluster_size(tiles, p.groups, sms) : 1;
  if (want > 1) {
    auto kern = bf16 ? gemm_channel_kernel<true, kSplitK> : gemm_channel_kernel<false, kSplitK>;
    static DeviceFlags done[2];
    rc = ensure_smem_limit(kern, kSmemBytes, done[bf16 ? 1 : 0]);
    if (rc != BFP8_OK) return rc;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.numAttrs = 2;
    static ClusterCaps caps[2];
    for (int cs = want; cs > 1; --cs) {                // the largest cluster of which the device holds all `tiles` at once
      attr[1].val.clusterDim.x = static_cast<unsigned>(cs);
      cfg.gridDim = dim3(static_cast<unsigned>(tiles * cs), 1, 1);
      if (max_active_clusters(kern, cfg, cs, caps[bf16 ? 1 : 0]) < tiles) continue;
      p.split = cs;
      BFP8_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tmap_a, tmap_w, tmap_out, p));
      return BFP8_OK;
    }
    cfg.numAttrs = 1;
  }
  auto kern = bf16 ? gemm_channel_kernel<true, kOne> : gemm_channel_kernel<false, kOne>;
  static DeviceFlags done[2];
  rc = ensure_smem_limit(kern, kSmemBytes, done[bf16 ? 1 : 0]);
  if (rc != BFP8_OK) return rc;
  cfg.gridDim = dim3(static_cast<unsigned>(grid), 1, 1);
  BFP8_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tmap_a, tmap_w, tmap_out, p));
  return BFP8_OK;
}

}  // namespace bfp8
