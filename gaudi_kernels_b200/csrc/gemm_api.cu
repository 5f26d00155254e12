// C entry points of the block-scaled GEMM: argument checks and schedule selection.
#include "common.cuh"

namespace bfp8 {
struct PushTarget {
  const void* recv[8];
  int world, rank, rows;
};
struct SmallPush {
  const void* recv[8];
  int world, rank, rows;
};
int launch_gemm_large(const uint8_t* a_codes, int64_t lda, const float* a_scales, int64_t ldsa,
                      const uint8_t* w_codes, int64_t ldw, const float* w_scales, const float* bias, void* out,
                      int out_dtype, int64_t ldo, int64_t m, int64_t n, int64_t k, uint32_t* status_dev,
                      long long wait_limit, int max_ctas, int band, int inter, const PushTarget* push, bool may_split,
                      cudaStream_t st);
int launch_gemm_pair(const uint8_t* a_codes, int64_t lda, const float* a_scales, int64_t ldsa,
                     const uint8_t* w_codes, int64_t ldw, const float* w_scales, const float* bias, void* out,
                     int out_dtype, int64_t ldo, int64_t m, int64_t n, int64_t k, uint32_t* status_dev,
                     long long wait_limit, int max_ctas, cudaStream_t st);
int launch_gemm_smallm(const uint8_t* a_codes, int64_t lda, const float* a_scales, int64_t ldsa,
                       const uint8_t* w_codes, int64_t ldw, const float* w_scales, const float* bias, void* out,
                       int out_dtype, int64_t ldo, int64_t m, int64_t n, int64_t k, void* workspace,
                       uint32_t* status_dev, long long wait_limit, int max_ctas, int inter, const SmallPush* push,
                       bool fresh_weight, cudaStream_t st);
int launch_gemm_channel(const uint8_t* a_codes, int64_t lda, const float* a_scales, const uint8_t* w_codes,
                        int64_t ldw, const float* w_scales, const float* bias, void* out, int out_dtype, int64_t ldo,
                        int64_t m, int64_t n, int64_t k, uint32_t* status_dev, long long wait_limit, int max_ctas,
                        cudaStream_t st);
int launch_gemm_smallm_token(const uint8_t* a_codes, int64_t lda, const float* a_scales, const uint8_t* w_codes,
                             int64_t ldw, const float* w_scales, const float* bias, void* out, int out_dtype,
                             int64_t ldo, int64_t m, int64_t n, int64_t k, uint32_t* status_dev, long long wait_limit,
                             cudaStream_t st);
size_t smallm_workspace_bytes(int64_t m, int64_t n, int max_ctas);
int set_weights_at_rest(int on);
bool smallm_supported(int64_t n);
int smallm_cluster_size(int64_t tiles, int64_t groups, int sms);
int large_k_split(int64_t m, int64_t n, int64_t groups, int sms);
int channel_k_split(int64_t m, int64_t n, int64_t groups, int sms);
}

using namespace bfp8;

namespace {
// About one second at B200 clocks: far beyond any legitimate wait, short enough that a broken
// launch returns with BFP8_STATUS_WAIT_TIMEOUT instead of hanging the device.
constexpr long long kDefaultWaitLimit = 2000000000LL;
constexpr int64_t kSmallMRows = 128;     // up to this many activation rows the weight-streaming schedule runs
// The same of the token/channel GEMM, one pass over W (K=4096, N=14336: 24.3 -> 14.8 us at 16 rows, 23.6 -> 19.7 at 64; its
// epilogue paces it beyond: 24.7 at 128 rows, where a pair of CTAs per large tile takes 20.4)
constexpr int64_t kTokenStreamRows = 64;
constexpr int kMaxCtas = 256;            // workspace is sized for this many CTAs, whatever the device has
}

extern "C" size_t bfp8_gemm_block128_workspace_bytes(int64_t m, int64_t n, int64_t k) {
  (void)k;
  if (m <= 0 || n <= 0) return 0;
  // Sized for the small-M schedule whenever it could be selected (automatically or by `schedule`).
  return (m <= kSmallMRows && smallm_supported(n)) ? smallm_workspace_bytes(m, n, kMaxCtas) : 0;
}

extern "C" int bfp8_gemm_block128_ex(const uint8_t* a_codes, int64_t lda, const float* a_scales, int64_t ldsa,
                                     const uint8_t* w_codes, int64_t ldw, const float* w_scales,
                                     const float* bias, void* out, int out_dtype, int64_t ldo,
                                     int64_t m, int64_t n, int64_t k,
                                     void* workspace, size_t workspace_bytes, uint32_t* status_dev, void* stream,
                                     int schedule, int max_ctas, int64_t wait_limit_cycles) {
  if (!a_codes || !a_scales || !w_codes || !w_scales || !out || !status_dev) return BFP8_ERR_NULL;
  if (m <= 0 || n <= 0 || k <= 0 || m > (1 << 30) || n > (1 << 30) || k > (1 << 30)) return BFP8_ERR_SHAPE;
  if (lda < k || ldw < k || ldo < n || ldsa < m) return BFP8_ERR_SHAPE;
  if (out_dtype != BFP8_OUT_F32 && out_dtype != BFP8_OUT_BF16) return BFP8_ERR_SHAPE;
  if (!aligned(a_codes, 16) || !aligned(w_codes, 16) || lda % 16 != 0 || ldw % 16 != 0) return BFP8_ERR_ALIGN;
  if (!aligned(a_scales, 4) || !aligned(w_scales, 4) || !aligned(status_dev, 4)) return BFP8_ERR_ALIGN;
  if (bias && !aligned(bias, 4)) return BFP8_ERR_ALIGN;
  if (out_dtype == BFP8_OUT_BF16 && (!aligned(out, 16) || ldo % 8 != 0)) return BFP8_ERR_ALIGN;
  if (out_dtype == BFP8_OUT_F32 && !aligned(out, 4)) return BFP8_ERR_ALIGN;
  const bool fresh_weight = (schedule & BFP8_SCHEDULE_FRESH_WEIGHT) != 0;
  schedule &= ~BFP8_SCHEDULE_FRESH_WEIGHT;
  if (schedule < 0 || schedule > 3 || (schedule == 2 && (m > kSmallMRows || !smallm_supported(n)))) return BFP8_ERR_SHAPE;
  const bool small = schedule == 2 || (schedule == 0 && m <= kSmallMRows && smallm_supported(n));
  const long long limit = wait_limit_cycles > 0 ? wait_limit_cycles : kDefaultWaitLimit;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (small) {
    const size_t need = bfp8_gemm_block128_workspace_bytes(m, n, k);
    if (!workspace || workspace_bytes < need) return BFP8_ERR_WORKSPACE;
    if (!aligned(workspace, 256)) return BFP8_ERR_ALIGN;
    if (sm_count() > kMaxCtas) return BFP8_ERR_UNSUPPORTED;
    return launch_gemm_smallm(a_codes, lda, a_scales, ldsa, w_codes, ldw, w_scales, bias, out, out_dtype, ldo,
                              m, n, k, workspace, status_dev, limit, max_ctas, /*inter=*/0, /*push=*/nullptr,
                              fresh_weight, st);
  }
  if (schedule == 3)
    return launch_gemm_pair(a_codes, lda, a_scales, ldsa, w_codes, ldw, w_scales, bias, out, out_dtype, ldo, m, n, k,
                            status_dev, limit, max_ctas, st);
  return launch_gemm_large(a_codes, lda, a_scales, ldsa, w_codes, ldw, w_scales, bias, out, out_dtype, ldo, m, n, k,
                           status_dev, limit, max_ctas, /*band=*/0, /*inter=*/0, /*push=*/nullptr, /*may_split=*/schedule == 0, st);
}

extern "C" int bfp8_gemm_block128(const uint8_t* a_codes, int64_t lda, const float* a_scales, int64_t ldsa,
                                  const uint8_t* w_codes, int64_t ldw, const float* w_scales,
                                  const float* bias, void* out, int out_dtype, int64_t ldo,
                                  int64_t m, int64_t n, int64_t k,
                                  void* workspace, size_t workspace_bytes, uint32_t* status_dev, void* stream) {
  return bfp8_gemm_block128_ex(a_codes, lda, a_scales, ldsa, w_codes, ldw, w_scales, bias, out, out_dtype, ldo,
                               m, n, k, workspace, workspace_bytes, status_dev, stream, 0, 0, 0);
}

extern "C" int bfp8_set_weights_at_rest(int on) { return set_weights_at_rest(on); }

extern "C" int bfp8_gemm_k_split(int64_t m, int64_t n, int64_t k, int token_channel, int sms) {
  if (m <= 0 || n <= 0 || k <= 0) return BFP8_ERR_SHAPE;
  if (sms <= 0) sms = sm_count();
  const int64_t groups = (k + 127) / 128;
  if (token_channel ? m <= kTokenStreamRows : m <= kSmallMRows && smallm_supported(n)) {
    const int cluster = smallm_cluster_size((n + 127) / 128, groups, sms);
    return cluster > 1 ? cluster : 1;
  }
  return token_channel ? channel_k_split(m, n, groups, sms) : large_k_split(m, n, groups, sms);
}

extern "C" int bfp8_gemm_token_channel(const uint8_t* a_codes, int64_t lda, const float* a_scales,
                                       const uint8_t* w_codes, int64_t ldw, const float* w_scales,
                                       const float* bias, void* out, int out_dtype, int64_t ldo,
                                       int64_t m, int64_t n, int64_t k, uint32_t* status_dev, void* stream) {
  if (!a_codes || !a_scales || !w_codes || !w_scales || !out || !status_dev) return BFP8_ERR_NULL;
  if (m <= 0 || n <= 0 || k <= 0 || m > (1 << 30) || n > (1 << 30) || k > (1 << 30)) return BFP8_ERR_SHAPE;
  if (lda < k || ldw < k || ldo < n) return BFP8_ERR_SHAPE;
  if (out_dtype != BFP8_OUT_F32 && out_dtype != BFP8_OUT_BF16) return BFP8_ERR_SHAPE;
  if (!aligned(a_codes, 16) || !aligned(w_codes, 16) || lda % 16 != 0 || ldw % 16 != 0) return BFP8_ERR_ALIGN;
  if (!aligned(a_scales, 4) || !aligned(w_scales, 4) || !aligned(status_dev, 4)) return BFP8_ERR_ALIGN;
  if (bias && !aligned(bias, 4)) return BFP8_ERR_ALIGN;
  if (out_dtype == BFP8_OUT_BF16 && (!aligned(out, 16) || ldo % 8 != 0)) return BFP8_ERR_ALIGN;
  if (out_dtype == BFP8_OUT_F32 && !aligned(out, 4)) return BFP8_ERR_ALIGN;
  if (m <= kTokenStreamRows)
    return launch_gemm_smallm_token(a_codes, lda, a_scales, w_codes, ldw, w_scales, bias, out, out_dtype, ldo, m, n, k,
                                    status_dev, kDefaultWaitLimit, static_cast<cudaStream_t>(stream));
  return launch_gemm_channel(a_codes, lda, a_scales, w_codes, ldw, w_scales, bias, out, out_dtype, ldo, m, n, k,
                             status_dev, kDefaultWaitLimit, 0, static_cast<cudaStream_t>(stream));
}

// ---- code rows of any length, given the 16-byte pitch that TMA needs --------------------------------------

namespace {
// Both operands of a GEMM in one launch: K that is not a multiple of 16 would otherwise take a fill and a strided copy
// for each (16.5 us of device time at M=777, K=1000, N=1003 before a GEMM of 11).  A thread writes one 16-byte vector of a
// destination row from the five aligned words that hold its source bytes, shifted into place; vectors at the ends of
// the source, and bytes at or beyond k, are formed byte by byte.
__global__ void __launch_bounds__(256)
repitch_kernel(const uint8_t* __restrict__ a, int64_t rows_a, uint8_t* __restrict__ dst_a, const uint8_t* __restrict__ w,
               int64_t rows_w, uint8_t* __restrict__ dst_w, int64_t k, uint32_t vecs) {
  // launched with programmatic stream serialization (see launch_overlapped)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int64_t vecs_a = rows_a * vecs, total = vecs_a + rows_w * vecs;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const bool first = i < vecs_a;
    const int64_t j = first ? i : i - vecs_a;
    const uint8_t* src = first ? a : w;
    const int64_t bytes = (first ? rows_a : rows_w) * k;
    const int64_t row = j / vecs, col = (j - row * vecs) * 16, from = row * k + col;
    const int valid = static_cast<int>(k - col < 16 ? k - col : 16);
    uint32_t v[4] = {0u, 0u, 0u, 0u};
    const uint32_t skew = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(src) + from) & 3u);
    if (from >= 4 && from + 20 <= bytes) {                       // the five words lie inside the source
      const uint32_t* p = reinterpret_cast<const uint32_t*>(src + from - skew);
      uint32_t x[5];
#pragma unroll
      for (int q = 0; q < 5; ++q) x[q] = __ldg(p + q);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        v[q] = __funnelshift_r(x[q], x[q + 1], skew * 8);
        const int keep = valid - 4 * q;                          // bytes of this word that belong to the row
        if (keep < 4) v[q] = keep <= 0 ? 0u : v[q] & ((1u << (8 * keep)) - 1u);
      }
    } else {
#pragma unroll
      for (int q = 0; q < 16; ++q)
        if (q < valid) v[q >> 2] |= static_cast<uint32_t>(src[from + q]) << (8 * (q & 3));
    }
    uint4* dst = reinterpret_cast<uint4*>(first ? dst_a : dst_w) + j;
    *dst = make_uint4(v[0], v[1], v[2], v[3]);
  }
}
}  // namespace

extern "C" int bfp8_repitch_codes(const uint8_t* a_codes, int64_t m, uint8_t* a_out, const uint8_t* w_codes, int64_t n,
                                  uint8_t* w_out, int64_t k, int64_t ld_out, void* stream) {
  if (m < 0 || n < 0 || m + n <= 0 || k <= 0 || m > (1 << 30) || n > (1 << 30) || k > (1 << 30)) return BFP8_ERR_SHAPE;
  if ((m > 0 && (!a_codes || !a_out)) || (n > 0 && (!w_codes || !w_out))) return BFP8_ERR_NULL;
  if (ld_out != (k + 15) / 16 * 16) return BFP8_ERR_SHAPE;
  if (!aligned(a_out, 16) || !aligned(w_out, 16)) return BFP8_ERR_ALIGN;
  const int64_t vecs = ld_out / 16, want = ((m + n) * vecs + 255) / 256, cap = static_cast<int64_t>(sm_count()) * 16;
  return launch_overlapped(repitch_kernel, dim3(static_cast<unsigned>(want < cap ? want : cap)), dim3(256), 0,
                           static_cast<cudaStream_t>(stream), a_codes, m, a_out, w_codes, n, w_out, k,
                           static_cast<uint32_t>(vecs));
}

// ---- gate/up GEMM with the SwiGLU step fused into its epilogue ---------------------------------------

namespace {
constexpr int kSwigluChunk = 64;

// Rows [0, inter) of src are the gate projection, rows [inter, 2 inter) the up projection.  Chunk c of 64
// outputs becomes dst rows [128 c, 128 c + 64) (gate) and [128 c + 64, 128 c + 128) (up).  16 bytes per thread.
__global__ void __launch_bounds__(256)
swiglu_interleave_kernel(const uint8_t* __restrict__ src, int64_t ld_src, uint8_t* __restrict__ dst, int64_t ld_dst,
                         int64_t inter, int64_t vecs_per_row) {
  const int64_t total = 2 * inter * vecs_per_row;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = i / vecs_per_row, v = i - r * vecs_per_row;          // destination row, 16-byte column
    const int64_t chunk = r / (2 * kSwigluChunk), in_chunk = r - chunk * 2 * kSwigluChunk;
    const int64_t s_row = in_chunk < kSwigluChunk ? chunk * kSwigluChunk + in_chunk
                                                  : inter + chunk * kSwigluChunk + (in_chunk - kSwigluChunk);
    const uint4 x = __ldcs(reinterpret_cast<const uint4*>(src + s_row * ld_src) + v);
    __stcs(reinterpret_cast<uint4*>(dst + r * ld_dst) + v, x);
  }
}
}  // namespace

extern "C" int bfp8_swiglu_interleave_weight(const uint8_t* w_codes, int64_t ld_src, uint8_t* out, int64_t ld_dst,
                                             int64_t inter, int64_t k, void* stream) {
  if (!w_codes || !out) return BFP8_ERR_NULL;
  if (inter <= 0 || k <= 0 || ld_src < k || ld_dst < k || inter > (1 << 29)) return BFP8_ERR_SHAPE;
  if (inter % 128 != 0) return BFP8_ERR_UNSUPPORTED;
  if (k % 16 != 0 || ld_src % 16 != 0 || ld_dst % 16 != 0 || !aligned(w_codes, 16) || !aligned(out, 16))
    return BFP8_ERR_ALIGN;
  if (w_codes == out) return BFP8_ERR_SHAPE;                       // not an in-place operation
  const int64_t vecs = k / 16, total = 2 * inter * vecs;
  const int64_t want = (total + 255) / 256;
  const int grid = static_cast<int>(want < static_cast<int64_t>(sm_count()) * 16 ? want : static_cast<int64_t>(sm_count()) * 16);
  swiglu_interleave_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(w_codes, ld_src, out, ld_dst, inter, vecs);
  BFP8_CUDA_TRY(cudaGetLastError());
  return BFP8_OK;
}

extern "C" int bfp8_gemm_block128_swiglu(const uint8_t* a_codes, int64_t lda, const float* a_scales, int64_t ldsa,
                                         const uint8_t* w_codes, int64_t ldw, const float* w_scales,
                                         const float* bias, void* out, int64_t ldo,
                                         int64_t m, int64_t inter, int64_t k,
                                         void* workspace, size_t workspace_bytes, uint32_t* status_dev, void* stream) {
  if (!a_codes || !a_scales || !w_codes || !w_scales || !out || !status_dev) return BFP8_ERR_NULL;
  if (m <= 0 || inter <= 0 || k <= 0 || m > (1 << 30) || inter > (1 << 29) || k > (1 << 30)) return BFP8_ERR_SHAPE;
  if (lda < k || ldw < k || ldo < inter || ldsa < m) return BFP8_ERR_SHAPE;
  if (inter % 128 != 0) return BFP8_ERR_UNSUPPORTED;               // gate / up boundary on a scale-block boundary
  if (!aligned(a_codes, 16) || !aligned(w_codes, 16) || lda % 16 != 0 || ldw % 16 != 0) return BFP8_ERR_ALIGN;
  if (!aligned(a_scales, 4) || !aligned(w_scales, 4) || !aligned(status_dev, 4)) return BFP8_ERR_ALIGN;
  if (bias && !aligned(bias, 4)) return BFP8_ERR_ALIGN;
  if (!aligned(out, 16) || ldo % 8 != 0) return BFP8_ERR_ALIGN;
  // decode bucket: the weight-streaming schedule, when the caller brought its scratch
  if (m <= kSmallMRows && smallm_supported(2 * inter) && workspace != nullptr) {
    if (workspace_bytes < bfp8_gemm_block128_workspace_bytes(m, 2 * inter, k)) return BFP8_ERR_WORKSPACE;
    if (!aligned(workspace, 256)) return BFP8_ERR_ALIGN;
    if (sm_count() > kMaxCtas) return BFP8_ERR_UNSUPPORTED;
    return launch_gemm_smallm(a_codes, lda, a_scales, ldsa, w_codes, ldw, w_scales, bias, out, BFP8_OUT_BF16, ldo, m,
                              2 * inter, k, workspace, status_dev, kDefaultWaitLimit, 0, static_cast<int>(inter),
                              /*push=*/nullptr, /*fresh_weight=*/false, static_cast<cudaStream_t>(stream));
  }
  return launch_gemm_large(a_codes, lda, a_scales, ldsa, w_codes, ldw, w_scales, bias, out, BFP8_OUT_BF16, ldo,
                           m, 2 * inter, k, status_dev, kDefaultWaitLimit, 0, /*band=*/0, static_cast<int>(inter),
                           /*push=*/nullptr, /*may_split=*/false, static_cast<cudaStream_t>(stream));
}

// ---- the SwiGLU step on its own, for results of the schedules that have no fused form (decode bucket) -------

namespace {
// One 16-byte vector (8 outputs) per thread and iteration; gate at column c, up at column c + inter of a row.
__global__ void __launch_bounds__(256)
silu_and_mul_kernel(const uint16_t* __restrict__ gate_up, int64_t ld_in, uint16_t* __restrict__ out, int64_t ld_out,
                    int64_t rows, int64_t inter, int vec_ok) {
  // launched with programmatic stream serialization (see launch_overlapped)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (vec_ok) {
    const int64_t vecs = inter >> 3, total = rows * vecs;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
      const int64_t r = i / vecs, v = i - r * vecs;
      const uint4 g = __ldcs(reinterpret_cast<const uint4*>(gate_up + r * ld_in) + v);
      const uint4 u = __ldcs(reinterpret_cast<const uint4*>(gate_up + r * ld_in + inter) + v);
      const uint32_t* gw = reinterpret_cast<const uint32_t*>(&g);
      const uint32_t* uw = reinterpret_cast<const uint32_t*>(&u);
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        o[j] = pack_bf16x2(silu_mul(bf16_lo_to_float(gw[j]), bf16_lo_to_float(uw[j])),
                           silu_mul(bf16_hi_to_float(gw[j]), bf16_hi_to_float(uw[j])));
      __stcs(reinterpret_cast<uint4*>(out + r * ld_out) + v, make_uint4(o[0], o[1], o[2], o[3]));
    }
  } else {
    const int64_t total = rows * inter;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
      const int64_t r = i / inter, c = i - r * inter;
      const float g = bf16_bits_to_float(gate_up[r * ld_in + c]), u = bf16_bits_to_float(gate_up[r * ld_in + inter + c]);
      out[r * ld_out + c] = static_cast<uint16_t>(float_to_bf16_bits(silu_mul(g, u)));
    }
  }
}
}  // namespace

extern "C" int bfp8_silu_and_mul_bf16(const uint16_t* gate_up, int64_t ld_in, uint16_t* out, int64_t ld_out,
                                      int64_t rows, int64_t inter, void* stream) {
  if (!gate_up || !out) return BFP8_ERR_NULL;
  if (rows <= 0 || inter <= 0 || ld_in < 2 * inter || ld_out < inter || rows > (1LL << 40) / inter) return BFP8_ERR_SHAPE;
  if (!aligned(gate_up, 2) || !aligned(out, 2)) return BFP8_ERR_ALIGN;
  const int vec = aligned(gate_up, 16) && aligned(out, 16) && inter % 8 == 0 && ld_in % 8 == 0 && ld_out % 8 == 0;
  const int64_t work = vec ? rows * (inter / 8) : rows * inter;
  const int64_t want = (work + 255) / 256, cap = static_cast<int64_t>(sm_count()) * 8;
  return launch_overlapped(silu_and_mul_kernel, dim3(static_cast<unsigned>(want < cap ? want : cap)), dim3(256), 0,
                           static_cast<cudaStream_t>(stream), gate_up, ld_in, out, ld_out, rows, inter, vec);
}

// ---- row-parallel GEMM whose epilogue scatters its tiles to the GPUs that reduce them -------------------

extern "C" int bfp8_gemm_block128_push(const uint8_t* a_codes, int64_t lda, const float* a_scales, int64_t ldsa,
                                       const uint8_t* w_codes, int64_t ldw, const float* w_scales,
                                       void* const* recv, int rank, int world_size,
                                       int64_t m, int64_t n, int64_t k,
                                       void* workspace, size_t workspace_bytes, uint32_t* status_dev, void* stream) {
  if (!a_codes || !a_scales || !w_codes || !w_scales || !recv || !status_dev) return BFP8_ERR_NULL;
  if (m <= 0 || n <= 0 || k <= 0 || m > (1 << 30) || n > (1 << 30) || k > (1 << 30)) return BFP8_ERR_SHAPE;
  if (world_size < 2 || world_size > 8 || rank < 0 || rank >= world_size) return BFP8_ERR_UNSUPPORTED;
  if (lda < k || ldw < k || ldsa < m) return BFP8_ERR_SHAPE;
  // decode bucket: the weight-streaming schedule stores each activation row to the GPU that owns it
  const bool small = m <= kSmallMRows && m % world_size == 0 && n % 64 == 0 && smallm_supported(n) && workspace != nullptr;
  if (!small && (m % (128 * world_size) != 0 || n % 64 != 0)) return BFP8_ERR_UNSUPPORTED;
  if (!aligned(a_codes, 16) || !aligned(w_codes, 16) || lda % 16 != 0 || ldw % 16 != 0) return BFP8_ERR_ALIGN;
  if (!aligned(a_scales, 4) || !aligned(w_scales, 4) || !aligned(status_dev, 4)) return BFP8_ERR_ALIGN;
  PushTarget t = {};
  for (int o = 0; o < world_size; ++o) {
    if (!recv[o]) return BFP8_ERR_NULL;
    if (!aligned(recv[o], 16)) return BFP8_ERR_ALIGN;
    t.recv[o] = recv[o];
  }
  t.world = world_size;
  t.rank = rank;
  t.rows = static_cast<int>(m / world_size);
  if (small) {
    if (workspace_bytes < bfp8_gemm_block128_workspace_bytes(m, n, k)) return BFP8_ERR_WORKSPACE;
    if (!aligned(workspace, 256)) return BFP8_ERR_ALIGN;
    if (sm_count() > kMaxCtas) return BFP8_ERR_UNSUPPORTED;
    SmallPush sp = {};
    for (int o = 0; o < world_size; ++o) sp.recv[o] = t.recv[o];
    sp.world = t.world;
    sp.rank = t.rank;
    sp.rows = t.rows;
    return launch_gemm_smallm(a_codes, lda, a_scales, ldsa, w_codes, ldw, w_scales, nullptr, const_cast<void*>(t.recv[rank]),
                              BFP8_OUT_BF16, n, m, n, k, workspace, status_dev, kDefaultWaitLimit, 0, /*inter=*/0, &sp,
                              /*fresh_weight=*/false, static_cast<cudaStream_t>(stream));
  }
  return launch_gemm_large(a_codes, lda, a_scales, ldsa, w_codes, ldw, w_scales, nullptr, const_cast<void*>(t.recv[rank]),
                           BFP8_OUT_BF16, n, m, n, k, status_dev, kDefaultWaitLimit, 0, /*band=*/0, /*inter=*/0, &t,
                           /*may_split=*/false, static_cast<cudaStream_t>(stream));
}
