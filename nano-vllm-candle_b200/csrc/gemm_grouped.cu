// Grouped product of the routed experts: C[r] = act(A[r] . W[group of r]^T), bf16 x bf16 -> fp32 in tensor memory.  The rows of A are sorted by
// group and every group starts at a multiple of 128 rows, so a tile of 128 rows has one group (tile_group, made on the device: the host knows only
// an upper bound of the rows); tiles behind the last group have a negative one and are passed over.
//
// A persistent grid, one CTA per SM, walks the 128 x BN tiles, the column tiles of a row tile first (they share its rows, and neighbouring row
// tiles of a group its weights, through L2):
//   warp 0     TMA producer: 128 x 64 boxes of A and BN x 64 boxes of W, a ring of four (BN 256), six (128) or four (64, two k-blocks
//              each) stages that runs on into the next tile
//   warp 1     tcgen05.mma M 128, N BN, K 16; two accumulators in tensor memory, so that a tile's epilogue runs under the next one's main loop
//   warps 2-5  epilogue: tcgen05.ld, activation, rows through a staging buffer (RowStage)
// What bounds it: a k-block brings (128 + BN) x 128 bytes into shared memory for 2 BN cycles of the tensor pipe, 96 and 128 bytes per cycle where an
// SM takes about 75; with a few rows per group (decode) the weights' way from memory.  One CTA per tile had the start, the first loads and the
// epilogue of every tile exposed: 4 000 tokens, 16 experts,
// top 2: 1 024 -> 3 072 79 us, 1 536 -> 1 024 38 us, where this takes 49 and 30; 64 tokens 35 and 16 us, where this takes 25 and 16.
#include "common.cuh"
#include "ptx.cuh"
#include "internal.h"
#include "gemm_epilogue.cuh"

#include <algorithm>
#include <cmath>

namespace {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int kThreads = 192;

template <int BN>
struct GroupedCfg {
  static constexpr int kBytesA = BM * BK * 2, kBytesB = BN * BK * 2;
  static constexpr int KPS = BN == 64 ? 2 : 1;                               // k-blocks per stage: a round trip over the barriers is long beside a narrow one
  static constexpr int kStageBytes = KPS * (kBytesA + kBytesB);
  static constexpr int kStages = BN == 128 ? 6 : 4;                          // 192 KB
  static constexpr int kOffStaging = kStages * kStageBytes;                  // 4 KB per epilogue warp
  static constexpr int kOffBar = kOffStaging + 4 * 4096;
  static constexpr int kNumBars = 2 * kStages + 4;                           // full, empty, accumulator full x 2, accumulator empty x 2
  static constexpr int kSmemBytes = kOffBar + kNumBars * 8 + 16 + 1024;      // 1024: alignment by hand
  static constexpr int kTmemCols = 2 * BN;
};

template <int BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_grouped_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, void* __restrict__ C, int ldc, int out_f32, int M, int N,
                    int num_kb, int num_tiles, int n_tiles, int epi, int zero, const int32_t* tile_group) {
  using cfg = GroupedCfg<BN>;
  pdl_trigger();
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bar0 = base + cfg::kOffBar;
  auto full_bar = [&](int s) { return bar0 + 8u * s; };
  auto empty_bar = [&](int s) { return bar0 + 8u * (cfg::kStages + s); };
  auto acc_full = [&](int a) { return bar0 + 8u * (2 * cfg::kStages + a); };
  auto acc_empty = [&](int a) { return bar0 + 8u * (2 * cfg::kStages + 2 + a); };
  const uint32_t tmem_slot = bar0 + 8u * cfg::kNumBars;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 0) {
    if (lane == 0) {
      ptx::tma_prefetch_desc(&tma_a);
      ptx::tma_prefetch_desc(&tma_b);
      for (int s = 0; s < cfg::kStages; ++s) {
        ptx::mbar_init(full_bar(s), 1);
        ptx::mbar_init(empty_bar(s), 1);
      }
      for (int a = 0; a < 2; ++a) {
        ptx::mbar_init(acc_full(a), 1);
        ptx::mbar_init(acc_empty(a), 4);
      }
      ptx::fence_barrier_init();
    }
    __syncwarp();
  } else if (warp == 1) {
    ptx::tmem_alloc(tmem_slot, cfg::kTmemCols);
    ptx::tmem_relinquish();
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  ptx::tcgen05_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(gen + cfg::kOffBar + cfg::kNumBars * 8);
  pdl_wait();
  // every role walks the same tiles; the group of the next one is fetched a tile ahead (past L1: an earlier kernel of the stream wrote the table)
  auto group_of = [&](int tile) { return tile < num_tiles ? __ldcg(tile_group + tile / n_tiles) : -1; };
  int next = group_of(blockIdx.x);
  if (warp == 0) {
    uint32_t it = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      const int grp = next, m = tile / n_tiles, n = tile - m * n_tiles;
      next = group_of(tile + gridDim.x);
      if (grp < 0) continue;
      for (int kb = 0; kb < num_kb; kb += cfg::KPS, ++it) {
        const int s = it % cfg::kStages;
        ptx::mbar_wait(empty_bar(s), ((it / cfg::kStages) & 1) ^ 1u);      // first lap: falls through
        if (ptx::elect_one()) {
          const int nsub = min(cfg::KPS, num_kb - kb);
          ptx::mbar_arrive_expect_tx(full_bar(s), (uint32_t)(nsub * (cfg::kBytesA + cfg::kBytesB)));
#pragma unroll
          for (int j = 0; j < cfg::KPS; ++j) {
            if (j < nsub) {
              const uint32_t dst = base + s * cfg::kStageBytes + j * (cfg::kBytesA + cfg::kBytesB);
              ptx::tma_load_2d(dst + cfg::kBytesA, &tma_b, full_bar(s), (kb + j) * BK, grp * N + n * BN);
              ptx::tma_load_2d(dst, &tma_a, full_bar(s), (kb + j) * BK, m * BM);
            }
          }
        }
        __syncwarp();
      }
    }
  } else if (warp == 1) {
    constexpr uint32_t idesc = ptx::umma_idesc_bf16(BM, BN, 0, 0), desc_hi = ptx::umma_desc_hi_sw128(1024);
    const uint32_t a_lo0 = ptx::umma_desc_lo(base, 16);
    uint32_t it = 0, ti = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      const int grp = next;
      next = group_of(tile + gridDim.x);
      if (grp < 0) continue;
      const int acc = ti & 1;
      ptx::mbar_wait(acc_empty(acc), ((ti >> 1) & 1) ^ 1u);                // its last tile has been read out
      ptx::tcgen05_fence_after();
      for (int kb = 0; kb < num_kb; kb += cfg::KPS, ++it) {
        const int s = it % cfg::kStages;
        ptx::mbar_wait(full_bar(s), (it / cfg::kStages) & 1);
        ptx::tcgen05_fence_after();
        if (ptx::elect_one()) {
          const int nsub = min(cfg::KPS, num_kb - kb);
#pragma unroll
          for (int j = 0; j < cfg::KPS; ++j) {
            if (j < nsub) {
              const uint32_t a_lo = a_lo0 + ((s * cfg::kStageBytes + j * (cfg::kBytesA + cfg::kBytesB)) >> 4), b_lo = a_lo + (cfg::kBytesA >> 4);
#pragma unroll
              for (int k = 0; k < BK / 16; ++k)
                ptx::umma_bf16_ss(tmem + acc * BN, ptx::umma_desc(a_lo + 2 * k, desc_hi), ptx::umma_desc(b_lo + 2 * k, desc_hi), idesc, (kb | j | k) != 0 ? 1u : 0u);
            }
          }
          ptx::umma_commit(empty_bar(s));
          if (kb + cfg::KPS >= num_kb) ptx::umma_commit(acc_full(acc));
        }
        __syncwarp();
      }
      ++ti;
    }
  } else {
    const int q = warp & 3;                                                // the quadrant of tensor memory lanes this warp may read
    const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16);
    uint32_t ti = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      const int grp = next, m = tile / n_tiles, n = tile - m * n_tiles;
      next = group_of(tile + gridDim.x);
      if (grp < 0 && !zero) continue;
      RowStage st = make_row_stage(gen + cfg::kOffStaging + q * 4096, C, out_f32, epi, ldc, m * BM + q * 32, M, n * BN, BN, N);
      if (grp < 0) {                                                       // rows that no group computes
        const float f[32] = {};
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) st.emit32(lane, out_f32, NVC_EPI_NONE, f);
        st.finish(lane);
        continue;
      }
      const int acc = ti & 1;
      ptx::mbar_wait(acc_full(acc), (ti >> 1) & 1);
      ptx::tcgen05_fence_after();
#pragma unroll 1
      for (int c = 0; c < BN; c += 32) {
        uint32_t v[32];
        ptx::tmem_ld_32x32b_x32(taddr + acc * BN + c, v);
        ptx::tmem_ld_wait();
        float f[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
        st.emit32(lane, out_f32, epi, f);
      }
      st.finish(lane);
      ptx::tcgen05_fence_before();
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(acc_empty(acc));
      ++ti;
    }
  }
  ptx::tcgen05_fence_before();
  __syncthreads();
  if (warp == 1) {
    ptx::tcgen05_fence_after();
    ptx::tmem_dealloc(tmem, cfg::kTmemCols);
  }
}

int make_map(nvc_ctx* ctx, CUtensorMap* map, const void* base, uint64_t inner, uint64_t rows, uint64_t row_bytes, uint32_t box_rows) {
  cuuint64_t gdim[2] = {inner, rows}, gstr[1] = {row_bytes};
  cuuint32_t box[2] = {BK, box_rows}, estr[2] = {1, 1};
  const CUresult r = ctx->encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r == CUDA_SUCCESS) return NVC_OK;
  nvc_set_error(ctx, "cuTensorMapEncodeTiled failed with CUresult " + std::to_string((int)r));
  return NVC_EINVAL;
}

template <int BN>
int launch(nvc_ctx* ctx, const nvc_bf16* A, int lda, const nvc_bf16* W, void* C, int ldc, int out_f32, int M, int N, int K, const int32_t* tile_group, int groups,
           int epi, int zero, cudaStream_t st) {
  CUtensorMap ta, tb;
  int rc = make_map(ctx, &ta, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BM);
  if (!rc) rc = make_map(ctx, &tb, W, (uint64_t)K, (uint64_t)N * groups, (uint64_t)K * 2, BN);
  if (rc) return rc;
  const int n_tiles = (N + BN - 1) / BN;
  const long long tiles = (long long)(M / BM) * n_tiles;
  NVC_REQUIRE(ctx, tiles <= 0x7fffffffLL - ctx->num_sms && (long long)N * groups <= 0x7fffffffLL, NVC_ESHAPE, "too many tiles or weight rows");
  const int grid = (int)(tiles < ctx->num_sms ? tiles : ctx->num_sms);
  NVC_CUDA_CHECK(ctx, nvc_launch(ctx, gemm_grouped_kernel<BN>, dim3(grid), dim3(kThreads), GroupedCfg<BN>::kSmemBytes, st, ta, tb, C, ldc, out_f32, M, N, K / BK,
                                 (int)tiles, n_tiles, epi, zero, tile_group));
  NVC_CUDA_CHECK(ctx, cudaGetLastError());
  ctx->launches++;
  return NVC_OK;
}

}  // namespace

extern "C" int nvc_gemm_grouped_init(nvc_ctx* ctx) {
  NVC_CUDA_CHECK(ctx, cudaFuncSetAttribute(gemm_grouped_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, GroupedCfg<256>::kSmemBytes));
  NVC_CUDA_CHECK(ctx, cudaFuncSetAttribute(gemm_grouped_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, GroupedCfg<128>::kSmemBytes));
  NVC_CUDA_CHECK(ctx, cudaFuncSetAttribute(gemm_grouped_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, GroupedCfg<64>::kSmemBytes));
  return NVC_OK;
}

// M_cap is the host-known upper bound of the padded row count (a multiple of 128); which tiles exist is decided on the device by tile_group, so
// the launch needs no host round trip and replays inside a CUDA graph.
static int grouped(nvc_ctx* ctx, const nvc_bf16* A, int lda, const nvc_bf16* W, void* C, int ldc, int out_dtype, int M_cap, int Nout, int K, const int32_t* tile_group,
                   int groups, int act, int zero, void* stream) {
  NVC_REQUIRE(ctx, ctx && A && W && C && tile_group, NVC_EINVAL, "null pointer");
  NVC_REQUIRE(ctx, M_cap >= 0 && M_cap % BM == 0 && Nout > 0 && K > 0 && groups > 0, NVC_EINVAL, "bad sizes (M_cap must be a multiple of 128)");
  NVC_REQUIRE(ctx, K % 64 == 0 && Nout % 16 == 0, NVC_ESHAPE, "K must be a multiple of 64 and Nout of 16");
  NVC_REQUIRE(ctx, lda % 8 == 0 && lda >= K && ldc % 8 == 0 && ldc >= Nout, NVC_ESHAPE, "row strides must cover the rows and be multiples of 8");
  NVC_REQUIRE(ctx, out_dtype == NVC_DT_BF16 || out_dtype == NVC_DT_F32, NVC_EINVAL, "bad out_dtype");
  NVC_REQUIRE(ctx, act == NVC_ACT_NONE || act == NVC_ACT_RELU2, NVC_EINVAL, "activation must be NVC_ACT_NONE or NVC_ACT_RELU2");
  NVC_REQUIRE(ctx, ((uintptr_t)A % 16) == 0 && ((uintptr_t)W % 16) == 0 && ((uintptr_t)C % 16) == 0, NVC_EINVAL, "pointers must be 16-byte aligned");
  NVC_REQUIRE(ctx, ctx->encode_tiled != nullptr, NVC_EDEVICE, "cuTensorMapEncodeTiled unavailable");
  if (M_cap == 0) return NVC_OK;
  const int epi = act == NVC_ACT_RELU2 ? NVC_EPI_RELU2 : NVC_EPI_NONE, f32 = out_dtype == NVC_DT_F32;
  cudaStream_t st = nvc_stream(stream);
  // Wide tiles bring fewer bytes per column, narrow ones spread few tiles over more SMs.  256 columns from two tiles per SM on (of M_cap's), and with long
  // k-loops where waves of tiles times a k-block's (128 + BN) x 128 bytes are fewer.  How many row tiles there will be is the device's to know: M_cap holds the
  // rows, groups x 127 of padding and up to 127 of rounding; a group of up to 112 rows on average fills one tile, a larger one half a tile more than its rows.
  // us, 128 / 256 columns wide: 16 groups of 4 rows, 3 072 x 1 024 24 / 27; 4 of 200, 4 096 x 2 048 23.6 / 21.2, of 400 40 / 33; 24 of 375, 768 x 2 048 42 / 35;
  // 64 columns only where they are one wave of a long k-loop: 8 groups of 4 to 60 rows, 768 x 2 048 13.0 / 10.3
  const double rows = std::max((double)M_cap - 127.0 * groups - 64.0, 1.0), per = rows / groups;
  const double m_tiles = groups * (per <= 112.0 ? std::min(per, 1.0) : per / BM + 0.5);
  auto cost = [&](int bn) { return std::max(std::ceil(m_tiles * ((Nout + bn - 1) / bn) / ctx->num_sms - 0.08), 1.0) * (128 + bn); };
  if ((long long)(M_cap / BM) * ((Nout + 63) / 64) <= ctx->num_sms && K >= 2048)
    return launch<64>(ctx, A, lda, W, C, ldc, f32, M_cap, Nout, K, tile_group, groups, epi, zero, st);
  const long long wide = (long long)(M_cap / BM) * ((Nout + 255) / 256);
  if (wide >= 2LL * ctx->num_sms || (K >= 1024 && cost(256) < 0.97 * cost(128))) return launch<256>(ctx, A, lda, W, C, ldc, f32, M_cap, Nout, K, tile_group, groups, epi, zero, st);
  return launch<128>(ctx, A, lda, W, C, ldc, f32, M_cap, Nout, K, tile_group, groups, epi, zero, st);
}

extern "C" int nvc_gemm_bf16_grouped(nvc_ctx* ctx, const nvc_bf16* A, int lda, const nvc_bf16* W, void* C, int ldc, int out_dtype, int M_cap, int Nout, int K,
                                     const int32_t* tile_group, int groups, int act, void* stream) {
  return grouped(ctx, A, lda, W, C, ldc, out_dtype, M_cap, Nout, K, tile_group, groups, act, 0, stream);
}
extern "C" int nvc_gemm_bf16_grouped_zero(nvc_ctx* ctx, const nvc_bf16* A, int lda, const nvc_bf16* W, void* C, int ldc, int out_dtype, int M_cap, int Nout, int K,
                                          const int32_t* tile_group, int groups, int act, void* stream) {
  return grouped(ctx, A, lda, W, C, ldc, out_dtype, M_cap, Nout, K, tile_group, groups, act, 1, stream);
}
