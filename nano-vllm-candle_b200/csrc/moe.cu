// Mixture-of-experts routing around the grouped matrix products (linear_generic.cu, moe_gemm): everything is sized
// by device-resident counts, so a step needs no host round trip and replays inside a CUDA graph.
//   nvc_moe_route    router logits in fp32, sigmoid scores, biased top-k choice, normalised weights, shared-expert gate
//   nvc_moe_sort     counting sort of the (token, choice) pairs by expert: group offsets, source rows, positions
//   nvc_moe_combine  weighted sum of a token's expert rows plus the gated shared expert, fp32
#include "ptx.cuh"
#include "typed.cuh"

namespace {

// one warp per token.  Scores of up to 32 * PER experts live in registers: one per lane up to 32 experts (4 000 tokens, 16 experts, cold
// cache: 8.5 -> 5.6 us against eight), else eight.
constexpr int kMaxPerLane = 8;   // experts <= 256

// top-k by repeated arg-max over the choice scores c (ties -> the lower expert index); expert e lives in lane e % 32,
// slot e / 32.  Writes idx / weights of token n: s_chosen / (sum of the chosen s + 1e-20) * scale.  idx names an expert whatever the scores are.
template <int PER>
__device__ __forceinline__ void topk_write(float (&s)[PER], float (&c)[PER], int lane, int E, int top, float scale,
                                           int32_t* __restrict__ idx, float* __restrict__ wout, int64_t n, bool normalize = true) {
  // top-k by repeated arg-max over the choice scores (ties -> the lower expert index)
  float sel_sum = 0.f, my_w = 0.f;
  int my_e = 0;
  for (int t = 0; t < top; ++t) {
    float bv = -INFINITY;
    int be = 0x7fffffff;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = lane + 32 * i;
      if (e < E && (c[i] > bv || (c[i] == bv && e < be))) { bv = c[i]; be = e; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
      const int oe = __shfl_xor_sync(0xffffffffu, be, o);
      if (ov > bv || (ov == bv && oe < be)) { bv = ov; be = oe; }
    }
    if (be >= E) be = 0;                      // only NaNs are left, which compare with nothing: expert 0, with the weight NaN
    // the owner lane publishes the unbiased score and retires the expert
    float sv = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i == be) { sv = s[i]; c[i] = -INFINITY; }
    sv = __shfl_sync(0xffffffffu, sv, be & 31);
    sel_sum += sv;
    if (lane == t % 32) { my_w = sv; my_e = be; }
    if (t % 32 == 31 || t == top - 1) {
      // flush up to 32 choices (weights are scaled after the loop: keep raw scores for now)
      const int t0 = t - (t % 32);
      if (t0 + lane <= t) { idx[(int64_t)n * top + t0 + lane] = my_e; wout[(int64_t)n * top + t0 + lane] = my_w; }
    }
  }
  __syncwarp();
  const float inv = normalize ? scale / (sel_sum + 1e-20f) : scale;
  for (int t = lane; t < top; t += 32) wout[(int64_t)n * top + t] *= inv;
}

// scores from logits that a matrix product has already taken: z [N, ldz] fp32, column gate_col (if >= 0) = the shared gate
template <int PER>
__global__ void moe_topk_kernel(const float* z, int ldz, const float* __restrict__ corr, int E, int top, float scale,
                                int gate_col, int score, int normalize, int32_t* __restrict__ idx, float* __restrict__ wout,
                                float* __restrict__ gate, int N) {
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * (blockDim.x >> 5) + warp;
  if (n >= N) return;
  const float* zr = z + (int64_t)n * ldz;
  float s[PER], c[PER];
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = lane + 32 * i;
    s[i] = 0.f;
    c[i] = -INFINITY;
    if (e < E) s[i] = zr[e];
  }
  if (score == NVC_ROUTE_SOFTMAX) {       // over all E columns, fp32
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i < E) mx = fmaxf(mx, s[i]);
    mx = warp_max(mx);
    float den = 0.f;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i < E) { s[i] = expf(s[i] - mx); den += s[i]; }
    den = warp_sum(den);
#pragma unroll
    for (int i = 0; i < PER; ++i) s[i] = s[i] / den;
  } else if (score == NVC_ROUTE_CHOSEN) { // choice by biased logits; the scores are their exponentials (the largest logit is always chosen)
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i < E) { c[i] = s[i] + __ldg(corr + lane + 32 * i); mx = fmaxf(mx, c[i]); }
    mx = warp_max(mx);
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i < E) s[i] = expf(c[i] - mx);
  } else {
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i < E) s[i] = sigmoid_f32(s[i]);
  }
  if (score != NVC_ROUTE_CHOSEN) {
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (lane + 32 * i < E) c[i] = s[i] + __ldg(corr + lane + 32 * i);
  }
  if (gate_col >= 0 && gate && lane == 0) gate[n] = sigmoid_f32(zr[gate_col]);
  topk_write(s, c, lane, E, top, scale, idx, wout, n, normalize != 0);
}

template <typename T>
__global__ void moe_route_kernel(const T* h, int ldh, const float* __restrict__ wr, const float* __restrict__ corr,
                                 const float* __restrict__ wsg, int E, int top, float scale, int32_t* __restrict__ idx,
                                 float* __restrict__ wout, float* __restrict__ gate, int N, int H) {
  extern __shared__ float hs[];   // [warps][H]
  pdl_trigger();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.x * (blockDim.x >> 5) + warp;
  if (n >= N) return;
  float* x = hs + (size_t)warp * H;
  for (int j = lane; j < H; j += 32) x[j] = ld_f(h + (int64_t)n * ldh + j);
  __syncwarp();
  // expert e's score lives in lane e % 32, slot e / 32; every dot product is taken by the whole warp (coalesced weight rows)
  float s[kMaxPerLane], c[kMaxPerLane];
#pragma unroll
  for (int i = 0; i < kMaxPerLane; ++i) { s[i] = 0.f; c[i] = -INFINITY; }
  for (int e0 = 0; e0 < E; e0 += 4) {           // four experts at a time: independent loads and sums
    float z[4] = {0.f, 0.f, 0.f, 0.f};
    const float* w0 = wr + (int64_t)e0 * H;
#pragma unroll 4
    for (int j = lane; j < H; j += 32) {
      const float xv = x[j];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (e0 + u < E) z[u] = fmaf(xv, __ldg(w0 + (int64_t)u * H + j), z[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int e = e0 + u;
      const float zu = warp_sum(z[u]);
      if (e < E && lane == (e & 31)) {
        const float sv = sigmoid_f32(zu), cv = sv + __ldg(corr + e);
#pragma unroll
        for (int i = 0; i < kMaxPerLane; ++i)
          if (i == (e >> 5)) { s[i] = sv; c[i] = cv; }
      }
    }
  }
  if (wsg && gate) {
    float z = 0.f;
    for (int j = lane; j < H; j += 32) z = fmaf(x[j], __ldg(wsg + j), z);
    z = warp_sum(z);
    if (lane == 0) gate[n] = sigmoid_f32(z);
  }
  topk_write(s, c, lane, E, top, scale, idx, wout, n);
}

// Stable counting sort by expert in one CTA of 32 warps or a cluster of C (pairs = N * top).  Warp w owns the contiguous segment w of the
// pairs: it counts its pairs per expert, a prefix over (expert, warp) gives every warp its first position in every
// expert's group, and the warp then places its pairs in order (__match_any_sync ranks equal experts inside a batch of
// 32).  Within an expert the pairs keep token order, so the layout - and every sum downstream - is deterministic.
// One CTA's latencies are its time: a warp requests 8 x 32 of its pairs at once and keeps the first 256 for the second pass, and both prefixes go by
// exchange (8 000 pairs, 16 experts, cold cache: 11.1 -> 10.6 us against loads one behind the other and prefixes thread by thread; 128 pairs 6.0 -> 5.3).
// Of many pairs it is one SM's scattered 4-byte stores and matches: eight CTAs take a stretch each and read each other's counts per expert (8 000 pairs, 16 experts
// 8.3 -> 4.6 us; 32 000 pairs, 128 experts 49.8 -> 11.0).  Counts lie in rows of an odd length: 128 of them put a column of 32 into one bank (512 pairs 11.1 -> 7.3).
template <int C>
__global__ void __launch_bounds__(1024)
moe_sort_kernel(const int32_t* idx, int P, int top, int E, int E_real, int align, int32_t* __restrict__ offsets,
                int32_t* __restrict__ src_rows, int32_t* __restrict__ pos, int32_t* __restrict__ tile_group, int tiles_cap, int tail_cap, int tail) {
  extern __shared__ int32_t sm[];   // [32][E | 1] counts -> pairs of earlier warps, then [E + 1] offsets, [E] sizes and, of several CTAs, [E] pairs here and [E] pairs of earlier CTAs
  const int Es = E | 1;                                  // a column of an even number of counts would lie in few banks
  int32_t* cnt = sm;
  int32_t* off = sm + 32 * Es;
  int32_t* size = off + E + 1;
  int32_t* here = C > 1 ? size + E : size;
  int32_t* before = here + E;
  constexpr int kBatch = 8;
  pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, rank = C > 1 ? blockIdx.x : 0, run = rank * 32 + warp;
  for (int i = threadIdx.x; i < 32 * Es; i += blockDim.x) cnt[i] = 0;
  pdl_wait();
  const int seg = ((P + 32 * C - 1) / (32 * C) + 31) / 32 * 32;      // pairs per warp, a multiple of 32
  const int p_begin = min(P, run * seg), p_end = min(P, run * seg + seg);
  int e[kBatch];
  auto load = [&](int p0) {
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      e[i] = p0 + 32 * i + lane < p_end ? idx[p0 + 32 * i + lane] : -1;
      if ((uint32_t)e[i] >= (uint32_t)E) e[i] = -1 - lane;                   // absent lanes match nobody; no expert, no place
    }
  };
  load(p_begin);
  __syncthreads();
  for (int p0 = p_begin; p0 < p_end; p0 += 32 * kBatch) {
    if (p0 > p_begin) load(p0);
#pragma unroll
    for (int i = 0; i < kBatch; ++i)
      if (e[i] >= 0) atomicAdd(&cnt[warp * Es + e[i]], 1);
  }
  __syncthreads();
  for (int x = warp; x < E; x += 32) {                   // an expert's pairs in earlier warps
    const int v = cnt[lane * Es + x];
    int sum = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += up;
    }
    cnt[lane * Es + x] = sum - v;
    if (lane == 31) here[x] = sum;
  }
  if constexpr (C > 1) {
    __syncwarp();                                        // the barrier is for whole warps
    ptx::cluster_sync_all();
    for (int x = threadIdx.x; x < E; x += blockDim.x) {
      int all = 0, earlier = 0;
#pragma unroll
      for (int r = 0; r < C; ++r) {
        const int v = ptx::ld_cluster_s32(ptx::mapa_u32(smem_u32(here + x), r));
        all += v;
        earlier += r < rank ? v : 0;
      }
      size[x] = all;
      before[x] = earlier;
    }
  }
  __syncthreads();
  if (warp == 0) {                                       // every group starts at a multiple of `align` rows
    int base = 0;
    for (int x0 = 0; x0 < E; x0 += 32) {
      int sum = x0 + lane < E ? (size[x0 + lane] + align - 1) / align * align : 0;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += up;
      }
      if (x0 + lane < E) off[x0 + lane + 1] = base + sum;
      base += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) off[0] = 0;
  }
  __syncthreads();
  if (align > 1) {
    // rows between a group's last pair and the next group's start have no source; tiles of `align` rows -> their group
    for (int x = run; x < E; x += 32 * C) {
      for (int r = off[x] + size[x] + lane; r < off[x + 1]; r += 32) src_rows[r] = -1;
      if (tile_group)
        for (int t = off[x] / align + lane; t < off[x + 1] / align; t += 32) tile_group[t] = x < E_real ? x : -1;   // no product behind an identity expert
    }
    if (tile_group)
      for (int t = off[E] / align + rank * blockDim.x + threadIdx.x; t < tiles_cap; t += C * blockDim.x) tile_group[t] = -1;
    for (int r = off[E] + rank * blockDim.x + threadIdx.x; r < tail_cap; r += C * blockDim.x) src_rows[r] = tail;       // behind the last group
  }
  if (rank == 0)
    for (int x = threadIdx.x; x <= E; x += blockDim.x) offsets[x] = off[x];
  const bool kept = p_end - p_begin <= 32 * kBatch;
  for (int p0 = p_begin; p0 < p_end; p0 += 32 * kBatch) {
    if (!kept) load(p0);
#pragma unroll
    for (int i = 0; i < kBatch; ++i) {
      if (p0 + 32 * i >= p_end) break;                   // warp-uniform
      const int p = p0 + 32 * i + lane, x = e[i];
      const unsigned peers = __match_any_sync(0xffffffffu, x);
      if (x >= 0) {
        const int at = off[x] + (C > 1 ? before[x] : 0) + cnt[warp * Es + x] + __popc(peers & ((1u << lane) - 1));
        src_rows[at] = p / top;
        pos[p] = at;
      } else if (p < p_end) {
        pos[p] = 0;                                      // no expert, no place: a row that exists, so that what reads it stays in bounds
      }
      __syncwarp();
      if (x >= 0 && lane == 31 - __clz(peers)) cnt[warp * Es + x] += __popc(peers);   // the last peer advances the group
      __syncwarp();
    }
  }
  if constexpr (C > 1) {                                 // the other CTAs have read this one's counts
    __syncwarp();
    ptx::cluster_sync_all();
  }
}

// out[r] = in[src_rows[r]] for r < *num_rows (a device count), zeros where src_rows[r] < 0, `two` (a pair of bf16) behind them when fill is set;
// 16 bytes per thread
__global__ void gather_rows_kernel(const uint4* in, int ld_in, const int32_t* src_rows,
                                   const int32_t* num_rows, uint4* __restrict__ out, int ld_out, int rows_cap, int per_row,
                                   int rows_per_cta, int fill, uint32_t two) {
  pdl_trigger();
  pdl_wait();
  const int n = min(rows_cap, *num_rows);
  for (int i = threadIdx.x; i < rows_per_cta * per_row; i += blockDim.x) {
    const int r = blockIdx.x * rows_per_cta + i / per_row, c = i % per_row;
    if (r >= n) {
      if (!fill || r >= rows_cap) break;
      out[(int64_t)r * ld_out + c] = make_uint4(two, two, two, two);
      continue;
    }
    const int src = src_rows[r];
    out[(int64_t)r * ld_out + c] = src >= 0 ? in[(int64_t)src * ld_in + c] : make_uint4(0u, 0u, 0u, 0u);
  }
}

// The same for rows of 512 numbers and more: a warp per row, four accesses per lane in flight, no division (10 000 x 1 024, cold cache: 8.5 -> 7.0 us)
__global__ void __launch_bounds__(128) gather_rows_warp_kernel(const uint4* in, int ld_in, const int32_t* src_rows,
                                                               const int32_t* num_rows, uint4* out, int ld_out, int rows_cap, int per_row,
                                                               int fill, uint32_t two) {
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const bool behind = r >= min(rows_cap, *num_rows);
  if (r >= rows_cap || (behind && !fill)) return;
  const int src = behind ? -1 : src_rows[r];
  const uint32_t v = behind ? two : 0u;
  const uint4* x = in + (int64_t)max(src, 0) * ld_in;
  uint4* y = out + (int64_t)r * ld_out;
  for (int c = lane; c < per_row; c += 128) {
    uint4 q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[i] = src >= 0 && c + 32 * i < per_row ? x[c + 32 * i] : make_uint4(v, v, v, v);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (c + 32 * i < per_row) y[c + 32 * i] = q[i];
  }
}

// experts from E_real on are identity experts: their pairs read the token's own row x[n] instead of a row of y
template <typename TY, typename TX>
__global__ void moe_combine_identity_kernel(const TY* y, int ldy, const int32_t* pos, const float* w,
                                            const int32_t* idx, int top, int E_real, const TX* x, int ldx,
                                            float* __restrict__ out, int ldo, int H) {
  pdl_trigger();
  pdl_wait();
  const int n = blockIdx.x;
  for (int j = threadIdx.x; j < H; j += blockDim.x) {
    float a = 0.f;
    for (int t = 0; t < top; ++t) {
      const int64_t p = (int64_t)n * top + t;
      const float v = idx[p] < E_real ? ld_f(y + (int64_t)pos[p] * ldy + j) : ld_f(x + (int64_t)n * ldx + j);
      a = fmaf(w[p], v, a);
    }
    out[(int64_t)n * ldo + j] = a;
  }
}

template <typename TY, typename TS>
__global__ void moe_combine_kernel(const TY* y, int ldy, const int32_t* pos, const float* w,
                                   int top, const TS* shared, int lds, const float* gate,
                                   float* __restrict__ out, int ldo, int H) {
  pdl_trigger();
  pdl_wait();
  const int n = blockIdx.x;
  for (int j = threadIdx.x; j < H; j += blockDim.x) {
    float a = 0.f;
    for (int t = 0; t < top; ++t) a = fmaf(w[(int64_t)n * top + t], ld_f(y + (int64_t)pos[(int64_t)n * top + t] * ldy + j), a);
    if (shared) a += ld_f(shared + (int64_t)n * lds + j) * (gate ? gate[n] : 1.0f);
    out[(int64_t)n * ldo + j] = a;
  }
}

// the same sum on fp32 rows whose width and strides are multiples of 4: 16-byte loads and stores, same order of additions.  TOP: the choices when they are
// 1 .. 4 (their rows are requested together), else 0
template <int TOP>
__global__ void moe_combine_f4_kernel(const float4* y, int ldy4, const int32_t* pos, const float* w,
                                      int top, const float4* shared, int lds4, const float* gate,
                                      float4* out, int ldo4, int H4) {
  pdl_trigger();
  pdl_wait();
  const int n = blockIdx.x;
  const float g = shared ? (gate ? gate[n] : 1.0f) : 0.f;
  constexpr int KEEP = TOP > 0 ? TOP : 1;
  int at[KEEP];
  float wt[KEEP];
  if constexpr (TOP > 0) {
#pragma unroll
    for (int t = 0; t < TOP; ++t) { at[t] = pos[(int64_t)n * TOP + t]; wt[t] = w[(int64_t)n * TOP + t]; }
  }
  for (int j = threadIdx.x; j < H4; j += blockDim.x) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [&](float f, const float4& v) { a.x = fmaf(f, v.x, a.x); a.y = fmaf(f, v.y, a.y); a.z = fmaf(f, v.z, a.z); a.w = fmaf(f, v.w, a.w); };
    if constexpr (TOP > 0) {
      float4 v[KEEP];
#pragma unroll
      for (int t = 0; t < TOP; ++t) v[t] = y[(int64_t)at[t] * ldy4 + j];
#pragma unroll
      for (int t = 0; t < TOP; ++t) add(wt[t], v[t]);
    } else {
      for (int t = 0; t < top; ++t) add(w[(int64_t)n * top + t], y[(int64_t)pos[(int64_t)n * top + t] * ldy4 + j]);
    }
    if (shared) {
      const float4 v = shared[(int64_t)n * lds4 + j];
      a.x += v.x * g; a.y += v.y * g; a.z += v.z * g; a.w += v.w * g;
    }
    out[(int64_t)n * ldo4 + j] = a;
  }
}

// one CTA per (token, choice): the token's row times the pair's router weight, written where the sort put the pair
template <typename T>
__global__ void moe_scatter_scaled_kernel(const T* h, int ldh, const int32_t* pos, const float* topk_w,
                                          T* __restrict__ out, int ldo, int top, int H) {
  pdl_trigger();
  pdl_wait();
  const int pair = blockIdx.x, n = pair / top;
  const float w = topk_w[pair];
  const T* x = h + (int64_t)n * ldh;
  T* y = out + (int64_t)pos[pair] * ldo;
  for (int j = threadIdx.x; j < H; j += blockDim.x) st_f(y + j, w * ld_f(x + j));
}

}  // namespace

extern "C" {

int nvc_moe_route(nvc_ctx* ctx, const void* h, int h_dtype, int ldh, const float* w_router, const float* correction,
                  const float* w_shared_gate, int E, int top, float scale, int32_t* topk_idx, float* topk_w, float* gate, int N,
                  int H, void* stream) {
  NVC_REQUIRE(ctx, ctx && h && w_router && correction && topk_idx && topk_w, NVC_EINVAL, "null pointer");
  NVC_REQUIRE(ctx, (w_shared_gate == nullptr) == (gate == nullptr), NVC_EINVAL, "the shared gate needs its weight and its output");
  NVC_REQUIRE(ctx, E > 0 && E <= 32 * kMaxPerLane && top > 0 && top <= E, NVC_ESHAPE, "experts must be in [1, 256], top in [1, experts]");
  NVC_REQUIRE(ctx, N >= 0 && H > 0 && ldh >= H && H <= 12288, NVC_EINVAL, "bad sizes");
  if (N == 0) return NVC_OK;
  const int warps = H <= 3072 ? 4 : 1;
  const size_t smem = (size_t)warps * H * sizeof(float);
  NVC_DISPATCH_DT(h_dtype, T,
                  NVC_CUDA_CHECK(ctx, nvc_launch(ctx, moe_route_kernel<T>, dim3((N + warps - 1) / warps), dim3(32 * warps), smem,
                                                 nvc_stream(stream), reinterpret_cast<const T*>(h), ldh, w_router, correction,
                                                 w_shared_gate, E, top, scale, topk_idx, topk_w, gate, N, H)));
  ctx->launches++;
  return NVC_OK;
}

int nvc_moe_route_logits(nvc_ctx* ctx, const float* z, int ldz, const float* correction, int E, int top, float scale, int gate_col,
                         int32_t* topk_idx, float* topk_w, float* gate, int N, void* stream) {
  return nvc_moe_route_logits_ex(ctx, z, ldz, correction, E, top, scale, gate_col, NVC_ROUTE_SIGMOID, 1, topk_idx, topk_w, gate, N, stream);
}

int nvc_moe_route_logits_ex(nvc_ctx* ctx, const float* z, int ldz, const float* correction, int E, int top, float scale, int gate_col,
                            int score, int normalize, int32_t* topk_idx, float* topk_w, float* gate, int N, void* stream) {
  NVC_REQUIRE(ctx, ctx && z && correction && topk_idx && topk_w, NVC_EINVAL, "null pointer");
  NVC_REQUIRE(ctx, score >= NVC_ROUTE_SIGMOID && score <= NVC_ROUTE_CHOSEN, NVC_EINVAL, "unknown score function");
  NVC_REQUIRE(ctx, E > 0 && E <= 32 * kMaxPerLane && top > 0 && top <= E, NVC_ESHAPE, "experts must be in [1, 256], top in [1, experts]");
  NVC_REQUIRE(ctx, N >= 0 && ldz >= E && gate_col < ldz && (gate_col < 0 || gate), NVC_EINVAL, "bad sizes");
  if (N == 0) return NVC_OK;
  NVC_CUDA_CHECK(ctx, nvc_launch(ctx, E <= 32 ? moe_topk_kernel<1> : moe_topk_kernel<kMaxPerLane>, dim3((N + 3) / 4), dim3(128), 0, nvc_stream(stream), z, ldz, correction, E, top, scale,
                                 gate_col, score, normalize, topk_idx, topk_w, gate, N));
  ctx->launches++;
  return NVC_OK;
}

int nvc_moe_sort(nvc_ctx* ctx, const int32_t* topk_idx, int N, int top, int E, int32_t* offsets, int32_t* src_rows, int32_t* pos,
                 void* stream) {
  return nvc_moe_sort_padded(ctx, topk_idx, N, top, E, 1, offsets, src_rows, pos, nullptr, 0, stream);
}

int nvc_moe_sort_padded(nvc_ctx* ctx, const int32_t* topk_idx, int N, int top, int E, int align, int32_t* offsets, int32_t* src_rows,
                        int32_t* pos, int32_t* tile_group, int tiles_cap, void* stream) {
  return nvc_moe_sort_padded_ex(ctx, topk_idx, N, top, E, E, align, offsets, src_rows, pos, tile_group, tiles_cap, stream);
}

static int sort_padded(nvc_ctx* ctx, const int32_t* topk_idx, int N, int top, int E, int E_real, int align, int32_t* offsets, int32_t* src_rows, int32_t* pos,
                       int32_t* tile_group, int tiles_cap, int tail_cap, int tail, void* stream) {
  NVC_REQUIRE(ctx, ctx && topk_idx && offsets && src_rows && pos, NVC_EINVAL, "null pointer");
  NVC_REQUIRE(ctx, E_real >= 0 && E_real <= E, NVC_EINVAL, "E_real must be in [0, E]");
  NVC_REQUIRE(ctx, N >= 0 && top > 0 && E > 0 && E <= 320 && align >= 1, NVC_EINVAL, "bad sizes");
  NVC_REQUIRE(ctx, !tile_group || (align > 1 && (int64_t)tiles_cap * align >= (int64_t)N * top + (int64_t)E * (align - 1)), NVC_EINVAL,
              "tile_group needs align > 1 and room for every group's padding");
  const int P = N * top;
  // Eight CTAs cost 0.8 - 1.1 us of cluster launch and barriers.  They divide the pairs, which take longer the more experts there are, and the walks over padded groups, 32 of them at a time (us, one /
  // eight CTAs, pairs to experts, groups of 128 rows: to 8 experts 3 200 4.2 / 4.4, 4 800 4.8 / 4.4; to 16 2 000 4.0 / 4.5, 3 200 4.8 / 4.5, 8 000 7.6 / 4.6; to 32 2 000 5.0 / 5.5, 3 200 5.95 /
  // 5.55; to 64 1 000 5.3 / 6.05, 2 000 6.4 / 6.2; to 95 32 4.7 / 5.1, 1 000 6.45 / 6.5, 2 000 7.6 / 6.6; to 128 8 5.35 / 5.5, with the rows behind the groups filled 6.15 / 5.6, 128 6.5 / 5.9,
  // 32 000 43.8 / 11.0; to 256 8 8.2 / 7.15; unpadded to 128 2 000 6.2 / 6.3, 3 200 7.25 / 6.5)
  const int C = P + (int64_t)E * E * (align - 1) / 690 > (E > 16 ? 3000 : 3500) ? 8 : 1;
  auto kernel = C == 8 ? moe_sort_kernel<8> : moe_sort_kernel<1>;
  NVC_CUDA_CHECK(ctx, nvc_launch_cluster(ctx, kernel, dim3(C), dim3(1024), (size_t)(32 * (E | 1) + (C > 1 ? 4 : 2) * E + 1) * sizeof(int32_t), nvc_stream(stream), C,
                                         topk_idx, P, top, E, E_real, align, offsets, src_rows, pos, tile_group, tiles_cap, tail_cap, tail));
  ctx->launches++;
  return NVC_OK;
}

int nvc_moe_sort_padded_ex(nvc_ctx* ctx, const int32_t* topk_idx, int N, int top, int E, int E_real, int align, int32_t* offsets,
                           int32_t* src_rows, int32_t* pos, int32_t* tile_group, int tiles_cap, void* stream) {
  return sort_padded(ctx, topk_idx, N, top, E, E_real, align, offsets, src_rows, pos, tile_group, tiles_cap, 0, 0, stream);
}

int nvc_moe_sort_padded_fill(nvc_ctx* ctx, const int32_t* topk_idx, int N, int top, int E, int E_real, int align, int32_t* offsets,
                             int32_t* src_rows, int32_t* pos, int32_t* tile_group, int tiles_cap, int tail, void* stream) {
  NVC_REQUIRE(ctx, align > 1 && tile_group, NVC_EINVAL, "groups of rows and their table are wanted");
  return sort_padded(ctx, topk_idx, N, top, E, E_real, align, offsets, src_rows, pos, tile_group, tiles_cap, tiles_cap * align, tail, stream);
}

static int gather(nvc_ctx* ctx, const nvc_bf16* in, int ld_in, const int32_t* src_rows, const int32_t* num_rows, nvc_bf16* out, int ld_out, int rows_cap, int width,
                  int fill, nvc_bf16 value, void* stream) {
  NVC_REQUIRE(ctx, ctx && in && src_rows && num_rows && out, NVC_EINVAL, "null pointer");
  NVC_REQUIRE(ctx, rows_cap >= 0 && width > 0 && width % 8 == 0 && ld_in % 8 == 0 && ld_out % 8 == 0 && ld_in >= width && ld_out >= width,
              NVC_ESHAPE, "width and row strides must be multiples of 8");
  NVC_REQUIRE(ctx, ((uintptr_t)in % 16) == 0 && ((uintptr_t)out % 16) == 0, NVC_EINVAL, "pointers must be 16-byte aligned");
  if (rows_cap == 0) return NVC_OK;
  const int per_row = width / 8;                                   // 16-byte chunks per row
  if (per_row >= 64) {
    NVC_CUDA_CHECK(ctx, nvc_launch(ctx, gather_rows_warp_kernel, dim3((rows_cap + 3) / 4), dim3(128), 0, nvc_stream(stream), reinterpret_cast<const uint4*>(in),
                                   ld_in / 8, src_rows, num_rows, reinterpret_cast<uint4*>(out), ld_out / 8, rows_cap, per_row, fill, (uint32_t)value * 0x10001u));
    ctx->launches++;
    return NVC_OK;
  }
  const int rows_per_cta = std::max(1, 256 / per_row);
  NVC_CUDA_CHECK(ctx, nvc_launch(ctx, gather_rows_kernel, dim3((rows_cap + rows_per_cta - 1) / rows_per_cta), dim3(256), 0, nvc_stream(stream),
                                 reinterpret_cast<const uint4*>(in), ld_in / 8, src_rows, num_rows, reinterpret_cast<uint4*>(out), ld_out / 8,
                                 rows_cap, per_row, rows_per_cta, fill, (uint32_t)value * 0x10001u));
  ctx->launches++;
  return NVC_OK;
}

int nvc_gather_rows_bf16(nvc_ctx* ctx, const nvc_bf16* in, int ld_in, const int32_t* src_rows, const int32_t* num_rows, nvc_bf16* out,
                         int ld_out, int rows_cap, int width, void* stream) {
  return gather(ctx, in, ld_in, src_rows, num_rows, out, ld_out, rows_cap, width, 0, 0, stream);
}

int nvc_gather_rows_bf16_fill(nvc_ctx* ctx, const nvc_bf16* in, int ld_in, const int32_t* src_rows, const int32_t* num_rows, nvc_bf16* out,
                              int ld_out, int rows_cap, int width, nvc_bf16 value, void* stream) {
  return gather(ctx, in, ld_in, src_rows, num_rows, out, ld_out, rows_cap, width, 1, value, stream);
}

int nvc_moe_combine(nvc_ctx* ctx, const void* y, int y_dtype, int ldy, const int32_t* pos, const float* topk_w, int top,
                    const void* shared, int shared_dtype, int lds, const float* gate, float* out, int ldo, int N, int H,
                    void* stream) {
  NVC_REQUIRE(ctx, ctx && y && pos && topk_w && out, NVC_EINVAL, "null pointer");
  NVC_REQUIRE(ctx, N >= 0 && H > 0 && top > 0 && ldy >= H && ldo >= H && (!shared || lds >= H), NVC_EINVAL, "bad sizes");
  if (N == 0) return NVC_OK;
  if (y_dtype == NVC_DT_F32 && (!shared || shared_dtype == NVC_DT_F32) && H % 4 == 0 && ldy % 4 == 0 && ldo % 4 == 0 &&
      (!shared || lds % 4 == 0) && ((uintptr_t)y % 16) == 0 && ((uintptr_t)out % 16) == 0 && ((uintptr_t)shared % 16) == 0) {
    auto* kernel = top == 1 ? moe_combine_f4_kernel<1> : (top == 2 ? moe_combine_f4_kernel<2> : (top == 3 ? moe_combine_f4_kernel<3> :
                                                                                                    (top == 4 ? moe_combine_f4_kernel<4> : moe_combine_f4_kernel<0>)));
    NVC_CUDA_CHECK(ctx, nvc_launch(ctx, kernel, dim3(N), dim3(H / 4 >= 256 ? 256 : (H / 4 > 32 ? 128 : 32)), 0, nvc_stream(stream),
                                   reinterpret_cast<const float4*>(y), ldy / 4, pos, topk_w, top, reinterpret_cast<const float4*>(shared), lds / 4,
                                   gate, reinterpret_cast<float4*>(out), ldo / 4, H / 4));
    ctx->launches++;
    return NVC_OK;
  }
  const dim3 grid(N), block(H >= 1024 ? 512 : 128);
#define NVC_COMBINE(TY, TS)                                                                                                        \
  NVC_CUDA_CHECK(ctx, nvc_launch(ctx, moe_combine_kernel<TY, TS>, grid, block, 0, nvc_stream(stream), reinterpret_cast<const TY*>(y), \
                                 ldy, pos, topk_w, top, reinterpret_cast<const TS*>(shared), lds, gate, out, ldo, H))
  if (y_dtype == NVC_DT_F32 && shared_dtype == NVC_DT_F32) NVC_COMBINE(float, float);
  else if (y_dtype == NVC_DT_F32) NVC_COMBINE(float, __nv_bfloat16);
  else if (shared_dtype == NVC_DT_F32) NVC_COMBINE(__nv_bfloat16, float);
  else NVC_COMBINE(__nv_bfloat16, __nv_bfloat16);
#undef NVC_COMBINE
  ctx->launches++;
  return NVC_OK;
}

int nvc_moe_combine_identity(nvc_ctx* ctx, const void* y, int y_dtype, int ldy, const int32_t* pos, const float* topk_w,
                             const int32_t* topk_idx, int top, int E_real, const void* x, int x_dtype, int ldx, float* out, int ldo,
                             int N, int H, void* stream) {
  NVC_REQUIRE(ctx, ctx && y && pos && topk_w && topk_idx && x && out, NVC_EINVAL, "null pointer");
  NVC_REQUIRE(ctx, N >= 0 && H > 0 && top > 0 && E_real >= 0 && ldy >= H && ldo >= H && ldx >= H, NVC_EINVAL, "bad sizes");
  if (N == 0) return NVC_OK;
  const dim3 grid(N), block(H >= 1024 ? 512 : 128);
#define NVC_COMBINE(TY, TX)                                                                                                                  \
  NVC_CUDA_CHECK(ctx, nvc_launch(ctx, moe_combine_identity_kernel<TY, TX>, grid, block, 0, nvc_stream(stream), reinterpret_cast<const TY*>(y), \
                                 ldy, pos, topk_w, topk_idx, top, E_real, reinterpret_cast<const TX*>(x), ldx, out, ldo, H))
  if (y_dtype == NVC_DT_F32 && x_dtype == NVC_DT_F32) NVC_COMBINE(float, float);
  else if (y_dtype == NVC_DT_F32) NVC_COMBINE(float, __nv_bfloat16);
  else if (x_dtype == NVC_DT_F32) NVC_COMBINE(__nv_bfloat16, float);
  else NVC_COMBINE(__nv_bfloat16, __nv_bfloat16);
#undef NVC_COMBINE
  ctx->launches++;
  return NVC_OK;
}

int nvc_moe_scatter_scaled(nvc_ctx* ctx, const void* h, int dtype, int ldh, const int32_t* pos, const float* topk_w, int top, void* out,
                           int ldo, int N, int H, void* stream) {
  NVC_REQUIRE(ctx, ctx && h && pos && topk_w && out, NVC_EINVAL, "null pointer");
  NVC_REQUIRE(ctx, N >= 0 && H > 0 && top > 0 && ldh >= H && ldo >= H, NVC_EINVAL, "bad sizes");
  if (N == 0) return NVC_OK;
  NVC_DISPATCH_DT(dtype, T,
                  NVC_CUDA_CHECK(ctx, nvc_launch(ctx, moe_scatter_scaled_kernel<T>, dim3(N * top), dim3(H >= 1024 ? 256 : 128), 0, nvc_stream(stream),
                                                 reinterpret_cast<const T*>(h), ldh, pos, topk_w, reinterpret_cast<T*>(out), ldo, top, H)));
  ctx->launches++;
  return NVC_OK;
}

}  // extern "C"
