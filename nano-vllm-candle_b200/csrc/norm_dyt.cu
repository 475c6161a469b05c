// Norms and row operations of the models whose residual stream and norms are fp32 end to end:
//   nvc_embed_gather_f32    token rows of the embedding table as fp32
//   nvc_dyt_norm            Dynamic Tanh norm (no mean, no variance) fused with the residual accumulation
//   nvc_latent_norm_store   plain-weight RMS norms of the two low-rank latents of latent attention, the key / value
//                           latent scattered into the paged cache in the same pass
//   nvc_act_mul             gated / plain feed-forward activations (tanh-gelu gate, squared relu)
// Every kernel exists for bf16 and fp32 storage; arithmetic is fp32.
#include "typed.cuh"

namespace {

template <typename T>
__global__ void embed_gather_f32_kernel(const int32_t* ids, const T* __restrict__ table, int ldt,
                                        float* __restrict__ out, int ldo, int N, int H) {
  pdl_trigger();
  pdl_wait();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)N * H) return;
  const int n = (int)(i / H), j = (int)(i % H);
  out[(int64_t)n * ldo + j] = ld_f(table + (int64_t)ids[n] * ldt + j);
}

// one CTA per output row
template <typename T>
__global__ void dyt_norm_kernel(const float* res_in, const float* a0, const float* a1,
                                const float* a2, float* __restrict__ res_out, int ld, const float* __restrict__ w,
                                const float* __restrict__ b, const float* __restrict__ alpha, T* __restrict__ out, int ldo,
                                const int32_t* rows, int H) {
  pdl_trigger();
  const float al = w ? __ldg(alpha) : 0.f;
  pdl_wait();
  const int64_t src = rows ? rows[blockIdx.x] : blockIdx.x;
  for (int j = threadIdx.x; j < H; j += blockDim.x) {
    const int64_t k = src * ld + j;
    float s = res_in ? res_in[k] : 0.f;
    if (a0) s += a0[k];
    if (a1) s += a1[k];
    if (a2) s += a2[k];
    if (res_out) res_out[k] = s;
    if (w) st_f(out + (int64_t)blockIdx.x * ldo + j, tanh_f32(al * s) * __ldg(w + j) + __ldg(b + j));
  }
}

// one warp per row: segment 0 = columns [0, n0) -> out0; segment 1 = columns [off1, off1 + n1) -> the cache row of the slot
template <typename T>
__global__ void latent_norm_store_kernel(const float* in, int ldi, int n0, int off1, int n1,
                                         const float* __restrict__ w0, const float* __restrict__ w1, float eps,
                                         T* __restrict__ out0, int ld0, T* __restrict__ cache, int ldc,
                                         const int32_t* __restrict__ slots, int rot_dim, int rot_dims, int rot_half,
                                         const float* __restrict__ rot_table, const int32_t* __restrict__ positions, int N) {
  pdl_trigger();
  pdl_wait();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (row >= N) return;
  const float* x = in + (int64_t)row * ldi;
  float ss = 0.f;
  for (int j = lane; j < n0; j += 32) ss += x[j] * x[j];
  ss = warp_sum(ss);
  float r = 1.0f / sqrtf(ss / (float)n0 + eps);
  for (int j = lane; j < n0; j += 32) st_f(out0 + (int64_t)row * ld0 + j, x[j] * r * __ldg(w0 + j));
  const int slot = slots ? slots[row] : -1;
  if (slot < 0 || !cache) return;
  ss = 0.f;
  for (int j = lane; j < n1; j += 32) ss += x[off1 + j] * x[off1 + j];
  ss = warp_sum(ss);
  r = 1.0f / sqrtf(ss / (float)n1 + eps);
  for (int j = lane; j < n1; j += 32) st_f(cache + (int64_t)slot * ldc + j, x[off1 + j] * r * __ldg(w1 + j));
  // the key part that all heads share, behind the latent: turned by the token's position, not normed
  const float* kr = x + off1 + n1;
  const int half = rot_dims >> 1;
  const float2* tab = reinterpret_cast<const float2*>(rot_table) + (int64_t)(rot_dims ? positions[row] : 0) * half;
  for (int j = lane; j < rot_dim; j += 32) {
    float y = kr[j];
    if (j < rot_dims) {
      int i, partner;
      float sign;
      if (rot_half) { i = j < half ? j : j - half; partner = j < half ? j + half : j - half; sign = j < half ? -1.f : 1.f; }
      else { i = j >> 1; partner = j ^ 1; sign = (j & 1) ? 1.f : -1.f; }
      const float2 cs = __ldg(tab + i);
      y = y * cs.x + sign * kr[partner] * cs.y;
    }
    st_f(cache + (int64_t)slot * ldc + n1 + j, y);
  }
}

// four neighbouring numbers in the storage format
__device__ __forceinline__ void st_f4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void st_f4(__nv_bfloat16* p, const float4& v) { *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w)); }
__device__ __forceinline__ float4 scale4(const float4& x, float r, const float4& w) { return make_float4(x.x * r * w.x, x.y * r * w.y, x.z * r * w.z, x.w * r * w.w); }
__device__ __forceinline__ float dot4(const float4& x) { return x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w; }

// The same where the rows allow 16-byte accesses, n0 <= 128 V and latent and rotated part fit in 128 numbers: a warp requests all of its row at once, keeps
// it in registers, and finds weights, slot and angles (static operands) already there.  The general kernel reads the row twice, number by number, and the slot, the
// second part and the angles one behind the other: 64 rows of 512 + 96 + 32 took 4.5 us, here 2.1; 2 400 rows of 512 + 112 + 16 5.9, here 3.0 (calls in a row).
template <typename T, int V>
__global__ void __launch_bounds__(128) latent_norm_store_row_kernel(const float* in, int ldi, int n0, int off1, int n1, const float* __restrict__ w0,
                                                                    const float* __restrict__ w1, float eps, T* out0, int ld0, T* cache,
                                                                    int ldc, const int32_t* __restrict__ slots, int rot_dim, int rot_dims, int rot_half,
                                                                    const float* __restrict__ rot_table, const int32_t* __restrict__ positions, int N) {
  pdl_trigger();
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= N) return;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const int j = 4 * lane, jr = j - n1, half = rot_dims >> 1;          // this lane's numbers of the second part; of its rotated part
  const bool rotated = jr >= 0 && jr < rot_dims;
  // what no kernel of the step writes: weights, the slot, the angles
  float4 w[V], wl = zero, c0 = zero, c1 = zero;
#pragma unroll
  for (int v = 0; v < V; ++v) w[v] = j + 128 * v < n0 ? __ldg(reinterpret_cast<const float4*>(w0 + j + 128 * v)) : zero;
  const int slot = cache ? slots[row] : -1;
  if (cache) {
    if (j < n1) wl = __ldg(reinterpret_cast<const float4*>(w1 + j));
    if (rotated) {
      const float4* cs = reinterpret_cast<const float4*>(rot_table + (int64_t)positions[row] * rot_dims + (rot_half ? 2 * (jr < half ? jr : jr - half) : jr));
      c0 = __ldg(cs);
      if (rot_half) c1 = __ldg(cs + 1);
    }
  }
  pdl_wait();
  const float* x = in + (int64_t)row * ldi;
  float4 a[V], k = zero;
#pragma unroll
  for (int v = 0; v < V; ++v) a[v] = j + 128 * v < n0 ? *reinterpret_cast<const float4*>(x + j + 128 * v) : zero;
  if (slot >= 0 && j < n1 + rot_dim) k = *reinterpret_cast<const float4*>(x + off1 + j);
  float ss = 0.f;
#pragma unroll
  for (int v = 0; v < V; ++v) ss += dot4(a[v]);
  const float r0 = 1.0f / sqrtf(warp_sum(ss) / (float)n0 + eps);
#pragma unroll
  for (int v = 0; v < V; ++v)
    if (j + 128 * v < n0) st_f4(out0 + (int64_t)row * ld0 + j + 128 * v, scale4(a[v], r0, w[v]));
  if (slot < 0) return;
  const float r1 = 1.0f / sqrtf(warp_sum(j < n1 ? dot4(k) : 0.f) / (float)n1 + eps);
  // (i, i + half) by exchange, neighbouring pairs inside the lane
  const int from = lane + (jr < half ? half >> 2 : -(half >> 2));
  const float4 z = make_float4(__shfl_sync(0xffffffffu, k.x, from), __shfl_sync(0xffffffffu, k.y, from), __shfl_sync(0xffffffffu, k.z, from),
                               __shfl_sync(0xffffffffu, k.w, from));
  if (j < n1) {
    k = scale4(k, r1, wl);
  } else if (rotated) {
    if (rot_half) {
      const float s = jr < half ? -1.f : 1.f;
      k = make_float4(k.x * c0.x + s * z.x * c0.y, k.y * c0.z + s * z.y * c0.w, k.z * c1.x + s * z.z * c1.y, k.w * c1.z + s * z.w * c1.w);
    } else {
      k = make_float4(k.x * c0.x - k.y * c0.y, k.y * c0.x + k.x * c0.y, k.z * c0.z - k.w * c0.w, k.w * c0.z + k.z * c0.w);
    }
  }
  if (j < n1 + rot_dim) st_f4(cache + (int64_t)slot * ldc + j, k);
}

// NVC_ACT_GELU_TANH_MUL: out[n, j] = gelu_tanh(in[n, j]) * in[n, Fp + j];  NVC_ACT_RELU2: out[n, j] = relu(in[n, j])^2;
// NVC_ACT_SILU_MUL: silu(in[n, j]) * in[n, Fp + j];  NVC_ACT_GELU_TANH: gelu_tanh(in[n, j]);  NVC_ACT_GLU_CLAMP: g sigmoid(p1 g) (u + 1), g = min(in[n, j], p0), u = clamp(in[n, Fp + j], +-p0)
// T: what the result is stored as; the gates of a bf16 result take the hardware's exponential and reciprocal (typed.cuh; silu, 10 112 x 1 536, cold cache:
// 19.5 -> 14.4 us, 64 tokens' 2 176 rows 6.4 -> 5.2)
template <typename T>
__device__ __forceinline__ float act_unit(int kind, float g, float u, float p0, float p1) {
  if (kind == NVC_ACT_GELU_TANH_MUL) return gelu_tanh_f32(g) * u;
  if (kind == NVC_ACT_GELU_TANH) return gelu_tanh_f32(g);
  if (kind == NVC_ACT_SILU_MUL) return g * sigmoid_to<T>(g) * u;
  if (kind == NVC_ACT_GLU_CLAMP) {
    const float gc = fminf(g, p0);
    return gc * sigmoid_to<T>(p1 * gc) * (fminf(fmaxf(u, -p0), p0) + 1.0f);
  }
  const float t = fmaxf(g, 0.f);
  return t * t;
}

// rows_per_cta rows per CTA, the threads walk along a row: no division per element
template <typename T>
__global__ void act_mul_kernel(const T* in, int ldi, T* __restrict__ out, int ldo, int N, int F, int Fp, int kind, float p0,
                               float p1, int rows_per_cta) {
  pdl_trigger();
  pdl_wait();
  const bool two = kind == NVC_ACT_GELU_TANH_MUL || kind == NVC_ACT_GLU_CLAMP || kind == NVC_ACT_SILU_MUL;
  for (int rr = 0; rr < rows_per_cta; ++rr) {
    const int64_t n = (int64_t)blockIdx.x * rows_per_cta + rr;
    if (n >= N) return;
    const T* x = in + n * ldi;
    T* y = out + n * ldo;
    for (int j = threadIdx.x; j < F; j += blockDim.x) st_f(y + j, act_unit<T>(kind, ld_f(x + j), two ? ld_f(x + Fp + j) : 0.f, p0, p1));
  }
}

// The same 16 bytes at a time (every row start 16-byte aligned in both buffers, F and Fp multiples of the access).  A stream of 6 bytes per number; a thread
// requests its share of R rows before the first use of any, the CTA is as wide as the row (up to 512 accesses) and the kind of unit is fixed.  R = 4 where the
// rows fill the chip so (32 per SM; one pass per row: rows of two passes lost 4 % with R = 4), else 1.  Against a CTA of 64 to 256 threads per row that tests the
// kind per number, cold cache, gated units, bf16 rows x columns: 64 x 1 536: 2.0 -> 1.4 us; 512 x 3 072: 4.8 -> 3.8; 4 000 x 1 536: 9.5 -> 8.5; 10 048 x 1 536: 20.0 -> 17.2 gelu
// (5.4 TB/s), 20.7 -> 19.6 clamped; 8 192 x 64: 15.3 -> 4.7; 16 000 x 256: 11.6 -> 6.5; fp32 10 048 x 1 536: 32.8 -> 27.0; squared relu 10 048 x 1 536: 12.2 -> 8.8 (7.0 TB/s)
// `in` and `out` may be the same rows (one stride, the second halves behind the first ones): a number is written by the thread that has read it, and
// nobody else reads it.
template <typename T, int kKind, int R>
__global__ void __launch_bounds__(512) act_mul_rows_kernel(const T* in, int ldi, T* out, int ldo, int N, int F, int Fp, float p0, float p1) {
  pdl_trigger();
  pdl_wait();
  constexpr bool two = kKind == NVC_ACT_GELU_TANH_MUL || kKind == NVC_ACT_GLU_CLAMP || kKind == NVC_ACT_SILU_MUL;
  constexpr int PER = 16 / sizeof(T);                // numbers per 16-byte access
  const int64_t n0 = (int64_t)blockIdx.x * R;
  for (int j = threadIdx.x * PER; j < F; j += blockDim.x * PER) {
    __align__(16) T g[R][PER];
    __align__(16) T u[R][PER];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const T* x = in + (n0 + r < N ? n0 + r : n0) * ldi + j;
      *reinterpret_cast<uint4*>(g[r]) = *reinterpret_cast<const uint4*>(x);
      if constexpr (two) *reinterpret_cast<uint4*>(u[r]) = *reinterpret_cast<const uint4*>(x + Fp);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      __align__(16) T o[PER];
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        float f = 0.f;
        if constexpr (two) f = ld_f(u[r] + k);
        st_f(o + k, act_unit<T>(kKind, ld_f(g[r] + k), f, p0, p1));
      }
      if (n0 + r < N) *reinterpret_cast<uint4*>(out + (n0 + r) * ldo + j) = *reinterpret_cast<const uint4*>(o);
    }
  }
}

template <typename T, int kKind>
cudaError_t launch_act_mul_rows(nvc_ctx* ctx, cudaStream_t st, const T* in, int ldi, T* out, int ldo, int N, int F, int Fp, float p0, float p1) {
  const int lanes = F / (int)(16 / sizeof(T)), passes = (lanes + 511) / 512;
  const int threads = ((lanes + passes - 1) / passes + 31) & ~31;
  // narrow rows from half of that on: a CTA of one warp per row is bound by the rate at which CTAs start (fp32 4 000 x 100: 4.5 us, so 1.9)
  if (passes == 1 && N >= (lanes <= 32 ? 16 : 32) * ctx->num_sms)
    return nvc_launch(ctx, act_mul_rows_kernel<T, kKind, 4>, dim3((unsigned)(((int64_t)N + 3) / 4)), dim3(threads), 0, st, in, ldi, out, ldo, N, F, Fp, p0, p1);
  return nvc_launch(ctx, act_mul_rows_kernel<T, kKind, 1>, dim3((unsigned)N), dim3(threads), 0, st, in, ldi, out, ldo, N, F, Fp, p0, p1);
}

}  // namespace

extern "C" {

int nvc_embed_gather_f32(nvc_ctx* ctx, const int32_t* ids, const void* table, int table_dtype, int ldt, float* out, int ldo,
                         int N, int H, void* stream) {
  NVC_REQUIRE(ctx, ctx && ids && table && out, NVC_EINVAL, "null pointer");
  NVC_REQUIRE(ctx, N >= 0 && H > 0 && ldt >= H && ldo >= H, NVC_EINVAL, "bad sizes");
  if (N == 0) return NVC_OK;
  const int64_t total = (int64_t)N * H;
  NVC_DISPATCH_DT(table_dtype, T,
                  NVC_CUDA_CHECK(ctx, nvc_launch(ctx, embed_gather_f32_kernel<T>, dim3((unsigned)((total + 255) / 256)), dim3(256), 0,
                                                 nvc_stream(stream), ids, reinterpret_cast<const T*>(table), ldt, out, ldo, N, H)));
  ctx->launches++;
  return NVC_OK;
}

int nvc_dyt_norm(nvc_ctx* ctx, const float* res_in, const float* a0, const float* a1, const float* a2, float* res_out, int ld,
                 const float* w, const float* b, const float* alpha, void* out, int out_dtype, int ldo, const int32_t* rows,
                 int N, int H, void* stream) {
  NVC_REQUIRE(ctx, ctx && (res_in || a0), NVC_EINVAL, "null pointer");
  NVC_REQUIRE(ctx, (w == nullptr) == (out == nullptr) && (!w || (b && alpha)), NVC_EINVAL, "norm needs weight, bias, alpha and an output");
  NVC_REQUIRE(ctx, N >= 0 && H > 0 && ld >= H && (!w || ldo >= H), NVC_EINVAL, "bad sizes");
  NVC_REQUIRE(ctx, !(rows && res_out), NVC_EINVAL, "a gathering call does not write the residual back");
  if (N == 0) return NVC_OK;
  const int threads = H >= 1024 ? 512 : (H >= 256 ? 256 : 128);
  NVC_DISPATCH_DT(out_dtype, T,
                  NVC_CUDA_CHECK(ctx, nvc_launch(ctx, dyt_norm_kernel<T>, dim3(N), dim3(threads), 0, nvc_stream(stream), res_in, a0, a1, a2,
                                                 res_out, ld, w, b, alpha, reinterpret_cast<T*>(out), ldo, rows, H)));
  ctx->launches++;
  return NVC_OK;
}

int nvc_latent_norm_store(nvc_ctx* ctx, const float* in, int ldi, int n0, int off1, int n1, const float* w0, const float* w1,
                          float eps, void* out0, int ld0, void* cache, int ldc, const int32_t* slot_mapping, int dtype, int N,
                          void* stream) {
  return nvc_latent_norm_store_rot(ctx, in, ldi, n0, off1, n1, w0, w1, eps, out0, ld0, cache, ldc, slot_mapping, 0, 0, 0, nullptr, nullptr,
                                   dtype, N, stream);
}

int nvc_latent_norm_store_rot(nvc_ctx* ctx, const float* in, int ldi, int n0, int off1, int n1, const float* w0, const float* w1,
                              float eps, void* out0, int ld0, void* cache, int ldc, const int32_t* slot_mapping, int rot_dim,
                              int rot_dims, int rot_half, const float* rot_table, const int32_t* positions, int dtype, int N,
                              void* stream) {
  NVC_REQUIRE(ctx, ctx && in && w0 && out0, NVC_EINVAL, "null pointer");
  NVC_REQUIRE(ctx, rot_dim >= 0 && rot_dims >= 0 && rot_dims % 2 == 0 && rot_dims <= rot_dim && (rot_dims == 0 || (rot_table && positions)),
              NVC_EINVAL, "bad rotary arguments");
  if (!cache) rot_dim = rot_dims = 0;
  NVC_REQUIRE(ctx, !cache || (w1 && slot_mapping), NVC_EINVAL, "a cache needs its norm weight and the slot mapping");
  NVC_REQUIRE(ctx, N >= 0 && n0 > 0 && n1 >= 0 && off1 >= n0 && ldi >= off1 + n1 + rot_dim && ld0 >= n0 && (!cache || ldc >= n1 + rot_dim),
              NVC_EINVAL, "bad sizes");
  if (N == 0) return NVC_OK;
  auto al16 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
  const bool vec = n0 <= 1024 && ((n0 | off1 | n1 | rot_dim | rot_dims | ldi | ld0 | ldc) & 3) == 0 && (!rot_half || rot_dims % 8 == 0) && al16(in) && al16(w0) &&
                   al16(out0) && (!cache || (n1 > 0 && n1 + rot_dim <= 128 && al16(w1) && al16(cache) && (rot_dims == 0 || al16(rot_table))));
  if (vec) {
    NVC_DISPATCH_DT(dtype, T,
                    NVC_CUDA_CHECK(ctx, nvc_launch(ctx, n0 <= 512 ? latent_norm_store_row_kernel<T, 4> : latent_norm_store_row_kernel<T, 8>, dim3((N + 3) / 4), dim3(128), 0,
                                                   nvc_stream(stream), in, ldi, n0, off1, n1, w0, w1, eps, reinterpret_cast<T*>(out0), ld0,
                                                   reinterpret_cast<T*>(cache), ldc, slot_mapping, rot_dim, rot_dims, rot_half, rot_table, positions, N)));
    ctx->launches++;
    return NVC_OK;
  }
  NVC_DISPATCH_DT(dtype, T,
                  NVC_CUDA_CHECK(ctx, nvc_launch(ctx, latent_norm_store_kernel<T>, dim3((N + 3) / 4), dim3(128), 0, nvc_stream(stream), in,
                                                 ldi, n0, off1, n1, w0, w1, eps, reinterpret_cast<T*>(out0), ld0,
                                                 reinterpret_cast<T*>(cache), ldc, slot_mapping, rot_dim, rot_dims, rot_half, rot_table,
                                                 positions, N)));
  ctx->launches++;
  return NVC_OK;
}

int nvc_act_mul(nvc_ctx* ctx, const void* in, int ldi, void* out, int ldo, int dtype, int N, int F, int Fp, int kind, void* stream) {
  NVC_REQUIRE(ctx, kind == NVC_ACT_GELU_TANH_MUL || kind == NVC_ACT_RELU2, NVC_EINVAL, "bad arguments");
  return nvc_act_mul_p(ctx, in, ldi, out, ldo, dtype, N, F, Fp, kind, 0.f, 0.f, stream);
}

int nvc_act_mul_p(nvc_ctx* ctx, const void* in, int ldi, void* out, int ldo, int dtype, int N, int F, int Fp, int kind, float p0, float p1,
                  void* stream) {
  NVC_REQUIRE(ctx, ctx && in && out, NVC_EINVAL, "null pointer");
  const bool two = kind == NVC_ACT_GELU_TANH_MUL || kind == NVC_ACT_GLU_CLAMP || kind == NVC_ACT_SILU_MUL;
  NVC_REQUIRE(ctx, N >= 0 && F > 0 && (two || kind == NVC_ACT_RELU2 || kind == NVC_ACT_GELU_TANH), NVC_EINVAL, "bad arguments");
  NVC_REQUIRE(ctx, ldo >= F && ldi >= (two ? Fp + F : F), NVC_EINVAL, "bad strides");
  // with other strides, or halves that overlap, a CTA would write what another one (a thread, what another one) still has to read
  NVC_REQUIRE(ctx, in != out || ((ldi == ldo || N <= 1) && (!two || Fp >= F)), NVC_EINVAL, "in place: one row stride, and the second half behind the first");
  if (N == 0) return NVC_OK;
  const int per = dtype == NVC_DT_F32 ? 4 : 8;
  const bool vec = F % per == 0 && Fp % per == 0 && ldi % per == 0 && ldo % per == 0 && (reinterpret_cast<uintptr_t>(in) & 15) == 0 &&
                   (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  cudaStream_t st = nvc_stream(stream);
  NVC_DISPATCH_DT(dtype, T, {
    const T* x = reinterpret_cast<const T*>(in);
    T* y = reinterpret_cast<T*>(out);
    cudaError_t e;
    if (!vec) {
      const int threads = F >= 256 ? 256 : (F >= 128 ? 128 : 64);
      const int rows_per_cta = F >= 64 ? 1 : 64 / F;
      e = nvc_launch(ctx, act_mul_kernel<T>, dim3((unsigned)((N + rows_per_cta - 1) / rows_per_cta)), dim3(threads), 0, st, x, ldi, y, ldo, N, F, Fp, kind, p0, p1,
                     rows_per_cta);
    } else if (kind == NVC_ACT_GELU_TANH_MUL) {
      e = launch_act_mul_rows<T, NVC_ACT_GELU_TANH_MUL>(ctx, st, x, ldi, y, ldo, N, F, Fp, p0, p1);
    } else if (kind == NVC_ACT_RELU2) {
      e = launch_act_mul_rows<T, NVC_ACT_RELU2>(ctx, st, x, ldi, y, ldo, N, F, Fp, p0, p1);
    } else if (kind == NVC_ACT_SILU_MUL) {
      e = launch_act_mul_rows<T, NVC_ACT_SILU_MUL>(ctx, st, x, ldi, y, ldo, N, F, Fp, p0, p1);
    } else if (kind == NVC_ACT_GELU_TANH) {
      e = launch_act_mul_rows<T, NVC_ACT_GELU_TANH>(ctx, st, x, ldi, y, ldo, N, F, Fp, p0, p1);
    } else {
      e = launch_act_mul_rows<T, NVC_ACT_GLU_CLAMP>(ctx, st, x, ldi, y, ldo, N, F, Fp, p0, p1);
    }
    NVC_CUDA_CHECK(ctx, e);
  });
  ctx->launches++;
  return NVC_OK;
}

}  // extern "C"
