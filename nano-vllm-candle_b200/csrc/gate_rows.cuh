// The output stage of a mixer in groups of up to 1 024 columns, 16-byte accesses: y = x / rms(x) * out_scale * w * gate(z), or with the gate in front
// of the norm.  Included by norm_rms.cu (heads) and norm_blend.cu (groups).
//
// The stage moves 10 bytes per number (x, z, the bf16 result) and is bound by them.  One unit (row, group) per warp that reads x, reduces, reads x again
// and then z keeps 0.5 - 1 KB per warp on the way and pays three latencies and two 64-bit divisions per unit; a CTA per unit adds its barriers.  Here W lanes
// request x AND z of L units before their first use of either, four 16-byte accesses of each per lane (V per unit, V L = 4; V = 8 from 513 columns on),
// and divide once, in 32 bits.  Grids that do not fill the chip with that (under 64 units per SM) take one unit per W lanes, for the latency's sake.
// silu gate, cold cache, a warp per unit (head) | a CTA per unit (group) -> here, us:
//   rows x groups x columns   8 x 16 x 128: 1.9 | 1.9 -> 1.7     64 x 16 x 128: 2.2 | 2.5 -> 2.0      1 000 x 16 x 128: 7.9 | 18.6 -> 7.9
//   4 480 x 16 x 128: 27.9 | 76 -> 21.0 (4.4 TB/s; the sigmoid's exponential and division share the time)      4 480 x 16 x 64: 26.6 | 76 -> 11.9
//   4 480 x 4 x 512: 21.0 | 41 -> 17.0 (5.4 TB/s)    4 480 x 2 x 1 024: 23.9 | 27.4 -> 20.7     16 000 x 4 x 512: 66 | 143 -> 52 (6.3 TB/s)
#pragma once
#include "typed.cuh"

namespace {

__device__ __forceinline__ void gate_store(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void gate_store(__nv_bfloat16* p, const float4& v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

// w: gsize numbers per group, wstride apart (0: the same for every group).  gsize is a multiple of 4 and at most 4 W V.
// W lanes per unit.
template <typename T, int W, int V, int L>
__global__ void __launch_bounds__(128) gate_rows_kernel(const float* o, int ldo, const float* g, int ldg, const float* __restrict__ w,
                                                        int wstride, T* out, int ldout, int groups, int gsize, int norm, int gate_first, float eps,
                                                        int act, float out_scale, uint32_t units) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x % W, v4 = gsize >> 2;
  const uint32_t u0 = (blockIdx.x * (128 / W) + threadIdx.x / W) * L;
  uint32_t n = min(u0, units - 1) / (uint32_t)groups, k = min(u0, units - 1) - n * groups;
  const uint32_t n0 = n, k0 = k;
  auto gated = [&](float4 v, const float4& z) {
    if (act == NVC_GATE_SILU) { v.x *= z.x * sigmoid_to<T>(z.x); v.y *= z.y * sigmoid_to<T>(z.y); v.z *= z.z * sigmoid_to<T>(z.z); v.w *= z.w * sigmoid_to<T>(z.w); }
    else { v.x *= sigmoid_to<T>(z.x); v.y *= sigmoid_to<T>(z.y); v.z *= sigmoid_to<T>(z.z); v.w *= sigmoid_to<T>(z.w); }
    return v;
  };
  float4 x[L][V], z[L][V];
#pragma unroll
  for (int i = 0; i < L; ++i) {
    const float* po = o + (int64_t)n * ldo + k * gsize;
    const float* pz = g + (int64_t)n * ldg + k * gsize;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int j = lane + W * v;
      x[i][v] = j < v4 ? *reinterpret_cast<const float4*>(po + 4 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
      if (g) z[i][v] = j < v4 ? *reinterpret_cast<const float4*>(pz + 4 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (u0 + i + 1 < units && ++k == (uint32_t)groups) { k = 0; ++n; }         // past the end: the last unit again
  }
  n = n0;
  k = k0;
  float r[L];
#pragma unroll
  for (int i = 0; i < L; ++i) {
    float ss = 0.f;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      if (g && gate_first) x[i][v] = gated(x[i][v], z[i][v]);
      const float4 a = x[i][v];
      ss += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
    }
    r[i] = out_scale;
    if (norm) {
#pragma unroll
      for (int w = W / 2; w > 0; w >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, w);
      r[i] *= 1.0f / sqrtf(ss / (float)gsize + eps);
    }
  }
#pragma unroll
  for (int i = 0; i < L; ++i) {
    if (u0 + i >= units) return;
    T* const dst = out + (int64_t)n * ldout + k * gsize;
    const float* const pw = w ? w + k * wstride : nullptr;
#pragma unroll
    for (int v = 0; v < V; ++v) {
      const int j = lane + W * v;
      if (j >= v4) break;
      float4 a = x[i][v];
      a.x *= r[i]; a.y *= r[i]; a.z *= r[i]; a.w *= r[i];
      if (pw) {
        const float4 c = *reinterpret_cast<const float4*>(pw + 4 * j);
        a.x *= c.x; a.y *= c.y; a.z *= c.z; a.w *= c.w;
      }
      if (g && !gate_first) a = gated(a, z[i][v]);
      gate_store(dst + 4 * j, a);
    }
    if (++k == (uint32_t)groups) { k = 0; ++n; }
  }
}

template <typename T>
cudaError_t launch_gate_rows(nvc_ctx* ctx, cudaStream_t st, const float* o, int ldo, const float* g, int ldg, const float* w, int wstride, T* out, int ldout,
                             int groups, int gsize, int norm, int gate_first, float eps, int act, float out_scale, int N) {
  const uint32_t units = (uint32_t)N * groups;
  const bool full = units >= 64u * ctx->num_sms;
  auto run = [&](auto kernel, uint32_t per_cta) {
    return nvc_launch(ctx, kernel, dim3((units + per_cta - 1) / per_cta), dim3(128), 0, st, o, ldo, g, ldg, w, wstride, out, ldout, groups, gsize, norm,
                      gate_first, eps, act, out_scale, units);
  };
  if (gsize <= 64) return full ? run(gate_rows_kernel<T, 16, 1, 4>, 32) : run(gate_rows_kernel<T, 16, 1, 1>, 8);
  if (gsize <= 128) return full ? run(gate_rows_kernel<T, 32, 1, 4>, 16) : run(gate_rows_kernel<T, 32, 1, 1>, 4);
  if (gsize <= 256) return full ? run(gate_rows_kernel<T, 32, 2, 2>, 8) : run(gate_rows_kernel<T, 32, 2, 1>, 4);
  if (gsize <= 512) return run(gate_rows_kernel<T, 32, 4, 1>, 4);
  return run(gate_rows_kernel<T, 32, 8, 1>, 4);
}

}  // namespace
