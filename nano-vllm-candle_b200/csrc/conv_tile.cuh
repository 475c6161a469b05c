// A short causal convolution over time for a tile of neighbouring rows, four channels per lane (delta_rule.cu, ssd_prep.cu): the taps slide along
// the rows in registers, so a projection row is read once - and not once per tap - and a tile's loads are in flight together.
#pragma once
#include "typed.cuh"

namespace {

// The sequence of a row, found by the whole warp (cu: first rows of B sequences and the end; rows behind empty sequences belong to the last of
// their first rows).
struct RowSeq {
  int b, r0, r1;
  bool fresh;         // the portion starts at position 0
  int slot;
  __device__ __forceinline__ void set(const int32_t* cu, const int32_t* slots, const int32_t* positions) {
    r0 = cu[b];
    r1 = cu[b + 1];
    fresh = positions[r0] == 0;
    slot = slots[b];
  }
  __device__ __forceinline__ void find(const int32_t* cu, const int32_t* slots, const int32_t* positions, int B, int n, int lane) {
    b = 0;
    for (int i = 1; i < B; i += 32) b += __popc(__ballot_sync(0xffffffffu, i + lane < B && cu[i + lane] <= n));
    set(cu, slots, positions);
  }
  __device__ __forceinline__ void next(const int32_t* cu, const int32_t* slots, const int32_t* positions, int B, int n) {
    while (b + 1 < B && cu[b + 1] <= n) ++b;
    set(cu, slots, positions);
  }
};

// y[i] = bias + sum_j w[j] x_(n0 + i - TAPS + 1 + j) for rows n0 .. n0 + cnt - 1 of four channels: in, state and w point at the first of them.  All
// lanes of the warp call it; `on`: this lane has channels.
template <int TAPS, int TT>
__device__ __forceinline__ void conv_tile(float4 (&y)[TT], const float* in, int64_t ldi, const float* state, int C, const float* w, const float4& bias,
                                          const int32_t* cu, const int32_t* slots, const int32_t* positions, int B, int n0, int cnt, bool on, int lane) {
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < TT; ++i) y[i] = on && i < cnt ? *reinterpret_cast<const float4*>(in + (int64_t)(n0 + i) * ldi) : zero;
  float4 wt[TAPS], h[TAPS];
#pragma unroll
  for (int i = 0; i < TAPS; ++i) wt[i] = on ? __ldg(reinterpret_cast<const float4*>(w + (int64_t)i * C)) : zero;
  RowSeq s;
  s.find(cu, slots, positions, B, n0, lane);
  auto history = [&](int n) {
#pragma unroll
    for (int k = 0; k + 1 < TAPS; ++k) {
      const int src = n - (TAPS - 1) + k;
      h[k] = zero;
      if (on && src >= s.r0) h[k] = *reinterpret_cast<const float4*>(in + (int64_t)src * ldi);
      else if (on && !s.fresh) h[k] = *reinterpret_cast<const float4*>(state + ((int64_t)s.slot * (TAPS - 1) + (src - s.r0 + TAPS - 1)) * C);
    }
  };
  history(n0);
#pragma unroll
  for (int i = 0; i < TT; ++i) {
    if (i < cnt) {
      if (n0 + i >= s.r1) {
        s.next(cu, slots, positions, B, n0 + i);
        history(n0 + i);
      }
      h[TAPS - 1] = y[i];
      float4 a = bias;
#pragma unroll
      for (int k = 0; k < TAPS; ++k) {
        a.x = fmaf(wt[k].x, h[k].x, a.x);
        a.y = fmaf(wt[k].y, h[k].y, a.y);
        a.z = fmaf(wt[k].z, h[k].z, a.z);
        a.w = fmaf(wt[k].w, h[k].w, a.w);
      }
      y[i] = a;
#pragma unroll
      for (int k = 0; k + 1 < TAPS; ++k) h[k] = h[k + 1];
    }
  }
}

__device__ __forceinline__ float4 silu4(const float4& a) {
  return make_float4(a.x * sigmoid_f32(a.x), a.y * sigmoid_f32(a.y), a.z * sigmoid_f32(a.z), a.w * sigmoid_f32(a.w));
}

}  // namespace
