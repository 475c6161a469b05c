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

// x sigmoid(x) of every convolution here, rows of a decode step and tiles of a prompt alike, without a division's branch and range checks, which are most of a convolved number's
// instructions: with t = exp(-|x|) the sigmoid is 1 / (1 + t) or t / (1 + t), its divisor lies in [1, 2], and one Newton step on the hardware's reciprocal (off by one unit in the last
// place at most) and one on the quotient correct it (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990); what 1 + t rounds away takes part in
// the second.  Infinities and NaN come out as those of x / (1 + exp(-x)).  Error at most 4 units of 2^-23 and a step of 2^-149 times |x|, as tested: below -87.34 the exponential is
// subnormal and rounded to such a step (by x / (1 + exp(-x)) everything below -88.72 is 0; a scaled exponential there would cost what the missing division gains, 4.8 us a layer).
// Against 64 bits, relative 2-norm, that division / this: x from N(0, 1) 4.54e-8 / 3.49e-8, from N(0, 1e-8) 5.0e-8 / 3.9e-8.  4 480 rows of 4 096 channels 46.2 -> 42.2 us, of 2 560 31.5 -> 28.6.
__device__ __forceinline__ float silu_f32(float x) {
  const float t = expf(-fabsf(x)), d = 1.0f + t, rest = t - (d - 1.0f), a = x < 0.f ? t : 1.0f;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(fmaf(-d, r, 1.0f), r, r);
  const float q = a * r;
  return x * fmaf(fmaf(-rest, q, fmaf(-d, q, a)), r, q);
}
__device__ __forceinline__ float4 silu4(const float4& a) { return make_float4(silu_f32(a.x), silu_f32(a.y), silu_f32(a.z), silu_f32(a.w)); }

}  // namespace
