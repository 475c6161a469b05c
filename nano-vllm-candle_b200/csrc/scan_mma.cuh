// Products of fp32 numbers on the tensor pipe for the chunked recurrences (retention.cu, delta_rule.cu).
//
// An fp32 number is the exact sum of three bf16 numbers (8 + 8 + 8 bits: high, middle, low), and a product of two numbers is the sum of nine
// products of parts.  The six largest are taken (mma.sync m16n8k16, exact products, fp32 sums); the three that are left out are below
// 2^-24 of the whole.  The pipe's own sums round towards zero, so no more than 64 terms of high parts share an accumulator before an
// ordinary fp32 add takes over, and the five small products are summed apart from them, or in front of them (the observation and the
// remedy are Ootomo and Yokota's, "Recovering single precision accuracy from Tensor Cores", 2022).
// Measured against 64 bits, relative error of sums of 64 products of normal numbers: 7.0e-8, a chain of 64 fp32 FMAs 1.45e-7; of
// positive numbers 8.9e-8 and 1.2e-7.  Rate: 555 TFLOP/s of bf16 products, so 92 of fp32 ones, against 72 of the FMA pipe - and
// without its operands' way through shared memory and issue slots, which is what bound the FMA form of the recurrences.
#pragma once
#include "scan_common.cuh"

namespace {

struct FragA { uint32_t r[3][4]; };        // a 16 x 16 operand in its three parts
struct FragB { uint32_t r[3][2]; };        // a 16 x 8 operand

// the three parts of two numbers, two bf16 to a register
__device__ __forceinline__ void split_pair(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& low) {
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(y), "f"(x));
  x -= __uint_as_float(hi << 16);
  y -= __uint_as_float(hi & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(mid) : "f"(y), "f"(x));
  x -= __uint_as_float(mid << 16);
  y -= __uint_as_float(mid & 0xffff0000u);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(low) : "f"(y), "f"(x));
}
// two neighbouring 16 x 8 accumulator tiles as the left operand of the next product (the register layouts agree)
__device__ __forceinline__ void frag_of_tiles(FragA& a, const float (&t0)[4], const float (&t1)[4]) {
  split_pair(t0[0], t0[1], a.r[0][0], a.r[1][0], a.r[2][0]);
  split_pair(t0[2], t0[3], a.r[0][1], a.r[1][1], a.r[2][1]);
  split_pair(t1[0], t1[1], a.r[0][2], a.r[1][2], a.r[2][2]);
  split_pair(t1[2], t1[3], a.r[0][3], a.r[1][3], a.r[2][3]);
}
__device__ __forceinline__ void mma_bf16_acc(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// The five small products of a b[t], and the large one.  One part after the other over all tiles: a chain of products on one accumulator
// advances every 20 cycles, the pipe takes one every 8.
template <int NT>
__device__ __forceinline__ void mma_small(float (&acc)[NT][4], const FragA& a, const FragB (&b)[NT]) {
  constexpr int pa[5] = {2, 0, 1, 1, 0}, pb[5] = {0, 2, 1, 0, 1};
#pragma unroll
  for (int i = 0; i < 5; ++i)
#pragma unroll
    for (int t = 0; t < NT; ++t) mma_bf16_acc(acc[t], a.r[pa[i]], b[t].r[pb[i]]);
}
template <int NT>
__device__ __forceinline__ void mma_high(float (&acc)[NT][4], const FragA& a, const FragB (&b)[NT]) {
#pragma unroll
  for (int t = 0; t < NT; ++t) mma_bf16_acc(acc[t], a.r[0], b[t].r[0]);
}

__device__ __forceinline__ void ldsm4(uint32_t& x, uint32_t& y, uint32_t& z, uint32_t& w, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(addr));
}
__device__ __forceinline__ void ldsm4_t(uint32_t& x, uint32_t& y, uint32_t& z, uint32_t& w, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(addr));
}

// (Planes are written and read by volatile asm alone, which keeps its order, barriers included: no memory clobbers.)
// Matrices in shared memory are kept as three planes of bf16 parts, `rows` rows of `ld` numbers each (ld = a multiple of 16 plus 8, so that the
// eight rows of an 8 x 8 block fall into different banks).
struct Planes {
  uint32_t base;      // shared address
  int ld, plane;      // numbers per row, bytes per plane
  __device__ __forceinline__ uint32_t at(int r, int c) const { return base + (uint32_t)(r * ld + c) * 2u; }
};
__device__ __forceinline__ Planes planes(const void* p, int rows, int ld) {
  return Planes{(uint32_t)__cvta_generic_to_shared(p), ld, rows * ld * 2};
}
// rows r0 .. r0 + 15, columns c0 .. c0 + 15 as the left operand
__device__ __forceinline__ void load_a(FragA& a, const Planes& m, int r0, int c0, int lane) {
  const uint32_t p = m.at(r0 + (lane & 15), c0 + (lane >> 4) * 8);
#pragma unroll
  for (int i = 0; i < 3; ++i) ldsm4(a.r[i][0], a.r[i][1], a.r[i][2], a.r[i][3], p + i * m.plane);
}
// the matrix holds the right operand's columns as rows: rows n0 .. n0 + 15 (two operands of eight columns), columns k0 .. k0 + 15
__device__ __forceinline__ void load_b2(FragB& x, FragB& y, const Planes& m, int n0, int k0, int lane) {
  const uint32_t p = m.at(n0 + (lane & 7) + ((lane >> 4) << 3), k0 + ((lane >> 3) & 1) * 8);
#pragma unroll
  for (int i = 0; i < 3; ++i) ldsm4(x.r[i][0], x.r[i][1], y.r[i][0], y.r[i][1], p + i * m.plane);
}
// the matrix holds the right operand as it is: rows k0 .. k0 + 15, columns n0 .. n0 + 15
__device__ __forceinline__ void load_b2_t(FragB& x, FragB& y, const Planes& m, int k0, int n0, int lane) {
  const uint32_t p = m.at(k0 + (lane & 7) + ((lane >> 3) & 1) * 8, n0 + (lane >> 4) * 8);
#pragma unroll
  for (int i = 0; i < 3; ++i) ldsm4_t(x.r[i][0], x.r[i][1], y.r[i][0], y.r[i][1], p + i * m.plane);
}
// NT operands of eight columns side by side (NT even)
template <int NT>
__device__ __forceinline__ void load_b(FragB (&x)[NT], const Planes& m, int n0, int k0, int lane) {
#pragma unroll
  for (int t = 0; t < NT; t += 2) load_b2(x[t], x[t + 1], m, n0 + 8 * t, k0, lane);
}
template <int NT>
__device__ __forceinline__ void load_b_t(FragB (&x)[NT], const Planes& m, int k0, int n0, int lane) {
#pragma unroll
  for (int t = 0; t < NT; t += 2) load_b2_t(x[t], x[t + 1], m, k0, n0 + 8 * t, lane);
}
// two neighbouring numbers of a row into the planes
__device__ __forceinline__ void store_pair(const Planes& m, int r, int c, float x, float y) {
  uint32_t v[3];
  split_pair(x, y, v[0], v[1], v[2]);
#pragma unroll
  for (int i = 0; i < 3; ++i) asm volatile("st.shared.b32 [%0], %1;" ::"r"(m.at(r, c) + i * m.plane), "r"(v[i]));
}
// four neighbouring numbers (c a multiple of 4)
__device__ __forceinline__ void store_quad(const Planes& m, int r, int c, const float4& x) {
  uint32_t u[3], v[3];
  split_pair(x.x, x.y, u[0], u[1], u[2]);
  split_pair(x.z, x.w, v[0], v[1], v[2]);
#pragma unroll
  for (int i = 0; i < 3; ++i) asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(m.at(r, c) + i * m.plane), "r"(u[i]), "r"(v[i]));
}
constexpr int kMT = 32;                 // tokens per chunk
constexpr int kMC = 64;                 // value columns per CTA: 16 for each of its four state warps
constexpr int kMV = kMC + 4;            // row stride of staged values
constexpr int kMP = kMT + 8;            // row stride of the token-by-token planes

// What the chunked recurrences on the tensor pipe have in common.  One CTA of eight warps per (sequence, head, 64 value columns), one CTA per SM:
//   warps 4 .. 7  prepare the chunks of 32 tokens, up to two ahead: rows from global memory into bf16 planes in shared memory, decays, the
//                 token-by-token products
//   warps 0 .. 3  carry the state, 16 value columns each.  It is kept TRANSPOSED in the warp's accumulator registers (16 columns x all channels: 64
//                 numbers per thread at 128 channels), where it is at once the left operand of its products with the chunk's rows and
//                 the accumulator of its own update: it never travels, and a state warp waits for nobody but the preparing ones.
// The chain of a sequence's chunks is what takes the time, and it holds only what depends on the state.  (The same products by eight warps that
// do everything in turn, two CTAs per SM: bound by latency, 500 us for the delta rule over eight prompts of 245 to 1 050 tokens, 16 heads of
// 128 x 128, where this takes 266.)
enum { kFull = 1, kEmpty = 3, kPrepare = 5 };                 // named barriers: a buffer of a chunk is filled / free (two each); the preparing warps
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// four neighbouring numbers of a row of `dim` (zeros behind it, or everywhere)
__device__ __forceinline__ float4 load_quad(const float* row, int c, int dim, bool in, bool vec) {
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  if (in && c < dim) {
    if (vec) return *reinterpret_cast<const float4*>(row + c);
    x.x = row[c];
    if (c + 1 < dim) x.y = row[c + 1];
    if (c + 2 < dim) x.z = row[c + 2];
    if (c + 3 < dim) x.w = row[c + 3];
  }
  return x;
}
// 32 rows of up to DZ (a multiple of 16, up to 128) numbers by four warps, in registers between global and shared memory
template <int DZ>
struct RowTile {
  static constexpr int kLanes = DZ / 4, kRows = 32 / kLanes, kPasses = 8 / kRows;
  float4 x[kPasses];
  __device__ __forceinline__ static int row(int i, int pw, int lane) { return (4 * i + pw) * kRows + lane / kLanes; }
  __device__ __forceinline__ void load(const float* src, int64_t ld, int dim, int n, bool vec, int pw, int lane) {
#pragma unroll
    for (int i = 0; i < kPasses; ++i) {
      const int r = row(i, pw, lane);
      x[i] = load_quad(src + r * ld, 4 * (lane % kLanes), dim, r < n, vec);
    }
  }
  __device__ __forceinline__ void split_to(const Planes& m, int pw, int lane) const {
#pragma unroll
    for (int i = 0; i < kPasses; ++i) store_quad(m, row(i, pw, lane), 4 * (lane % kLanes), x[i]);
  }
  __device__ __forceinline__ void store_to(float* dst, int ld, int pw, int lane) const {
#pragma unroll
    for (int i = 0; i < kPasses; ++i) *reinterpret_cast<float4*>(dst + row(i, pw, lane) * ld + 4 * (lane % kLanes)) = x[i];
  }
};

// The sequence of a block when the longest are to start first (one wave of CTAs rarely holds them all): the one with `rank` longer ones.
// Sequences beyond 256 keep their order.
__device__ __forceinline__ int sequence_of_rank(const int32_t* cu, int B, int rank, int* found) {
  if (B > 256 || B == 1) return rank;
  for (int i = threadIdx.x; i < B; i += blockDim.x) {
    const int len = cu[i + 1] - cu[i];
    int longer = 0;
    for (int j = 0; j < B; ++j) {
      const int l = cu[j + 1] - cu[j];
      longer += l > len || (l == len && j < i);
    }
    if (longer == rank) *found = i;
  }
  __syncthreads();
  return *found;
}

// Token-by-token products: rows x0 .. x0 + 15 of X against rows y0 .. y0 + 15 of Y, two tiles of eight columns; KS blocks of 16 channels,
// alternately with sums of their own (at most 64 terms each)
template <int KS>
__device__ __forceinline__ void token_products(float (&out)[2][4], const Planes& X, int x0, const Planes& Y, int y0, int lane) {
  float x[2][2][4] = {}, rest[2][2][4] = {};
#pragma unroll 2
  for (int ks = 0; ks < KS; ks += 2) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      FragA a;
      FragB b[2];
      load_a(a, X, x0, (ks + p) * 16, lane);
      load_b(b, Y, y0, (ks + p) * 16, lane);
      mma_high(x[p], a, b);
      mma_small(rest[p], a, b);
    }
  }
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) out[t][i] = (x[0][t][i] + x[1][t][i]) + (rest[0][t][i] + rest[1][t][i]);
}

// The state of a warp: tile i holds channels 8 i + 2 tq (+ 1), columns g (0, 1) and g + 8 (2, 3) of the warp's 16 (g = lane / 4, tq = lane % 4)
template <int KS>
__device__ __forceinline__ void load_state(float (&S)[2 * KS][4], const float* sp, int64_t ld, int dim, int c, int cols, bool fresh, int lane) {
#pragma unroll
  for (int i = 0; i < 2 * KS; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = 8 * i + 2 * (lane & 3) + (e & 1), cc = c + 4 * (e & 2);
      S[i][e] = (!fresh && d < dim && cc < cols) ? sp[(int64_t)d * ld + cc] : 0.f;
    }
}
template <int KS>
__device__ __forceinline__ void store_state(const float (&S)[2 * KS][4], float* sp, int64_t ld, int dim, int c, int cols, int lane) {
#pragma unroll
  for (int i = 0; i < 2 * KS; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int d = 8 * i + 2 * (lane & 3) + (e & 1), cc = c + 4 * (e & 2);
      if (d < dim && cc < cols) sp[(int64_t)d * ld + cc] = S[i][e];
    }
}
// S <- gn S + u K  (u: 16 columns x 32 tokens)
template <int KS>
__device__ __forceinline__ void state_update(float (&S)[2 * KS][4], float gn, const FragA (&u)[2], const Planes& K, int lane) {
#pragma unroll
  for (int i = 0; i < 2 * KS; i += 4) {
    float r[4][4] = {};
    FragB x[2][4];
#pragma unroll
    for (int s = 0; s < 2; ++s) load_b_t(x[s], K, 16 * s, 8 * i, lane);
    mma_small(r, u[0], x[0]);                 // the small products first, so that only the large ones meet a large sum
    mma_small(r, u[1], x[1]);
    mma_high(r, u[0], x[0]);
    mma_high(r, u[1], x[1]);
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[i + t][e] = fmaf(gn, S[i + t][e], r[t][e]);
  }
}
// out += f M^T: 16 columns x 8 NT tokens from 16 tokens of a token-by-token matrix
template <int NT>
__device__ __forceinline__ void add_tokens(float (&out)[NT][4], const FragA& f, const Planes& M, int m0, int k0, int lane) {
  float r[NT][4] = {};
  FragB x[NT];
  load_b(x, M, m0, k0, lane);
  mma_small(r, f, x);
  mma_high(r, f, x);
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) out[t][e] += r[t][e];
}

}  // namespace
