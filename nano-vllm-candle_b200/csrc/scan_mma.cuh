// Products of fp32 numbers on the tensor pipe for the chunked recurrences (retention.cu, delta_rule.cu).
//
// An fp32 number is the exact sum of three bf16 numbers (8 + 8 + 8 bits: high, middle, low), and a product of two numbers is the sum of nine
// products of parts.  The six largest are taken (mma.sync m16n8k16, exact products, fp32 sums); the three that are left out are below
// 2^-24 of the whole.  That holds for every number by itself, whatever its neighbours are.  (Two fp16 parts under one scale per row or state column, three
// products: 177 us for the delta rule where this takes 213, but 22 bits of the row's largest number for all of them: a channel 2^11 below its
// neighbours came out with errors of 5e-6 to 5e-5, one 2^20 below with none of its digits.)
// The pipe's own sums round towards zero, relative to the sum: the large products, which make that sum, are added up in short chains of their own (16 - 64 terms)
// that ordinary fp32 adds take over, the small ones apart from them, or in front of them (the observation and the remedy are Ootomo and Yokota's, "Recovering
// single precision accuracy from Tensor Cores", 2022).  Against 64 bits, relative, over eight prompts of 245 to 1 050 tokens: delta rule of 16 heads of
// 128 x 128, outputs 1.2e-7, state 0.96e-7; 32 heads of 128 x 64 with a decay per token, 0.97e-7 and 0.63e-7.
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

constexpr int kBuffers = 3, kScanThreads = 512, kPrep0 = 8;       // threads, first preparing warp

// What the chunked recurrences on the tensor pipe have in common.  One CTA of sixteen warps per (sequence, head, 64 value columns), one CTA per SM:
//   warps 8 .. 15 prepare the chunks of 32 tokens, in two groups that take every other chunk (and the first one together, so that a short portion does
//                 not wait for its keys behind its queries): rows from global memory into planes of bf16 parts in shared memory, decays, the
//                 token-by-token products
//   warps 0 .. 7  carry the state, 16 value columns of one half of the channels each.  It is kept TRANSPOSED in the warp's accumulator registers
//                 (16 columns x 64 channels: 32 numbers per thread at 128 channels), where it is at once the left operand of its products
//                 with the chunk's rows and the accumulator of its own update: it never travels.  The two warps of a pair (w, w + 4) add what their halves
//                 of the channels give to the chunk's rows by way of shared memory.
// The tensor pipe is what takes the time: half of all cycles in the mean over the SMs, with some 700 products per SM quarter and chunk, and the warps that
// wait for it or for one another are the rest.  Against four and four warps, whose preparation asks for queries, keys and values at once (us): eight prompts of 245 to
// 1 050 tokens, delta rule of 16 heads of 128 x 128 238 -> 212, of 8 heads of 64 x 128 158 -> 133; 32 heads of 128 x 64 with a decay per token 152 -> 141; 64
// portions of 20 tokens 123 -> 116, delta rule 176 -> 178, of 64 x 128 64 -> 73.  Not kept: the pair's sums exchanged behind the state's update instead of in front
// of it (ssm 146 -> 150), both warps of a pair solving for the chunk's U instead of one that hands it on (delta 222 -> 232), two buffers instead of three at 128
// channels (no change), queries and keys of every chunk at once (213 -> 223, for want of registers).
// 128 registers per thread: a few numbers are spilled (8 - 52 bytes loaded per thread); moving registers from the preparing warps to the state's
// (144 and 112: 277 -> 281 us for the delta rule with its preparation) only moves the spills there.
// Named barriers: a buffer is filled / free for its next chunk; a group of preparing warps; a pair.  (Of three buffers, chunks i and i + 3 share one but not
// the group that fills it, so each group waits for a free buffer at barriers of its own: chunk i at kEmpty + i % 6; of two, at kEmpty + i % 4.)
enum { kFull = 1, kEmpty = kFull + kBuffers, kPrepare = kEmpty + 2 * kBuffers, kPair = kPrepare + 2 };
static_assert(kPair + 4 <= 16, "barriers");
constexpr int kBufThreads = 384;        // the state warps and one group
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
// 32 rows of up to DZ (64 or 128) numbers by a group of preparing warps, in registers between global and shared memory
template <int DZ>
struct RowTile {
  static constexpr int kLanes = DZ / 4, kRows = 32 / kLanes, kPasses = kMT / (kRows * 4);
  float4 x[kPasses];
  __device__ __forceinline__ static int row(int i, int pw, int lane) { return (4 * i + pw) * kRows + lane / kLanes; }
  __device__ __forceinline__ void load(const float* src, int64_t ld, int dim, int n, bool vec, int pw, int lane) {
    if (vec && dim == DZ) {                   // no question per row: those behind the end repeat the last one, as zeros
      const float* p = src + 4 * (lane % kLanes);
#pragma unroll
      for (int i = 0; i < kPasses; ++i) x[i] = *reinterpret_cast<const float4*>(p + min(row(i, pw, lane), n - 1) * ld);
      if (n < kMT)
#pragma unroll
        for (int i = 0; i < kPasses; ++i)
          if (row(i, pw, lane) >= n) x[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    } else {
#pragma unroll
      for (int i = 0; i < kPasses; ++i) {
        const int r = row(i, pw, lane);
        x[i] = load_quad(src + r * ld, 4 * (lane % kLanes), dim, r < n, vec);
      }
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

// 32 rows of up to kMC values into shared memory by a group of preparing warps; they are there behind values_wait() of every thread
__device__ __forceinline__ void fetch_values(float* dst, const float* src, int64_t ld, int cols, int n, bool vec, int pw, int lane) {
  using Tile = RowTile<kMC>;
  if (vec && cols == kMC) {
#pragma unroll
    for (int i = 0; i < Tile::kPasses; ++i) {
      const int r = Tile::row(i, pw, lane), c = 4 * (lane % Tile::kLanes);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst + r * kMV + c)), "l"(src + min(r, n - 1) * ld + c), "r"(r < n ? 16 : 0) : "memory");
    }
  } else {
    Tile v;
    v.load(src, ld, cols, n, vec, pw, lane);
    v.store_to(dst, kMV, pw, lane);
  }
}
__device__ __forceinline__ void values_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The sequence of a block when the longest are to start first (one wave of CTAs rarely holds them all): the one with `rank` longer ones.
// Sequences beyond 256 keep their order.  All threads of the CTA call it; every sequence is compared by two of them.
struct RankScratch { int len[256], longer[256], found; };
__device__ __forceinline__ int sequence_of_rank(const int32_t* cu, int B, int rank, RankScratch& s) {
  static_assert(kScanThreads == 512, "two threads per sequence");
  if (B > 256 || B == 1) return rank;
  const int i = threadIdx.x & 255, part = threadIdx.x >> 8, mid = B >> 1;
  if (part == 0 && i < B) {
    s.len[i] = cu[i + 1] - cu[i];
    s.longer[i] = 0;
  }
  __syncthreads();
  if (i < B) {
    const int len = s.len[i];
    int longer = 0;
    for (int j = part ? mid : 0; j < (part ? B : mid); ++j) longer += s.len[j] > len || (s.len[j] == len && j < i);
    atomicAdd(&s.longer[i], longer);
  }
  __syncthreads();
  if (part == 0 && i < B && s.longer[i] == rank) s.found = i;
  __syncthreads();
  return s.found;
}

// Token-by-token products: rows x0 .. x0 + 15 of X against rows y0 .. y0 + 15 of Y, two tiles of eight columns; KS blocks of 16 channels, two side by side with
// sums of their own (at most 32 terms each).  A chain of products on one accumulator waits for each of them, so the two blocks' products alternate: one block behind the other
// took 3 100 cycles per 16 x 16 tokens of 128 channels.
template <int KS>
__device__ __forceinline__ void token_products(float (&out)[2][4], const Planes& X, int x0, const Planes& Y, int y0, int lane) {
  constexpr int pa[5] = {2, 0, 1, 1, 0}, pb[5] = {0, 2, 1, 0, 1};
  float rest[2][2][4] = {};
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) out[t][i] = 0.f;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    float x[2][2][4] = {};
#pragma unroll
    for (int ks = half * (KS / 2); ks < (half + 1) * (KS / 2); ks += 2) {
      FragA a[2];
      FragB b[2][2];
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        load_a(a[p], X, x0, (ks + p) * 16, lane);
        load_b(b[p], Y, y0, (ks + p) * 16, lane);
      }
#pragma unroll
      for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (i == 0) mma_bf16_acc(x[p][t], a[p].r[0], b[p][t].r[0]);
            else mma_bf16_acc(rest[p][t], a[p].r[pa[i - 1]], b[p][t].r[pb[i - 1]]);
          }
    }
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int i = 0; i < 4; ++i) out[t][i] += x[0][t][i] + x[1][t][i];
  }
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int i = 0; i < 4; ++i) out[t][i] += rest[0][t][i] + rest[1][t][i];
}

// Decays are differences of running sums of log decays over a chunk's tokens, kept in 64 bits and handed on in two parts: sums of 32 tokens reach 30 and
// more, and e^x in fp32 is off by its argument's rounding, |x| 2^-25.  What the first part leaves over comes back as e^lo = 1 + lo.
__device__ __forceinline__ float exp_parts(float hi, float lo) {
  const float e = expf(hi);
  return fmaf(e, lo, e);
}
struct LogSum {
  double l;                               // of a warp's 32 tokens, a token per lane
  __device__ __forceinline__ LogSum(float log_decay, int lane) {
    l = (double)log_decay;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, l, o);
      if (lane >= o) l += up;
    }
  }
  __device__ __forceinline__ static float power(double x) {
    const float hi = (float)x;
    return exp_parts(hi, (float)(x - (double)hi));
  }
  __device__ __forceinline__ float from() const { return power(l); }                                          // from the chunk's start up to the token
  __device__ __forceinline__ float to() const { return power(__shfl_sync(0xffffffffu, l, 31) - l); }            // behind the token up to the chunk's end
};
// decays between the tokens of a thread's numbers in a 16 x 16 block
struct Decays {
  float th[2], tl[2], jh[4], jl[4];
  __device__ __forceinline__ void load(const float* Lh, const float* Ll, int t0, int j0, int lane) {
#pragma unroll
    for (int i = 0; i < 2; ++i) { th[i] = Lh[t0 + (lane >> 2) + 8 * i]; tl[i] = Ll[t0 + (lane >> 2) + 8 * i]; }
#pragma unroll
    for (int i = 0; i < 4; ++i) { jh[i] = Lh[j0 + 2 * (lane & 3) + (i & 1) + 4 * (i & 2)]; jl[i] = Ll[j0 + 2 * (lane & 3) + (i & 1) + 4 * (i & 2)]; }
  }
  // number e of tile y; the sum of a later token is the larger one in size, so what the difference rounds away is (a - d) - b
  __device__ __forceinline__ float operator()(int y, int e) const {
    const float a = th[e >> 1], b = jh[2 * y + (e & 1)], d = a - b;
    return exp_parts(d, ((a - d) - b) + (tl[e >> 1] - jl[2 * y + (e & 1)]));
  }
};
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
// S <- gn S + u K  (u: 16 columns x 32 tokens; the channels from d0 on)
template <int KS>
__device__ __forceinline__ void state_update(float (&S)[2 * KS][4], float gn, const float (&u)[4][4], const Planes& K, int d0, int lane) {
  FragA a[2];
  frag_of_tiles(a[0], u[0], u[1]);
  frag_of_tiles(a[1], u[2], u[3]);
#pragma unroll
  for (int i = 0; i < 2 * KS; i += 4) {
    float r[4][4] = {};
    FragB x[2][4];
#pragma unroll
    for (int s = 0; s < 2; ++s) load_b_t(x[s], K, 16 * s, d0 + 8 * i, lane);
    mma_small(r, a[0], x[0]);                 // the small products first, so that only the large ones meet a large sum
    mma_small(r, a[1], x[1]);
    mma_high(r, a[0], x[0]);
    mma_high(r, a[1], x[1]);
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
