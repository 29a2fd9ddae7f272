// Router logits on mma.sync, softmax and top-k of the single-launch route+plan kernel of small batches
// (routing.cu).
//
// What bounds it: a batch of at most a few thousand copies is a chain of dependent loads and launches, not
// bytes.  A 128-row tcgen05 tile keeps one SM per 128 tokens busy and its k-blocks are one dependent chain of
// loads; 16-row mma.sync tiles with the row split over the warps of a CTA put many times as many loads in
// flight (1000 tokens of the Mixtral shape, router and plan: 46 us with one warp per token on CUDA cores, 13 us
// with these tiles).
//
// Tile: 16 tokens by NT x 8 experts per pass; the reduction dimension is dealt to KS warps in 64-element
// steps.  Fragments are loaded straight from global memory, 16 bytes per lane: the order of the
// reduction index inside a 32-element piece is free as long as both operands use the same one, so
// lane (g, q) takes the eight consecutive elements 8q.. of rows g and g + 8 (tokens) and of row g
// (experts), which are the operands of two MMAs.
//
// Precision: the tensor core truncates when it adds into its accumulator, and a chain over the whole
// row loses 2e-7 .. 4e-6 of a weight that way.  Each MMA therefore starts from zero and the
// running sums are fp32 adds.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "sm100_ptx.cuh"
#include "topk.cuh"

namespace b200 {

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

template <int NT, int KS>
struct RouterTile {
  static constexpr int TOK = 16;           // tokens per tile
  static constexpr int EXP = NT * 8;       // experts per pass over the rows
  static constexpr int THREADS = KS * 32;
  static constexpr int U = NT <= 2 ? 4 : 1;   // 64-element steps whose loads are in flight together
  static constexpr int PART = KS * TOK * EXP; // partial logits (floats)
  static __host__ __device__ constexpr int smem_bytes(int E) { return (PART + TOK * E) * 4; }

  // Logits of tokens [t0, t0 + TOK) (those below T) against all E experts into lg[TOK][E].
  // Every thread of the CTA takes part; ends with a barrier.
  static __device__ __forceinline__ void logits(const __nv_bfloat16* x,
                                                const __nv_bfloat16* __restrict__ wr_kmajor,
                                                const float* __restrict__ bias, int T, int D, int E, int t0,
                                                float* part, float* lg) {
    const int tid = threadIdx.x, ks = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, q = lane & 3;
    const int d16 = D / 8;            // 16-byte pieces per row
    const int steps = (d16 + 7) / 8;  // 64-element steps
    const uint4* xr[2];
#pragma unroll
    for (int h = 0; h < 2; ++h)       // rows past the batch repeat the last one; nothing reads their logits
      xr[h] = reinterpret_cast<const uint4*>(x) + static_cast<size_t>(min(t0 + h * 8 + g, T - 1)) * d16 + q;
    for (int e0 = 0; e0 < E; e0 += EXP) {
      const uint4* wp = reinterpret_cast<const uint4*>(wr_kmajor) + q;
      int wo[NT];
#pragma unroll
      for (int n = 0; n < NT; ++n) wo[n] = min(e0 + n * 8 + g, E - 1) * d16;
      float acc[NT][4];
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[n][j] = 0.f;
      for (int s0 = ks; s0 < steps; s0 += U * KS) {
        uint4 xv[U][2][2], wv[U][2][NT];
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const int i = (s0 + u * KS) * 8 + j * 4;
            const bool in = i + q < d16;
#pragma unroll
            for (int h = 0; h < 2; ++h) xv[u][j][h] = in ? ld_16(xr[h] + i) : zero;
#pragma unroll
            for (int n = 0; n < NT; ++n) wv[u][j][n] = in ? __ldg(wp + wo[n] + i) : zero;
          }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int n = 0; n < NT; ++n) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const uint4 a = xv[u][j][0], b = xv[u][j][1], w = wv[u][j][n];
              float c[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {0.f, 0.f, 0.f, 0.f};
              mma_bf16_16816(c, a.x, b.x, a.y, b.y, w.x, w.y);
              mma_bf16_16816(d, a.z, b.z, a.w, b.w, w.z, w.w);
#pragma unroll
              for (int v = 0; v < 4; ++v) acc[n][v] += c[v] + d[v];
            }
          }
      }
#pragma unroll
      for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          *reinterpret_cast<float2*>(part + (ks * TOK + h * 8 + g) * EXP + n * 8 + 2 * q) =
              make_float2(acc[n][2 * h], acc[n][2 * h + 1]);
      __syncthreads();
      for (int i = tid; i < TOK * EXP; i += THREADS) {
        const int t = i / EXP, e = e0 + i % EXP;
        if (e < E) {
          float v[KS];                 // pairwise: half the rounding error of a running sum
#pragma unroll
          for (int w = 0; w < KS; ++w) v[w] = part[w * TOK * EXP + i];
#pragma unroll
          for (int o = KS / 2; o > 0; o >>= 1)
#pragma unroll
            for (int w = 0; w < o; ++w) v[w] += v[w + o];
          lg[t * E + e] = bias ? v[0] + bias[e] : v[0];
        }
      }
      __syncthreads();
    }
  }
};

// Softmax over one token's E <= 32 * PER logits (shared memory) and its k best experts, by one warp: lane
// r < k returns choice r in my_i (`none` when no expert with a logit above -inf is left) and its
// (renormalised) probability in my_w.  Ties go to the lower index.  Logits are compared as
// order-preserving 32-bit keys, one warp-wide reduction for the value and one for the index a round.
template <int PER>
__device__ __forceinline__ void warp_softmax_topk(const float* lg, int E, int k, int renorm, int none, int lane,
                                                  int& my_i, float& my_w) {
  float v[PER];
  uint32_t key[PER];
  uint32_t best = 0u;
#pragma unroll
  for (int j = 0; j < PER; ++j) {
    const int e = lane + 32 * j;
    v[j] = e < E ? lg[e] : -INFINITY;
    const uint32_t b = __float_as_uint(v[j]);
    key[j] = v[j] > -INFINITY ? ((b >> 31) ? ~b : (b | 0x80000000u)) : 0u;   // NaN and -inf: never chosen
    if (v[j] == 0.f) key[j] = 0x80000000u;                                   // -0 and +0 tie
    best = max(best, key[j]);
  }
  best = __reduce_max_sync(0xffffffffu, best);
  auto value = [](uint32_t u) {
    return u == 0u ? -INFINITY : __uint_as_float((u >> 31) ? (u & 0x7fffffffu) : ~u);
  };
  const float mx = value(best);
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < PER; ++j)
    if (lane + 32 * j < E) sum += __expf(v[j] - mx);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  float my_p = 0.f;
  my_i = 0;
  for (int r = 0; r < k; ++r) {
    int mine = 0x7fffffff;
#pragma unroll
    for (int j = PER - 1; j >= 0; --j)
      if (key[j] == best && best != 0u) mine = lane + 32 * j;
    const int win = __reduce_min_sync(0xffffffffu, mine);
    if (lane == r) {
      my_p = __expf(value(best) - mx);
      my_i = best != 0u ? win : none;
    }
    uint32_t next = 0u;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      if (win == lane + 32 * j) key[j] = 0u;
      next = max(next, key[j]);
    }
    best = __reduce_max_sync(0xffffffffu, next);
  }
  my_w = my_p / sum;
  if (renorm) {
    float wsum = 0.f;
    for (int r = 0; r < k; ++r) wsum += __shfl_sync(0xffffffffu, my_w, r);
    my_w = my_w / wsum;
  }
}

// One tile: logits, then one warp per token for softmax and top-k.  `smem` holds
// RouterTile::smem_bytes(E) bytes.
template <int NT, int KS>
__device__ __forceinline__ void route_tile(const __nv_bfloat16* x, const __nv_bfloat16* wr_kmajor, const float* bias,
                                           int T, int D, int E, int k, int renorm, int none, int t0, int* topk_idx,
                                           float* topk_w, float* smem) {
  using R = RouterTile<NT, KS>;
  float* lg = smem + R::PART;
  R::logits(x, wr_kmajor, bias, T, D, E, t0, smem, lg);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t = warp; t < R::TOK && t0 + t < T; t += KS) {
    int my_i;
    float my_w;
    if (NT <= 4) warp_softmax_topk<1>(lg + t * E, E, k, renorm, none, lane, my_i, my_w);
    else if (E <= 64) warp_softmax_topk<2>(lg + t * E, E, k, renorm, none, lane, my_i, my_w);
    else warp_softmax_topk<8>(lg + t * E, E, k, renorm, none, lane, my_i, my_w);
    if (lane < k) {
      topk_idx[static_cast<size_t>(t0 + t) * k + lane] = my_i;
      topk_w[static_cast<size_t>(t0 + t) * k + lane] = my_w;
    }
  }
}

}  // namespace b200
