// Deterministic reduction over the batch axis: out[r] += sum_b f(r, b) for r < n.
// Two fixed stages (ascending b inside a chunk, ascending chunk order after), so
// the result depends only on (n, B, SM count), never on scheduling.
#pragma once
#include "common.cuh"

template <class F>
__global__ void __launch_bounds__(128) k_batch_reduce_partial(F f, size_t n, uint32_t B, uint32_t chunk,
                                                             float* __restrict__ partial,
                                                             float* __restrict__ out, int direct) {
  dyb_grid_dep_sync();
  size_t r = (size_t)blockIdx.x * 128 + threadIdx.x;
  if (r >= n) return;
  uint32_t b0 = blockIdx.y * chunk, b1 = min(B, b0 + chunk);
  float acc = 0.f;
  for (uint32_t b = b0; b < b1; b += 8) {   // eight loads in flight, summed in ascending order
    // (the last few too: one by one they were most of a chunk of 14, 14 of the 14 + 5 us of a layer norm's gain, 4096 x 1024 terms: now 10.5 + 5)
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = f(r, min(b + q, b1 - 1));
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (b + q < b1) acc += v[q];
  }
  if (direct) out[r] += acc;
  else partial[(size_t)blockIdx.y * n + r] = acc;
}

// 32 outputs per CTA, its eight warps an eighth of the partials each, added in warp order (one thread per output took 5.4 us for 4096 outputs of 74
// partials, a chain of ten loads on 32 CTAs; 2.5 - 3.7 now)
static __global__ void __launch_bounds__(256) k_batch_reduce_final(const float* __restrict__ partial, uint32_t S,
                                                                   size_t n, float* __restrict__ out) {
  dyb_grid_dep_sync();
  __shared__ float part[8][32];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, per = (S + 7) / 8, s0 = min(w * per, S), s1 = min(s0 + per, S);
  const size_t r = (size_t)blockIdx.x * 32 + lane;
  float acc = 0.f;
  if (r < n) {
    for (uint32_t s = s0; s < s1; s += 8) {
      float v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = partial[(size_t)min(s + q, s1 - 1) * n + r];
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (s + q < s1) acc += v[q];
    }
  }
  part[w][lane] = acc;
  __syncthreads();
  if (w == 0 && r < n) {
#pragma unroll
    for (int q = 1; q < 8; ++q) acc += part[q][lane];
    out[r] += acc;
  }
}
// The same for few outputs and many partial sums (a bias gradient over 100 000 columns: n = 45, S = 2368): a warp per
// output, lane l adds the partials l, l + 32, ... in ascending order (four loads in flight), then the lanes are added by a
// butterfly - a fixed order, so the result is reproducible.
static __global__ void __launch_bounds__(128) k_batch_reduce_final_warp(const float* __restrict__ partial, uint32_t S,
                                                                        size_t n, float* __restrict__ out) {
  dyb_grid_dep_sync();
  const size_t r = (size_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (r >= n) return;
  const uint32_t lane = threadIdx.x & 31;
  float acc = 0.f;
  uint32_t s = lane;
  for (; s + 96 < S; s += 128) {
    const float v0 = partial[(size_t)s * n + r], v1 = partial[(size_t)(s + 32) * n + r], v2 = partial[(size_t)(s + 64) * n + r],
                v3 = partial[(size_t)(s + 96) * n + r];
    acc += v0; acc += v1; acc += v2; acc += v3;
  }
  for (; s < S; s += 32) acc += partial[(size_t)s * n + r];
  acc = warp_sum(acc);
  if (lane == 0) out[r] += acc;
}

// Both stages in one CTA per 32 outputs, for few terms: 32 warps add a stretch of b each, in ascending order, then a warp per output the 32 stretches
// by a butterfly.  (5003 outputs of some 50 terms: 2.0 + 2.0 us in two launches, 3.1 in
// one; a pass of a tagger of 520 tokens, three launches less, 447 -> 444.5.)
constexpr uint32_t kReduceOneCols = 1024;
constexpr size_t kReduceOneTerms = 1u << 18;
template <class F>
__global__ void __launch_bounds__(1024) k_batch_reduce_one(F f, size_t n, uint32_t B, float* __restrict__ out) {
  dyb_grid_dep_sync();
  __shared__ float part[32][33];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, per = (B + 31) / 32, b0 = min(w * per, B), b1 = min(b0 + per, B);
  const size_t r = (size_t)blockIdx.x * 32 + lane, mine = (size_t)blockIdx.x * 32 + w;
  float acc = 0.f;
  if (r < n)
#pragma unroll 1
    for (uint32_t b = b0; b < b1; b += 8) {
      float v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = f(r, min(b + q, b1 - 1));
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (b + q < b1) acc += v[q];
    }
  part[w][lane] = acc;
  __syncthreads();
  acc = warp_sum(part[lane][w]);
  if (lane == 0 && mine < n) out[mine] += acc;
}

template <class F>
static int batch_reduce_add(dyb200_ctx* ctx, F f, size_t n, uint32_t B, float* out) {
  if (n == 0 || B == 0) return DYB200_OK;
  unsigned gx = (unsigned)((n + 127) / 128);
  unsigned want = (16u * ctx->sm_count + gx - 1) / gx;   // about 16 CTAs of 128 threads per SM
  unsigned S = want < 1 ? 1 : want;
  if (S > (B + 15) / 16) S = (B + 15) / 16;
  if (S < 1) S = 1;
  uint32_t chunk = (B + S - 1) / S;
  S = (B + chunk - 1) / chunk;
  if (S == 1) {
    dyb_launch(k_batch_reduce_partial<F>, dim3(gx, 1), 128, 0, ctx, f, n, B, chunk, nullptr, out, 1);
    DYB_LAUNCHED(ctx);
    return DYB200_OK;
  }
  if (B <= kReduceOneCols && n * B <= kReduceOneTerms) {
    dyb_launch(k_batch_reduce_one<F>, (unsigned)((n + 31) / 32), 1024, 0, ctx, f, n, B, out);
    DYB_LAUNCHED(ctx);
    return DYB200_OK;
  }
  void* scratch = nullptr;
  int rc = dyb200_scratch(ctx, (size_t)S * n * sizeof(float), &scratch);
  if (rc) return rc;
  dyb_launch(k_batch_reduce_partial<F>, dim3(gx, S), 128, 0, ctx, f, n, B, chunk, (float*)scratch, out, 0);
  DYB_LAUNCHED(ctx);
  if (n <= 512 && S >= 64) dyb_launch(k_batch_reduce_final_warp, (unsigned)((n + 3) / 4), 128, 0, ctx, (const float*)scratch, S, n, out);
  else dyb_launch(k_batch_reduce_final, (unsigned)((n + 31) / 32), 256, 0, ctx, (const float*)scratch, S, n, out);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}
