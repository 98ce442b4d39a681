// Products with one narrow side and a long one, in fp32 on the CUDA cores: the per-token layers of a tagger (32 or 45 rows times
// 100 000 tokens), their gradients by the tokens and by the weights.
//   a short reduction (up to 64), many columns:   C (M x N) = epilogue(op(A) B)      k_gemm_narrow
//   few rows, more to reduce over, many columns:  the same                           k_gemm_slices
//   both sides small, a long reduction:           C (M x N) (+)= A B^T               k_gemm_narrow_k
// On the tensor path such a product is bound by everything but its arithmetic: the long operand is read, written as two split planes
// and read again, three quarters of the rows of a 128-row tile are padding, and accumulating stores go by registers.  32 x 107 000 x 256
// took 111 + 56 us (split + product), its gradient by the tokens 111 + 263, that by the weights 219 + 263.  Here the small
// operand sits in shared memory, the long one streams through it once, and the fp32 multiply-adds (1.8 G, 24 us at the cores' full
// rate) stay under what the split planes alone cost.
#include "gemm.cuh"

namespace {

constexpr int kThreadsN = 256;
constexpr uint32_t kNarrow = 64;                 // what counts as narrow
constexpr uint32_t kSmallMax = 16 * 1024;        // floats of op(A) kept in shared memory
constexpr size_t kSmemNarrow = 224 * 1024;       // (the most a launch takes)

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(void* dst, const float* src, uint32_t bytes) {   // bytes < 16: the rest is zero
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const float* src, uint32_t bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

struct Narrow {
  const float *A, *B; uint32_t lda, ldb; int transA;
  uint32_t M, N, K;
  uint32_t MP;        // rows of A in a CTA's shared memory: one or more row blocks (grid.y CTAs share the rows)
  uint32_t KC, pitch; // k per piece of B; floats per column of a piece (an odd number of float4: eight columns, eight bank groups)
  int vec_b, vec_c;   // 16-byte loads of B / accesses of C
  float* C; uint32_t ldc; const float* bias; int mode;
};

constexpr int kStagesN = 3;

// Thread: 8 rows x NJ columns, ML threads along the rows; a block is 8 ML rows x 256 / ML NJ columns.  Per four k a thread reads
// 8 + NJ float4 for 32 NJ multiply-adds: shared memory, two to four cycles per read, is what bounds this kernel up to NJ = 4 (4 x 4
// outputs per thread took 63 us where 8 x 4 take 48, 32 x 107 000 x 256).  Either there is one row block (few rows: B comes in
// several pieces, the sums stay in registers) or one piece (short reduction: every row block uses the piece that is there).
// CTAs are persistent; their pieces run through a ring of three.
template <int ML, int NJ>
__global__ void __launch_bounds__(kThreadsN) k_gemm_narrow(const Narrow a) {
  dyb_grid_dep_sync();
  constexpr uint32_t NL = 32 / ML, TN = kThreadsN / ML * NJ, MB = 8 * ML;   // NL: threads of a warp along the columns
  extern __shared__ __align__(16) float nsm[];
  float* As = nsm;                                   // [K][MP]
  float* ring = nsm + (size_t)a.K * a.MP;
  const uint32_t tid = threadIdx.x, mg = tid % ML, n_t = (tid >> 5) * (NL * NJ) + (tid & 31) / ML;
  const uint32_t m_base = blockIdx.y * a.MP;
  const uint32_t tiles = (a.N + TN - 1) / TN, nkc = (a.K + a.KC - 1) / a.KC, nmb = a.MP / MB;
  const uint32_t my_tiles = blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0, items = my_tiles * nkc;
  // this thread's part of a piece: the same k of every f_step-th column
  const uint32_t f_q = a.vec_b ? a.KC / 4 : a.KC, f_step = kThreadsN / f_q, f_k = (tid % f_q) * (a.vec_b ? 4 : 1);
  const uint32_t f_n = tid < f_step * f_q ? tid / f_q : TN;
  auto fetch = [&](uint32_t item) {
    if (item < items) {
      const uint32_t n0 = (blockIdx.x + (item / nkc) * gridDim.x) * TN, k0 = (item % nkc) * a.KC, kn = min(a.KC, a.K - k0);
      float* st = ring + (size_t)(item % kStagesN) * TN * a.pitch;
      if (f_n < TN) {
        const uint32_t w = a.vec_b ? 4 : 1, left = f_k < kn ? min(w, kn - f_k) * 4 : 0;
        float* d = st + f_n * a.pitch + f_k;
        const float* src = a.B + (left ? (size_t)a.ldb * (n0 + f_n) + k0 + f_k : 0);
        for (uint32_t n = f_n; n < TN; n += f_step, d += f_step * a.pitch, src += left ? (size_t)a.ldb * f_step : 0) {
          const bool in = left && n0 + n < a.N;
          if (a.vec_b) cp_async16(d, in ? src : a.B, in ? left : 0);
          else cp_async4(d, in ? src : a.B, in ? 4 : 0);
        }
      }
    }
    cp_commit();
  };
  fetch(0);
  fetch(1);
  for (uint32_t m = tid & 31; m < a.MP; m += 32) {
    const uint32_t mm = m_base + m;
    const size_t step = a.transA ? 1 : a.lda;
    const float* src = a.A + (mm < a.M ? a.transA ? (size_t)a.lda * mm : mm : 0);
#pragma unroll 8
    for (uint32_t k = tid >> 5; k < a.K; k += kThreadsN / 32) As[(size_t)k * a.MP + m] = mm < a.M ? src[k * step] : 0.f;
  }
  float acc[8][NJ];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[i][j] = 0.f;
  for (uint32_t item = 0; item < items; ++item) {
    cp_wait<kStagesN - 2>();
    __syncthreads();            // this piece is here, and every thread is done with the one before it
    fetch(item + 2);
    const uint32_t n0 = (blockIdx.x + (item / nkc) * gridDim.x) * TN, kc = item % nkc, k0 = kc * a.KC, kn = min(a.KC, a.K - k0);
    const float* bs = ring + (size_t)(item % kStagesN) * TN * a.pitch + (size_t)n_t * a.pitch;
    for (uint32_t mb = 0; mb < nmb; ++mb) {
      const float* as = As + (size_t)k0 * a.MP + mb * MB + 4 * mg;
      const bool last = kc + 1 == nkc, add = a.mode == EPI_ACCUM && a.vec_c && last;
      float4 old[NJ][2];   // (read before the products, which cover the time that takes)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t n = n0 + n_t + NL * j, m = m_base + mb * MB + 4 * ML * h + 4 * mg;
          old[j][h] = add && n < a.N && m < a.M ? ld4(a.C + m + (size_t)a.ldc * n) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      const uint32_t k4 = kn / 4 * 4;
      for (uint32_t k = 0; k < k4; k += 4) {
        float4 b[NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) b[j] = ld4(bs + NL * j * a.pitch + k);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          float w[8];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float4 v = ld4(as + (size_t)(k + kk) * a.MP + 4 * ML * h);
            w[4 * h] = v.x; w[4 * h + 1] = v.y; w[4 * h + 2] = v.z; w[4 * h + 3] = v.w;
          }
#pragma unroll
          for (int j = 0; j < NJ; ++j) {
            const float x = kk == 0 ? b[j].x : kk == 1 ? b[j].y : kk == 2 ? b[j].z : b[j].w;
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(w[i], x, acc[i][j]);
          }
        }
      }
      for (uint32_t k = k4; k < kn; ++k)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 v = ld4(as + (size_t)k * a.MP + 4 * ML * h);
#pragma unroll
          for (int j = 0; j < NJ; ++j) {
            const float x = bs[NL * j * a.pitch + k];
            acc[4 * h][j] = fmaf(v.x, x, acc[4 * h][j]);
            acc[4 * h + 1][j] = fmaf(v.y, x, acc[4 * h + 1][j]);
            acc[4 * h + 2][j] = fmaf(v.z, x, acc[4 * h + 2][j]);
            acc[4 * h + 3][j] = fmaf(v.w, x, acc[4 * h + 3][j]);
          }
        }
      if (!last) continue;
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t n = n0 + n_t + NL * j, m = m_base + mb * MB + 4 * ML * h + 4 * mg;
          float v[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) { v[i] = acc[4 * h + i][j]; acc[4 * h + i][j] = 0.f; }
          if (n >= a.N || m >= a.M) continue;
          float* c = a.C + m + (size_t)a.ldc * n;
          if (a.vec_c) {
            if (a.mode == EPI_BIAS) { const float4 b = ld4(a.bias + m); v[0] += b.x; v[1] += b.y; v[2] += b.z; v[3] += b.w; }
            if (a.mode == EPI_ACCUM) { const float4 o = old[j][h]; v[0] += o.x; v[1] += o.y; v[2] += o.z; v[3] += o.w; }
            st4(c, make_float4(v[0], v[1], v[2], v[3]));
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (m + i < a.M) c[i] = v[i] + (a.mode == EPI_BIAS ? a.bias[m + i] : a.mode == EPI_ACCUM ? c[i] : 0.f);
          }
        }
    }
  }
  cp_wait<0>();
}

// ---- few rows, a reduction of more than 64 ----
struct Slices {
  const float *A, *B; uint32_t lda, ldb; int transA;
  uint32_t M, N, K;   // (at most 64 rows: one row block)
  uint32_t KS, CS;    // KS CS = 8: slices of a piece's reduction and stretches of columns that the warps share out
  uint32_t KC, pieces, TN, pitch;   // k per piece of B and pieces of the reduction; columns per tile; floats per column of a piece (an odd number of float4: eight columns, eight bank groups)
  int vec_b, vec_c;   // 16-byte loads of B / accesses of C
  float* C; uint32_t ldc; const float* bias; int mode;
};

// Lane: 8 rows x NJ columns, ML lanes along the rows, so that a warp has 8 ML rows x 32 / ML NJ columns: per four k a lane reads 8 + NJ float4 for 32 NJ multiply-adds,
// with NJ = 8 half as many reads per multiply-add as 8 x 4 per thread.  What bounds it then is two warps per scheduler (58 % of the issue slots, 42 % of the
// multiply-adds' rate at 32 x 107 000 x 256).  B comes in pieces of 64 k (of 16 each piece took a barrier per 2000 cycles), one on its way while the other is used.
// The eight warps share out columns and, where there are fewer tiles than SMs, slices of a piece's reduction, whose sums meet, in their order, in the buffer just read:
// without slices a few hundred columns were 15 us of one CTA's latencies.
// us, k_gemm_narrow / here, by columns:  520  2300  13 400  107 000
//   32 rows, K = 256   15.2 / 5.9  15.3 / 9.4  28.0 / 18.6  99 / 67      K = 128   8.7 / 5.7  8.8 / 5.7  15.3 / 12.8  52 / 37
//   64 rows, K = 256   16.4 / 7.3  18.7 / 10.7  31.1 / 26.2  142 / 109   K = 128   9.3 / 6.1  9.3 / 7.4  17.3 / 16.5  76 / 59
// Up to 64 k k_gemm_narrow is the faster one (32 rows, K = 32, 13 400 columns 5.5 / 8.8): there B's pieces are few and its tiles store while others load.
template <int ML, int NJ>
__global__ void __launch_bounds__(kThreadsN) k_gemm_slices(const Slices a) {
  dyb_grid_dep_sync();
  constexpr uint32_t NL = 32 / ML, WN = NL * NJ, MB = 8 * ML;   // NL: lanes along the columns; WN: columns of a warp
  extern __shared__ __align__(16) float nsm[];
  float* As = nsm;                                   // [K][MB]
  float* ring = nsm + (size_t)a.K * MB;              // [2][TN][pitch]
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, mg = lane % ML, nl = lane / ML;
  const uint32_t ks = warp % a.KS, cs = warp / a.KS, buffer = a.TN * a.pitch, tiles = (a.N + a.TN - 1) / a.TN;
  const uint32_t my_tiles = blockIdx.x < tiles ? (tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0, items = my_tiles * a.pieces;
  // this thread's part of a piece: the same k of every f_step-th column
  const uint32_t f_q = a.vec_b ? a.KC / 4 : a.KC, f_step = kThreadsN / f_q, f_k = (tid % f_q) * (a.vec_b ? 4 : 1), f_n = tid / f_q;
  auto fetch = [&](uint32_t item) {
    if (item < items && f_n < f_step) {
      const uint32_t n0 = (blockIdx.x + item / a.pieces * gridDim.x) * a.TN, k = item % a.pieces * a.KC + f_k, cols = min(a.TN, a.N - n0);
      if (k < a.K) {
        float* d = ring + (item & 1) * buffer + f_n * a.pitch + f_k;
        const float* src = a.B + (size_t)a.ldb * (n0 + f_n) + k;
        const uint32_t bytes = 4 * min(4u, a.K - k);
        for (uint32_t n = f_n; n < cols; n += f_step, d += f_step * a.pitch, src += (size_t)a.ldb * f_step) {
          if (a.vec_b) cp_async16(d, src, bytes); else cp_async4(d, src, 4);
        }
      }
    }
    cp_commit();
  };
  fetch(0);
  for (uint32_t m = lane; m < MB; m += 32) {
    const size_t step = a.transA ? 1 : a.lda;
    const float* src = a.A + (m < a.M ? a.transA ? (size_t)a.lda * m : m : 0);
#pragma unroll 8
    for (uint32_t k = warp; k < a.K; k += kThreadsN / 32) As[(size_t)k * MB + m] = m < a.M ? src[k * step] : 0.f;
  }
  const uint32_t per = a.KC / a.KS, k_of = ks * per;                                          // this warp's slice of a piece
  // the thread's part of a tile's results, where they go by shared memory
  const uint32_t o_q = a.vec_c ? a.M / 4 : a.M, o_step = kThreadsN / o_q, o_m = (tid % o_q) * (a.vec_c ? 4 : 1), o_n = tid / o_q;
  float acc[8][NJ];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) acc[i][j] = 0.f;
  uint32_t piece = 0, tile = blockIdx.x;
  for (uint32_t item = 0; item < items; ++item) {
    float* const st = ring + (item & 1) * buffer;
    fetch(item + 1);
    cp_wait<1>();
    __syncthreads();            // this piece (the first time: A too) is here
    const uint32_t n0 = tile * a.TN, k0 = piece * a.KC, kn = min(per, k0 + k_of < a.K ? a.K - k0 - k_of : 0);   // k of this warp's slice
    const float *bs = st + (size_t)(cs * WN + nl) * a.pitch + k_of, *as = As + (size_t)(k0 + k_of) * MB + 4 * mg;
    float4 b[NJ];
    if (kn >= 4) {
#pragma unroll
      for (int j = 0; j < NJ; ++j) b[j] = ld4(bs + NL * j * a.pitch);
    }
    uint32_t k = 0;
#pragma unroll 2
    for (; k + 4 <= kn; k += 4, as += 4 * MB) {
      float4 next[NJ];
      const uint32_t kx = k + 8 <= kn ? k + 4 : k;   // (asked for a step ahead)
#pragma unroll
      for (int j = 0; j < NJ; ++j) next[j] = ld4(bs + NL * j * a.pitch + kx);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        float w[8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float4 v = ld4(as + (size_t)kk * MB + 4 * ML * h);
          w[4 * h] = v.x; w[4 * h + 1] = v.y; w[4 * h + 2] = v.z; w[4 * h + 3] = v.w;
        }
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const float x = kk == 0 ? b[j].x : kk == 1 ? b[j].y : kk == 2 ? b[j].z : b[j].w;
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i][j] = fmaf(w[i], x, acc[i][j]);
        }
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) b[j] = next[j];
    }
    for (; k < kn; ++k, as += MB)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 v = ld4(as + 4 * ML * h);
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const float x = bs[NL * j * a.pitch + k];
          acc[4 * h][j] = fmaf(v.x, x, acc[4 * h][j]);
          acc[4 * h + 1][j] = fmaf(v.y, x, acc[4 * h + 1][j]);
          acc[4 * h + 2][j] = fmaf(v.z, x, acc[4 * h + 2][j]);
          acc[4 * h + 3][j] = fmaf(v.w, x, acc[4 * h + 3][j]);
        }
      }
    __syncthreads();            // everybody is done with the buffer
    if (++piece < a.pieces) continue;
    piece = 0;
    tile += gridDim.x;
    if (a.KS == 1 && a.vec_c) {
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t n = n0 + cs * WN + nl + NL * j, m = 4 * mg + 4 * ML * h;
          float4 v = make_float4(acc[4 * h][j], acc[4 * h + 1][j], acc[4 * h + 2][j], acc[4 * h + 3][j]);
          acc[4 * h][j] = acc[4 * h + 1][j] = acc[4 * h + 2][j] = acc[4 * h + 3][j] = 0.f;
          if (n >= a.N || m >= a.M) continue;
          float* c = a.C + m + (size_t)a.ldc * n;
          if (a.mode == EPI_BIAS) { const float4 o = ld4(a.bias + m); v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
          if (a.mode == EPI_ACCUM) { const float4 o = ld4(c); v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w; }
          st4(c, v);
        }
      continue;
    }
    // the slices' sums side by side: [slice][column][row]
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        st4(st + ((size_t)ks * a.TN + cs * WN + nl + NL * j) * MB + 4 * mg + 4 * ML * h, make_float4(acc[4 * h][j], acc[4 * h + 1][j], acc[4 * h + 2][j], acc[4 * h + 3][j]));
        acc[4 * h][j] = acc[4 * h + 1][j] = acc[4 * h + 2][j] = acc[4 * h + 3][j] = 0.f;
      }
    __syncthreads();
    const uint32_t slice = a.TN * MB, cols = min(a.TN, a.N - n0);
    if (o_n < o_step)
      for (uint32_t n = o_n; n < cols; n += o_step) {
        float* c = a.C + o_m + (size_t)a.ldc * (n0 + n);
        const float* v = st + (size_t)n * MB + o_m;
        if (a.vec_c) {
          float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
          if (a.mode == EPI_BIAS) o = ld4(a.bias + o_m);
          if (a.mode == EPI_ACCUM) o = ld4(c);
          float4 r = ld4(v);
          for (uint32_t x = 1; x < a.KS; ++x) { const float4 w = ld4(v + x * slice); r.x += w.x; r.y += w.y; r.z += w.z; r.w += w.w; }
          st4(c, make_float4(r.x + o.x, r.y + o.y, r.z + o.z, r.w + o.w));
        } else {
          float r = *v;
          for (uint32_t x = 1; x < a.KS; ++x) r += v[x * slice];
          *c = r + (a.mode == EPI_BIAS ? a.bias[o_m] : a.mode == EPI_ACCUM ? *c : 0.f);
        }
      }
    __syncthreads();            // the buffer is free again
  }
  cp_wait<0>();
}

// ---- long reductions -------------------------------------------------------------------------------------------------------
struct NarrowK {
  const float *A, *B; uint32_t lda, ldb;
  uint32_t M, N, K;
  uint32_t MT, NT;          // output block of a CTA (multiples of 8); grid.y counts the blocks along the side that has several
  uint32_t groups, KC;      // groups of threads that share a piece's k; k per piece (a multiple of `groups`)
  uint32_t kspan;           // k per CTA
  int vec_a, vec_b;
  int meet;                 // the groups' sums meet in shared memory (else: a partial product per group)
  float* part;              // [grid.x][groups, or 1][M N]
};
constexpr uint32_t kTilesMax = kThreadsN / 2;   // 8 x 8 outputs per thread and at least two groups: 8192 outputs per CTA

// CTA: k in [kspan x, + kspan) of an MT x NT block; a group of MT NT / 64 threads covers the block, several groups share
// the k.  8 x 8 outputs per thread: four reads of shared memory, up to four cycles each, for 64 multiply-adds, 16 cycles of the SM.
__global__ void __launch_bounds__(kThreadsN) k_gemm_narrow_k(const NarrowK a) {
  dyb_grid_dep_sync();
  extern __shared__ __align__(16) float nsm[];
  const uint32_t tid = threadIdx.x, mt = a.MT / 8, nt = a.NT / 8, per = mt * nt;
  const uint32_t grp = tid / per, t = tid % per, mi = t % mt, ni = t / mt;
  const bool on = grp < a.groups;
  const bool rows_split = a.MT < a.M;   // the blocks of grid.y lie along M (else along N)
  const uint32_t m0 = rows_split ? blockIdx.y * a.MT : 0, n0 = rows_split ? 0 : blockIdx.y * a.NT;
  const uint32_t mn = min(a.MT, a.M - m0), nn = min(a.NT, a.N - n0);
  const uint32_t k_lo = blockIdx.x * a.kspan, k_hi = min(a.K, k_lo + a.kspan), pieces = (k_hi - k_lo + a.KC - 1) / a.KC;
  const uint32_t row = a.MT + a.NT, stage = a.KC * row;
  auto side = [&](float* dst, const float* src, uint32_t ld, uint32_t k0, uint32_t kn, uint32_t width, uint32_t have, int vec) {
    if (vec) {
      const uint32_t q = width / 4, step = kThreadsN / q;
      if (tid >= q * step) return;
      const uint32_t r = 4 * (tid % q), left = r < have ? min(4u, have - r) * 4 : 0;
      uint32_t k = tid / q;
      float* d = dst + k * row + r;
      const float* from = src + (left ? (size_t)ld * (k0 + k) + r : 0);
      for (; k < kn; k += step, d += step * row, from += left ? (size_t)ld * step : 0) cp_async16(d, from, left);
      for (; k < a.KC; k += step, d += step * row) cp_async16(d, src, 0);
    } else {
      for (uint32_t r = tid & 31; r < width; r += 32)
        for (uint32_t k = tid >> 5; k < a.KC; k += kThreadsN / 32) {
          const bool in = k < kn && r < have;
          cp_async4(dst + k * row + r, src + (in ? (size_t)ld * (k0 + k) + r : 0), in ? 4 : 0);
        }
    }
  };
  auto fetch = [&](uint32_t p) {
    if (p < pieces) {
      const uint32_t k0 = k_lo + p * a.KC, kn = min(a.KC, k_hi - k0);
      float* st = nsm + (size_t)(p % kStagesN) * stage;
      side(st, a.A + m0, a.lda, k0, kn, a.MT, mn, a.vec_a);
      side(st + a.MT, a.B + n0, a.ldb, k0, kn, a.NT, nn, a.vec_b);
    }
    cp_commit();
  };
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  fetch(0);
  fetch(1);
  for (uint32_t p = 0; p < pieces; ++p) {
    cp_wait<kStagesN - 2>();
    __syncthreads();
    fetch(p + 2);
    if (!on) continue;
    const float* st = nsm + (size_t)(p % kStagesN) * stage + grp * row + 4 * mi;
    const uint32_t to_y = 4 * mt, to_b = a.MT + 4 * ni - 4 * mi, to_d = to_b + 4 * nt;
#pragma unroll 4
    for (uint32_t k = grp; k < a.KC; k += a.groups, st += a.groups * row) {   // (k beyond the end are zeros)
      const float4 x = ld4(st), y = ld4(st + to_y), b = ld4(st + to_b), d = ld4(st + to_d);
      const float w[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w}, c[8] = {b.x, b.y, b.z, b.w, d.x, d.y, d.z, d.w};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(w[i], c[j], acc[i][j]);
    }
  }
  cp_wait<0>();
  const uint32_t outs = a.MT * a.NT;
  float* const out = a.part + (size_t)blockIdx.x * (a.meet ? 1 : a.groups) * a.M * a.N + m0 + (size_t)a.M * n0;
  if (!a.meet) {
    // every group's sums go out as they are: the launch that adds up the CTAs adds the groups too, in order
    if (!on) return;
    float* o = out + (size_t)grp * a.M * a.N;
    const bool quads = a.M % 4 == 0;   // (the partial products start on 16 bytes)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t n = 4 * (ni + j / 4 * nt) + j % 4;
      if (n >= nn) continue;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t m = 4 * (mi + h * mt);
        float* c = o + m + (size_t)a.M * n;
        if (quads) {
          if (m < mn) st4(c, make_float4(acc[4 * h][j], acc[4 * h + 1][j], acc[4 * h + 2][j], acc[4 * h + 3][j]));
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (m + i < mn) c[i] = acc[4 * h + i][j];
        }
      }
    }
    return;
  }
  // the groups' sums, then out: each output's group sums are added in group order
  __syncthreads();
  if (on) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        st4(nsm + (size_t)grp * outs + (size_t)(4 * (ni + j / 4 * nt) + j % 4) * a.MT + 4 * (mi + h * mt), make_float4(acc[4 * h][j], acc[4 * h + 1][j], acc[4 * h + 2][j], acc[4 * h + 3][j]));
  }
  __syncthreads();
  for (uint32_t e = tid; e < outs; e += kThreadsN) {
    const uint32_t m = e % a.MT, n = e / a.MT;
    if (m >= mn || n >= nn) continue;
    float s = nsm[e];
    for (uint32_t g = 1; g < a.groups; ++g) s += nsm[(size_t)g * outs + e];
    out[m + (size_t)a.M * n] = s;
  }
}

// C (+)= the sums of the CTAs, in order: 32 outputs per CTA, eight warps each add a stretch of the partial products.
__global__ void __launch_bounds__(256) k_narrow_reduce(const float* __restrict__ part, uint32_t S, uint32_t M, uint32_t N, float* __restrict__ C,
                                                       uint32_t ldc, int accumulate) {
  dyb_grid_dep_sync();
  __shared__ float red[8][33];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, e = blockIdx.x * 32 + lane, MN = M * N, per = (S + 7) / 8;
  float s = 0.f;
  if (e < MN) {
    const uint32_t hi = min(S, (w + 1) * per);
#pragma unroll 8
    for (uint32_t q = w * per; q < hi; ++q) s += __ldcs(part + (size_t)q * MN + e);
  }
  red[w][lane] = s;
  __syncthreads();
  if (w || e >= MN) return;
#pragma unroll
  for (int q = 1; q < 8; ++q) s += red[q][lane];
  float* c = C + e % M + (size_t)ldc * (e / M);
  *c = accumulate ? *c + s : s;
}

uint32_t up(uint32_t v, uint32_t step) { return (v + step - 1) / step * step; }

template <int ML, int NJ>
int launch_narrow(dyb200_ctx* ctx, Narrow a) {
  const uint32_t TN = kThreadsN / ML * NJ, tiles = (a.N + TN - 1) / TN, blocks = (a.M + 8 * ML - 1) / (8 * ML);
  // row blocks on CTAs of their own as long as there are fewer CTAs than SMs
  uint32_t per = blocks;
  while (per > 1 && (uint64_t)tiles * ((blocks + per - 1) / per) < (uint32_t)ctx->sm_count) per = (per + 1) / 2;
  a.MP = per * 8 * ML;
  const uint32_t by = (blocks + per - 1) / per;
  const size_t smem = sizeof(float) * ((size_t)a.K * a.MP + (size_t)kStagesN * TN * a.pitch);
  DYB_CUDA(ctx, dyb_smem_limit(k_gemm_narrow<ML, NJ>, smem, kSmemNarrow));
  const uint32_t per_sm = smem <= 72 * 1024 ? 3 : smem <= 110 * 1024 ? 2 : 1, cap = per_sm * (uint32_t)ctx->sm_count;
  dyb_launch(k_gemm_narrow<ML, NJ>, dim3(tiles < cap ? tiles : cap, by), kThreadsN, smem, ctx, a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

// -1: the tile does not fit shared memory
template <int ML, int NJ>
int launch_slices(dyb200_ctx* ctx, Slices a) {
  constexpr uint32_t MB = 8 * ML, WN = 32 / ML * NJ;
  const uint32_t sms = (uint32_t)ctx->sm_count;
  // slices by what the fullest SM has to do: whole rounds of tiles, 6 % more for each doubling (the sums' way through shared memory)
  double best = 0;
  size_t smem = 0;
  for (uint32_t KS = 1; KS <= 8 && (KS == 1 || 16 * KS <= up(a.K, 8)); KS *= 2) {
    const uint32_t TN = 8 / KS * WN, tiles = (a.N + TN - 1) / TN;
    // k per piece; floats per column of the slices' sums (rows stored one by one go by the buffer as well)
    const uint32_t most = KS == 8 ? 128 : 64, KC = a.K <= most ? up(a.K, 4 * KS) : most, need = KS > 1 || !a.vec_c ? KS * MB : 0;
    const uint32_t pitch = (((KC > need ? KC : need) + 3) / 4 | 1) * 4;
    const size_t bytes = sizeof(float) * ((size_t)a.K * MB + 2 * (size_t)TN * pitch);
    const double t = (double)((tiles + sms - 1) / sms) * TN * (KS == 1 ? 1.0 : KS == 2 ? 1.06 : KS == 4 ? 1.12 : 1.18);
    if (bytes > kSmemNarrow || (best != 0 && t >= best)) continue;
    best = t; smem = bytes;
    a.KS = KS; a.CS = 8 / KS; a.TN = TN; a.KC = KC; a.pitch = pitch; a.pieces = (a.K + KC - 1) / KC;
  }
  if (best == 0) return -1;
  DYB_CUDA(ctx, dyb_smem_limit(k_gemm_slices<ML, NJ>, smem, kSmemNarrow));
  const uint32_t tiles = (a.N + a.TN - 1) / a.TN, cap = (smem <= 72 * 1024 ? 3 : smem <= 110 * 1024 ? 2 : 1) * sms;
  dyb_launch(k_gemm_slices<ML, NJ>, tiles < cap ? tiles : cap, kThreadsN, smem, ctx, a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

// Row block: 32 rows, or 64 where that leaves less padding or reads the pieces less often.
uint32_t row_block(uint32_t M) { return M <= 32 || (M > kNarrow && up(M, 32) < up(M, 64)) ? 32 : 64; }

}  // namespace

// Few rows or a short reduction (one side at most 64) and a small operand that fits shared memory, with columns enough to fill the
// tiles; or a reduction of at least 256 with one output side at most 64 and the other at most 1024.  From 64 on the multiply-adds (M
// per element of the long operand, 2.9 ps at 64) cost more than splitting that element and a quarter-filled tensor tile (4 ps at
// any M).  Below 256 columns the tiles are too few to spread over the chip.
bool dyb200_narrow_takes(uint32_t M, uint32_t N, int npairs, const GemmPair* pairs, const GemmEpilogue& epi) {
  if (npairs != 1 || pairs[0].maskB || epi.split_m || pairs[0].K == 0) return false;
  const GemmPair& p = pairs[0];
  if (!p.transB) {
    if (epi.mode != EPI_STORE && epi.mode != EPI_BIAS && epi.mode != EPI_ACCUM) return false;
    return (M <= kNarrow || p.K <= kNarrow) && N >= 256 && N >= M && (uint64_t)up(M, row_block(M)) * p.K <= kSmallMax;
  }
  return !p.transA && (epi.mode == EPI_STORE || epi.mode == EPI_ACCUM) && (M <= kNarrow || N <= kNarrow) && M <= 1024 && N <= 1024 && p.K >= 256 && p.K >= M && p.K >= N;
}

int dyb200_gemm_narrow(dyb200_ctx* ctx, uint32_t M, uint32_t N, const GemmPair& p, const GemmEpilogue& epi) {
  GemmProfScope scope(ctx, 2.0 * M * N * p.K, 0, M, N, p.K, (uint32_t)epi.mode);
  if (!p.transB) {
    const uint32_t mb = row_block(M);
    if (p.K > 64) {   // (M <= 64)
      Slices a{p.A, p.B, p.lda, p.ldb, p.transA, M, N, p.K, 0, 0, 0, 0, 0, 0, 0, 0, epi.C, epi.ldc, epi.bias, epi.mode};
      a.vec_b = p.ldb % 4 == 0 && aligned16(p.B);
      a.vec_c = epi.ldc % 4 == 0 && M % 4 == 0 && aligned16(epi.C) && (epi.mode != EPI_BIAS || aligned16(epi.bias));
      // eight columns per lane, fewer where those tiles would leave SMs without one or do not fit
      const uint32_t sms = (uint32_t)ctx->sm_count;
      int rc = -1;
      for (uint32_t nj = 8; nj >= 1 && rc == -1; nj /= 2) {
        if (nj > 1 && (uint64_t)N < (uint64_t)sms * nj * (mb == 32 ? 8 : 4)) continue;
        if (mb == 32) rc = nj == 8 ? launch_slices<4, 8>(ctx, a) : nj == 4 ? launch_slices<4, 4>(ctx, a) : nj == 2 ? launch_slices<4, 2>(ctx, a) : launch_slices<4, 1>(ctx, a);
        else rc = nj == 8 ? launch_slices<8, 8>(ctx, a) : nj == 4 ? launch_slices<8, 4>(ctx, a) : nj == 2 ? launch_slices<8, 2>(ctx, a) : launch_slices<8, 1>(ctx, a);
      }
      return rc == -1 ? dyb200_fail(ctx, DYB200_ERUNTIME, "narrow product: %u x %u x %u does not fit shared memory", M, N, p.K) : rc;
    }
    Narrow a{p.A, p.B, p.lda, p.ldb, p.transA, M, N, p.K, 0, 0, 0, 0, 0, epi.C, epi.ldc, epi.bias, epi.mode};
    // one piece holds the whole reduction when there are several row blocks (then it is at most 64 long)
    const bool several = M > mb;
    
    a.vec_b = p.ldb % 4 == 0 && aligned16(p.B);
    a.vec_c = epi.ldc % 4 == 0 && M % 4 == 0 && aligned16(epi.C) && (epi.mode != EPI_BIAS || aligned16(epi.bias));
    // tiles of 256 columns (128 when pieces are long), or narrower ones where those would leave SMs without a tile
    const uint32_t sms = (uint32_t)ctx->sm_count;
    const bool wide = N >= 192u * sms, mid = N >= (mb == 32 ? 64u : 32u) * sms;
    const uint32_t most = wide ? 16 : mid ? 32 : 64;   // (20 KB a piece at most)
    a.KC = several || p.K <= most ? up(p.K, 4) : most;
    a.pitch = (a.KC / 4 | 1) * 4;
    if (mb == 32) return wide ? (several ? launch_narrow<4, 2>(ctx, a) : launch_narrow<4, 4>(ctx, a)) : mid ? launch_narrow<4, 2>(ctx, a) : launch_narrow<4, 1>(ctx, a);
    return wide ? (several ? launch_narrow<8, 4>(ctx, a) : launch_narrow<8, 8>(ctx, a)) : mid ? launch_narrow<8, 2>(ctx, a) : launch_narrow<8, 1>(ctx, a);
  }
  NarrowK a;
  a.A = p.A; a.B = p.B; a.lda = p.lda; a.ldb = p.ldb; a.M = M; a.N = N; a.K = p.K;
  if (M <= kNarrow) {
    a.MT = up(M, 8);
    const uint32_t most = kTilesMax / (a.MT / 8) * 8, blocks = (N + most - 1) / most;
    a.NT = up((N + blocks - 1) / blocks, 8);
  } else {
    a.NT = up(N, 8);
    const uint32_t most = kTilesMax / (a.NT / 8) * 8, blocks = (M + most - 1) / most;
    a.MT = up((M + blocks - 1) / blocks, 8);
  }
  const uint32_t by = M <= kNarrow ? (N + a.NT - 1) / a.NT : (M + a.MT - 1) / a.MT;
  a.groups = kThreadsN / (a.MT / 8 * (a.NT / 8));
  // Two groups or one write their sums as they are: where the outputs are many, meeting in shared memory and a thread adding the groups of 32 outputs one after the
  // other took longer than twice the partial products do (us: 32 x 256 x 520 11.3 / 5.7, x 13 400 27.2 / 20.6, x 107 000 80 / 66, the last with pieces of 32 KB and
  // addresses that walk; with 10 groups of 48 x 32 meeting is the faster one, 7.8 / 14.6 at 520).
  a.meet = a.groups > 2;
  a.vec_a = p.lda % 4 == 0 && aligned16(p.A);
  a.vec_b = p.ldb % 4 == 0 && aligned16(p.B);
  uint32_t gx;
  void* part;
  auto cut = [&]() {
    a.KC = a.meet ? up(4096 / (a.MT + a.NT), a.groups) : up(8192 / (a.MT + a.NT), 4 * a.groups);   // 16 or 32 KB a piece
    gx = 2 * (uint32_t)ctx->sm_count / by;
    if (gx < 1) gx = 1;
    a.kspan = up((p.K + gx - 1) / gx, a.KC);
    gx = (p.K + a.kspan - 1) / a.kspan;
    return dyb200_scratch(ctx, (size_t)gx * (a.meet ? 1 : a.groups) * M * N * sizeof(float), &part);
  };
  int rc = cut();
  if (rc == DYB200_ENOMEM && !a.meet) {   // (half as much, up to 10 MB, may still fit)
    a.meet = 1;
    rc = cut();
  }
  if (rc) return rc;
  a.part = (float*)part;
  const size_t ring = (size_t)kStagesN * a.KC * (a.MT + a.NT), sums = a.meet ? (size_t)a.groups * a.MT * a.NT : 0;
  const size_t smem = sizeof(float) * (ring > sums ? ring : sums);
  DYB_CUDA(ctx, dyb_smem_limit(k_gemm_narrow_k, smem, kSmemNarrow));
  dyb_launch(k_gemm_narrow_k, dim3(gx, by), kThreadsN, smem, ctx, a);
  DYB_LAUNCHED(ctx);
  dyb_launch(k_narrow_reduce, (M * N + 31) / 32, 256, 0, ctx, (const float*)a.part, gx * (a.meet ? 1 : a.groups), M, N, epi.C, epi.ldc, epi.mode == EPI_ACCUM ? 1 : 0);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}
