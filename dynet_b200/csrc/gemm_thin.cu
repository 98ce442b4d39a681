// Products with few columns: C[M x N] = epilogue(A0 B0 (+ A1 B1)), A column-major, N <= 32 - one token at a time of a text
// generator, the small batches of a test run, the last steps of a ragged batch.
//
// What bounds it: every weight is used N times, so the product is one pass over A (from L2 when the model fits there).  The
// tensor path moved 128-row tiles of 64 columns, nearly all of them padding, out of split operand planes of twice the bytes,
// after a launch that split B: 17 + 2 us for the 4096 x 1 x 2048 gate product of a 1024-unit layer and 25 us for a
// 10000 x 1 x 1024 projection.  Here A is read once, as it lies, in fp32 with plain multiply-adds: a CTA owns 32 rows (the four
// gates of 8 hidden units, or 32 consecutive rows), 8 lanes x 16 bytes cover them for one k, the other lanes and warps take
// other k; two batches of eight 16-byte loads are in
// flight per thread, the first of them before B is fetched.  Plain products of up to four columns share their rows out evenly over the SMs
// instead (thin_launch).  B (all of its k, N columns) sits in shared memory as [k][column], so
// that a thread gets the N factors of a k with 16-byte loads that the warp shares.  The partial sums of the k lanes meet by
// shuffles, those of the warps in shared memory as a tree: the result does not depend on the run.
// Up to 16 columns per CTA (64 sums per thread); beyond that a second column of CTAs reads A again (from L2).
#include "gemm.cuh"

namespace {

constexpr uint32_t kRows = 32;      // rows per CTA
// the longest reduction: B has to fit in shared memory (160 KB at most)
constexpr uint32_t thin_k_max(uint32_t n) { return n > 8 ? 2560u : n > 4 ? 4096u : 8192u; }

struct ThinPair {
  const float* A; uint32_t lda, K; const float* B; uint32_t ldb; const float* mask; uint32_t mask_ld; int mask_full;
  int vec;                          // B and its mask can be read 16 bytes at a time when the pair's first k is a multiple of 4
};
struct ThinArgs {
  ThinPair p[2];
  int npairs, mode, pre_in_c;       // pre_in_c: (gates) C holds the rest of the pre-activation, bias included
  uint32_t M, N, quads;             // quads: (up to kFlexColumns) groups of four rows per CTA
  float* C; uint32_t ldc;
  const float* bias; uint32_t H; float fb;
  const float* c_prev; float *c_out, *h_out;        // gates with the cell update (null: gates only)
  float *hn_hi, *hn_lo; uint32_t hn_pitch; const float* hmask; uint32_t hmask_ld; int hmask_full;
};

// A thread's walk over its k's (`step` apart, pair 0 and then pair 1), one batch of IN loads after another
struct ThinCursor { const float* p; size_t stride; uint32_t k, K, off; };   // next address; elements to the next k; k, end of the pair, its first row of xs
template <int IN, bool VEC>
__device__ __forceinline__ void thin_load(ThinCursor& c, uint32_t step, float4 (&w)[IN]) {
  const float* p = c.p;
  if (c.k + (IN - 1) * step < c.K) {
#pragma unroll
    for (int j = 0; j < IN; ++j, p += c.stride) {
      if (VEC) w[j] = __ldg(reinterpret_cast<const float4*>(p));
      else w[j].x = __ldg(p);
    }
  } else {
#pragma unroll
    for (int j = 0; j < IN; ++j, p += c.stride)
      if (c.k + j * step < c.K) {
        if (VEC) w[j] = __ldg(reinterpret_cast<const float4*>(p));
        else w[j].x = __ldg(p);
      }
  }
  c.p = p;
}
// the multiply-adds on a batch whose first k is k (row k of xs, `step` rows apart)
template <int NB, int IN, bool VEC>
__device__ __forceinline__ void thin_fma(const float4 (&w)[IN], uint32_t k, uint32_t K, uint32_t step, const float* xs, float (&acc)[VEC ? 4 : 1][NB]) {
  const float* xp = xs + (size_t)k * NB;
#pragma unroll
  for (int j = 0; j < IN; ++j, xp += step * NB) {
    if (k + j * step >= K) break;
    float x[NB];
    if (NB % 4 == 0) {
#pragma unroll
      for (int c = 0; c < NB / 4; ++c) {
        const float4 v = ld4(xp + 4 * c);
        x[4 * c] = v.x; x[4 * c + 1] = v.y; x[4 * c + 2] = v.z; x[4 * c + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int c = 0; c < NB; ++c) x[c] = xp[c];
    }
#pragma unroll
    for (int c = 0; c < NB; ++c) {
      acc[0][c] = fmaf(w[j].x, x[c], acc[0][c]);
      if (VEC) {
        acc[VEC ? 1 : 0][c] = fmaf(w[j].y, x[c], acc[VEC ? 1 : 0][c]);
        acc[VEC ? 2 : 0][c] = fmaf(w[j].z, x[c], acc[VEC ? 2 : 0][c]);
        acc[VEC ? 3 : 0][c] = fmaf(w[j].w, x[c], acc[VEC ? 3 : 0][c]);
      }
    }
  }
}

// four consecutive k (`left` of them exist) of column n of B .* mask, the reduction running over pair 0 and then pair 1
__device__ __forceinline__ float4 thin_b(const ThinArgs& a, uint32_t kg, uint32_t left, uint32_t K0, uint32_t n) {
  float v[4] = {0.f, 0.f, 0.f, 0.f}, m[4] = {1.f, 1.f, 1.f, 1.f};
  const bool second = kg >= K0;
  const ThinPair& p = a.p[second];
  if (left == 4 && p.vec && (second || kg + 4 <= K0)) {
    const uint32_t k = second ? kg - K0 : kg;
    const float4 x = ld4(p.B + k + (size_t)p.ldb * n);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
    if (p.mask) { const float4 y = ld4(p.mask + k + (p.mask_full ? (size_t)p.mask_ld * n : 0)); m[0] = y.x; m[1] = y.y; m[2] = y.z; m[3] = y.w; }
  } else {
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i)
      if (i < left) {
        const ThinPair& q = a.p[kg + i >= K0];
        const uint32_t k = kg + i >= K0 ? kg + i - K0 : kg + i;
        v[i] = q.B[k + (size_t)q.ldb * n];
        if (q.mask) m[i] = q.mask[k + (q.mask_full ? (size_t)q.mask_ld * n : 0)];
      }
  }
  return make_float4(v[0] * m[0], v[1] * m[1], v[2] * m[2], v[3] * m[3]);
}

// Plain products of up to four columns: any number of row quads per CTA, so that one CTA per SM takes an equal share of the rows.
constexpr uint32_t kFlexColumns = 4;

// grid (row blocks, column blocks); 256 or 512 threads
template <int NB, bool GATES, bool VEC>
__global__ void __launch_bounds__(512, 1) k_gemm_thin(const __grid_constant__ ThinArgs a) {
  extern __shared__ __align__(16) float thin_smem[];
  // No early launch of the dependent kernel: the CTAs of a following product would settle two and more on the SMs that this one leaves free
  // and read their shares of the weights from there (a token of a 2-layer, 1024-unit generator: 40.4 us with it, 31.5 without).
  dyb_grid_dep_wait();
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x / 32, n0 = blockIdx.y * NB;
  // row of the CTA's 32 that this thread's first value belongs to
  constexpr bool FLEX = VEC && !GATES && NB <= kFlexColumns;
  const uint32_t quads = FLEX ? a.quads : 8u, rows = FLEX ? 4 * quads : kRows;
  const uint32_t r = VEC ? 4 * (FLEX ? tid % quads : tid & 7) : lane;
  const uint32_t u = blockIdx.x * 8 + r % 8, m = GATES ? (r / 8) * a.H + u : blockIdx.x * rows + r;
  float acc[VEC ? 4 : 1][NB];
#pragma unroll
  for (int i = 0; i < (VEC ? 4 : 1); ++i)
#pragma unroll
    for (int c = 0; c < NB; ++c) acc[i][c] = 0.f;
  constexpr int IN = NB >= 16 && VEC ? 4 : 8;   // loads per batch; two batches are on their way at any time
  const uint32_t sub = VEC ? tid / quads : warp, step = VEC ? blockDim.x / quads : warps;
  const bool row_live = (GATES ? u < a.H : m < a.M) && sub < step;
  const uint32_t K0 = a.p[0].K, K = a.npairs > 1 ? K0 + a.p[1].K : K0;
  ThinCursor cur;
  auto pair_start = [&](int q) {
    cur.p = a.p[q].A + m + (size_t)a.p[q].lda * sub;
    cur.stride = (size_t)a.p[q].lda * step;
    cur.off = q ? K0 : 0;
    cur.k = sub;
    cur.K = row_live ? a.p[q].K : 0;
  };
  // the next batch into w: its first row of xs and the end of its pair there (equal: there is none left)
  auto next = [&](float4 (&w)[IN], uint32_t& k, uint32_t& kend) {
    if (cur.k >= cur.K && cur.off == 0 && a.npairs > 1) pair_start(1);
    k = cur.off + cur.k;
    kend = cur.off + cur.K;
    if (cur.k < cur.K) {
      thin_load<IN, VEC>(cur, step, w);
      cur.k += IN * step;
    }
  };
  float4 w0[IN], w1[IN];
  uint32_t k0, e0, k1, e1;
  pair_start(0);
  next(w0, k0, e0);   // (on their way while B is fetched)
  next(w1, k1, e1);
  // gates: what the thread that finishes (unit tid % 8, column tid / 8) adds, fetched now
  const uint32_t f_u = blockIdx.x * 8 + tid % 8, f_n = n0 + tid / 8;
  const bool f_live = GATES && tid < 8 * NB && f_u < a.H && f_n < a.N;
  float f_pre[4] = {0.f, 0.f, 0.f, 0.f}, f_c = 0.f, f_m = 1.f;
  if (f_live) {
    const float* g = a.pre_in_c ? a.C + f_u + (size_t)a.ldc * f_n : a.bias + f_u;
#pragma unroll
    for (int q = 0; q < 4; ++q) f_pre[q] = g[(size_t)q * a.H];
    if (a.c_out) f_c = a.c_prev[f_u + (size_t)a.H * f_n];
    if (a.hn_hi && a.hmask) f_m = a.hmask[f_u + (a.hmask_full ? (size_t)a.hmask_ld * f_n : 0)];
  }
  // B as [k][column]: an item is four consecutive k of one column, four items per thread on their way at a time (one by one they
  // cost a latency of L2 each, 3 us in all)
  const uint32_t items = (K + 3) / 4 * NB;
  for (uint32_t i0 = tid; i0 < items; i0 += 4 * blockDim.x) {
    float4 v[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const uint32_t e = i0 + x * blockDim.x, n = n0 + e % NB, kg = e / NB * 4;
      v[x] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (e < items && n < a.N) v[x] = thin_b(a, kg, min(K - kg, 4u), K0, n);
    }
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const uint32_t e = i0 + x * blockDim.x;
      if (e < items) {
        float* dst = thin_smem + (size_t)(e / NB * 4) * NB + e % NB;
        if (NB == 1) st4(dst, v[x]);
        else { dst[0] = v[x].x; dst[NB] = v[x].y; dst[2 * NB] = v[x].z; dst[3 * NB] = v[x].w; }
      }
    }
  }
  __syncthreads();
  while (k0 < e0) {
    thin_fma<NB, IN, VEC>(w0, k0, e0, step, thin_smem, acc);
    next(w0, k0, e0);
    if (k1 < e1) thin_fma<NB, IN, VEC>(w1, k1, e1, step, thin_smem, acc);
    next(w1, k1, e1);
  }
  if (k1 < e1) thin_fma<NB, IN, VEC>(w1, k1, e1, step, thin_smem, acc);
  if (FLEX) {   // the k lanes of a warp by shuffles where its quads divide it, the rest in order, one thread per (column, row)
    uint32_t parts = step, part = sub;
    bool holds = sub < step;
    if (32 % quads == 0) {
      for (uint32_t d = quads; d < 32; d <<= 1)
#pragma unroll
        for (int i = 0; i < (VEC ? 4 : 1); ++i)
#pragma unroll
          for (int c = 0; c < NB; ++c) acc[i][c] += __shfl_xor_sync(0xffffffffu, acc[i][c], d);
      parts = warps; part = warp; holds = lane < quads;
    }
    __syncthreads();
    float* red = thin_smem;   // [column][row][parts, odd pitch]
    const uint32_t rp = parts | 1;
    if (holds) {
#pragma unroll
      for (int c = 0; c < NB; ++c)
#pragma unroll
        for (int i = 0; i < (VEC ? 4 : 1); ++i) red[(size_t)(c * rows + r + i) * rp + part] = acc[i][c];
    }
    __syncthreads();
    for (uint32_t e = tid; e < rows * NB; e += blockDim.x) {
      const uint32_t mm = blockIdx.x * rows + e % rows, n = n0 + e / rows;
      if (mm >= a.M || n >= a.N) continue;
      float v = 0.f;
#pragma unroll 8
      for (uint32_t k = 0; k < parts; ++k) v += red[(size_t)e * rp + k];
      float* dst = a.C + mm + (size_t)a.ldc * n;
      if (a.mode == EPI_BIAS) v += a.bias[mm];
      else if (a.mode == EPI_ACCUM) v += *dst;
      *dst = v;
    }
    return;
  }
  // the k lanes of a warp (VEC: lanes 8 j + s hold rows 4 s .. 4 s + 3), then the warps in order
  if (VEC) {
#pragma unroll
    for (int i = 0; i < (VEC ? 4 : 1); ++i)
#pragma unroll
      for (int c = 0; c < NB; ++c) {
        acc[i][c] += __shfl_xor_sync(0xffffffffu, acc[i][c], 8);
        acc[i][c] += __shfl_xor_sync(0xffffffffu, acc[i][c], 16);
      }
  }
  __syncthreads();
  float* red = thin_smem;   // [column][row][warps + 1]
  const uint32_t rp = warps + 1;
  if (!VEC || lane < 8) {
#pragma unroll
    for (int c = 0; c < NB; ++c)
#pragma unroll
      for (int i = 0; i < (VEC ? 4 : 1); ++i) red[((size_t)c * kRows + r + i) * rp + warp] = acc[i][c];
  }
  __syncthreads();
  // one thread per (column, row, warp) value: a tree over the warps, the total left at [column][row][0]
  for (uint32_t e0 = 0; e0 < kRows * NB * warps; e0 += blockDim.x) {
    const uint32_t o = (e0 + tid) / warps, w = tid % warps;
    float v = red[(size_t)o * rp + w];
    for (uint32_t d = warps / 2; d >= 1; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    if (w == 0) red[(size_t)o * rp] = v;
  }
  __syncthreads();
  if (GATES) {
    if (f_live) {
      float z[4];
      float* g = a.C + f_u + (size_t)a.ldc * f_n;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float v = red[((size_t)(tid / 8) * kRows + 8 * q + tid % 8) * rp] + f_pre[q];
        if (q == 1) v += a.fb;
        z[q] = q == 3 ? gate_tanh(v) : gate_sigmoid(v);
        g[(size_t)q * a.H] = z[q];
      }
      if (a.c_out) {
        const size_t ei = f_u + (size_t)a.H * f_n;
        const float cn = lstm_cell_c(z[0], z[3], z[1], f_c), hv = lstm_cell_h(z[2], cn);
        a.c_out[ei] = cn;
        a.h_out[ei] = hv;
        if (a.hn_hi) {
          float hi, lo;
          split_tf32(a.hmask ? hv * f_m : hv, hi, lo);
          a.hn_hi[(size_t)f_n * a.hn_pitch + f_u] = hi;
          a.hn_lo[(size_t)f_n * a.hn_pitch + f_u] = lo;
        }
      }
    }
  } else {
    for (uint32_t e = tid; e < kRows * NB; e += blockDim.x) {
      const uint32_t c = e / kRows, rr = e % kRows, mm = blockIdx.x * kRows + rr, n = n0 + c;
      if (mm >= a.M || n >= a.N) continue;
      float v = red[(size_t)e * rp];
      float* dst = a.C + mm + (size_t)a.ldc * n;
      if (a.mode == EPI_BIAS) v += a.bias[mm];
      else if (a.mode == EPI_ACCUM) v += *dst;
      *dst = v;
    }
  }
}

template <bool GATES, bool VEC>
void (*thin_kernel(uint32_t nb))(ThinArgs) {
  switch (nb) {
    case 1: return k_gemm_thin<1, GATES, VEC>;
    case 2: return k_gemm_thin<2, GATES, VEC>;
    case 4: return k_gemm_thin<4, GATES, VEC>;
    case 8: return k_gemm_thin<8, GATES, VEC>;
    default: return k_gemm_thin<16, GATES, VEC>;
  }
}

int thin_launch(dyb200_ctx* ctx, ThinArgs& a, bool gates, double flops) {
  uint32_t nb = 1;
  while (nb < a.N && nb < 16) nb *= 2;
  bool vec = gates ? a.H % 4 == 0 : a.M % 4 == 0;
  uint32_t ktot = 0;
  for (int q = 0; q < a.npairs; ++q) {
    vec = vec && a.p[q].lda % 4 == 0 && aligned16(a.p[q].A);
    a.p[q].vec = ktot % 4 == 0 && a.p[q].ldb % 4 == 0 && aligned16(a.p[q].B) &&
                 (!a.p[q].mask || (aligned16(a.p[q].mask) && (!a.p[q].mask_full || a.p[q].mask_ld % 4 == 0)));
    ktot += a.p[q].K;
  }
  uint32_t blocks = gates ? (a.H + 7) / 8 : (a.M + kRows - 1) / kRows;
  uint32_t threads = blocks <= (uint32_t)ctx->sm_count ? 512u : 256u;   // (one CTA per SM: more loads in flight from it)
  size_t red = (size_t)(threads / 32 + 1) * nb * kRows * 4;
  if (vec && !gates && nb <= kFlexColumns) {
    // One CTA of 512 threads per SM with up to 32 quads of rows, at least 32 bytes of a column; more rows in whole rounds of two CTAs per
    // SM.  (us for 1 / 4 columns, against CTAs of 32 rows whatever the number of rows: 10000 x 1024 10.2 / 12.1 against 12.3 / 17.3 in
    // 313 CTAs, 50000 x 128 8.3 / 10.5 against 13.7 / 20.7, 1024 x 4096 6.4 / 9.9 against 10.2 / 15.5 in 32 CTAs.)
    const uint32_t sms = (uint32_t)ctx->sm_count, all = a.M / 4;
    a.quads = (all + sms - 1) / sms;
    threads = 512;
    if (a.quads <= 8) a.quads = a.quads <= 2 ? 2 : a.quads <= 4 ? 4 : 8;   // (so that shuffles add up a warp's k lanes)
    if (a.quads > 32) {
      threads = 256;
      const uint32_t rounds = (all + 64 * sms - 1) / (64 * sms);
      a.quads = (all + 2 * sms * rounds - 1) / (2 * sms * rounds);
    }
    blocks = (all + a.quads - 1) / a.quads;
    red = (size_t)((threads / a.quads) | 1) * nb * 4 * a.quads * 4;
  }
  const size_t xs = (size_t)(ktot + 3) / 4 * 4 * nb * 4;
  const size_t smem = xs > red ? xs : red;
  void (*k)(ThinArgs) = gates ? (vec ? thin_kernel<true, true>(nb) : thin_kernel<true, false>(nb))
                              : (vec ? thin_kernel<false, true>(nb) : thin_kernel<false, false>(nb));
  DYB_CUDA(ctx, dyb_smem_limit(k, smem, 160 * 1024));
  GemmProfScope scope(ctx, flops, 0, a.M, a.N, a.p[0].K + (a.npairs > 1 ? a.p[1].K : 0), (uint32_t)a.mode);
  dyb_launch(k, dim3(blocks, (a.N + nb - 1) / nb), threads, smem, ctx, a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

}  // namespace

// Measured (us per call, this path / the tensor path with its operand split): 4096 x N x 2048: N = 1 8.2 / 19, N = 4 12.6 / 19,
// N = 8 18.5 / 20, N = 16 30 / 21; 4096 x N x 1024: 8 12.3 / 18, 16 18.5 / 18; 10000 x N x 1024: 4 18.5 / 28, 8 29 / 29; 1024 x N x 512:
// 32 12 / 18.  So: at most 32 columns and 64 M multiply-adds (0.2 us per million from 4.5 us on).  A long reduction over few rows
// has too few CTAs here and stays with the K-split forms.
bool dyb200_thin_columns(uint32_t M, uint32_t N, uint32_t K) { return N <= 32 && K <= thin_k_max(N) && (double)M * N * K <= 64.0 * 1048576.0; }

bool dyb200_thin_takes(uint32_t M, uint32_t N, int npairs, const GemmPair* pairs, const GemmEpilogue& epi) {
  if (epi.split_m || (epi.mode != EPI_STORE && epi.mode != EPI_BIAS && epi.mode != EPI_ACCUM && epi.mode != EPI_GATES)) return false;
  uint64_t K = 0;
  for (int p = 0; p < npairs; ++p) {
    if (pairs[p].transA || pairs[p].transB || pairs[p].K == 0 || N > 32) return false;
    K += pairs[p].K;
  }
  return dyb200_thin_columns(M, N, (uint32_t)K) && (K <= 8ull * M || K <= 256);
}

int dyb200_gemm_thin(dyb200_ctx* ctx, uint32_t M, uint32_t N, int npairs, const GemmPair* pairs, const GemmEpilogue& epi) {
  ThinArgs a;
  memset(&a, 0, sizeof(a));
  double flops = 0;
  for (int p = 0; p < npairs; ++p) {
    const GemmPair& g = pairs[p];
    a.p[p] = ThinPair{g.A, g.lda, g.K, g.B, g.ldb, g.maskB, g.mask_ld, g.mask_full, 0};
    flops += 2.0 * M * N * g.K;
  }
  a.npairs = npairs; a.mode = epi.mode; a.M = M; a.N = N; a.C = epi.C; a.ldc = epi.ldc; a.bias = epi.bias; a.H = epi.H; a.fb = epi.forget_bias;
  return thin_launch(ctx, a, epi.mode == EPI_GATES, flops);
}

int dyb200_lstm_thin(dyb200_ctx* ctx, uint32_t H, uint32_t B, int npairs, const GemmPair* pairs, int pre_in_gates, const GemmEpilogue& epi) {
  ThinArgs a;
  memset(&a, 0, sizeof(a));
  double flops = 0;
  for (int p = 0; p < npairs; ++p) {
    const GemmPair& g = pairs[p];
    a.p[p] = ThinPair{g.A, g.lda, g.K, g.B, g.ldb, g.maskB, g.mask_ld, g.mask_full, 0};
    flops += 8.0 * H * B * g.K;
  }
  a.npairs = npairs; a.mode = EPI_LSTM_CELL; a.pre_in_c = pre_in_gates; a.M = 4 * H; a.N = B; a.C = epi.C; a.ldc = epi.ldc;
  a.bias = epi.bias; a.H = H; a.fb = epi.forget_bias; a.c_prev = epi.c_prev; a.c_out = epi.c_out; a.h_out = epi.h_out;
  a.hn_hi = epi.hn_hi; a.hn_lo = epi.hn_lo; a.hn_pitch = epi.hn_pitch;
  a.hmask = epi.hmask; a.hmask_ld = epi.hmask_ld; a.hmask_full = epi.hmask_full;
  return thin_launch(ctx, a, true, flops);
}
