// Products with few columns: C[M x N] = epilogue(A0 B0 (+ A1 B1)), A column-major, N <= 32 - one token at a time of a text
// generator, the small batches of a test run, the last steps of a ragged batch.
//
// What bounds it: every weight is used N times, so the product is one pass over A (from L2 when the model fits there).  The
// tensor path moved 128-row tiles of 64 columns, nearly all of them padding, out of split operand planes of twice the bytes,
// after a launch that split B: 17 + 2 us for the 4096 x 1 x 2048 gate product of a 1024-unit layer and 25 us for a
// 10000 x 1 x 1024 projection.  Here A is read once, as it lies, in fp32 with plain multiply-adds: a CTA owns 32 rows (the four
// gates of 8 hidden units, or 32 consecutive rows), 8 lanes x 16 bytes cover them for one k, the other lanes and warps take
// other k; eight 16-byte loads are in flight per thread.  B (all of its k, N columns) sits in shared memory as [k][column], so
// that a thread gets the N factors of a k with 16-byte loads that the warp shares.  The partial sums of the k lanes meet by
// shuffles, those of the warps in shared memory in warp order: the result does not depend on the run.
// Up to 16 columns per CTA (64 sums per thread); beyond that a second column of CTAs reads A again (from L2).
#include "gemm.cuh"

namespace {

constexpr uint32_t kRows = 32;      // rows per CTA
constexpr uint32_t kChunk = 2048;   // reduction elements of B in shared memory at a time

struct ThinPair { const float* A; uint32_t lda, K; const float* B; uint32_t ldb; const float* mask; uint32_t mask_ld; int mask_full; };
struct ThinArgs {
  ThinPair p[2];
  int npairs, mode, pre_in_c;       // pre_in_c: (gates) C holds the rest of the pre-activation, bias included
  uint32_t M, N;
  float* C; uint32_t ldc;
  const float* bias; uint32_t H; float fb;
  const float* c_prev; float *c_out, *h_out;        // gates with the cell update (null: gates only)
  float *hn_hi, *hn_lo; uint32_t hn_pitch; const float* hmask; uint32_t hmask_ld; int hmask_full;
};

// one pair over k in [k_lo, k_hi) (xs holds B from k_lo on)
template <int NB, bool VEC>
__device__ __forceinline__ void thin_pass(const float* __restrict__ A, uint32_t lda, bool row_live, uint32_t k_lo, uint32_t k_hi, const float* xs,
                                          float (&acc)[VEC ? 4 : 1][NB]) {
  const uint32_t sub = VEC ? threadIdx.x / 8 : threadIdx.x / 32, step = VEC ? blockDim.x / 8 : blockDim.x / 32;
  constexpr int kIn = VEC ? 8 : 16;   // loads in flight
  if (!row_live) return;
  for (uint32_t k0 = k_lo + sub; k0 < k_hi; k0 += kIn * step) {
    float4 w[kIn];
#pragma unroll
    for (int j = 0; j < kIn; ++j) {
      const uint32_t k = k0 + j * step;
      if (VEC) w[j] = k < k_hi ? __ldg(reinterpret_cast<const float4*>(A + (size_t)lda * k)) : make_float4(0.f, 0.f, 0.f, 0.f);
      else w[j].x = k < k_hi ? __ldg(A + (size_t)lda * k) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < kIn; ++j) {
      const uint32_t k = k0 + j * step;
      if (k < k_hi) {
        const float* xp = xs + (size_t)(k - k_lo) * NB;
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
  }
}

// grid (row blocks, column blocks); 256 or 512 threads
template <int NB, bool GATES, bool VEC>
__global__ void __launch_bounds__(512, NB <= 4 ? 2 : 1) k_gemm_thin(const __grid_constant__ ThinArgs a) {
  extern __shared__ __align__(16) float thin_smem[];
  dyb_grid_dep_sync();
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x / 32, n0 = blockIdx.y * NB;
  // row of the CTA's 32 that this thread's first value belongs to
  const uint32_t r = VEC ? 4 * (tid & 7) : lane;
  const uint32_t u = blockIdx.x * 8 + r % 8, m = GATES ? (r / 8) * a.H + u : blockIdx.x * kRows + r;
  const bool row_live = GATES ? u < a.H : m < a.M;
  float acc[VEC ? 4 : 1][NB];
#pragma unroll
  for (int i = 0; i < (VEC ? 4 : 1); ++i)
#pragma unroll
    for (int c = 0; c < NB; ++c) acc[i][c] = 0.f;
  for (int q = 0; q < a.npairs; ++q) {
    const ThinPair& p = a.p[q];
    for (uint32_t k0 = 0; k0 < p.K; k0 += kChunk) {
      const uint32_t kn = min(kChunk, p.K - k0);
      if (q || k0) __syncthreads();
      // (a warp takes CL columns x 32 / CL consecutive k: its stores are contiguous, or two-way conflicts with 16 columns)
      constexpr uint32_t CL = NB < 8 ? NB : 8, KL = 32 / CL, CB = NB / CL;
      for (uint32_t e = tid; e < (kn + KL - 1) / KL * KL * NB; e += blockDim.x) {
        const uint32_t c = e % CL + CL * (e / 32 % CB), k = e % 32 / CL + KL * (e / 32 / CB), n = n0 + c;
        if (k >= kn) continue;
        float v = 0.f;
        if (n < a.N) {
          v = p.B[k0 + k + (size_t)p.ldb * n];
          if (p.mask) v *= p.mask[k0 + k + (p.mask_full ? (size_t)p.mask_ld * n : 0)];
        }
        thin_smem[(size_t)k * NB + c] = v;
      }
      __syncthreads();
      thin_pass<NB, VEC>(p.A + m, p.lda, row_live, k0, k0 + kn, thin_smem, acc);
    }
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
  float* red = thin_smem;   // [warp][column][32 rows]
  if (!VEC || lane < 8) {
#pragma unroll
    for (int c = 0; c < NB; ++c)
#pragma unroll
      for (int i = 0; i < (VEC ? 4 : 1); ++i) red[((size_t)warp * NB + c) * kRows + r + i] = acc[i][c];
  }
  __syncthreads();
  if (GATES) {
    for (uint32_t e = tid; e < 8 * NB; e += blockDim.x) {
      const uint32_t c = e / 8, ul = e % 8, uu = blockIdx.x * 8 + ul, n = n0 + c;
      if (uu >= a.H || n >= a.N) continue;
      float z[4];
      float* g = a.C + uu + (size_t)a.ldc * n;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float v = 0.f;
        for (uint32_t w = 0; w < warps; ++w) v += red[((size_t)w * NB + c) * kRows + 8 * q + ul];
        v += a.pre_in_c ? g[(size_t)q * a.H] : a.bias[(size_t)q * a.H + uu];
        if (q == 1) v += a.fb;
        z[q] = q == 3 ? gate_tanh(v) : gate_sigmoid(v);
        g[(size_t)q * a.H] = z[q];
      }
      if (a.c_out) {
        const size_t ei = uu + (size_t)a.H * n;
        const float cn = lstm_cell_c(z[0], z[3], z[1], a.c_prev[ei]), hv = lstm_cell_h(z[2], cn);
        a.c_out[ei] = cn;
        a.h_out[ei] = hv;
        if (a.hn_hi) {
          float hi, lo;
          split_tf32(a.hmask ? hv * a.hmask[uu + (a.hmask_full ? (size_t)a.hmask_ld * n : 0)] : hv, hi, lo);
          a.hn_hi[(size_t)n * a.hn_pitch + uu] = hi;
          a.hn_lo[(size_t)n * a.hn_pitch + uu] = lo;
        }
      }
    }
  } else {
    for (uint32_t e = tid; e < kRows * NB; e += blockDim.x) {
      const uint32_t c = e / kRows, rr = e % kRows, mm = blockIdx.x * kRows + rr, n = n0 + c;
      if (mm >= a.M || n >= a.N) continue;
      float v = 0.f;
      for (uint32_t w = 0; w < warps; ++w) v += red[((size_t)w * NB + c) * kRows + rr];
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

int thin_launch(dyb200_ctx* ctx, const ThinArgs& a, bool gates, double flops) {
  uint32_t nb = 1;
  while (nb < a.N && nb < 16) nb *= 2;
  bool vec = gates ? a.H % 4 == 0 : a.M % 4 == 0;
  uint32_t kmax = 0;
  for (int q = 0; q < a.npairs; ++q) {
    vec = vec && a.p[q].lda % 4 == 0 && aligned16(a.p[q].A);
    if (a.p[q].K > kmax) kmax = a.p[q].K;
  }
  const uint32_t blocks = gates ? (a.H + 7) / 8 : (a.M + kRows - 1) / kRows;
  const uint32_t threads = blocks <= (uint32_t)ctx->sm_count ? 512u : 256u;   // (one CTA per SM: more loads in flight from it)
  const size_t xs = (size_t)(kmax < kChunk ? kmax : kChunk) * nb * 4, red = (size_t)threads / 32 * nb * kRows * 4;
  const size_t smem = xs > red ? xs : red;
  void (*k)(ThinArgs) = gates ? (vec ? thin_kernel<true, true>(nb) : thin_kernel<true, false>(nb))
                              : (vec ? thin_kernel<false, true>(nb) : thin_kernel<false, false>(nb));
  if (smem > 48 * 1024) DYB_CUDA(ctx, cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  GemmProfScope scope(ctx, flops, 0, a.M, a.N, a.p[0].K + (a.npairs > 1 ? a.p[1].K : 0), (uint32_t)a.mode);
  dyb_launch(k, dim3(blocks, (a.N + nb - 1) / nb), threads, smem, ctx, a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

}  // namespace

// Up to 32 columns: at 32 columns and 4096 x 2048 the multiply-adds take 14 us, as long as the tensor path with its split.  A long
// reduction over few rows has too few CTAs here and stays with the K-split forms.
bool dyb200_thin_columns(uint32_t N) { return N <= 32; }

bool dyb200_thin_takes(uint32_t M, uint32_t N, int npairs, const GemmPair* pairs, const GemmEpilogue& epi) {
  if (!dyb200_thin_columns(N) || epi.split_m || (epi.mode != EPI_STORE && epi.mode != EPI_BIAS && epi.mode != EPI_ACCUM && epi.mode != EPI_GATES)) return false;
  uint64_t K = 0;
  for (int p = 0; p < npairs; ++p) {
    if (pairs[p].transA || pairs[p].transB || pairs[p].K == 0) return false;
    K += pairs[p].K;
  }
  return K <= 8ull * M || K <= 256;
}

int dyb200_gemm_thin(dyb200_ctx* ctx, uint32_t M, uint32_t N, int npairs, const GemmPair* pairs, const GemmEpilogue& epi) {
  ThinArgs a;
  memset(&a, 0, sizeof(a));
  double flops = 0;
  for (int p = 0; p < npairs; ++p) {
    const GemmPair& g = pairs[p];
    a.p[p] = ThinPair{g.A, g.lda, g.K, g.B, g.ldb, g.maskB, g.mask_ld, g.mask_full};
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
    a.p[p] = ThinPair{g.A, g.lda, g.K, g.B, g.ldb, g.maskB, g.mask_ld, g.mask_full};
    flops += 8.0 * H * B * g.K;
  }
  a.npairs = npairs; a.mode = EPI_LSTM_CELL; a.pre_in_c = pre_in_gates; a.M = 4 * H; a.N = B; a.C = epi.C; a.ldc = epi.ldc;
  a.bias = epi.bias; a.H = H; a.fb = epi.forget_bias; a.c_prev = epi.c_prev; a.c_out = epi.c_out; a.h_out = epi.h_out;
  a.hn_hi = epi.hn_hi; a.hn_lo = epi.hn_lo; a.hn_pitch = epi.hn_pitch;
  a.hmask = epi.hmask; a.hmask_ld = epi.hmask_ld; a.hmask_full = epi.hmask_full;
  return thin_launch(ctx, a, true, flops);
}
