// The forward recurrence of a wide LSTM layer (more than 384 units) over a whole sequence of few columns in one launch: a prompt
// read by a generator, or a layer at a small batch.
//
// What bounds it.  As one launch per step (gemm_thin.cu) a step of 1024 units and one column took 6.4 us: 2.6 us to read the 16.8 MB
// of Wh from L2, the rest launch, reduction and tail.  All of Wh fits the registers of the whole GPU (113 KB per SM), so here CTA g
// keeps the 32 gate rows of its 8 units for the whole sequence, and a step is one trip of h_t through L2: every value goes out
// as one 8-byte store of the value and the number of its step, and whoever needs it polls that word - no fence, no counter, no second
// round trip.  Two buffers: a CTA writes h_{t+1} only after it has read all of h_t, which every CTA wrote after reading h_{t-1}.
// 2.1 us per step of 1024 units, one column.
//
// Thread (q, s) of 4 x 128: gate q of the 8 units, k = 512 j + 4 s + 0..3.  Sums over s by a butterfly that leaves each group of four
// lanes one unit, then over four warps through shared memory; thread (column, unit) of the first ones finishes the cell.
#include "lstm_rec.cuh"

#include "gemm.cuh"
#include "lstm_wide.cuh"

namespace {

constexpr uint32_t kWideThreads = 512, kWideUnits = 8;
constexpr uint32_t kWidePolls = 1u << 22;   // polls of one word before a thread gives up (~ seconds)

template <int KJ>
__global__ void __launch_bounds__(kWideThreads, 1) k_lstm_wide_fwd(const __grid_constant__ WideFwd a) {
  constexpr uint32_t HP = 512 * KJ;
  extern __shared__ __align__(16) float wide_smem[];      // h [B][HP], sums [B][16 warps][8 units]
  dyb_grid_dep_sync();
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = tid >> 7, s = tid & 127, H = a.H, B = a.B, u0 = blockIdx.x * kWideUnits;
  float* hs = wide_smem;
  float* red = hs + (size_t)B * HP;
  float w[4 * KJ][8];
  {
    const bool vec = (H & 3) == 0 && aligned16(a.Wh);
#pragma unroll
    for (int x = 0; x < 4 * KJ; ++x) {
      const uint32_t k = 512 * (x / 4) + 4 * s + x % 4;
      const float* p = a.Wh + (size_t)q * H + u0 + (size_t)4 * H * k;
      float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
      if (k < H) {
        if (vec) {   // (units come in fours then)
          if (u0 < H) lo = __ldg(reinterpret_cast<const float4*>(p));
          if (u0 + 4 < H) hi = __ldg(reinterpret_cast<const float4*>(p + 4));
        } else {
          if (u0 < H) lo.x = __ldg(p);
          if (u0 + 1 < H) lo.y = __ldg(p + 1);
          if (u0 + 2 < H) lo.z = __ldg(p + 2);
          if (u0 + 3 < H) lo.w = __ldg(p + 3);
          if (u0 + 4 < H) hi.x = __ldg(p + 4);
          if (u0 + 5 < H) hi.y = __ldg(p + 5);
          if (u0 + 6 < H) hi.z = __ldg(p + 6);
          if (u0 + 7 < H) hi.w = __ldg(p + 7);
        }
      }
      w[x][0] = lo.x; w[x][1] = lo.y; w[x][2] = lo.z; w[x][3] = lo.w; w[x][4] = hi.x; w[x][5] = hi.y; w[x][6] = hi.z; w[x][7] = hi.w;
    }
  }
  // the cell of this thread
  const uint32_t cc = tid / kWideUnits, ul = tid % kWideUnits, u = u0 + ul;
  const bool cell = cc < B && u < H;
  float cst = 0.f, mk = 1.f;
  if (cell) {
    cst = a.c0[u + (size_t)H * cc];
    if (a.mask) mk = a.mask[u + (a.mask_full ? (size_t)H * cc : 0)];
  }
  for (uint32_t e = tid; e < B * HP; e += kWideThreads) {
    const uint32_t c = e / HP, k = e % HP;
    float v = 0.f;
    if (k < H) {
      v = a.h0[k + (size_t)H * c];
      if (a.mask) v *= a.mask[k + (a.mask_full ? (size_t)H * c : 0)];
    }
    hs[e] = v;
  }
  bool ok = true;
  for (uint32_t t = 0; t < a.T; ++t) {
    float pre[4];
    float* g = a.gates + u + (size_t)4 * H * (t * (size_t)B + cc);
    if (cell)
#pragma unroll
      for (int p = 0; p < 4; ++p) pre[p] = g[(size_t)p * H];
    if (t) {
      const unsigned long long* x = a.xchg + (size_t)(t & 1) * B * H;
      // (eight words at a time: one after the other, each cost its own trip to L2)
      for (uint32_t e0 = tid; e0 < B * H; e0 += 8 * kWideThreads) {
        unsigned long long v[8];
#pragma unroll
        for (uint32_t r = 0; r < 8; ++r)
          if (e0 + r * kWideThreads < B * H) asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[r]) : "l"(x + e0 + r * kWideThreads) : "memory");
#pragma unroll
        for (uint32_t r = 0; r < 8; ++r) {
          const uint32_t e = e0 + r * kWideThreads;
          if (e >= B * H) break;
          for (uint32_t it = 0; ok && (uint32_t)(v[r] >> 32) != t; ++it) {
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[r]) : "l"(x + e) : "memory");
            if (it == kWidePolls) ok = false;
          }
          const uint32_t c = e / H;
          hs[(size_t)c * HP + (e - c * H)] = __uint_as_float((uint32_t)v[r]);
        }
      }
    }
    __syncthreads();
    for (uint32_t c = 0; c < B; ++c) {
      float acc[8];
#pragma unroll
      for (int r = 0; r < 8; ++r) acc[r] = 0.f;
#pragma unroll
      for (int j = 0; j < KJ; ++j) {
        const float4 h = ld4(hs + (size_t)c * HP + 512 * j + 4 * s);
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r] = fmaf(w[4 * j][r], h.x, acc[r]);
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r] = fmaf(w[4 * j + 1][r], h.y, acc[r]);
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r] = fmaf(w[4 * j + 2][r], h.z, acc[r]);
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r] = fmaf(w[4 * j + 3][r], h.w, acc[r]);
      }
#pragma unroll
      for (int m = 4; m >= 1; m >>= 1) {   // lane bits 4, 3, 2 choose the unit
        const bool up = (lane & (4 * m)) != 0;
#pragma unroll
        for (int r = 0; r < 4; ++r)
          if (r < m) {
            const float keep = up ? acc[r + m] : acc[r], send = up ? acc[r] : acc[r + m];
            acc[r] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * m);
          }
      }
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
      acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
      if ((lane & 3) == 0) red[(c * 16 + warp) * 8 + (lane >> 2)] = acc[0];
    }
    __syncthreads();
    if (cell) {
      float z[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        const float* r = red + (cc * 16 + 4 * p) * 8 + ul;
        z[p] = ((r[0] + r[8]) + (r[16] + r[24])) + pre[p];
      }
      z[0] = gate_sigmoid(z[0]);
      z[1] = gate_sigmoid(z[1] + a.fb);
      z[2] = gate_sigmoid(z[2]);
      z[3] = gate_tanh(z[3]);
      cst = lstm_cell_c(z[0], z[3], z[1], cst);
      const float hv = lstm_cell_h(z[2], cst), hm = hv * mk;
      if (t + 1 < a.T) {
        const unsigned long long v = (unsigned long long)(t + 1) << 32 | __float_as_uint(hm);
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(a.xchg + (size_t)((t + 1) & 1) * B * H + (size_t)H * cc + u), "l"(v) : "memory");
      }
#pragma unroll
      for (int p = 0; p < 4; ++p) g[(size_t)p * H] = z[p];
      const size_t col = (size_t)t * B + cc;
      a.c[u + (size_t)H * col] = cst;
      a.h[u + (size_t)H * col] = hv;
      if (a.hn_hi && t + 1 < a.T) {
        float hi, lo;
        split_tf32(hm, hi, lo);
        a.hn_hi[(col + B) * a.hn_pitch + u] = hi;
        a.hn_lo[(col + B) * a.hn_pitch + u] = lo;
      }
    }
  }
  if (!ok) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
}

}  // namespace

// Up to 8 columns (each costs a step 0.6 - 0.8 us of polls and multiply-adds; 1024 units: 2.1 us at 1, 5.3 at 4, 7.8 at 8 columns, launch by
// launch 5.0, 7.3 and 10.4) and as many units as the SMs hold, 8 each; narrower layers
// belong to the clusters of lstm_rec.cu.
bool dyb200_wide_takes(const dyb200_ctx* ctx, uint32_t H, uint32_t B) { return !ctx->wide_refused && H > 384 && H <= 1536 && H <= kWideUnits * (uint32_t)ctx->sm_count && B <= 8; }

int dyb200_wide_fwd(dyb200_ctx* ctx, WideFwd a, bool* launched) {
  *launched = true;
  void* x;
  const size_t bytes = (size_t)2 * a.B * a.H * sizeof(unsigned long long);
  int rc = dyb200_scratch(ctx, bytes, &x);
  if (rc) return rc;
  a.xchg = (unsigned long long*)x;
  a.flags = ctx->dev_flags;
  DYB_CUDA(ctx, cudaMemsetAsync(x, 0, bytes, ctx->stream));   // (no step has number 0)
  const uint32_t kj = (a.H + 511) / 512;
  void (*k)(WideFwd) = kj == 1 ? k_lstm_wide_fwd<1> : kj == 2 ? k_lstm_wide_fwd<2> : k_lstm_wide_fwd<3>;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = dim3((a.H + kWideUnits - 1) / kWideUnits); cfg.blockDim = dim3(kWideThreads);
  cfg.dynamicSmemBytes = (size_t)a.B * (512 * kj + 128) * sizeof(float); cfg.stream = ctx->stream;
  DYB_CUDA(ctx, dyb_smem_limit(k, cfg.dynamicSmemBytes, 8 * (512 * 3 + 128) * sizeof(float)));
  // The CTAs wait on one another: launched as one gang.  A driver that refuses that gets the launches step by step; where the
  // caller has asked for launches without the attribute (dyb200_ctx_sequence_kernels), or the sequence kernels found it refused, a plain one.
  cudaLaunchAttribute attr[1];
  if (ctx->seq_coop >= 0) {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, k, a) != cudaSuccess) {
      (void)cudaGetLastError();
      ctx->wide_refused = 1;
      *launched = false;
      return DYB200_OK;
    }
    ctx->launches++;
    return DYB200_OK;
  }
  cudaLaunchKernelEx(&cfg, k, a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}
