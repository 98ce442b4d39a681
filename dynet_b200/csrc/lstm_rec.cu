// The recurrence of an LSTM layer of moderate width (H <= 384) over a whole sequence, forward and backward, one launch per
// pass: the call pattern of CompactVanillaLSTMBuilder::add_input_impl (dynet/lstm.cc:1044-1080) for a batch of sequences, or
// for the shrinking batches that the autobatching executor makes of ragged sentences (dynet/exec.cc:481-895).
//
// What bounds it.  Per time step a layer of 256 units and 32 columns is 17 MFLOP: as one launch per step (operand split,
// product, cell pass) a step took 12 us forward and 24 us backward, all of it launch latency, pipeline fill and K-split
// exchange of products that fill a fraction of the GPU.  Batch columns never meet in the recurrence, so here a thread-block
// CLUSTER owns a few columns for all time steps and never talks to another cluster:
//   * Wh is held on chip for the whole sequence: CTA r of the cluster keeps the 4 gate rows of its U hidden units (forward)
//     / the same rows as the reduction index of Wh^T (backward) in REGISTERS, up to 192 floats per thread; Wh is read once
//     per launch and cluster instead of once per step.
//   * h_t (forward) goes to every CTA of the cluster through distributed shared memory, double-buffered, with one hardware
//     cluster barrier per step (no polling, no global-memory hand-over); backward, each CTA reduces over its own gate rows
//     and sends partial sums of dE/dh_{t-1} to the CTA that owns the unit, 4 x fewer bytes than handing dgates around.
//   * plain fp32 multiply-adds (two per instruction, fma.rn.f32x2): more accurate than the 3xTF32 products of the per-step
//     form, and at 1 - 8 columns per cluster the tensor pipe could not be filled anyway.
// The arithmetic order is fixed by the shape (cluster count, ranks, lanes): reproducible run to run.
//
// Thread layout, forward: 8 lanes per hidden unit (slice s of the reduction index: k = 32 j + 4 s + 0..3, so the 8 slices of
// a unit read 128 contiguous bytes of h: no bank conflicts, the 4 units of a warp broadcast), 4 gates x KD k per lane.
// NB columns at a time; a butterfly over the 8 lanes leaves each lane with all four gates of one column.
// Backward: 8 lanes per group of 8 units of dE/dh_{t-1}, slices of the CTA's own 4 U gate rows in the same pattern.
#include "lstm_rec.cuh"

#include "gemm.cuh"
#include "lstm_cell.cuh"
#include "lstm_rec_api.h"

namespace {

typedef unsigned long long u64;
__device__ __forceinline__ u64 pack2(float a, float b) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float sum2(u64 v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return a + b;
}
__device__ __forceinline__ void fma2(u64& acc, u64 a, u64 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ float xor_add(float keep, float send, int m) { return keep + __shfl_xor_sync(0xffffffffu, send, m); }

// columns of this cluster that are active at a step of width B: those i < ncol with g + G (i0 + i) < B
__device__ __forceinline__ uint32_t active_cols(uint32_t B, uint32_t g, uint32_t G, uint32_t i0, uint32_t ncol) {
  if (B <= g) return 0;
  const uint32_t n = (B - g + G - 1) / G;
  return n > i0 ? min(n - i0, ncol) : 0;
}

// grid (C, G, directions), cluster (C, 1, 1); block = 8 U threads.  Dynamic shared memory: h[2][ncap][8 KD], c[ncap][U].
template <int KD, int NB>
__global__ void __launch_bounds__(256, 1) k_lstm_rec_fwd(const __grid_constant__ RecFwd a) {
  constexpr int HP = 8 * KD;
  extern __shared__ __align__(16) float rec_smem[];
  const RecDirF d = blockIdx.z ? a.d[1] : a.d[0];
  const uint32_t H = a.H, U = a.U, G = a.G, g = blockIdx.y, rank = blockIdx.x, C = gridDim.x;
  const uint32_t tid = threadIdx.x, s = tid & 7, ul = tid >> 3, u = rank * U + ul;
  const bool live_u = u < H;
  float* hbuf = rec_smem;
  float* cbuf = rec_smem + (size_t)2 * a.ncap * HP;
  dyb_grid_dep_sync();

  u64 w[4][KD / 2];
#pragma unroll
  for (int j = 0; j < KD / 4; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t k = 32 * j + 4 * s + i;
        v[i] = (live_u && k < H) ? __ldg(d.Wh + (size_t)q * H + u + (size_t)4 * H * k) : 0.f;
      }
      w[q][2 * j] = pack2(v[0], v[1]);
      w[q][2 * j + 1] = pack2(v[2], v[3]);
    }

  // the column of a block that this lane finishes; 8 / NB lanes share one (they hold equal values; dup == 0 stores)
  const uint32_t lc = NB == 8 ? s : NB == 4 ? s >> 1 : NB == 2 ? s >> 2 : 0;
  const uint32_t dup = NB == 8 ? 0 : NB == 4 ? (s & 1) : NB == 2 ? (s & 3) : s;
  constexpr uint32_t DUPS = 8 / NB;
  const uint32_t nloc = a.N > g ? (a.N - g + G - 1) / G : 0;

  for (uint32_t i0 = 0; i0 < nloc; i0 += a.ncap) {
    const uint32_t ncol = min(a.ncap, nloc - i0);
    // h_{-1} of this chunk's columns; zeros in the padding (both buffers)
    for (uint32_t e = tid; e < a.ncap * HP; e += blockDim.x) {
      const uint32_t i = e / HP, k = e % HP, sc = g + G * (i0 + i);
      float v = 0.f;
      if (d.h0 && i < ncol && k < H) {
        v = d.h0[k + (size_t)H * sc];
        if (d.mask) v *= d.mask[k + (a.mask_full ? (size_t)H * sc : 0)];
      }
      hbuf[e] = v;
      hbuf[(size_t)a.ncap * HP + e] = 0.f;
    }
    for (uint32_t e = tid; e < ncol * U; e += blockDim.x) {
      const uint32_t i = e / U, uu = rank * U + e % U, sc = g + G * (i0 + i);
      cbuf[e] = (d.c0 && uu < H) ? d.c0[uu + (size_t)H * sc] : 0.f;
    }
    __syncthreads();
    if (d.hn_hi)   // the planes of the first step's h input
      for (uint32_t e = tid; e < ncol * U; e += blockDim.x) {
        const uint32_t i = e / U, uu = rank * U + e % U, sc = g + G * (i0 + i);
        if (uu < H) {
          float hi, lo;
          split_tf32(hbuf[(size_t)i * HP + uu], hi, lo);
          d.hn_hi[(size_t)sc * a.hn_pitch + uu] = hi;
          d.hn_lo[(size_t)sc * a.hn_pitch + uu] = lo;
        }
      }
    cluster_arrive();
    cluster_wait();

    uint32_t col0 = 0, B = a.prefix ? a.prefix[1] : a.N;      // first column and width of the step
    uint32_t n = active_cols(B, g, G, i0, ncol);
    float pre[4], mk;
    auto fetch = [&](uint32_t c0, uint32_t nact, uint32_t nb) {   // Wx x + b and the mask of this lane's column of a block
      const uint32_t i = nb + lc, sc = g + G * (i0 + i);
      if (live_u && i < nact) {
        const float* p = d.gates + u + (size_t)4 * H * (c0 + sc);
#pragma unroll
        for (int q = 0; q < 4; ++q) pre[q] = p[(size_t)q * H];
        mk = d.mask ? d.mask[u + (a.mask_full ? (size_t)H * sc : 0)] : 1.f;
      } else {
        pre[0] = pre[1] = pre[2] = pre[3] = mk = 0.f;
      }
    };
    fetch(col0, n, 0);
    for (uint32_t t = 0; t < a.T && n > 0; ++t) {
      const float* hcur = hbuf + (size_t)(t & 1) * a.ncap * HP;
      const uint32_t hnext = smem_addr(hbuf + (size_t)((t + 1) & 1) * a.ncap * HP);
      const uint32_t col1 = col0 + B;                                          // the next step
      const uint32_t B1 = t + 1 < a.T ? (a.prefix ? a.prefix[t + 2] - a.prefix[t + 1] : a.N) : 0;
      const uint32_t n1 = active_cols(B1, g, G, i0, ncol);
      float z[4], cn = 0.f, hv = 0.f, hm = 0.f;
      uint32_t sc = 0;
      bool mine = false;
      auto store = [&]() {   // gates, c, h and the operand planes of the block just finished
        if (!mine || dup) return;
        float* p = d.gates + u + (size_t)4 * H * (col0 + sc);
#pragma unroll
        for (int q = 0; q < 4; ++q) p[(size_t)q * H] = z[q];
        d.c[u + (size_t)H * (col0 + sc)] = cn;
        d.h[u + (size_t)H * (col0 + sc)] = hv;
        if (d.hn_hi && sc < B1) {
          float hi, lo;
          split_tf32(hm, hi, lo);
          d.hn_hi[(size_t)(col1 + sc) * a.hn_pitch + u] = hi;
          d.hn_lo[(size_t)(col1 + sc) * a.hn_pitch + u] = lo;
        }
      };
#pragma unroll 1
      for (uint32_t nb = 0; nb < n; nb += NB) {
        u64 acc[4][NB];
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int c = 0; c < NB; ++c) acc[q][c] = 0ull;
        const float* hp = hcur + (size_t)nb * HP + 4 * s;
#pragma unroll
        for (int j = 0; j < KD / 4; ++j)
#pragma unroll
          for (int c = 0; c < NB; ++c) {
            const ulonglong2 hh = *reinterpret_cast<const ulonglong2*>(hp + (size_t)c * HP + 32 * j);
#pragma unroll
            for (int q = 0; q < 4; ++q) { fma2(acc[q][c], w[q][2 * j], hh.x); fma2(acc[q][c], w[q][2 * j + 1], hh.y); }
          }
        // sum over the 8 slices: columns are split between the lanes as long as there are several, then added on both sides
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float v[NB];
#pragma unroll
          for (int c = 0; c < NB; ++c) v[c] = sum2(acc[q][c]);
#pragma unroll
          for (int m = 4; m >= 1; m >>= 1) {
            const int half = NB * m / 8;            // columns each side keeps (0: one is left, added on both sides)
            const bool up = (s & m) != 0;
            if (half >= 1) {
#pragma unroll
              for (int c = 0; c < NB / 2; ++c)
                if (c < half) v[c] = xor_add(up ? v[c + half] : v[c], up ? v[c] : v[c + half], m);
            } else {
              v[0] = xor_add(v[0], v[0], m);
            }
          }
          z[q] = v[0];
        }
        const uint32_t i = nb + lc;
        mine = live_u && i < n;
        if (mine) {
          sc = g + G * (i0 + i);
          z[0] = gate_sigmoid(z[0] + pre[0]);
          z[1] = gate_sigmoid(z[1] + pre[1] + a.fb);
          z[2] = gate_sigmoid(z[2] + pre[2]);
          z[3] = gate_tanh(z[3] + pre[3]);
          cn = lstm_cell_c(z[0], z[3], z[1], cbuf[i * U + ul]);
          hv = lstm_cell_h(z[2], cn);
          hm = hv * mk;
        }
        __syncwarp();   // (all lanes of the unit have read the old cell state)
        if (mine) {
          if (!dup) cbuf[i * U + ul] = cn;
          const uint32_t off = hnext + 4u * (i * HP + u);
          for (uint32_t r = dup; r < C; r += DUPS) st_cluster(map_rank(off, r), hm);
        }
        if (nb + NB < n) {
          store();
          fetch(col0, n, nb + NB);
        }
      }
      cluster_arrive();
      store();                       // (the last block's results go out while the cluster meets)
      if (n1) fetch(col1, n1, 0);
      cluster_wait();
      col0 = col1; B = B1; n = n1;
    }
    cluster_arrive();                // nobody overwrites a neighbour's buffers before it is through with this chunk
    cluster_wait();
  }
}

// grid (C, G, directions), cluster (C, 1, 1); block = 8 ceil(H / 8) threads rounded up to warps.
// Dynamic shared memory: part[2][C][ncap][U], dg[ncap][8 KD], dcs[ncap][U].  KD = gate rows per slice: 8 KD >= 4 U.
template <int KD, int NB>
__global__ void __launch_bounds__(KD == 16 ? 256 : 384, 1) k_lstm_rec_bwd(const __grid_constant__ RecBwd a) {
  constexpr int KP = 8 * KD;
  extern __shared__ __align__(16) float rec_smem[];
  const RecDirB d = blockIdx.z ? a.d[1] : a.d[0];
  const uint32_t H = a.H, U = a.U, G = a.G, g = blockIdx.y, rank = blockIdx.x, C = gridDim.x, ncap = a.ncap;
  const uint32_t tid = threadIdx.x, s = tid & 7, og = tid >> 3;
  float* part = rec_smem;                                   // [parity][source rank][column][unit]
  float* dg = part + (size_t)2 * C * ncap * U;
  float* dcs = dg + (size_t)ncap * KP;
  dyb_grid_dep_sync();

  // weights: outputs o = 8 og + 0..7 (units of h_{t-1}) x this CTA's gate rows kk = q U + unit, slice s
  u64 w[8][KD / 2];
#pragma unroll
  for (int o = 0; o < 8; ++o)
#pragma unroll
    for (int j = 0; j < KD / 4; ++j) {
      float v[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t kk = 32 * j + 4 * s + i, q = kk / U, uu = rank * U + kk % U, oo = 8 * og + o;
        v[i] = (q < 4 && uu < H && oo < H) ? __ldg(d.Wh + (size_t)q * H + uu + (size_t)4 * H * oo) : 0.f;
      }
      w[o][2 * j] = pack2(v[0], v[1]);
      w[o][2 * j + 1] = pack2(v[2], v[3]);
    }
  // after the butterfly this lane holds unit o_mine of dE/dh_{t-1}; it belongs to CTA o_mine / U
  const uint32_t o_mine = 8 * og + s, o_rank = o_mine / U, o_ul = o_mine % U;
  const bool o_live = o_mine < H;
  const uint32_t o_base = map_rank(smem_addr(part), o_live ? o_rank : rank) + 4u * (rank * ncap * U + o_ul);
  // cell pass: thread -> (unit c_ul, columns c_i0, c_i0 + c_step, ...)
  const uint32_t c_step = blockDim.x / U, c_ul = tid % U, c_i0 = tid / U, c_u = rank * U + c_ul;
  const bool c_live = c_i0 < c_step && c_u < H;
  float db[4] = {0.f, 0.f, 0.f, 0.f};
  const uint32_t nloc = a.N > g ? (a.N - g + G - 1) / G : 0;

  for (uint32_t i0 = 0; i0 < nloc; i0 += ncap) {
    const uint32_t ncol = min(ncap, nloc - i0);
    for (uint32_t e = tid; e < ncap * KP; e += blockDim.x) dg[e] = 0.f;
    for (uint32_t e = tid; e < ncap * U; e += blockDim.x) dcs[e] = 0.f;
    cluster_arrive();
    cluster_wait();
    // the last step that has a column of this chunk: widths never grow, so the steps before it have one too
    uint32_t T = a.T;
    while (a.prefix && T > 0 && active_cols(a.prefix[T] - a.prefix[T - 1], g, G, i0, ncol) == 0) --T;

    // saved values of the first (column, unit) item of the cell pass of a step, requested one step ahead
    float gt[4], cv, cp, dhv, dcv;
    auto fetch = [&](uint32_t t, uint32_t col, uint32_t colm1, uint32_t sc) {
      const float* p = d.gates + c_u + (size_t)4 * H * (col + sc);
#pragma unroll
      for (int q = 0; q < 4; ++q) gt[q] = p[(size_t)q * H];
      cv = d.c[c_u + (size_t)H * (col + sc)];
      cp = t ? d.c[c_u + (size_t)H * (colm1 + sc)] : (d.c0 ? d.c0[c_u + (size_t)H * sc] : 0.f);
      dhv = d.dh[c_u + (size_t)H * (col + sc)];
      dcv = d.dc ? d.dc[c_u + (size_t)H * (col + sc)] : 0.f;
    };
    auto start_of = [&](uint32_t t) { return a.prefix ? a.prefix[t] : t * a.N; };
    uint32_t n_later = 0;            // columns that were active at step t + 1
    uint32_t col = T ? start_of(T - 1) : 0;
    uint32_t n = T ? active_cols(start_of(T) - col, g, G, i0, ncol) : 0;
    if (T && c_live && c_i0 < n) fetch(T - 1, col, T > 1 ? start_of(T - 2) : 0, g + G * (i0 + c_i0));
    for (uint32_t t = T; t-- > 0;) {
      const uint32_t colm1 = t ? start_of(t - 1) : 0;
      const float* pin = part + (size_t)((t + 1) & 1) * C * ncap * U;
      // ---- gradients of the gate pre-activations of this CTA's units ----
      if (c_live)
        for (uint32_t i = c_i0; i < n; i += c_step) {
          const uint32_t sc = g + G * (i0 + i);
          if (i != c_i0) fetch(t, col, colm1, sc);
          float dh = dhv;
          if (i < n_later) {
            float r = 0.f;
            for (uint32_t q = 0; q < C; ++q) r += pin[((size_t)q * ncap + i) * U + c_ul];
            if (d.mask) r *= d.mask[c_u + (a.mask_full ? (size_t)H * sc : 0)];
            dh += r;
            d.dh[c_u + (size_t)H * (col + sc)] = dh;
          }
          float dcp = 0.f, pr[4];
          const float dci = dcv + dcs[i * U + c_ul];
          if (d.dc && i < n_later) d.dc[c_u + (size_t)H * (col + sc)] = dci;
          lstm_cell_grad(gt[0], gt[1], gt[2], gt[3], cv, cp, dh, dci, true, dcp, pr[0], pr[1], pr[2], pr[3]);
          dcs[i * U + c_ul] = dcp;
          float* dgi = dg + (size_t)i * KP + c_ul;
          float* ph = d.dn_hi + (size_t)(col + sc) * a.dn_pitch + c_u;
          float* pl = d.dn_lo + (size_t)(col + sc) * a.dn_pitch + c_u;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            dgi[q * U] = pr[q];
            db[q] += pr[q];
            float hi, lo;
            split_tf32(pr[q], hi, lo);
            ph[(size_t)q * H] = hi;
            pl[(size_t)q * H] = lo;
          }
        }
      if (t == 0) break;             // (no earlier state to hand dE/dh to)
      __syncthreads();
      const uint32_t nm1 = active_cols(col - colm1, g, G, i0, ncol);
      if (c_live && c_i0 < nm1) fetch(t - 1, colm1, t > 1 ? start_of(t - 2) : 0, g + G * (i0 + c_i0));
      // ---- partial sums of dE/dh_{t-1} over this CTA's gate rows ----
      const uint32_t pout = o_base + 4u * ((t & 1) * C * ncap * U);
#pragma unroll 1
      for (uint32_t nb = 0; nb < n; nb += NB) {
        u64 acc[8][NB];
#pragma unroll
        for (int o = 0; o < 8; ++o)
#pragma unroll
          for (int c = 0; c < NB; ++c) acc[o][c] = 0ull;
        const float* gp = dg + (size_t)nb * KP + 4 * s;
#pragma unroll
        for (int j = 0; j < KD / 4; ++j)
#pragma unroll
          for (int c = 0; c < NB; ++c) {
            const ulonglong2 hh = *reinterpret_cast<const ulonglong2*>(gp + (size_t)c * KP + 32 * j);
#pragma unroll
            for (int o = 0; o < 8; ++o) { fma2(acc[o][c], w[o][2 * j], hh.x); fma2(acc[o][c], w[o][2 * j + 1], hh.y); }
          }
#pragma unroll
        for (int c = 0; c < NB; ++c) {
          float v[8];
#pragma unroll
          for (int o = 0; o < 8; ++o) v[o] = sum2(acc[o][c]);
#pragma unroll
          for (int m = 4; m >= 1; m >>= 1) {
            const bool up = (s & m) != 0;
#pragma unroll
            for (int o = 0; o < 4; ++o)
              if (o < m) v[o] = xor_add(up ? v[o + m] : v[o], up ? v[o] : v[o + m], m);
          }
          if (o_live && nb + c < n) st_cluster(pout + 4u * ((nb + c) * U), v[0]);
        }
      }
      cluster_arrive();
      cluster_wait();
      n_later = n; n = nm1; col = colm1;
    }
    cluster_arrive();
    cluster_wait();
  }
  // row sums of dgates: the threads of one unit, in ascending order (part is free: every CTA is through)
  float* red = part;
  if (c_live)
#pragma unroll
    for (int q = 0; q < 4; ++q) red[(c_i0 * 4 + q) * U + c_ul] = db[q];
  __syncthreads();
  for (uint32_t e = tid; e < 4 * U; e += blockDim.x) {
    const uint32_t q = e / U, ul = e % U, u = rank * U + ul;
    if (u < H) {
      float r = 0.f;
      for (uint32_t k = 0; k < c_step; ++k) r += red[(k * 4 + q) * U + ul];
      d.dbpart[(size_t)g * 4 * H + q * H + u] = r;
    }
  }
}

// db += sum over the clusters, in ascending order
__global__ void __launch_bounds__(256) k_rec_db(const float* __restrict__ part0, const float* __restrict__ part1, uint32_t G, uint32_t rows,
                                                float* __restrict__ db0, float* __restrict__ db1) {
  dyb_grid_dep_sync();
  const float* part = blockIdx.y ? part1 : part0;
  float* db = blockIdx.y ? db1 : db0;
  const uint32_t r = blockIdx.x * 256 + threadIdx.x;
  if (r >= rows) return;
  float acc = 0.f;
#pragma unroll 8
  for (uint32_t k = 0; k < G; ++k) acc += part[(size_t)k * rows + r];
  db[r] += acc;
}

}  // namespace

// ---- host side -----------------------------------------------------------------------------------------------------------
namespace {

constexpr size_t kRecSmemMax = 208 * 1024;
constexpr uint32_t kRecCols = 64;   // most columns a cluster carries through the sequence at once (more: one batch of them after another)

typedef void (*FwdKernel)(RecFwd);
typedef void (*BwdKernel)(RecBwd);
// (registers: 4 KD weights + 8 NB accumulator words forward, 8 KD2 + 16 NB backward, at most 255 per thread)
FwdKernel fwd_kernel(uint32_t kd, uint32_t nb) {
#define REC_F(K) (nb == 1 ? k_lstm_rec_fwd<K, 1> : nb == 2 ? k_lstm_rec_fwd<K, 2> : nb == 4 ? k_lstm_rec_fwd<K, 4> : k_lstm_rec_fwd<K, 8>)
  switch (kd) {
    case 8: return REC_F(8);
    case 16: return REC_F(16);
    case 24: return REC_F(24);
    case 32: return REC_F(32);
    case 40: return nb == 1 ? k_lstm_rec_fwd<40, 1> : nb == 2 ? k_lstm_rec_fwd<40, 2> : k_lstm_rec_fwd<40, 4>;
    default: return nb == 1 ? k_lstm_rec_fwd<48, 1> : k_lstm_rec_fwd<48, 2>;
  }
#undef REC_F
}
uint32_t fwd_nb_max(uint32_t kd) { return kd <= 32 ? 8 : kd == 40 ? 4 : 2; }
// (16 gate rows per lane: at most 256 units and threads, 255 registers each; fewer: up to 384 threads of 168 registers)
BwdKernel bwd_kernel(uint32_t kd, uint32_t nb) {
#define REC_B(K) (nb == 1 ? k_lstm_rec_bwd<K, 1> : nb == 2 ? k_lstm_rec_bwd<K, 2> : k_lstm_rec_bwd<K, 4>)
  switch (kd) {
    case 8: return REC_B(8);
    case 12: return nb == 1 ? k_lstm_rec_bwd<12, 1> : k_lstm_rec_bwd<12, 2>;
    default: return REC_B(16);
  }
#undef REC_B
}
uint32_t bwd_nb_max(uint32_t kd) { return kd == 12 ? 2 : 4; }
uint32_t block_cols(uint32_t n, uint32_t most) {
  uint32_t nb = 1;
  while (nb < n && nb < most) nb *= 2;
  return nb;
}
uint32_t fwd_threads(const RecPlan& p) { return 8 * p.U; }
uint32_t bwd_threads(uint32_t H) { return ((H + 7) / 8 * 8 + 31) / 32 * 32; }
size_t fwd_col_bytes(const RecPlan& p) { return sizeof(float) * (2 * 8 * p.KD + p.U); }
size_t bwd_col_bytes(const RecPlan& p) { return sizeof(float) * (2 * p.C * p.U + 8 * p.KD2 + p.U); }

int launch_cfg(dyb200_ctx* ctx, const void* kernel, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, dim3 grid, uint32_t threads, size_t smem) {
  DYB_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRecSmemMax));
  if (grid.x > 8) DYB_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  memset(cfg, 0, sizeof(*cfg));
  cfg->gridDim = grid; cfg->blockDim = dim3(threads, 1, 1); cfg->dynamicSmemBytes = smem; cfg->stream = ctx->stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = grid.x; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg->attrs = attr; cfg->numAttrs = 1;
  return DYB200_OK;
}
// How many clusters run side by side (remembered per context and width class): the columns are dealt out over that many.
int clusters_that_fit(dyb200_ctx* ctx, const RecPlan& p, bool bwd, uint32_t threads) {
  int16_t& fit = ctx->rec_fit[bwd][p.KD / 8 - 1][p.C];
  if (fit == 0) {
    const void* k = bwd ? (const void*)bwd_kernel(p.KD2, bwd_nb_max(p.KD2)) : (const void*)fwd_kernel(p.KD, fwd_nb_max(p.KD));
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    if (launch_cfg(ctx, k, &cfg, attr, dim3(p.C, 1, 1), threads, kRecSmemMax)) return -1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = -1; }
    fit = (int16_t)(n > 0 ? n : -1);
  }
  return fit;
}
// Columns per cluster and per pass of it over the sequence.
void deal_columns(uint32_t N, int fit, int ndir, size_t col_bytes, uint32_t* G, uint32_t* ncap) {
  const uint32_t g = fit > ndir ? (uint32_t)(fit / ndir) : 1u;
  *G = N < g ? N : g;
  const uint32_t nloc = (N + *G - 1) / *G;
  uint32_t most = (uint32_t)(kRecSmemMax / col_bytes) / 8 * 8;
  if (most > kRecCols) most = kRecCols;
  const uint32_t chunks = (nloc + most - 1) / most;
  *ncap = ((nloc + chunks - 1) / chunks + 7) / 8 * 8;
}

}  // namespace

bool dyb200_rec_plan(dyb200_ctx* ctx, uint32_t H, RecPlan* out) {
  if (H == 0 || H > 384) return false;
  RecPlan p;
  // up to 256 units: 32 per CTA and at most 8 CTAs, the portable cluster size; beyond: 16 CTAs
  p.U = H <= 256 ? (H < 32 ? (H + 3) / 4 * 4 : 32u) : ((H + 15) / 16 + 3) / 4 * 4;
  p.C = (H + p.U - 1) / p.U;
  p.KD = (H + 63) / 64 * 8;
  p.KD2 = p.U <= 16 ? 8 : p.U <= 24 ? 12 : 16;
  if (clusters_that_fit(ctx, p, false, fwd_threads(p)) <= 0 || clusters_that_fit(ctx, p, true, bwd_threads(H)) <= 0) return false;
  *out = p;
  return true;
}

int dyb200_rec_fwd(dyb200_ctx* ctx, const RecPlan& p, RecFwd* a, int ndir) {
  a->U = p.U;
  deal_columns(a->N, clusters_that_fit(ctx, p, false, fwd_threads(p)), ndir, fwd_col_bytes(p), &a->G, &a->ncap);
  const uint32_t per_pass = a->ncap < (a->N + a->G - 1) / a->G ? a->ncap : (a->N + a->G - 1) / a->G;
  FwdKernel k = fwd_kernel(p.KD, block_cols(per_pass, fwd_nb_max(p.KD)));
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  int rc = launch_cfg(ctx, (const void*)k, &cfg, attr, dim3(p.C, a->G, ndir), fwd_threads(p), a->ncap * fwd_col_bytes(p));
  if (rc) return rc;
  cudaLaunchKernelEx(&cfg, k, *a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

int dyb200_rec_bwd(dyb200_ctx* ctx, const RecPlan& p, RecBwd* a, int ndir, float* const* db) {
  a->U = p.U;
  deal_columns(a->N, clusters_that_fit(ctx, p, true, bwd_threads(a->H)), ndir, bwd_col_bytes(p), &a->G, &a->ncap);
  const uint32_t per_pass = a->ncap < (a->N + a->G - 1) / a->G ? a->ncap : (a->N + a->G - 1) / a->G;
  void* part;
  int rc = dyb200_scratch(ctx, (size_t)ndir * a->G * 4 * a->H * sizeof(float), &part);
  if (rc) return rc;
  for (int k = 0; k < ndir; ++k) a->d[k].dbpart = (float*)part + (size_t)k * a->G * 4 * a->H;
  BwdKernel k = bwd_kernel(p.KD2, block_cols(per_pass, bwd_nb_max(p.KD2)));
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  rc = launch_cfg(ctx, (const void*)k, &cfg, attr, dim3(p.C, a->G, ndir), bwd_threads(a->H), a->ncap * bwd_col_bytes(p));
  if (rc) return rc;
  cudaLaunchKernelEx(&cfg, k, *a);
  DYB_LAUNCHED(ctx);
  const uint32_t rows = 4 * a->H;
  dyb_launch(k_rec_db, dim3((rows + 255) / 256, ndir), 256, 0, ctx, (const float*)a->d[0].dbpart, (const float*)a->d[ndir - 1].dbpart, a->G, rows,
             db[0], db[ndir - 1]);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

// ---- products over all columns around the recurrence -----------------------------------------------------------------------
namespace {

// dst += src .* mask, all `rows` x n; the mask repeats every `period` columns (0: one column for all)
__global__ void __launch_bounds__(256) k_masked_add(const float* __restrict__ src, const float* __restrict__ mask, uint32_t rows, uint32_t period,
                                                    size_t total, float* __restrict__ dst) {
  dyb_grid_dep_sync();
  for (size_t e = (size_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (size_t)gridDim.x * 256) {
    const uint32_t n = (uint32_t)(e / rows), r = (uint32_t)(e % rows);
    dst[e] = __fmaf_rn(src[e], mask[r + (period ? (size_t)rows * (n % period) : 0)], dst[e]);
  }
}

// Steps from which a sequence is worth the fixed costs of the recurrence kernels: reading Wh into registers (3 - 5 us), the
// separate input product and the separate dx product.  Shorter ones stay on the per-step calls.
constexpr uint32_t kRecMinSteps = 8;

}  // namespace

extern "C" {

int dyb200i_rec_takes(dyb200_ctx* ctx, uint32_t H, uint32_t T) {
  RecPlan p;
  return ctx->seq_kernels && T >= kRecMinSteps && dyb200_rec_plan(ctx, H, &p) ? 1 : 0;
}

int dyb200i_rec_inputs(dyb200_ctx* ctx, dyb200_wgrad* w, const float* Wx, const float* b, uint32_t I, uint32_t H, uint32_t columns, float* gates) {
  { int rc0__ = dyb200_scratch_begin(ctx); if (rc0__) return rc0__; }
  const uint32_t G = 4 * H;
  PackedOp A, X, Hs;
  DYB_CHECK_ARG(ctx, dyb200_wgrad_rows(w) == G && dyb200_wgrad_column_planes(w, columns, nullptr, &X, &Hs) && X.K == I && Hs.K == H,
                "lstm recurrence: the accumulator does not hold the inputs of this layer");
  // (Wx split as it lies, I rows of 4H values, and read MN-major: the planes that the dx product reads K-major)
  int rc = dyb200_tc_param(ctx, Wx, G, true, I, G, &A);
  if (rc) return rc;
  A.rows = G; A.K = I; A.mn_major = 1;
  GemmEpilogue e{EPI_BIAS, gates, G, b, 0, 0.f, nullptr, 0, 0};
  return dyb200_tc_gemm_packed(ctx, G, columns, 1, &A, &X, e);
}

int dyb200i_rec_fwd(dyb200_ctx* ctx, int ndir, const dyb200i_rec_dir* dirs, uint32_t H, uint32_t T, uint32_t N, const uint32_t* prefix_dev,
                    int mask_full, float forget_bias) {
  RecPlan p;
  DYB_CHECK_ARG(ctx, (ndir == 1 || ndir == 2) && dyb200_rec_plan(ctx, H, &p), "lstm recurrence: %u units are outside its range", H);
  RecFwd a;
  memset(&a, 0, sizeof(a));
  for (int k = 0; k < ndir; ++k) {
    const dyb200i_rec_dir& s = dirs[k];
    RecDirF& d = a.d[k];
    d.Wh = s.Wh; d.gates = s.gates; d.c = s.c; d.h = s.h; d.h0 = s.h0; d.c0 = s.c0; d.mask = s.mask_h;
    if (s.w) {
      PackedOp X, Hs;
      DYB_CHECK_ARG(ctx, dyb200_wgrad_column_planes(s.w, 1, nullptr, &X, &Hs) && Hs.K == H && (k == 0 || Hs.pitch == a.hn_pitch),
                    "lstm recurrence: the accumulator does not hold the inputs of this layer");
      d.hn_hi = Hs.hi; d.hn_lo = Hs.lo; a.hn_pitch = Hs.pitch;
    }
  }
  a.H = H; a.T = T; a.N = N; a.mask_full = mask_full; a.fb = forget_bias; a.prefix = prefix_dev;
  int rc = dyb200_rec_fwd(ctx, p, &a, ndir);
  for (int k = 0; k < ndir && !rc; ++k) if (dirs[k].w) dyb200_wgrad_h_done(dirs[k].w);
  return rc;
}

int dyb200i_rec_bwd(dyb200_ctx* ctx, int ndir, const dyb200i_rec_dir* dirs, uint32_t H, uint32_t T, uint32_t N, const uint32_t* prefix_dev,
                    int mask_full, uint32_t columns) {
  { int rc0__ = dyb200_scratch_begin(ctx); if (rc0__) return rc0__; }
  RecPlan p;
  DYB_CHECK_ARG(ctx, (ndir == 1 || ndir == 2) && dyb200_rec_plan(ctx, H, &p), "lstm recurrence: %u units are outside its range", H);
  RecBwd a;
  memset(&a, 0, sizeof(a));
  float* db[2] = {nullptr, nullptr};
  for (int k = 0; k < ndir; ++k) {
    const dyb200i_rec_dir& s = dirs[k];
    RecDirB& d = a.d[k];
    d.Wh = s.Wh; d.gates = s.gates; d.c = s.c; d.c0 = s.c0; d.dh = s.dh; d.dc = s.dc; d.mask = s.mask_h;
    DYB_CHECK_ARG(ctx, s.w && dyb200_wgrad_rows(s.w) == 4 * H, "lstm recurrence: the accumulator does not belong to this layer");
    int rc = dyb200_wgrad_reserve_a_at(s.w, 0, columns, &d.dn_hi, &d.dn_lo, &a.dn_pitch, ctx);
    if (rc) return rc;
    db[k] = s.db;
  }
  a.H = H; a.T = T; a.N = N; a.mask_full = mask_full; a.prefix = prefix_dev;
  return dyb200_rec_bwd(ctx, p, &a, ndir, db);
}

int dyb200i_rec_dx(dyb200_ctx* ctx, dyb200_wgrad* w, const float* Wx, uint32_t I, uint32_t H, uint32_t columns, const float* mask_x, int mask_full,
                   uint32_t period, float* dx) {
  { int rc0__ = dyb200_scratch_begin(ctx); if (rc0__) return rc0__; }
  const uint32_t G = 4 * H;
  PackedOp A, D;
  DYB_CHECK_ARG(ctx, dyb200_wgrad_rows(w) == G && dyb200_wgrad_column_planes(w, columns, &D, nullptr, nullptr), "lstm recurrence: the accumulator does not belong to this layer");
  int rc = dyb200_tc_param(ctx, Wx, G, true, I, G, &A);
  if (rc) return rc;
  if (!mask_x) {
    GemmEpilogue e{EPI_ACCUM, dx, I, nullptr, 0, 0.f, nullptr, 0, 0};
    return dyb200_tc_gemm_packed(ctx, I, columns, 1, &A, &D, e);
  }
  void* tmp;
  if ((rc = dyb200_scratch(ctx, (size_t)I * columns * sizeof(float), &tmp))) return rc;
  GemmEpilogue e{EPI_STORE, (float*)tmp, I, nullptr, 0, 0.f, nullptr, 0, 0};
  if ((rc = dyb200_tc_gemm_packed(ctx, I, columns, 1, &A, &D, e))) return rc;
  const size_t total = (size_t)I * columns;
  dyb_launch(k_masked_add, stream_grid(ctx, total, 256), 256, 0, ctx, (const float*)tmp, mask_x, I, mask_full ? period : 0u, total, dx);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

}  // extern "C"
