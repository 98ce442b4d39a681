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
//   * h_t (forward) goes to every CTA of the cluster through distributed shared memory as 16-byte messages that complete an
//     mbarrier of the receiver (st.async): no fence, no polling of global memory, two buffers.  A barrier of the whole cluster
//     per step instead took 1.9 us per step at 2 - 4 columns, most of it the release of the step's global stores.  Backward,
//     each CTA reduces over its own gate rows and sends partial sums of dE/dh_{t-1} to the CTA that owns the unit, 4 x fewer
//     bytes than handing dgates around.
//   * plain fp32 multiply-adds: more accurate than the 3xTF32 products of the per-step form, and at 1 - 8 columns per cluster
//     the tensor pipe could not be filled anyway.  (Not fma.rn.f32x2: with two 64-bit register operands and a 64-bit
//     accumulator it issued once in four cycles here, half the rate of the scalar form.)
// The arithmetic order is fixed by the shape (cluster count, ranks, lanes): reproducible run to run.
//
// Every warp sends its own part as soon as it has it (no barrier of the CTA).  Buffers are free to be overwritten without a
// further hand-shake: a warp sends h_t only after the h_{t-1} of every warp of the cluster has arrived, and each of those was
// sent after that warp had read the buffer that h_t goes to.
//
// Thread layout, forward: 16 lanes per pair of hidden units (slice s of the reduction index: k = 64 j + 4 s + 0..3, so the
// slices read 256 contiguous bytes of h without bank conflicts), 8 gate rows x KD k per lane - with one unit per 8 lanes the
// loads of h took as many cycles as the multiply-adds.  NB columns at a time; a butterfly over the 16 lanes leaves each lane
// with all four gates of one unit and column.
// Backward: 8 lanes per group of 8 units of dE/dh_{t-1}, slices of the CTA's own 4 U gate rows in the same pattern.
#include "lstm_rec.cuh"

#include "gemm.cuh"
#include "lstm_cell.cuh"
#include "lstm_rec_api.h"
#include "lstm_rec_dev.cuh"

namespace {

__device__ __forceinline__ float xor_add(float keep, float send, int m) { return keep + __shfl_xor_sync(0xffffffffu, send, m); }

// columns of a cluster that are active at a step of width B: those i < cap with first + step i < B
__device__ __forceinline__ uint32_t active_cols(uint32_t B, uint32_t first, uint32_t step, uint32_t cap) {
  return B > first ? min((B - first + step - 1) / step, cap) : 0;
}

// grid (C, G, directions), cluster (C, 1, 1); block = 8 U threads.
// Dynamic shared memory: h[2][ncap][16 KD], c[ncap][U].  NB columns per block, NF of them computed (3 of 4, or all).
template <int KD, int NB, int NF = NB>
__global__ void __launch_bounds__(256, 1) k_lstm_rec_fwd(const __grid_constant__ RecFwd a) {
  constexpr int HP = 16 * KD;
  extern __shared__ __align__(16) float rec_smem[];
  __shared__ __align__(8) uint64_t got[2];
  __shared__ __align__(16) float stage_all[8][NB * 4];
  const RecDirF d = blockIdx.z ? a.d[1] : a.d[0];
  const uint32_t H = a.H, U = a.U, g = blockIdx.y, g0 = g * a.first, gi = a.step, gc = a.cap, rank = blockIdx.x, C = gridDim.x, ncap = a.ncap;
  const uint32_t tid = threadIdx.x, s = tid & 15, ul0 = 2 * (tid >> 4);   // slice, first of the lane's two units
  const uint32_t ul = ul0 + (s >> 3), u = rank * U + ul;                  // the unit this lane finishes
  const bool live_u = u < H;
  float* hbuf = rec_smem;
  float* cbuf = hbuf + (size_t)2 * ncap * HP;
  float* stage = stage_all[tid >> 5];                                     // h of this warp's 4 units, column by column
  const uint32_t lane = tid & 31, u_warp = rank * U + 4 * (tid >> 5);
  if (tid == 0) {
    msg_init(&got[0]);
    msg_init(&got[1]);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  dyb_grid_dep_wait();   // (the next kernel starts when this one's CTAs end: early, its own would hold SMs for a whole sequence)

  // the column of a block that this lane finishes; 8 / NB lanes share one (they hold equal values; dup == 0 stores)
  const uint32_t lc = NB == 8 ? (s & 7) : NB == 4 ? (s & 7) >> 1 : NB == 2 ? (s & 7) >> 2 : 0;
  const uint32_t dup = NB == 8 ? 0 : NB == 4 ? (s & 1) : NB == 2 ? (s & 3) : (s & 7);
  const uint32_t ncol = active_cols(a.N, g0, gi, gc);
  uint32_t phase[2] = {0, 0};
  bool ok = true;
  uint32_t col0 = 0, B = a.prefix ? a.prefix[1] : a.N;      // first column and width of the step
  uint32_t n = active_cols(B, g0, gi, gc);
  float pre[4], mk, pre_next[4], mk_next;
  // Wx x + b and the mask of this lane's column of a block, asked for a block or step ahead.  (Behind a block's stores they came in after the h they are
  // added to: 200 - 480 of a step's 3 800 cycles at 256 units and 3 columns.)
  auto fetch = [&](uint32_t c0, uint32_t nact, uint32_t nb) {
    const uint32_t i = nb + lc, sc = g0 + gi * i;
    if (live_u && i < nact) {
      const float* p = d.gates + u + (size_t)4 * H * (c0 + sc);
#pragma unroll
      for (int q = 0; q < 4; ++q) pre_next[q] = p[(size_t)q * H];
      mk_next = d.mask ? d.mask[u + (a.mask_full ? (size_t)H * sc : 0)] : 1.f;
    } else {
      pre_next[0] = pre_next[1] = pre_next[2] = pre_next[3] = mk_next = 0.f;
    }
  };
  fetch(col0, n, 0);

  // The CTA's rows of Wh come in as they lie in memory (16 bytes of U neighbouring units of one gate and column per lane), pass
  // through shared memory and stay in registers.  For 128 KB: 3 000 cycles; 4-byte loads took 4 500 - 7 000 (twice that when
  // they miss L2), 128-byte bulk copies 7 500.  Row k is shifted by the slice that reads it, so that the 16 slices meet 16
  // pairs of banks.
  const uint32_t WP = 4 * U + 32;
  {
    const bool vec = (H & 3) == 0 && aligned16(d.Wh);
    const uint32_t nq = U / 4, total = 64 * KD * nq;
    for (uint32_t e0 = tid; e0 < total; e0 += 8 * blockDim.x) {
      float4 v[8];
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const uint32_t e = e0 + x * blockDim.x, seg = e / nq, k = seg / 4, q = seg % 4, uu = rank * U + 4 * (e % nq);
        const float* p = d.Wh + (size_t)q * H + uu + (size_t)4 * H * k;
        v[x] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k < H && uu < H) {
          if (vec) v[x] = __ldg(reinterpret_cast<const float4*>(p));
          else {
            v[x].x = __ldg(p);
            if (uu + 1 < H) v[x].y = __ldg(p + 1);
            if (uu + 2 < H) v[x].z = __ldg(p + 2);
            if (uu + 3 < H) v[x].w = __ldg(p + 3);
          }
        }
      }
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const uint32_t e = e0 + x * blockDim.x, seg = e / nq, k = seg / 4, q = seg % 4;
        if (e < total) {
          float2* dst = reinterpret_cast<float2*>(rec_smem + (size_t)k * WP + 2 * (k / 4 % 16) + q * U + 4 * (e % nq));
          dst[0] = make_float2(v[x].x, v[x].y);
          dst[1] = make_float2(v[x].z, v[x].w);
        }
      }
    }
  }
  __syncthreads();
  float w[8][KD];   // row 4 (unit of the pair) + gate
#pragma unroll
  for (int x = 0; x < KD; ++x)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float2 v = *reinterpret_cast<const float2*>(rec_smem + (size_t)(64 * (x / 4) + 4 * s + x % 4) * WP + 2 * s + q * U + ul0);
      w[q][x] = v.x;
      w[4 + q][x] = v.y;
    }
  __syncthreads();

  // h_{-1} and c_{-1} of the cluster's columns, the operand planes of the first step's h input; zeros in the padding of h
  for (uint32_t e = tid; e < 2 * ncap * HP / 4; e += blockDim.x) reinterpret_cast<float4*>(hbuf)[e] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
#pragma unroll 2
  for (uint32_t e = tid; e < ncol * H; e += blockDim.x) {
    const uint32_t i = e / H, k = e % H, sc = g0 + gi * i;
    const bool own = k / U == rank;
    float v = d.h0 ? __ldg(d.h0 + k + (size_t)H * sc) : 0.f;
    const float m = d.mask ? __ldg(d.mask + k + (a.mask_full ? (size_t)H * sc : 0)) : 1.f, c = own && d.c0 ? __ldg(d.c0 + k + (size_t)H * sc) : 0.f;
    v *= m;
    hbuf[(size_t)i * HP + k] = v;
    if (own) {
      cbuf[i * U + k % U] = c;
      if (d.hn_hi) {
        float hi, lo;
        split_tf32(v, hi, lo);
        d.hn_hi[(size_t)sc * a.hn_pitch + k] = hi;
        d.hn_lo[(size_t)sc * a.hn_pitch + k] = lo;
      }
    }
  }
  cluster_arrive();
  cluster_wait();

  for (uint32_t t = 0; t < a.T && n > 0; ++t) {
    const uint32_t pt = t & 1, pn = pt ^ 1;
    const float* hcur = hbuf + (size_t)pt * ncap * HP;
    const uint32_t hnext = smem_addr(hbuf + (size_t)pn * ncap * HP);
    const uint32_t col1 = col0 + B;                                          // the next step
    const uint32_t B1 = t + 1 < a.T ? (a.prefix ? a.prefix[t + 2] - a.prefix[t + 1] : a.N) : 0;
    const uint32_t n1 = active_cols(B1, g0, gi, gc);
    if (n1 && tid == 0) msg_expect(&got[pn], n1 * C * U * 4);   // (only the columns that go on are handed over)
    if (t > 0) {
      ok = ok && msg_wait(&got[pt], phase[pt]);
      phase[pt] ^= 1;
    }
#pragma unroll 1
    for (uint32_t nb = 0; nb < n; nb += NB) {
#pragma unroll
      for (int q = 0; q < 4; ++q) pre[q] = pre_next[q];
      mk = mk_next;
      if (nb + NB < n) fetch(col0, n, nb + NB);
      else if (n1) fetch(col1, n1, 0);
      float acc[8][NB];   // (columns NF .. NB - 1 stay zero)
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < NB; ++c) acc[r][c] = 0.f;
      const float* hp = hcur + (size_t)nb * HP + 4 * s;
#pragma unroll
      for (int j = 0; j < KD / 4; ++j)
#pragma unroll
        for (int c = 0; c < NF; ++c) {
          const float4 hh = ld4(hp + (size_t)c * HP + 64 * j);
#pragma unroll
          for (int r = 0; r < 8; ++r) acc[r][c] = fmaf(w[r][4 * j], hh.x, acc[r][c]);
#pragma unroll
          for (int r = 0; r < 8; ++r) acc[r][c] = fmaf(w[r][4 * j + 1], hh.y, acc[r][c]);
#pragma unroll
          for (int r = 0; r < 8; ++r) acc[r][c] = fmaf(w[r][4 * j + 2], hh.z, acc[r][c]);
#pragma unroll
          for (int r = 0; r < 8; ++r) acc[r][c] = fmaf(w[r][4 * j + 3], hh.w, acc[r][c]);
        }
      // sum over the 16 slices: first the units, then the columns are split between the lanes; what is left is added on both
      float z[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float v[NB];
        const bool hi_unit = (s & 8) != 0;
#pragma unroll
        for (int c = 0; c < NB; ++c) {
          const float v0 = acc[q][c], v1 = acc[4 + q][c];
          v[c] = xor_add(hi_unit ? v1 : v0, hi_unit ? v0 : v1, 8);
        }
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
      const uint32_t i = nb + lc, sc = g0 + gi * i;
      const bool mine = live_u && i < n;
      float cn = 0.f, hv = 0.f, hm = 0.f;
      if (mine) {
        z[0] = gate_sigmoid(z[0] + pre[0]);
        z[1] = gate_sigmoid(z[1] + pre[1] + a.fb);
        z[2] = gate_sigmoid(z[2] + pre[2]);
        z[3] = gate_tanh(z[3] + pre[3]);
        cn = lstm_cell_c(z[0], z[3], z[1], cbuf[i * U + ul]);
        hv = lstm_cell_h(z[2], cn);
        hm = hv * mk;
      }
      if (dup == 0) stage[lc * 4 + (ul & 3)] = hm;
      __syncwarp();             // (also: all lanes of the unit have read the old cell state)
      if (n1 > nb) {
        // the warp hands its 4 units of the block over: one 16-byte message per column and CTA
        const uint32_t n_send = min(n1 - nb, (uint32_t)NB);
        for (uint32_t e = lane; e < NB * C; e += 32) {
          const uint32_t c = e % NB, r = e / NB;
          if (c < n_send)
            send4(map_rank(hnext + 4u * ((nb + c) * HP + u_warp), r), *reinterpret_cast<const float4*>(stage + 4 * c), map_rank(smem_addr(&got[pn]), r));
        }
      }
      if (mine && dup == 0) {   // gates, c, h and the operand planes of the next step's input
        cbuf[i * U + ul] = cn;
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
      }
      __syncwarp();             // (the unit's other lanes read the new cell state in the next step)
    }
    col0 = col1; B = B1; n = n1;
  }
  cluster_arrive();                // nobody leaves while a neighbour may still send to it
  cluster_wait();
  if (!ok) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
}

// grid (C, G, directions), cluster (C, 1, 1); block = C U threads rounded up to warps.  KD = gate rows per slice: 8 KD >= 4 U.
// Dynamic shared memory: part[2][C][ncap][U], dg[2][ncap][8 KD], dcs[ncap][U].  (dg in two: a step's gradients are written as soon
// as the sums of the step before have arrived, which some warps of this CTA may still be forming for other CTAs.)
template <int KD, int NB, int NF = NB, int MT = KD == 16 ? 256 : 384>   // MT: most threads of a CTA
__global__ void __launch_bounds__(MT, 1) k_lstm_rec_bwd(const __grid_constant__ RecBwd a) {
  constexpr int KP = 8 * KD;
  extern __shared__ __align__(16) float rec_smem[];
  __shared__ __align__(8) uint64_t got[2];
  __shared__ __align__(16) float stage_all[12][NB * 32];
  const RecDirB d = blockIdx.z ? a.d[1] : a.d[0];
  const uint32_t H = a.H, U = a.U, g = blockIdx.y, g0 = g * a.first, gi = a.step, gc = a.cap, rank = blockIdx.x, C = gridDim.x, ncap = a.ncap;
  const uint32_t tid = threadIdx.x, s = tid & 7, og = tid >> 3;
  float* part = rec_smem;                                   // [parity][source rank][column][unit]
  float* dg = part + (size_t)2 * C * ncap * U;
  float* dcs = dg + (size_t)2 * ncap * KP;
  float* stage = stage_all[tid >> 5];                       // partial sums of this warp's 32 units, column by column
  // message of this lane: 4 units of column lane / 8 of a block, for the CTA that owns them
  const uint32_t lane = tid & 31, o_msg = 32 * (tid >> 5) + 4 * (lane & 7), r_msg = o_msg / U;
  const bool msg_live = o_msg < C * U;
  if (tid == 0) {
    msg_init(&got[0]);
    msg_init(&got[1]);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  dyb_grid_dep_wait();

  // weights: outputs o = 8 og + 0..7 (units of h_{t-1}) x this CTA's gate rows kk = q U + unit, slice s
  float w[8][KD];
  const bool quads = (H & 3) == 0 && aligned16(d.Wh);
#pragma unroll
  for (int o = 0; o < 8; ++o)
#pragma unroll
    for (int j = 0; j < KD / 4; ++j) {
      // (U is a multiple of 4: the four rows are one gate's rows of four neighbouring units)
      const uint32_t kk = 32 * j + 4 * s, q = kk / U, uu = rank * U + kk % U, oo = 8 * og + o;
      const float* p = d.Wh + (size_t)q * H + uu + (size_t)4 * H * oo;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (q < 4 && uu < H && oo < H) {
        if (quads) v = __ldg(reinterpret_cast<const float4*>(p));
        else {
          v.x = __ldg(p);
          if (uu + 1 < H) v.y = __ldg(p + 1);
          if (uu + 2 < H) v.z = __ldg(p + 2);
          if (uu + 3 < H) v.w = __ldg(p + 3);
        }
      }
      w[o][4 * j] = v.x; w[o][4 * j + 1] = v.y; w[o][4 * j + 2] = v.z; w[o][4 * j + 3] = v.w;
    }
  // cell pass: thread -> (unit c_ul, columns c_i0, c_i0 + c_step, ...)
  const uint32_t c_step = blockDim.x / U, c_ul = tid % U, c_i0 = tid / U, c_u = rank * U + c_ul;
  const bool c_live = c_i0 < c_step && c_u < H;
  float db[4] = {0.f, 0.f, 0.f, 0.f};
  uint32_t phase[2] = {0, 0};
  bool ok = true;

  for (uint32_t e = tid; e < 2 * ncap * KP; e += blockDim.x) dg[e] = 0.f;
  for (uint32_t e = tid; e < ncap * U; e += blockDim.x) dcs[e] = 0.f;
  cluster_arrive();
  cluster_wait();
  // the last step that has a column of this cluster: widths never grow, so the steps before it have one too
  uint32_t T = a.T;
  while (a.prefix && T > 0 && active_cols(a.prefix[T] - a.prefix[T - 1], g0, gi, gc) == 0) --T;

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
  uint32_t n = T ? active_cols(start_of(T) - col, g0, gi, gc) : 0;
  if (T && c_live && c_i0 < n) fetch(T - 1, col, T > 1 ? start_of(T - 2) : 0, g0 + gi * c_i0);
  for (uint32_t t = T; t-- > 0;) {
    const uint32_t colm1 = t ? start_of(t - 1) : 0, pin = (t + 1) & 1, pout = t & 1;
    const float* from = part + (size_t)pin * C * ncap * U;
    if (t && tid == 0) msg_expect(&got[pout], n * C * U * 4);
    if (n_later) {
      ok = ok && msg_wait(&got[pin], phase[pin]);
      phase[pin] ^= 1;
    }
    // ---- gradients of the gate pre-activations of this CTA's units ----
    if (c_live)
      for (uint32_t i = c_i0; i < n; i += c_step) {
        const uint32_t sc = g0 + gi * i;
        if (i != c_i0) fetch(t, col, colm1, sc);
        float dh = dhv;
        if (i < n_later) {
          float r = 0.f;
          for (uint32_t q = 0; q < C; ++q) r += from[((size_t)q * ncap + i) * U + c_ul];
          if (d.mask) r *= d.mask[c_u + (a.mask_full ? (size_t)H * sc : 0)];
          dh += r;
          d.dh[c_u + (size_t)H * (col + sc)] = dh;
        }
        float dcp = 0.f, pr[4];
        const float dci = dcv + dcs[i * U + c_ul];
        if (d.dc && i < n_later) d.dc[c_u + (size_t)H * (col + sc)] = dci;
        lstm_cell_grad(gt[0], gt[1], gt[2], gt[3], cv, cp, dh, dci, true, dcp, pr[0], pr[1], pr[2], pr[3]);
        dcs[i * U + c_ul] = dcp;
        float* dgi = dg + (size_t)((t & 1) * ncap + i) * KP + c_ul;
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
    const uint32_t nm1 = active_cols(col - colm1, g0, gi, gc);
    if (c_live && c_i0 < nm1) fetch(t - 1, colm1, t > 1 ? start_of(t - 2) : 0, g0 + gi * c_i0);
    // ---- partial sums of dE/dh_{t-1} over this CTA's gate rows ----
#pragma unroll 1
    for (uint32_t nb = 0; nb < n; nb += NB) {
      float acc[8][NB];
#pragma unroll
      for (int o = 0; o < 8; ++o)
#pragma unroll
        for (int c = 0; c < NB; ++c) acc[o][c] = 0.f;
      const float* gp = dg + (size_t)((t & 1) * ncap + nb) * KP + 4 * s;
#pragma unroll
      for (int j = 0; j < KD / 4; ++j)
#pragma unroll
        for (int c = 0; c < NF; ++c) {
          const float4 hh = ld4(gp + (size_t)c * KP + 32 * j);
#pragma unroll
          for (int o = 0; o < 8; ++o) acc[o][c] = fmaf(w[o][4 * j], hh.x, acc[o][c]);
#pragma unroll
          for (int o = 0; o < 8; ++o) acc[o][c] = fmaf(w[o][4 * j + 1], hh.y, acc[o][c]);
#pragma unroll
          for (int o = 0; o < 8; ++o) acc[o][c] = fmaf(w[o][4 * j + 2], hh.z, acc[o][c]);
#pragma unroll
          for (int o = 0; o < 8; ++o) acc[o][c] = fmaf(w[o][4 * j + 3], hh.w, acc[o][c]);
        }
#pragma unroll
      for (int c = 0; c < NF; ++c) {
        float v[8];
#pragma unroll
        for (int o = 0; o < 8; ++o) v[o] = acc[o][c];
#pragma unroll
        for (int m = 4; m >= 1; m >>= 1) {
          const bool up = (s & m) != 0;
#pragma unroll
          for (int o = 0; o < 4; ++o)
            if (o < m) v[o] = xor_add(up ? v[o + m] : v[o], up ? v[o] : v[o + m], m);
        }
        stage[c * 32 + lane] = v[0];   // (lane 8 g + s holds unit 8 g + s of the warp's 32)
      }
      __syncwarp();
      // the warp hands its sums over: 8 messages of 4 units per column, each to the CTA that owns those units
      if (NB * 8 >= 32 || lane < NB * 8) {
        const uint32_t c = lane >> 3;
        if (msg_live && nb + c < n)
          send4(map_rank(smem_addr(part + (((size_t)pout * C + rank) * ncap + nb + c) * U + o_msg % U), r_msg),
                *reinterpret_cast<const float4*>(stage + c * 32 + 4 * (lane & 7)), map_rank(smem_addr(&got[pout]), r_msg));
      }
      __syncwarp();
    }
    n_later = n; n = nm1; col = colm1;
  }
  cluster_arrive();                // nobody leaves while a neighbour may still send to it
  cluster_wait();
  if (!ok) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
  // row sums of dgates: the threads of one unit, in ascending order (part is free: every CTA is through)
  __syncthreads();
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

constexpr size_t kRecSmemMax = 216 * 1024;
// Most columns a cluster carries: at 32 - 64 columns a step takes 0.3 us per column and cluster, as much as the per-step tensor
// products take for the whole GPU; wider batches stay with those.
constexpr uint32_t kRecCols = 64;

typedef void (*FwdKernel)(RecFwd);
typedef void (*BwdKernel)(RecBwd);
// (registers: 8 KD weights + 8 NB sums in both kernels, at most 255 per thread.  Three columns are a variant of their own: up to
// 45 columns on the 15 clusters of 8 CTAs that fit.)
FwdKernel fwd_kernel(uint32_t kd, uint32_t n) {
#define REC_F4(K) n == 1 ? k_lstm_rec_fwd<K, 1> : n == 2 ? k_lstm_rec_fwd<K, 2> : n == 3 ? k_lstm_rec_fwd<K, 4, 3>
#define REC_F(K) (REC_F4(K) : k_lstm_rec_fwd<K, 4>)
  switch (kd) {
    case 4: return REC_F(4);
    case 8: return REC_F(8);
    case 12: return REC_F(12);
    case 16: return REC_F(16);
    case 20: return REC_F(20);
    default: return n == 1 ? k_lstm_rec_fwd<24, 1> : k_lstm_rec_fwd<24, 2>;
  }
#undef REC_F
#undef REC_F4
}
// (16 gate rows per lane: 255 registers at up to 256 units and threads, 168 at up to 320, where the instances of two and of three columns spill 48 and 28
// bytes; fewer rows: up to 384 threads of 168)
BwdKernel bwd_kernel(uint32_t kd, uint32_t n, uint32_t threads) {
#define REC_B(K) (n == 1 ? k_lstm_rec_bwd<K, 1> : n == 2 ? k_lstm_rec_bwd<K, 2> : n == 3 ? k_lstm_rec_bwd<K, 4, 3> : k_lstm_rec_bwd<K, 4>)
  if (kd == 16 && threads > 256)
    return n == 1 ? k_lstm_rec_bwd<16, 1, 1, 320> : n == 2 ? k_lstm_rec_bwd<16, 2, 2, 320> : n == 3 ? k_lstm_rec_bwd<16, 4, 3, 320> : k_lstm_rec_bwd<16, 4, 4, 320>;
  switch (kd) {
    case 8: return REC_B(8);
    case 12: return REC_B(12);
    default: return REC_B(16);
  }
#undef REC_B
}
uint32_t fwd_threads(const RecPlan& p) { return 8 * p.U; }
uint32_t bwd_threads(const RecPlan& p) { return (p.C * p.U + 31) / 32 * 32; }
// shared memory: per column carried, and for Wh on its way into registers (forward)
size_t fwd_col_bytes(const RecPlan& p) { return sizeof(float) * (2 * 16 * p.KD + p.U); }
size_t bwd_col_bytes(const RecPlan& p) { return sizeof(float) * (2 * p.C * p.U + 2 * 8 * p.KD2 + p.U); }
size_t fwd_smem(const RecPlan& p, uint32_t ncap) {
  const size_t cols = ncap * fwd_col_bytes(p), weights = sizeof(float) * (16 * p.KD * (4 * p.U + 32) + 32);
  return cols > weights ? cols : weights;
}

}  // namespace

int dyb200_rec_launch_cfg(dyb200_ctx* ctx, const void* kernel, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, dim3 grid, uint32_t threads, size_t smem) {
  DYB_CUDA(ctx, dyb_smem_limit(kernel, smem, kRecSmemMax));
  if (grid.x > 8) DYB_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  memset(cfg, 0, sizeof(*cfg));
  cfg->gridDim = grid; cfg->blockDim = dim3(threads, 1, 1); cfg->dynamicSmemBytes = smem; cfg->stream = ctx->stream;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = grid.x; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg->attrs = attr; cfg->numAttrs = 1;
  return DYB200_OK;
}
namespace {

// How many clusters run side by side (remembered per context and width class): the columns are dealt out over that many.
int clusters_that_fit(dyb200_ctx* ctx, const RecPlan& p, bool bwd, uint32_t threads) {
  const uint32_t C = p.C;
  int16_t& fit = ctx->rec_fit[bwd][p.KD / 4 - 1][C];
  if (fit == 0) {
    const void* k = bwd ? (const void*)bwd_kernel(p.KD2, 4, threads) : (const void*)fwd_kernel(p.KD, 4);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    if (dyb200_rec_launch_cfg(ctx, k, &cfg, attr, dim3(C, 1, 1), threads, kRecSmemMax)) return -1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = -1; }
    fit = (int16_t)(n > 0 ? n : -1);
  }
  return fit;
}
// Clusters per direction and columns per cluster; false when a cluster would have to carry more than it can.
bool deal_columns(uint32_t N, int fit, int ndir, size_t col_bytes, uint32_t* G, uint32_t* ncap) {
  const uint32_t g = fit > ndir ? (uint32_t)(fit / ndir) : 1u;
  *G = N < g ? N : g;
  *ncap = ((N + *G - 1) / *G + 7) / 8 * 8;
  return *ncap <= kRecCols && *ncap * col_bytes <= kRecSmemMax;
}

}  // namespace

bool dyb200_rec_plan(dyb200_ctx* ctx, uint32_t H, uint32_t N, int ndir, RecPlan* out) {
  if (H == 0 || H > 384 || N == 0) return false;
  RecPlan p;
  // up to 256 units: 32 per CTA and at most 8 CTAs, the portable cluster size; beyond: 16 CTAs
  p.U = H <= 256 ? (H < 32 ? (H + 3) / 4 * 4 : 32u) : ((H + 15) / 16 + 3) / 4 * 4;
  // From 8 columns on: 32 per CTA also up to 320 units (beyond, a CTA's weights do not pass through its shared memory), since more clusters
  // of 10 CTAs than of 16 run side by side: 300 units, 35 steps, forward: 30 columns 149 -> 94 us, 130 317 -> 222, 300 656 -> 466; backward, 30 columns
  // 115 -> 86 us.  Below, every column has a cluster of its own either way, and the smaller CTAs are through sooner: 4 columns 70 against 75 us.
  if (H > 256 && H <= 320 && N >= 8) p.U = 32;
  p.C = (H + p.U - 1) / p.U;
  p.KD = (H + 63) / 64 * 4;
  p.KD2 = p.U <= 16 ? 8 : p.U <= 24 ? 12 : 16;
  const int ff = clusters_that_fit(ctx, p, false, fwd_threads(p)), fb = clusters_that_fit(ctx, p, true, bwd_threads(p));
  const bool sf = ff > 0 && deal_columns(N, ff, ndir, fwd_col_bytes(p), &p.Gf, &p.ncapf), sb = fb > 0 && deal_columns(N, fb, ndir, bwd_col_bytes(p), &p.Gb, &p.ncapb);
  // More than four columns per cluster: the tensor pipe, where the width lets it (256 units, a step: 1.8 us here at 3 columns,
  // 8.0 at 37; there 2.5 at any number)
  p.tcf = !(sf && (N + p.Gf - 1) / p.Gf <= 4) && dyb200_rec_tc_plan(ctx, false, H, N, ndir, &p.tf);
  p.tcb = !(sb && (N + p.Gb - 1) / p.Gb <= 4) && dyb200_rec_tc_plan(ctx, true, H, N, ndir, &p.tb);
  if (!(sf || p.tcf) || !(sb || p.tcb)) return false;
  *out = p;
  return true;
}

// Clusters that a sequence of constant width runs on: as many as it takes with the columns that the fullest one has anyway (16 columns over 15
// clusters are two columns' time, and so they are over 8).  The others' SMs are left to other streams: three language models of 256
// units and 16 columns on three streams 103.6 -> 85.9 us a step, of 300 units and 30 columns 475 -> 440; a layer by itself is as fast.  (Where the width shrinks from step to step
// more clusters have fewer columns for longer.)
constexpr uint32_t kBlockCols = 4;   // the most columns an instance of the kernels takes at a time
static uint32_t clusters_needed(uint32_t N, uint32_t G, const uint32_t* prefix) {
  const uint32_t cols = (N + G - 1) / G;
  return prefix && cols > kBlockCols ? G : (N + cols - 1) / cols;
}
// Which columns cluster g has: first * g + step * i, i < cap.  Neighbouring ones where they are one block of the kernel, which costs the same whatever is
// left of it: the clusters of a ragged batch's short sequences then end early: taggers of 16 sentences of 5 to
// 60 tokens on three streams 198 -> 188 us a step (one by itself: forward 100 -> 103 us, where the last steps of every cluster had a column left, backward
// 97 both; of 24 sentences, four columns a cluster: forward 125 -> 130, backward 114 both, a pass by itself 453 -> 457, three on three streams 236 -> 193).  More than a block: every G-th column, so that all
// clusters lose columns alike.
template <class Args>
static void deal(Args* a, uint32_t G) {
  const uint32_t cols = (a->N + G - 1) / G;
  const bool block = cols <= kBlockCols;
  a->G = G; a->first = block ? cols : 1u; a->step = block ? 1u : G; a->cap = block ? cols : 0xffffffffu;
}

int dyb200_rec_fwd(dyb200_ctx* ctx, const RecPlan& p, RecFwd* a, int ndir) {
  if (p.tcf) return dyb200_rec_tc_fwd(ctx, p.tf, a, ndir);
  const uint32_t G = clusters_needed(a->N, p.Gf, a->prefix);
  deal(a, G);
  a->U = p.U; a->ncap = p.ncapf; a->flags = ctx->dev_flags;
  FwdKernel k = fwd_kernel(p.KD, (a->N + G - 1) / G);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  int rc = dyb200_rec_launch_cfg(ctx, (const void*)k, &cfg, attr, dim3(p.C, G, ndir), fwd_threads(p), fwd_smem(p, p.ncapf));
  if (rc) return rc;
  cudaLaunchKernelEx(&cfg, k, *a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

int dyb200_rec_bwd(dyb200_ctx* ctx, const RecPlan& p, RecBwd* a, int ndir, float* const* db) {
  const uint32_t rows = 4 * a->H, G = p.tcb ? p.tb.G : clusters_needed(a->N, p.Gb, a->prefix);
  deal(a, G);
  a->U = p.U; a->ncap = p.ncapb; a->flags = ctx->dev_flags;
  void* part;
  int rc = dyb200_scratch(ctx, (size_t)ndir * G * rows * sizeof(float), &part);
  if (rc) return rc;
  for (int k = 0; k < ndir; ++k) a->d[k].dbpart = (float*)part + (size_t)k * G * rows;
  if (p.tcb) {
    if ((rc = dyb200_rec_tc_bwd(ctx, p.tb, a, ndir))) return rc;
  } else {
    BwdKernel k = bwd_kernel(p.KD2, (a->N + G - 1) / G, bwd_threads(p));
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    rc = dyb200_rec_launch_cfg(ctx, (const void*)k, &cfg, attr, dim3(p.C, G, ndir), bwd_threads(p), p.ncapb * bwd_col_bytes(p));
    if (rc) return rc;
    cudaLaunchKernelEx(&cfg, k, *a);
    DYB_LAUNCHED(ctx);
  }
  dyb_launch(k_rec_db, dim3((rows + 255) / 256, ndir), 256, 0, ctx, (const float*)a->d[0].dbpart, (const float*)a->d[ndir - 1].dbpart, G, rows,
             db[0], db[ndir - 1]);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

// ---- products over all columns around the recurrence -----------------------------------------------------------------------
namespace {

// dst (+)= src .* mask, all `rows` x n; the mask repeats every `period` columns (0: one column for all)
__global__ void __launch_bounds__(256) k_masked_add(const float* __restrict__ src, const float* __restrict__ mask, uint32_t rows, uint32_t period,
                                                    size_t total, float* __restrict__ dst, int overwrite) {
  dyb_grid_dep_sync();
  for (size_t e = (size_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (size_t)gridDim.x * 256) {
    const uint32_t n = (uint32_t)(e / rows), r = (uint32_t)(e % rows);
    dst[e] = __fmaf_rn(src[e], mask[r + (period ? (size_t)rows * (n % period) : 0)], overwrite ? 0.f : dst[e]);
  }
}

}  // namespace

extern "C" {

int dyb200i_rec_takes(dyb200_ctx* ctx, uint32_t H, uint32_t T, uint32_t N, int ndir) {
  RecPlan p;
  return ctx->seq_kernels && T >= kRecMinSteps && dyb200_rec_plan(ctx, H, N, ndir, &p) ? 1 : 0;
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
  DYB_CHECK_ARG(ctx, (ndir == 1 || ndir == 2) && dyb200_rec_plan(ctx, H, N, ndir, &p), "lstm recurrence: %u units x %u columns are outside its range", H, N);
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
  DYB_CHECK_ARG(ctx, (ndir == 1 || ndir == 2) && dyb200_rec_plan(ctx, H, N, ndir, &p), "lstm recurrence: %u units x %u columns are outside its range", H, N);
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
                   uint32_t period, float* dx, int overwrite) {
  { int rc0__ = dyb200_scratch_begin(ctx); if (rc0__) return rc0__; }
  const uint32_t G = 4 * H;
  PackedOp A, D;
  DYB_CHECK_ARG(ctx, dyb200_wgrad_rows(w) == G && dyb200_wgrad_column_planes(w, columns, &D, nullptr, nullptr), "lstm recurrence: the accumulator does not belong to this layer");
  int rc = dyb200_tc_param(ctx, Wx, G, true, I, G, &A);
  if (rc) return rc;
  if (!mask_x) {
    GemmEpilogue e{overwrite ? EPI_STORE : EPI_ACCUM, dx, I, nullptr, 0, 0.f, nullptr, 0, 0};
    return dyb200_tc_gemm_packed(ctx, I, columns, 1, &A, &D, e);
  }
  void* tmp;
  if ((rc = dyb200_scratch(ctx, (size_t)I * columns * sizeof(float), &tmp))) return rc;
  GemmEpilogue e{EPI_STORE, (float*)tmp, I, nullptr, 0, 0.f, nullptr, 0, 0};
  if ((rc = dyb200_tc_gemm_packed(ctx, I, columns, 1, &A, &D, e))) return rc;
  const size_t total = (size_t)I * columns;
  dyb_launch(k_masked_add, stream_grid(ctx, total, 256), 256, 0, ctx, (const float*)tmp, mask_x, I, mask_full ? period : 0u, total, dx, overwrite);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

}  // extern "C"
