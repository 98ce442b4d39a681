// One LSTM layer over ALL time steps of a sequence in one kernel (forward): the call pattern of
// CompactVanillaLSTMBuilder::add_input_impl (dynet/lstm.cc:1044-1080) driven through RNNBuilder::add_input
// (dynet/rnn.h:120) for a batch of equally long sequences, i.e. T times
//     gates_t = VanillaLSTMGates(x_t, h_{t-1}, Wx, Wh, b [, masks]);  c_t = VanillaLSTMC(c_{t-1}, gates_t);
//     h_t = VanillaLSTMH(c_t, gates_t).
// The per-step form (dyb200_vanilla_lstm_fwd_fused_at) launches one 3xTF32 product per step (wide layers: this kernel with T = 1).  Here the CTAs of that
// product stay resident for the whole sequence: CTA (mt, nt[, split]) owns the same 128 interleaved gate rows (32 hidden
// units) x BNT batch columns in every step.  What that buys per step: no launch gap, no TMEM allocation / barrier set-up /
// tensor-map fetch, and the Wx x_{t+1} share of a step's k-blocks (which does not depend on h_t) runs while the epilogue of
// step t is still writing and handing over.  The weights are not kept in shared memory; their split planes stay in L2.
//
// Hand-over of h_t: the epilogue writes h_t .* mask_h as TF32 hi / lo operand planes (rows = batch columns) and then
// adds 1 to a counter of its column block; the TMA warp of every CTA of that column block waits for the count of the
// previous step before its first Wh h k-block.  The wait is bounded like every other wait of these kernels: on expiry
// the CTA sets DYB200_FLAG_WAIT_TIMEOUT, skips its stores, keeps taking part in the hand-shakes so that nothing else
// stalls, frees its TMEM and returns.
//
// Values are bit for bit those of the per-step calls: the same k-blocks in the same accumulation chains (cut every
// kChunkKB k-blocks), the same K split (k_split) reduced in split order through distributed shared memory, the same epilogue.
#include "seq_dev.cuh"
#include "lstm_rec_api.h"
#include "lstm_wide.cuh"

namespace {

struct SeqFwd {
  uint32_t T, B, H;                 // time steps, batch columns per step, hidden units (M = 4H gate rows)
  uint32_t kb0, kb1;                // k-blocks of Wx x and of Wh h
  float* gates; float* cs; float* hs;   // outputs of step t at + t * 4H * B / + t * H * B
  const float* c0;                  // cell state before the first step
  const float* bias; float forget_bias;
  // operand planes of h .* mask_h: row = column of the sequence (K-major right operand of the gate products; the layer's
  // weight-gradient product reads the same planes MN-major)
  float *hn_hi, *hn_lo; uint32_t hn_pitch;
  const float* hmask; uint32_t hmask_ld; int hmask_full;
  int emit_last;                    // the last step's h goes out as operand planes too (a single step of a sequence driven from outside)
  // F16: scale words of the gate rows (row q H + u of Wx, 4H further on of Wh), of the columns of x (sequence columns), of h_{-1} (batch columns) and of all
  // later h (batch columns, or one for all; null: |h| < 1), and the planes of h .* mask_h as fp16 pairs: two slots of B rows, step t reads
  // slot t % 2
  const uint32_t *gate_scale, *x_scale, *h0_scale, *h_scale; int h_scale_full;
  __half *h16_hi, *h16_lo; uint32_t h16_pitch;
  uint32_t* ready;                  // one arrival counter per column block, zero at launch
  uint32_t* flags;
};

__device__ __forceinline__ uint32_t h_word(const SeqFwd& a, uint32_t n) { return a.h_scale && n < a.B ? __ldg(a.h_scale + (a.h_scale_full ? n : 0)) : 0x3f800000u; }

// F16: the products of wide layers on scaled fp16 pairs (gemm.cuh) in k-blocks of 64 - half the weight bytes from L2 per step and 0.61 us per 64 k
// instead of 2 x 0.66.  The weights' planes are MN-major as they lie, their rows interleaved like the TF32 ones; a scale per gate row of Wx and of Wh.
// A column of x has a scale of its own, h .* mask_h one that is known beforehand (|h| < 1: the largest mask value of the column), h_{-1} the
// larger of that and its own; so accumulation chains end between Wx x and Wh h, and a chain is unscaled as it is drained.  (Elements of h below 2^-28 of
// the mask's largest value keep an absolute error of 2^-50 of it, as those of a column of x and of a row of weights do of theirs: below the 2^-24
// that an activation is rounded to, as long as a column's largest |x| times a row's sum of |w|, and a row's largest |w| times a column's sum of |x|, stay below 2^25.)
// grid = (4H / 128, B / BNT, S); with S > 1 the S CTAs of a tile are one thread-block cluster (1 x 1 x S).  S (1, 2, 4 or 8) is
// a template parameter so that the column exchange indexes registers statically.
// VEC: units in fours, on 16 bytes (otherwise, F16 only, a value at a time; those on 128-column tiles spill 464 - 592 bytes: 512 x 777 x 500 columns 23 us a
// step, launch by launch 53).
template <int BNT, uint32_t S, bool F16, bool VEC = true>
__global__ void __launch_bounds__(kThreads, 1) k_lstm_seq_fwd(const __grid_constant__ TmapPack tm, const SeqFwd a) {
  if (a.T == 1) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // (behind a sequence the next kernel starts when this one ends)
  // 64-column tiles need 48 KiB per stage, so the ring holds four of them: at 0.4 us per k-block three stages do not cover
  // the latency of a tile fetch
  constexpr int kStages = BNT == 64 ? 4 : 3;
  constexpr int kStageBytes = 2 * TILE_BYTES + 2 * BNT * BK * 4;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kStages], empty_bar[kStages], acc_full[kSeqBufs], acc_empty[kSeqBufs], park_full, park_free;
  __shared__ uint32_t tmem_base_slot;
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* park = reinterpret_cast<float*>(ring + (size_t)kStages * kStageBytes);   // 64 columns x BM rows
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int TILE_B_BYTES = BNT * BK * 4;
  constexpr int STAGE_TX = 2 * TILE_BYTES + 2 * TILE_B_BYTES;
  const uint32_t rank = blockIdx.z;
  const uint32_t m0 = blockIdx.x * BM, n0 = blockIdx.y * BNT;
  const KSplit ks = k_split(a.kb0, a.kb1, rank, S);
  const uint32_t total = ks.n0 + ks.n1;          // k-blocks of this CTA per time step
  const uint32_t M = 4 * a.H, N = a.B;
  constexpr uint32_t kAccCols = F16 ? 2 * BNT : BN, kBufs = F16 ? kSeqBufs * BN / kAccCols : kSeqBufs, kChunk = F16 ? kChunkF16 : kChunkKB;
  constexpr int EL = F16 ? 64 : 32;
  constexpr uint32_t kHalf = BNT / 2, kParkBytes = 64 * BM * 4;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (uint32_t q = 0; q < kSeqBufs; ++q) { mbar_init(&acc_full[q], 1); mbar_init(&acc_empty[q], kEpiWarps); }
    mbar_init(&park_full, 1); mbar_init(&park_free, S);   // the bytes of a pass, 64 columns, whoever sends them / an arrival per CTA
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (S > 1) mbar_expect_tx(&park_full, kParkBytes);
  }
  if (threadIdx.x == 32 * 2) {
#pragma unroll
    for (int q = 0; q < 8; ++q) asm volatile("prefetch.tensormap [%0];" ::"l"(&tm.t[q]) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(kSeqBufs * BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_slot;
  if (S > 1) cluster_sync_all();   // every CTA's barriers exist before anyone arrives on them remotely
  dyb_grid_dep_wait();

  if (warp == 0) {
    if (elect_one()) {
      // TMA producer.  Step t reads Wx / Wh rows [m0, m0 + 128) and the operand planes of columns [t B + n0, + BNT).
      uint32_t s = 0, ph = 0;
      bool fail = false;
      const uint32_t per_step = gridDim.x * S;   // arrivals per column block and step: every CTA that writes a piece of h_t
      for (uint32_t t = 0; t < a.T && !fail; ++t) {
        const int brow = (int)(t * a.B + n0), hrow = F16 ? (int)((t & 1) * a.B + n0) : brow;
        for (uint32_t it = 0; it < total;) {
          if (it == ks.n0 && t > 0) {
            // The Wh h share of this step needs the planes of h_{t-1}, complete for this column block.  The weight tiles
            // of its first k-blocks do not: they are requested before the wait (a stage's barrier completes when both its
            // weight and its activation tiles have arrived), so only the small activation tiles are still to come afterwards.
            const uint32_t pre = min((uint32_t)kStages, ks.n1);
            uint32_t s2 = s, ph2 = ph;
            for (uint32_t j = 0; j < pre && !fail; ++j) {
              if (!mbar_wait(&empty_bar[s2], ph2 ^ 1)) { fail = true; break; }
              unsigned char* st = ring + (size_t)s2 * kStageBytes;
              mbar_expect_tx(&full_bar[s2], STAGE_TX);
              load_a_tile<EL>(st, &tm.t[4], &full_bar[s2], ks.b1 + j, m0, F16);
              load_a_tile<EL>(st + TILE_BYTES, &tm.t[5], &full_bar[s2], ks.b1 + j, m0, F16);
              if (++s2 == kStages) { s2 = 0; ph2 ^= 1; }
            }
            if (fail) break;
            if (!wait_counter(a.ready + blockIdx.y, t * per_step)) { fail = true; break; }
            asm volatile("fence.proxy.async.global;" ::: "memory");   // generic-proxy stores of other CTAs -> this CTA's TMA reads
            for (uint32_t j = 0; j < pre; ++j) {
              unsigned char* st = ring + (size_t)s * kStageBytes;
              tma_load_2d(st + 2 * TILE_BYTES, &tm.t[6], &full_bar[s], (int)((ks.b1 + j) * EL), hrow);
              tma_load_2d(st + 2 * TILE_BYTES + TILE_B_BYTES, &tm.t[7], &full_bar[s], (int)((ks.b1 + j) * EL), hrow);
              if (++s == kStages) { s = 0; ph ^= 1; }
            }
            it += pre;
            continue;
          }
          if (!mbar_wait(&empty_bar[s], ph ^ 1)) { fail = true; break; }
          const uint32_t pair = it < ks.n0 ? 0 : 1, kblk = pair ? ks.b1 + (it - ks.n0) : ks.b0 + it;
          unsigned char* st = ring + (size_t)s * kStageBytes;
          mbar_expect_tx(&full_bar[s], STAGE_TX);
          load_a_tile<EL>(st, &tm.t[4 * pair + 0], &full_bar[s], kblk, m0, F16);
          load_a_tile<EL>(st + TILE_BYTES, &tm.t[4 * pair + 1], &full_bar[s], kblk, m0, F16);
          tma_load_2d(st + 2 * TILE_BYTES, &tm.t[4 * pair + 2], &full_bar[s], (int)(kblk * EL), pair ? hrow : brow);
          tma_load_2d(st + 2 * TILE_BYTES + TILE_B_BYTES, &tm.t[4 * pair + 3], &full_bar[s], (int)(kblk * EL), pair ? hrow : brow);
          if (++s == kStages) { s = 0; ph ^= 1; }
          ++it;
        }
      }
      if (fail) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = (1u << 4) | (F16 ? 1u << 15 : (2u << 7) | (2u << 10)) | ((uint32_t)(BNT >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      const uint32_t idesc_wide = idesc + ((uint32_t)(BNT >> 3) << 17);
      uint64_t d_a_hi[kStages], d_a_lo[kStages], d_b_hi[kStages], d_b_lo[kStages];
#pragma unroll
      for (int q = 0; q < kStages; ++q) {
        const uint32_t base = smem_u32(ring + (size_t)q * kStageBytes);
        d_a_hi[q] = F16 ? umma_desc_mn16(base) : umma_desc(base); d_a_lo[q] = F16 ? umma_desc_mn16(base + TILE_BYTES) : umma_desc(base + TILE_BYTES);
        d_b_hi[q] = umma_desc(base + 2 * TILE_BYTES); d_b_lo[q] = umma_desc(base + 2 * TILE_BYTES + TILE_B_BYTES);
      }
      // stage, phase and chunk counters run on across time steps; an accumulation chain never crosses a step
      uint32_t s = 0, ph = 0, chunk = 0, buf = 0;
      bool fail = false;
      for (uint32_t t = 0; t < a.T && !fail; ++t) {
        uint32_t in_chunk = 0;
        for (uint32_t it = 0; it < total; ++it) {
          if (in_chunk == 0 && chunk >= kBufs) {
            if (!mbar_wait(&acc_empty[buf], ((chunk / kBufs) - 1) & 1)) { fail = true; break; }
          }
          if (!mbar_wait(&full_bar[s], ph)) { fail = true; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          uint64_t a_hi, a_lo, b_hi, b_lo;   // select without dynamic register indexing
          if (s == 0) { a_hi = d_a_hi[0]; a_lo = d_a_lo[0]; b_hi = d_b_hi[0]; b_lo = d_b_lo[0]; }
          else if (s == 1) { a_hi = d_a_hi[1]; a_lo = d_a_lo[1]; b_hi = d_b_hi[1]; b_lo = d_b_lo[1]; }
          else if (s == 2 || kStages == 3) { a_hi = d_a_hi[2]; a_lo = d_a_lo[2]; b_hi = d_b_hi[2]; b_lo = d_b_lo[2]; }
          else { a_hi = d_a_hi[kStages - 1]; a_lo = d_a_lo[kStages - 1]; b_hi = d_b_hi[kStages - 1]; b_lo = d_b_lo[kStages - 1]; }
          if (F16) issue_kblock_f16(tmem_base + buf * kAccCols, tmem_base + buf * kAccCols + BNT, a_hi, a_lo, b_hi, idesc_wide, idesc, in_chunk, 128, 2);
          else issue_kblock(tmem_base + buf * kAccCols, a_hi, a_lo, b_hi, b_lo, idesc, in_chunk);
          umma_commit(&empty_bar[s]);
          const bool chunk_ends = in_chunk == kChunk - 1 || it == total - 1 || (F16 && it + 1 == ks.n0);
          if (chunk_ends) { umma_commit(&acc_full[buf]); in_chunk = 0; ++chunk; buf = chunk % kBufs; }
          else ++in_chunk;
          if (++s == kStages) { s = 0; ph ^= 1; }
        }
      }
      if (fail) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
    }
  } else {
    // epilogue warps 2..9: TMEM lanes 32 (warp % 4) .. +31; warps 2-5 drain the tile's first BNT / 2 columns, warps 6-9 the others
    const uint32_t quarter = warp & 3, half = (warp - 2) >> 2, row = quarter * 32 + lane;
    const uint32_t te = threadIdx.x - 64;
    const uint32_t x_chunks = (ks.n0 + kChunk - 1) / kChunk;   // (F16: those of Wx x)
    const uint32_t nchunks = F16 ? x_chunks + (ks.n1 + kChunk - 1) / kChunk : (total + kChunk - 1) / kChunk;
    // The tile is finished in passes of 64 columns: pass hh takes columns [32 hh, + 32) of either half, position p of a pass being column p % 32 of the
    // half p / 32.  In the cooperative pass this thread owns hidden units [u, u + 4) (rows 32 q + l of the tile are gate q of unit 32 mt + l) at the
    // positions te / 8 and te / 8 + 32.
    const uint32_t l = 4 * (te & 7), u = blockIdx.x * 32 + l;
    const bool own_u = u < a.H;
    const uint32_t left = a.H - u;   // (own_u) units from u on
    auto column = [&](int hh, uint32_t p) { return (p >> 5) * kHalf + 32 * hh + (p & 31); };
    // F16: 2^-s of this thread's gate row in Wx and in Wh; of the columns lane (and lane + 32) of its half (h after the first step); and 2^s of the columns it finishes
    float row_x = 1.f, row_h = 1.f, h_f[kHalf / 32], h_s[BNT / 64][2];
    const uint32_t hn0 = n0 + half * kHalf + lane;
    if (F16) {
      if (32 * blockIdx.x + lane < a.H) {
        row_x = inv_scale_of(__ldg(a.gate_scale + (size_t)quarter * a.H + 32 * blockIdx.x + lane));
        row_h = inv_scale_of(__ldg(a.gate_scale + (size_t)(4 + quarter) * a.H + 32 * blockIdx.x + lane));
      }
#pragma unroll
      for (uint32_t k = 0; k < kHalf / 32; ++k) h_f[k] = inv_scale_of(h_word(a, hn0 + 32 * k));
#pragma unroll
      for (int hh = 0; hh < BNT / 64; ++hh)
#pragma unroll
        for (int k = 0; k < 2; ++k) h_s[hh][k] = scale_of(h_word(a, n0 + column(hh, (te >> 3) + 32 * k)));
    }
    // The positions of a pass are finished by the S CTAs of the cluster, w each: rank r takes [r w, + w).  Every CTA sends its partial sums of those
    // columns straight into rank r's exchange buffer (slot = sender's rank), so the owner adds S slots from its own shared memory - no remote loads, whose
    // round trips would sit on the step's critical path.  Without a K split (S = 1) the buffer is simply the parked pass.
    constexpr uint32_t w = 64 / S;
    const uint32_t c_lo = rank * w, c_hi = c_lo + w;
    float4 bias[4];   // the same for every step
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      bias[q] = own_u ? ldu<VEC>(a.bias + (size_t)q * a.H + u, left) : make_float4(0.f, 0.f, 0.f, 0.f);
      if (q == 1) { bias[q].x += a.forget_bias; bias[q].y += a.forget_bias; bias[q].z += a.forget_bias; bias[q].w += a.forget_bias; }
    }
    uint32_t cg = 0, pf_phase = 0, pr_phase = 0;
    bool ok = true;   // the same for all 256 epilogue threads after every bar_and below
    const size_t HB = (size_t)a.H * a.B;
#pragma unroll 1
    for (uint32_t t = 0; t < a.T; ++t) {
      float* const gates_t = a.gates + (size_t)t * 4 * HB;
      const float* const c_prev = t ? a.cs + (size_t)(t - 1) * HB : a.c0;
      float* const c_out = a.cs + (size_t)t * HB;
      float* const h_out = a.hs + (size_t)t * HB;
      const bool emit = t + 1 < a.T || a.emit_last;   // h_t is the next step's input
      // h_t .* mask_h as operand planes of step t + 1: rows (t + 1) B .. of the planes
      float* const hn_hi = a.hn_hi + (size_t)(t + 1) * a.B * a.hn_pitch;
      float* const hn_lo = a.hn_lo + (size_t)(t + 1) * a.B * a.hn_pitch;
      // previous cell states and mask values of the columns this thread finishes (c_prev was written by this same thread one
      // step earlier); fetched now, while the products of the step run
      float4 cp[BNT / 64][2], hm[BNT / 64][2];
#pragma unroll
      for (int hh = 0; hh < BNT / 64; ++hh)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const uint32_t c = (te >> 3) + 32 * k, n = n0 + column(hh, c);
          const bool mine = own_u && n < N && c >= c_lo && c < c_hi;
          cp[hh][k] = mine ? ldu<VEC>(c_prev + u + (size_t)a.H * n, left) : make_float4(0.f, 0.f, 0.f, 0.f);
          hm[hh][k] = (mine && a.hmask) ? ldu<VEC>(a.hmask + u + (a.hmask_full ? (size_t)a.hmask_ld * n : 0), left) : make_float4(1.f, 1.f, 1.f, 1.f);
        }
      float f[kHalf / 32], row_f = row_x;   // F16: 2^-s of the columns lane (and lane + 32) in the coming chains, and of the row
#pragma unroll
      for (uint32_t k = 0; k < kHalf / 32; ++k) f[k] = F16 && hn0 + 32 * k < N ? inv_scale_of(__ldg(a.x_scale + (size_t)t * a.B + hn0 + 32 * k)) : 1.f;
      float sum[kHalf];
#pragma unroll
      for (uint32_t q = 0; q < kHalf; ++q) sum[q] = 0.f;
#pragma unroll 1
      for (uint32_t c = 0; c < nchunks; ++c, ++cg) {
        const uint32_t buf = cg % kBufs;
        if (F16 && c == x_chunks) {
          row_f = row_h;
#pragma unroll
          for (uint32_t k = 0; k < kHalf / 32; ++k) f[k] = t || hn0 + 32 * k >= N ? h_f[k] : inv_scale_of(__ldg(a.h0_scale + hn0 + 32 * k));
        }
        if (!ok) continue;
        if (!mbar_wait(&acc_full[buf], (cg / kBufs) & 1)) { ok = false; continue; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr = tmem_base + buf * kAccCols + ((quarter * 32) << 16) + half * kHalf;
        if (F16) {
#pragma unroll
          for (uint32_t p = 0; p < kHalf / 16; ++p) {   // (16 columns of both accumulators at a time)
            float v1[16], v2[16];
            tmem_ld16x2(taddr + 16 * p, taddr + BNT + 16 * p, v1, v2);
#pragma unroll
            for (int q = 0; q < 16; ++q)
              // (both factors at once: the sum times one of them may leave fp32's range where the product does not)
              sum[16 * p + q] = fmaf(fmaf(v2[q], kLoScale, v1[q]), row_f * __shfl_sync(0xffffffffu, f[p / 2], 16 * (p % 2) + q), sum[16 * p + q]);
          }
        } else {
#pragma unroll
          for (uint32_t p = 0; p < kHalf / 32; ++p) {
            float v[32];
            tmem_ld32(taddr + 32 * p, v);
#pragma unroll
            for (int q = 0; q < 32; ++q) sum[32 * p + q] += v[q];
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);
      }
#pragma unroll
      for (int hh = 0; hh < BNT / 64; ++hh) {
        // Every CTA's exchange buffer is free once its owner has read the previous pass: the owners say so on park_free
        // (S > 1), or this CTA's own threads have left the previous pass (the barrier at its end).
        if (S > 1 && ok && !mbar_wait_cluster(&park_free, pr_phase ^ 1)) ok = false;
        if (S > 1) {
#pragma unroll
          for (uint32_t rr = 0; rr < S / 2; ++rr) {
            const uint32_t to = mapa_u32(smem_u32(park), half * (S / 2) + rr) + 4u * (rank * w * BM), bar = mapa_u32(smem_u32(&park_full), half * (S / 2) + rr);
#pragma unroll
            for (uint32_t q = 0; q < w; q += 4)   // position q + lane % 4 of the rank's, rows of the lane's quad
              send4(to + 4u * park_at(q + (lane & 3), row >> 2), transpose4(sum + (32 * hh + rr * w + q) % kHalf, lane), bar);
          }
          const bool got = mbar_wait_cluster(&park_full, pf_phase);
          ok = bar_and(1, 256, ok && got) != 0;
          pf_phase ^= 1; pr_phase ^= 1;
          if (te == 0) mbar_expect_tx(&park_full, kParkBytes);   // (the next pass; it begins when this CTA has arrived on the others' park_free)
        } else {
#pragma unroll
          for (uint32_t q = 0; q < 32; ++q) park[park_at(32 * half + q, row >> 2) + (row & 3)] = sum[32 * hh + q];
          ok = bar_and(1, 256, ok) != 0;
        }
        // ---- the LSTM epilogue on this CTA's columns of the half: the arithmetic of epilogue_pass (EPI_LSTM_CELL), the S
        // partial sums added in split order, c / h / the operand planes of h.  The planes of h, which the next step waits for,
        // go out first and are published before the other stores are issued.
        const bool last_pass = hh == BNT / 64 - 1;
        float4 g[2][4], cn[2], hv[2], phi[2], plo[2];
        bool live[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const uint32_t c = (te >> 3) + 32 * k, n = n0 + column(hh, c);
          live[k] = ok && own_u && n < N && c >= c_lo && c < c_hi;
          if (!live[k]) continue;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float* col = park + park_at(c - c_lo, 8 * q + (te & 7));
            float4 acc = ld4(col);
#pragma unroll
            for (uint32_t r = 1; r < S; ++r) { const float4 pv = ld4(col + (size_t)r * w * BM); acc.x += pv.x; acc.y += pv.y; acc.z += pv.z; acc.w += pv.w; }
            const float4 x = make_float4(acc.x + bias[q].x, acc.y + bias[q].y, acc.z + bias[q].z, acc.w + bias[q].w);
            g[k][q] = q == 3 ? make_float4(gate_tanh(x.x), gate_tanh(x.y), gate_tanh(x.z), gate_tanh(x.w))
                             : make_float4(gate_sigmoid(x.x), gate_sigmoid(x.y), gate_sigmoid(x.z), gate_sigmoid(x.w));
          }
          const float4 cv = cp[hh][k];
          cn[k] = make_float4(lstm_cell_c(g[k][0].x, g[k][3].x, g[k][1].x, cv.x), lstm_cell_c(g[k][0].y, g[k][3].y, g[k][1].y, cv.y),
                              lstm_cell_c(g[k][0].z, g[k][3].z, g[k][1].z, cv.z), lstm_cell_c(g[k][0].w, g[k][3].w, g[k][1].w, cv.w));
          hv[k] = make_float4(lstm_cell_h(g[k][2].x, cn[k].x), lstm_cell_h(g[k][2].y, cn[k].y), lstm_cell_h(g[k][2].z, cn[k].z), lstm_cell_h(g[k][2].w, cn[k].w));
          if (!VEC) { if (left < 2) hv[k].y = 0.f; if (left < 3) hv[k].z = 0.f; if (left < 4) hv[k].w = 0.f; }   // (the planes' padding stays zero)
          if (emit) {
            // h .* mask_h as the next step's operand planes (the values of epi_emit_h)
            const float4 mk = hm[hh][k];
            const float4 hmk = a.hmask ? make_float4(hv[k].x * mk.x, hv[k].y * mk.y, hv[k].z * mk.z, hv[k].w * mk.w) : hv[k];
            split_tf32(hmk.x, phi[k].x, plo[k].x); split_tf32(hmk.y, phi[k].y, plo[k].y);
            split_tf32(hmk.z, phi[k].z, plo[k].z); split_tf32(hmk.w, phi[k].w, plo[k].w);
            if (a.hn_hi) {
              st4(hn_hi + (size_t)n * a.hn_pitch + u, phi[k]);
              st4(hn_lo + (size_t)n * a.hn_pitch + u, plo[k]);
            }
            if (F16 && t + 1 < a.T) {
              // (of the value that the TF32 pair stands for, as a single step's call makes it of those planes)
              const float hs = h_s[hh][k];
              __half ph[4], pl[4];
              split_f16((phi[k].x + plo[k].x) * hs, ph[0], pl[0]); split_f16((phi[k].y + plo[k].y) * hs, ph[1], pl[1]);
              split_f16((phi[k].z + plo[k].z) * hs, ph[2], pl[2]); split_f16((phi[k].w + plo[k].w) * hs, ph[3], pl[3]);
              const size_t o = (size_t)(((t + 1) & 1) * a.B + n) * a.h16_pitch + u;
              *reinterpret_cast<uint2*>(a.h16_hi + o) = *reinterpret_cast<const uint2*>(ph);
              *reinterpret_cast<uint2*>(a.h16_lo + o) = *reinterpret_cast<const uint2*>(pl);
            }
          }
        }
        // all reads of the exchange buffer are done (the next pass may overwrite it) and, in the last pass, every thread has
        // issued its stores of the operand planes
        bar_sync(1, 256);
        if (S > 1 && te < S) mbar_arrive_remote(&park_free, te);
        if (last_pass && emit && te == 0) {
          // One thread publishes: its release orders all stores it has observed, through the barrier, before the counter
          // update (cumulativity), for the generic and for the async proxy (the readers are TMA loads).
          asm volatile("fence.proxy.async.global;" ::: "memory");
          signal_counter(a.ready + blockIdx.y);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          if (!live[k]) continue;
          const uint32_t n = n0 + column(hh, (te >> 3) + 32 * k);
#pragma unroll
          for (int q = 0; q < 4; ++q) stu<VEC>(gates_t + (size_t)q * a.H + u + (size_t)M * n, g[k][q], left);
          const size_t ei = u + (size_t)a.H * n;
          stu<VEC>(c_out + ei, cn[k], left);
          stu<VEC>(h_out + ei, hv[k], left);
        }
      }
    }
    if (!ok && lane == 0) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (S > 1) cluster_sync_all();   // no CTA leaves while another may still arrive on its barriers
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kSeqBufs * BN) : "memory");
  }
}

}  // namespace

// ---- host side ---------------------------------------------------------------------------------------------------------
namespace {

// How many clusters of S CTAs of the sequence kernel fit on the GPU at once (remembered per context = per device).
template <int BNT, uint32_t S, bool F16, bool VEC>
int seq_clusters_that_fit(dyb200_ctx* ctx) {
  int& mc = ctx->seq_max_clusters[(BNT == 64 ? 0 : 1) + (F16 ? VEC ? 2 : 4 : 0)][S];
  if (mc == 0) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(1, 1, S); cfg.blockDim = dim3(kThreads, 1, 1); cfg.dynamicSmemBytes = SMEM_SEQ_BYTES; cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = S;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_lstm_seq_fwd<BNT, S, F16, VEC>, &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = -1; }
    mc = n > 0 ? n : -1;
  }
  return mc;
}

template <int BNT, uint32_t S, bool F16, bool VEC>
int launch_seq_fwd(dyb200_ctx* ctx, const TmapPack& tm, const SeqFwd& a, dim3 grid, double flops, uint32_t K) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = grid; cfg.blockDim = dim3(kThreads, 1, 1); cfg.dynamicSmemBytes = SMEM_SEQ_BYTES; cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (grid.z > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = grid.z;
    ++na;
  }
  // All CTAs wait on one another, so they have to be resident together.  The grid never exceeds what the GPU holds at
  // once (checked by the caller); the cooperative attribute additionally makes the driver schedule them as one gang.  A
  // driver that refuses the attribute for this launch shape gets a plain launch (the waits are bounded either way).
  if (ctx->seq_coop >= 0 && a.T > 1) {   // (a single step's CTAs wait for nobody but their cluster)
    attr[na].id = cudaLaunchAttributeCooperative;
    attr[na].val.cooperative = 1;
    cfg.attrs = attr; cfg.numAttrs = na + 1;
    GemmProfScope scope(ctx, flops, F16 ? 2 : 1, 4 * a.H, a.B * a.T, K, EPI_LSTM_CELL);
    cudaError_t e = cudaLaunchKernelEx(&cfg, k_lstm_seq_fwd<BNT, S, F16, VEC>, tm, a);
    if (e == cudaSuccess) { ctx->seq_coop = 1; ctx->launches++; return DYB200_OK; }
    (void)cudaGetLastError();
    if (ctx->seq_coop == 1) return dyb200_fail(ctx, DYB200_ECUDA, "sequence kernel launch failed: %s", cudaGetErrorString(e));
    ctx->seq_coop = -1;
  }
  if (F16 && a.T == 1 && ctx->pdl) {   // (a single step's prologue runs beside the short kernel that makes its pairs)
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    ++na;
  }
  cfg.attrs = attr; cfg.numAttrs = na;
  GemmProfScope scope(ctx, flops, F16 ? 2 : 1, 4 * a.H, a.B * a.T, K, EPI_LSTM_CELL);
  cudaLaunchKernelEx(&cfg, k_lstm_seq_fwd<BNT, S, F16, VEC>, tm, a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

// the (tile width, K splits) instantiations behind one switch
enum SeqOp { SEQ_SET_SMEM, SEQ_FIT, SEQ_LAUNCH };
template <int BNT, uint32_t S, bool F16, bool VEC>
int seq_fwd_do(SeqOp op, dyb200_ctx* ctx, const TmapPack* tm, const SeqFwd* a, dim3 grid, double flops, uint32_t K) {
  if (op == SEQ_SET_SMEM) {
    // (the shared-memory limit of the kernel has to be raised before its occupancy is asked for)
    const uint32_t log_s = S == 1 ? 0 : S == 2 ? 1 : S == 4 ? 2 : 3, bit = (F16 ? (BNT == 64 ? 1u << 12 : 1u << 16) : BNT == 64 ? 16u : 256u) << log_s;
    uint32_t& done = VEC ? ctx->func_attr_done : ctx->seq_odd_attr_done;
    if (!(done & bit)) {
      DYB_CUDA(ctx, cudaFuncSetAttribute(k_lstm_seq_fwd<BNT, S, F16, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_SEQ_BYTES));
      done |= bit;
    }
    return DYB200_OK;
  }
  if (op == SEQ_FIT) return seq_clusters_that_fit<BNT, S, F16, VEC>(ctx);
  return launch_seq_fwd<BNT, S, F16, VEC>(ctx, *tm, *a, grid, flops, K);
}
template <bool F16, bool VEC = true>
int seq_fwd_dispatch(SeqOp op, uint32_t bn, uint32_t S, dyb200_ctx* ctx, const TmapPack* tm = nullptr, const SeqFwd* a = nullptr,
                     dim3 grid = dim3(), double flops = 0, uint32_t K = 0) {
  if (bn == 64) {
    switch (S) {
      case 1: return seq_fwd_do<64, 1, F16, VEC>(op, ctx, tm, a, grid, flops, K);
      case 2: return seq_fwd_do<64, 2, F16, VEC>(op, ctx, tm, a, grid, flops, K);
      case 4: return seq_fwd_do<64, 4, F16, VEC>(op, ctx, tm, a, grid, flops, K);
      default: return seq_fwd_do<64, 8, F16, VEC>(op, ctx, tm, a, grid, flops, K);
    }
  }
  switch (S) {
    case 1: return seq_fwd_do<128, 1, F16, VEC>(op, ctx, tm, a, grid, flops, K);
    case 2: return seq_fwd_do<128, 2, F16, VEC>(op, ctx, tm, a, grid, flops, K);
    case 4: return seq_fwd_do<128, 4, F16, VEC>(op, ctx, tm, a, grid, flops, K);
    default: return seq_fwd_do<128, F16 ? 4 : 8, F16, VEC>(op, ctx, tm, a, grid, flops, K);
  }
}

// the F16 form for units in fours and for others
int seq_f16_dispatch(SeqOp op, bool vec, uint32_t bn, uint32_t S, dyb200_ctx* ctx, const TmapPack* tm = nullptr, const SeqFwd* a = nullptr, dim3 grid = dim3(), double flops = 0,
                     uint32_t K = 0) {
  return vec ? seq_fwd_dispatch<true, true>(op, bn, S, ctx, tm, a, grid, flops, K) : seq_fwd_dispatch<true, false>(op, bn, S, ctx, tm, a, grid, flops, K);
}

// ---- the inputs of the F16 form, one launch: a warp per line ----
// x: planes of the columns' inputs (hi + lo, or the values themselves without lo planes) -> fp16 pairs, a word per line.  h_{-1}: h0 .* mask -> TF32 planes (unless they are in place) and
// fp16 pairs of what those stand for, a word per line: the largest of its values and the mask's.  mask: the words alone.
struct SeqPrep {
  const float *x_hi, *x_lo; uint32_t x_ld, I, x_lines; __half *x16_hi, *x16_lo; uint32_t x16_pitch; uint32_t* x_scale;
  const float *h0, *mask; uint32_t H, B; int mask_full, h0_done; float *hn_hi, *hn_lo; uint32_t hn_pitch; __half *h16_hi, *h16_lo; uint32_t h16_pitch; uint32_t* h0_scale;
  uint32_t mask_lines; uint32_t* h_scale;
};
__global__ void __launch_bounds__(256) k_seq_prep(const __grid_constant__ SeqPrep a) {
  dyb_grid_dep_sync();
  uint32_t line = blockIdx.x * 8 + (threadIdx.x >> 5);
  const uint32_t lane = threadIdx.x & 31;
  const int kind = line < a.x_lines ? 0 : line < a.x_lines + a.B ? 1 : 2;
  line -= kind == 0 ? 0 : kind == 1 ? a.x_lines : a.x_lines + a.B;
  if (kind == 2 && line >= a.mask_lines) return;
  const uint32_t n = kind == 0 ? a.I : a.H;
  const float *p = kind == 0 ? a.x_hi + (size_t)line * a.x_ld : kind == 1 ? a.h0 + (size_t)line * a.H : a.mask + (size_t)line * a.H;
  const float *p2 = kind == 0 ? (a.x_lo ? a.x_lo + (size_t)line * a.x_ld : nullptr) : kind == 1 && a.mask ? a.mask + (a.mask_full ? (size_t)line * a.H : 0) : nullptr;
  const bool vec = aligned16(p) && (!p2 || aligned16(p2));
  auto mag = [](float4 v) { return max(max(finite_mag(v.x), finite_mag(v.y)), max(finite_mag(v.z), finite_mag(v.w))); };
  uint32_t m = kind == 1 && !p2 ? 0x3f800000u : 0;   // (h_{-1}: no smaller than the scale of later h, which an h_{-1} from a call for the step before is)
  auto four = [&](const float* q, uint32_t e) {   // (zeros past the line's end)
    if (vec && e + 4 <= n) return ld4(q + e);
    return make_float4(q[e], e + 1 < n ? q[e + 1] : 0.f, e + 2 < n ? q[e + 2] : 0.f, e + 3 < n ? q[e + 3] : 0.f);
  };
  auto value = [&](uint32_t e) {   // elements [e, e + 4)
    float4 v = four(p, e);
    if (p2) {
      const float4 w = four(p2, e);
      if (kind == 0) v = make_float4(v.x + w.x, v.y + w.y, v.z + w.z, v.w + w.w);
      else {
        v = make_float4(v.x * w.x, v.y * w.y, v.z * w.z, v.w * w.w);
        m = max(m, mag(w));
      }
    }
    if (kind == 1) {
      float4 hi, lo;
      split_tf32(v.x, hi.x, lo.x); split_tf32(v.y, hi.y, lo.y); split_tf32(v.z, hi.z, lo.z); split_tf32(v.w, hi.w, lo.w);
      if (!a.h0_done && a.hn_hi) { st4(a.hn_hi + (size_t)line * a.hn_pitch + e, hi); st4(a.hn_lo + (size_t)line * a.hn_pitch + e, lo); }
      v = make_float4(hi.x + lo.x, hi.y + lo.y, hi.z + lo.z, hi.w + lo.w);
    }
    return v;
  };
  float4 keep[8];   // lines of up to 1024 values stay in registers between the scale and the split
#pragma unroll
  for (uint32_t k = 0; k < 8; ++k) if (4 * lane + 128 * k < n) { keep[k] = value(4 * lane + 128 * k); m = max(m, mag(keep[k])); }
  for (uint32_t e = 1024 + 4 * lane; e < n; e += 128) m = max(m, mag(value(e)));
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0) (kind == 0 ? a.x_scale : kind == 1 ? a.h0_scale : a.h_scale)[line] = m;
  if (kind == 2) return;
  const float s = scale_of(m);
  __half* const dh = kind == 0 ? a.x16_hi + (size_t)line * a.x16_pitch : a.h16_hi + (size_t)line * a.h16_pitch;
  __half* const dl = kind == 0 ? a.x16_lo + (size_t)line * a.x16_pitch : a.h16_lo + (size_t)line * a.h16_pitch;
  auto split = [&](uint32_t e, float4 v) {
    __half hi[4], lo[4];
    split_f16(v.x * s, hi[0], lo[0]); split_f16(v.y * s, hi[1], lo[1]); split_f16(v.z * s, hi[2], lo[2]); split_f16(v.w * s, hi[3], lo[3]);
    *reinterpret_cast<uint2*>(dh + e) = *reinterpret_cast<const uint2*>(hi);
    *reinterpret_cast<uint2*>(dl + e) = *reinterpret_cast<const uint2*>(lo);
  };
#pragma unroll
  for (uint32_t k = 0; k < 8; ++k) if (4 * lane + 128 * k < n) split(4 * lane + 128 * k, keep[k]);
  for (uint32_t e = 1024 + 4 * lane; e < n; e += 128) split(e, value(e));
}

// gates = Wx x + b over all columns: from the accumulator's input planes, or from x itself without one (no mask then)
int layer_inputs(dyb200_ctx* ctx, dyb200_wgrad* deferred, const float* Wx, const float* x, const float* b, uint32_t I, uint32_t H, uint32_t columns,
                 float* gates) {
  if (deferred) return dyb200i_rec_inputs(ctx, deferred, Wx, b, I, H, columns, gates);
  { int rc0__ = dyb200_scratch_begin(ctx); if (rc0__) return rc0__; }
  GemmPair p{Wx, 4 * H, 0, x, I, 0, I, nullptr, 0, 0, 1};
  GemmEpilogue e{EPI_BIAS, gates, 4 * H, b, 0, 0.f, nullptr, 0, 0};
  return dyb200_gemm_fused(ctx, 4 * H, columns, 1, &p, e);
}

}  // namespace

// Layers of more than 384 units (narrower ones: lstm_rec.cu and the TF32 form) and batches of more than eight columns (fewer: lstm_wide.cu) whose tiles are
// all resident (one CTA per SM: 225 KB of shared memory).  64-column tiles where there are SMs for them (us per step, I = H = 1024, TF32 / this form
// with 128 / with 64 columns: batch 128 16.5 / 14.3 / 10.5, 256 23.3 / 17.4 / 14.8; batch 512 has 128 columns only, 40.8 / 25.4; batch 64 11.1 / - / 8.4),
// then as many K splits as there are SMs for, four k-blocks each on average and more (Wx and Wh are cut separately, so the last share may be short or
// empty: 9 + 9 k-blocks make 6, 6, 6, 0, the longest still shorter than the 10 of two splits).  They are clusters whatever dyb200_ctx_cluster_splitk
// says: there is no other form, and another number of splits would give other bits.  Columns and units past the end of a tile are computed and
// dropped: a launch and more per step, which such layers took before, was 19 us at (512, 1024, 100 columns), 25 at (300, 600, 30), 24 at (512, 768, 300),
// 31 at (512, 1000, 100) and 18 at (256, 1024, 16); here it is 8.9, 7.1, 10.8, 8.9 and 7.1.  Units that do not come in fours have instantiations that
// read and write a value at a time: 28 -> 10.1 at (512, 777, 100), 26 -> 8.0 at (300, 601, 30).  At the rule's edges, the forms before / here: (64, 385, 9) 12.0 / 8.8,
// (512, 385, 40) 21.7 / 8.4, (512, 416, 64) 15.4 / 7.5 and (512, 448, 512) 15.3 / 10.0 (TF32 pairs in whole tiles there), (512, 2048, 256) 45.4 / 44.1,
// (512, 4096, 64) 67.3 / 64.9, (64, 4736, 128) 91.1 / 90.3, (512, 1023, 500) 58.7 / 25.7; two steps with the weights' pairs made for them: (512, 512, 64) 28.0 / 21.7,
// (512, 385, 40) 38.5 / 27.6, (64, 400, 9) 20.9 / 18.4.
// Error of whole sequences against float64 (2-norm, forms before / here): gates 0.13 - 0.97 of what it was at 32 - 1024 inputs, 385 - 1024 units, 9 - 512 columns; with 1 - 16
// inputs and at most 32 columns, all plain fp32 before, 1.00 - 1.03 (6.8e-8).
bool dyb200_seq_f16_plan(dyb200_ctx* ctx, uint32_t I, uint32_t H, uint32_t B, uint32_t* bn, uint32_t* S) {
  if (H <= 384 || I == 0 || B <= 8) return false;
  const uint32_t sms = (uint32_t)ctx->sm_count, tiles_m = (H + 31) / 32, kb = (I + 63) / 64 + (H + 63) / 64;
  *bn = tiles_m * ((B + 63) / 64) <= sms ? 64 : 128;
  const uint32_t tiles_n = (B + *bn - 1) / *bn, tiles = tiles_m * tiles_n;
  if (tiles_n > 32) return false;   // (one hand-over counter per column block)
  for (uint32_t s = *bn == 64 ? 8 : 4; s >= 1; s /= 2) {
    if (tiles * s > sms || (s > 1 && kb / s < 4)) continue;
    if (seq_f16_dispatch(SEQ_SET_SMEM, H % 4 == 0, *bn, s, ctx) != DYB200_OK) return false;
    if (s > 1) {
      const int fit = seq_f16_dispatch(SEQ_FIT, H % 4 == 0, *bn, s, ctx);
      if (fit <= 0 || tiles > (uint32_t)fit) continue;
    }
    *S = s;
    return true;
  }
  return false;
}

int dyb200_seq_f16(dyb200_ctx* ctx, const SeqF16Call& q) {
  const uint32_t I = q.I, H = q.H, B = q.B, T = q.T, G = 4 * H, tiles_m = (H + 31) / 32, rows = tiles_m * BM;
  uint32_t bn, S;
  DYB_CHECK_ARG(ctx, dyb200_seq_f16_plan(ctx, I, H, B, &bn, &S), "lstm_seq_fwd: shape %u, %u x %u", I, H, B);
  F16Gates W;
  int rc;
  if ((rc = dyb200_f16_gates(ctx, q.Wx, q.Wh, I, H, &W))) return rc;
  const uint32_t xp = (I + 63) / 64 * 64, hp = (H + 63) / 64 * 64, slots = T > 1 ? 2 : 1;
  const size_t xn = (size_t)T * B * xp, hn = (size_t)slots * B * hp;
  void *p16, *words;
  if ((rc = dyb200_scratch(ctx, 2 * (xn + hn) * sizeof(__half), &p16)) || (rc = dyb200_scratch(ctx, ((size_t)T * B + 2 * (size_t)B) * sizeof(uint32_t), &words))) return rc;
  SeqPrep p;
  memset(&p, 0, sizeof(p));
  p.x_hi = q.X.hi; p.x_lo = q.X.lo; p.x_ld = q.X.pitch; p.I = I; p.x_lines = T * B;
  p.x16_hi = (__half*)p16; p.x16_lo = p.x16_hi + xn; p.x16_pitch = xp; p.x_scale = (uint32_t*)words;
  p.h0 = q.h0; p.mask = q.mh; p.H = H; p.B = B; p.mask_full = q.mh_full; p.h0_done = q.h0_done; p.hn_hi = q.Hs.hi; p.hn_lo = q.Hs.lo; p.hn_pitch = q.Hs.pitch;
  p.h16_hi = p.x16_lo + xn; p.h16_lo = p.h16_hi + hn; p.h16_pitch = hp; p.h0_scale = p.x_scale + (size_t)T * B;
  p.mask_lines = q.mh ? (q.mh_full ? B : 1) : 0; p.h_scale = p.h0_scale + B;
  dyb_launch(k_seq_prep, (unsigned)(((size_t)T * B + B + p.mask_lines + 7) / 8), 256, 0, ctx, p);
  DYB_LAUNCHED(ctx);
  TmapPack tm;
  memset(&tm, 0, sizeof(tm));
  struct { __half* plane; uint32_t n, K, pitch, box; bool mn; } maps[8] = {
      {W.x_hi, rows, I, rows, BM, true}, {W.x_lo, rows, I, rows, BM, true}, {p.x16_hi, T * B, I, xp, bn, false}, {p.x16_lo, T * B, I, xp, bn, false},
      {W.h_hi, rows, H, rows, BM, true}, {W.h_lo, rows, H, rows, BM, true}, {p.h16_hi, slots * B, H, hp, bn, false}, {p.h16_lo, slots * B, H, hp, bn, false}};
  for (int k = 0; k < 8; ++k)
    if ((rc = dyb200_tc_make_tmap_f16(ctx, &tm.t[k], maps[k].plane, maps[k].n, maps[k].K, maps[k].pitch, maps[k].box, maps[k].mn))) return rc;
  SeqFwd a;
  memset(&a, 0, sizeof(a));
  a.T = T; a.B = B; a.H = H; a.kb0 = xp / 64; a.kb1 = hp / 64;
  a.gates = q.gates; a.cs = q.c; a.hs = q.h; a.c0 = q.c0; a.bias = q.b; a.forget_bias = q.forget_bias;
  a.hn_hi = q.Hs.hi; a.hn_lo = q.Hs.lo; a.hn_pitch = q.Hs.pitch;
  a.hmask = q.mh; a.hmask_ld = H; a.hmask_full = q.mh_full; a.emit_last = q.emit_last;
  a.gate_scale = W.scale; a.x_scale = p.x_scale; a.h0_scale = p.h0_scale; a.h_scale = q.mh ? p.h_scale : nullptr; a.h_scale_full = q.mh_full;
  a.h16_hi = p.h16_hi; a.h16_lo = p.h16_lo; a.h16_pitch = hp;
  a.ready = ctx->dev_flags + DYB200_DEV_SEQ0;
  a.flags = ctx->dev_flags;
  if (T > 1) DYB_CUDA(ctx, cudaMemsetAsync(a.ready, 0, 32 * sizeof(uint32_t), ctx->stream));   // (a single step's CTAs count, but nobody waits)
  return seq_f16_dispatch(SEQ_LAUNCH, H % 4 == 0, bn, S, ctx, &tm, &a, dim3(tiles_m, (B + bn - 1) / bn, S), 2.0 * G * (double)B * (I + H) * T, I + H);
}

extern "C" {

// Whether the forward products of such a layer run on fp16 pairs (1 or 0), and their column tile and K splits.
int dyb200i_seq_f16_tiling(dyb200_ctx* ctx, uint32_t I, uint32_t H, uint32_t B, uint32_t* tile, uint32_t* splits) {
  return dyb200_seq_f16_plan(ctx, I, H, B, tile, splits) ? 1 : 0;
}

int dyb200_vanilla_lstm_seq_fwd(const dyb200_tensor* x_all, const dyb200_tensor* h0, const dyb200_tensor* c0,
                                const dyb200_tensor* Wx, const dyb200_tensor* Wh, const dyb200_tensor* b,
                                const dyb200_tensor* mask_x, const dyb200_tensor* mask_h, const dyb200_lstm_gates_attrs* attrs,
                                dyb200_tensor* gates_all, dyb200_tensor* c_all, dyb200_tensor* h_all, dyb200_wgrad* deferred,
                                uint32_t steps, dyb200_ctx* ctx) {
  DYB_CHECK_ARG(ctx, x_all && h0 && c0 && Wx && Wh && b && attrs && gates_all && c_all && h_all && steps > 0, "lstm_seq_fwd: null argument");
  DYB_CHECK_ARG(ctx, (attrs->dropout != 0) == (mask_x != nullptr && mask_h != nullptr), "lstm_seq_fwd: masks must be given exactly when dropout is set");
  DYB_CHECK_ARG(ctx, x_all->nd == 1 && x_all->bd % steps == 0, "lstm_seq_fwd: x_all must be Dim({I}, steps * batch)");
  const uint32_t T = steps, B = x_all->bd / T, I = t_dim(x_all, 0), H = t_dim(h0, 0), G = 4 * H;
  const size_t HB = (size_t)H * B;
  DYB_CHECK_ARG(ctx, h0->nd == 1 && h0->bd == B && c0->bd == B && t_dim(c0, 0) == H, "lstm_seq_fwd: h0 / c0 must be Dim({H}, batch)");
  DYB_CHECK_ARG(ctx, t_size(gates_all) == 4 * HB * T && t_size(c_all) == HB * T && t_size(h_all) == HB * T, "lstm_seq_fwd: outputs must hold all %u steps", T);
  if (HB == 0) return DYB200_OK;
  int rc;
  if (deferred && (rc = dyb200_wgrad_pack_inputs(deferred, x_all, mask_x, B, ctx))) return rc;
  const float* mx = attrs->dropout ? mask_x->v : nullptr;
  const float* mh = attrs->dropout ? mask_h->v : nullptr;
  const int mh_full = mh ? mask_h->bd == B : 0;
  (void)mx;

  // ---- one kernel for the whole sequence, when its CTAs can all be resident ----
  // (It comes first because it gives the per-step calls' values bit for bit.  It is not the fastest form for narrow layers in whole tiles:
  // forward and backward over 35 steps, I = H, this kernel at 64 / 128 / 256 columns against the clusters of lstm_rec.cu at 66 / 132 / 260:
  // 128 units 732 / 1113 / 1564 against 184 / 214 / 306 us, 256 units 772 / 1115 / 1480 against 314 / 341 / 398, 384 units
  // 763 / 1228 / 2070 against 535 / 930 / 1738.)
  const uint32_t bn = dyb200_tc_tile_cols(B);
  const uint32_t kb0 = (I + 31) / 32, kb1 = (H + 31) / 32, kb_total = kb0 + kb1;
  const bool sequence = ctx->seq_kernels && T >= 2 && attrs->weightnoise_std == 0.f && Wx->nd == 2 && Wx->d[0] == G && Wx->d[1] == I && Wh->nd == 2 &&
                    Wh->d[0] == G && Wh->d[1] == H && t_size(b) == G &&
                    (H % 4 != 0 || (aligned16(gates_all->v) && aligned16(b->v) && aligned16(c0->v) && aligned16(c_all->v) && aligned16(h_all->v) && (!mh || aligned16(mh)))) &&
                    (!attrs->dropout || ((mask_h->bd == B || mask_h->bd == 1) && t_dim(mask_h, 0) == H));
  const bool resident = sequence && deferred && H % 32 == 0 && I % 4 == 0 && dyb200_tc_eligible(G, B, 2.0 * G * B * (I + H));
  uint32_t S = 1, f16_bn;
  bool wide_fits = true;
  SeqPlanes pl;
  // (wide layers.  Without an accumulator the inputs are x itself, and a sequence has to be worth making the weights' pairs for.  A short sequence of few
  // columns keeps the step calls' own sums, plain fp32 there: gemm_thin.cu)
  const bool short_thin = T < kRecMinSteps && dyb200_thin_columns(G, B, I + H);
  if (sequence && !short_thin && (deferred || (!attrs->dropout && T >= kRecMinSteps && I % 4 == 0)) && dyb200_seq_f16_plan(ctx, I, H, B, &f16_bn, &S) &&
      (!deferred || dyb200_wgrad_seq_planes(deferred, T, B, &pl))) {
    { int rc0__ = dyb200_scratch_begin(ctx); if (rc0__) return rc0__; }
    if (deferred) DYB_CHECK_ARG(ctx, dyb200_wgrad_rows(deferred) == G, "lstm_seq_fwd: the deferred accumulator has %u rows, the layer %u", dyb200_wgrad_rows(deferred), G);
    else { pl.X.hi = x_all->v; pl.X.lo = nullptr; pl.X.pitch = I; pl.Hs.hi = pl.Hs.lo = nullptr; pl.Hs.pitch = 0; }
    SeqF16Call q{I, H, B, T, Wx->v, Wh->v, b->v, h0->v, c0->v, mh, mh_full, attrs->forget_gate_bias, gates_all->v, c_all->v, h_all->v, pl.X, pl.Hs, 0, 0};
    rc = dyb200_seq_f16(ctx, q);
    if (rc != DYB200_ENOMEM) {
      if (!rc && deferred) dyb200_wgrad_seq_done(deferred);
      return rc;
    }
    wide_fits = false;   // (no room for the pairs of all steps: the single-step calls, with those of one)
  }
  bool persistent = resident && wide_fits && B % bn == 0;
  if (persistent) {
    S = dyb200_tc_splits(ctx, G, B, kb_total);
    const uint32_t per = (kb_total + S - 1) / S;
    S = (kb_total + per - 1) / per;
    const uint32_t tiles = (G / BM) * (B / bn);
    if (S > 8 || (S & (S - 1)) != 0 || (S > 1 && !ctx->cluster_splitk)) persistent = false;   // (the column exchange wants a power of two)
    else {
      if ((rc = seq_fwd_dispatch<false>(SEQ_SET_SMEM, bn, S, ctx))) return rc;
      if (S > 1) {
        const int fit = seq_fwd_dispatch<false>(SEQ_FIT, bn, S, ctx);
        persistent = fit > 0 && tiles <= (uint32_t)fit;
      } else {
        persistent = tiles <= (uint32_t)ctx->sm_count;   // one CTA per SM (225 KB of shared memory each)
      }
    }
    if (B / bn > 32) persistent = false;                // one hand-over counter per column block
    if (persistent) persistent = dyb200_wgrad_seq_planes(deferred, T, B, &pl);
  }
  if (persistent) {
    { int rc0__ = dyb200_scratch_begin(ctx); if (rc0__) return rc0__; }
    DYB_CHECK_ARG(ctx, dyb200_wgrad_rows(deferred) == G, "lstm_seq_fwd: the deferred accumulator has %u rows, the layer %u", dyb200_wgrad_rows(deferred), G);
    PackedOp A[2];
    if ((rc = dyb200_tc_param_gates(ctx, Wx->v, G, G, I, &A[0]))) return rc;
    if ((rc = dyb200_tc_param_gates(ctx, Wh->v, G, G, H, &A[1]))) return rc;
    PackJobs batch;
    dyb200_tc_pack_begin(&batch);
    if ((rc = dyb200_wgrad_seq_h0(deferred, h0->v, mh, mh_full, ctx, &batch))) return rc;
    if ((rc = dyb200_tc_pack_flush(ctx, &batch))) return rc;
    TmapPack tm;
    memset(&tm, 0, sizeof(tm));
    if ((rc = dyb200_tc_make_tmap(ctx, &tm.t[0], A[0].hi, G, I, A[0].pitch, BM))) return rc;
    if ((rc = dyb200_tc_make_tmap(ctx, &tm.t[1], A[0].lo, G, I, A[0].pitch, BM))) return rc;
    if ((rc = dyb200_tc_make_tmap(ctx, &tm.t[2], pl.X.hi, T * B, I, pl.X.pitch, bn))) return rc;
    if ((rc = dyb200_tc_make_tmap(ctx, &tm.t[3], pl.X.lo, T * B, I, pl.X.pitch, bn))) return rc;
    if ((rc = dyb200_tc_make_tmap(ctx, &tm.t[4], A[1].hi, G, H, A[1].pitch, BM))) return rc;
    if ((rc = dyb200_tc_make_tmap(ctx, &tm.t[5], A[1].lo, G, H, A[1].pitch, BM))) return rc;
    if ((rc = dyb200_tc_make_tmap(ctx, &tm.t[6], pl.Hs.hi, T * B, H, pl.Hs.pitch, bn))) return rc;
    if ((rc = dyb200_tc_make_tmap(ctx, &tm.t[7], pl.Hs.lo, T * B, H, pl.Hs.pitch, bn))) return rc;
    SeqFwd a;
    memset(&a, 0, sizeof(a));
    a.T = T; a.B = B; a.H = H; a.kb0 = kb0; a.kb1 = kb1;
    a.gates = gates_all->v; a.cs = c_all->v; a.hs = h_all->v; a.c0 = c0->v; a.bias = b->v; a.forget_bias = attrs->forget_gate_bias;
    a.hn_hi = pl.Hs.hi; a.hn_lo = pl.Hs.lo; a.hn_pitch = pl.Hs.pitch;
    a.hmask = mh; a.hmask_ld = H; a.hmask_full = mh_full;
    a.ready = ctx->dev_flags + DYB200_DEV_SEQ0;
    a.flags = ctx->dev_flags;
    DYB_CUDA(ctx, cudaMemsetAsync(a.ready, 0, 32 * sizeof(uint32_t), ctx->stream));
    const dim3 grid(G / BM, B / bn, S);
    const double flops = 2.0 * G * (double)B * (I + H) * T;
    rc = seq_fwd_dispatch<false>(SEQ_LAUNCH, bn, S, ctx, &tm, &a, grid, flops, I + H);
    if (rc) return rc;
    dyb200_wgrad_seq_done(deferred);
    return DYB200_OK;
  }

  // ---- layers of moderate width: the input products of all steps as one GEMM, then the recurrence in clusters (lstm_rec.cu) ----
  if (!persistent && attrs->weightnoise_std == 0.f && I > 0 && Wx->nd == 2 && Wx->d[0] == G && Wx->d[1] == I && Wh->nd == 2 && Wh->d[0] == G &&
      Wh->d[1] == H && t_size(b) == G && (deferred || !attrs->dropout) &&
      (!attrs->dropout || ((mask_h->bd == B || mask_h->bd == 1) && t_dim(mask_h, 0) == H)) && dyb200i_rec_takes(ctx, H, T, B, 1)) {
    if ((rc = layer_inputs(ctx, deferred, Wx->v, x_all->v, b->v, I, H, T * B, gates_all->v))) return rc;
    dyb200i_rec_dir d;
    memset(&d, 0, sizeof(d));
    d.Wh = Wh->v; d.h0 = h0->v; d.c0 = c0->v; d.mask_h = mh; d.gates = gates_all->v; d.c = c_all->v; d.h = h_all->v; d.w = deferred;
    return dyb200i_rec_fwd(ctx, 1, &d, H, T, B, nullptr, mh_full, attrs->forget_gate_bias);
  }

  // ---- few columns: the input products of all steps as one GEMM, then one pass over Wh per step (gemm_thin.cu) ----
  // (from as many steps up as the recurrence kernels; a shorter sequence keeps the per-step calls' own sums)
  if (!persistent && ctx->seq_kernels && T >= kRecMinSteps && attrs->weightnoise_std == 0.f && I > 0 && dyb200_thin_columns(G, B, H) && Wx->nd == 2 && Wx->d[0] == G &&
      Wx->d[1] == I && Wh->nd == 2 && Wh->d[0] == G && Wh->d[1] == H && t_size(b) == G && (deferred || !attrs->dropout) &&
      (!attrs->dropout || ((mask_h->bd == B || mask_h->bd == 1) && t_dim(mask_h, 0) == H))) {
    { int rc0__ = dyb200_scratch_begin(ctx); if (rc0__) return rc0__; }
    if ((rc = layer_inputs(ctx, deferred, Wx->v, x_all->v, b->v, I, H, T * B, gates_all->v))) return rc;
    if (deferred) {
      PackJobs batch;
      dyb200_tc_pack_begin(&batch);
      if ((rc = dyb200_wgrad_seq_h0(deferred, h0->v, mh, mh_full, ctx, &batch))) return rc;
      if ((rc = dyb200_tc_pack_flush(ctx, &batch))) return rc;
    }
    // (h0 on the first step's outputs is read from a copy: a step's launch reads h_{t-1} while it stores its own)
    const float* h_first = h0->v;
    if (t_overlap(h0->v, HB, h_all->v, HB) || t_overlap(h0->v, HB, c_all->v, HB)) {
      void* copy;
      if ((rc = dyb200_scratch(ctx, HB * sizeof(float), &copy))) return rc;
      DYB_CUDA(ctx, cudaMemcpyAsync(copy, h0->v, HB * sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
      h_first = (const float*)copy;
    }
    if (dyb200_wide_takes(ctx, H, B)) {   // all steps in one launch, Wh in the registers of the whole GPU (lstm_wide.cu)
      WideFwd a;
      memset(&a, 0, sizeof(a));
      a.Wh = Wh->v; a.gates = gates_all->v; a.c = c_all->v; a.h = h_all->v; a.h0 = h_first; a.c0 = c0->v; a.mask = mh; a.mask_full = mh_full;
      a.H = H; a.B = B; a.T = T; a.fb = attrs->forget_gate_bias;
      if (deferred) {
        PackedOp X, Hs;
        DYB_CHECK_ARG(ctx, dyb200_wgrad_column_planes(deferred, T * B, nullptr, &X, &Hs) && Hs.K == H, "lstm sequence: the accumulator does not hold the inputs of this layer");
        a.hn_hi = Hs.hi; a.hn_lo = Hs.lo; a.hn_pitch = Hs.pitch;
      }
      bool launched;
      if ((rc = dyb200_wide_fwd(ctx, a, &launched))) return rc;
      if (launched) {
        if (deferred) dyb200_wgrad_seq_done(deferred);
        return DYB200_OK;
      }
    }
    for (uint32_t t = 0; t < T; ++t) {
      GemmPair p{Wh->v, G, 0, t ? h_all->v + (size_t)(t - 1) * HB : h_first, H, 0, H, mh, H, mh_full, 1};
      GemmEpilogue e{EPI_LSTM_CELL, gates_all->v + (size_t)t * 4 * HB, G, nullptr, H, attrs->forget_gate_bias, nullptr, 0, 0};
      e.c_prev = t ? c_all->v + (size_t)(t - 1) * HB : c0->v;
      e.c_out = c_all->v + (size_t)t * HB; e.h_out = h_all->v + (size_t)t * HB;
      if (deferred && dyb200_wgrad_next_h(deferred, t * B, B, &e)) { e.hmask = mh; e.hmask_ld = H; e.hmask_full = mh_full; }
      if ((rc = dyb200_lstm_thin(ctx, H, B, 1, &p, 1, e))) return rc;
    }
    if (deferred) dyb200_wgrad_seq_done(deferred);
    return DYB200_OK;
  }

  // ---- the same sequence as one call per time step ----
  for (uint32_t t = 0; t < T; ++t) {
    dyb200_tensor x = *x_all, hp = *h0, cp = *c0, g = *gates_all, c = *c_all, h = *h_all;
    x.bd = B; x.v = x_all->v + (size_t)t * I * B;
    g.bd = B; g.v = gates_all->v + (size_t)t * 4 * HB;
    c.bd = B; c.v = c_all->v + (size_t)t * HB;
    h.bd = B; h.v = h_all->v + (size_t)t * HB;
    if (t > 0) { hp.v = h_all->v + (size_t)(t - 1) * HB; cp.v = c_all->v + (size_t)(t - 1) * HB; }
    if ((rc = dyb200_vanilla_lstm_fwd_fused_at(&x, &hp, &cp, Wx, Wh, b, mask_x, mask_h, attrs, &g, &c, &h, deferred, t * B, ctx))) return rc;
  }
  return DYB200_OK;
}

}  // extern "C"
