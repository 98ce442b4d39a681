// The recurrence of lstm_rec.cu for batches of more columns, on the tensor pipe: layers of at most 256 units, one launch per pass.
//
// What bounds it.  With more than four columns per cluster the fp32 multiply-adds of lstm_rec.cu bound its steps (0.2 us per column
// and step at 256 units: 8 us forward at 37 columns).  A step here is the same hand-over between CTAs around a product of 128 x
// 2 NC x K on tcgen05: the operands are 2 x 11 bit fp16 pairs (gemm.cuh), of which a CTA's share of Wh is 128 KB, so that it stays in
// half of the TMEM for the whole sequence and leaves shared memory to the columns; TF32 pairs of the same precision would need all of
// it.  A step is a chain of product, cell pass and one trip through the cluster.
//
// Columns: a cluster takes kGroups groups of 16 neighbours.  More clusters than fit run one after the other (no cluster waits for another):
// ragged batches come longest first, so every group ends with its own longest sentence.
//
// Cells: a warp's lanes are the CTA's 32 units of one column, so that every access to gates, states and operand planes is a full
// 128-byte line (8 units x 4 columns per access took four requests each: 3400 of a step's 9000 cycles went into the stores alone).
// Sixteen cell warps: with eight, a step waited on its own latencies (15000 cycles backward instead of 9000).
//
// Forward: CTA r owns 32 hidden units, 128 gate rows (row 32 q + unit); D (gate row x column) = Wh_r h, accumulators in TMEM.  The four
// warps that read the four gates of a group of columns exchange them through shared memory.  h_t goes to every CTA of the cluster as
// fp16 pairs in the layout of the MMA's right operand, one bulk copy per CTA (messages of 16 bytes, st.async, moved 10 bytes per cycle:
// 5000 cycles for 48 columns).  |h| < 1 and the largest dropout factor give one scale for the whole launch; an initial state has its own.
// (Elements of h down to 2^-28 keep all their bits; smaller ones an absolute error below 2^-50, which is what rounding adds to any
// pre-activation from 2^-26 up.)
// Backward: D (unit of h_{t-1} x column) = Wh_r^T dgates_r over the CTA's own 128 gate rows, partial sums to the unit's owner.  dgates
// have no bound known in advance: a column's scale is the largest value of its 128 rows, found in the cell pass.
#include "lstm_rec.cuh"

#include "gemm.cuh"
#include "lstm_cell.cuh"
#include "lstm_rec_dev.cuh"
#include "tc_dev.cuh"

namespace {

// Two groups of columns per CTA, each with its own loop, barriers and buffers (only Wh is shared): one's cell pass runs beside the other's
// product and messages (one group of 32 or 64 columns: 302 and 450 us where two of 16 take 247 and 278, 256 sentences of up to 100
// words; two of 32 spill registers, three of 16 too).  Warps 0 and 1 issue the groups' products and copies (the oldest warps of their
// schedulers go first), 2 .. 9 and 10 .. 17 are the groups' cell warps.
constexpr uint32_t kGroups = 2, kGroupWarps = 8, kGroupThreads = 32 * kGroupWarps;
constexpr uint32_t kCellThreads = kGroups * kGroupThreads, kTcThreads = kCellThreads + 32 * kGroups;
constexpr uint32_t kTcUnits = 32;      // hidden units per CTA
constexpr uint32_t kTcCols = 16;       // columns per group

// Positions of a column's K-major operand row: byte offset of element k (even or odd) of row r in a plane block of `rows` rows per 64 k.
__device__ __forceinline__ uint32_t op_off(uint32_t rows, uint32_t r, uint32_t k) {
  return (k >> 6) * rows * 128 + r * 128 + ((((k & 63) >> 3) ^ (r & 7)) << 4) + (k & 7) * 2;
}
// The same in the layout of h: blocks of 32 k (one CTA's units), rows of 64 bytes in the 64-byte swizzle, so that what a CTA contributes
// lies in one piece.
__device__ __forceinline__ uint32_t h_off(uint32_t rows, uint32_t r, uint32_t k) {
  return (k >> 5) * rows * 64 + r * 64 + ((((k & 31) >> 3) ^ ((r >> 1) & 3)) << 4) + (k & 7) * 2;
}
__device__ __forceinline__ uint64_t umma_desc64(uint32_t smem_addr) {   // K-major, 64-byte swizzle, 8-row groups 512 bytes apart
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;
  return d;
}
// shared memory of this CTA -> of a CTA of the cluster, counted by that CTA's mbarrier
__device__ __forceinline__ void send_bulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(smem_u32(src)),
               "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// two values as fp16 pairs, the words of either plane
__device__ __forceinline__ void pack_pair2(float a, float b, float scale, uint32_t& hi, uint32_t& lo) {
  __half ah, al, bh, bl;
  split_f16(a * scale, ah, al);
  split_f16(b * scale, bh, bl);
  hi = (uint32_t)__half_as_ushort(ah) | (uint32_t)__half_as_ushort(bh) << 16;
  lo = (uint32_t)__half_as_ushort(al) | (uint32_t)__half_as_ushort(bl) << 16;
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// four bytes of global memory into this thread's place in shared memory, beside everything else it does
__device__ __forceinline__ void copy4(uint32_t dst, const float* src) { asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory"); }
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// p + col * bytes: one multiply-add of 32 x 32 + 64 bits (indexing by floats adds a shift of 64 bits to every address; addresses were a
// third of the cell passes' instructions)
__device__ __forceinline__ float* at(float* p, uint32_t col, uint32_t bytes) { return reinterpret_cast<float*>(reinterpret_cast<char*>(p) + (uint64_t)col * bytes); }
__device__ __forceinline__ const float* at(const float* p, uint32_t col, uint32_t bytes) {
  return reinterpret_cast<const float*>(reinterpret_cast<const char*>(p) + (uint64_t)col * bytes);
}
// columns of the block from `base` on that are active at a step of width B
__device__ __forceinline__ uint32_t tc_active(uint32_t B, uint32_t base, uint32_t ncap) { return B > base ? min(B - base, ncap) : 0; }
__device__ __forceinline__ uint32_t tmem_cols(uint32_t need) { return need <= 64 ? 64 : need <= 128 ? 128 : need <= 256 ? 256 : 512; }

// One k step of 16: A_hi x [B_hi | B_lo] -> wide (2 NC columns), A_lo x B_hi -> narrow.  A in TMEM: lane = row, a column holds two k.
template <int NC>
__device__ __forceinline__ void tc_kstep(uint32_t wide, uint32_t narrow, uint32_t a_hi, uint32_t a_lo, uint64_t b, uint32_t add_wide, uint32_t add_narrow) {
  constexpr uint32_t base = (1u << 4) | ((uint32_t)(BM >> 4) << 24);   // fp32 accumulator, fp16 operands, both K-major
  asm volatile(
      "{\n\t.reg .pred pw, pn;\n\t"
      "setp.ne.b32 pw, %7, 0;\n\tsetp.ne.b32 pn, %8, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%2], %4, %5, pw;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [%3], %4, %6, pn;\n\t}"
      ::"r"(wide), "r"(narrow), "r"(a_hi), "r"(a_lo), "l"(b), "r"(base | ((uint32_t)(2 * NC >> 3) << 17)), "r"(base | ((uint32_t)(NC >> 3) << 17)),
        "r"(add_wide), "r"(add_narrow)
      : "memory");
}

// grid (C, clusters x directions), cluster (C, 1, 1).  Dynamic shared memory (1024-byte aligned), for each group:
// h [2][2 KB blocks of 32 units][NC hi rows, NC lo rows][64 bytes], then gates on their way [NC][4][32], then Wx x + b [2][2 cells x 4 gates][threads];
// KB = ceil(H / 64).
// TMEM: each group's accumulators (3 NC columns: A_hi B_hi, A_hi B_lo, A_lo B_hi - the last apart, so that the chain of one waits on
// the other's MMAs, not on its own), Wh_hi and Wh_lo (32 KB columns each).
template <uint32_t kH, bool kCopies = true>
__global__ void __launch_bounds__(kTcThreads, 1) k_rec_tc_fwd(const __grid_constant__ RecFwd a) {
  constexpr uint32_t NC = kTcCols, kBlock = 2 * NC * 64;   // bytes of a CTA's part of h
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t got_[kGroups][2], acc_full_[kGroups], h_ready_[kGroups];
  __shared__ uint32_t tmem_slot, hword_[kGroups][2], wmax[128];
  const uint32_t ndir = a.ndir, dir = blockIdx.y % ndir;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t grp = warp < kGroups ? warp : (warp - kGroups) / kGroupWarps, gw = (warp - kGroups) % kGroupWarps;   // (gw: cell warps)
  const RecDirF d = dir ? a.d[1] : a.d[0];
  const uint32_t H = kH ? kH : a.H, rank = blockIdx.x, C = kH ? kH / kTcUnits : gridDim.x, KB = (H + 63) / 64;
  const uint32_t base = (blockIdx.y / ndir * kGroups + grp) * NC;
  const uint32_t hbytes = 2 * KB * kBlock;
  unsigned char* hall = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* hbuf = hall + grp * 2 * hbytes;
  float* exch = reinterpret_cast<float*>(hall + kGroups * 2 * hbytes) + grp * NC * 128;
  float* ahead = reinterpret_cast<float*>(hall + kGroups * 2 * hbytes) + (kGroups + 2 * grp) * NC * 128;
  uint64_t *got = got_[grp], &acc_full = acc_full_[grp], &h_ready = h_ready_[grp];
  uint32_t* hword = hword_[grp];
  if (tid == 0) {
    for (uint32_t k = 0; k < kGroups; ++k) {
      msg_init(&got_[k][0]);
      msg_init(&got_[k][1]);
      mbar_init(&acc_full_[k], 1);
      mbar_init(&h_ready_[k], kGroupWarps);
      hword_[k][0] = hword_[k][1] = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 128) wmax[tid] = 0;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(tmem_cols(kGroups * 3 * NC + 64 * KB)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  dyb_grid_dep_wait();
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t ncol = tc_active(a.N, base, NC);

  // Wh of this CTA: lane = unit (128 contiguous bytes per load), a warp has 64 k of one gate.  The scale of a row is that of its largest
  // value.
  if (warp >= kGroups) {
    float v[64];
    const uint32_t u = rank * kTcUnits + lane, q = warp & 3, kb = (warp - kGroups) >> 2, row = 32 * q + lane;
    const float* src = d.Wh + (size_t)q * H + u;
    uint32_t m = 0;
#pragma unroll
    for (int x = 0; x < 64; ++x) {
      const uint32_t k = 64 * kb + x;
      v[x] = k < H && u < H ? __ldg(at(src, k, 16 * H)) : 0.f;
    }
#pragma unroll
    for (int x = 0; x < 64; ++x) m = max(m, finite_mag(v[x]));
    atomicMax(&wmax[row], m);
    bar_sync(1, kCellThreads);
    if (kb < KB) {
      const float scale = scale_of(wmax[row]);
      const uint32_t to = tmem + kGroups * 3 * NC + 32 * kb + ((32 * q) << 16);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int y = 0; y < 8; ++y) pack_pair2(v[16 * x + 2 * y], v[16 * x + 2 * y + 1], scale, hi[y], lo[y]);
        tmem_st8(to + 8 * x, hi);
        tmem_st8(to + 32 * KB + 8 * x, lo);
      }
      tmem_st_wait();
    }
    tc_before();
  }
  // scales of h: the largest dropout factor (1 without); of the initial state: its largest value
  for (uint32_t e = tid; e < kGroups * 2 * hbytes / 16; e += kTcThreads) reinterpret_cast<uint4*>(hall)[e] = make_uint4(0, 0, 0, 0);
  const uint32_t gt0 = gw * 32 + lane;   // (cell warps: thread of the group)
  if (warp >= kGroups && (d.mask || d.h0)) {
    uint32_t m0 = 0, m1 = 0;
    for (uint32_t e = gt0; e < ncol * H; e += kGroupThreads) {
      const uint32_t i = e / H, k = e % H, sc = base + i;
      const float m = d.mask ? __ldg(d.mask + k + (a.mask_full ? (size_t)H * sc : 0)) : 1.f;
      m1 = max(m1, finite_mag(m));
      if (d.h0) m0 = max(m0, finite_mag(__ldg(d.h0 + k + (size_t)H * sc) * m));
    }
    atomicMax(&hword[0], m0);
    if (d.mask) atomicMax(&hword[1], m1);
  }
  __syncthreads();
  const uint32_t word0 = hword[0], word1 = d.mask ? hword[1] : 0x3f800000u;
  if (warp >= kGroups) {
    const float s0 = scale_of(word0);
    for (uint32_t e = gt0; e < ncol * H; e += kGroupThreads) {
      const uint32_t i = e / H, k = e % H, sc = base + i;
      float v = 0.f;
      if (d.h0) v = __ldg(d.h0 + k + (size_t)H * sc) * (d.mask ? __ldg(d.mask + k + (a.mask_full ? (size_t)H * sc : 0)) : 1.f);
      __half hi, lo;
      split_f16(v * s0, hi, lo);
      *reinterpret_cast<__half*>(hbuf + h_off(2 * NC, i, k)) = hi;
      *reinterpret_cast<__half*>(hbuf + h_off(2 * NC, NC + i, k)) = lo;
      if (d.hn_hi && k / kTcUnits == rank) {
        float thi, tlo;
        split_tf32(v, thi, tlo);
        d.hn_hi[(size_t)sc * a.hn_pitch + k] = thi;
        d.hn_lo[(size_t)sc * a.hn_pitch + k] = tlo;
      }
    }
  }
  fence_async();
  cluster_arrive();
  cluster_wait();

  // first columns of the steps t, t + 1, t + 2 (the end when there is none), each read a step before it is needed
  auto start_of = [&](uint32_t t) { t = min(t, a.T); return a.prefix ? a.prefix[t] : t * a.N; };
  uint32_t col0 = 0, col1 = start_of(1), col2 = start_of(2), n = tc_active(col1, base, NC);
  bool ok = true;
  if (warp < kGroups) {
    uint32_t phase[2] = {0, 0};
    const uint32_t whi = tmem + kGroups * 3 * NC, wlo = whi + 32 * KB, acc = tmem + grp * 3 * NC;
    for (uint32_t t = 0; t < a.T && n > 0; ++t) {
      const uint32_t pt = t & 1, pn = pt ^ 1, col3 = start_of(t + 3), n1 = tc_active(col2 - col1, base, NC);
      unsigned char* h = hbuf + pt * hbytes;
      if (n1 && lane == 0) msg_expect(&got[pn], (C - 1) * kBlock);
      if (t > 0) {
        // this CTA's units of h_{t-1} are complete (and the accumulators of that step read): on their way, the others' in
        unsigned char* own = h + rank * kBlock;
        const uint32_t dst = map_rank(smem_u32(own), lane < C ? lane : 0), bar = map_rank(smem_u32(&got[pt]), lane < C ? lane : 0);
        ok = ok && mbar_wait(&h_ready, (t - 1) & 1);
        fence_async();
        if (lane < C && lane != rank) send_bulk(dst, own, kBlock, bar);
        ok = ok && msg_wait(&got[pt], phase[pt]);
        phase[pt] ^= 1;
      }
      if (elect_one()) {
        fence_async();
        tc_after();
        const uint32_t hb = smem_u32(h);
        for (uint32_t blk = 0; blk < 2 * KB; ++blk) {
          const uint64_t bd = umma_desc64(hb + blk * kBlock);
          tc_kstep<NC>(acc, acc + 2 * NC, whi + 16 * blk, wlo + 16 * blk, bd, blk, blk);
          tc_kstep<NC>(acc, acc + 2 * NC, whi + 16 * blk + 8, wlo + 16 * blk + 8, bd + 2, 1, 1);
        }
        umma_commit(&acc_full);
      }
      __syncwarp();
      col1 = col2; col2 = col3; n = n1;
    }
  } else {
    // reads gate `quad` of the columns c8 .. c8 + 7, finishes columns c8 + quad + 4 j; lane = unit
    constexpr int kCells = NC / 8;
    const uint32_t quad = warp & 3, c8 = 8 * (gw >> 2), u = rank * kTcUnits + lane, i0 = c8 + quad;
    const bool live_u = u < H;
    const uint32_t uc = min(u, H - 1);                  // (units that are not there read another's values and store nothing)
    const int wf = scale_field(wmax[32 * quad + lane]), t0 = wf + scale_field(word0) - 282, t1 = wf + scale_field(word1) - 282;
    const float hscale = live_u ? scale_of(word1) : 0.f;
    const uint32_t tq = tmem + grp * 3 * NC + ((32 * quad) << 16) + c8;
    const float* mask = d.mask ? d.mask + uc : nullptr;
    float *pg = d.gates + uc, *pc = d.c + uc, *ph = d.h + uc, *phi = d.hn_hi ? d.hn_hi + uc : nullptr, *plo = phi ? d.hn_lo + uc : nullptr;
    float cst[kCells], mk[kCells];
    // Wx x + b of this thread's cells, of this step and of the next, asked for a whole step before its use.  (In registers the wait for it fell wherever the
    // compiler's few scoreboards put it, before the cell pass of the step that asked: 256 units 1187 us forward, 1039 like this; 200 units, 600 sentences 250 against
    // 230; 99 units, 600 sentences 127 against 119.  Fewer than 64 units, whose steps are the shortest, keep the registers, kCopies off: 600 sentences, 8 units 95 against 101, 33
    // 102 against 105, 56 100 against 104; 64 units 102 against 94.  160 steps of 600 columns, inputs out of L2: 8 units 237 against 254, 56 272 against 264.)
    float* const mine = ahead + gt0;
    const uint32_t pitch = kH ? kH : a.hn_pitch;
    uint32_t ho[kCells];                                   // where h of cell j goes in this CTA's block
    float next[kCells][4];   // (without copies)
    auto fetch = [&](uint32_t to, uint32_t c0, uint32_t nact) {
      if (!kCopies) {
#pragma unroll
        for (int j = 0; j < kCells; ++j) {   // (columns and units that are not there: another's)
          const uint32_t i = i0 + 4 * j;
#pragma unroll
          for (int q = 0; q < 4; ++q) next[j][q] = at(pg, c0 + base + (i < nact ? i : 0), 16 * H)[(size_t)q * H];
        }
        return;
      }
      const uint32_t dst = smem_u32(mine) + to * (NC * 128 * 4);
#pragma unroll
      for (int j = 0; j < kCells; ++j)
        if (live_u && i0 + 4 * j < nact) {   // (units that are not there ask for nothing: 29 lanes on one address took 0.9 us a step, 99 units)
#pragma unroll
          for (int q = 0; q < 4; ++q) copy4(dst + (4 * j + q) * (kGroupThreads * 4), at(pg, c0 + base + i0 + 4 * j, 16 * H) + (size_t)q * H);
        }
    };
    if (n) fetch(0, 0, n);          // (a group may have no column at all)
#pragma unroll
    for (int j = 0; j < kCells; ++j) {
      const uint32_t i = i0 + 4 * j, sc = base + i;
      cst[j] = d.c0 && i < ncol ? __ldg(at(d.c0 + uc, sc, 4 * H)) : 0.f;
      mk[j] = mask && i < ncol ? __ldg(at(mask, a.mask_full ? sc : 0, 4 * H)) : 1.f;
      ho[j] = h_off(2 * NC, i, rank * kTcUnits + lane);
    }
    for (uint32_t t = 0; t < a.T && n > 0; ++t) {
      const uint32_t col3 = start_of(t + 3), n1 = tc_active(col2 - col1, base, NC);
      unsigned char* hnext = hbuf + ((t & 1) ^ 1) * hbytes;
      const int ts = t ? t1 : t0, th = ts >> 1;
      const float f0 = __int_as_float((th + 127) << 23), f1 = __int_as_float((ts - th + 127) << 23);
      const float* const pre = mine + (t & 1) * (NC * 128);
      float now[kCells][4];
      if (kCopies) copies_done();
      else
#pragma unroll
        for (int j = 0; j < kCells; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) now[j][q] = next[j][q];
      if (n1) fetch((t & 1) ^ 1, col1, n1);
      ok = ok && mbar_wait(&acc_full, t & 1);
      tc_after();
      {
        float z[8], z2[8], z3[8];
        tmem_ld8(tq, z);
        tmem_ld8(tq + NC, z2);
        tmem_ld8(tq + 2 * NC, z3);
        tmem_ld_wait();
#pragma unroll
        for (int x = 0; x < 8; ++x) exch[((c8 + x) * 4 + quad) * 32 + lane] = (fmaf(z2[x] + z3[x], kLoScale, z[x]) * f0) * f1;
      }
      tc_before();
      bar_sync(2 + 2 * grp + c8 / 8, 128);
      float hv[kCells], hm[kCells], y[kCells][4];
#pragma unroll
      for (int j = 0; j < kCells; ++j) {
        const uint32_t i = i0 + 4 * j;
#pragma unroll
        for (int q = 0; q < 4; ++q) y[j][q] = exch[(i * 4 + q) * 32 + lane];
        if (i >= n) continue;                            // (the same for the whole warp)
        y[j][0] = gate_sigmoid(y[j][0] + (kCopies ? pre[4 * j * kGroupThreads] : now[j][0]));
        y[j][1] = gate_sigmoid(y[j][1] + (kCopies ? pre[(4 * j + 1) * kGroupThreads] : now[j][1]) + a.fb);
        y[j][2] = gate_sigmoid(y[j][2] + (kCopies ? pre[(4 * j + 2) * kGroupThreads] : now[j][2]));
        y[j][3] = gate_tanh(y[j][3] + (kCopies ? pre[(4 * j + 3) * kGroupThreads] : now[j][3]));
        cst[j] = lstm_cell_c(y[j][0], y[j][3], y[j][1], cst[j]);
        hv[j] = lstm_cell_h(y[j][2], cst[j]);
        hm[j] = hv[j] * mk[j];
        __half hi, lo;
        split_f16(live_u ? hm[j] * hscale : 0.f, hi, lo);
        if (i < n1) {
          *reinterpret_cast<__half*>(hnext + ho[j]) = hi;
          *reinterpret_cast<__half*>(hnext + ho[j] + NC * 64) = lo;
        }
      }
      fence_async();
      __syncwarp();
      if (lane == 0) mbar_arrive(&h_ready);
#pragma unroll
      for (int j = 0; j < kCells; ++j) {
        const uint32_t i = i0 + 4 * j, sc = base + i;
        if (!live_u || i >= n) continue;
        float* const og = at(pg, col0 + sc, 16 * H);
#pragma unroll
        for (int q = 0; q < 4; ++q) og[(size_t)q * H] = y[j][q];
        *at(pc, col0 + sc, 4 * H) = cst[j];
        *at(ph, col0 + sc, 4 * H) = hv[j];
        if (phi && i < n1) {
          float hi, lo;
          split_tf32(hm[j], hi, lo);
          *at(phi, col1 + sc, 4 * pitch) = hi;
          *at(plo, col1 + sc, 4 * pitch) = lo;
        }
      }
      col0 = col1; col1 = col2; col2 = col3; n = n1;
    }
  }
  if (!ok) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
  tc_before();
  __syncthreads();
  cluster_arrive();                // nobody leaves while a neighbour may still send to it
  cluster_wait();
  if (warp == 0) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols(kGroups * 3 * NC + 64 * KB)) : "memory");
  }
}

// grid (C, clusters x directions), cluster (C, 1, 1).  Dynamic shared memory (1024-byte aligned), for each group: dgates [2 blocks of 64
// gate rows][NC hi rows, NC lo rows][128 bytes]; the partial sums [2][C ranks][NC columns][32 units].  TMEM: per group and row tile of 128
// units the accumulators (2 NC columns); then Wh^T hi and lo (64 columns each per row tile).  The slots of the sums that have just been
// read hold the outgoing ones: what comes into slot r next, rank r sends after it has what went out of that slot.  Gate row (unit ul,
// gate q) is element 4 ul + q of the reduction.
template <bool DC, uint32_t kH>
__global__ void __launch_bounds__(kTcThreads, 1) k_rec_tc_bwd(const __grid_constant__ RecBwd a) {
  constexpr uint32_t NC = kTcCols, kSlot = NC * kTcUnits;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t got_[kGroups][2], acc_full_[kGroups];
  __shared__ uint32_t tmem_slot, wmax[256];
  __shared__ __align__(16) float colscale_[kGroups][2][NC];
  const uint32_t ndir = a.ndir, dir = blockIdx.y % ndir, g = blockIdx.y / ndir;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t grp = warp < kGroups ? warp : (warp - kGroups) / kGroupWarps, gw = (warp - kGroups) % kGroupWarps;   // (gw: cell warps)
  const RecDirB d = dir ? a.d[1] : a.d[0];
  const uint32_t H = kH ? kH : a.H, rank = blockIdx.x, C = kH ? kH / kTcUnits : gridDim.x, MT = (H + 127) / 128;
  const uint32_t base = (g * kGroups + grp) * NC;
  unsigned char* dgall = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* dgb = dgall + grp * 2 * 2 * NC * 128;
  float* partall = reinterpret_cast<float*>(dgall + kGroups * 2 * 2 * NC * 128);
  float* part = partall + grp * 2 * C * kSlot;
  uint64_t *got = got_[grp], &acc_full = acc_full_[grp];
  float (*colscale)[NC] = colscale_[grp];
  if (tid == 0) {
    for (uint32_t k = 0; k < kGroups; ++k) {
      mbar_init(&got_[k][0], 2);   // (the bytes of the others, and this CTA's own warp)
      mbar_init(&got_[k][1], 2);
      mbar_init(&acc_full_[k], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 256) wmax[tid] = 0;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(tmem_cols(MT * (kGroups * 2 * NC + 128))) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  dyb_grid_dep_wait();
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = tmem_slot;

  // Lane = unit o of h_{t-1} (row o % 128 of its row tile), a warp has its weights in 16 of this CTA's units; scaled by the largest of all
  if (warp >= kGroups) {
    float4 v[4][4];
    const bool quads = (H & 3) == 0 && aligned16(d.Wh);
    const uint32_t q4 = warp & 3, p4 = (warp - kGroups) >> 2, mt = p4 >> 1, kh = p4 & 1, o = 128 * mt + 32 * q4 + lane;
    uint32_t m = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const uint32_t uu = rank * kTcUnits + 16 * kh + 4 * x;
        const float* p = at(d.Wh + (size_t)q * H + uu, o, 16 * H);
        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
        if (o < H && uu < H) {
          if (quads) w = __ldg(reinterpret_cast<const float4*>(p));
          else {
            w.x = __ldg(p);
            if (uu + 1 < H) w.y = __ldg(p + 1);
            if (uu + 2 < H) w.z = __ldg(p + 2);
            if (uu + 3 < H) w.w = __ldg(p + 3);
          }
        }
        v[q][x] = w;
        m = max(m, max(max(finite_mag(w.x), finite_mag(w.y)), max(finite_mag(w.z), finite_mag(w.w))));
      }
    if (mt < 2) atomicMax(&wmax[o], m);
    bar_sync(1, kCellThreads);
    if (mt < MT) {
      const float scale = scale_of(wmax[o]);
      const uint32_t to = tmem + MT * kGroups * 2 * NC + 64 * mt + 32 * kh + ((32 * q4) << 16);
#pragma unroll
      for (int x = 0; x < 4; ++x) {   // (a column holds two gates of a unit)
        uint32_t hi[8], lo[8];
        pack_pair2(v[0][x].x, v[1][x].x, scale, hi[0], lo[0]); pack_pair2(v[2][x].x, v[3][x].x, scale, hi[1], lo[1]);
        pack_pair2(v[0][x].y, v[1][x].y, scale, hi[2], lo[2]); pack_pair2(v[2][x].y, v[3][x].y, scale, hi[3], lo[3]);
        pack_pair2(v[0][x].z, v[1][x].z, scale, hi[4], lo[4]); pack_pair2(v[2][x].z, v[3][x].z, scale, hi[5], lo[5]);
        pack_pair2(v[0][x].w, v[1][x].w, scale, hi[6], lo[6]); pack_pair2(v[2][x].w, v[3][x].w, scale, hi[7], lo[7]);
        tmem_st8(to + 8 * x, hi);
        tmem_st8(to + 64 * MT + 8 * x, lo);
      }
      tmem_st_wait();
    }
    tc_before();
  }
  for (uint32_t e = tid; e < kGroups * 2 * 2 * NC * 128 / 16; e += kTcThreads) reinterpret_cast<uint4*>(dgall)[e] = make_uint4(0, 0, 0, 0);
  fence_async();
  cluster_arrive();
  cluster_wait();

  // the last step that has a column of this block: widths never grow, so the steps before it have one too
  uint32_t T = base < a.N ? a.T : 0;
  while (a.prefix && T > 0 && tc_active(a.prefix[T] - a.prefix[T - 1], base, NC) == 0) --T;
  auto start_of = [&](uint32_t t) { return a.prefix ? a.prefix[t] : t * a.N; };
  bool ok = true;
  float db[4] = {0.f, 0.f, 0.f, 0.f};
  if (warp < kGroups) {
    const uint32_t acc = tmem + grp * MT * 2 * NC, whi = tmem + MT * kGroups * 2 * NC, wlo = whi + 64 * MT, dg = smem_u32(dgb);
    for (uint32_t t = T; t-- > 1;) {
      bar_sync(2 + grp, kGroupThreads + 32);     // the step's gradients are in place
      if (elect_one()) {
        fence_async();
        tc_after();
#pragma unroll
        for (uint32_t ks = 0; ks < 8; ++ks) {
          const uint64_t bd = umma_desc(dg + (ks / 4) * 2 * NC * 128) + 2 * (ks % 4);
          for (uint32_t mt = 0; mt < MT; ++mt)
            tc_kstep<NC>(acc + mt * 2 * NC, acc + mt * 2 * NC + NC, whi + mt * 64 + 8 * ks, wlo + mt * 64 + 8 * ks, bd, ks, 1);
        }
        umma_commit(&acc_full);
      }
      __syncwarp();
    }
  } else {
    constexpr int kCells = NC / 8;
    const uint32_t u = rank * kTcUnits + lane;
    const bool live_u = u < H;
    const uint32_t uc = min(u, H - 1);                   // (units that are not there read another's values and store nothing)
    // this warp's piece of the product: 32 rows (the units of rank `to`)
    const uint32_t quad = warp & 3, mt = gw >> 2, to = 4 * mt + quad;
    const float wscale = __int_as_float((scale_field(wmax[32 * to + lane]) - 14) << 23);   // (undoes the scale of the row this lane reads)
    const uint32_t tq = tmem + (grp * MT + mt) * 2 * NC + ((32 * quad) << 16);
    const float *pg = d.gates + uc, *pc = d.c + uc, *pc0 = d.c0 ? d.c0 + uc : nullptr;
    float *pdh = d.dh + uc, *pdc = DC ? d.dc + uc : nullptr, *phi = d.dn_hi + uc, *plo = d.dn_lo + uc;
    const uint32_t pitch = kH ? 4 * kH : a.dn_pitch;
    uint32_t phase[2] = {0, 0};
    float gt[kCells][4], cv[kCells], cp[kCells], dhv[kCells], dcv[kCells], dcs[kCells];
    unsigned char* dgo = dgb + op_off(2 * NC, gw, 4 * lane);   // (eight columns on: 1024 bytes)
    // cell j: column 8 j + gw
    auto fetch = [&](bool first, uint32_t c0, uint32_t cm1, uint32_t nact) {
#pragma unroll
      for (int j = 0; j < kCells; ++j) {
        const uint32_t i = 8 * j + gw, sc = base + (i < nact ? i : 0);
#pragma unroll
        for (int q = 0; q < 4; ++q) gt[j][q] = at(pg, c0 + sc, 16 * H)[(size_t)q * H];
        cv[j] = *at(pc, c0 + sc, 4 * H);
        dhv[j] = *at(pdh, c0 + sc, 4 * H);
        cp[j] = dcv[j] = 0.f;
        const float* before = first ? pc0 : pc;
        if (before) cp[j] = *at(before, first ? sc : cm1 + sc, 4 * H);
        if (DC) dcv[j] = *at(pdc, c0 + sc, 4 * H);
      }
    };
    // first columns of the steps t, t - 1, t - 2, each read a step before it is needed; columns active at step t
    uint32_t col = T ? start_of(T - 1) : 0, colm1 = T > 1 ? start_of(T - 2) : 0, colm2 = T > 2 ? start_of(T - 3) : 0;
    uint32_t n = T ? tc_active(start_of(T) - col, base, NC) : 0;
#pragma unroll
    for (int j = 0; j < kCells; ++j) {
      dcs[j] = 0.f;
    }
    if (T) fetch(T == 1, col, colm1, n);
    uint32_t n_later = 0, full = 0;
    for (uint32_t t = T; t-- > 0;) {
      const uint32_t pin = (t + 1) & 1, pout = t & 1, colm3 = t > 2 ? start_of(t - 3) : 0;
      float* in = part + (size_t)pin * C * kSlot;
      if (t && gw == 0 && lane == 0) msg_expect(&got[pout], n * (C - 1) * kTcUnits * 4);
      if (n_later) {
        ok = ok && msg_wait(&got[pin], phase[pin]);
        phase[pin] ^= 1;
      }
      float pr[kCells][4];
#pragma unroll
      for (int j = 0; j < kCells; ++j) {
        const uint32_t i = 8 * j + gw, sc = base + i;
        pr[j][0] = pr[j][1] = pr[j][2] = pr[j][3] = 0.f;
        if (i < n) {                    // (the same for the whole warp)
          float dh = dhv[j], dcp = 0.f;
          const float dci = dcv[j] + dcs[j];
          if (i < n_later) {
            const float* from = in + i * kTcUnits + lane;
            float r = 0.f;
#pragma unroll
            for (int q = 0; q < 8; ++q)
              if ((uint32_t)q < C) r += from[(size_t)q * kSlot];
            dh = d.mask ? fmaf(r, __ldg(at(d.mask + uc, a.mask_full ? sc : 0, 4 * H)), dh) : dh + r;
            if (live_u) {
              *at(pdh, col + sc, 4 * H) = dh;
              if (DC) *at(pdc, col + sc, 4 * H) = dci;
            }
          }
          lstm_cell_grad(gt[j][0], gt[j][1], gt[j][2], gt[j][3], cv[j], cp[j], dh, dci, true, dcp, pr[j][0], pr[j][1], pr[j][2], pr[j][3]);
          dcs[j] = dcp;
          if (!live_u) pr[j][0] = pr[j][1] = pr[j][2] = pr[j][3] = 0.f;
        }
        if (t) {
          // the column's scale, and its gradients as eight bytes of either plane per unit
          const uint32_t m = __reduce_max_sync(0xffffffffu, max(max(finite_mag(pr[j][0]), finite_mag(pr[j][1])), max(finite_mag(pr[j][2]), finite_mag(pr[j][3]))));
          const float scale = scale_of(m);
          if (lane == 0) colscale[t & 1][i] = __int_as_float((scale_field(m) - 14) << 23);   // 2^(E - 141)
          __half hi[4], lo[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) split_f16(pr[j][q] * scale, hi[q], lo[q]);
          *reinterpret_cast<uint2*>(dgo + j * 1024) = *reinterpret_cast<uint2*>(hi);
          *reinterpret_cast<uint2*>(dgo + j * 1024 + NC * 128) = *reinterpret_cast<uint2*>(lo);
        }
      }
      if (t) {
        fence_async();
        tc_before();
        bar_sync(2 + grp, kGroupThreads + 32);
      }
      // while the product runs: the next step's values, the operand planes of the weight gradients
      const uint32_t nm1 = t ? tc_active(col - colm1, base, NC) : 0;
      if (t) fetch(t == 1, colm1, colm2, nm1);
#pragma unroll
      for (int j = 0; j < kCells; ++j) {
        const uint32_t i = 8 * j + gw, sc = base + i;
        if (!live_u || i >= n) continue;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          db[q] += pr[j][q];
          float hi, lo;
          split_tf32(pr[j][q], hi, lo);
          at(phi, col + sc, 4 * pitch)[(size_t)q * H] = hi;
          at(plo, col + sc, 4 * pitch)[(size_t)q * H] = lo;
        }
      }
      if (t == 0) break;           // (no earlier state to hand dE/dh to)
      ok = ok && mbar_wait(&acc_full, full);
      full ^= 1;
      tc_after();
      // (columns that are not there are not sent: what the slot's owner sends later does not come before it has this)
      if (to < C) {
        float* slot = (to == rank ? part + (size_t)pout * C * kSlot : in) + to * kSlot;
        const float* cs = colscale[t & 1];
#pragma unroll
        for (int x = 0; x < (int)NC / 8; ++x) {
          if (8u * x >= n) break;
          float z[8], z2[8];
          tmem_ld8(tq + 8 * x, z);
          tmem_ld8(tq + NC + 8 * x, z2);
          tmem_ld_wait();
#pragma unroll
          for (int y = 0; y < 8; y += 4) {
            const float4 c = *reinterpret_cast<const float4*>(cs + 8 * x + y);
            float* o = slot + (8 * x + y) * kTcUnits + lane;
            o[0] = fmaf(z2[y], kLoScale, z[y]) * wscale * c.x;
            o[kTcUnits] = fmaf(z2[y + 1], kLoScale, z[y + 1]) * wscale * c.y;
            o[2 * kTcUnits] = fmaf(z2[y + 2], kLoScale, z[y + 2]) * wscale * c.z;
            o[3 * kTcUnits] = fmaf(z2[y + 3], kLoScale, z[y + 3]) * wscale * c.w;
          }
        }
        if (to != rank) {
          fence_async();
          __syncwarp();
          if (lane == 0)
            send_bulk(map_rank(smem_u32(part + ((size_t)pout * C + rank) * kSlot), to), slot, n * kTcUnits * 4, map_rank(smem_u32(&got[pout]), to));
        }
      }
      if (to == rank) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&got[pout]);
      }
      tc_before();
      n_later = n; n = nm1; col = colm1; colm1 = colm2; colm2 = colm3;
    }
  }
  if (!ok) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
  tc_before();
  __syncthreads();
  cluster_arrive();                // nobody leaves while a neighbour may still send to it
  cluster_wait();
  if (warp == 0) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols(MT * (kGroups * 2 * NC + 128))) : "memory");
  }
  if (warp >= kGroups) {
    // row sums of dgates: the threads of a unit, in ascending order (part is free: every CTA is through)
#pragma unroll
    for (int q = 0; q < 4; ++q) partall[((warp - kGroups) * 4 + q) * kTcUnits + lane] = db[q];
  }
  __syncthreads();
  if (tid < 128) {
    const uint32_t q = tid / kTcUnits, ul = tid % kTcUnits, u = rank * kTcUnits + ul;
    if (u < H) {
      float r = 0.f;
      for (uint32_t k = 0; k < kCellThreads / 32; ++k) r += partall[(k * 4 + q) * kTcUnits + ul];
      d.dbpart[(size_t)g * 4 * H + q * H + u] = r;
    }
  }
}

constexpr uint32_t tc_smem(bool bwd, uint32_t H) {
  const uint32_t NC = kTcCols, KB = (H + 63) / 64, C = (H + kTcUnits - 1) / kTcUnits;
  // (the partial sums' room also holds the row sums of dgates at the end, 512 bytes per cell warp)
  const uint32_t need = 1024 + kGroups * (bwd ? 2 * 2 * NC * 128 + 2 * C * NC * kTcUnits * 4 : 2 * 2 * KB * 2 * NC * 64 + 3 * NC * 512);
  return need > kTmemSmem ? need : kTmemSmem;
}
static_assert(tc_smem(true, 1) >= kTmemSmem && tc_smem(false, 1) >= kTmemSmem, "a recurrence that fits beside a waiting product");

typedef void (*TcFwd)(RecFwd);
typedef void (*TcBwd)(RecBwd);
// The instance of a launch.  Widths in whole 64 units (whose planes have no padding) have instances of their own: with the strides known the addresses of a
// cell's 16 - 23 accesses are a base and immediates instead of a third of all instructions.  256 units, 4096 columns of up to 100 steps: 1039 against 951 us
// forward, 1392 against 1194 backward; 64 and 128 units, 1400 columns: 108 -> 96 and 130 -> 106 with the copies, 142 -> 128 and 147 -> 135.
TcFwd tc_fwd_kernel(uint32_t H, uint32_t pitch) {
  if (H < 64) return k_rec_tc_fwd<0, false>;   // (see its inputs)
  if (pitch && pitch != H) return k_rec_tc_fwd<0>;
  switch (H) {
    case 64: return k_rec_tc_fwd<64>;
    case 128: return k_rec_tc_fwd<128>;
    case 192: return k_rec_tc_fwd<192>;
    case 256: return k_rec_tc_fwd<256>;
    default: return k_rec_tc_fwd<0>;
  }
}
template <bool DC>
TcBwd tc_bwd_kernel(uint32_t H, uint32_t pitch) {
  if (pitch != 4 * H) return k_rec_tc_bwd<DC, 0>;
  switch (H) {
    case 64: return k_rec_tc_bwd<DC, 64>;
    case 128: return k_rec_tc_bwd<DC, 128>;
    case 192: return k_rec_tc_bwd<DC, 192>;
    case 256: return k_rec_tc_bwd<DC, 256>;
    default: return k_rec_tc_bwd<DC, 0>;
  }
}

}  // namespace

// Clusters per direction (of kGroups x 16 columns each); all of them are the grid's second dimension.
bool dyb200_rec_tc_plan(dyb200_ctx* ctx, bool bwd, uint32_t H, uint32_t N, int ndir, RecTcPlan* out) {
  const uint64_t clusters = ((uint64_t)N + kGroups * kTcCols - 1) / (kGroups * kTcCols);
  if (H > 256 || N == 0 || clusters * ndir > 65535u) return false;
  const uint32_t C = (H + kTcUnits - 1) / kTcUnits;
  int16_t& fit = ctx->rec_tc_fit[bwd][C - 1];
  if (fit == 0) {   // (asked once: whether a cluster fits this device at all)
    const void* k = bwd ? (const void*)tc_bwd_kernel<true>(H, 4 * H) : (const void*)tc_fwd_kernel(H, H);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    if (dyb200_rec_launch_cfg(ctx, k, &cfg, attr, dim3(C, 1, 1), kTcThreads, tc_smem(bwd, H))) return false;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = -1; }
    fit = (int16_t)(n > 0 ? n : -1);
  }
  if (fit <= 0) return false;
  out->G = (uint32_t)clusters;
  return true;
}
int dyb200_rec_tc_fwd(dyb200_ctx* ctx, const RecTcPlan& p, RecFwd* a, int ndir) {
  a->G = p.G; a->ndir = (uint32_t)ndir; a->flags = ctx->dev_flags;
  const TcFwd k = tc_fwd_kernel(a->H, a->hn_pitch);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  int rc = dyb200_rec_launch_cfg(ctx, (const void*)k, &cfg, attr, dim3((a->H + kTcUnits - 1) / kTcUnits, p.G * ndir, 1), kTcThreads, tc_smem(false, a->H));
  if (rc) return rc;
  cudaLaunchKernelEx(&cfg, k, *a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}
int dyb200_rec_tc_bwd(dyb200_ctx* ctx, const RecTcPlan& p, RecBwd* a, int ndir) {
  a->G = p.G; a->ndir = (uint32_t)ndir; a->flags = ctx->dev_flags;
  const TcBwd k = a->d[0].dc ? tc_bwd_kernel<true>(a->H, a->dn_pitch) : tc_bwd_kernel<false>(a->H, a->dn_pitch);   // (both directions give dE/dc or neither)
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  int rc = dyb200_rec_launch_cfg(ctx, (const void*)k, &cfg, attr, dim3((a->H + kTcUnits - 1) / kTcUnits, p.G * ndir, 1), kTcThreads, tc_smem(true, a->H));
  if (rc) return rc;
  cudaLaunchKernelEx(&cfg, k, *a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}
