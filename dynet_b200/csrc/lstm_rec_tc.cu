// The recurrence of lstm_rec.cu for batches of more columns, on the tensor pipe: layers of at most 256 units, one launch per pass.
//
// What bounds it.  With more than four columns per cluster the fp32 multiply-adds of lstm_rec.cu bound its steps (0.2 us per column
// and step at 256 units: 8 us forward at 37 columns).  A step here is the same hand-over between CTAs around a product of 128 x
// 2 NC x K on tcgen05: the operands are 2 x 11 bit fp16 pairs (gemm.cuh), of which a CTA's share of Wh is 128 KB, so that it stays in
// half of the TMEM for the whole sequence; TF32 pairs of the same precision would need all of it.  (From shared memory the 32 MMAs of
// a step took 2400 cycles, each waiting for its 4 KB of Wh.)  A step is a chain of product, cell pass and one trip through the cluster.
//
// Columns: a cluster takes up to 16 NCH.  More than the clusters that fit run one after the other (no cluster waits for another);
// ragged batches are then dealt out in blocks of neighbours, longest first, so that every block ends with its own longest sentence.
//
// Cells: a warp's lanes are the CTA's 32 units of one column, so that every access to gates, states and operand planes is a full
// 128-byte line (8 units x 4 columns per access took four requests each: 3400 of a step's 9000 cycles went into the stores alone).
// Sixteen cell warps: with eight, a step waited on its own latencies (15000 cycles backward instead of 9000).
//
// Forward: CTA r owns 32 hidden units, 128 gate rows (row 32 q + unit); D (gate row x column) = Wh_r h, accumulators in TMEM.  The four
// warps that read the four gates of a group of columns exchange them through shared memory.  h_t goes to every CTA of the cluster as
// fp16 pairs in the layout of the MMA's right operand, one bulk copy per CTA (messages of 16 bytes, st.async, moved 10 bytes per cycle:
// 5000 cycles for 48 columns).  |h| < 1 and the largest dropout factor give one scale for the whole launch; an initial state has its own.
// Backward: D (unit of h_{t-1} x column) = Wh_r^T dgates_r over the CTA's own 128 gate rows, partial sums to the unit's owner.  dgates
// have no bound known in advance: a column's scale is the largest value of its 128 rows, found in the cell pass.
#include "lstm_rec.cuh"

#include "gemm.cuh"
#include "lstm_cell.cuh"
#include "lstm_rec_dev.cuh"
#include "tc_dev.cuh"

namespace {

// Warp 0 issues the products and the copies (the oldest warp of its scheduler goes first), warps 1 .. 16 are the cell warps.
constexpr uint32_t kCellThreads = 512, kTcThreads = kCellThreads + 32;
constexpr uint32_t kTcUnits = 32;      // hidden units per CTA

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
__device__ __forceinline__ uint32_t finite_mag(float v) {
  const uint32_t u = __float_as_uint(v) & 0x7fffffffu;
  return u < 0x7f800000u ? u : 0u;
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
// element `col * step` floats behind p
__device__ __forceinline__ float* at(float* p, uint32_t col, uint32_t step) { return p + (uint64_t)col * step; }
__device__ __forceinline__ const float* at(const float* p, uint32_t col, uint32_t step) { return p + (uint64_t)col * step; }
// columns of the block from `base` on that are active at a step of width B
__device__ __forceinline__ uint32_t tc_active(uint32_t B, uint32_t base, uint32_t ncap) { return B > base ? min(B - base, ncap) : 0; }
__device__ __forceinline__ uint32_t tmem_cols(uint32_t need) { return need <= 64 ? 64 : need <= 128 ? 128 : need <= 256 ? 256 : 512; }

// One k-block of 64: A_hi x [B_hi | B_lo] -> acc (2 NC columns), A_lo x B_hi -> its upper half, four k steps of 16.  A in TMEM: lane = row,
// a column holds two k.  b0 / b1: descriptors of the right operand's first and second 32 k.
template <int NC>
__device__ __forceinline__ void tc_kblock(uint32_t acc, uint32_t a_hi, uint32_t a_lo, uint64_t b0, uint64_t b1, uint32_t accumulate) {
  constexpr uint32_t base = (1u << 4) | ((uint32_t)(BM >> 4) << 24);   // fp32 accumulator, fp16 operands, both K-major
  constexpr uint32_t wide = base | ((uint32_t)(2 * NC >> 3) << 17), narrow = base | ((uint32_t)(NC >> 3) << 17);
  asm volatile(
      "{\n\t.reg .pred pf, pt;\n\t.reg .b32 xa, xl;\n\t.reg .b64 yb;\n\t"
      "setp.ne.b32 pf, %8, 0;\n\tsetp.eq.b32 pt, 0, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%2], %4, %6, pf;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [%3], %4, %7, pt;\n\t"
      "add.u32 xa, %2, 8;\n\tadd.u32 xl, %3, 8;\n\tadd.s64 yb, %4, 2;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [xa], yb, %6, pt;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [xl], yb, %7, pt;\n\t"
      "add.u32 xa, xa, 8;\n\tadd.u32 xl, xl, 8;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [xa], %5, %6, pt;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [xl], %5, %7, pt;\n\t"
      "add.u32 xa, xa, 8;\n\tadd.u32 xl, xl, 8;\n\tadd.s64 yb, %5, 2;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [xa], yb, %6, pt;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], [xl], yb, %7, pt;\n\t}"
      ::"r"(acc), "r"(acc + NC), "r"(a_hi), "r"(a_lo), "l"(b0), "l"(b1), "r"(wide), "r"(narrow), "r"(accumulate)
      : "memory");
}

// grid (C, blocks x directions), cluster (C, 1, 1).  Dynamic shared memory (1024-byte aligned):
// h [2][2 KB blocks of 32 units][NC hi rows, NC lo rows][64 bytes]; gates on their way [NC][4][32]; KB = ceil(H / 64).
// TMEM: accumulators (2 NC columns), Wh_hi and Wh_lo (32 KB columns each).
template <int NCH>
__global__ void __launch_bounds__(kTcThreads, 1) k_rec_tc_fwd(const __grid_constant__ RecFwd a) {
  constexpr uint32_t NC = 16 * NCH, kBlock = 2 * NC * 64;   // bytes of a CTA's part of h
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t got[2], acc_full, h_ready;
  __shared__ uint32_t tmem_slot, hword[2], wmax[128];
  const uint32_t ndir = a.ndir, dir = blockIdx.y % ndir, g = blockIdx.y / ndir;
  const RecDirF d = dir ? a.d[1] : a.d[0];
  const uint32_t H = a.H, rank = blockIdx.x, C = gridDim.x, KB = (H + 63) / 64;
  const uint32_t base = g * NC;
  unsigned char* hbuf = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t hbytes = 2 * KB * kBlock;
  float* exch = reinterpret_cast<float*>(hbuf + 2 * hbytes);
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    msg_init(&got[0]);
    msg_init(&got[1]);
    mbar_init(&acc_full, 1);
    mbar_init(&h_ready, kCellThreads / 32);
    hword[0] = hword[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 128) wmax[tid] = 0;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(tmem_cols(2 * NC + 64 * KB)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  dyb_grid_dep_sync();
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t ncol = tc_active(a.N, base, NC);

  // Wh of this CTA: lane = unit (128 contiguous bytes per load), a warp has 64 k of one gate.  The scale of a row is that of its largest
  // value.
  if (warp > 0) {
    float v[64];
    const uint32_t u = rank * kTcUnits + lane, q = warp & 3, kb = (warp - 1) >> 2, row = 32 * q + lane;
    const float* src = d.Wh + (size_t)q * H + u;
    uint32_t m = 0;
#pragma unroll
    for (int x = 0; x < 64; ++x) {
      const uint32_t k = 64 * kb + x;
      v[x] = k < H && u < H ? __ldg(at(src, k, 4 * H)) : 0.f;
    }
#pragma unroll
    for (int x = 0; x < 64; ++x) m = max(m, finite_mag(v[x]));
    atomicMax(&wmax[row], m);
    bar_sync(1, kCellThreads);
    if (kb < KB) {
      const float scale = scale_of(wmax[row]);
      const uint32_t to = tmem + 2 * NC + 32 * kb + ((32 * q) << 16);
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
  for (uint32_t e = tid; e < 2 * hbytes / 16; e += kTcThreads) reinterpret_cast<uint4*>(hbuf)[e] = make_uint4(0, 0, 0, 0);
  if (d.mask || d.h0) {
    uint32_t m0 = 0, m1 = 0;
    for (uint32_t e = tid; e < ncol * H; e += kTcThreads) {
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
  {
    const float s0 = scale_of(word0);
    for (uint32_t e = tid; e < ncol * H; e += kTcThreads) {
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
  if (warp == 0) {
    uint32_t phase[2] = {0, 0};
    const uint32_t whi = tmem + 2 * NC, wlo = whi + 32 * KB;
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
      if (lane == 0) {
        fence_async();
        tc_after();
        const uint32_t hb = smem_u32(h);
        for (uint32_t kb = 0; kb < KB; ++kb)
          tc_kblock<NC>(tmem, whi + kb * 32, wlo + kb * 32, umma_desc64(hb + 2 * kb * kBlock), umma_desc64(hb + (2 * kb + 1) * kBlock), kb);
        umma_commit(&acc_full);
      }
      __syncwarp();
      col1 = col2; col2 = col3; n = n1;
    }
  } else {
    // reads gate `quad` of the columns 16 j + c4 .. + 3, finishes column 16 j + c4 + quad; lane = unit
    const uint32_t quad = warp & 3, c4 = 4 * ((warp - 1) >> 2), u = rank * kTcUnits + lane, i0 = c4 + quad;
    const bool live_u = u < H;
    const uint32_t uc = min(u, H - 1);                  // (units that are not there read another's values and store nothing)
    const int wf = scale_field(wmax[32 * quad + lane]), t0 = wf + scale_field(word0) - 282, t1 = wf + scale_field(word1) - 282;
    const float hscale = live_u ? scale_of(word1) : 0.f;
    const uint32_t tq = tmem + ((32 * quad) << 16) + c4;
    const float* mask = d.mask ? d.mask + uc : nullptr;
    float *pg = d.gates + uc, *pc = d.c + uc, *ph = d.h + uc, *phi = d.hn_hi ? d.hn_hi + uc : nullptr, *plo = phi ? d.hn_lo + uc : nullptr;
    float pre[NCH][4], cst[NCH], mk[NCH];
    uint32_t ho[NCH];                                    // where h of cell j goes in this CTA's block
    auto fetch = [&](uint32_t c0, uint32_t nact) {
#pragma unroll
      for (int j = 0; j < NCH; ++j) {
        const uint32_t i = 16 * j + i0, col = c0 + base + (i < nact ? i : 0);
#pragma unroll
        for (int q = 0; q < 4; ++q) pre[j][q] = *at(pg + (size_t)q * H, col, 4 * H);
      }
    };
    fetch(0, n);
#pragma unroll
    for (int j = 0; j < NCH; ++j) {
      const uint32_t i = 16 * j + i0, sc = base + (i < ncol ? i : 0);
      cst[j] = d.c0 ? __ldg(at(d.c0 + uc, sc, H)) : 0.f;
      mk[j] = mask ? __ldg(at(mask, a.mask_full ? sc : 0, H)) : 1.f;
      ho[j] = h_off(2 * NC, i, rank * kTcUnits + lane);
    }
    for (uint32_t t = 0; t < a.T && n > 0; ++t) {
      const uint32_t col3 = start_of(t + 3), n1 = tc_active(col2 - col1, base, NC);
      unsigned char* hnext = hbuf + ((t & 1) ^ 1) * hbytes;
      const int ts = t ? t1 : t0, th = ts >> 1;
      const float f0 = __int_as_float((th + 127) << 23), f1 = __int_as_float((ts - th + 127) << 23);
      ok = ok && mbar_wait(&acc_full, t & 1);
      tc_after();
      {
        float z[4 * NCH], z2[4 * NCH];
#pragma unroll
        for (int j = 0; j < NCH; ++j) {
          tmem_ld4(tq + 16 * j, z + 4 * j);
          tmem_ld4(tq + NC + 16 * j, z2 + 4 * j);
        }
        tmem_ld_wait();
        tc_before();
#pragma unroll
        for (int j = 0; j < NCH; ++j)
#pragma unroll
          for (int x = 0; x < 4; ++x)
            exch[((16 * j + c4 + x) * 4 + quad) * 32 + lane] = (fmaf(z2[4 * j + x], kLoScale, z[4 * j + x]) * f0) * f1;
      }
      bar_sync(2 + c4 / 4, 128);
      float hv[NCH], hm[NCH], y[NCH][4];
#pragma unroll
      for (int j = 0; j < NCH; ++j) {
        const uint32_t i = 16 * j + i0;
#pragma unroll
        for (int q = 0; q < 4; ++q) y[j][q] = exch[(i * 4 + q) * 32 + lane];
        if (i >= n) continue;                            // (the same for the whole warp)
        y[j][0] = gate_sigmoid(y[j][0] + pre[j][0]);
        y[j][1] = gate_sigmoid(y[j][1] + pre[j][1] + a.fb);
        y[j][2] = gate_sigmoid(y[j][2] + pre[j][2]);
        y[j][3] = gate_tanh(y[j][3] + pre[j][3]);
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
      for (int j = 0; j < NCH; ++j) {
        const uint32_t i = 16 * j + i0, sc = base + i;
        if (!live_u || i >= n) continue;
#pragma unroll
        for (int q = 0; q < 4; ++q) *at(pg + (size_t)q * H, col0 + sc, 4 * H) = y[j][q];
        *at(pc, col0 + sc, H) = cst[j];
        *at(ph, col0 + sc, H) = hv[j];
        if (phi && i < n1) {
          float hi, lo;
          split_tf32(hm[j], hi, lo);
          *at(phi, col1 + sc, a.hn_pitch) = hi;
          *at(plo, col1 + sc, a.hn_pitch) = lo;
        }
      }
      if (n1) fetch(col1, n1);
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
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols(2 * NC + 64 * KB)) : "memory");
  }
}

// grid (C, blocks x directions), cluster (C, 1, 1).  Dynamic shared memory (1024-byte aligned): dgates [2 blocks of 64 gate rows]
// [NC hi rows, NC lo rows][128 bytes]; the partial sums [2][C ranks][NC columns][32 units].  TMEM: per row tile of 128 units the
// accumulators (2 NC columns); then Wh^T hi and lo (64 columns each per row tile).  The slots of the sums that have just been read hold the outgoing ones: what comes into slot r next, rank r
// sends after it has what went out of that slot.  Gate row (unit ul, gate q) is element 4 ul + q of the reduction.
template <int NCH>
__global__ void __launch_bounds__(kTcThreads, 1) k_rec_tc_bwd(const __grid_constant__ RecBwd a) {
  constexpr uint32_t NC = 16 * NCH, kSlot = NC * kTcUnits;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t got[2], acc_full;
  __shared__ uint32_t tmem_slot, wmax[256];
  __shared__ float colscale[2][NC];
  const uint32_t ndir = a.ndir, dir = blockIdx.y % ndir, g = blockIdx.y / ndir;
  const RecDirB d = dir ? a.d[1] : a.d[0];
  const uint32_t H = a.H, rank = blockIdx.x, C = gridDim.x, MT = (H + 127) / 128;
  const uint32_t base = g * NC;
  unsigned char* dgb = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* part = reinterpret_cast<float*>(dgb + 2 * 2 * NC * 128);
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    mbar_init(&got[0], 3);   // (the bytes of the others, and this CTA's own two warps)
    mbar_init(&got[1], 3);
    mbar_init(&acc_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 256) wmax[tid] = 0;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(tmem_cols(MT * (2 * NC + 128))) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  dyb_grid_dep_sync();
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = tmem_slot;

  // Lane = unit o of h_{t-1} (row o % 128 of its row tile), a warp has its weights in 16 of this CTA's units; scaled by the largest of all
  if (warp > 0) {
    float4 v[4][4];
    const bool quads = (H & 3) == 0 && aligned16(d.Wh);
    const uint32_t q4 = warp & 3, p4 = (warp - 1) >> 2, mt = p4 >> 1, kh = p4 & 1, o = 128 * mt + 32 * q4 + lane;
    uint32_t m = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const uint32_t uu = rank * kTcUnits + 16 * kh + 4 * x;
        const float* p = at(d.Wh + (size_t)q * H + uu, o, 4 * H);
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
    atomicMax(&wmax[o], m);
    bar_sync(1, kCellThreads);
    if (mt < MT) {
      const float scale = scale_of(wmax[o]);
      const uint32_t to = tmem + MT * 2 * NC + 64 * mt + 32 * kh + ((32 * q4) << 16);
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
  for (uint32_t e = tid; e < 2 * 2 * NC * 128 / 16; e += kTcThreads) reinterpret_cast<uint4*>(dgb)[e] = make_uint4(0, 0, 0, 0);
  fence_async();
  cluster_arrive();
  cluster_wait();

  // the last step that has a column of this block: widths never grow, so the steps before it have one too
  uint32_t T = a.T;
  while (a.prefix && T > 0 && tc_active(a.prefix[T] - a.prefix[T - 1], base, NC) == 0) --T;
  auto start_of = [&](uint32_t t) { return a.prefix ? a.prefix[t] : t * a.N; };
  bool ok = true;
  float db[4] = {0.f, 0.f, 0.f, 0.f};
  if (warp == 0) {
    const uint32_t whi = tmem + MT * 2 * NC, wlo = whi + 64 * MT, dg = smem_u32(dgb);
    for (uint32_t t = T; t-- > 1;) {
      bar_sync(2, kTcThreads);     // the step's gradients are in place
      if (lane == 0) {
        fence_async();
        tc_after();
        for (uint32_t mt = 0; mt < MT; ++mt)
          for (uint32_t kb = 0; kb < 2; ++kb) {
            const uint64_t b = umma_desc(dg + kb * 2 * NC * 128);
            tc_kblock<NC>(tmem + mt * 2 * NC, whi + mt * 64 + kb * 32, wlo + mt * 64 + kb * 32, b, b + 4, kb);
          }
        umma_commit(&acc_full);
      }
      __syncwarp();
    }
  } else {
    const uint32_t cw = warp - 1, quad = warp & 3, part4 = cw >> 2, u = rank * kTcUnits + lane;
    const bool live_u = u < H;
    const uint32_t uc = min(u, H - 1);                   // (units that are not there read another's values and store nothing)
    // this warp's piece of the product: 32 rows (the units of rank `to`) x 8 NCH columns from `cols` on
    const uint32_t to = 4 * (part4 >> 1) + quad, half = part4 & 1, cols = 8 * NCH * half;
    const float wscale = __int_as_float((scale_field(wmax[32 * to + lane]) - 14) << 23);   // (undoes the scale of the row this lane reads)
    const uint32_t tq = tmem + (part4 >> 1) * 2 * NC + cols + ((32 * quad) << 16);
    const float *pg = d.gates + uc, *pc = d.c + uc, *pc0 = d.c0 ? d.c0 + uc : nullptr;
    float *pdh = d.dh + uc, *pdc = d.dc ? d.dc + uc : nullptr, *phi = d.dn_hi + uc, *plo = d.dn_lo + uc;
    uint32_t phase[2] = {0, 0};
    float gt[NCH][4], cv[NCH], cp[NCH], dhv[NCH], dcv[NCH], dcs[NCH], mk[NCH];
    // cell j: column 16 j + cw
    auto fetch = [&](bool first, uint32_t c0, uint32_t cm1, uint32_t nact) {
#pragma unroll
      for (int j = 0; j < NCH; ++j) {
        const uint32_t i = 16 * j + cw, sc = base + (i < nact ? i : 0);
#pragma unroll
        for (int q = 0; q < 4; ++q) gt[j][q] = *at(pg + (size_t)q * H, c0 + sc, 4 * H);
        cv[j] = *at(pc, c0 + sc, H);
        dhv[j] = *at(pdh, c0 + sc, H);
        cp[j] = dcv[j] = 0.f;
        const float* before = first ? pc0 : pc;
        if (before) cp[j] = *at(before, first ? sc : cm1 + sc, H);
        if (pdc) dcv[j] = *at(pdc, c0 + sc, H);
      }
    };
    // first columns of the steps t, t - 1, t - 2, each read a step before it is needed; columns active at step t
    uint32_t col = T ? start_of(T - 1) : 0, colm1 = T > 1 ? start_of(T - 2) : 0, colm2 = T > 2 ? start_of(T - 3) : 0;
    uint32_t n = T ? tc_active(start_of(T) - col, base, NC) : 0;
#pragma unroll
    for (int j = 0; j < NCH; ++j) {
      const uint32_t sc = base + 16 * j + cw;
      dcs[j] = 0.f;
      mk[j] = d.mask && sc < a.N ? __ldg(at(d.mask + uc, a.mask_full ? sc : 0, H)) : 1.f;
    }
    if (T) fetch(T == 1, col, colm1, n);
    uint32_t n_later = 0, full = 0;
    for (uint32_t t = T; t-- > 0;) {
      const uint32_t pin = (t + 1) & 1, pout = t & 1, colm3 = t > 2 ? start_of(t - 3) : 0;
      float* in = part + (size_t)pin * C * kSlot;
      if (t && tid == 32) msg_expect(&got[pout], n * (C - 1) * kTcUnits * 4);
      if (n_later) {
        ok = ok && msg_wait(&got[pin], phase[pin]);
        phase[pin] ^= 1;
      }
      float pr[NCH][4];
#pragma unroll
      for (int j = 0; j < NCH; ++j) {
        const uint32_t i = 16 * j + cw, sc = base + i;
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
            dh = fmaf(r, mk[j], dh);
            if (live_u) {
              *at(pdh, col + sc, H) = dh;
              if (pdc) *at(pdc, col + sc, H) = dci;
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
          *reinterpret_cast<uint2*>(dgb + op_off(2 * NC, i, 4 * lane)) = *reinterpret_cast<uint2*>(hi);
          *reinterpret_cast<uint2*>(dgb + op_off(2 * NC, NC + i, 4 * lane)) = *reinterpret_cast<uint2*>(lo);
        }
      }
      if (t) {
        fence_async();
        tc_before();
        bar_sync(2, kTcThreads);
      }
      // while the product runs: the next step's values, the operand planes of the weight gradients
      const uint32_t nm1 = t ? tc_active(col - colm1, base, NC) : 0;
      if (t) fetch(t == 1, colm1, colm2, nm1);
#pragma unroll
      for (int j = 0; j < NCH; ++j) {
        const uint32_t i = 16 * j + cw, sc = base + i;
        if (!live_u || i >= n) continue;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          db[q] += pr[j][q];
          float hi, lo;
          split_tf32(pr[j][q], hi, lo);
          *at(phi + (size_t)q * H, col + sc, a.dn_pitch) = hi;
          *at(plo + (size_t)q * H, col + sc, a.dn_pitch) = lo;
        }
      }
      if (t == 0) break;           // (no earlier state to hand dE/dh to)
      ok = ok && mbar_wait(&acc_full, full);
      full ^= 1;
      tc_after();
      // (columns that are not there are neither written nor sent: their part of the slot may already be filling again)
      const uint32_t out = n > cols ? min(n - cols, 8u * NCH) : 0;
      if (to < C && out) {
        float* slot = (to == rank ? part + (size_t)pout * C * kSlot : in) + to * kSlot + cols * kTcUnits;
        const float* cs = colscale[t & 1] + cols;
#pragma unroll
        for (int x = 0; x < NCH; ++x) {
          if (8u * x >= out) break;
          float z[8], z2[8];
          tmem_ld8(tq + 8 * x, z);
          tmem_ld8(tq + NC + 8 * x, z2);
          tmem_ld_wait();
#pragma unroll
          for (int y = 0; y < 8; ++y)
            if (8u * x + y < out) slot[(8 * x + y) * kTcUnits + lane] = fmaf(z2[y], kLoScale, z[y]) * wscale * cs[8 * x + y];
        }
        if (to != rank) {
          fence_async();
          __syncwarp();
          if (lane == 0)
            send_bulk(map_rank(smem_u32(part + ((size_t)pout * C + rank) * kSlot + cols * kTcUnits), to), slot, out * kTcUnits * 4, map_rank(smem_u32(&got[pout]), to));
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
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols(MT * (2 * NC + 128))) : "memory");
  } else {
    // row sums of dgates: the sixteen threads of a unit, in ascending order (part is free: every CTA is through)
#pragma unroll
    for (int q = 0; q < 4; ++q) part[((warp - 1) * 4 + q) * kTcUnits + lane] = db[q];
  }
  __syncthreads();
  if (tid < 128) {
    const uint32_t q = tid / kTcUnits, ul = tid % kTcUnits, u = rank * kTcUnits + ul;
    if (u < H) {
      float r = 0.f;
      for (uint32_t k = 0; k < 16; ++k) r += part[(k * 4 + q) * kTcUnits + ul];
      d.dbpart[(size_t)g * 4 * H + q * H + u] = r;
    }
  }
}

constexpr uint32_t kTcMostCols = 64;   // columns per cluster: 165 KB of shared memory and, backward, all of the TMEM

uint32_t tc_smem(bool bwd, uint32_t H, uint32_t nch) {
  const uint32_t NC = 16 * nch, KB = (H + 63) / 64, C = (H + kTcUnits - 1) / kTcUnits;
  // (the partial sums' room also holds the 16 x 128 row sums of dgates at the end)
  const uint32_t part = 2 * C * NC * kTcUnits * 4;
  return 1024 + (bwd ? 2 * 2 * NC * 128 + (part > 8192 ? part : 8192) : 2 * 2 * KB * 2 * NC * 64 + NC * 512);
}
typedef void (*TcFwdKernel)(RecFwd);
typedef void (*TcBwdKernel)(RecBwd);
TcFwdKernel tc_fwd(uint32_t nch) { return nch == 1 ? k_rec_tc_fwd<1> : nch == 2 ? k_rec_tc_fwd<2> : nch == 3 ? k_rec_tc_fwd<3> : k_rec_tc_fwd<4>; }
TcBwdKernel tc_bwd(uint32_t nch) { return nch == 1 ? k_rec_tc_bwd<1> : nch == 2 ? k_rec_tc_bwd<2> : nch == 3 ? k_rec_tc_bwd<3> : k_rec_tc_bwd<4>; }
const void* tc_kernel(bool bwd, uint32_t nch) { return bwd ? (const void*)tc_bwd(nch) : (const void*)tc_fwd(nch); }

}  // namespace

// Room for columns in a cluster (16 per unit) and blocks of columns per direction: one round of clusters where that holds all columns, else
// rounds of full blocks.
bool dyb200_rec_tc_plan(dyb200_ctx* ctx, bool bwd, uint32_t H, uint32_t N, int ndir, RecTcPlan* out) {
  if (H > 256 || N == 0) return false;
  const uint32_t C = (H + kTcUnits - 1) / kTcUnits;
  int16_t& fit = ctx->rec_tc_fit[bwd][C - 1];
  if (fit == 0) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    if (dyb200_rec_launch_cfg(ctx, tc_kernel(bwd, kTcMostCols / 16), &cfg, attr, dim3(C, 1, 1), kTcThreads, tc_smem(bwd, H, kTcMostCols / 16))) return false;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, tc_kernel(bwd, kTcMostCols / 16), &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = -1; }
    fit = (int16_t)(n > 0 ? n : -1);
  }
  if (fit <= 0) return false;
  const uint32_t side = fit > ndir ? (uint32_t)(fit / ndir) : 1u;   // clusters per direction that run at the same time
  const uint32_t each = (N + side - 1) / side;                      // columns per cluster in one round
  out->nch = each > kTcMostCols ? kTcMostCols / 16 : (each + 15) / 16;
  out->G = (N + 16 * out->nch - 1) / (16 * out->nch);
  return true;
}
int dyb200_rec_tc_fwd(dyb200_ctx* ctx, const RecTcPlan& p, RecFwd* a, int ndir) {
  a->G = p.G; a->ncap = 16 * p.nch; a->ndir = (uint32_t)ndir; a->flags = ctx->dev_flags;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  int rc = dyb200_rec_launch_cfg(ctx, tc_kernel(false, p.nch), &cfg, attr, dim3((a->H + kTcUnits - 1) / kTcUnits, p.G * ndir, 1), kTcThreads, tc_smem(false, a->H, p.nch));
  if (rc) return rc;
  cudaLaunchKernelEx(&cfg, tc_fwd(p.nch), *a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}
int dyb200_rec_tc_bwd(dyb200_ctx* ctx, const RecTcPlan& p, RecBwd* a, int ndir) {
  a->G = p.G; a->ncap = 16 * p.nch; a->ndir = (uint32_t)ndir; a->flags = ctx->dev_flags;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  int rc = dyb200_rec_launch_cfg(ctx, tc_kernel(true, p.nch), &cfg, attr, dim3((a->H + kTcUnits - 1) / kTcUnits, p.G * ndir, 1), kTcThreads, tc_smem(true, a->H, p.nch));
  if (rc) return rc;
  cudaLaunchKernelEx(&cfg, tc_bwd(p.nch), *a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}
