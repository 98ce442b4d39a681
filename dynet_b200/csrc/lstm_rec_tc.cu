// The recurrence of lstm_rec.cu for batches of more columns, on the tensor pipe: layers of at most 256 units, one launch per pass.
//
// What bounds it.  With more than four columns per cluster the fp32 multiply-adds of lstm_rec.cu bound its steps (0.2 us per column
// and step at 256 units: 8 us forward at 37 columns).  A step here is the same hand-over by messages around a product of 128 x
// 2 NC x K on tcgen05: the operands are 2 x 11 bit fp16 pairs (gemm.cuh), of which a CTA's share of Wh is 128 KB, so that it stays in
// shared memory for the whole sequence; TF32 pairs of the same precision would need 256 KB.  A product of up to 64 columns costs the
// 32 MMAs' reads of that operand, 0.5 us whatever the columns; the rest of a step is the cell pass and one trip through the cluster.
//
// Columns: a cluster takes up to 16 NCH.  More than the clusters that fit run one after the other (no cluster waits for another);
// ragged batches are then dealt out in blocks of neighbours, longest first, so that every block ends with its own longest sentence.
//
// Forward: CTA r owns 32 hidden units, 128 gate rows; D (gate row x column) = Wh_r h, accumulators in TMEM, lane = gate row.  Rows are
// ordered so that a warp's 32 lanes are four gates of 8 units: two shuffle stages give each lane the gates of one unit and column.
// h_t goes to every CTA of the cluster as fp16 pairs in the layout of the MMA's right operand (16-byte messages, eight units).  |h| < 1
// and the largest dropout factor give one scale for the whole launch; an initial state has its own.
// Backward: D (unit of h_{t-1} x column) = Wh_r^T dgates_r over the CTA's own 128 gate rows, partial sums to the unit's owner.  dgates
// have no bound known in advance: a column's scale is the largest value of its 128 rows, found in the cell pass.
#include "lstm_rec.cuh"

#include "gemm.cuh"
#include "lstm_cell.cuh"
#include "lstm_rec_dev.cuh"
#include "tc_dev.cuh"

namespace {

constexpr uint32_t kTcThreads = 288;   // eight cell warps, one MMA warp
constexpr uint32_t kTcUnits = 32;      // hidden units per CTA

// Positions of a column's K-major operand row: byte offset of element k (even or odd) of row r in a plane block of `rows` rows per 64 k.
__device__ __forceinline__ uint32_t op_off(uint32_t rows, uint32_t r, uint32_t k) {
  return (k >> 6) * rows * 128 + r * 128 + ((((k & 63) >> 3) ^ (r & 7)) << 4) + (k & 7) * 2;
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
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                 "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// eight values as fp16 pairs into 16 bytes of either plane
__device__ __forceinline__ void store_pair8(unsigned char* hi, unsigned char* lo, const float (&v)[8], float scale) {
  __half h[8], l[8];
#pragma unroll
  for (int x = 0; x < 8; ++x) split_f16(v[x] * scale, h[x], l[x]);
  *reinterpret_cast<uint4*>(hi) = *reinterpret_cast<uint4*>(h);
  *reinterpret_cast<uint4*>(lo) = *reinterpret_cast<uint4*>(l);
}
// columns of block g active at a step of width B
__device__ __forceinline__ uint32_t tc_active(uint32_t B, uint32_t base, uint32_t stride, uint32_t ncap) {
  const uint32_t n = B > base ? (B - base + stride - 1) / stride : 0;
  return n < ncap ? n : ncap;
}
__device__ __forceinline__ constexpr uint32_t tmem_cols(uint32_t need) { return need <= 32 ? 32 : need <= 64 ? 64 : need <= 128 ? 128 : 256; }

// One k-block of 64 (see issue_kblock_f16): the instruction descriptors for 2 NC and NC columns.
template <int NC>
__device__ __forceinline__ void tc_kblock(uint32_t acc, uint32_t a_hi, uint32_t a_lo, uint32_t b, uint32_t accumulate) {
  constexpr uint32_t base = (1u << 4) | ((uint32_t)(BM >> 4) << 24);   // fp32 accumulator, fp16 operands, both K-major
  issue_kblock_f16(acc, acc + NC, umma_desc(a_hi), umma_desc(a_lo), umma_desc(b), base | ((uint32_t)(2 * NC >> 3) << 17),
                   base | ((uint32_t)(NC >> 3) << 17), accumulate, 2, 2);
}

// grid (C, blocks x directions), cluster (C, 1, 1).  Dynamic shared memory (1024-byte aligned): Wh_hi, Wh_lo [KB][128 rows][128 bytes],
// h [2][KB][NC hi rows, NC lo rows][128 bytes]; KB = ceil(H / 64).
template <int NCH>
__global__ void __launch_bounds__(kTcThreads, 1) k_rec_tc_fwd(const __grid_constant__ RecFwd a) {
  constexpr uint32_t NC = 16 * NCH, kCells = 2 * NCH;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t got[2], acc_full, acc_empty;
  __shared__ uint32_t tmem_slot, hword[2], wmax[128];
  __shared__ __align__(16) __half stage_all[8][64];
  const uint32_t ndir = a.ndir, dir = blockIdx.y % ndir, g = blockIdx.y / ndir;
  const RecDirF d = dir ? a.d[1] : a.d[0];
  const uint32_t H = a.H, rank = blockIdx.x, C = gridDim.x, KB = (H + 63) / 64;
  const uint32_t base = a.contiguous ? g * NC : g, stride = a.contiguous ? 1 : a.G;
  unsigned char* Whi = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* Wlo = Whi + KB * 16384;
  unsigned char* hbuf = Wlo + KB * 16384;
  const uint32_t hbytes = KB * 2 * NC * 128;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    msg_init(&got[0]);
    msg_init(&got[1]);
    mbar_init(&acc_full, 1);
    mbar_init(&acc_empty, 8);
    hword[0] = hword[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 128) wmax[tid] = 0;
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(tmem_cols(2 * NC)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  dyb_grid_dep_sync();
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t ncol = tc_active(a.N, base, stride, NC);

  // Wh of this CTA: gate row of (unit ul, gate q) is row 32 (ul / 8) + 8 q + ul % 8.  Lane = unit (128 contiguous bytes per load), warp
  // w has k in [8 KB w, + 8 KB).  The scale of a row is that of its largest value.
  if (warp < 8) {
    float v[4][4][8];
    const uint32_t u = rank * kTcUnits + lane, k0 = 8 * KB * warp;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          const uint32_t k = k0 + 8 * c + x;
          v[q][c][x] = (uint32_t)c < KB && k < H && u < H ? __ldg(d.Wh + (size_t)q * H + u + (size_t)4 * H * k) : 0.f;
        }
    const uint32_t row0 = 32 * (lane >> 3) + (lane & 7);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t m = 0;
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int x = 0; x < 8; ++x) m = max(m, finite_mag(v[q][c][x]));
      atomicMax(&wmax[row0 + 8 * q], m);
    }
    bar_sync(1, 256);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float scale = scale_of(wmax[row0 + 8 * q]);
#pragma unroll
      for (int c = 0; c < 4; ++c)
        if ((uint32_t)c < KB) {
          const uint32_t off = op_off(128, row0 + 8 * q, k0 + 8 * c);
          store_pair8(Whi + off, Wlo + off, v[q][c], scale);
        }
    }
  }
  // scales of h: the largest dropout factor (1 without); of the initial state: its largest value
  for (uint32_t e = tid; e < 2 * hbytes / 16; e += kTcThreads) reinterpret_cast<uint4*>(hbuf)[e] = make_uint4(0, 0, 0, 0);
  if (d.mask || d.h0) {
    uint32_t m0 = 0, m1 = 0;
    for (uint32_t e = tid; e < ncol * H; e += kTcThreads) {
      const uint32_t i = e / H, k = e % H, sc = base + stride * i;
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
      const uint32_t i = e / H, k = e % H, sc = base + stride * i;
      float v = 0.f;
      if (d.h0) v = __ldg(d.h0 + k + (size_t)H * sc) * (d.mask ? __ldg(d.mask + k + (a.mask_full ? (size_t)H * sc : 0)) : 1.f);
      __half hi, lo;
      split_f16(v * s0, hi, lo);
      *reinterpret_cast<__half*>(hbuf + op_off(2 * NC, i, k)) = hi;
      *reinterpret_cast<__half*>(hbuf + op_off(2 * NC, NC + i, k)) = lo;
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

  uint32_t B = a.prefix ? a.prefix[1] : a.N, n = tc_active(B, base, stride, NC);
  bool ok = true;
  if (warp == 8) {
    if (lane == 0) {
      uint32_t phase[2] = {0, 0};
      for (uint32_t t = 0; t < a.T && n > 0; ++t) {
        const uint32_t pt = t & 1, pn = pt ^ 1;
        const uint32_t B1 = t + 1 < a.T ? (a.prefix ? a.prefix[t + 2] - a.prefix[t + 1] : a.N) : 0, n1 = tc_active(B1, base, stride, NC);
        if (n1) msg_expect(&got[pn], n1 * C * kTcUnits * 4);
        if (t > 0) {
          ok = ok && msg_wait(&got[pt], phase[pt]);
          phase[pt] ^= 1;
          ok = ok && mbar_wait(&acc_empty, (t - 1) & 1);   // the accumulators of the step before have been read
        }
        fence_async();
        tc_after();
        const uint32_t h = smem_u32(hbuf + pt * hbytes), whi = smem_u32(Whi), wlo = smem_u32(Wlo);
        for (uint32_t kb = 0; kb < KB; ++kb) tc_kblock<NC>(tmem, whi + kb * 16384, wlo + kb * 16384, h + kb * 2 * NC * 128, kb);
        umma_commit(&acc_full);
        n = n1;
      }
    }
    __syncwarp();
  } else {
    const uint32_t quad = warp & 3, half = warp >> 2, u8 = lane & 7, cx = lane >> 3;   // (cx: gate of this lane's TMEM row; then its column)
    const uint32_t ul = 8 * quad + u8, u = rank * kTcUnits + ul;
    const bool live_u = u < H;
    const int wf = scale_field(wmax[32 * quad + lane]), t0 = wf + scale_field(word0) - 282, t1 = wf + scale_field(word1) - 282;
    const float hscale = scale_of(word1);
    __half* stage = stage_all[warp];
    const uint32_t tq = tmem + ((32 * quad) << 16);
    float pre[kCells][4], cst[kCells];
    // cell e: column 16 (e / 2) + 8 half + 4 (e % 2) + cx
    auto column = [&](int e) { return 16u * (e >> 1) + 8 * half + 4 * (e & 1) + cx; };
    auto fetch = [&](uint32_t c0, uint32_t nact) {
#pragma unroll
      for (int e = 0; e < (int)kCells; ++e) {
        const uint32_t i = column(e);
        const float* p = d.gates + u + (size_t)4 * H * (c0 + base + stride * i);
#pragma unroll
        for (int q = 0; q < 4; ++q) pre[e][q] = live_u && i < nact ? p[(size_t)q * H] : 0.f;
      }
    };
    uint32_t col0 = 0;
    fetch(0, n);
#pragma unroll
    for (int e = 0; e < (int)kCells; ++e) {
      const uint32_t i = column(e);
      cst[e] = d.c0 && live_u && i < ncol ? __ldg(d.c0 + u + (size_t)H * (base + stride * i)) : 0.f;
    }
    for (uint32_t t = 0; t < a.T && n > 0; ++t) {
      const uint32_t pn = (t & 1) ^ 1, col1 = col0 + B;
      const uint32_t B1 = t + 1 < a.T ? (a.prefix ? a.prefix[t + 2] - a.prefix[t + 1] : a.N) : 0, n1 = tc_active(B1, base, stride, NC);
      const uint32_t hnext = smem_u32(hbuf + pn * hbytes), bar = smem_u32(&got[pn]);
      ok = ok && mbar_wait(&acc_full, t & 1);
      tc_after();
      float z[8 * NCH];
      {
        float z2[8 * NCH];
#pragma unroll
        for (int j = 0; j < NCH; ++j) {
          tmem_ld8(tq + 16 * j + 8 * half, z + 8 * j);
          tmem_ld8(tq + NC + 16 * j + 8 * half, z2 + 8 * j);
        }
        tmem_ld_wait();
        const int ts = t ? t1 : t0, th = ts >> 1;
        const float f0 = __int_as_float((th + 127) << 23), f1 = __int_as_float((ts - th + 127) << 23);
#pragma unroll
        for (int e = 0; e < 8 * NCH; ++e) z[e] = (fmaf(z2[e], kLoScale, z[e]) * f0) * f1;
      }
      tc_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty);
      // gates of (unit, column 4 x + cx): a 4 x 4 transpose over the lanes that differ in cx
#pragma unroll
      for (int e = 0; e < (int)kCells; ++e) {
        float* y = z + 4 * e;
        const bool b0 = (cx & 1) != 0, b1 = (cx & 2) != 0;
        float s;
        s = __shfl_xor_sync(0xffffffffu, b0 ? y[0] : y[1], 8);  if (b0) y[0] = s; else y[1] = s;
        s = __shfl_xor_sync(0xffffffffu, b0 ? y[2] : y[3], 8);  if (b0) y[2] = s; else y[3] = s;
        s = __shfl_xor_sync(0xffffffffu, b1 ? y[0] : y[2], 16); if (b1) y[0] = s; else y[2] = s;
        s = __shfl_xor_sync(0xffffffffu, b1 ? y[1] : y[3], 16); if (b1) y[1] = s; else y[3] = s;
      }
      float hv[kCells], hm[kCells];
#pragma unroll
      for (int e = 0; e < (int)kCells; ++e) {
        const uint32_t i = column(e);
        float* y = z + 4 * e;
        hv[e] = hm[e] = 0.f;
        if (16u * (e >> 1) >= n) continue;       // (the same for the whole warp)
        const bool mine = live_u && i < n;
        if (mine) {
          y[0] = gate_sigmoid(y[0] + pre[e][0]);
          y[1] = gate_sigmoid(y[1] + pre[e][1] + a.fb);
          y[2] = gate_sigmoid(y[2] + pre[e][2]);
          y[3] = gate_tanh(y[3] + pre[e][3]);
          cst[e] = lstm_cell_c(y[0], y[3], y[1], cst[e]);
          hv[e] = lstm_cell_h(y[2], cst[e]);
          hm[e] = d.mask ? hv[e] * __ldg(d.mask + u + (a.mask_full ? (size_t)H * (base + stride * i) : 0)) : hv[e];
        }
        if (16u * (e >> 1) + 8 * half + 4 * (e & 1) < n1) {
          // eight units of a column are 16 bytes of either plane; lane: column cx, rank u8
          __half hi, lo;
          split_f16(hm[e] * hscale, hi, lo);
          __syncwarp();
          stage[16 * cx + u8] = hi;
          stage[16 * cx + 8 + u8] = lo;
          __syncwarp();
          if (u8 < C && i < n1) {
            const uint32_t k = rank * kTcUnits + 8 * quad, dbar = map_rank(bar, u8);
            send4(map_rank(hnext + op_off(2 * NC, i, k), u8), *reinterpret_cast<const float4*>(stage + 16 * cx), dbar);
            send4(map_rank(hnext + op_off(2 * NC, NC + i, k), u8), *reinterpret_cast<const float4*>(stage + 16 * cx + 8), dbar);
          }
        }
      }
#pragma unroll
      for (int e = 0; e < (int)kCells; ++e) {
        const uint32_t i = column(e), sc = base + stride * i;
        if (!live_u || i >= n) continue;
        const float* y = z + 4 * e;
        float* p = d.gates + u + (size_t)4 * H * (col0 + sc);
#pragma unroll
        for (int q = 0; q < 4; ++q) p[(size_t)q * H] = y[q];
        d.c[u + (size_t)H * (col0 + sc)] = cst[e];
        d.h[u + (size_t)H * (col0 + sc)] = hv[e];
        if (d.hn_hi && i < n1) {
          float hi, lo;
          split_tf32(hm[e], hi, lo);
          d.hn_hi[(size_t)(col1 + sc) * a.hn_pitch + u] = hi;
          d.hn_lo[(size_t)(col1 + sc) * a.hn_pitch + u] = lo;
        }
      }
      fetch(col1, n1);
      col0 = col1; B = B1; n = n1;
    }
  }
  if (!ok) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
  tc_before();
  __syncthreads();
  cluster_arrive();                // nobody leaves while a neighbour may still send to it
  cluster_wait();
  if (warp == 8) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols(2 * NC)) : "memory");
  }
}

// grid (C, blocks x directions), cluster (C, 1, 1).  Dynamic shared memory (1024-byte aligned): Wh^T hi, lo [row tile of 128 units]
// [2 blocks of 64 gate rows][128 rows][128 bytes]; dgates [2][NC hi rows, NC lo rows][128 bytes]; the partial sums
// [2][C source ranks][32 units][NC + 4 columns].  Gate row (unit ul, gate q) is element 4 ul + q of the reduction.
template <int NCH>
__global__ void __launch_bounds__(kTcThreads, 1) k_rec_tc_bwd(const __grid_constant__ RecBwd a) {
  constexpr uint32_t NC = 16 * NCH, kCells = 2 * NCH, PP = NC + 4;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t got[2], acc_full;
  __shared__ uint32_t tmem_slot, colmax[2][NC];
  const uint32_t ndir = a.ndir, dir = blockIdx.y % ndir, g = blockIdx.y / ndir;
  const RecDirB d = dir ? a.d[1] : a.d[0];
  const uint32_t H = a.H, rank = blockIdx.x, C = gridDim.x, MT = (H + 127) / 128;
  const uint32_t base = a.contiguous ? g * NC : g, stride = a.contiguous ? 1 : a.G;
  unsigned char* Whi = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  unsigned char* Wlo = Whi + MT * 32768;
  unsigned char* dgb = Wlo + MT * 32768;
  float* part = reinterpret_cast<float*>(dgb + 2 * 2 * NC * 128);
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    msg_init(&got[0]);
    msg_init(&got[1]);
    mbar_init(&acc_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (tid < 2 * NC) colmax[tid / NC][tid % NC] = 0;
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(tmem_cols(4 * NC)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  dyb_grid_dep_sync();
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = tmem_slot;

  // Thread o: unit o of h_{t-1}, its 128 weights in this CTA's gate rows, scaled by the largest of them
  uint32_t wword = 0;
  if (tid < MT * 128) {
    float4 v[4][8];
    const bool quads = (H & 3) == 0 && aligned16(d.Wh);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const uint32_t uu = rank * kTcUnits + 4 * x;
        const float* p = d.Wh + (size_t)q * H + uu + (size_t)4 * H * tid;
        float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tid < H && uu < H) {
          if (quads) w = __ldg(reinterpret_cast<const float4*>(p));
          else {
            w.x = __ldg(p);
            if (uu + 1 < H) w.y = __ldg(p + 1);
            if (uu + 2 < H) w.z = __ldg(p + 2);
            if (uu + 3 < H) w.w = __ldg(p + 3);
          }
        }
        v[q][x] = w;
        wword = max(wword, max(max(finite_mag(w.x), finite_mag(w.y)), max(finite_mag(w.z), finite_mag(w.w))));
      }
    const float scale = scale_of(wword);
    unsigned char *hi = Whi + (tid / 128) * 32768, *lo = Wlo + (tid / 128) * 32768;
#pragma unroll
    for (int x = 0; x < 8; ++x) {
      const float r0[8] = {v[0][x].x, v[1][x].x, v[2][x].x, v[3][x].x, v[0][x].y, v[1][x].y, v[2][x].y, v[3][x].y};
      const float r1[8] = {v[0][x].z, v[1][x].z, v[2][x].z, v[3][x].z, v[0][x].w, v[1][x].w, v[2][x].w, v[3][x].w};
      const uint32_t o0 = op_off(128, tid % 128, 16 * x), o1 = op_off(128, tid % 128, 16 * x + 8);
      store_pair8(hi + o0, lo + o0, r0, scale);
      store_pair8(hi + o1, lo + o1, r1, scale);
    }
  }
  for (uint32_t e = tid; e < 2 * 2 * NC * 128 / 16; e += kTcThreads) reinterpret_cast<uint4*>(dgb)[e] = make_uint4(0, 0, 0, 0);
  fence_async();
  cluster_arrive();
  cluster_wait();

  // the last step that has a column of this block: widths never grow, so the steps before it have one too
  uint32_t T = a.T;
  while (a.prefix && T > 0 && tc_active(a.prefix[T] - a.prefix[T - 1], base, stride, NC) == 0) --T;
  auto start_of = [&](uint32_t t) { return a.prefix ? a.prefix[t] : t * a.N; };
  uint32_t col = T ? start_of(T - 1) : 0, n = T ? tc_active(start_of(T) - col, base, stride, NC) : 0;
  bool ok = true;
  float db[4] = {0.f, 0.f, 0.f, 0.f};
  if (warp == 8) {
    for (uint32_t t = T; t-- > 1;) {
      bar_sync(2, kTcThreads);     // the step's gradients are in place
      if (lane == 0) {
        fence_async();
        tc_after();
        for (uint32_t mt = 0; mt < MT; ++mt)
          for (uint32_t kb = 0; kb < 2; ++kb)
            tc_kblock<NC>(tmem + mt * 2 * NC, smem_u32(Whi) + mt * 32768 + kb * 16384, smem_u32(Wlo) + mt * 32768 + kb * 16384,
                          smem_u32(dgb) + kb * 2 * NC * 128, kb);
        umma_commit(&acc_full);
      }
      __syncwarp();
    }
  } else {
    const uint32_t quad = warp & 3, half = warp >> 2, u8 = lane & 7, cx = lane >> 3, ul = 8 * quad + u8, u = rank * kTcUnits + ul;
    const bool live_u = u < H;
    const uint32_t to = 4 * half + quad;                 // the rank that owns this warp's 32 rows of the product
    const int wf = scale_field(wword);                   // (this thread's row of it: unit 32 to + lane = tid)
    const uint32_t tq = tmem + half * 2 * NC + ((32 * quad) << 16);
    uint32_t phase[2] = {0, 0};
    float gt[kCells][4], cv[kCells], cp[kCells], dhv[kCells], dcv[kCells], dcs[kCells];
    auto column = [&](int e) { return 16u * (e >> 1) + 8 * half + 4 * (e & 1) + cx; };
    auto fetch = [&](uint32_t t, uint32_t c0, uint32_t cm1, uint32_t nact) {
#pragma unroll
      for (int e = 0; e < (int)kCells; ++e) {
        const uint32_t i = column(e), sc = base + stride * i;
        const bool in = live_u && i < nact;
        const float* p = d.gates + u + (size_t)4 * H * (c0 + sc);
#pragma unroll
        for (int q = 0; q < 4; ++q) gt[e][q] = in ? p[(size_t)q * H] : 0.f;
        cv[e] = in ? d.c[u + (size_t)H * (c0 + sc)] : 0.f;
        cp[e] = !in ? 0.f : t ? d.c[u + (size_t)H * (cm1 + sc)] : d.c0 ? d.c0[u + (size_t)H * sc] : 0.f;
        dhv[e] = in ? d.dh[u + (size_t)H * (c0 + sc)] : 0.f;
        dcv[e] = in && d.dc ? d.dc[u + (size_t)H * (c0 + sc)] : 0.f;
      }
    };
#pragma unroll
    for (int e = 0; e < (int)kCells; ++e) dcs[e] = 0.f;
    if (T) fetch(T - 1, col, T > 1 ? start_of(T - 2) : 0, n);
    uint32_t n_later = 0, full = 0;
    for (uint32_t t = T; t-- > 0;) {
      const uint32_t colm1 = t ? start_of(t - 1) : 0, pin = (t + 1) & 1, pout = t & 1;
      if (t && tid == 0) msg_expect(&got[pout], (n + 3) / 4 * 4 * C * kTcUnits * 4);
      if (n_later) {
        ok = ok && msg_wait(&got[pin], phase[pin]);
        phase[pin] ^= 1;
      }
      const float* from = part + (size_t)pin * C * kTcUnits * PP + ul * PP;
      float pr[kCells][4];
#pragma unroll
      for (int e = 0; e < (int)kCells; ++e) {
        const uint32_t i = column(e), sc = base + stride * i;
        const bool mine = live_u && i < n;
        pr[e][0] = pr[e][1] = pr[e][2] = pr[e][3] = 0.f;
        if (mine) {
          float dh = dhv[e];
          const float dci = dcv[e] + dcs[e];
          if (i < n_later) {
            float r = 0.f;
            for (uint32_t q = 0; q < C; ++q) r += from[(size_t)q * kTcUnits * PP + i];
            if (d.mask) r *= __ldg(d.mask + u + (a.mask_full ? (size_t)H * sc : 0));
            dh += r;
            d.dh[u + (size_t)H * (col + sc)] = dh;
            if (d.dc) d.dc[u + (size_t)H * (col + sc)] = dci;
          }
          float dcp = 0.f;
          lstm_cell_grad(gt[e][0], gt[e][1], gt[e][2], gt[e][3], cv[e], cp[e], dh, dci, true, dcp, pr[e][0], pr[e][1], pr[e][2], pr[e][3]);
          dcs[e] = dcp;
        }
        if (t) {
          // (every lane takes part: the others' values are zeros)
          uint32_t m = max(max(finite_mag(pr[e][0]), finite_mag(pr[e][1])), max(finite_mag(pr[e][2]), finite_mag(pr[e][3])));
          m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
          m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
          m = max(m, __shfl_xor_sync(0xffffffffu, m, 4));
          if (u8 == 0) atomicMax(&colmax[t & 1][i], m);
        }
      }
      if (t) {
        bar_sync(1, 256);          // the columns' largest values are known
        if (tid < NC) colmax[pin][tid] = 0;   // (those of the step before are not needed any more, and not yet again)
#pragma unroll
        for (int e = 0; e < (int)kCells; ++e) {
          const uint32_t i = column(e);
          const float scale = scale_of(colmax[t & 1][i]);
          __half hi[4], lo[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) split_f16(pr[e][q] * scale, hi[q], lo[q]);
          *reinterpret_cast<uint2*>(dgb + op_off(2 * NC, i, 4 * ul)) = *reinterpret_cast<uint2*>(hi);
          *reinterpret_cast<uint2*>(dgb + op_off(2 * NC, NC + i, 4 * ul)) = *reinterpret_cast<uint2*>(lo);
        }
        fence_async();
        tc_before();
        bar_sync(2, kTcThreads);
      }
      // while the product runs: the operand planes of the weight gradients, and the next step's values
#pragma unroll
      for (int e = 0; e < (int)kCells; ++e) {
        const uint32_t i = column(e), sc = base + stride * i;
        if (!live_u || i >= n) continue;
        float* ph = d.dn_hi + (size_t)(col + sc) * a.dn_pitch + u;
        float* pl = d.dn_lo + (size_t)(col + sc) * a.dn_pitch + u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          db[q] += pr[e][q];
          float hi, lo;
          split_tf32(pr[e][q], hi, lo);
          ph[(size_t)q * H] = hi;
          pl[(size_t)q * H] = lo;
        }
      }
      if (t == 0) break;           // (no earlier state to hand dE/dh to)
      const uint32_t nm1 = tc_active(col - colm1, base, stride, NC);
      fetch(t - 1, colm1, t > 1 ? start_of(t - 2) : 0, nm1);
      ok = ok && mbar_wait(&acc_full, full);
      full ^= 1;
      tc_after();
      if (to < C) {
        const uint32_t dst = map_rank(smem_u32(part + (((size_t)pout * C + rank) * kTcUnits + lane) * PP), to), bar = map_rank(smem_u32(&got[pout]), to);
#pragma unroll
        for (int j = 0; j < NCH; ++j) {
          if (16u * j >= n) break;
          float z[16], z2[16];
          tmem_ld16(tq + 16 * j, z);
          tmem_ld16(tq + NC + 16 * j, z2);
          tmem_ld_wait();
#pragma unroll
          for (int x = 0; x < 16; ++x) z[x] = unscale(fmaf(z2[x], kLoScale, z[x]), wf + scale_field(colmax[t & 1][16 * j + x]) - 282);
#pragma unroll
          for (int x = 0; x < 4; ++x)
            if (16u * j + 4 * x < n) send4(dst + 4 * (16 * j + 4 * x), make_float4(z[4 * x], z[4 * x + 1], z[4 * x + 2], z[4 * x + 3]), bar);
        }
      }
      tc_before();
      n_later = n; n = nm1; col = colm1;
    }
  }
  if (!ok) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
  tc_before();
  __syncthreads();
  cluster_arrive();                // nobody leaves while a neighbour may still send to it
  cluster_wait();
  if (warp == 8) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols(4 * NC)) : "memory");
  }
  // row sums of dgates: the eight threads of a unit, in ascending order (part is free: every CTA is through)
  if (warp < 8) {
    const uint32_t ul = 8 * (warp & 3) + (lane & 7), k = 4 * (warp >> 2) + (lane >> 3);
#pragma unroll
    for (int q = 0; q < 4; ++q) part[(k * 4 + q) * kTcUnits + ul] = db[q];
  }
  __syncthreads();
  if (tid < 128) {
    const uint32_t q = tid / kTcUnits, ul = tid % kTcUnits, u = rank * kTcUnits + ul;
    if (u < H) {
      float r = 0.f;
      for (uint32_t k = 0; k < 8; ++k) r += part[(k * 4 + q) * kTcUnits + ul];
      d.dbpart[(size_t)g * 4 * H + q * H + u] = r;
    }
  }
}

constexpr size_t kTcSmemMax = 231 * 1000;   // beside 1.7 KB of static shared memory

uint32_t tc_smem(bool bwd, uint32_t H, uint32_t nch) {
  const uint32_t NC = 16 * nch, KB = (H + 63) / 64, MT = (H + 127) / 128, C = (H + kTcUnits - 1) / kTcUnits;
  return 1024 + (bwd ? MT * 65536 + 2 * 2 * NC * 128 + 2 * C * kTcUnits * (NC + 4) * 4 : KB * 32768 + 2 * KB * 2 * NC * 128);
}
typedef void (*TcFwdKernel)(RecFwd);
typedef void (*TcBwdKernel)(RecBwd);
TcFwdKernel tc_fwd(uint32_t nch) { return nch == 1 ? k_rec_tc_fwd<1> : nch == 2 ? k_rec_tc_fwd<2> : k_rec_tc_fwd<3>; }
TcBwdKernel tc_bwd(uint32_t nch) { return nch == 1 ? k_rec_tc_bwd<1> : nch == 2 ? k_rec_tc_bwd<2> : k_rec_tc_bwd<3>; }
const void* tc_kernel(bool bwd, uint32_t nch) { return bwd ? (const void*)tc_bwd(nch) : (const void*)tc_fwd(nch); }

}  // namespace

// Room for columns in a cluster (16 per unit), blocks of columns per direction, whether blocks are neighbours.  One round of clusters
// where that holds all columns; else rounds of full blocks.
bool dyb200_rec_tc_plan(dyb200_ctx* ctx, bool bwd, uint32_t H, uint32_t N, int ndir, RecTcPlan* out) {
  if (H > 256 || N == 0) return false;
  const uint32_t C = (H + kTcUnits - 1) / kTcUnits;
  int16_t& fit = ctx->rec_tc_fit[bwd][C - 1];
  uint32_t most = 3;
  while (most > 1 && tc_smem(bwd, H, most) > kTcSmemMax) --most;
  if (tc_smem(bwd, H, most) > kTcSmemMax) return false;
  if (fit == 0) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    if (dyb200_rec_launch_cfg(ctx, tc_kernel(bwd, most), &cfg, attr, dim3(C, 1, 1), kTcThreads, tc_smem(bwd, H, most))) return false;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, tc_kernel(bwd, most), &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = -1; }
    fit = (int16_t)(n > 0 ? n : -1);
  }
  if (fit <= 0) return false;
  const uint32_t side = fit > ndir ? (uint32_t)(fit / ndir) : 1u;   // clusters per direction that run at the same time
  RecTcPlan p;
  const uint32_t each = (N + side - 1) / side;                      // columns per cluster in one round
  p.nch = each > 16 * most ? most : (each + 15) / 16;
  p.contiguous = each > 16 * most;
  p.G = p.contiguous ? (N + 16 * p.nch - 1) / (16 * p.nch) : N < side ? N : side;
  *out = p;
  return true;
}
int dyb200_rec_tc_fwd(dyb200_ctx* ctx, const RecTcPlan& p, RecFwd* a, int ndir) {
  a->G = p.G; a->ncap = 16 * p.nch; a->contiguous = p.contiguous; a->ndir = (uint32_t)ndir; a->flags = ctx->dev_flags;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  int rc = dyb200_rec_launch_cfg(ctx, tc_kernel(false, p.nch), &cfg, attr, dim3((a->H + kTcUnits - 1) / kTcUnits, p.G * ndir, 1), kTcThreads, tc_smem(false, a->H, p.nch));
  if (rc) return rc;
  cudaLaunchKernelEx(&cfg, tc_fwd(p.nch), *a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}
int dyb200_rec_tc_bwd(dyb200_ctx* ctx, const RecTcPlan& p, RecBwd* a, int ndir) {
  a->G = p.G; a->ncap = 16 * p.nch; a->contiguous = p.contiguous; a->ndir = (uint32_t)ndir; a->flags = ctx->dev_flags;
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr[1];
  int rc = dyb200_rec_launch_cfg(ctx, tc_kernel(true, p.nch), &cfg, attr, dim3((a->H + kTcUnits - 1) / kTcUnits, p.G * ndir, 1), kTcThreads, tc_smem(true, a->H, p.nch));
  if (rc) return rc;
  cudaLaunchKernelEx(&cfg, tc_bwd(p.nch), *a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}
