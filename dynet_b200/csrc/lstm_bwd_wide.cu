// The backward recurrence of wide LSTM layers (more than 384 units) on fp16 pairs: what T calls of VanillaLSTMH, VanillaLSTMC and VanillaLSTMGates
// backward (dynet/nodes-lstm.cc:262-330, 415-470, 530-580) do in the order of the executor's backward sweep (dynet/exec.cc:96-140), with the products
// that need no step's predecessor - dx of all columns - taken out of the chain:
//     dh_{t-1} += mask_h .* (Wh^T dgates_t),  then the cell pass of step t - 1, which makes dgates_{t-1}      (k_bwd_wide<.., true>, resident)
//     dx += mask_x .* (Wx^T dgates)                                            all columns, one launch        (k_bwd_wide<.., false>)
// A CTA owns 128 units x BNT batch columns of Wh^T dgates and the share `rank` of its reduction; the S CTAs of a tile are one cluster and send each
// other partial sums through distributed shared memory, so that CTA r finishes 1/S of the tile's columns - dE/dh and, from the same registers, the
// cell pass of the step before.  The only hand-over through global memory is that of dgates: a counter per column block, which the next
// product's TMA thread polls (bounded, then DYB200_FLAG_WAIT_TIMEOUT, as every wait here).
//
// dgates as fp16 pairs (gemm.cuh): a column's values fade by many powers of two over the steps and their largest is not known before the cell pass is
// through everywhere, so a pair's scale belongs to (column, block of 128 units, all four gates) - what one warp of the cell pass holds.  The
// reduction is ordered by these blocks (4 gates x 128 units = 8 k-blocks of 64), each one accumulation chain that is unscaled as it is drained.
//
// A pair has 2 x 11 bits down to 2^-28 of its scale's largest value and an absolute error of 2^-50 of it below, where the TF32 pairs of the form before had an
// exponent each.  Quads of values that lie that low are added in fp32 ("small quads" below): without them a sum that only such values reach - units 2^-40 of
// others of their block, the others' weights zero - was off by 3e-4 of itself; looking for them costs 0.1 - 0.5 us a step.  Everywhere else the sums are better than
// those of TF32 pairs, a third of the truncated accumulations: error of whole sequences against float64 (2-norm, before / here)
// dh 3.1 - 4.1e-7 / 0.5 - 1.2e-7, dx 0.5 - 2.1e-6 / 2.5 - 5.9e-7, db 0.5 - 1.4e-6 / 1.2 - 4.8e-7, dWx and dWh 0.4 - 0.9 of before (1 - 1024 inputs, 385 - 1024 units,
// 9 - 512 columns, weights as initialised).
//
// Measured (us per step of 35, all of a layer's backward call, I = H = 1024; TF32 pairs with dx inside the recurrence / this form): batch 512 48.2 / 29.8,
// 256 35.8 / 17.8, 128 21.8 / 14.6, 64 16.6 / 9.5; batch 100 (a launch and more per step before) 31 / 14; 600 units, batch 30: 21 / 7.6; 777 units, batch 100
// (a value at a time, the weights' gates moved apart so that a k-block's copy starts on 16 bytes): 37 / 10.4.  dx is 10 of
// the 29.8, at 430 TFLOP/s useful.  What bounds the recurrence: at batch 512, two column blocks per CTA in turn (one block of 128 columns had nothing
// to overlap its exchange and cell pass with: 25 us a step against 20), 196 MB of operands per step from L2 at 11 - 14 TB/s; at batch 64 the chain
// itself: 0.5 until the first pairs of dgates are there, 2.8 for 8 k-blocks, 0.5 to drain the last, 1.2 exchange, 1.0 cell pass, 0.8 until the stores are
// out and counted, 0.5 until the count is seen.
#include "lstm_cell.cuh"
#include "seq_dev.cuh"

namespace {

struct BwdWide {
  uint32_t T, B, H, Hp, Ha;         // steps, columns per step, units, units rounded up to 64, distance of the gates in a row of the weights' pairs
  uint32_t kbs;                     // k-blocks of the product
  uint32_t P;                       // products of a column block: T - 1, and one more when dh_prev is given; dx: tiles
  uint32_t ncb, tiles_n;            // column blocks that a CTA serves in turn, of how many (dx: 1)
  uint32_t M, tiles_m;              // rows of the product and its tiles of 128
  const float *gates, *cs, *c0;     // step t at + t * 4 H B / + t * H B
  float *dh, *dc;                   // dE/dh, dE/dc of the steps (accumulated; dc may be null: none from outside, T = 1)
  float *dh_prev, *dc_prev;         // those of the step before the first (null: not wanted)
  float *dn_hi, *dn_lo; uint32_t dn_pitch;       // TF32 planes of dgates for the weight gradients: row = column of the sequence
  __half *d16_hi, *d16_lo;          // fp16 pairs, row = column of the sequence, gate q's unit u at q Hp + u (zeros from H on)
  uint32_t* dsc; uint32_t dsc_ld;   // scale words [block of 128 units][column of the sequence]; bit 0: small quads
  const float* W;                   // Wh (dx: Wx)
  const uint32_t* wscale;           // of the rows of W^T; bit 0: small quads
  float* part;                      // row sums of dgates: [step in sweep order][column block, rank][4H]
  const float* mask; int mask_full; // of the result's rows; full: one column per batch column
  float* dx; uint32_t columns;      // dx only
  int fresh_dx, fresh_dc;           // dx is written and not added to; dE/dc of a step before it is added to: zeros, whatever dc holds
  uint32_t* done;                   // a counter per column block, zero at launch (cleared by the launch that sums up db)
  uint32_t* flags;
};

// k-block i of the reduction: block of 128 units (i / 8), gate, half.  The last block has 64 units or fewer when H % 128 is in 1 .. 64.
struct KBlock { int xa, xb; };
__device__ __forceinline__ KBlock k_block(uint32_t i, uint32_t H, uint32_t Ha, uint32_t Hp) {
  const uint32_t full = H / BM, blk = i >> 3;
  uint32_t q = (i >> 1) & 3, h = i & 1;
  if (blk >= full && H % BM <= 64) { q = i - 8 * full; h = 0; }
  const uint32_t u = BM * min(blk, full) + 64 * h;
  return KBlock{(int)(q * Ha + u), (int)(q * Hp + u)};
}

constexpr int kMaxBlocks = 4;   // column blocks per CTA
// A CTA that adds many small quads (below) is milliseconds late, and the others wait for it.  ms a step where every quad but one of a scale is small, of dgates / of
// weights: 1024 units, 512 columns 2.3 / 9, 2048 units, 500 columns 14 / 37, 3072 units, 1000 columns 93 / 148 (past the other kernels' bound).
constexpr uint32_t kLongWait = 16 * kWaitLimit;

struct CellIn { float4 gi, gf, go, gg, c, cp, dci, dcp; };
// What a thread of the eight warps that share a CTA's columns does of the cell pass: units [u, + 4) of block `blk`, `left` of them there (own: any)
struct CellUnits { uint32_t blk, u, left; bool own; };

template <bool VEC>
__device__ __forceinline__ void cell_load(const BwdWide& a, const CellUnits& q, CellIn& in, uint32_t t, uint32_t n) {
  const size_t HB = (size_t)a.H * a.B, e = (size_t)n * a.H + q.u;
  const float* g = a.gates + (size_t)t * 4 * HB + (size_t)n * 4 * a.H + q.u;
  in.gi = ldu<VEC>(g, q.left); in.gf = ldu<VEC>(g + a.H, q.left); in.go = ldu<VEC>(g + 2 * a.H, q.left); in.gg = ldu<VEC>(g + 3 * a.H, q.left);
  in.c = ldu<VEC>(a.cs + (size_t)t * HB + e, q.left);
  in.cp = ldu<VEC>((t ? a.cs + (size_t)(t - 1) * HB : a.c0) + e, q.left);
  const float* dcp = t ? a.dc + (size_t)(t - 1) * HB : a.dc_prev;
  in.dci = a.dc && !(a.fresh_dc && t == a.T - 1) ? ldu_cg<VEC>(a.dc + (size_t)t * HB + e, q.left) : make_float4(0.f, 0.f, 0.f, 0.f);
  in.dcp = dcp && !a.fresh_dc ? ldu_cg<VEC>(dcp + e, q.left) : make_float4(0.f, 0.f, 0.f, 0.f);
}
template <bool VEC>
__device__ __forceinline__ void planes_out(const BwdWide& a, const CellUnits& q, const float4 (&p)[4], uint32_t t, uint32_t n) {   // dgates for the weight gradients
  const size_t o = ((size_t)t * a.B + n) * a.dn_pitch + q.u;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float4 hi, lo;
    split_tf32(p[k].x, hi.x, lo.x); split_tf32(p[k].y, hi.y, lo.y); split_tf32(p[k].z, hi.z, lo.z); split_tf32(p[k].w, hi.w, lo.w);
    stu<VEC>(a.dn_hi + o + (size_t)k * a.H, hi, q.left); stu<VEC>(a.dn_lo + o + (size_t)k * a.H, lo, q.left);
  }
}
// Small quads: four neighbouring units' gradients of a gate, or four weights of a row side by side, that are not all zero and all lie 2^28 below the largest
// value of their scale, so that pairs would keep little of them.  They are zeros in the pairs, bit 0 of the scale's word tells of them, and the warp that
// finishes a column adds their products in fp32, from the planes of dgates for the weight gradients (small_parts).  So no value is further off than 2^-22 of
// the largest of its quad, whatever else shares its scale.  The rule of the flush, there a row's blocks of eight columns, for the same reason.
__device__ __forceinline__ uint32_t quad_mag(float4 v) { return max(max(finite_mag(v.x), finite_mag(v.y)), max(finite_mag(v.z), finite_mag(v.w))); }
// What the cell pass does besides where it finds one (small), or the weights have some: the column's planes go out before they are published, and the pairs again.
template <bool VEC>
__device__ __forceinline__ void cell_small(const BwdWide& a, CellUnits q, float4 p0, float4 p1, float4 p2, float4 p3, uint32_t t, uint32_t n, uint32_t word) {
  if (!q.own) return;
  const float4 p[4] = {p0, p1, p2, p3};
  planes_out<VEC>(a, q, p, t, n);
  if (!word) return;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float v[4], h, l;
#pragma unroll
    for (int i = 0; i < 4; ++i) { split_tf32((&p[k].x)[i], h, l); v[i] = h + l; }   // (what small_parts will see)
    if (!pair_loses(quad_mag(make_float4(v[0], v[1], v[2], v[3])), word)) continue;
    const size_t o = (((size_t)t * a.B + n) * 4 + k) * a.Hp + q.u;
    *reinterpret_cast<uint2*>(a.d16_hi + o) = *reinterpret_cast<uint2*>(a.d16_lo + o) = make_uint2(0, 0);
  }
}
// Quad of gate k from unit u on, of a column's planes (zeros past the last unit)
__device__ __forceinline__ float4 quad_of(const BwdWide& a, const float* hi, const float* lo, uint32_t k, uint32_t u) {
  float v[4];
#pragma unroll
  for (uint32_t i = 0; i < 4; ++i) v[i] = u + i < a.H ? __ldcg(hi + k * a.H + u + i) + __ldcg(lo + k * a.H + u + i) : 0.f;
  return make_float4(v[0], v[1], v[2], v[3]);
}
// The products of the small quads of column r (of the sequence) and of rows [m, + 4); a warp.
__device__ __noinline__ float4 small_parts(const BwdWide& a, uint32_t r, uint32_t m) {
  const uint32_t lane = threadIdx.x & 31, G = 4 * a.H;
  const float *hi = a.dn_hi + (size_t)r * a.dn_pitch, *lo = a.dn_lo + (size_t)r * a.dn_pitch;
  const bool vec = (a.H & 3) == 0 && aligned16(a.W);
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  for (uint32_t b = 0; b * BM < a.H; ++b) {
    const uint32_t word = __ldcg(a.dsc + (size_t)b * a.dsc_ld + r);
    if (!(word & 1)) continue;
    float4 v[4];
    uint32_t hits[4], n = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
      v[k] = quad_of(a, hi, lo, k, b * BM + 4 * lane);
      const bool hit = pair_loses(quad_mag(v[k]), word);
      if (!hit) v[k] = make_float4(0.f, 0.f, 0.f, 0.f);
      hits[k] = __ballot_sync(0xffffffffu, hit);
      n += __popc(hits[k]);
    }
    if (n <= 6) {   // a few: quad by quad, every lane its rows (32 sectors a load: 16 such loads a quad)
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k)
        for (uint32_t left = hits[k]; left; left &= left - 1) {
          const uint32_t src = __ffs(left) - 1, u = b * BM + 4 * src;
#pragma unroll
          for (uint32_t i = 0; i < 4; ++i) {
            const float x = __shfl_sync(0xffffffffu, (&v[k].x)[i], src);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
              if (u + i < a.H && m + j < a.M) acc[j] = fmaf(__ldg(a.W + k * a.H + u + i + (size_t)G * (m + j)), x, acc[j]);
          }
        }
    } else {   // many: row by row, every lane its quads (whole lines; 1024 units, 512 columns, all of them small: 39 ms -> 6.9 for three steps)
      const uint32_t u = b * BM + 4 * lane, left = u < a.H ? a.H - u : 0;
      for (uint32_t src = 0; src < 32; ++src)
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
          const uint32_t row = __shfl_sync(0xffffffffu, m, src) + j;
          float sum = 0.f;
          if (row < a.M && left) {
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
              const float* p = a.W + (size_t)G * row + k * a.H + u;
              const float4 w = vec ? __ldg(reinterpret_cast<const float4*>(p)) : ldu<false>(p, left);
              sum = fmaf(w.x, v[k].x, fmaf(w.y, v[k].y, fmaf(w.z, v[k].z, fmaf(w.w, v[k].w, sum))));
            }
          }
          sum = warp_sum(sum);
          if (lane == src) acc[j] += sum;
        }
    }
  }
  // those of the weights' rows, 32 quads at a time, with what has not been added above
  uint32_t rows[4];
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j) rows[j] = __ballot_sync(0xffffffffu, m + j < a.M && (__ldg(a.wscale + m + j) & 1));
  if ((rows[0] | rows[1] | rows[2] | rows[3]) == 0) return make_float4(acc[0], acc[1], acc[2], acc[3]);
  for (uint32_t e = 4 * lane; e < (G + 127) / 128 * 128; e += 128) {   // (G is a multiple of four)
    float v[4];
    bool have = false;   // (the dgates, once a row wants them)
#pragma unroll
    for (uint32_t j = 0; j < 4; ++j)
      for (uint32_t left = rows[j]; left; left &= left - 1) {
        const uint32_t src = __ffs(left) - 1, row = __shfl_sync(0xffffffffu, m, src) + j;
        const float* w = a.W + (size_t)G * row + e;
        const float4 x = e >= G ? make_float4(0.f, 0.f, 0.f, 0.f) : aligned16(a.W) ? __ldg(reinterpret_cast<const float4*>(w)) : make_float4(__ldg(w), __ldg(w + 1), __ldg(w + 2), __ldg(w + 3));
        const bool hit = pair_loses(quad_mag(x), __ldg(a.wscale + row));
        if (!__any_sync(0xffffffffu, hit)) continue;
        if (!have) {
          have = true;
#pragma unroll
          for (uint32_t i = 0; i < 4; ++i) {
            const uint32_t k = (e + i) / a.H, u = (e + i) % a.H;
            const float4 q = e < G ? quad_of(a, hi, lo, k, u / 4 * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[i] = e < G && !pair_loses(quad_mag(q), __ldcg(a.dsc + (size_t)(u / BM) * a.dsc_ld + r)) ? (u % 4 == 0 ? q.x : u % 4 == 1 ? q.y : u % 4 == 2 ? q.z : q.w) : 0.f;
          }
        }
        const float sum = warp_sum(hit ? fmaf(x.x, v[0], fmaf(x.y, v[1], fmaf(x.z, v[2], x.w * v[3]))) : 0.f);
        if (lane == src) acc[j] += sum;
      }
  }
  return make_float4(acc[0], acc[1], acc[2], acc[3]);
}
// The cell pass of units [u, + 4), column n of step t from dE/dh: dE/dc of the step before, and dgates as fp16 pairs with the word of the warp's
// (column, block).  The four gates' gradients come back in p and are added to rs.  (All lanes of a warp take part; those past the last unit with zeros.)
// Returns its word where there are small quads, else 0.
__device__ __forceinline__ uint32_t cell(const BwdWide& a, const CellUnits& q, CellIn& in, float4 dh, uint32_t t, uint32_t n, float4 (&p)[4], float4 (&rs)[4]) {
  uint32_t m = 0, low = 0xffffffffu;   // the largest magnitude, and that of the smallest quad that is not zero, less one
#pragma unroll
  for (int k = 0; k < 4; ++k) p[k] = make_float4(0.f, 0.f, 0.f, 0.f);
  if (q.own) {
    const float* f[8] = {&in.gi.x, &in.gf.x, &in.go.x, &in.gg.x, &in.c.x, &in.cp.x, &dh.x, &in.dci.x};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      lstm_cell_grad(f[0][k], f[1][k], f[2][k], f[3][k], f[4][k], f[5][k], f[6][k], f[7][k], a.dc != nullptr, (&in.dcp.x)[k], (&p[0].x)[k], (&p[1].x)[k],
                     (&p[2].x)[k], (&p[3].x)[k]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t w = quad_mag(p[k]);
      m = max(m, w);
      low = min(low, w - 1);
      rs[k].x += p[k].x; rs[k].y += p[k].y; rs[k].z += p[k].z; rs[k].w += p[k].w;
    }
  }
  m = __reduce_max_sync(0xffffffffu, m);
  const size_t r = (size_t)t * a.B + n;
  const float s = scale_of(m);
  if (q.u < a.Hp) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      __half hi[4], lo[4];
      split_f16(p[k].x * s, hi[0], lo[0]); split_f16(p[k].y * s, hi[1], lo[1]); split_f16(p[k].z * s, hi[2], lo[2]); split_f16(p[k].w * s, hi[3], lo[3]);
      const size_t o = (r * 4 + k) * a.Hp + q.u;
      *reinterpret_cast<uint2*>(a.d16_hi + o) = *reinterpret_cast<const uint2*>(hi);
      *reinterpret_cast<uint2*>(a.d16_lo + o) = *reinterpret_cast<const uint2*>(lo);
    }
  }
  const uint32_t small = __any_sync(0xffffffffu, pair_loses(low + 1, m));
  if ((threadIdx.x & 31) == 0) a.dsc[(size_t)q.blk * a.dsc_ld + r] = (m & ~1u) | small;
  return small ? m | 1u : 0u;
}
template <bool VEC>
__device__ __forceinline__ void cell_rest(const BwdWide& a, const CellUnits& q, const CellIn& in, const float4 (&p)[4], uint32_t t, uint32_t n) {   // dE/dc of the step before, the planes
  if (!q.own) return;
  float* dcp = t ? a.dc + (size_t)(t - 1) * a.H * a.B : a.dc_prev;
  if (dcp) stu<VEC>(dcp + (size_t)n * a.H + q.u, in.dcp, q.left);
  planes_out<VEC>(a, q, p, t, n);
}
// The row sums of a CTA's columns in a step (part: those of its column block and rank), through 4096 floats of shared memory: the eight warps' columns
// in order.  te: thread of the 256.
__device__ __forceinline__ void row_sums(const BwdWide& a, const float4 (&rs)[4], float* park, float* part, uint32_t blk, uint32_t te, uint32_t ew, uint32_t uq, bool ok) {
#pragma unroll
  for (int q = 0; q < 4; ++q) st4(park + (ew * 4 + q) * BM + uq, rs[q]);
  bar_sync(1, 256);
#pragma unroll
  for (uint32_t k = 0; k < 2; ++k) {
    const uint32_t r = te + 256 * k, q = r / BM, j = r % BM;
    float v[8];
#pragma unroll
    for (int x = 0; x < 8; ++x) v[x] = park[(x * 4 + q) * BM + j];
#pragma unroll
    for (int x = 1; x < 8; ++x) v[0] += v[x];
    if (ok && blk * BM + j < a.H) part[(size_t)q * a.H + blk * BM + j] = v[0];
  }
  bar_sync(1, 256);
}
__device__ __forceinline__ float* part_of(const BwdWide& a, uint32_t step, uint32_t block, uint32_t splits, uint32_t rank) {
  return a.part + (((size_t)step * a.tiles_n + block) * splits + rank) * 4 * a.H;
}

// The cell pass of a single step on its own: what a CTA of the recurrence does before its first product, its columns and their order included - the row sums
// of dgates are the sequence's bit for bit.  Bound by its few loads' latency (a column per warp at eight splits); no cluster, no TMEM, 16 KB.
// grid = (tiles_m, tiles_n, splits)
template <bool VEC>
__global__ void __launch_bounds__(256) k_bwd_cells(const __grid_constant__ BwdWide a) {
  dyb_grid_dep_sync();
  __shared__ __align__(16) float park[32 * BM];
  const uint32_t ew = threadIdx.x >> 5, u = blockIdx.x * BM + 4 * (threadIdx.x & 31), w = 64 / gridDim.z;
  const CellUnits un{blockIdx.x, u, a.H - u, u < a.H};
  float4 rs[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) rs[q] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
  for (uint32_t c = ew; c < w; c += 8) {
    const uint32_t n = 64 * blockIdx.y + blockIdx.z * w + c;
    if (n >= a.B) break;
    CellIn in = {};
    float4 dh = make_float4(0.f, 0.f, 0.f, 0.f), p[4];
    if (un.own) { cell_load<VEC>(a, un, in, 0, n); dh = ldu<VEC>(a.dh + (size_t)n * a.H + u, un.left); }
    const uint32_t word = cell(a, un, in, dh, 0, n, p, rs);
    if (word) cell_small<VEC>(a, un, p[0], p[1], p[2], p[3], 0, n, word);
    cell_rest<VEC>(a, un, in, p, 0, n);
  }
  row_sums(a, rs, park, part_of(a, 0, blockIdx.y, gridDim.z, blockIdx.z), blockIdx.x, threadIdx.x, ew, 4 * (threadIdx.x & 31), true);
}

// REC: the recurrence, grid = (tiles_m, column blocks, S).  Otherwise dx: grid = (clusters, 1, S), the clusters walk the tiles.
// VEC: units in fours, on 16 bytes (dx has a rule of its own for its rows).
template <int BNT, uint32_t S, bool REC, bool VEC>
__global__ void __launch_bounds__(kThreads, 1) k_bwd_wide(const __grid_constant__ TmapPack tm, const __grid_constant__ BwdWide a) {
  constexpr int kStages = BNT == 64 ? 4 : 3;
  constexpr int TILE_B_BYTES = BNT * BK * 4, kStageBytes = 2 * TILE_BYTES + 2 * TILE_B_BYTES;
  constexpr uint32_t kAccCols = 2 * BNT, kBufs = kSeqBufs * BN / kAccCols, kHalf = BNT / 2, kParkBytes = 64 * BM * 4;
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[kStages], empty_bar[kStages], acc_full[kBufs], acc_empty[kBufs], park_full, park_free, go[kMaxBlocks];
  __shared__ uint32_t tmem_base_slot;
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* park = reinterpret_cast<float*>(ring + (size_t)kStages * kStageBytes);   // 64 columns x BM rows
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.z;
  if (a.T == 1) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // this CTA's k-blocks: an equal share, or (dx with splits) one block of units, so that the sums are those of the unsplit form
  const uint32_t per = REC || S == 1 ? (a.kbs + S - 1) / S : 8, k0 = min(rank * per, a.kbs), total = min(k0 + per, a.kbs) - k0;
  const uint32_t slots = REC ? S : min(S, (a.kbs + 7) / 8);
  const uint32_t item0 = REC ? 0 : blockIdx.x, item_step = REC ? 1 : gridDim.x;
  const uint32_t block0 = REC ? blockIdx.y * a.ncb : 0, nblocks = REC ? min(a.ncb, a.tiles_n - block0) : 1;   // this CTA's column blocks

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (uint32_t q = 0; q < kBufs; ++q) { mbar_init(&acc_full[q], 1); mbar_init(&acc_empty[q], kEpiWarps); }
    mbar_init(&park_full, 1); mbar_init(&park_free, S);   // the bytes of a pass, 64 columns, whoever sends them / an arrival per CTA
    for (int q = 0; q < kMaxBlocks; ++q) mbar_init(&go[q], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (S > 1) mbar_expect_tx(&park_full, kParkBytes);
  }
  if (threadIdx.x == 32 * 2) {
#pragma unroll
    for (int q = 0; q < 4; ++q) asm volatile("prefetch.tensormap [%0];" ::"l"(&tm.t[q]) : "memory");
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
      // TMA producer: rows [m0, + 128) of the weights, rows [col0, + BNT) of the pairs of dgates
      uint32_t s = 0, ph = 0;
      bool fail = false;
      const uint32_t per_step = gridDim.x * S;   // REC: arrivals per column block and step
      for (uint32_t it = item0; it < a.P && !fail; it += item_step)
      for (uint32_t cb = 0; cb < nblocks && !fail; ++cb) {
        const int m0 = (int)(REC ? blockIdx.x * BM : it % a.tiles_m * BM);
        const int col0 = (int)(REC ? (a.T - 1 - it) * a.B + (block0 + cb) * BNT : it / a.tiles_m * BNT);
        uint32_t i = 0;
        if (REC) {
          // The weights of the first k-blocks do not depend on the cell pass and are requested as their stages become free; the pairs of dgates follow
          // as soon as the counter says so, with more column blocks than one before all of those stages are free.
          const uint32_t pre = min((uint32_t)kStages, total), want = a.T > 1 ? (it + 1) * per_step : 0;
          uint32_t sa = s, pa = ph, na = 0;   // next stage for weights, its phase, weights requested so far
          bool ready = false;
          for (uint32_t poll = 0; !fail && (!ready || i < pre); ++poll) {
            if (poll == kPollLimit) fail = true;
            if (!ready && peek_counter(a.done + block0 + cb) >= want) {
              ready = true;
              mbar_arrive(&go[cb]);                                       // (the scale words may be read)
              asm volatile("fence.proxy.async.global;" ::: "memory");     // generic-proxy stores of other CTAs -> this CTA's TMA reads
            }
            if (na < pre && mbar_test(&empty_bar[sa], pa ^ 1)) {
              unsigned char* st = ring + (size_t)sa * kStageBytes;
              const KBlock kb = k_block(k0 + na, a.H, a.Ha, a.Hp);
              mbar_expect_tx(&full_bar[sa], kStageBytes);
              tma_load_2d(st, &tm.t[0], &full_bar[sa], kb.xa, m0);
              tma_load_2d(st + TILE_BYTES, &tm.t[1], &full_bar[sa], kb.xa, m0);
              if (++sa == kStages) { sa = 0; pa ^= 1; }
              ++na;
            }
            if (ready && i < na) {
              unsigned char* st = ring + (size_t)s * kStageBytes;
              const KBlock kb = k_block(k0 + i, a.H, a.Ha, a.Hp);
              tma_load_2d(st + 2 * TILE_BYTES, &tm.t[2], &full_bar[s], kb.xb, col0);
              tma_load_2d(st + 2 * TILE_BYTES + TILE_B_BYTES, &tm.t[3], &full_bar[s], kb.xb, col0);
              if (++s == kStages) { s = 0; ph ^= 1; }
              ++i;
            }
          }
          if (fail) break;
        }
        for (; i < total; ++i) {
          if (!mbar_wait(&empty_bar[s], ph ^ 1, kLongWait)) { fail = true; break; }
          unsigned char* st = ring + (size_t)s * kStageBytes;
          const KBlock kb = k_block(k0 + i, a.H, a.Ha, a.Hp);
          mbar_expect_tx(&full_bar[s], kStageBytes);
          tma_load_2d(st, &tm.t[0], &full_bar[s], kb.xa, m0);
          tma_load_2d(st + TILE_BYTES, &tm.t[1], &full_bar[s], kb.xa, m0);
          tma_load_2d(st + 2 * TILE_BYTES, &tm.t[2], &full_bar[s], kb.xb, col0);
          tma_load_2d(st + 2 * TILE_BYTES + TILE_B_BYTES, &tm.t[3], &full_bar[s], kb.xb, col0);
          if (++s == kStages) { s = 0; ph ^= 1; }
        }
      }
      if (fail) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = (1u << 4) | ((uint32_t)(BNT >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      const uint32_t idesc_wide = idesc + ((uint32_t)(BNT >> 3) << 17);
      uint64_t d_a_hi[kStages], d_a_lo[kStages], d_b[kStages];
#pragma unroll
      for (int q = 0; q < kStages; ++q) {
        const uint32_t base = smem_u32(ring + (size_t)q * kStageBytes);
        d_a_hi[q] = umma_desc(base); d_a_lo[q] = umma_desc(base + TILE_BYTES); d_b[q] = umma_desc(base + 2 * TILE_BYTES);
      }
      // stage, phase and chain counters run on across products; a chain ends with its block of units, or with this CTA's share
      uint32_t s = 0, ph = 0, chain = 0, buf = 0;
      bool fail = false;
      for (uint32_t it = item0; it < a.P && !fail; it += item_step)
      for (uint32_t cb = 0; cb < nblocks && !fail; ++cb) {
        uint32_t in_chain = 0;
        for (uint32_t i = 0; i < total; ++i) {
          if (in_chain == 0 && chain >= kBufs) {
            if (!mbar_wait(&acc_empty[buf], ((chain / kBufs) - 1) & 1, kLongWait)) { fail = true; break; }
          }
          if (!mbar_wait(&full_bar[s], ph, kLongWait)) { fail = true; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          uint64_t a_hi, a_lo, b;   // select without dynamic register indexing
          if (s == 0) { a_hi = d_a_hi[0]; a_lo = d_a_lo[0]; b = d_b[0]; }
          else if (s == 1) { a_hi = d_a_hi[1]; a_lo = d_a_lo[1]; b = d_b[1]; }
          else if (s == 2 || kStages == 3) { a_hi = d_a_hi[2]; a_lo = d_a_lo[2]; b = d_b[2]; }
          else { a_hi = d_a_hi[kStages - 1]; a_lo = d_a_lo[kStages - 1]; b = d_b[kStages - 1]; }
          issue_kblock_f16(tmem_base + buf * kAccCols, tmem_base + buf * kAccCols + BNT, a_hi, a_lo, b, idesc_wide, idesc, in_chain, 2, 2);
          umma_commit(&empty_bar[s]);
          if (((k0 + i) & 7) == 7 || i == total - 1) { umma_commit(&acc_full[buf]); in_chain = 0; ++chain; buf = chain % kBufs; }
          else ++in_chain;
          if (++s == kStages) { s = 0; ph ^= 1; }
        }
      }
      if (fail) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
    }
  } else {
    // epilogue warps 2..9: TMEM lanes 32 (warp % 4) .. + 31; warps 2 - 5 drain the tile's first BNT / 2 columns, warps 6 - 9 the others
    const uint32_t quarter = warp & 3, half = (warp - 2) >> 2, row = quarter * 32 + lane;
    const uint32_t te = threadIdx.x - 64, ew = te >> 5;
    const uint32_t nchains = total ? ((k0 + total - 1) >> 3) - (k0 >> 3) + 1 : 0;
    // The exchange goes in passes of 64 columns: pass hh takes columns [32 hh, + 32) of either half, position p of a pass being column p % 32 of the
    // half p / 32.  Rank r finishes the positions [r w, + w); sender s's partial sums of them lie in slot s of r's buffer.
    constexpr uint32_t w = 64 / S, KC = w / 8, GB = KC < 2 ? KC : REC ? 2 : KC < 4 ? KC : 4;   // a warp holds one column: 8 columns of a slice at a time, GB of them in flight
    const uint32_t uq = 4 * (te & 31);                                  // this thread's four rows of the tile
    uint32_t cg = 0, pf_phase = 0, pr_phase = 0;
    bool ok = true;   // the same for all 256 threads after every bar_and below
    const size_t HB = (size_t)a.H * a.B;
    const uint32_t u = blockIdx.x * BM + uq;                            // REC: units [u, u + 4)
    const bool own_u = u < a.H;
    const uint32_t left = a.H - u;                                      // (own_u) units from u on
    const CellUnits un{blockIdx.x, u, left, own_u};
    float4 rs[4];   // REC: row sums of dgates over this thread's columns of a step

    auto column = [&](int hh, uint32_t k) { const uint32_t p = rank * w + ew + 8 * k; return (p >> 5) * kHalf + 32 * hh + (p & 31); };
    auto publish = [&](uint32_t cb) {   // (behind a barrier: one thread's release orders all the stores it has observed, for both proxies)
      if (te == 0) {
        asm volatile("fence.proxy.async.global;" ::: "memory");
        signal_counter(a.done + block0 + cb);
      }
    };
    auto clear_sums = [&]() {
#pragma unroll
      for (int q = 0; q < 4; ++q) rs[q] = make_float4(0.f, 0.f, 0.f, 0.f);
    };

    bool planes = false;   // small quads among the weights: the others look into the planes of every column
    if (REC && a.T > 1) {
      for (uint32_t k = te; k < a.M; k += 256) planes = planes || (__ldg(a.wscale + k) & 1);
      planes = !bar_and(1, 256, !planes);
    }
    for (uint32_t cb = 0; REC && a.T > 1 && cb < nblocks; ++cb) {   // the cell pass of the last step (of a single one: k_bwd_cells)
      const uint32_t t = a.T - 1, n0 = (block0 + cb) * BNT;
      clear_sums();
#pragma unroll 1
      for (int hh = 0; hh < BNT / 64; ++hh)
#pragma unroll 1
        for (uint32_t k = 0; k < KC; ++k) {
          const uint32_t n = n0 + column(hh, k);
          if (n >= a.B) continue;
          CellIn in = {};
          float4 dh = make_float4(0.f, 0.f, 0.f, 0.f), p[4];
          if (own_u) { cell_load<VEC>(a, un, in, t, n); dh = ldu<VEC>(a.dh + (size_t)t * HB + (size_t)n * a.H + u, left); }
          const uint32_t word = cell(a, un, in, dh, t, n, p, rs);
          if (word) cell_small<VEC>(a, un, p[0], p[1], p[2], p[3], t, n, word);
          cell_rest<VEC>(a, un, in, p, t, n);
        }
      row_sums(a, rs, park, part_of(a, 0, block0 + cb, S, rank), blockIdx.x, te, ew, uq, ok);
    }
    if (REC && a.T > 1)   // (all blocks at the end: the exchange buffer belongs to the others from the first one on)
      for (uint32_t cb = 0; cb < nblocks; ++cb) publish(cb);

    auto rows_of = [&](uint32_t m) {   // whether there are small quads among the weights of rows [m, + 4)
      uint32_t w = 0;
#pragma unroll
      for (uint32_t q = 0; q < 4; ++q) w |= m + q < a.M ? __ldg(a.wscale + m + q) : 0u;
      return w & 1;
    };
    uint32_t small_rows = REC ? rows_of(u) : 0u;
    float row_f = REC ? inv_scale_of(blockIdx.x * BM + row < a.M ? __ldg(a.wscale + blockIdx.x * BM + row) : 0x3f800000u) : 1.f;
#pragma unroll 1
    for (uint32_t it = item0; it < a.P; it += item_step)
#pragma unroll 1
    for (uint32_t cb = 0; cb < nblocks; ++cb) {
      const uint32_t n0 = REC ? (block0 + cb) * BNT : 0;
      const uint32_t m0 = REC ? blockIdx.x * BM : it % a.tiles_m * BM;
      const uint32_t t = REC ? a.T - 1 - it : 0;                           // REC: dgates of step t -> dE/dh of step t - 1
      const uint32_t col0 = REC ? n0 : it / a.tiles_m * BNT, cols = REC ? a.B : a.columns;   // first column of the tile and their end
      const uint32_t seq0 = REC ? t * a.B : 0;                             // ... as columns of the sequence
      float* const dst = REC ? (t ? a.dh + (size_t)(t - 1) * HB : a.dh_prev) : a.dx;
      const uint32_t m = m0 + uq;
      const bool own = m < a.M, vec = REC || ((a.M & 3) == 0 && aligned16(a.dx) && aligned16(a.mask));
      if (!REC) small_rows = rows_of(m);
      if (!REC) row_f = inv_scale_of(m0 + row < a.M ? __ldg(a.wscale + m0 + row) : 0x3f800000u);
      if (REC && t) {   // what the cell pass will read from HBM is asked for now (a request per 128-byte line)
        if (own_u && (te & 7) == 0) {
#pragma unroll
          for (int hh = 0; hh < BNT / 64; ++hh)
#pragma unroll
            for (uint32_t k = 0; k < KC; ++k) {
              const uint32_t n = n0 + column(hh, k);
              if (n >= a.B) continue;
              const size_t e = (size_t)n * a.H + u;
              const float* g = a.gates + (size_t)(t - 1) * 4 * HB + (size_t)n * 4 * a.H + u;
              const float* ps[7] = {g, g + a.H, g + 2 * a.H, g + 3 * a.H, (t > 1 ? a.cs + (size_t)(t - 2) * HB : a.c0) + e, dst + e, t > 1 && !a.fresh_dc ? a.dc + (size_t)(t - 2) * HB + e : dst + e};
#pragma unroll
              for (int q = 0; q < 7; ++q) asm volatile("prefetch.global.L2 [%0];" ::"l"(ps[q]));
            }
        }
      }
      if (!REC && own && !a.fresh_dx && (te & 7) == 0)   // (the values that this tile adds to)
#pragma unroll
        for (int hh = 0; hh < BNT / 64; ++hh)
#pragma unroll
          for (uint32_t k = 0; k < KC; ++k) {
            const uint32_t n = col0 + column(hh, k);
            if (n < cols) asm volatile("prefetch.global.L2 [%0];" ::"l"(dst + (size_t)n * a.M + m));
          }
      // ---- drain the chains of this product ----
      float sum[kHalf];
#pragma unroll
      for (uint32_t q = 0; q < kHalf; ++q) sum[q] = 0.f;
      // (a share without k-blocks waits too: once the counter is up, the others are done with their exchange buffers as scratch for row sums)
      if (REC && ok && !mbar_wait(&go[cb], it & 1, kLongWait)) ok = false;
      // (the words of the columns that this warp finishes: looked at once the partial sums are on their way)
      uint32_t words[KC * BNT / 64];
#pragma unroll
      for (uint32_t k = 0; k < KC * BNT / 64; ++k) {
        const uint32_t n = col0 + column(k / KC, k % KC);
        words[k] = ok && n < cols && lane * BM < a.H ? __ldcg(a.dsc + (size_t)lane * a.dsc_ld + seq0 + n) : 0u;
        if (a.H > 32 * BM && ok && n < cols) for (uint32_t b = lane + 32; b * BM < a.H; b += 32) words[k] |= __ldcg(a.dsc + (size_t)b * a.dsc_ld + seq0 + n);
      }
#pragma unroll 1
      for (uint32_t c = 0; c < nchains; ++c, ++cg) {
        const uint32_t buf = cg % kBufs;
        if (!ok) continue;
        float f[BNT / 64];   // 2^-s of the columns lane (and lane + 32) of this warp's half, and of its row
#pragma unroll
        for (int k = 0; k < BNT / 64; ++k) {
          const uint32_t n = col0 + half * kHalf + 32 * k + lane;
          f[k] = inv_scale_of(n < cols ? __ldcg(a.dsc + (size_t)((k0 >> 3) + c) * a.dsc_ld + seq0 + n) : 0x3f800000u);
        }
        if (!mbar_wait(&acc_full[buf], (cg / kBufs) & 1, kLongWait)) { ok = false; continue; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t taddr = tmem_base + buf * kAccCols + ((quarter * 32) << 16) + half * kHalf;
#pragma unroll
        for (uint32_t p = 0; p < kHalf / 16; ++p) {   // (16 columns of both accumulators at a time)
          float v1[16], v2[16];
          tmem_ld16x2(taddr + 16 * p, taddr + BNT + 16 * p, v1, v2);
#pragma unroll
          for (int q = 0; q < 16; ++q)
            // (both factors at once: the sum times one of them may leave fp32's range where the product does not; rounded before it is added, as where
            // another CTA adds it)
            sum[16 * p + q] = __fadd_rn(sum[16 * p + q], __fmul_rn(__fmaf_rn(v2[q], kLoScale, v1[q]), row_f * __shfl_sync(0xffffffffu, f[p / 2], 16 * (p % 2) + q)));
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);
      }
      if (REC) clear_sums();
#pragma unroll
      for (int hh = 0; hh < BNT / 64; ++hh) {
        uint32_t any = small_rows;
#pragma unroll
        for (uint32_t k = 0; k < KC; ++k) any |= words[KC * hh + k];
        const bool quads = __any_sync(0xffffffffu, any & 1);
        // ---- partial sums to the ranks that finish them ----
        if (S > 1 && ok && !mbar_wait_cluster(&park_free, pr_phase ^ 1, kLongWait)) ok = false;
        if (S > 1) {
#pragma unroll
          for (uint32_t rr = 0; rr < S / 2; ++rr) {
            const uint32_t to = mapa_u32(smem_u32(park), half * (S / 2) + rr) + 4u * (rank * w * BM), bar = mapa_u32(smem_u32(&park_full), half * (S / 2) + rr);
#pragma unroll
            for (uint32_t q = 0; q < w; q += 4)   // column q + lane % 4, rows of the lane's quad
              send4(to + 4u * park_at(q + (lane & 3), row >> 2), transpose4(sum + (32 * hh + rr * w + q) % kHalf, lane), bar);
          }
        } else {
#pragma unroll
          for (uint32_t q = 0; q < 32; ++q) park[park_at(32 * half + q, row >> 2) + (row & 3)] = sum[32 * hh + q];
        }
        const bool last_pass = hh == BNT / 64 - 1;
        if (quads) {   // ---- the products of small quads, into what these columns are added to ----
#pragma unroll 1
          for (uint32_t k = 0; k < KC; ++k) {
            const uint32_t n = col0 + column(hh, k);
            if (n >= cols || !ok) continue;   // (the same for a whole warp)
            const float4 x = small_parts(a, seq0 + n, m);
            for (uint32_t q = 0; q < 4 && m + q < a.M; ++q) {
              float* d = dst + (size_t)n * a.M + m + q;
              *d = __fmaf_rn((&x.x)[q], a.mask ? a.mask[m + q + (a.mask_full ? (size_t)(REC ? n : n % a.B) * a.M : 0)] : 1.f, !REC && a.fresh_dx ? 0.f : __ldcg(d));
            }
          }
        }
#pragma unroll 1
        for (uint32_t kb = 0; kb < KC; kb += GB) {
          CellIn in[GB];
          float4 old[GB], mk[GB], p[GB][4];
          uint32_t n[GB], word[GB];
#pragma unroll
          for (uint32_t g = 0; g < GB; ++g) {   // everything that comes from memory, before the wait
            n[g] = col0 + column(hh, kb + g);
            in[g] = CellIn{};
            word[g] = 0;
            mk[g] = make_float4(1.f, 1.f, 1.f, 1.f);
            old[g] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!own || n[g] >= cols || !vec) continue;
            if (REC || !a.fresh_dx || quads) old[g] = REC ? ldu_cg<VEC>(dst + (size_t)n[g] * a.M + m, left) : __ldcg(reinterpret_cast<const float4*>(dst + (size_t)n[g] * a.M + m));
            if (a.mask) {
              const float* mp = a.mask + m + (a.mask_full ? (size_t)(REC ? n[g] : n[g] % a.B) * a.M : 0);
              mk[g] = REC ? ldu<VEC>(mp, left) : ld4(mp);
            }
            if (REC && t) cell_load<VEC>(a, un, in[g], t - 1, n[g]);
          }
          if (kb == 0) {
            const bool got = S > 1 ? mbar_wait_cluster(&park_full, pf_phase, kLongWait) : true;
            ok = bar_and(1, 256, ok && got) != 0;
            pf_phase ^= 1; pr_phase ^= 1;
            if (S > 1 && te == 0) mbar_expect_tx(&park_full, kParkBytes);   // (the next pass; it begins when this CTA has arrived on the others' park_free)
          }
#pragma unroll
          for (uint32_t g = 0; g < GB; ++g) {
            if (n[g] >= cols) continue;   // (the same for a whole warp)
            const float* col = park + park_at(ew + 8 * (kb + g), te & 31);
            float4 v = ld4(col);
#pragma unroll
            for (uint32_t r = 1; r < S; ++r)
              if (REC || r < slots) { const float4 x = ld4(col + (size_t)r * w * BM); v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w; }
            if (vec) {
              if (a.mask) v = make_float4(__fmaf_rn(v.x, mk[g].x, old[g].x), __fmaf_rn(v.y, mk[g].y, old[g].y), __fmaf_rn(v.z, mk[g].z, old[g].z), __fmaf_rn(v.w, mk[g].w, old[g].w));
              else v = make_float4(v.x + old[g].x, v.y + old[g].y, v.z + old[g].z, v.w + old[g].w);
            }
            old[g] = v;
            if (REC && t && ok) word[g] = cell(a, un, in[g], v, t - 1, n[g], p[g], rs);
            if (vec || !own || !ok) continue;
            for (uint32_t q = 0; q < 4 && m + q < a.M; ++q) {
              float* d = dst + (size_t)n[g] * a.M + m + q;
              *d = __fmaf_rn((&v.x)[q], a.mask ? a.mask[m + q + (a.mask_full ? (size_t)(n[g] % a.B) * a.M : 0)] : 1.f, !REC && a.fresh_dx && !quads ? 0.f : *d);
            }
          }
          if (REC && t && ok) {
#pragma unroll
            for (uint32_t g = 0; g < GB; ++g)
              if ((word[g] || planes) && n[g] < cols) cell_small<VEC>(a, un, p[g][0], p[g][1], p[g][2], p[g][3], t - 1, n[g], word[g]);
          }
          if (REC && t && last_pass && kb + GB >= KC) {
            bar_sync(1, 256);   // all stores of the pairs and their words are issued; what nobody waits for goes out behind them
            publish(cb);
          }
          if (!ok) continue;
#pragma unroll
          for (uint32_t g = 0; g < GB; ++g) {
            if (n[g] >= cols) continue;
            if (own && vec) { if (REC) stu<VEC>(dst + (size_t)n[g] * a.M + m, old[g], left); else st4(dst + (size_t)n[g] * a.M + m, old[g]); }
            if (REC && t) cell_rest<VEC>(a, un, in[g], p[g], t - 1, n[g]);
          }
        }
        if (REC && t && last_pass) row_sums(a, rs, park, part_of(a, it + 1, block0 + cb, S, rank), blockIdx.x, te, ew, uq, ok);
        else bar_sync(1, 256);    // every read of the exchange buffer is done
        if (S > 1 && te < S) mbar_arrive_remote(&park_free, te);
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

// ---- host side ---------------------------------------------------------------------------------------------------------
enum WideOp { WIDE_FIT, WIDE_LAUNCH };

template <int BNT, uint32_t S, bool REC, bool VEC = true>
int wide_do(WideOp op, dyb200_ctx* ctx, int slot, const TmapPack* tm, const BwdWide* a, dim3 grid, double flops) {
  const auto kernel = k_bwd_wide<BNT, S, REC, VEC>;
  int16_t& fit = ctx->bwd_wide_fit[slot];
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = op == WIDE_FIT ? dim3(1, 1, S) : grid; cfg.blockDim = dim3(kThreads, 1, 1); cfg.dynamicSmemBytes = SMEM_SEQ_BYTES; cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[2];
  int na = 0;
  if (S > 1) {
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = 1; attr[na].val.clusterDim.y = 1; attr[na].val.clusterDim.z = S;
    ++na;
  }
  cfg.attrs = attr; cfg.numAttrs = na;
  if (op == WIDE_FIT) {   // clusters (S = 1: CTAs) that fit on the GPU at once; the kernel's shared-memory limit is raised with the first question
    if (fit == 0) {
      int n = ctx->sm_count;   // (225 KB of shared memory: one CTA per SM)
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_SEQ_BYTES) != cudaSuccess ||
          (S > 1 && cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess)) { (void)cudaGetLastError(); n = -1; }
      fit = (int16_t)(n > 0 ? n : -1);
    }
    return fit;
  }
  GemmProfScope scope(ctx, flops, 2, a->M, REC ? a->B * a->T : a->columns, 4 * a->H, EPI_ACCUM_MASK);
  if (REC && a->T > 1 && ctx->seq_coop >= 0) {
    // all CTAs wait on one another (a single step's for none beside those of their cluster): as many as fit at once (the plan), scheduled as one gang where the driver takes the attribute
    attr[na].id = cudaLaunchAttributeCooperative;
    attr[na].val.cooperative = 1;
    cfg.numAttrs = na + 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, *tm, *a);
    if (e == cudaSuccess) { ctx->seq_coop = 1; ctx->launches++; return DYB200_OK; }
    (void)cudaGetLastError();
    if (ctx->seq_coop == 1) return dyb200_fail(ctx, DYB200_ECUDA, "backward recurrence: launch failed: %s", cudaGetErrorString(e));
    ctx->seq_coop = -1;
    cfg.numAttrs = na;
  }
  if (a->T == 1 && ctx->pdl) {   // (a single step's kernels are short: each one's prologue runs beside the one before)
    attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[na].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = na + 1;
  }
  cudaLaunchKernelEx(&cfg, kernel, *tm, *a);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}
constexpr uint32_t kRecCols = 64;
template <bool VEC>
int wide_rec_of(WideOp op, uint32_t S, dyb200_ctx* ctx, const TmapPack* tm, const BwdWide* a, dim3 grid, double flops) {
  constexpr int slot = VEC ? 0 : 7;
  if (S == 8) return wide_do<kRecCols, 8, true, VEC>(op, ctx, slot, tm, a, grid, flops);
  if (S == 4) return wide_do<kRecCols, 4, true, VEC>(op, ctx, slot + 1, tm, a, grid, flops);
  if (S == 2) return wide_do<kRecCols, 2, true, VEC>(op, ctx, slot + 2, tm, a, grid, flops);
  return wide_do<kRecCols, 1, true, VEC>(op, ctx, slot + 3, tm, a, grid, flops);
}
int wide_rec(WideOp op, uint32_t H, uint32_t S, dyb200_ctx* ctx, const TmapPack* tm = nullptr, const BwdWide* a = nullptr, dim3 grid = dim3(), double flops = 0) {
  return H % 4 == 0 ? wide_rec_of<true>(op, S, ctx, tm, a, grid, flops) : wide_rec_of<false>(op, S, ctx, tm, a, grid, flops);
}
enum DxForm { DX_128, DX_64, DX_SPLIT };   // tiles of 128 or 64 columns, a CTA each; tiles of 64 columns, a CTA of eight for each block of 128 units
int wide_dx(WideOp op, DxForm f, dyb200_ctx* ctx, const TmapPack* tm = nullptr, const BwdWide* a = nullptr, dim3 grid = dim3(), double flops = 0) {
  if (f == DX_128) return wide_do<128, 1, false>(op, ctx, 4, tm, a, grid, flops);
  if (f == DX_64) return wide_do<64, 1, false>(op, ctx, 5, tm, a, grid, flops);
  return wide_do<64, 8, false>(op, ctx, 6, tm, a, grid, flops);
}
uint32_t k_blocks(uint32_t H) { return 8 * (H / BM) + (H % BM == 0 ? 0 : H % BM <= 64 ? 4 : 8); }

}  // namespace

// Column blocks per CTA and K splits: the fastest by what a product was measured to take - 0.36 us per k-block on the tensor pipe and 6 us from its last
// MMA to the next step's first, which another block's MMAs overlap (both from 1024 units).  The rule's edges, us per step, the forms before / this one: (64, 385, 9)
// 37.8 / 8.2, (512, 385, 9) 20.3 / 8.2, (512, 416, 64) 21.2 / 7.4, (512, 448, 512) 26.6 / 13.1, (512, 777, 500) 81.5 / 31.7, (64, 1024, 1024) 58.5 / 49.9, (64, 2048, 1000) 164 / 127,
// (64, 4096, 64) 107 / 78, (64, 4096, 500) 272 / 216; two steps with the weights' pairs made for them: (512, 512, 64) 24.4 / 23.7, (512, 385, 40) 33.0 / 27.1.
bool dyb200_bwd_wide_plan(dyb200_ctx* ctx, uint32_t H, uint32_t B, uint32_t* ncb, uint32_t* S) {
  if (H <= 384 || B <= 8 || (H % 8 != 0 && 4 * H > kF16PadMax)) return false;
  const uint32_t tiles_m = (H + BM - 1) / BM, tiles_n = (B + kRecCols - 1) / kRecCols, kbs = k_blocks(H);
  if (tiles_n > DYB200_DEV_BWD_WORDS) return false;   // (a hand-over counter per column block)
  struct { double t; uint32_t n, s; } c[12];
  int nc = 0;
  for (uint32_t n = 1; n <= kMaxBlocks && n <= tiles_n; n *= 2)
    for (uint32_t s = 8; s >= 1; s /= 2) {
      if (tiles_m * ((tiles_n + n - 1) / n) * s > (uint32_t)ctx->sm_count) continue;
      const double mma = (kbs + s - 1) / s * 0.36;
      c[nc].t = n == 1 ? mma + 6.0 : n * (mma > 6.0 ? mma : 6.0) + 1.5; c[nc].n = n; c[nc].s = s;
      ++nc;
    }
  while (nc > 0) {   // (the best one first: asking how many clusters fit loads the kernel, a few ms each)
    int k = 0;
    for (int q = 1; q < nc; ++q) if (c[q].t < c[k].t) k = q;
    const int fit = wide_rec(WIDE_FIT, H, c[k].s, ctx);
    if (fit > 0 && tiles_m * ((tiles_n + c[k].n - 1) / c[k].n) <= (uint32_t)fit) { *ncb = c[k].n; *S = c[k].s; return true; }
    c[k] = c[--nc];
  }
  return false;
}

int dyb200_bwd_wide(dyb200_ctx* ctx, const BwdWideCall& q) {
  const uint32_t H = q.H, I = q.I, B = q.B, T = q.T, G = 4 * H, Hp = (H + 63) / 64 * 64, tiles_m = (H + BM - 1) / BM, columns = T * B;
  uint32_t ncb, S;
  DYB_CHECK_ARG(ctx, dyb200_bwd_wide_plan(ctx, H, B, &ncb, &S), "lstm_seq_bwd: shape %u, %u x %u", I, H, B);
  const uint32_t tiles_n = (B + kRecCols - 1) / kRecCols;
  F16Job wh, wx;
  int rc;
  void *p16, *words, *part;
  const size_t plane = (size_t)columns * 4 * Hp;
  if ((rc = dyb200_scratch(ctx, 2 * plane * sizeof(__half), &p16)) || (rc = dyb200_scratch(ctx, (size_t)tiles_m * columns * sizeof(uint32_t), &words)) ||
      (rc = dyb200_scratch(ctx, (size_t)T * tiles_n * S * G * sizeof(float), &part))) return rc;
  // (a k-block's copy starts at a gate's units: on 16 bytes as the weights lie, or with the gates moved apart)
  const uint32_t pad = H % 8 == 0 ? 0 : H, K = pad ? 4 * Hp : G;
  if ((rc = dyb200_f16_param(ctx, q.Wh, G, H, G, F16_LINE, &wh, pad, 1))) return rc;
  if (q.dx && (rc = dyb200_f16_param(ctx, q.Wx, G, I, G, F16_LINE, &wx, pad, 1))) return rc;
  BwdWide a;
  memset(&a, 0, sizeof(a));
  a.T = T; a.B = B; a.H = H; a.Hp = Hp; a.Ha = pad ? Hp : H; a.kbs = k_blocks(H); a.P = T - 1 + (q.dh_prev ? 1 : 0); a.M = H; a.tiles_m = tiles_m;
  a.ncb = ncb; a.tiles_n = tiles_n;
  a.gates = q.gates; a.cs = q.c; a.c0 = q.c0; a.dh = q.dh; a.dc = q.dc; a.dh_prev = q.dh_prev; a.dc_prev = q.dc_prev;
  a.dn_hi = q.dn_hi; a.dn_lo = q.dn_lo; a.dn_pitch = q.dn_pitch;
  a.d16_hi = (__half*)p16; a.d16_lo = a.d16_hi + plane;
  a.dsc = (uint32_t*)words; a.dsc_ld = columns; a.W = q.Wh; a.wscale = wh.scale; a.part = (float*)part;
  a.mask = q.mh; a.mask_full = q.mh_full; a.fresh_dx = q.fresh_dx; a.fresh_dc = q.fresh_dc;
  a.done = ctx->dev_flags + DYB200_DEV_BWD0; a.flags = ctx->dev_flags;
  TmapPack tm;
  memset(&tm, 0, sizeof(tm));
  if ((rc = dyb200_tc_make_tmap_f16(ctx, &tm.t[0], wh.hi, H, K, wh.pitch, BM, false)) || (rc = dyb200_tc_make_tmap_f16(ctx, &tm.t[1], wh.lo, H, K, wh.pitch, BM, false)) ||
      (rc = dyb200_tc_make_tmap_f16(ctx, &tm.t[2], a.d16_hi, columns, 4 * Hp, 4 * Hp, kRecCols, false)) ||
      (rc = dyb200_tc_make_tmap_f16(ctx, &tm.t[3], a.d16_lo, columns, 4 * Hp, 4 * Hp, kRecCols, false))) return rc;
  const dim3 grid(tiles_m, (tiles_n + ncb - 1) / ncb, S);
  // A single step's cell pass is a launch of its own, and the product behind it polls no counter: a step's call depends on no CTA beside those of its
  // cluster being on the GPU with it.  The bits are those of the sequence.  (us, a gang that does both and hands over through counters / so, each kernel's
  // prologue beside the one before: 512 x 1024 x 64 columns 26.5 / 24.3, 512 x 512 x 64 24.5 / 19.7, 1024 x 1024 x 512 66.5 / 66.3.  As two launches of the
  // recurrence kernel one after the other: 30.4, 29.5, 72.9.)
  if (T == 1) {
    dyb_launch(H % 4 == 0 ? k_bwd_cells<true> : k_bwd_cells<false>, dim3(tiles_m, tiles_n, S), 256, 0, ctx, a);
    DYB_LAUNCHED(ctx);
    if ((rc = dyb200_seq_db(ctx, a.part, 1, tiles_n * S, G, q.db, nullptr))) return rc;
  }
  if (a.P && (rc = wide_rec(WIDE_LAUNCH, H, S, ctx, &tm, &a, grid, 2.0 * G * (double)H * B * a.P))) return rc;
  if (T > 1 && (rc = dyb200_seq_db(ctx, a.part, T, tiles_n * S, G, q.db, a.done))) return rc;
  if (!q.dx) return DYB200_OK;
  // dx of all columns
  a.M = I; a.tiles_m = (I + BM - 1) / BM; a.columns = columns; a.dx = q.dx; a.mask = q.mx; a.mask_full = q.mx_full; a.W = q.Wx; a.wscale = wx.scale;
  // The form by what a round of tiles was measured to take.  All give the same bits, whatever the number of columns: chains are added in the order of
  // the blocks of units.  (1024 x 64 of a single step: 17 us with two CTAs per tile, 9 with
  // eight; 1024 x 17 920: 350 on 128-column tiles.)
  DxForm form = DX_128;
  double best = 0;
  for (const DxForm f : {DX_128, DX_64, DX_SPLIT}) {
    if (f == DX_SPLIT && a.kbs > 64) continue;
    const uint32_t n = f == DX_128 ? 128 : 64, tiles = a.tiles_m * ((columns + n - 1) / n), room = f == DX_SPLIT ? (uint32_t)ctx->sm_count / 10 + 1 : (uint32_t)ctx->sm_count;
    const double t = (tiles + room - 1) / room * (f == DX_128 ? a.kbs * 0.55 + 6.0 : f == DX_64 ? a.kbs * 0.36 + 4.0 : 8 * 0.36 + 4.5);
    if (best == 0 || t < best) { best = t; form = f; }
  }
  int fit = wide_dx(WIDE_FIT, form, ctx);
  if (fit <= 0 && form == DX_SPLIT) fit = wide_dx(WIDE_FIT, form = DX_64, ctx);
  if (fit <= 0) return dyb200_fail(ctx, DYB200_ECUDA, "lstm_seq_bwd: no launch of the dx product fits");
  const uint32_t dn = form == DX_128 ? 128 : 64;
  a.P = a.tiles_m * ((columns + dn - 1) / dn);
  if ((rc = dyb200_tc_make_tmap_f16(ctx, &tm.t[0], wx.hi, I, K, wx.pitch, BM, false)) || (rc = dyb200_tc_make_tmap_f16(ctx, &tm.t[1], wx.lo, I, K, wx.pitch, BM, false)) ||
      (rc = dyb200_tc_make_tmap_f16(ctx, &tm.t[2], a.d16_hi, columns, 4 * Hp, 4 * Hp, dn, false)) ||
      (rc = dyb200_tc_make_tmap_f16(ctx, &tm.t[3], a.d16_lo, columns, 4 * Hp, 4 * Hp, dn, false))) return rc;
  return wide_dx(WIDE_LAUNCH, form, ctx, &tm, &a, dim3(a.P < (uint32_t)fit ? a.P : (uint32_t)fit, 1, form == DX_SPLIT ? 8 : 1), 2.0 * G * (double)I * columns);
}

// Whether the backward pass of such a layer takes this form (1 or 0), and its column blocks per CTA and K splits.
extern "C" int dyb200i_bwd_wide_tiling(dyb200_ctx* ctx, uint32_t H, uint32_t B, uint32_t* blocks, uint32_t* splits) {
  return dyb200_bwd_wide_plan(ctx, H, B, blocks, splits) ? 1 : 0;
}
