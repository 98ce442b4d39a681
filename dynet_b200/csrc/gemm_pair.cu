// Large products on scaled fp16 pairs (gemm.cuh, "2 x 11 bits in fp16"), one 256 x 256 output tile per PAIR of SMs
// (tcgen05.mma.cta_group::2): CTA r of a cluster of two holds rows [128 r, +128) of the left operand's tile and columns [128 r, +128)
// of the right one's, the tensor cores of both SMs read both halves, and each CTA's tensor memory receives its own 128 rows x 256 columns.
//
// Why a pair: a 128 x 128 tile of fp16 pairs on one SM (gemm_tc.cu) moves 144 KB through shared memory per 64 k - 64 KB written by TMA,
// 80 KB read by the MMAs - which at 128 bytes per cycle is 1125 cycles for 768 cycles of MMAs: 444 TFLOP/s useful on 128 SMs where the
// tensor pipe alone would give 660.  Here a CTA moves 64 KB in and 96 KB out per 1536 cycles of MMAs, below the limit.
//
// Tensor memory: D1 = hi hi and D2 = hi lo + lo hi take 256 columns each, so nothing is left for a second pair of accumulators.
// What keeps the pipe busy while an accumulator is drained is the order of the MMAs.  D1's chain is cut every kChunkF16 k-blocks (the
// tensor core truncates when it adds): the last two k-blocks of a chunk issue their hi hi products first, D1 is handed over, and
// their eight hi lo / lo hi MMAs each (2048 cycles) run while the epilogue warps of both CTAs add D1 into registers.  D2 carries
// 2^-11 of the result and its truncation with it, so its chain runs through the whole reduction; it is drained at the end of a tile
// while the hi hi products of the next tile's first three k-blocks (all stages of the ring) run.
//
// Measured (useful TFLOP/s, this kernel against the one-SM tiles): 50000 x 4096 x 512 456 / 387, 50000 x 512 x 4096 460 / 355,
// 512 x 4096 x 50000 484 / 417, 10000 x 17920 x 1024 501 / 425, 1024 x 17920 x 10000 512 / 405, 4096 x 1024 x 17920 495 on 64 of the 74
// pairs (a third of cuBLAS's bf16 rate is 551): the MMAs of a k-block take 1.05 us.  What is left below that is partly filled last
// rounds and, where K is short, the drain between tiles.
//
// Roles per CTA (three groups of four warps): warp 0 loads this CTA's tiles (its arrivals go to the leader's barrier), warp 1 of the leader
// issues every MMA, warps 4-11 drain (128 columns of one row per thread) and write out through two 8 KB buffers per four warps: TMA
// stores, or TMA adds where the result is accumulated, so that 128 rows x 16 columns leave per instruction and no thread waits for the
// old values.  Destinations that TMA cannot address (leading dimension no multiple of 4, misaligned) are written from registers.
// Persistent: pair p takes work items p, p + pairs, ... (K splits as further items, added in split order by k_splitk_reduce).
#include "seq_dev.cuh"

namespace {

constexpr int kPairTile = 256;
constexpr uint32_t kPairHead = STAGES, kPairTail = 2;   // k-blocks whose hi hi products go first: at a tile's start, at a chunk's end
constexpr int kPairPiece = 16;                           // columns per staging buffer
constexpr int kPairThreads = 384;
// Registers: 168 per thread at launch (384 x 168 = 64512); the first group gives 112 of them up to the other two, 56 + 2 x 224 = 3 x 168.
// The epilogue keeps 128 sums per thread (at 168 it spilled 700 bytes).
constexpr int kPairRegsLow = 56, kPairRegsHigh = 224;
constexpr int kPairBuf = BM * kPairPiece;                // floats
constexpr int SMEM_PAIR_BYTES = SMEM_BYTES + 4 * kPairBuf * (int)sizeof(float);

struct PairArgs {
  uint32_t M, N, kb, tiles_m, tiles_n, gm, S;
  float* C; uint32_t ldc; const float* bias; int accumulate;   // (splits: C = the partial products, split z at columns z N)
  uint32_t* flags;
  const uint32_t* unless;   // a device word: where it is not zero there is nothing to do (null: always run)
};

// This CTA's tile, its bytes reported to the barrier of the leader (both CTAs' loads complete one phase of it).
__device__ __forceinline__ void pair_load(void* dst, const CUtensorMap* map, uint32_t bar, uint32_t kblk, uint32_t row0, uint32_t mn) {
  if (mn)
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
                 "l"(map), "r"(bar), "r"(0), "r"((int)(kblk * 64)), "r"((int)(row0 / 64))
                 : "memory");
  else
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
                 "l"(map), "r"(bar), "r"((int)(kblk * 64)), "r"((int)row0)
                 : "memory");
}
// Arrival on the barrier of both CTAs once every MMA issued so far has completed.
__device__ __forceinline__ void pair_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
// d (+)= a b over one 64-wide k-block: four k steps, 256 x 256 x 16 each.
__device__ __forceinline__ void pair_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, uint64_t a_step, uint64_t b_step) {
  asm volatile(
      "{\n\t.reg .pred pf, pt;\n\t.reg .b64 xa, xb;\n\t"
      "setp.ne.b32 pf, %4, 0;\n\tsetp.eq.b32 pt, 0, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, pf;\n\t"
      "add.s64 xa, %1, %5;\n\tadd.s64 xb, %2, %6;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], xa, xb, %3, pt;\n\t"
      "add.s64 xa, xa, %5;\n\tadd.s64 xb, xb, %6;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], xa, xb, %3, pt;\n\t"
      "add.s64 xa, xa, %5;\n\tadd.s64 xb, xb, %6;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], xa, xb, %3, pt;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "l"(a_step), "l"(b_step)
      : "memory");
}

struct PairItem { uint32_t m0, n0, z, b0, nkb; };
// Work item w: split-major, so that the pairs of a round share k-blocks; within a split groups of gm tile rows, row fastest (the tiles in
// flight then share their operands in L2).
__device__ __forceinline__ PairItem pair_item(const PairArgs& a, uint32_t w) {
  PairItem it;
  const uint32_t tiles = a.tiles_m * a.tiles_n, per_group = a.gm * a.tiles_n;
  it.z = w / tiles;
  const uint32_t t = w - it.z * tiles, g = t / per_group, r = t - g * per_group, rows = min(a.gm, a.tiles_m - g * a.gm);
  it.n0 = (r / rows) * kPairTile;
  it.m0 = (g * a.gm + r % rows) * kPairTile;
  const KSplit ks = k_split(a.kb, 0, it.z, a.S);
  it.b0 = ks.b0; it.nkb = ks.n0;
  return it;
}

__device__ __forceinline__ void pair_producer(const TmapPack* tm, const PairArgs* a, unsigned char* ring, uint64_t* full_bar, uint64_t* empty_bar, uint32_t rank) {
  uint32_t s = 0, ph = 0;
  const uint32_t items = a->tiles_m * a->tiles_n * a->S, pairs = gridDim.x >> 1;
  uint32_t lead[STAGES];   // the leader's barriers
#pragma unroll
  for (int q = 0; q < STAGES; ++q) asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(lead[q]) : "r"(smem_u32(&full_bar[q])));
  for (uint32_t w = blockIdx.x >> 1; w < items; w += pairs) {
    const PairItem it = pair_item(*a, w);
    for (uint32_t k = 0; k < it.nkb; ++k) {
      if (!mbar_wait(&empty_bar[s], ph ^ 1)) { atomicOr(a->flags, DYB200_FLAG_WAIT_TIMEOUT); return; }
      unsigned char* st = ring + (size_t)s * STAGE_BYTES;
      if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * STAGE_BYTES);
      const uint32_t bar = s == 0 ? lead[0] : s == 1 ? lead[1] : lead[2];
      pair_load(st, &tm->t[0], bar, it.b0 + k, it.m0 + rank * BM, tm->a_mn);
      pair_load(st + TILE_BYTES, &tm->t[1], bar, it.b0 + k, it.m0 + rank * BM, tm->a_mn);
      pair_load(st + 2 * TILE_BYTES, &tm->t[2], bar, it.b0 + k, it.n0 + rank * BN, tm->b_mn);
      pair_load(st + 3 * TILE_BYTES, &tm->t[3], bar, it.b0 + k, it.n0 + rank * BN, tm->b_mn);
      if (++s == STAGES) { s = 0; ph ^= 1; }
    }
  }
}

__device__ __forceinline__ void pair_issue(const TmapPack* tm, const PairArgs* a, unsigned char* ring, uint64_t* full_bar, uint64_t* empty_bar, uint64_t* acc_full,
                                           uint64_t* acc_empty, uint32_t tmem) {
  const uint32_t items = a->tiles_m * a->tiles_n * a->S, pairs = gridDim.x >> 1;
  const uint32_t idesc = (1u << 4) | ((uint32_t)(kPairTile >> 3) << 17) | ((uint32_t)(kPairTile >> 4) << 24) | (tm->a_mn ? 1u << 15 : 0u) | (tm->b_mn ? 1u << 16 : 0u);
  const uint32_t base = smem_u32(ring);
  const uint64_t da = tm->a_mn ? umma_desc_mn16(base) : umma_desc(base), db = tm->b_mn ? umma_desc_mn16(base + 2 * TILE_BYTES) : umma_desc(base + 2 * TILE_BYTES);
  const uint64_t a_step = tm->a_mn ? 128 : 2, b_step = tm->b_mn ? 128 : 2;
  // (stage s: + s STAGE_BYTES in the address field, which the ring's top does not overflow; the lo planes one tile further)
  constexpr uint64_t kStage = STAGE_BYTES >> 4, kLo = TILE_BYTES >> 4;
  uint32_t sh = 0, ph = 0, sx = 0, chunk = 0, tile = 0;   // stage and phase of the next hi hi product, stage of the next cross products
  for (uint32_t w = blockIdx.x >> 1; w < items; w += pairs, ++tile) {
    const uint32_t nkb = pair_item(*a, w).nkb;
    uint32_t in_chunk = 0;
    for (uint32_t it = 0; it < nkb;) {
      const uint32_t left = min(kChunkF16 - in_chunk, nkb - it);
      const uint32_t g = it == 0 ? min(kPairHead, left) : left <= kPairTail ? left : 1u;
      if (in_chunk == 0 && chunk > 0 && !mbar_wait_cluster(&acc_empty[0], (chunk - 1) & 1)) { atomicOr(a->flags, DYB200_FLAG_WAIT_TIMEOUT); return; }
      for (uint32_t j = 0; j < g; ++j) {
        if (!mbar_wait(&full_bar[sh], ph)) { atomicOr(a->flags, DYB200_FLAG_WAIT_TIMEOUT); return; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        pair_mma(tmem, da + sh * kStage, db + sh * kStage, idesc, in_chunk + j, a_step, b_step);
        if (++sh == STAGES) { sh = 0; ph ^= 1; }
      }
      if (g == left) { pair_commit(&acc_full[0]); ++chunk; }
      if (it == 0 && tile > 0) {
        if (!mbar_wait_cluster(&acc_empty[1], (tile - 1) & 1)) { atomicOr(a->flags, DYB200_FLAG_WAIT_TIMEOUT); return; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      for (uint32_t j = 0; j < g; ++j) {
        const uint64_t a_hi = da + sx * kStage, b_hi = db + sx * kStage;
        pair_mma(tmem + kPairTile, a_hi, b_hi + kLo, idesc, it + j, a_step, b_step);
        pair_mma(tmem + kPairTile, a_hi + kLo, b_hi, idesc, 1u, a_step, b_step);
        pair_commit(&empty_bar[sx]);
        if (++sx == STAGES) sx = 0;
      }
      it += g;
      in_chunk = g == left ? 0 : in_chunk + g;
    }
    pair_commit(&acc_full[1]);
  }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1) k_gemm_pair(const __grid_constant__ TmapPack tm, const __grid_constant__ PairArgs a) {
  if (a.unless) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (*(const volatile uint32_t*)a.unless) return;   // (the same in every CTA)
  }
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];   // acc: 0 = D1, 1 = D2
  __shared__ uint32_t tmem_base_slot;
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.x & 1;   // (= the CTA's rank in its cluster)

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int q = 0; q < 2; ++q) { mbar_init(&acc_full[q], 1); mbar_init(&acc_empty[q], 2 * kEpiWarps); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 128) {
#pragma unroll
    for (int q = 0; q < 5; ++q) asm volatile("prefetch.tensormap [%0];" ::"l"(&tm.t[q]) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(2u * kPairTile) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();   // the barriers of both CTAs exist, and so do both allocations
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base_slot;
  asm volatile("griddepcontrol.wait;" ::: "memory");

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPairRegsLow));
    if (warp == 0) {
      if (elect_one()) pair_producer(&tm, &a, ring, full_bar, empty_bar, rank);
    } else if (warp == 1) {
      if (rank == 0 && elect_one()) pair_issue(&tm, &a, ring, full_bar, empty_bar, acc_full, acc_empty, tmem);
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPairRegsHigh));
    // warps 4..11: TMEM lanes 32 (warp % 4) .. +31 (rows of this CTA's half of the tile); warps 4-7 hold columns 0-127, warps 8-11 128-255
    const uint32_t quarter = warp & 3, half = (warp - 4) >> 2, th = threadIdx.x & 127;
    const uint32_t row = quarter * 32 + lane, lanes = tmem + ((quarter * 32) << 16) + 128 * half;
    float* const stage = reinterpret_cast<float*>(ring + (size_t)STAGES * STAGE_BYTES) + half * 2 * kPairBuf;
    const uint32_t items = a.tiles_m * a.tiles_n * a.S, pairs = gridDim.x >> 1;
    uint32_t chunk = 0, tile = 0, piece = 0;
    bool ok = true;
#pragma unroll 1
    for (uint32_t w = blockIdx.x >> 1; w < items; w += pairs, ++tile) {
      const PairItem it = pair_item(a, w);
      const uint32_t m = it.m0 + rank * BM + row, n0 = it.n0 + 128 * half;
      float sum[128];
#pragma unroll
      for (int q = 0; q < 128; ++q) sum[q] = 0.f;
      const uint32_t nchunks = (it.nkb + kChunkF16 - 1) / kChunkF16;
#pragma unroll 1
      for (uint32_t c = 0; c < nchunks; ++c, ++chunk) {
        if (ok && !mbar_wait(&acc_full[0], chunk & 1)) ok = false;
        if (!ok) continue;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          float v[32];
          tmem_ld32(lanes + 32 * p, v);
#pragma unroll
          for (int q = 0; q < 32; ++q) sum[32 * p + q] += v[q];
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(&acc_empty[0], 0);
      }
      if (ok && !mbar_wait(&acc_full[1], tile & 1)) ok = false;
      if (ok) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          float v[32];
          tmem_ld32(lanes + kPairTile + 32 * p, v);
#pragma unroll
          for (int q = 0; q < 32; ++q) sum[32 * p + q] = fmaf(v[q], kLoScale, sum[32 * p + q]);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive_remote(&acc_empty[1], 0);
      }
      // (the scales are applied as in unscale_tile: a lane fetches the words of four columns and hands them round)
      {
        const int ea = scale_field(__ldg(tm.sa + min(m, a.M - 1))) - 282;
        const float b = a.bias ? __ldg(a.bias + min(m, a.M - 1)) : 0.f;
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const int f = scale_field(__ldg(tm.sb + min(n0 + 32 * p + lane, a.N - 1)));
#pragma unroll
          for (int q = 0; q < 32; ++q) sum[32 * p + q] = unscale(sum[32 * p + q], ea + __shfl_sync(0xffffffffu, f, q)) + b;
        }
      }
      ok = bar_and(1 + half, 128, ok) != 0;
      if (!ok || it.m0 + rank * BM >= a.M || n0 >= a.N) continue;
      if (tm.store_map) {
#pragma unroll
        for (int p = 0; p < 128 / kPairPiece; ++p, ++piece) {
          if (n0 + kPairPiece * p >= a.N) break;
          float* const buf = stage + (piece & 1) * kPairBuf;
          if (th == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");   // the store before the last one has left this buffer
          bar_sync(1 + half, 128);
#pragma unroll
          for (int q = 0; q < kPairPiece; ++q) buf[q * BM + row] = sum[kPairPiece * p + q];
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          bar_sync(1 + half, 128);
          if (th == 0) {
            const int x = (int)(it.m0 + rank * BM), y = (int)(n0 + kPairPiece * p);
            if (a.accumulate)
              asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(&tm.t[4]), "r"(smem_u32(buf)), "r"(x),
                           "r"(y), "r"((int)it.z)
                           : "memory");
            else
              asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(&tm.t[4]), "r"(smem_u32(buf)), "r"(x), "r"(y),
                           "r"((int)it.z)
                           : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
          __syncwarp();
        }
      } else if (m < a.M) {
        float* dst = a.C + m + (size_t)a.ldc * ((size_t)it.z * a.N + n0);
        const uint32_t cols = min(128u, a.N - n0);
#pragma unroll
        for (int p = 0; p < 128; p += 8) {
          float old[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) old[q] = a.accumulate && p + q < cols ? dst[(size_t)a.ldc * q] : 0.f;
#pragma unroll
          for (int q = 0; q < 8; ++q)
            if (p + q < cols) dst[(size_t)a.ldc * q] = a.accumulate ? old[q] + sum[p + q] : sum[p + q];
          dst += (size_t)a.ldc * 8;
        }
      }
    }
    if (th == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    if (!ok && lane == 0) atomicOr(a.flags, DYB200_FLAG_WAIT_TIMEOUT);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync_all();   // neither CTA leaves while the other may still arrive on its barriers or read its tiles
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2u * kPairTile) : "memory");
  }
}

}  // namespace

// Which products take the pair kernel: plain results (the other epilogues are those of small products) with more than one tile of the
// one-SM kernel in either direction - with fewer rows or columns at least half of a 256 x 256 tile is padding.
bool dyb200_pair_takes(const dyb200_ctx* ctx, uint32_t M, uint32_t N, const GemmEpilogue& epi) {
  return ctx->sm_count >= 2 && M > BM && N > BN && epi.split_m == 0 && (epi.mode == EPI_STORE || epi.mode == EPI_ACCUM || epi.mode == EPI_BIAS);
}

// tm: the operand maps and scale words of dyb200_tc_gemm_packed (boxes of 128 rows x 64 k); K in k-blocks of 64.
int dyb200_gemm_pair(dyb200_ctx* ctx, TmapPack* tm, uint32_t M, uint32_t N, uint32_t kb, double flops, const GemmEpilogue& epi, const uint32_t* unless) {
  if (!(ctx->func_attr_done & (1u << 24))) {
    DYB_CUDA(ctx, cudaFuncSetAttribute(k_gemm_pair, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_PAIR_BYTES));
    // (the epilogue warps' share comes out of what the block is launched with; a build with fewer registers would wait for it without end)
    cudaFuncAttributes fa;
    DYB_CUDA(ctx, cudaFuncGetAttributes(&fa, k_gemm_pair));
    DYB_CHECK_ARG(ctx, 3 * fa.numRegs >= kPairRegsLow + 2 * kPairRegsHigh, "pair kernel built with %d registers per thread, its split needs %d", fa.numRegs,
                  (kPairRegsLow + 2 * kPairRegsHigh) / 3);
    ctx->func_attr_done |= 1u << 24;
  }
  const uint32_t pairs = (uint32_t)ctx->sm_count / 2;
  PairArgs a;
  memset(&a, 0, sizeof(a));
  a.M = M; a.N = N; a.kb = kb; a.flags = ctx->dev_flags; a.unless = unless;
  a.tiles_m = (M + kPairTile - 1) / kPairTile; a.tiles_n = (N + kPairTile - 1) / kPairTile; a.gm = 8;
  const uint32_t tiles = a.tiles_m * a.tiles_n;
  // K splits: rounds of the pairs x (k-blocks x 1.05 us + 2 us between items), and for more than one split the second stage, (S + 2) M N
  // floats through HBM at 5 TB/s and its launch.  (10000 x 1024 x 17920: 160 tiles on 74 pairs, 925 us unsplit, 800 in 4 splits with the
  // second stage, 791 in 6; 4096 x 1024 x 17920: 64 tiles, 304 unsplit, 322 in 9.)
  auto est = [&](uint32_t q) {
    return (double)((tiles * (uint64_t)q + pairs - 1) / pairs) * (((kb + q - 1) / q) * 1.05 + 2.0) + (q > 1 ? (q + 2) * 4.0e-6 * M * N / 5.0 + 8.0 : 0.0);
  };
  a.S = 1;
  double best = est(1);
  for (uint32_t q = 2; q <= 16 && kb / q >= 8; ++q) {
    const uint32_t per = (kb + q - 1) / q;
    if ((kb + per - 1) / per == q && est(q) < 0.97 * best) { best = est(q); a.S = q; }   // (no empty split)
  }
  GemmEpilogue e = epi;
  if (a.S > 1) {
    void* part;
    if (dyb200_scratch(ctx, (size_t)a.S * M * N * sizeof(float), &part) == DYB200_OK) e = GemmEpilogue{EPI_STORE, (float*)part, M, nullptr, 0, 0.f, nullptr, 0, 0};
    else a.S = 1;   // (no room for partial products)
  }
  a.C = e.C; a.ldc = e.ldc; a.bias = e.mode == EPI_BIAS ? e.bias : nullptr; a.accumulate = e.mode == EPI_ACCUM;
  tm->store_map = e.ldc % 4 == 0 && aligned16(e.C);
  if (tm->store_map) {
    int rc = dyb200_tc_make_store_map(ctx, &tm->t[4], e.C, M, N, a.S, e.ldc, kPairPiece);
    if (rc) return rc;
  }
  GemmProfScope scope(ctx, flops, 2, M, N, kb * 64, (uint32_t)epi.mode);
  dyb_launch(k_gemm_pair, dim3(2 * pairs), kPairThreads, SMEM_PAIR_BYTES, ctx, *tm, a);
  DYB_LAUNCHED(ctx);
  return a.S > 1 ? dyb200_splitk_reduce(ctx, e.C, a.S, M, N, epi, 0, unless) : DYB200_OK;
}
