// 3xTF32 GEMM on the 5th-generation tensor cores: tcgen05.mma (kind::tf32) with the accumulator
// in TMEM, operands staged in shared memory by TMA (cp.async.bulk.tensor, 128-byte swizzle, no
// multicast), one CTA per 128 x 128 output tile.
//
// fp32 accuracy from TF32 hardware: every operand x is split as x = hi + lo with hi = tf32(x) and
// lo = tf32(x - hi); the product a*b is accumulated as a_lo*b_hi + a_hi*b_lo + a_hi*b_hi (the
// lo*lo term, ~2^-22 relative, is dropped).  The split is done once per operand by a packing
// kernel that also brings the operand to K-major order (the reduction index contiguous) and
// applies the dropout mask, so the GEMM kernel itself only moves tiles and issues MMAs:
//   warp 0     TMA producer: 4 tiles (A_hi, A_lo, B_hi, B_lo) per 32-wide k-block, 3-stage ring
//   warp 1     allocates TMEM, issues 3 MMAs per 8-wide k-step, commits to the ring's mbarriers;
//              the accumulation chain is cut every kChunkKB k-blocks (two TMEM accumulators, used alternately)
//   warps 2-9  add every finished chunk (tcgen05.ld of their 32 accumulator lanes x 64 columns) into fp32
//              registers, park the finished tile in the idle operand ring and run the epilogue as a short
//              cooperative loop over it: 16-byte accesses along the rows (whole 512-byte tile columns per warp),
//              what it adds to fetched while the last MMAs run; the LSTM epilogue reads the four gates of a
//              hidden unit from the tile and also forms c and h
// Products with few output tiles are split along K over blockIdx.z; the splits store raw partial
// tiles and a second kernel adds them in split order and applies the epilogue (deterministic).
// Products with more tiles than SMs run on a persistent variant (one CTA per SM walks the tiles) whose
// epilogue overlaps the next tile's main loop.
// Every mbarrier wait is bounded; a wait that runs out sets DYB200_FLAG_WAIT_TIMEOUT and the
// kernel still frees its TMEM and returns.

#include "tc_dev.cuh"
#include "seq_dev.cuh"

namespace {

// instruction descriptor: D = f32, A = B = tf32 or f16, M = 128, N = cols (bits 15 / 16: A / B is MN-major)
__device__ __forceinline__ uint32_t tile_idesc(uint32_t cols, bool f16, uint32_t a_mn, uint32_t b_mn) {
  return (1u << 4) | (f16 ? 0u : (2u << 7) | (2u << 10)) | ((cols >> 3) << 17) | ((uint32_t)(BM >> 4) << 24) | (a_mn ? 1u << 15 : 0u) |
         (b_mn ? 1u << 16 : 0u);
}
// shared-memory descriptor of an operand tile, and what one MMA's k step adds to it (in units of 16 bytes)
__device__ __forceinline__ uint64_t tile_desc(uint32_t addr, bool f16, uint32_t mn) {
  return !mn ? umma_desc(addr) : f16 ? umma_desc_mn16(addr) : umma_desc_mn(addr);
}
__device__ __forceinline__ uint64_t mma_step(bool f16, uint32_t mn) { return !mn ? 2 : f16 ? 128 : 64; }
// F16: the sums of row m, columns [n0, n0 + 64), divided by the scales of the row and the columns
__device__ __forceinline__ void unscale_tile(const TmapPack& tm, float (&sum)[64], uint32_t m, uint32_t M, uint32_t n0, uint32_t N) {
  // (a lane fetches the words of two columns and hands them round)
  const int ea = scale_field(__ldg(tm.sa + min(m, M - 1))) - 282;
  const uint32_t lane = threadIdx.x & 31;
  const int f0 = scale_field(__ldg(tm.sb + min(n0 + lane, N - 1))), f1 = scale_field(__ldg(tm.sb + min(n0 + 32 + lane, N - 1)));
#pragma unroll
  for (int j = 0; j < 64; ++j) sum[j] = unscale(sum[j], ea + __shfl_sync(0xffffffffu, j < 32 ? f0 : f1, j & 31));
}

// The epilogue is what a short product spends its time on, and cold code is what an epilogue spends it on: a CTA runs it once, and
// unrolled or with the modes told apart inside, its instructions took longer to fetch than its data.  So: one short loop per mode,
// and what a tile adds to is copied into an idle stage of the operand ring while the last MMAs run, each thread's pieces by itself.
// us for a launch in a running program, before / after (fetched at the end, by the pass that knows every mode, and by K splits with their
// ranks' words read one after another): 1024 x 320 x 128 stored 8.2 / 6.0, 2000 x 256 x 320 added to 14.8 / 9.7, 1024 x 384 x 320 13.4 / 9.6,
// 5003 x 300 x 1050 (pieces of 4 bytes) 31 / 25, 1024 x 384 x 1600 in six splits 15.0 / 13.2, 300 x 1050 x 1200 in four 15.5 / 12.5.
template <int BYTES>
__device__ __forceinline__ void copy_piece(float* dst, const float* src) {
  if (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
// columns [c, c_hi) of the tile, STEP apart: what is there already, to the same place in `old` (stored like the tile)
template <int BYTES, int STEP>
__device__ __forceinline__ void fetch_old(float* old, const float* src, size_t ldc, uint32_t c, uint32_t c_hi) {
  src += ldc * c;
#pragma unroll 4
  for (; c < c_hi; c += STEP, src += STEP * ldc) copy_piece<BYTES>(old + (size_t)c * BM, src);
}
__device__ __forceinline__ float piece_add(float a, float b) { return a + b; }
__device__ __forceinline__ float4 piece_add(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
// (rounded as in every kernel with this epilogue)
__device__ __forceinline__ float piece_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float4 piece_fma(float4 a, float4 b, float4 c) {
  return make_float4(__fmaf_rn(a.x, b.x, c.x), __fmaf_rn(a.y, b.y, c.y), __fmaf_rn(a.z, b.z, c.z), __fmaf_rn(a.w, b.w, c.w));
}
// The plain epilogues on columns [c, c_hi) of a tile in shared memory, STEP apart, a piece V (4 rows or one) per thread and column;
// dst, mask and bias are those of the thread's first row, in column 0 of the tile; a thread whose rows are not there (no columns: c >= c_hi) reads none of them -
// its bias would be one value short of a whole piece, or beyond the last.
template <class V, int STEP>
__device__ __forceinline__ void write_pieces(int mode, const float* tile, const float* old, float* dst, size_t ldc, const float* mask,
                                             size_t mstep, const float* bias, uint32_t c, uint32_t c_hi) {
  if (c >= c_hi) return;
  auto at = [](const float* p) { return *reinterpret_cast<const V*>(p); };
  dst += ldc * c;
  tile += (size_t)c * BM; old += (size_t)c * BM;
  if (mode == EPI_STORE) {
#pragma unroll 4
    for (; c < c_hi; c += STEP, dst += STEP * ldc, tile += STEP * BM) *reinterpret_cast<V*>(dst) = at(tile);
  } else if (mode == EPI_BIAS) {
    const V b = at(bias);
#pragma unroll 4
    for (; c < c_hi; c += STEP, dst += STEP * ldc, tile += STEP * BM) *reinterpret_cast<V*>(dst) = piece_add(at(tile), b);
  } else if (mode == EPI_ACCUM) {
#pragma unroll 4
    for (; c < c_hi; c += STEP, dst += STEP * ldc, tile += STEP * BM, old += STEP * BM) *reinterpret_cast<V*>(dst) = piece_add(at(tile), at(old));
  } else {
    mask += mstep * c;
#pragma unroll 4
    for (; c < c_hi; c += STEP, dst += STEP * ldc, tile += STEP * BM, old += STEP * BM, mask += STEP * mstep)
      *reinterpret_cast<V*>(dst) = piece_fma(at(tile), at(mask), at(old));
  }
}
// K splits as a cluster: the sums over the S partial tiles of the 16-byte pieces of columns [c, c_hi), 8 apart, in split order, put into
// this CTA's own tile; BATCH columns x RANKS tiles requested at a time.
template <int RANKS, int BATCH>
__device__ __forceinline__ void slice_sums(float* tile, uint32_t S, uint32_t rq, uint32_t c, uint32_t c_hi) {
  const uint32_t here = smem_u32(tile) + 16 * rq;
  uint32_t base[RANKS];
#pragma unroll
  for (int r = 0; r < RANKS; ++r) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(base[r]) : "r"(here), "r"(min((uint32_t)r, S - 1)));
#pragma unroll 1
  for (; c < c_hi; c += 8 * BATCH) {
    float4 p[BATCH][RANKS];
#pragma unroll
    for (int k = 0; k < BATCH; ++k)
#pragma unroll
      for (int r = 0; r < RANKS; ++r)
        if ((uint32_t)r < S && c + 8 * k < c_hi)
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(p[k][r].x), "=f"(p[k][r].y), "=f"(p[k][r].z), "=f"(p[k][r].w)
                       : "r"(base[r] + 4u * BM * (c + 8u * k)) : "memory");
#pragma unroll
    for (int k = 0; k < BATCH; ++k) {
      float4 a = p[k][0];
#pragma unroll
      for (int r = 1; r < RANKS; ++r)
        if ((uint32_t)r < S) a = piece_add(a, p[k][r]);
      if (c + 8 * k < c_hi) st4(tile + (size_t)(c + 8 * k) * BM + 4 * rq, a);
    }
  }
}

// BNT = columns of the output tile: 128, or 64 for products with N <= 64 (small per-GPU batches), where a 128-wide tile
// would spend half of every MMA and half of the B traffic on padding.
// CLUSTER: the gridDim.z K-splits of a tile form one thread-block cluster (1 x 1 x S); every CTA parks its partial tile in
// its own shared memory, and CTA r adds all partial tiles of its 1 / S of the columns through distributed shared memory, in
// split order, and runs the epilogue on that slice - no workspace round trip and no second kernel.
// F16: the operands are fp16 pairs (tc_dev.cuh) in k-blocks of 64; an accumulator is D1 | D2, 2 BNT columns of TMEM.
// TWO: two right operands side by side, each with its own destination (TmapPack::n_split).  A variant of its own, since the choice of the
// destination costs the epilogue registers; the persistent kernel leaves it to k_splitk_reduce: with it in its epilogue, its three
// products in a step of a language model of 128 units (vocabulary 1901, 10560 tokens) took 60 us each instead of 38.
template <int BNT, bool CLUSTER, bool F16 = false, bool TWO = false>
__global__ void __launch_bounds__(kThreads, 1) k_gemm_tc(const __grid_constant__ TmapPack tm, uint32_t M, uint32_t N,
                                                         uint32_t kb0, uint32_t kb1, uint32_t kb_per_split,
                                                         GemmEpilogue epi, uint32_t* flags) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // (the wait comes after the prologue, below)
  if (TWO && !CLUSTER && tm.sa) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!*(const volatile uint32_t*)tm.sa) return;   // (the same in every CTA)
  }
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2], old_free;
  __shared__ uint32_t tmem_base_slot;
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int TILE_B_BYTES = BNT * BK * 4;                      // one B plane of a stage
  constexpr int STAGE_TX = 2 * TILE_BYTES + 2 * TILE_B_BYTES;     // bytes a stage receives (stages stay STAGE_BYTES apart)
  const uint32_t m0 = blockIdx.x * BM, n0 = blockIdx.y * BNT;
  // K splits: split z of S takes the z-th share of EACH pair's k-blocks (pair 0 first, then pair 1), so that in
  // Wx x + Wh h every split holds the same mix of the two products (the sequence-persistent LSTM kernel relies on
  // it: only the Wh h share of a split waits for the previous time step).  With one pair this is the plain contiguous cut.
  const KSplit ks = k_split(kb0, kb1, blockIdx.z, gridDim.z);
  const uint32_t total = ks.n0 + ks.n1;
  (void)kb_per_split;
  constexpr uint32_t kChunk = F16 ? kChunkF16 : kChunkKB, kAccCols = F16 ? 2 * BN : BN, kTmem = F16 ? 2 * kTmemCols : kTmemCols;
  constexpr int EL = F16 ? 64 : 32;
  const uint32_t nchunks = (total + kChunk - 1) / kChunk;
  if (!CLUSTER && gridDim.z > 1) epi.C += (size_t)blockIdx.z * epi.ldc * N;   // raw partial tile of this split (mode is EPI_STORE)
  // What the tile adds to goes into the stage after the last k-block's (not the first one, where the tile will be), once k-block
  // it_old - STAGES has been read from it.
  const uint32_t it_old = total + (total % STAGES == 0 ? 1 : 0);
  __shared__ uint32_t split_ok;   // CLUSTER: this CTA's partial tile is complete

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int q = 0; q < 2; ++q) { mbar_init(&acc_full[q], 1); mbar_init(&acc_empty[q], kEpiWarps); }
    mbar_init(&old_free, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 32 * 2) {   // (an epilogue thread, idle until the first chunk is done) descriptors of the first loads
#pragma unroll
    for (int q = 0; q < 8; ++q) asm volatile("prefetch.tensormap [%0];" ::"l"(&tm.t[q]) : "memory");
  }
  if (warp == 1) {   // the whole warp allocates the accumulator columns
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(kTmem) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_slot;
  // Barrier initialisation and the TMEM allocation above may overlap the previous kernel of the stream; nothing below
  // (TMA loads, c_prev prefetch, stores) starts before that kernel has completed.
  // (the scales of fp16 pairs go by __ldg, which an asm statement alone does not keep behind it)
  dyb_grid_dep_wait();

  if (warp == 0) {
    if (elect_one()) {
      uint32_t s = 0, ph = 0;
      const bool second = TWO && n0 >= tm.n_split;
      const uint32_t nb0 = second ? n0 - tm.n_split : n0, tb = second ? 6u : 2u;
      for (uint32_t it = 0; it < total; ++it) {
        if (!mbar_wait(&empty_bar[s], ph ^ 1)) { atomicOr(flags, DYB200_FLAG_WAIT_TIMEOUT); break; }
        const uint32_t pair = it < ks.n0 ? 0 : 1, kblk = pair ? ks.b1 + (it - ks.n0) : ks.b0 + it;
        unsigned char* st = ring + (size_t)s * STAGE_BYTES;
        mbar_expect_tx(&full_bar[s], STAGE_TX);
        load_a_tile<EL>(st, &tm.t[4 * pair + 0], &full_bar[s], kblk, m0, tm.a_mn);
        load_a_tile<EL>(st + TILE_BYTES, &tm.t[4 * pair + 1], &full_bar[s], kblk, m0, tm.a_mn);
        load_b_tile<EL>(st + 2 * TILE_BYTES, &tm.t[4 * pair + tb], &full_bar[s], kblk, nb0, tm.b_mn);
        load_b_tile<EL>(st + 2 * TILE_BYTES + TILE_B_BYTES, &tm.t[4 * pair + tb + 1], &full_bar[s], kblk, nb0, tm.b_mn);
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
    if (CLUSTER) {   // all lanes: the two cluster barriers of the epilogue warps (see there)
      __syncwarp();
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // This one thread issues every MMA of the tile, and the tensor pipe is only as busy as this loop is short:
      // descriptors of the three stages are built once, stage / phase / chunk counters are carried instead of divided,
      // and the 12 MMAs of a k-block go out in one block of PTX.
      // instruction descriptor: D = f32, A = B = tf32, both K-major, N = BNT, M = 128
      // (bits 15 / 16: A / B is MN-major)
      const uint32_t a_mn = tm.a_mn, b_mn = tm.b_mn;
      const uint32_t idesc = tile_idesc(BNT, F16, a_mn, b_mn), idesc_wide = tile_idesc(2 * BNT, F16, a_mn, b_mn);
      const uint64_t a_step = mma_step(F16, a_mn), b_step = mma_step(F16, b_mn);
      uint64_t d_a_hi[STAGES], d_a_lo[STAGES], d_b_hi[STAGES], d_b_lo[STAGES];
#pragma unroll
      for (int q = 0; q < STAGES; ++q) {
        const uint32_t base = smem_u32(ring + (size_t)q * STAGE_BYTES);
        d_a_hi[q] = tile_desc(base, F16, a_mn);
        d_a_lo[q] = tile_desc(base + TILE_BYTES, F16, a_mn);
        d_b_hi[q] = tile_desc(base + 2 * TILE_BYTES, F16, b_mn);
        d_b_lo[q] = tile_desc(base + 2 * TILE_BYTES + TILE_B_BYTES, F16, b_mn);
      }
      // The tensor core truncates when it aligns addends to the accumulator, a bias that grows with the length of
      // the accumulation chain.  So the chain is cut every kChunkKB k-blocks: chunk c accumulates into TMEM buffer
      // c & 1 from zero, and the epilogue warps add finished chunks into fp32 registers with ordinary rounding.
      uint32_t s = 0, ph = 0, in_chunk = 0, chunk = 0, buf = 0;
      for (uint32_t it = 0; it < total; ++it) {
        if (in_chunk == 0 && chunk >= 2) {   // buffer reuse: the epilogue warps must have drained chunk - 2
          if (!mbar_wait(&acc_empty[buf], ((chunk >> 1) - 1) & 1)) { atomicOr(flags, DYB200_FLAG_WAIT_TIMEOUT); break; }
        }
        if (!mbar_wait(&full_bar[s], ph)) { atomicOr(flags, DYB200_FLAG_WAIT_TIMEOUT); break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint64_t a_hi, a_lo, b_hi, b_lo;   // select without dynamic register indexing
        if (s == 0) { a_hi = d_a_hi[0]; a_lo = d_a_lo[0]; b_hi = d_b_hi[0]; b_lo = d_b_lo[0]; }
        else if (s == 1) { a_hi = d_a_hi[1]; a_lo = d_a_lo[1]; b_hi = d_b_hi[1]; b_lo = d_b_lo[1]; }
        else { a_hi = d_a_hi[2]; a_lo = d_a_lo[2]; b_hi = d_b_hi[2]; b_lo = d_b_lo[2]; }
        const uint32_t acc = tmem_base + buf * kAccCols;
        if (F16) issue_kblock_f16(acc, acc + BNT, a_hi, a_lo, b_hi, idesc_wide, idesc, in_chunk, a_step, b_step);
        else issue_kblock(acc, a_hi, a_lo, b_hi, b_lo, idesc, in_chunk, a_step, b_step);
        umma_commit(&empty_bar[s]);   // frees the stage once these MMAs have read it
        if (it + STAGES == it_old) umma_commit(&old_free);
        const bool chunk_ends = in_chunk == kChunk - 1 || it == total - 1;
        if (chunk_ends) { umma_commit(&acc_full[buf]); in_chunk = 0; ++chunk; buf ^= 1; }
        else ++in_chunk;
        if (++s == STAGES) { s = 0; ph ^= 1; }
      }
    }
    if (CLUSTER) {
      __syncwarp();
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
  } else {
    // epilogue warps 2..9: TMEM lanes 32*(warp % 4) .. +31 (row of the tile = lane of TMEM); warps 2-5
    // take columns 0-63, warps 6-9 columns 64-127
    const uint32_t quarter = warp & 3, half = (warp - 2) >> 2;
    const uint32_t te = threadIdx.x - 64;   // 0..255 among the epilogue threads
    // EPI_LSTM_CELL: in the cooperative pass below this thread owns hidden units [4 (te % 8), +4) of the tile's 32 for
    // the columns te / 8 + 32 k; their previous cell states are fetched now, while the MMAs run
    float4 cprev[4];
    if (epi.mode == EPI_LSTM_CELL) {
      const uint32_t u = blockIdx.x * 32 + 4 * (te & 7);
#pragma unroll
      for (int k = 0; k < BNT / 32; ++k) {
        const uint32_t n = n0 + (te >> 3) + 32 * k;
        cprev[k] = n < N ? ld4(epi.c_prev + u + (size_t)epi.H * n) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    uint32_t ne0 = n0, Ne = N;
    if (TWO) epi_side(epi, ne0, Ne);
    // the columns this CTA finishes (K splits as a cluster: its slice), and the pieces of them this thread does in the plain epilogues:
    // 4 rows of every eighth column where rows and destinations allow it, a row of every second one otherwise
    const uint32_t S = CLUSTER ? gridDim.z : 1, w = CLUSTER ? ((BNT + S - 1) / S + 7) & ~7u : BNT;
    const uint32_t c_lo = CLUSTER ? min(blockIdx.z * w, (uint32_t)BNT) : 0, c_hi = CLUSTER ? min(c_lo + w, (uint32_t)BNT) : BNT;
    const bool adds = epi.mode == EPI_ACCUM || epi.mode == EPI_ACCUM_MASK;
    const bool plain = adds || epi.mode == EPI_STORE || epi.mode == EPI_BIAS, vec = plain && epi_in_pieces(epi, M);
    const uint32_t my_r = vec ? 4 * (te & 31) : te & 127, my_c = c_lo + (vec ? te >> 5 : te >> 7);
    const uint32_t my_hi = m0 + my_r < M && ne0 < Ne ? min(c_hi, Ne - ne0) : 0;
    const EpiRow row = epi_row(epi, min(m0 + my_r, M - 1));
    float* const dst = row.c + (size_t)row.ldc * ne0;
    float* const old = reinterpret_cast<float*>(ring + (size_t)(it_old % STAGES) * STAGE_BYTES) + my_r;
    float sum[64];   // this thread's row of the tile, columns [64 half, 64 half + 64)
#pragma unroll
    for (int j = 0; j < 64; ++j) sum[j] = 0.f;
    bool ok = true;
#pragma unroll 1
    for (uint32_t c = 0; c < nchunks; ++c) {
      const uint32_t buf = c & 1;
      if (adds && c == nchunks - 1) {   // (the chunks before are drained: the MMAs that free the stage wait for nothing here)
        if (it_old >= STAGES && !mbar_wait(&old_free, 0)) { ok = false; break; }
        if (vec) fetch_old<16, 8>(old, dst, row.ldc, my_c, my_hi);
        else fetch_old<4, 2>(old, dst, row.ldc, my_c, my_hi);
      }
      if (!mbar_wait(&acc_full[buf], (c >> 1) & 1)) { ok = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (64 * half < BNT) {   // (with a 64-column tile the second column half does not exist)
        // (two 32-column loads: one 64-column load per flush measured slower)
        float v[32];
        const uint32_t taddr = tmem_base + buf * kAccCols + ((quarter * 32) << 16) + 2 * half * 32;
        tmem_ld32(taddr, v);
#pragma unroll
        for (int j = 0; j < 32; ++j) sum[j] += v[j];
        tmem_ld32(taddr + 32, v);
#pragma unroll
        for (int j = 0; j < 32; ++j) sum[32 + j] += v[j];
        if (F16) {
          tmem_ld32(taddr + BNT, v);
#pragma unroll
          for (int j = 0; j < 32; ++j) sum[j] = fmaf(v[j], kLoScale, sum[j]);
          tmem_ld32(taddr + BNT + 32, v);
#pragma unroll
          for (int j = 0; j < 32; ++j) sum[32 + j] = fmaf(v[j], kLoScale, sum[32 + j]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[buf]);
    }
    if (!ok && lane == 0) atomicOr(flags, DYB200_FLAG_WAIT_TIMEOUT);
    // The tile goes through shared memory (the operand ring is idle once the last chunk has been drained: every MMA
    // has completed and no TMA load is in flight), stored like C: column-major, 128 rows per column.  The pass that
    // follows is a short rolled loop in which consecutive threads take consecutive rows, so global accesses are
    // 16-byte vectors covering whole 512-byte columns of the tile.  Every epilogue warp reaches the named barrier,
    // whatever its waits did; a failed wait anywhere cancels the stores.
    float* tile = reinterpret_cast<float*>(ring);
    if (F16 && 64 * half < BNT) unscale_tile(tm, sum, m0 + quarter * 32 + lane, M, n0 + 64 * half, N);
    if (64 * half < BNT) {
      float* col = tile + (size_t)(64 * half) * BM + quarter * 32 + lane;
#pragma unroll
      for (int j = 0; j < 64; ++j) col[(size_t)j * BM] = sum[j];
    }
    if (adds) asm volatile("cp.async.wait_all;" ::: "memory");   // (each thread reads what it has fetched itself)
    uint32_t all_ok;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.cta.red.and.pred p, 1, 256, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(all_ok) : "r"((uint32_t)ok) : "memory");
    auto finish = [&]() {
      const float* mask = epi.mode == EPI_ACCUM_MASK ? row.mask + (row.mask_full ? (size_t)row.mask_ld * ne0 : 0) : nullptr;
      const size_t mstep = row.mask_full ? row.mask_ld : 0;
      const float* bias = epi.bias + min(m0 + my_r, M - 1);
      if (vec) write_pieces<float4, 8>(epi.mode, tile + my_r, old, dst, row.ldc, mask, mstep, bias, my_c, my_hi);
      else if (plain) write_pieces<float, 2>(epi.mode, tile + my_r, old, dst, row.ldc, mask, mstep, bias, my_c, my_hi);
      else epilogue_pass<BNT, 256>(epi, tile, te, blockIdx.x, m0, ne0, M, Ne, cprev, c_lo, c_hi);
    };
    if (!CLUSTER) {
      if (all_ok) finish();
    } else {
      // every thread of every CTA of the cluster takes part in the two cluster barriers below (the TMA and MMA warps
      // reach them further down); between them rank 0 reads the other CTAs' tiles
      if (te == 0) split_ok = all_ok;
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      // Rank r (= blockIdx.z: the cluster is 1 x 1 x gridDim.z) finishes columns [c_lo, c_hi) of the tile: it adds the
      // S partial tiles of that slice in split order (the order of the split-K reduction kernel), its own from its
      // shared memory and the others through distributed shared memory, and runs the epilogue on the slice.
      uint32_t ra, v;   // (one rank's word per lane)
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(smem_u32(&split_ok)), "r"(min((uint32_t)lane, S - 1)));
      asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(ra) : "memory");
      {   // (whatever the words say: the sums go no further than this tile yet)
        const uint32_t rq = te & 31, c = c_lo + (te >> 5);
        if (S <= 2) slice_sums<2, 4>(tile, S, rq, c, c_hi);
        else if (S <= 4) slice_sums<4, 2>(tile, S, rq, c, c_hi);
        else slice_sums<8, 2>(tile, S, rq, c, c_hi);
      }
      const bool ok_all = __all_sync(0xffffffffu, v != 0);
      if (!ok_all && te == 0 && blockIdx.z == 0) atomicOr(flags, DYB200_FLAG_WAIT_TIMEOUT);
      __syncwarp();
      // every tile stays until all ranks have read it
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      if (ok_all) {
        if (!vec) asm volatile("barrier.cta.sync 1, 256;" ::: "memory");   // the pass below reads other threads' pieces
        finish();
      }
      __syncwarp();
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmem) : "memory");
  }
}

// ---- persistent variant for products with more tiles than SMs -----------------------------------------------------------
// One CTA per SM walks the tiles blockIdx.x, blockIdx.x + gridDim.x, ... (the same order in which the one-tile kernel's
// CTAs would run, so CTAs that share operand tiles still work on the same k-blocks at the same time).  The epilogue of a
// tile runs while the TMA and MMA warps are already on the next one: the finished tile waits in the epilogue warps'
// registers (the TMEM accumulators are free again as soon as their last chunk is drained) and goes through a 32 KiB
// staging buffer beside the operand ring, one 64-column half at a time: warps 2-5 park and write out columns 0-63, then
// warps 6-9 columns 64-127.  What this saves is the pipeline fill and the epilogue of every tile but the last, about
// 9 us per tile: a third of the time of the output layer's product (K = 1024, 75 tiles per SM).
constexpr int SMEM_PERSIST_BYTES = SMEM_BYTES + BM * 64 * 4;
// Four accumulators (all 512 TMEM columns): the MMA warp may run four chunks - a whole tile of the output layer's
// product - ahead of the epilogue warps, which drain nothing while they write out the previous tile.
constexpr uint32_t kPersistBufs = 4;

// Tile order.  gm == 0: row block fastest (the launch order of the one-tile kernel).  gm > 0: groups of gm row blocks, row
// block fastest within a group, then the column block, then the next group.  The 148 tiles in flight then touch gm A
// blocks and ~148 / gm B blocks instead of all A blocks and two B blocks, and the A blocks of a group stay in L2 while
// the B blocks stream past them (output layer, gm = 16: 25 MB of operands per round instead of 83 MB).
__device__ __forceinline__ void persist_tile_coords(uint32_t tile, uint32_t tiles_m, uint32_t tiles_n, uint32_t gm, uint32_t& mt,
                                                    uint32_t& nt) {
  if (gm == 0) { mt = tile % tiles_m; nt = tile / tiles_m; return; }
  const uint32_t per_group = gm * tiles_n;
  const uint32_t g = tile / per_group, r = tile - g * per_group;
  const uint32_t rows = min(gm, tiles_m - g * gm);   // the last group may be lower
  nt = r / rows;
  mt = g * gm + r % rows;
}

// The two single-thread roles are functions of their own: their loops pace the tensor pipe and keep their own registers.
template <int BNT, bool F16>
__device__ __noinline__ void persist_producer(const TmapPack* tm, unsigned char* ring, uint64_t* full_bar, uint64_t* empty_bar,
                                              uint32_t tiles, uint32_t tiles_m, uint32_t tiles_n, uint32_t gm, uint32_t kb0,
                                              uint32_t kb1, uint32_t S, uint32_t* flags) {
  constexpr int TILE_B_BYTES = BNT * BK * 4;
  constexpr int STAGE_TX = 2 * TILE_BYTES + 2 * TILE_B_BYTES;
  uint32_t s = 0, ph = 0;
  bool fail = false;
  // work item w = (K split z, tile): all tiles of split 0 first, so that the CTAs of a round share operand k-blocks
  for (uint32_t w = blockIdx.x; w < tiles * S && !fail; w += gridDim.x) {
    const uint32_t z = w / tiles, tile = w - z * tiles;
    const KSplit ks = k_split(kb0, kb1, z, S);
    uint32_t mt, nt;
    persist_tile_coords(tile, tiles_m, tiles_n, gm, mt, nt);
    const uint32_t m0 = mt * BM, n0 = nt * BNT;
    const bool second = tm->n_split && n0 >= tm->n_split;
    const uint32_t nb0 = second ? n0 - tm->n_split : n0, tb = second ? 6u : 2u;
    for (uint32_t g = 0; g < ks.n0 + ks.n1; ++g) {
      if (!mbar_wait(&empty_bar[s], ph ^ 1)) { fail = true; break; }
      const uint32_t pair = g < ks.n0 ? 0 : 1, kblk = pair ? ks.b1 + (g - ks.n0) : ks.b0 + g;
      unsigned char* st = ring + (size_t)s * STAGE_BYTES;
      mbar_expect_tx(&full_bar[s], STAGE_TX);
      load_a_tile<F16 ? 64 : 32>(st, &tm->t[4 * pair + 0], &full_bar[s], kblk, m0, tm->a_mn);
      load_a_tile<F16 ? 64 : 32>(st + TILE_BYTES, &tm->t[4 * pair + 1], &full_bar[s], kblk, m0, tm->a_mn);
      load_b_tile<F16 ? 64 : 32>(st + 2 * TILE_BYTES, &tm->t[4 * pair + tb], &full_bar[s], kblk, nb0, tm->b_mn);
      load_b_tile<F16 ? 64 : 32>(st + 2 * TILE_BYTES + TILE_B_BYTES, &tm->t[4 * pair + tb + 1], &full_bar[s], kblk, nb0, tm->b_mn);
      if (++s == STAGES) { s = 0; ph ^= 1; }
    }
  }
  if (fail) atomicOr(flags, DYB200_FLAG_WAIT_TIMEOUT);
}

template <int BNT, bool F16>
__device__ __noinline__ void persist_issue(unsigned char* ring, uint64_t* full_bar, uint64_t* empty_bar, uint64_t* acc_full,
                                           uint64_t* acc_empty, uint32_t tmem_base, uint32_t tiles, uint32_t kb0, uint32_t kb1, uint32_t S,
                                           uint32_t a_mn, uint32_t b_mn, uint32_t* flags) {
  constexpr int TILE_B_BYTES = BNT * BK * 4;
  constexpr uint32_t kBufs = F16 ? kPersistBufs / 2 : kPersistBufs, kChunk = F16 ? kChunkF16 : kChunkKB, kAccCols = F16 ? 2 * BN : BN;
  const uint32_t idesc = tile_idesc(BNT, F16, a_mn, b_mn), idesc_wide = tile_idesc(2 * BNT, F16, a_mn, b_mn);
  const uint64_t a_step = mma_step(F16, a_mn), b_step = mma_step(F16, b_mn);
  uint64_t d_a_hi[STAGES], d_a_lo[STAGES], d_b_hi[STAGES], d_b_lo[STAGES];
#pragma unroll
  for (int q = 0; q < STAGES; ++q) {
    const uint32_t base = smem_u32(ring + (size_t)q * STAGE_BYTES);
    d_a_hi[q] = tile_desc(base, F16, a_mn);
    d_a_lo[q] = tile_desc(base + TILE_BYTES, F16, a_mn);
    d_b_hi[q] = tile_desc(base + 2 * TILE_BYTES, F16, b_mn);
    d_b_lo[q] = tile_desc(base + 2 * TILE_BYTES + TILE_B_BYTES, F16, b_mn);
  }
  // stage, phase and chunk counters run on across tiles; an accumulation chain never crosses a tile boundary
  uint32_t s = 0, ph = 0, chunk = 0, buf = 0;
  bool fail = false;
  for (uint32_t w = blockIdx.x; w < tiles * S && !fail; w += gridDim.x) {
    const KSplit ks = k_split(kb0, kb1, w / tiles, S);
    const uint32_t kb = ks.n0 + ks.n1;
    uint32_t in_chunk = 0;
    for (uint32_t it = 0; it < kb; ++it) {
      if (in_chunk == 0 && chunk >= kBufs) {
        if (!mbar_wait(&acc_empty[buf], ((chunk / kBufs) - 1) & 1)) { fail = true; break; }
      }
      if (!mbar_wait(&full_bar[s], ph)) { fail = true; break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint64_t a_hi, a_lo, b_hi, b_lo;
      if (s == 0) { a_hi = d_a_hi[0]; a_lo = d_a_lo[0]; b_hi = d_b_hi[0]; b_lo = d_b_lo[0]; }
      else if (s == 1) { a_hi = d_a_hi[1]; a_lo = d_a_lo[1]; b_hi = d_b_hi[1]; b_lo = d_b_lo[1]; }
      else { a_hi = d_a_hi[2]; a_lo = d_a_lo[2]; b_hi = d_b_hi[2]; b_lo = d_b_lo[2]; }
      const uint32_t acc = tmem_base + buf * kAccCols;
      if (F16) issue_kblock_f16(acc, acc + BNT, a_hi, a_lo, b_hi, idesc_wide, idesc, in_chunk, a_step, b_step);
      else issue_kblock(acc, a_hi, a_lo, b_hi, b_lo, idesc, in_chunk, a_step, b_step);
      umma_commit(&empty_bar[s]);
      const bool chunk_ends = in_chunk == kChunk - 1 || it == kb - 1;
      if (chunk_ends) { umma_commit(&acc_full[buf]); in_chunk = 0; ++chunk; buf = chunk % kBufs; }
      else ++in_chunk;
      if (++s == STAGES) { s = 0; ph ^= 1; }
    }
  }
  if (fail) atomicOr(flags, DYB200_FLAG_WAIT_TIMEOUT);
}


template <int BNT, bool F16 = false>
__global__ void __launch_bounds__(kThreads, 1) k_gemm_persist(const __grid_constant__ TmapPack tm, uint32_t M, uint32_t N,
                                                              uint32_t kb0, uint32_t kb1, uint32_t tiles_m, uint32_t tiles,
                                                              uint32_t gm, uint32_t S, GemmEpilogue epi, uint32_t* flags) {
  // (no early start of the next kernel: this one has every SM for its whole time)
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[kPersistBufs], acc_empty[kPersistBufs];
  __shared__ uint32_t tmem_base_slot;
  unsigned char* ring = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* stage = reinterpret_cast<float*>(ring + (size_t)STAGES * STAGE_BYTES);   // 64 columns x BM rows
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (uint32_t q = 0; q < kPersistBufs; ++q) { mbar_init(&acc_full[q], 1); mbar_init(&acc_empty[q], kEpiWarps); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(kPersistBufs * BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_base_slot;
  asm volatile("griddepcontrol.wait;" ::: "memory");

  if (warp == 0) {
    if (elect_one()) persist_producer<BNT, F16>(&tm, ring, full_bar, empty_bar, tiles, tiles_m, (N + BNT - 1) / BNT, gm, kb0, kb1, S, flags);
  } else if (warp == 1) {
    if (elect_one()) persist_issue<BNT, F16>(ring, full_bar, empty_bar, acc_full, acc_empty, tmem_base, tiles, kb0, kb1, S, tm.a_mn, tm.b_mn, flags);
  } else {
    // epilogue warps 2..9: TMEM lanes 32 (warp % 4) .. +31; warps 2-5 hold columns 0-63 of the tile, warps 6-9 columns 64-127
    const uint32_t quarter = warp & 3, half = (warp - 2) >> 2;
    const uint32_t th = (threadIdx.x - 64) & 127;   // 0..127 within this half's four warps
    const bool has_cols = 64 * half < BNT;
    constexpr uint32_t kBufs = F16 ? kPersistBufs / 2 : kPersistBufs, kChunk = F16 ? kChunkF16 : kChunkKB, kAccCols = F16 ? 2 * BN : BN;
    uint32_t cg = 0;   // chunks drained so far (selects the TMEM buffer and the barrier phase)
    bool ok = true;
#pragma unroll 1
    for (uint32_t w = blockIdx.x, j = 0; w < tiles * S; w += gridDim.x, ++j) {
      const uint32_t z = w / tiles, tile = w - z * tiles;
      const KSplit ks = k_split(kb0, kb1, z, S);
      const uint32_t nchunks = (ks.n0 + ks.n1 + kChunk - 1) / kChunk;
      // (K splits: epi is a plain store with ldc = M into S partial products side by side, so split z writes columns z N ..)
      const uint32_t n_shift = z * N;
      uint32_t mt, nt;
      persist_tile_coords(tile, tiles_m, (N + BNT - 1) / BNT, gm, mt, nt);
      const uint32_t m0 = mt * BM, n0 = nt * BNT + 64 * half;
      float sum[64];
#pragma unroll
      for (int q = 0; q < 64; ++q) sum[q] = 0.f;
#pragma unroll 1
      for (uint32_t c = 0; c < nchunks; ++c, ++cg) {
        const uint32_t buf = cg % kBufs;
        if (!ok) continue;
        if (!mbar_wait(&acc_full[buf], (cg / kBufs) & 1)) { ok = false; continue; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (has_cols) {
          float v[32];
          const uint32_t taddr = tmem_base + buf * kAccCols + ((quarter * 32) << 16) + 2 * half * 32;
          tmem_ld32(taddr, v);
#pragma unroll
          for (int q = 0; q < 32; ++q) sum[q] += v[q];
          tmem_ld32(taddr + 32, v);
#pragma unroll
          for (int q = 0; q < 32; ++q) sum[32 + q] += v[q];
          if (F16) {
            tmem_ld32(taddr + BNT, v);
#pragma unroll
            for (int q = 0; q < 32; ++q) sum[q] = fmaf(v[q], kLoScale, sum[q]);
            tmem_ld32(taddr + BNT + 32, v);
#pragma unroll
            for (int q = 0; q < 32; ++q) sum[32 + q] = fmaf(v[q], kLoScale, sum[32 + q]);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[buf]);
      }
      if (F16 && has_cols) unscale_tile(tm, sum, m0 + quarter * 32 + lane, M, n0, N);
      if (!has_cols) continue;   // (64-column tiles: warps 6-9 only take part in the accumulator hand-shake)
      // The staging buffer is free once the other half has written out its columns of the previous turn (128-column
      // tiles), or once this half's own warps have all left the previous pass (64-column tiles).
      if (BNT == 128) {
        if (half == 1) bar_sync(2, 256);
        else if (j > 0) bar_sync(4, 256);
      } else if (j > 0) {
        bar_sync(2, 128);
      }
      {
        float* col = stage + quarter * 32 + lane;
        const float b = tm.store_map && epi.mode == EPI_BIAS ? __ldg(epi.bias + min(m0 + quarter * 32 + lane, M - 1)) : 0.f;
#pragma unroll
        for (int q = 0; q < 64; ++q) col[(size_t)q * BM] = sum[q] + b;
      }
      if (tm.store_map) {
        // A plain store: the staged 64 columns x 128 rows go out as one TMA store (rows and columns past the edge are clipped),
        // and these warps go on to drain the next tile.  The generic pass below took longer than the tensor pipe needs for a tile
        // of K = 512 fp16 pairs.
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        const uint32_t fine = bar_and(1u + 2u * half, 128, ok);
        if (fine && th == 0) {
          asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(&tm.t[4]), "r"(smem_u32(stage)),
                       "r"((int)m0), "r"((int)n0), "r"((int)z) : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the buffer may be overwritten
        }
        __syncwarp();
        if (BNT == 128) {
          if (half == 0) bar_arrive(2, 256);
          else if (w + gridDim.x < tiles * S) bar_arrive(4, 256);
        }
        continue;
      }
      float4 cprev[4];
      if (epi.mode == EPI_LSTM_CELL) {
        const uint32_t u = mt * 32 + 4 * (th & 7);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t n = n0 + (th >> 3) + 16 * k;
          cprev[k] = n < N ? ld4(epi.c_prev + u + (size_t)epi.H * n) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
      uint32_t all_ok;
      asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbarrier.cta.red.and.pred p, %2, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                   : "=r"(all_ok) : "r"((uint32_t)ok), "r"(1u + 2u * half) : "memory");
      if (all_ok && (epi.mode == EPI_STORE || epi.mode == EPI_BIAS)) {
        // (5003 x 1050 x 300 with a bias, 4-byte pieces: the pass for every mode took longer than a tile's MMAs, 37.0 us in all, 33.5 here)
        const bool vec = epi_in_pieces(epi, M);
        const uint32_t r = vec ? 4 * (th & 31) : th, c = vec ? th >> 5 : 0, c_hi = m0 + r < M && n0 < N ? min(N - n0, 64u) : 0;
        const EpiRow row = epi_row(epi, min(m0 + r, M - 1));
        float* const dst = row.c + (size_t)row.ldc * (n0 + n_shift);
        const float* bias = epi.bias + min(m0 + r, M - 1);
        if (vec) write_pieces<float4, 4>(epi.mode, stage + r, stage, dst, row.ldc, nullptr, 0, bias, c, c_hi);
        else write_pieces<float, 1>(epi.mode, stage + r, stage, dst, row.ldc, nullptr, 0, bias, c, c_hi);
      } else if (all_ok) {
        epilogue_pass<64, 128>(epi, stage, th, mt, m0, n0 + n_shift, M, N + n_shift, cprev);
      }
      if (BNT == 128) {
        if (half == 0) bar_arrive(2, 256);
        else if (w + gridDim.x < tiles * S) bar_arrive(4, 256);
      }
    }
    if (!ok && lane == 0) atomicOr(flags, DYB200_FLAG_WAIT_TIMEOUT);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kPersistBufs * BN) : "memory");
  }
}

// ---- split-K second stage: C = epilogue(sum_s part[s]) in ascending split order ----------------
__global__ void __launch_bounds__(256) k_splitk_reduce(const float* __restrict__ part, uint32_t S, uint32_t M, uint32_t N,
                                                      GemmEpilogue epi, int vec, size_t stride, const uint32_t* unless) {
  dyb_grid_dep_sync();
  if (unless && *(const volatile uint32_t*)unless) return;
  const size_t MN = (size_t)M * N;
  if (vec) {   // M % 4 == 0 and 16-byte aligned C / mask: four rows of one column per thread
    const size_t MN4 = MN / 4;
    for (size_t q = (size_t)blockIdx.x * 256 + threadIdx.x; q < MN4; q += (size_t)gridDim.x * 256) {
      const size_t e = 4 * q;
      const uint32_t m = (uint32_t)(e % M), n = (uint32_t)(e / M);
      // (eight splits requested at a time: one after another, ten splits of 512 x 4096 took 133 us)
      float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
      for (uint32_t s0 = 0; s0 < S; s0 += 8) {
        float4 v[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) if (s0 + k < S) v[k] = ld4_stream(part + (size_t)(s0 + k) * stride + e);
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
          if (s0 + k >= S) break;
          if (s0 + k == 0) acc = v[0];
          else { acc.x += v[k].x; acc.y += v[k].y; acc.z += v[k].z; acc.w += v[k].w; }
        }
      }
      const EpiRow row = epi_row(epi, m);   // split_m is a multiple of 4 here: the four rows share a destination
      float* dst = row.c + (size_t)row.ldc * n;
      if (epi.mode == EPI_STORE) st4(dst, acc);
      else if (epi.mode == EPI_BIAS) {
        float4 b = ld4(epi.bias + m);
        st4(dst, make_float4(acc.x + b.x, acc.y + b.y, acc.z + b.z, acc.w + b.w));
      } else if (epi.mode == EPI_ACCUM) {
        float4 o = ld4(dst);
        st4(dst, make_float4(o.x + acc.x, o.y + acc.y, o.z + acc.z, o.w + acc.w));
      } else {   // EPI_ACCUM_MASK
        float4 o = ld4(dst), mk = ld4(row.mask + (row.mask_full ? (size_t)row.mask_ld * n : 0));
        st4(dst, make_float4(__fmaf_rn(acc.x, mk.x, o.x), __fmaf_rn(acc.y, mk.y, o.y), __fmaf_rn(acc.z, mk.z, o.z), __fmaf_rn(acc.w, mk.w, o.w)));
      }
    }
    return;
  }
  for (size_t e = (size_t)blockIdx.x * 256 + threadIdx.x; e < MN; e += (size_t)gridDim.x * 256) {
    const uint32_t m = (uint32_t)(e % M), n = (uint32_t)(e / M);
    float acc = 0.f;
    for (uint32_t s2 = 0; s2 < S; ++s2) acc += part[(size_t)s2 * stride + e];
    const EpiRow row = epi_row(epi, m);
    float* dst = row.c + (size_t)row.ldc * n;
    if (epi.mode == EPI_STORE) *dst = acc;
    else if (epi.mode == EPI_BIAS) *dst = acc + epi.bias[m];
    else if (epi.mode == EPI_ACCUM) *dst += acc;
    else if (epi.mode == EPI_GATES) {
      acc += epi.bias[m] + ((m >= epi.H && m < 2 * epi.H) ? epi.forget_bias : 0.f);
      *dst = m < 3 * epi.H ? gate_sigmoid(acc) : gate_tanh(acc);   // (the activations of every gate epilogue)
    } else {
      *dst = __fmaf_rn(acc, row.mask[row.mask_full ? (size_t)row.mask_ld * n : 0], *dst);
    }
  }
}

// Split-K second stage of the LSTM forward product (EPI_LSTM_CELL): rows are the interleaved gate rows of
// dyb200_tc_param_gates.  One thread owns four consecutive hidden units of one column: it adds the partial tiles in
// split order, applies bias + sigmoid / tanh, writes the four gate rows and forms c and h.
__global__ void __launch_bounds__(256) k_splitk_reduce_cell(const float* __restrict__ part, uint32_t S, uint32_t M, uint32_t N,
                                                           GemmEpilogue epi) {
  dyb_grid_dep_sync();
  const uint32_t H = epi.H, H4 = H / 4;
  const size_t MN = (size_t)M * N, total = (size_t)H4 * N;
  for (size_t q = (size_t)blockIdx.x * 256 + threadIdx.x; q < total; q += (size_t)gridDim.x * 256) {
    const uint32_t u = 4 * (uint32_t)(q % H4), n = (uint32_t)(q / H4);
    const uint32_t row0 = 128 * (u / 32) + (u % 32);   // interleaved row of gate 0; gate g is 32 g rows further
    float4 a[4];
    // all loads of up to four splits are issued before the first add (this kernel is latency-bound at small batch)
    for (uint32_t s0 = 0; s0 < S; s0 += 4) {
      float4 v[4][4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int g = 0; g < 4; ++g)
          v[k][g] = s0 + k < S ? ld4_stream(part + row0 + 32 * g + (size_t)M * n + (size_t)(s0 + k) * MN) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        if (s0 == 0) a[g] = v[0][g];
        else { a[g].x += v[0][g].x; a[g].y += v[0][g].y; a[g].z += v[0][g].z; a[g].w += v[0][g].w; }
#pragma unroll
        for (int k = 1; k < 4; ++k)
          if (s0 + k < S) { a[g].x += v[k][g].x; a[g].y += v[k][g].y; a[g].z += v[k][g].z; a[g].w += v[k][g].w; }
      }
    }
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const float4 b = ld4(epi.bias + (size_t)g * H + u);
      const float fb = g == 1 ? epi.forget_bias : 0.f;
      a[g].x += b.x + fb; a[g].y += b.y + fb; a[g].z += b.z + fb; a[g].w += b.w + fb;
      if (g == 3) a[g] = make_float4(gate_tanh(a[g].x), gate_tanh(a[g].y), gate_tanh(a[g].z), gate_tanh(a[g].w));
      else a[g] = make_float4(gate_sigmoid(a[g].x), gate_sigmoid(a[g].y), gate_sigmoid(a[g].z), gate_sigmoid(a[g].w));
      st4(epi.C + (size_t)g * H + u + (size_t)epi.ldc * n, a[g]);
    }
    const size_t e = u + (size_t)H * n;
    const float4 cp = ld4(epi.c_prev + e);
    const float4 c = make_float4(lstm_cell_c(a[0].x, a[3].x, a[1].x, cp.x), lstm_cell_c(a[0].y, a[3].y, a[1].y, cp.y),
                                 lstm_cell_c(a[0].z, a[3].z, a[1].z, cp.z), lstm_cell_c(a[0].w, a[3].w, a[1].w, cp.w));
    st4(epi.c_out + e, c);
    const float4 hv = make_float4(lstm_cell_h(a[2].x, c.x), lstm_cell_h(a[2].y, c.y), lstm_cell_h(a[2].z, c.z), lstm_cell_h(a[2].w, c.w));
    st4(epi.h_out + e, hv);
    if (epi.hn_hi) epi_emit_h(epi, u, n, hv);
  }
}

// ---- operand packing: fp32 (masked, possibly transposed) -> K-major hi / lo planes ------------
// One launch packs up to kMaxPackJobs operands.  A job is cut into units of one CTA each: for a source whose
// k index is fast (element (r, k) at src[k + ld * r]) a unit is 1024 consecutive k of one row; for a source whose
// row index is fast (element (r, k) at src[r + ld * k]) a unit is a 32 x 32 tile transposed through shared memory.
__global__ void __launch_bounds__(256) k_pack_multi(const PackJobs jobs) {
  dyb_grid_dep_sync();
  __shared__ float tile[32][33];
  int j = 0;
#pragma unroll
  for (int q = 1; q < kMaxPackJobs; ++q) if (q < jobs.n && blockIdx.x >= jobs.start[q]) j = q;
  const PackJob& job = jobs.job[j];
  const uint32_t unit = blockIdx.x - jobs.start[j];
  const float* __restrict__ src = job.src;
  const float* __restrict__ mask = job.mask;
  float* __restrict__ hi = job.hi;
  float* __restrict__ lo = job.lo;
  const uint32_t ld = job.ld, rows = job.rows, K = job.K, pitch = job.pitch, mask_ld = job.mask_ld;
  const int mask_full = job.mask_full;
  const uint32_t mask_period = job.mask_period;
  if (job.k_is_fast) {
    if (job.vec) {
      // rows end to end, 1024 float4 per CTA whatever their length: a CTA for each row of 256 values (64 of its threads at work)
      // took 111 us for 107 000 rows
      const uint32_t K4 = K / 4;
      const uint64_t e0 = (uint64_t)unit * 1024;
      const uint32_t first = (uint32_t)(e0 / K4), rem = (uint32_t)(e0 - (uint64_t)first * K4);
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t e = rem + 256 * i + threadIdx.x, r = first + e / K4, k = 4 * (e % K4);
        if (r >= rows) break;
        const uint32_t mr = mask_period ? r % mask_period : r;   // batch column of the mask
        float4 v = ld4(src + k + (size_t)ld * r);
        if (mask) {
          float4 mk = ld4(mask + k + (mask_full ? (size_t)mask_ld * mr : 0));
          v.x *= mk.x; v.y *= mk.y; v.z *= mk.z; v.w *= mk.w;
        }
        float4 h, l;
        split_tf32(v.x, h.x, l.x); split_tf32(v.y, h.y, l.y); split_tf32(v.z, h.z, l.z); split_tf32(v.w, h.w, l.w);
        st4(hi + k + (size_t)pitch * r, h);
        st4(lo + k + (size_t)pitch * r, l);
      }
    } else {
      const uint32_t r = unit / job.gx, bx = unit % job.gx, mr = mask_period ? r % mask_period : r;
      for (uint32_t k = bx * 1024 + threadIdx.x; k < min(K, (bx + 1) * 1024); k += 256) {
        float v = src[k + (size_t)ld * r];
        if (mask) v *= mask[k + (mask_full ? (size_t)mask_ld * mr : 0)];
        float h, l;
        split_tf32(v, h, l);
        hi[k + (size_t)pitch * r] = h;
        lo[k + (size_t)pitch * r] = l;
      }
    }
    return;
  }
  const uint32_t r0 = (unit % job.gx) * 32, k0 = (unit / job.gx) * 32;
  const uint32_t tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t r = r0 + tx, k = k0 + ty + 8 * i;
    float v = 0.f;
    if (r < rows && k < K) {
      v = src[r + (size_t)ld * k];
      if (mask) v *= mask[r + (mask_full ? (size_t)mask_ld * (mask_period ? k % mask_period : k) : 0)];
    }
    tile[ty + 8 * i][tx] = v;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    uint32_t r = r0 + ty + 8 * i, k = k0 + tx;
    if (r < rows && k < K) {
      float h, l;
      split_tf32(tile[tx][ty + 8 * i], h, l);
      uint32_t rd = r;
      if (job.perm_H) { const uint32_t q = r / job.perm_H, u = r % job.perm_H; rd = 128 * (u / 32) + 32 * q + (u % 32); }
      hi[k + (size_t)pitch * rd] = h;
      lo[k + (size_t)pitch * rd] = l;
    }
  }
}

// ---- fp16 operand planes: the largest |x| per line, per position or in all, then the split ---------------------------------
// Both passes read the source once; a line of a wide operand is shared by several CTAs, maxima meet by atomicMax on the bit
// patterns (the same from run to run).  Infinities and NaNs do not count: they come through the split as they are.
// A unit of work is one CTA's; the 16-byte loads of a batch are requested together (behind a branch per load they went out one by one:
// 219 instead of 122 us for the scales of 50000 x 4096, 433 instead of 282 us for its split).
constexpr uint32_t kMaxLines = 64;      // F16_ELEM: lines of each thread
constexpr uint32_t kWarpLine = 2048;    // F16_LINE: lines up to this length are a warp's, kWarpLines of them; longer ones go in pieces of kPiece
constexpr uint32_t kWarpLines = 4, kPiece = 8192;
struct F16Units { uint32_t groups, x, total; };   // F16_ELEM: groups of threads with lines of their own, units along the line
__host__ __device__ __forceinline__ F16Units f16_max_units(const F16Job& j) {
  F16Units u;
  u.groups = 1; u.x = 1;
  if (j.mode == F16_ELEM) {
    const uint32_t q = (j.n + 3) / 4;
    u.groups = q < 256 ? 256 / q : 1;
    u.x = (q + 255) / 256;
    u.total = u.x * ((j.lines + kMaxLines * u.groups - 1) / (kMaxLines * u.groups));
  } else if (j.n <= kWarpLine) {
    u.total = (j.lines + 8 * kWarpLines - 1) / (8 * kWarpLines);
  } else {
    u.x = (j.n + kPiece - 1) / kPiece;
    u.total = u.x * j.lines;
  }
  return u;
}
__device__ __forceinline__ uint32_t f16_job_of(const F16Jobs& jobs) {
  uint32_t z = 0;
#pragma unroll
  for (int q = 1; q < kF16MaxJobs; ++q) if (q < jobs.n && blockIdx.x >= jobs.start[q]) z = q;
  return z;
}
__device__ __forceinline__ uint32_t mag4(float4 v) { return max(max(finite_mag(v.x), finite_mag(v.y)), max(finite_mag(v.z), finite_mag(v.w))); }
// elements [e, e + 4) of a line of n (zeros past its end)
__device__ __forceinline__ float4 f16_load4(const float* line, uint32_t e, uint32_t n, bool vec) {
  if (vec && e + 4 <= n) return ld4(line + e);
  float v[4];
#pragma unroll
  for (uint32_t i = 0; i < 4; ++i) v[i] = e + i < n ? line[e + i] : 0.f;
  return make_float4(v[0], v[1], v[2], v[3]);
}
// LOW: jobs with `low` words (F16Jobs::wide).
template <bool LOW>
__global__ void __launch_bounds__(256) k_f16_absmax(const __grid_constant__ F16Jobs jobs) {
  dyb_grid_dep_sync();
  const uint32_t z = f16_job_of(jobs), unit = blockIdx.x - jobs.start[z];
  const F16Job& j = jobs.job[z];
  const bool vec = (j.ld & 3) == 0 && aligned16(j.src);
  const F16Units us = f16_max_units(j);
  if (j.mode == F16_ELEM) {   // four positions per thread; short lines: groups of threads with lines of their own meet in shared memory
    __shared__ uint32_t top[1024], bot[LOW ? 1024 : 1];
    const uint32_t q = us.groups > 1 ? (j.n + 3) / 4 : 256u, grp = threadIdx.x / q, e = 4 * ((unit % us.x) * 256 + threadIdx.x % q);
    const uint32_t l0 = (unit / us.x * us.groups + grp) * kMaxLines;
    const bool live = grp < us.groups && e < j.n;
    uint32_t m[4] = {0, 0, 0, 0}, low[4] = {0, 0, 0, 0};   // low: ~(the smallest of the blocks' maxima that are not zero)
    if (live) {
      for (uint32_t b = 0; b < kMaxLines && l0 + b < j.lines; b += 8) {
        float4 v[8];
        const uint32_t l = l0 + b;
        const float* p = j.src + (size_t)j.ld * l;
        if (vec && e + 4 <= j.n && l + 7 < j.lines) {
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k) v[k] = ld4(p + (size_t)j.ld * k + e);
        } else {
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k) v[k] = l + k < j.lines ? f16_load4(p + (size_t)j.ld * k, e, j.n, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
          w[0] = max(w[0], finite_mag(v[k].x)); w[1] = max(w[1], finite_mag(v[k].y)); w[2] = max(w[2], finite_mag(v[k].z)); w[3] = max(w[3], finite_mag(v[k].w));
        }
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) { m[i] = max(m[i], w[i]); if (LOW && w[i]) low[i] = max(low[i], ~w[i]); }
      }
    }
    if (us.groups > 1) {
      for (uint32_t i = threadIdx.x; i < 1024; i += 256) { top[i] = 0; if (LOW) bot[i] = 0; }
      __syncthreads();
      if (live) {
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) { atomicMax(top + e + i, m[i]); if (LOW) atomicMax(bot + e + i, low[i]); }
      }
      __syncthreads();
      for (uint32_t i = threadIdx.x; i < j.n; i += 256) { atomicMax(j.scale + i, top[i]); if (LOW) atomicMax(j.low + i, bot[i]); }
    } else if (live) {
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i)
        if (e + i < j.n) { atomicMax(j.scale + e + i, m[i]); if (LOW) atomicMax(j.low + e + i, low[i]); }
    }
    return;
  }
  if (j.n <= kWarpLine) {
    const uint32_t lane = threadIdx.x & 31, l0 = (unit * 8 + (threadIdx.x >> 5)) * kWarpLines;
    uint32_t m[kWarpLines] = {0, 0, 0, 0};
    for (uint32_t e = 4 * lane; e < j.n; e += 256) {
      float4 v[kWarpLines][2];
      if (vec && e + 132 <= j.n && l0 + kWarpLines <= j.lines) {
#pragma unroll
        for (uint32_t k = 0; k < kWarpLines; ++k)
#pragma unroll
          for (uint32_t h = 0; h < 2; ++h) v[k][h] = ld4(j.src + (size_t)j.ld * (l0 + k) + e + 128 * h);
      } else {
#pragma unroll
        for (uint32_t k = 0; k < kWarpLines; ++k)
#pragma unroll
          for (uint32_t h = 0; h < 2; ++h)
            v[k][h] = l0 + k < j.lines ? f16_load4(j.src + (size_t)j.ld * (l0 + k), e + 128 * h, j.n, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (uint32_t k = 0; k < kWarpLines; ++k) m[k] = max(m[k], max(mag4(v[k][0]), mag4(v[k][1])));
    }
#pragma unroll
    for (uint32_t k = 0; k < kWarpLines; ++k) {
      m[k] = __reduce_max_sync(0xffffffffu, m[k]);
      if (lane == 0 && l0 + k < j.lines) j.scale[l0 + k] = m[k] & ~j.mark;
    }
    return;
  }
  __shared__ uint32_t red[8];
  const uint32_t line = unit / us.x, e0 = unit % us.x * kPiece + 4 * threadIdx.x;
  float4 v[8];
  const float* p = j.src + (size_t)j.ld * line;
  if (vec && e0 + 7 * 1024 + 4 <= j.n) {
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) v[k] = ld4(p + e0 + 1024 * k);
  } else {
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) v[k] = f16_load4(p, e0 + 1024 * k, j.n, vec);
  }
  uint32_t m = 0;
#pragma unroll
  for (uint32_t k = 0; k < 8; ++k) m = max(m, mag4(v[k]));
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) m = max(m, red[w]);
    m &= ~j.mark;
    if (us.x == 1) j.scale[line] = m; else atomicMax(j.scale + line, m);
  }
}
__device__ __forceinline__ void split4_f16(float4 v, float4 s, uint2& hi, uint2& lo) {
  __half h[4], l[4];
  split_f16(v.x * s.x, h[0], l[0]); split_f16(v.y * s.y, h[1], l[1]); split_f16(v.z * s.z, h[2], l[2]); split_f16(v.w * s.w, h[3], l[3]);
  hi = *reinterpret_cast<const uint2*>(h);
  lo = *reinterpret_cast<const uint2*>(l);
}
// Positions [e, + 4) of a line to the planes: as they lie, or those of gate rows where they go (F16Job::perm_H; four units of a gate stay together
// where the units come in fours).  The pitch is a multiple of 64: the last item's padding stays inside the line's pitch.
__device__ __forceinline__ void store_pairs(const F16Job& j, uint32_t line, uint32_t e, uint2 hi, uint2 lo) {
  __half *ph = j.hi + (size_t)j.pitch * line, *pl = j.lo + (size_t)j.pitch * line;
  auto perm = [&](uint32_t x) { const uint32_t g = x / j.perm_H, u = x % j.perm_H; return 128 * (u / 32) + 32 * g + u % 32; };
  if (j.perm_H && (j.perm_H & 3)) {
    const __half *h = reinterpret_cast<const __half*>(&hi), *l = reinterpret_cast<const __half*>(&lo);
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i)
      if (e + i < j.n) { const uint32_t to = perm(e + i); ph[to] = h[i]; pl[to] = l[i]; }
    return;
  }
  if (j.perm_H) e = perm(e);
  *reinterpret_cast<uint2*>(ph + e) = hi;
  *reinterpret_cast<uint2*>(pl + e) = lo;
}
// A unit: kSplitItems items of four values, the lines end to end.  (A pair of planes is added up, hi + lo: the fp32 value that it stands for.)
constexpr uint32_t kSplitItems = 1024;
__global__ void __launch_bounds__(256) k_f16_split(const __grid_constant__ F16Jobs jobs) {
  dyb_grid_dep_sync();
  const uint32_t z = f16_job_of(jobs), unit = blockIdx.x - jobs.start[z];
  const F16Job& j = jobs.job[z];
  const bool vec = (j.ld & 3) == 0 && aligned16(j.src) && (!j.src_lo || aligned16(j.src_lo));
  const uint32_t q = (j.n + 3) / 4;
  const uint64_t first = (uint64_t)unit * kSplitItems;
  const uint32_t line0 = (uint32_t)(first / q), rem = (uint32_t)(first - (uint64_t)line0 * q);
  float4 v[4];
  uint32_t line[4], e[4];
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) {
    const uint32_t it = rem + 256 * k + threadIdx.x;
    line[k] = line0 + it / q; e[k] = 4 * (it % q);
  }
  // (the last item is the furthest in the source; lines that are whole quads: one straight set of loads)
  const bool plain = vec && (j.n & 3) == 0 && line[3] < j.lines;
  if (plain) {
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) v[k] = ld4(j.src + (size_t)j.ld * line[k] + e[k]);
  } else {
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) v[k] = line[k] < j.lines ? f16_load4(j.src + (size_t)j.ld * line[k], e[k], j.n, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (j.src_lo) {
    float4 w[4];
    if (plain) {
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) w[k] = ld4(j.src_lo + (size_t)j.ld * line[k] + e[k]);
    } else {
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) w[k] = line[k] < j.lines ? f16_load4(j.src_lo + (size_t)j.ld * line[k], e[k], j.n, vec) : v[k];
    }
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) v[k] = make_float4(v[k].x + w[k].x, v[k].y + w[k].y, v[k].z + w[k].z, v[k].w + w[k].w);
  }
#pragma unroll
  for (uint32_t k = 0; k < 4; ++k) {
    if (line[k] >= j.lines) break;
    float4 s;
    if (j.low && line[k] == 0) {   // (a position's words are looked at where its first line is split)
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i) {
        const uint32_t p = min(e[k] + i, j.n - 1), low = j.low[p];
        if (low && (j.scale[p] >> 23) > ((~low) >> 23) + kF16Span) *jobs.wide = 1;
      }
    }
    if (j.mode == F16_ELEM) {
      const uint32_t top = j.n - 1;
      if (e[k] + 4 <= j.n) {
        const uint4 w = __ldg(reinterpret_cast<const uint4*>(j.scale + e[k]));
        s = make_float4(scale_of(w.x), scale_of(w.y), scale_of(w.z), scale_of(w.w));
      } else {
        s = make_float4(scale_of(__ldg(j.scale + min(e[k], top))), scale_of(__ldg(j.scale + min(e[k] + 1, top))), scale_of(__ldg(j.scale + min(e[k] + 2, top))), 1.f);
      }
    } else {
      const uint32_t word = j.mark ? __ldcg(j.scale + line[k]) : __ldg(j.scale + line[k]);   // (bit 0 may be set meanwhile)
      s.x = s.y = s.z = s.w = scale_of(word);
      if (j.mark && pair_loses(mag4(v[k]), word)) { v[k] = make_float4(0.f, 0.f, 0.f, 0.f); atomicOr(j.scale + line[k], 1u); }
    }
    uint2 hi, lo;
    split4_f16(v[k], s, hi, lo);
    store_pairs(j, line[k], e[k], hi, lo);
  }
}

// ---- both in one pass, for operands whose rows fit into registers between the scale and the split ----
// (The passes above read an operand twice and are two launches and a clear.  us, those / one pass: gate weights of 1024 + 1024 columns x 4096 (34 MB) 28 / 17, 1024 lines of
// 10 000 positions (41 MB) 27 / 22, 1024 lines of 4096 11 / 7, of 10 000 24 / 17.  Strips of 32 positions store 64-byte pieces: from memory, not L2, that is the
// slower form, 512 lines of 50 000 positions 60 / 94.)
// Positions: a CTA takes strips of 32 positions, 128 bytes of every line; thread -> positions [p, p + 4) of the lines t / 8, t / 8 + 32, ...
template <int R, bool ODD = false>   // (ODD: gate rows whose units do not come in fours.  As a branch of the same kernel it cost the others 10 - 20 of 15 - 22 us)
__global__ void __launch_bounds__(256) k_f16_strip(const __grid_constant__ F16Jobs jobs) {
  dyb_grid_dep_sync();
  __shared__ uint32_t top[8][32];
  const uint32_t z = f16_job_of(jobs), unit = blockIdx.x - jobs.start[z];
  const F16Job& j = jobs.job[z];
  const bool vec = (j.ld & 3) == 0 && aligned16(j.src);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, q = 4 * (threadIdx.x & 7), e = 32 * unit + q, l0 = threadIdx.x >> 3;
  float4 v[R];
  if (vec && e + 4 <= j.n && j.lines >= 32 * R) {
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = ld4(j.src + (size_t)j.ld * (l0 + 32 * k) + e);
  } else {
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = l0 + 32 * k < j.lines && e < j.n ? f16_load4(j.src + (size_t)j.ld * (l0 + 32 * k), e, j.n, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  uint32_t m[4] = {0, 0, 0, 0};
#pragma unroll
  for (int k = 0; k < R; ++k) {
    m[0] = max(m[0], finite_mag(v[k].x)); m[1] = max(m[1], finite_mag(v[k].y)); m[2] = max(m[2], finite_mag(v[k].z)); m[3] = max(m[3], finite_mag(v[k].w));
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m[i] = max(m[i], __shfl_xor_sync(0xffffffffu, m[i], 8));
    m[i] = max(m[i], __shfl_xor_sync(0xffffffffu, m[i], 16));
    if (lane < 8) top[warp][q + i] = m[i];
  }
  __syncthreads();
  float s[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int w = 0; w < 8; ++w) m[i] = max(m[i], top[w][q + i]);
    s[i] = scale_of(m[i]);
    if (threadIdx.x < 8 && e + i < j.n) j.scale[e + i] = m[i];
  }
  if (e >= j.n) return;
  uint32_t to = e;
  if (j.perm_H && !ODD) { const uint32_t g = e / j.perm_H, u = e % j.perm_H; to = 128 * (u / 32) + 32 * g + u % 32; }   // (once, not line by line)
#pragma unroll
  for (int k = 0; k < R; ++k) {
    const uint32_t line = l0 + 32 * k;
    if (line >= j.lines) break;
    uint2 hi, lo;
    split4_f16(v[k], make_float4(s[0], s[1], s[2], s[3]), hi, lo);
    if (ODD) { store_pairs(j, line, e, hi, lo); continue; }
    *reinterpret_cast<uint2*>(j.hi + (size_t)j.pitch * line + to) = hi;
    *reinterpret_cast<uint2*>(j.lo + (size_t)j.pitch * line + to) = lo;
  }
}
// Lines: a warp per line of up to 1024 values, a CTA per longer one.
constexpr uint32_t kOneLine = kF16PadMax, kOneStrip = 1024;   // longest line, most lines of a strip
template <uint32_t R, bool PAD, bool MARK>
__device__ __forceinline__ void line_pairs(const F16Job& j, uint32_t line, uint32_t e0, uint32_t step, uint32_t* red) {
  const float* p = j.src + (size_t)j.ld * line;
  const bool vec = aligned16(p);
  float4 v[R];
  if (vec && e0 + (R - 1) * step + 4 <= j.n) {
#pragma unroll
    for (uint32_t k = 0; k < R; ++k) v[k] = ld4(p + e0 + step * k);
  } else {
#pragma unroll
    for (uint32_t k = 0; k < R; ++k) v[k] = e0 + step * k < j.n ? f16_load4(p, e0 + step * k, j.n, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  uint32_t m = 0;
#pragma unroll
  for (uint32_t k = 0; k < R; ++k) m = max(m, mag4(v[k]));
  m = __reduce_max_sync(0xffffffffu, m);
  if (red) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) m = max(m, red[w]);
  }
  if (MARK && j.mark) {
    bool loses = false;
#pragma unroll
    for (uint32_t k = 0; k < R; ++k)
      if (pair_loses(mag4(v[k]), m)) { v[k] = make_float4(0.f, 0.f, 0.f, 0.f); loses = true; }
    loses = red ? __syncthreads_or(loses) : __any_sync(0xffffffffu, loses);
    m = (m & ~1u) | loses;
  }
  if (e0 == 0) j.scale[line] = m;
  const float s = scale_of(m);
#pragma unroll
  for (uint32_t k = 0; k < R; ++k) {
    const uint32_t e = e0 + step * k;
    if (e >= j.n) break;
    uint2 hi, lo;
    split4_f16(v[k], make_float4(s, s, s, s), hi, lo);
    __half *ph = j.hi + (size_t)j.pitch * line, *pl = j.lo + (size_t)j.pitch * line;
    if (PAD && j.pad_H) {
      const __half *h = reinterpret_cast<const __half*>(&hi), *l = reinterpret_cast<const __half*>(&lo);
      const uint32_t gap = (j.pad_H + 63) / 64 * 64 - j.pad_H;
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i)
        if (e + i < j.n) { const uint32_t to = e + i + (e + i) / j.pad_H * gap; ph[to] = h[i]; pl[to] = l[i]; }
    } else {
      *reinterpret_cast<uint2*>(ph + e) = hi;
      *reinterpret_cast<uint2*>(pl + e) = lo;
    }
  }
  if (PAD && j.pad_H) {   // (the product meets zeros of the other operand here: any finite value would do)
    const uint32_t Hp = (j.pad_H + 63) / 64 * 64, gap = Hp - j.pad_H;
    for (uint32_t x = e0 / 4; x < 4 * gap; x += step / 4) {
      const size_t to = (size_t)j.pitch * line + x / gap * Hp + j.pad_H + x % gap;
      j.hi[to] = j.lo[to] = __float2half_rn(0.f);
    }
  }
}
template <uint32_t R, bool PAD, bool MARK>   // (R 16: lines of more than 8192; PAD, MARK: jobs with pad_H, with mark - registers that the others do without, 95 against 80)
__global__ void __launch_bounds__(256) k_f16_line(const __grid_constant__ F16Jobs jobs) {
  dyb_grid_dep_sync();
  __shared__ uint32_t red[8];
  const uint32_t z = f16_job_of(jobs), unit = blockIdx.x - jobs.start[z];
  const F16Job& j = jobs.job[z];
  if (j.n > 1024) {
    line_pairs<R, PAD, MARK>(j, unit, 4 * threadIdx.x, 1024, red);
  } else {
    const uint32_t line = 8 * unit + (threadIdx.x >> 5);
    if (line < j.lines) line_pairs<8, PAD, MARK>(j, line, 4 * (threadIdx.x & 31), 128, nullptr);
  }
}
constexpr uint64_t kOneValues = 12u << 20;   // (48 MB and as much again of pairs: L2 still holds most of both)
bool f16_one_pass(const F16Job& j) { return !j.src_lo && !j.low && (j.mode == F16_ELEM ? j.lines <= kOneStrip && (uint64_t)j.lines * j.n <= kOneValues : j.n <= kOneLine); }

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int get_encoder(dyb200_ctx* ctx, EncodeTiledFn* fn) {
  if (!ctx->encode_tiled) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    DYB_CUDA(ctx, cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    if (q != cudaDriverEntryPointSuccess || !p) return dyb200_fail(ctx, DYB200_ECUDA, "cuTensorMapEncodeTiled is not available in this driver");
    ctx->encode_tiled = p;
  }
  *fn = (EncodeTiledFn)ctx->encode_tiled;
  return DYB200_OK;
}

// Plane of `rows` rows and K valid floats per row, row pitch `pitch` floats; box = 32 (k) x 128 (rows).
int make_map(dyb200_ctx* ctx, EncodeTiledFn enc, CUtensorMap* map, float* plane, uint32_t rows, uint32_t K, uint32_t pitch,
             uint32_t box_rows = BM, bool f16 = false) {
  cuuint64_t dims[2] = {K, rows};
  cuuint64_t strides[1] = {(cuuint64_t)pitch * (f16 ? 2 : 4)};
  cuuint32_t box[2] = {f16 ? 64u : 32u, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, plane, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return dyb200_fail(ctx, DYB200_ECUDA, "cuTensorMapEncodeTiled failed with code %d (rows %u, K %u, pitch %u)", (int)r, rows, K, pitch);
  return DYB200_OK;
}

// MN-major plane: element (m, k) at plane[k * pitch + m], `rows` valid m and K valid k, as a 3-D tensor (m within a group
// of 32, k, group): one box = 4 groups x 32 k x 32 m, in the 128-byte swizzle with 32-byte atoms that umma_desc_mn describes.
// The last group may reach past `rows` into the pitch (those rows of the product are never stored).
int make_map_mn(dyb200_ctx* ctx, EncodeTiledFn enc, CUtensorMap* map, float* plane, uint32_t rows, uint32_t K, uint32_t pitch,
                uint32_t box_rows = BM, bool f16 = false) {
  // (32 m, k, group of 32 m): one box brings box_rows / 32 groups x 32 k rows x 128 bytes, group after group; F16: 64 of each, in
  // the plain 128-byte swizzle
  const uint32_t el = f16 ? 64u : 32u;
  cuuint64_t dims[3] = {el, K, (rows + el - 1) / el};
  cuuint64_t strides[2] = {(cuuint64_t)pitch * (f16 ? 2 : 4), 128};
  cuuint32_t box[3] = {el, el, box_rows / el};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, plane, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, f16 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return dyb200_fail(ctx, DYB200_ECUDA, "cuTensorMapEncodeTiled failed with code %d (MN-major, rows %u, K %u, pitch %u)", (int)r, rows, K, pitch);
  return DYB200_OK;
}

int pack_flush_impl(dyb200_ctx* ctx, PackJobs* jobs) {
  if (jobs->n == 0) return DYB200_OK;
  const uint32_t total = jobs->start[jobs->n];
  dyb_launch(k_pack_multi, total, 256, 0, ctx, *jobs);
  jobs->n = 0;
  jobs->start[0] = 0;
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

// Queues one operand in `batch` (launching the queue first when it is full); with batch == nullptr it is packed at once.
// layout: 0 = the row index is fast in the source, 1 = the k index is fast, kLayoutGates = row index fast and the
// rows = 4H gate rows are written interleaved (destination row 128 t + 32 q + l <- source row q H + 32 t + l) so that
// every 128-row tile holds the four gates of 32 hidden units.
int pack(dyb200_ctx* ctx, const float* src, uint32_t ld, int layout, uint32_t rows, uint32_t K, const float* mask,
         uint32_t mask_ld, int mask_full, float* hi, float* lo, uint32_t pitch, PackJobs* batch = nullptr,
         uint32_t mask_period = 0) {
  const bool k_is_fast = layout == 1;
  if (rows == 0 || K == 0) return DYB200_OK;
  PackJobs local;
  local.n = 0; local.start[0] = 0;
  PackJobs* q = batch ? batch : &local;
  if (q->n == kMaxPackJobs) { int rc = pack_flush_impl(ctx, q); if (rc) return rc; }
  PackJob& j = q->job[q->n];
  j.src = src; j.mask = mask; j.hi = hi; j.lo = lo;
  j.ld = ld; j.rows = rows; j.K = K; j.mask_ld = mask_ld; j.pitch = pitch;
  j.k_is_fast = k_is_fast ? 1 : 0; j.mask_full = mask_full; j.mask_period = mask_period;
  j.perm_H = layout == kLayoutGates ? rows / 4 : 0;
  uint64_t units;
  if (k_is_fast) {
    j.vec = (K % 4 == 0) && (ld % 4 == 0) && aligned16(src) && (!mask || ((mask_ld % 4 == 0 || !mask_full) && aligned16(mask)));
    j.gx = (K + 1023) / 1024;
    units = j.vec ? ((uint64_t)(K / 4) * rows + 1023) / 1024 : (uint64_t)j.gx * rows;
  } else {
    j.vec = 0;
    j.gx = (rows + 31) / 32;
    units = (uint64_t)j.gx * ((K + 31) / 32);
  }
  DYB_CHECK_ARG(ctx, (uint64_t)q->start[q->n] + units < 0x7fffffffull, "pack: operand too large (%u x %u)", rows, K);
  q->start[q->n + 1] = q->start[q->n] + (uint32_t)units;
  q->n++;
  return batch ? DYB200_OK : pack_flush_impl(ctx, q);
}

inline uint32_t round_up(uint32_t x, uint32_t m) { return (x + m - 1) / m * m; }

// fp16 planes of the gate weights (F16Gates): I lines of Wx, then H lines of Wh, the scale words in the same order.  A line is tiles of 32 units, 128 rows.
inline uint32_t gates_f16_pitch(uint32_t H) { return 128 * ((H + 31) / 32); }
int gates_f16_pack(dyb200_ctx* ctx, const float* Wx, const float* Wh, uint32_t I, uint32_t H, __half* hi, __half* lo, uint32_t* scale) {
  F16Jobs jobs;
  jobs.n = 2;
  for (int q = 0; q < 2; ++q) {
    const size_t at = q ? (size_t)I * gates_f16_pitch(H) : 0;
    jobs.job[q] = F16Job{q ? Wh : Wx, 4 * H, q ? H : I, 4 * H, gates_f16_pitch(H), F16_ELEM, scale + q * 4 * H, hi + at, lo + at};
    jobs.job[q].perm_H = H;
  }
  jobs.words = scale; jobs.n_words = 8 * (size_t)H;
  return dyb200_f16_pack(ctx, &jobs);
}

// Returns the cached packed form of a parameter matrix, packing it first if it is new or stale (3xTF32 planes: as jobs of `queue` if there is
// one; the entry then counts as packed, and a caller that does not launch the queue, or fails to, makes the cache stale).
// (k_is_fast = kLayoutF16 + F16_LINE or F16_ELEM: fp16 planes of the matrix as it lies, its scale words behind the hi plane)
int cached_param_pack(dyb200_ctx* ctx, const float* src, uint32_t ld, int k_is_fast, uint32_t rows, uint32_t K, uint32_t pitch,
                      float** hi, float** lo, const float* src2 = nullptr, uint32_t rows2 = 0, PackJobs* queue = nullptr) {
  const int cap = (int)(sizeof(ctx->param_pack) / sizeof(ctx->param_pack[0]));
  dyb200_ctx::ParamPack* hit = nullptr;
  dyb200_ctx::ParamPack* victim = &ctx->param_pack[0];
  for (int k = 0; k < cap; ++k) {
    dyb200_ctx::ParamPack* e = &ctx->param_pack[k];
    if (e->hi && e->src == src && e->src2 == src2 && e->rows2 == rows2 && e->ld == ld && e->rows == rows && e->K == K && e->k_is_fast == (int)k_is_fast) { hit = e; break; }
    if (!e->hi) { if (victim->hi) victim = e; }
    else if (victim->hi && e->last_use < victim->last_use) victim = e;
  }
  dyb200_ctx::ParamPack* e = hit ? hit : victim;
  const size_t floats = k_is_fast == kLayoutGatesF16 ? (size_t)(K + rows2) * pitch / 2 + 2 * rows : k_is_fast >= kLayoutF16 ? (size_t)rows * pitch / 2 + (k_is_fast == kLayoutF16 + F16_LINE || k_is_fast >= kLayoutPadF16 ? rows : K) : (size_t)(rows + rows2) * pitch;
  if (!hit) {
    if (e->hi && e->floats < floats) {   // evicted entry is too small: its buffers may still be read by queued kernels
      DYB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      cudaFree(e->hi); cudaFree(e->lo);
      e->hi = e->lo = nullptr;
    }
    if (!e->hi) {
      if (cudaMalloc((void**)&e->hi, floats * sizeof(float)) != cudaSuccess || cudaMalloc((void**)&e->lo, floats * sizeof(float)) != cudaSuccess) {
        cudaGetLastError();
        if (e->hi) cudaFree(e->hi);
        e->hi = e->lo = nullptr;
        return dyb200_fail(ctx, DYB200_ENOMEM, "parameter cache: cudaMalloc of %zu bytes failed", 2 * floats * sizeof(float));
      }
      e->floats = floats;
    }
    e->src = src; e->src2 = src2; e->rows2 = rows2; e->ld = ld; e->rows = rows; e->K = K; e->pitch = pitch; e->k_is_fast = (int)k_is_fast;
    e->version = ~0ull;
  }
  if (e->version != ctx->param_version && k_is_fast == kLayoutGatesF16) {   // (rows2 = columns of the second matrix)
    int rc = gates_f16_pack(ctx, src, src2, K, rows2, (__half*)e->hi, (__half*)e->lo, reinterpret_cast<uint32_t*>(e->hi + (size_t)(K + rows2) * pitch / 2));
    if (rc) return rc;
    e->version = ctx->param_version;
  } else if (e->version != ctx->param_version && k_is_fast >= kLayoutF16) {
    F16Jobs jobs;
    jobs.n = 1;
    const bool pad = k_is_fast == kLayoutPadF16, mark = k_is_fast >= kLayoutPadF16;
    jobs.job[0] = F16Job{src, ld, rows, K, pitch, mark ? (int)F16_LINE : k_is_fast - kLayoutF16, reinterpret_cast<uint32_t*>(e->hi + (size_t)rows * pitch / 2), (__half*)e->hi, (__half*)e->lo};
    if (pad) jobs.job[0].pad_H = K / 4;
    jobs.job[0].mark = mark;
    int rc = dyb200_f16_pack(ctx, &jobs);
    if (rc) return rc;
    e->version = ctx->param_version;
  } else if (e->version != ctx->param_version) {
    PackJobs own;
    dyb200_tc_pack_begin(&own);
    PackJobs* const batch = queue ? queue : &own;
    int rc = pack(ctx, src, ld, k_is_fast, rows, K, nullptr, 0, 0, e->hi, e->lo, pitch, batch);
    if (!rc && rows2) rc = pack(ctx, src2, ld, k_is_fast, rows2, K, nullptr, 0, 0, e->hi + (size_t)rows * pitch, e->lo + (size_t)rows * pitch, pitch, batch);
    if (!rc && !queue) rc = pack_flush_impl(ctx, &own);
    if (rc) return rc;
    e->version = ctx->param_version;
  }
  e->last_use = ++ctx->param_tick;
  *hi = e->hi; *lo = e->lo;
  return DYB200_OK;
}

}  // namespace

// ---- fp16 operand planes ----
int dyb200_f16_planes(dyb200_ctx* ctx, const float* src, uint32_t ld, uint32_t lines, uint32_t n, int mode, F16Job* job, uint32_t pad_H) {
  const uint32_t pitch = pad_H ? 4 * round_up(pad_H, 64) : round_up(n, 64);
  const size_t plane = (size_t)lines * pitch * sizeof(__half), words = mode == F16_LINE ? lines : mode == F16_ELEM ? n : 1;
  void *h, *l, *sc;
  int rc;
  if ((rc = dyb200_scratch(ctx, plane, &h)) || (rc = dyb200_scratch(ctx, plane, &l)) || (rc = dyb200_scratch(ctx, words * sizeof(uint32_t), &sc))) return rc;
  *job = F16Job{src, ld, lines, n, pitch, mode, (uint32_t*)sc, (__half*)h, (__half*)l};
  job->pad_H = pad_H;
  return DYB200_OK;
}
int dyb200_f16_pack(dyb200_ctx* ctx, F16Jobs* jobs) {
  if (jobs->n == 0) return DYB200_OK;
  F16Jobs rest = *jobs;
  rest.n = 0;
  // (the words of all jobs at once, those that a pass below writes among them: before it)
  bool two_pass = false;
  for (int k = 0; k < jobs->n; ++k) two_pass = two_pass || !f16_one_pass(jobs->job[k]);
  if (jobs->words && two_pass) DYB_CUDA(ctx, cudaMemsetAsync(jobs->words, 0, jobs->n_words * sizeof(uint32_t), ctx->stream));
  for (const int mode : {F16_ELEM, F16_LINE}) {   // (a launch per kind)
    F16Jobs part;
    part.n = 0; part.start[0] = 0;
    uint32_t lines = 0, longest = 0;
    bool odd = false, pad = false, mark = false;   // (pad: only with mark)
    for (int k = 0; k < jobs->n; ++k) {
      const F16Job& j = jobs->job[k];
      if (j.mode != mode) continue;
      if (!f16_one_pass(j)) { rest.job[rest.n++] = j; continue; }
      if (j.lines > lines) lines = j.lines;
      if (j.n > longest) longest = j.n;
      odd = odd || j.perm_H % 4 != 0; pad = pad || j.pad_H; mark = mark || j.mark || j.pad_H;
      part.job[part.n] = j;
      part.start[part.n + 1] = part.start[part.n] + (mode == F16_ELEM ? (j.n + 31) / 32 : j.n > 1024 ? j.lines : (j.lines + 7) / 8);
      ++part.n;
    }
    if (part.n == 0 || part.start[part.n] == 0) continue;
    void (*k)(F16Jobs);
    if (mode == F16_LINE && !mark) k = longest <= 8192 ? k_f16_line<8, false, false> : k_f16_line<16, false, false>;
    else if (mode == F16_LINE) k = longest <= 8192 ? (pad ? k_f16_line<8, true, true> : k_f16_line<8, false, true>) : pad ? k_f16_line<16, true, true> : k_f16_line<16, false, true>;
    else if (odd) k = lines <= 512 ? k_f16_strip<16, true> : k_f16_strip<32, true>;
    else k = lines <= 256 ? k_f16_strip<8> : lines <= 512 ? k_f16_strip<16> : k_f16_strip<32>;
    dyb_launch(k, part.start[part.n], 256, 0, ctx, part);
    DYB_LAUNCHED(ctx);
  }
  jobs = &rest;
  if (jobs->n == 0) return DYB200_OK;
  jobs->start[0] = 0;
  for (int k = 0; k < jobs->n; ++k) {
    const F16Job& j = jobs->job[k];
    const bool one_store = j.mode == F16_LINE && j.n <= kPiece;   // (every word is written once, no maximum to start from)
    if (!one_store && !jobs->words) DYB_CUDA(ctx, cudaMemsetAsync(j.scale, 0, (j.mode == F16_LINE ? j.lines : j.n) * sizeof(uint32_t), ctx->stream));
    const uint64_t end = (uint64_t)jobs->start[k] + f16_max_units(j).total;
    DYB_CHECK_ARG(ctx, end < 0x7fffffffull, "fp16 planes: operand too large (%u x %u)", j.lines, j.n);
    jobs->start[k + 1] = (uint32_t)end;
  }
  dyb_launch(jobs->wide ? k_f16_absmax<true> : k_f16_absmax<false>, jobs->start[jobs->n], 256, 0, ctx, *jobs);
  DYB_LAUNCHED(ctx);
  for (int k = 0; k < jobs->n; ++k) {
    const uint64_t end = jobs->start[k] + ((uint64_t)((jobs->job[k].n + 3) / 4) * jobs->job[k].lines + kSplitItems - 1) / kSplitItems;
    DYB_CHECK_ARG(ctx, end < 0x7fffffffull, "fp16 planes: operand too large (%u x %u)", jobs->job[k].lines, jobs->job[k].n);
    jobs->start[k + 1] = (uint32_t)end;
  }
  dyb_launch(k_f16_split, jobs->start[jobs->n], 256, 0, ctx, *jobs);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}
int dyb200_f16_param(dyb200_ctx* ctx, const float* src, uint32_t ld, uint32_t lines, uint32_t n, int mode, F16Job* job, uint32_t pad_H, uint32_t mark) {
  if (!ctx->param_cache_on) {
    F16Jobs jobs;
    jobs.n = 1;
    int rc = dyb200_f16_planes(ctx, src, ld, lines, n, mode, &jobs.job[0], pad_H);
    jobs.job[0].mark = mark;
    if (!rc) rc = dyb200_f16_pack(ctx, &jobs);
    *job = jobs.job[0];
    return rc;
  }
  const uint32_t pitch = pad_H ? 4 * round_up(pad_H, 64) : round_up(n, 64);
  float *hi, *lo;
  int rc = cached_param_pack(ctx, src, ld, pad_H ? kLayoutPadF16 : mark ? kLayoutMarkF16 : kLayoutF16 + mode, lines, n, pitch, &hi, &lo);
  if (rc) return rc;
  *job = F16Job{src, ld, lines, n, pitch, mode, reinterpret_cast<uint32_t*>(hi + (size_t)lines * pitch / 2), (__half*)hi, (__half*)lo};
  return DYB200_OK;
}
int dyb200_f16_gates(dyb200_ctx* ctx, const float* Wx, const float* Wh, uint32_t I, uint32_t H, F16Gates* out) {
  const uint32_t G = 4 * H, pitch = gates_f16_pitch(H);
  const size_t plane = (size_t)(I + H) * pitch;
  float *hi, *lo;
  uint32_t* scale;
  int rc;
  if (ctx->param_cache_on) {
    if ((rc = cached_param_pack(ctx, Wx, G, kLayoutGatesF16, G, I, pitch, &hi, &lo, Wh, H))) return rc;
    scale = reinterpret_cast<uint32_t*>(hi + plane / 2);
  } else {
    void *h, *l, *sc;
    if ((rc = dyb200_scratch(ctx, plane * sizeof(__half), &h)) || (rc = dyb200_scratch(ctx, plane * sizeof(__half), &l)) || (rc = dyb200_scratch(ctx, 2 * G * sizeof(uint32_t), &sc))) return rc;
    hi = (float*)h; lo = (float*)l; scale = (uint32_t*)sc;
    if ((rc = gates_f16_pack(ctx, Wx, Wh, I, H, (__half*)hi, (__half*)lo, scale))) return rc;
  }
  const size_t at = (size_t)I * pitch;
  *out = F16Gates{(__half*)hi, (__half*)lo, (__half*)hi + at, (__half*)lo + at, scale};
  return DYB200_OK;
}
PackedOp dyb200_f16_op(const F16Job& j, bool mn_major) {
  PackedOp p;
  p.hi = (float*)j.hi; p.lo = (float*)j.lo; p.pitch = j.pitch; p.f16 = 1; p.mn_major = mn_major ? 1u : 0u;
  p.rows = mn_major ? j.n : j.lines; p.K = mn_major ? j.lines : j.n;
  p.scale = j.scale;
  return p;
}

// ---- building blocks shared with the fused LSTM entry points ----------------------------------
int dyb200_tc_pack_flush(dyb200_ctx* ctx, PackJobs* batch) { return pack_flush_impl(ctx, batch); }

int dyb200_tc_pack(dyb200_ctx* ctx, const float* src, uint32_t ld, bool k_is_fast, uint32_t rows, uint32_t K,
                   const float* mask, uint32_t mask_ld, int mask_full, PackedOp* out, PackJobs* batch) {
  const uint32_t pitch = round_up(K, 32);
  void* buf;
  int rc = dyb200_scratch(ctx, (size_t)2 * rows * pitch * sizeof(float) + 256, &buf);
  if (rc) return rc;
  out->hi = (float*)buf;
  out->lo = (float*)(((uintptr_t)(out->hi + (size_t)rows * pitch) + 255) & ~(uintptr_t)255);
  out->rows = rows; out->K = K; out->pitch = pitch;
  return pack(ctx, src, ld, k_is_fast ? 1 : 0, rows, K, mask, mask_ld, mask_full, out->hi, out->lo, pitch, batch);
}

int dyb200_tc_planes(dyb200_ctx* ctx, uint32_t rows, uint32_t K, PackedOp* out) {
  const uint32_t pitch = round_up(K, 32);
  void* buf;
  int rc = dyb200_scratch(ctx, (size_t)2 * rows * pitch * sizeof(float) + 256, &buf);
  if (rc) return rc;
  out->hi = (float*)buf;
  out->lo = (float*)(((uintptr_t)(out->hi + (size_t)rows * pitch) + 255) & ~(uintptr_t)255);
  out->rows = rows; out->K = K; out->pitch = pitch;
  return DYB200_OK;
}

int dyb200_tc_param(dyb200_ctx* ctx, const float* src, uint32_t ld, bool k_is_fast, uint32_t rows, uint32_t K, PackedOp* out, PackJobs* batch) {
  if (!ctx->param_cache_on) return dyb200_tc_pack(ctx, src, ld, k_is_fast, rows, K, nullptr, 0, 0, out, batch);
  out->rows = rows; out->K = K; out->pitch = round_up(K, 32);
  return cached_param_pack(ctx, src, ld, k_is_fast ? 1 : 0, rows, K, out->pitch, &out->hi, &out->lo, nullptr, 0, batch);
}

int dyb200_tc_param_gates(dyb200_ctx* ctx, const float* src, uint32_t ld, uint32_t rows, uint32_t K, PackedOp* out) {
  const uint32_t pitch = round_up(K, 32);
  out->rows = rows; out->K = K; out->pitch = pitch;
  if (ctx->param_cache_on) return cached_param_pack(ctx, src, ld, kLayoutGates, rows, K, pitch, &out->hi, &out->lo);
  void* buf;
  int rc = dyb200_scratch(ctx, (size_t)2 * rows * pitch * sizeof(float) + 256, &buf);
  if (rc) return rc;
  out->hi = (float*)buf;
  out->lo = (float*)(((uintptr_t)(out->hi + (size_t)rows * pitch) + 255) & ~(uintptr_t)255);
  return pack(ctx, src, ld, kLayoutGates, rows, K, nullptr, 0, 0, out->hi, out->lo, pitch, nullptr);
}

inline uint32_t tile_cols(uint32_t N) { return N <= 64 ? 64 : BN; }

// Cost model of one launch (us): waves x (k-blocks per CTA x t_kb + 9 us of pipeline fill and epilogue), waves =
// ceil(tiles x S / SMs); S > 1 adds the second kernel that sums the S partial products into C ((S + 2) M N floats through
// HBM + a launch).  Measured on B200: within 2 us of the per-step LSTM products (dx / dh: 64 or 48 tiles, K = 4096 ->
// S = 2 and 3).
static double split_cost(double sms, uint32_t tiles, uint32_t kb_total, uint32_t S, double t_kb, double mn_bytes) {
  const uint32_t kb_split = (kb_total + S - 1) / S;
  double t = ceil((double)tiles * S / sms) * (kb_split * t_kb + 9.0);
  if (S > 1) t += (S + 2) * mn_bytes / 5.0e6 + 5.0;   // bytes / (5 TB/s) in us
  return t;
}
static uint32_t best_split(double sms, uint32_t tiles, uint32_t kb_total, double t_kb, double mn_bytes, double* cost) {
  uint32_t best = 1;
  double best_t = split_cost(sms, tiles, kb_total, 1, t_kb, mn_bytes);
  for (uint32_t S = 2; S <= 8; ++S) {
    if (kb_total / S < 8) break;   // at least 8 k-blocks per split
    const uint32_t kb_split = (kb_total + S - 1) / S;
    if ((kb_total + kb_split - 1) / kb_split != S) continue;
    const double t = split_cost(sms, tiles, kb_total, S, t_kb, mn_bytes);
    if (t < best_t * 0.97) { best = S; best_t = t; }   // a split must win by 3 %
  }
  if (cost) *cost = best_t;
  return best;
}
// The partly filled last round of a many-tile product can run as a product of its own (see dyb200_tc_gemm_packed) when K is
// long and its tiles form a rectangle: 2 = the last tail / tiles_n row blocks of every column of tiles (the persistent kernel
// keeps its grouped tile order on the row blocks before them), 1 = the last `tail` row blocks of the last column of tiles
// (row-block-fastest order), 0 = neither.
static int tail_can_run_apart(const dyb200_ctx* ctx, uint32_t tiles_m, uint32_t tiles, uint32_t kb_total, uint32_t bn) {
  const uint32_t tail = tiles % (uint32_t)ctx->sm_count, tiles_n = tiles / tiles_m;
  if (!(tiles > (uint32_t)ctx->sm_count && tail > 0 && 2 * tail <= (uint32_t)ctx->sm_count && kb_total >= 64 && bn == BN)) return 0;
  if (tail % tiles_n == 0 && tail / tiles_n < tiles_m) return 2;
  return tail <= tiles_m ? 1 : 0;
}

// Number of K splits of a product: the one the cost model says is fastest.  For a product with more tiles than SMs the
// unsplit form is the persistent kernel (epilogues overlapped, ~3 us left per tile) with its last round split apart.
uint32_t dyb200_tc_splits(const dyb200_ctx* ctx, uint32_t M, uint32_t N, uint32_t kb_total) {
  const uint32_t bn = tile_cols(N);
  const uint32_t tiles_m = (M + BM - 1) / BM, tiles = tiles_m * ((N + bn - 1) / bn);
  const double sms = (double)ctx->sm_count, t_kb = bn == 64 ? 0.40 : 0.66;
  const double mn_bytes = 4.0 * (double)M * (double)N;
  double cost;
  const uint32_t S = best_split(sms, tiles, kb_total, t_kb, mn_bytes, &cost);
  if (S > 1 && tail_can_run_apart(ctx, tiles_m, tiles, kb_total, bn)) {
    const uint32_t tail = tiles % (uint32_t)ctx->sm_count;
    double tail_cost;
    best_split(sms, tail, kb_total, t_kb, mn_bytes * tail / tiles, &tail_cost);
    const double persistent = (tiles / (uint32_t)ctx->sm_count) * (kb_total * t_kb + 3.0) + tail_cost;
    if (persistent < cost) return 1;
  }
  return S;
}

bool dyb200_lstm_bwd_tiling(const dyb200_ctx* ctx, uint32_t I, uint32_t H, uint32_t B, LstmBwdTiling* out) {
  // 128-column tiles from 256 columns up; two column blocks per CTA whenever the batch has an even number of them (128
  // columns: two blocks of 64), so that each CTA of the sequence kernel alternates between two independent chains
  const uint32_t bn = (B >= 256 && B % 128 == 0) ? 128u : 64u;
  if (B == 0 || B % bn != 0 || B / bn > 32 || H % 64 != 0 || I % 4 != 0) return false;
  const uint32_t tiles_m = (I + H + BM - 1) / BM, tiles_n = B / bn, kb = 4 * H / 32;
  const uint32_t ncb = tiles_n % 2 == 0 ? 2u : 1u;
  // as many K splits as keep every CTA of the sequence kernel resident (one per SM), at least 8 k-blocks each
  const uint32_t groups = tiles_m * (tiles_n / ncb);
  uint32_t S = (uint32_t)ctx->sm_count / groups;
  if (S == 0 || tiles_m * tiles_n > 160) return false;
  if (S > 8) S = 8;
  while (S > 1 && kb / S < 8) --S;
  const uint32_t per = (kb + S - 1) / S;
  S = (kb + per - 1) / per;
  out->bn = bn; out->ncb = ncb; out->S = S;
  return true;
}

int dyb200_tc_param2(dyb200_ctx* ctx, const float* src, uint32_t rows, const float* src2, uint32_t rows2, uint32_t ld,
                     bool k_is_fast, uint32_t K, PackedOp* out) {
  const uint32_t pitch = round_up(K, 32);
  out->rows = rows + rows2; out->K = K; out->pitch = pitch;
  if (ctx->param_cache_on) return cached_param_pack(ctx, src, ld, k_is_fast, rows, K, pitch, &out->hi, &out->lo, src2, rows2);
  void* buf;
  int rc = dyb200_scratch(ctx, (size_t)2 * out->rows * pitch * sizeof(float) + 256, &buf);
  if (rc) return rc;
  out->hi = (float*)buf;
  out->lo = (float*)(((uintptr_t)(out->hi + (size_t)out->rows * pitch) + 255) & ~(uintptr_t)255);
  PackJobs batch;
  dyb200_tc_pack_begin(&batch);
  rc = pack(ctx, src, ld, k_is_fast, rows, K, nullptr, 0, 0, out->hi, out->lo, pitch, &batch);
  if (!rc) rc = pack(ctx, src2, ld, k_is_fast, rows2, K, nullptr, 0, 0, out->hi + (size_t)rows * pitch, out->lo + (size_t)rows * pitch, pitch, &batch);
  if (!rc) rc = pack_flush_impl(ctx, &batch);
  return rc;
}

// One-tile products start under the kernel before them (see dyb_launch): 0.7 us of barriers, TMEM and descriptors, and the launch itself.  One
// layer of 256 units on 32 sequences, forward and backward: 227.5 -> 222.6 us; steps of models on several streams are the same within the
// noise; the persistent kernel so launched gained nothing and is not.  (A CTA that waits holds TMEM: no kernel that allocates any
// fits beside it, kTmemSmem sees to that, so none can be waiting for what it holds.)
// The kernels by tile width and form.  Their limit on dynamic shared memory is raised when one is first asked for (function attributes are per
// device, so the context remembers what it has set on its own; a limit loads its kernel, and a program needs a few of them).
using TcKernel = void (*)(TmapPack, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, GemmEpilogue, uint32_t*);
using PersistKernel = void (*)(TmapPack, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, GemmEpilogue, uint32_t*);
enum TcKind { TC_TF32, TC_F16, TC_TWO };
template <class K>
static int tc_limit(dyb200_ctx* ctx, uint32_t index, K kernel, int bytes) {
  if (ctx->gemm_attr_done & (1u << index)) return DYB200_OK;
  DYB_CUDA(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  ctx->gemm_attr_done |= 1u << index;
  return DYB200_OK;
}
static int tc_kernel(dyb200_ctx* ctx, uint32_t bn, bool cluster, TcKind kind, TcKernel* k) {
  static const TcKernel table[3][2][2] = {{{k_gemm_tc<64, false>, k_gemm_tc<128, false>}, {k_gemm_tc<64, true>, k_gemm_tc<128, true>}},
                                          {{k_gemm_tc<64, false, true>, k_gemm_tc<128, false, true>}, {k_gemm_tc<64, true, true>, k_gemm_tc<128, true, true>}},
                                          {{k_gemm_tc<64, false, false, true>, k_gemm_tc<128, false, false, true>}, {k_gemm_tc<64, true, false, true>, k_gemm_tc<128, true, false, true>}}};
  const uint32_t w = bn == 64 ? 0 : 1, c = cluster ? 1 : 0;
  *k = table[kind][c][w];
  return tc_limit(ctx, 4 * kind + 2 * c + w, *k, SMEM_BYTES);
}
static int persist_kernel(dyb200_ctx* ctx, uint32_t bn, bool f16, PersistKernel* k) {
  static const PersistKernel table[2][2] = {{k_gemm_persist<64>, k_gemm_persist<128>}, {k_gemm_persist<64, true>, k_gemm_persist<128, true>}};
  const uint32_t w = bn == 64 ? 0 : 1, f = f16 ? 1 : 0;
  *k = table[f][w];
  return tc_limit(ctx, 12 + 2 * f + w, *k, SMEM_PERSIST_BYTES);
}
// Whether `clusters` clusters of S one-tile CTAs are resident at once (asked for once per device, tile width and size).
static bool cluster_fits(dyb200_ctx* ctx, uint32_t bn, uint32_t S, uint32_t clusters) {
  int& mc = ctx->max_clusters[bn == 64 ? 0 : 1][S];
  if (mc == 0) {
    TcKernel k;
    if (tc_kernel(ctx, bn, true, TC_TF32, &k)) return false;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(1, 1, S); cfg.blockDim = dim3(kThreads, 1, 1); cfg.dynamicSmemBytes = SMEM_BYTES; cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = S;
    cfg.attrs = attr; cfg.numAttrs = 1;
    int n = 0;
    const cudaError_t e = cudaOccupancyMaxActiveClusters(&n, k, &cfg);
    if (e != cudaSuccess) { (void)cudaGetLastError(); n = -1; }
    mc = n > 0 ? n : -1;
  }
  return mc > 0 && clusters <= (uint32_t)mc;
}

int dyb200_tc_gemm_packed(dyb200_ctx* ctx, uint32_t M, uint32_t N, int npairs, const PackedOp* A, const PackedOp* B,
                          const GemmEpilogue& epi, uint32_t force_splits, const uint32_t* unless) {
  EncodeTiledFn enc;
  int rc = get_encoder(ctx, &enc);
  if (rc) return rc;
  const uint32_t bn = tile_cols(N);
  TmapPack tm;
  memset(&tm, 0, sizeof(tm));
  double flops = 0;
  const bool a_mn = A[0].mn_major != 0, b_mn = B[0].mn_major != 0, f16 = A[0].f16 != 0;
  const uint32_t el = f16 ? 64u : 32u;
  DYB_CHECK_ARG(ctx, !f16 || (npairs == 1 && B[0].f16 && A[0].scale && B[0].scale && A[0].pitch % 64 == 0 && B[0].pitch % 64 == 0),
                "tensor GEMM: fp16 operands come in one pair, both with scale words and a pitch that is a multiple of 64");
  DYB_CHECK_ARG(ctx, f16 || !B[0].f16, "tensor GEMM: operands of two kinds");
  tm.sa = A[0].scale; tm.sb = B[0].scale;
  // (an MN-major plane is read in groups of 32 rows: its pitch covers the rows rounded up to 32)
  DYB_CHECK_ARG(ctx, !a_mn || (npairs == 1 && A[0].pitch % 32 == 0 && A[0].pitch >= M && aligned16(A[0].hi) && aligned16(A[0].lo)),
                "tensor GEMM: an MN-major left operand needs a single pair, a pitch that is a multiple of 32 and covers the rows, and 16-byte aligned planes");
  DYB_CHECK_ARG(ctx, !b_mn || (npairs == 1 && B[0].pitch % 32 == 0 && B[0].pitch >= N && aligned16(B[0].hi) && aligned16(B[0].lo)),
                "tensor GEMM: an MN-major right operand needs a single pair, a pitch that is a multiple of 32 and covers the rows, and 16-byte aligned planes");
  tm.a_mn = a_mn ? 1u : 0u;
  tm.b_mn = b_mn ? 1u : 0u;
  for (int p = 0; p < npairs; ++p) {
    DYB_CHECK_ARG(ctx, A[p].rows == M && B[p].rows == N && A[p].K == B[p].K && A[p].pitch % 32 == 0 && B[p].pitch % 32 == 0,
                  "tensor GEMM: packed operand shapes do not match (M %u, N %u)", M, N);
    flops += 2.0 * M * N * A[p].K;
    if (a_mn) {
      if ((rc = make_map_mn(ctx, enc, &tm.t[0], A[0].hi, M, A[0].K, A[0].pitch, BM, f16))) return rc;
      if ((rc = make_map_mn(ctx, enc, &tm.t[1], A[0].lo, M, A[0].K, A[0].pitch, BM, f16))) return rc;
    } else {
      if ((rc = make_map(ctx, enc, &tm.t[4 * p + 0], A[p].hi, M, A[p].K, A[p].pitch, BM, f16))) return rc;
      if ((rc = make_map(ctx, enc, &tm.t[4 * p + 1], A[p].lo, M, A[p].K, A[p].pitch, BM, f16))) return rc;
    }
    if (b_mn) {
      if ((rc = make_map_mn(ctx, enc, &tm.t[2], B[0].hi, N, B[0].K, B[0].pitch, bn, f16))) return rc;
      if ((rc = make_map_mn(ctx, enc, &tm.t[3], B[0].lo, N, B[0].K, B[0].pitch, bn, f16))) return rc;
    } else {
      if ((rc = make_map(ctx, enc, &tm.t[4 * p + 2], B[p].hi, N, B[p].K, B[p].pitch, bn, f16))) return rc;
      if ((rc = make_map(ctx, enc, &tm.t[4 * p + 3], B[p].lo, N, B[p].K, B[p].pitch, bn, f16))) return rc;
    }
  }
  if (npairs == 1) for (int k = 0; k < 4; ++k) tm.t[4 + k] = tm.t[k];
  uint32_t kb0 = round_up(A[0].K, el) / el, kb1 = npairs > 1 ? round_up(A[1].K, el) / el : 0;
  const uint32_t kb_total = kb0 + kb1;
  if (f16 && !force_splits && dyb200_pair_takes(ctx, M, N, epi)) return dyb200_gemm_pair(ctx, &tm, M, N, kb_total, flops, epi, unless);
  DYB_CHECK_ARG(ctx, !unless, "tensor GEMM: a conditional product of a shape that the pair kernel does not take");
  dim3 grid((M + BM - 1) / BM, (N + bn - 1) / bn, 1);
  DYB_CHECK_ARG(ctx, epi.mode != EPI_LSTM_CELL || (M % BM == 0 && epi.H * 4 == M && epi.ldc % 4 == 0 && aligned16(epi.C) &&
                                                      aligned16(epi.bias) && aligned16(epi.c_prev) && aligned16(epi.c_out) && aligned16(epi.h_out)),
                "tensor GEMM: the LSTM-cell epilogue needs whole tiles of interleaved gate rows and 16-byte aligned tensors");
  // Split K when the output has too few tiles to occupy the SMs (e.g. dx = W^T dgate: 16-32 tiles, K = 4096).
  uint32_t S = force_splits ? (force_splits < kb_total ? force_splits : kb_total) : dyb200_tc_splits(ctx, M, N, kb_total);
  uint32_t kb_per_split = (kb_total + S - 1) / S;
  S = k_splits_used(kb0, kb1, (kb_total + kb_per_split - 1) / kb_per_split);
  GemmEpilogue kepi = epi;
  float* part = nullptr;
  // K splits as one thread-block cluster per tile (partial tiles meet in distributed shared memory) when every cluster
  // of the launch can be resident at once; dyb200_ctx_cluster_splitk(ctx, 0) keeps the workspace + second-kernel form.
  if (S > 1 && ctx->cluster_splitk) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.blockDim = dim3(kThreads, 1, 1); cfg.dynamicSmemBytes = SMEM_BYTES; cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->pdl ? 2 : 1;
    // (a smaller cluster size that fits was tried when the model's count does not - batch 64, 16 tiles: 7 instead of 8 -
    // and measured slower than the workspace form of the model's count: 4.73 vs 4.60 ms per step)
    const uint32_t Sc = (S <= 8 && cluster_fits(ctx, bn, S, grid.x * grid.y)) ? S : 0;
    if (Sc) {
      kb_per_split = (kb_total + Sc - 1) / Sc;
      cfg.gridDim = dim3(grid.x, grid.y, Sc);
      attr[0].val.clusterDim.z = Sc;
      GemmProfScope scope(ctx, flops, f16 ? 2 : 1, M, N, kb_total * el, (uint32_t)epi.mode);
      TcKernel kern;
      if ((rc = tc_kernel(ctx, bn, true, f16 ? TC_F16 : TC_TF32, &kern))) return rc;
      cudaLaunchKernelEx(&cfg, kern, tm, M, N, kb0, kb1, kb_per_split, epi, ctx->dev_flags);
      DYB_LAUNCHED(ctx);
      return DYB200_OK;
    }
  }
  if (S > 1) {
    void* pw;
    rc = dyb200_scratch(ctx, (size_t)S * M * N * sizeof(float), &pw);
    if (rc) return rc;
    part = (float*)pw;
    kepi = GemmEpilogue{EPI_STORE, part, M, nullptr, 0, 0.f, nullptr, 0, 0};   // (no second destination)
    grid.z = S;
  }
  if (S == 1 && grid.x * grid.y > (uint32_t)ctx->sm_count) {
    // A partly filled last round (dR: 632 tiles = 4 rounds of 148 + 40) would keep 108 SMs idle for a whole tile time.
    // When those last tiles form a rectangle (dR: the last 5 row blocks of all 8 columns of tiles) and K is long, the
    // persistent kernel stops before them and they run as a product of their own (the sub-matrices of the same operands),
    // which the cost model splits along K.
    uint32_t tiles_run = grid.x * grid.y;
    const uint32_t tail = tiles_run % (uint32_t)ctx->sm_count;
    const bool plain_epi = (epi.mode == EPI_STORE || epi.mode == EPI_ACCUM || epi.mode == EPI_BIAS) && epi.split_m == 0;
    const int tail_form = plain_epi ? tail_can_run_apart(ctx, grid.x, tiles_run, kb_total, bn) : 0;
    const bool tail_apart = tail_form != 0;
    if (tail_apart) tiles_run -= tail;
    // row blocks the persistent launch covers (all of them, unless the last ones run apart in every column of tiles)
    const uint32_t rows_run = tail_form == 2 ? grid.x - tail / grid.y : grid.x;
    // A long reduction whose tiles fill the last round badly (the deferred weight gradients: 256 tiles of 560 k-blocks on
    // 148 SMs = two rounds, the second 73 % full) is cut into Sp K splits as further work items of the same persistent
    // launch: 1024 items of 140 k-blocks make seven nearly full rounds.  The partial products go to a workspace and
    // k_splitk_reduce adds them in split order and applies the epilogue.  Same cost form as dyb200_tc_splits, with the 3 us
    // that a persistent CTA spends between items.
    uint32_t Sp = 1;
    if (!tail_apart && epi.mode != EPI_LSTM_CELL && epi.mode != EPI_GATES) {
      const double sms = (double)ctx->sm_count, t_kb = bn == 64 ? 0.40 : 0.66, mn_bytes = 4.0 * (double)M * (double)N;
      auto est = [&](uint32_t q) {
        const double rounds = ceil((double)tiles_run * q / sms);
        return rounds * ((double)((kb_total + q - 1) / q) * t_kb + 3.0) + (q > 1 ? (q + 2) * mn_bytes / 5.0e6 + 8.0 : 0.0);
      };
      double best = est(1);
      for (uint32_t q = 2; q <= 4; ++q)
        if (kb_total / q >= 64 && est(q) < 0.95 * best && est(q) < 0.95 * est(1)) { best = est(q); Sp = q; }
    }
    GemmEpilogue pepi = epi;
    float* ppart = nullptr;
    if (Sp > 1) {
      void* pw;
      if ((rc = dyb200_scratch(ctx, (size_t)Sp * M * N * sizeof(float), &pw))) return rc;
      ppart = (float*)pw;
      pepi = GemmEpilogue{EPI_STORE, ppart, M, nullptr, 0, 0.f, nullptr, 0, 0};
    }
    // one TMA store per finished half tile where the destination allows it
    if (npairs == 1 && (pepi.mode == EPI_STORE || pepi.mode == EPI_BIAS) && pepi.split_m == 0 && pepi.ldc % 4 == 0 && aligned16(pepi.C)) {
      if ((rc = dyb200_tc_make_store_map(ctx, &tm.t[4], pepi.C, M, N, Sp, pepi.ldc, 64))) return rc;
      tm.store_map = 1;
    }
    {
      GemmProfScope scope(ctx, flops * ((double)tiles_run / (grid.x * grid.y)), f16 ? 2 : 1, M, N, kb_total * el, (uint32_t)epi.mode);
      // grouped tile order when the A operand has many row blocks (unless the last round runs apart as part of the last
      // column of tiles, which relies on the row-block-fastest order)
      const uint32_t gm = (tail_form != 1 && rows_run > 16) ? 16u : 0u;
      PersistKernel kern;
      if ((rc = persist_kernel(ctx, bn, f16, &kern))) return rc;
      dyb_launch(kern, dim3(ctx->sm_count), kThreads, SMEM_PERSIST_BYTES, ctx, tm, M, N, kb0, kb1, rows_run, tiles_run, gm, Sp, pepi, ctx->dev_flags);
      DYB_LAUNCHED(ctx);
      if (Sp > 1 && (rc = dyb200_splitk_reduce(ctx, ppart, Sp, M, N, epi))) return rc;
    }
    if (!tail_apart) return DYB200_OK;
    // the last `tail` row blocks of the last column of tiles, or the last tail / tiles_n row blocks of every column
    const uint32_t m_off = (tail_form == 2 ? rows_run : grid.x - tail) * BM, n_off = tail_form == 2 ? 0u : (grid.y - 1) * bn;
    PackedOp A2[2], B2[2];
    for (int p = 0; p < npairs; ++p) {
      A2[p] = A[p]; A2[p].rows = M - m_off;   // (MN-major planes: the rows are the fast index)
      auto ahead = [&](float* q, size_t n) { return f16 ? (float*)((__half*)q + n) : q + n; };
      const size_t ao = a_mn ? (size_t)m_off : (size_t)m_off * A[p].pitch, bo = b_mn ? (size_t)n_off : (size_t)n_off * B[p].pitch;
      A2[p].hi = ahead(A[p].hi, ao); A2[p].lo = ahead(A[p].lo, ao);
      if (f16) A2[p].scale += m_off;
      B2[p] = B[p]; B2[p].rows = N - n_off;
      B2[p].hi = ahead(B[p].hi, bo); B2[p].lo = ahead(B[p].lo, bo);
      if (f16) B2[p].scale += n_off;
    }
    GemmEpilogue e2 = epi;
    e2.C += m_off + (size_t)epi.ldc * n_off;
    if (epi.mode == EPI_BIAS) e2.bias += m_off;
    return dyb200_tc_gemm_packed(ctx, M - m_off, N - n_off, npairs, A2, B2, e2);
  }
  {
    // times the MMA kernel (and the split-K reduction); the packing launches show up in the step time
    GemmProfScope scope(ctx, flops, f16 ? 2 : 1, M, N, kb_total * el, (uint32_t)epi.mode);
    TcKernel kern;
    if ((rc = tc_kernel(ctx, bn, false, f16 ? TC_F16 : TC_TF32, &kern))) return rc;
    dyb_launch_as(true, kern, grid, kThreads, SMEM_BYTES, ctx, tm, M, N, kb0, kb1, kb_per_split, kepi, ctx->dev_flags);
    DYB_LAUNCHED(ctx);
    if (S > 1 && epi.mode == EPI_LSTM_CELL) {
      dyb_launch(k_splitk_reduce_cell, stream_grid(ctx, (size_t)M / 16 * N + 1, 256), 256, 0, ctx, part, S, M, N, epi);
      DYB_LAUNCHED(ctx);
    } else if (S > 1) {
      int vec = M % 4 == 0 && epi.ldc % 4 == 0 && aligned16(epi.C) && epi.mode != EPI_GATES &&
                (epi.mode != EPI_BIAS || aligned16(epi.bias)) &&
                (epi.mode != EPI_ACCUM_MASK || (aligned16(epi.maskC) && (!epi.maskc_full || epi.maskc_ld % 4 == 0)));
      if (epi.split_m)
        vec = vec && epi.split_m % 4 == 0 && epi.ldc2 % 4 == 0 && aligned16(epi.C2) &&
              (epi.mode != EPI_ACCUM_MASK || (aligned16(epi.maskC2) && (!epi.maskc2_full || epi.maskc2_ld % 4 == 0)));
      dyb_launch(k_splitk_reduce, stream_grid(ctx, (size_t)M * N / 4 + 1, 256), 256, 0, ctx, part, S, M, N, epi, vec, (size_t)M * N, nullptr);
      DYB_LAUNCHED(ctx);
    }
  }
  return DYB200_OK;
}

// Second stage of a K split for callers outside this file: C = epilogue(sum over s of part[s]), the S partial products
// (M x N each, leading dimension M) added in ascending order.
int dyb200_splitk_reduce(dyb200_ctx* ctx, const float* part, uint32_t S, uint32_t M, uint32_t N, const GemmEpilogue& epi, size_t split_stride,
                         const uint32_t* unless) {
  int vec = M % 4 == 0 && split_stride % 4 == 0 && aligned16(part) && epi.ldc % 4 == 0 && aligned16(epi.C) && epi.mode != EPI_GATES && (epi.mode != EPI_BIAS || aligned16(epi.bias)) &&
            (epi.mode != EPI_ACCUM_MASK || (aligned16(epi.maskC) && (!epi.maskc_full || epi.maskc_ld % 4 == 0)));
  if (epi.split_m)
    vec = vec && epi.split_m % 4 == 0 && epi.ldc2 % 4 == 0 && aligned16(epi.C2) &&
          (epi.mode != EPI_ACCUM_MASK || (aligned16(epi.maskC2) && (!epi.maskc2_full || epi.maskc2_ld % 4 == 0)));
  dyb_launch(k_splitk_reduce, stream_grid(ctx, (size_t)M * N / 4 + 1, 256), 256, 0, ctx, part, S, M, N, epi, vec, split_stride ? split_stride : (size_t)M * N, unless);
  DYB_LAUNCHED(ctx);
  return DYB200_OK;
}

// Two products with one left operand, C0 += A B0^T and C1 += A B1^T, as one over the columns of both (each side's columns rounded up to whole
// tiles): a short product of its own is mostly pipeline fill and epilogue, and the few tiles of one leave SMs idle.  K splits as clusters
// where they fit, or as work items of the persistent kernel with a second stage, by the estimates of dyb200_tc_splits.
// us for a flush (events), as two launches / in one: 1024 x (128 + 256), K = 300 36 / 22, 520 44 / 21, 1600 38 / 21, 13000 99 / 68, 107000 538 / 378;
// 1200 x (200 + 300) x 1050 36 / 27; 512 x (32 + 128) x 10560 71 / 34; 2816 x (704 + 704) x 35 28 / 27; 2048 x (512 + 512) x 4480 120 / 103.
int dyb200_tc_gemm_packed2(dyb200_ctx* ctx, uint32_t M, const PackedOp& A, const PackedOp* B, float* C0, uint32_t ldc0, float* C1, uint32_t ldc1,
                           const uint32_t* only_if) {
  EncodeTiledFn enc;
  int rc = get_encoder(ctx, &enc);
  if (rc) return rc;
  const uint32_t N0 = B[0].rows, N1 = B[1].rows, bn = N0 <= 64 && N1 <= 64 ? 64 : BN, split = N1 ? round_up(N0, bn) : 0, N = N1 ? split + N1 : N0;
  const uint32_t tiles_m = (M + BM - 1) / BM, tiles = tiles_m * ((N + bn - 1) / bn), kb = round_up(A.K, 32) / 32;
  TmapPack tm;
  memset(&tm, 0, sizeof(tm));
  tm.a_mn = tm.b_mn = 1;
  tm.n_split = split;
  DYB_CHECK_ARG(ctx, A.mn_major && B[0].mn_major && !A.f16 && A.K == B[0].K && A.rows == M && (N1 ? B[1].mn_major && A.K == B[1].K : only_if != nullptr),
                "tensor GEMM: operands of a grouped product");
  if ((rc = make_map_mn(ctx, enc, &tm.t[0], A.hi, M, A.K, A.pitch, BM)) || (rc = make_map_mn(ctx, enc, &tm.t[1], A.lo, M, A.K, A.pitch, BM))) return rc;
  for (int q = 0; q < (N1 ? 2 : 1); ++q)
    if ((rc = make_map_mn(ctx, enc, &tm.t[q ? 6 : 2], B[q].hi, B[q].rows, B[q].K, B[q].pitch, bn)) ||
        (rc = make_map_mn(ctx, enc, &tm.t[q ? 7 : 3], B[q].lo, B[q].rows, B[q].K, B[q].pitch, bn))) return rc;
  if (!N1) { tm.t[6] = tm.t[2]; tm.t[7] = tm.t[3]; }   // (n_split = 0: every tile is of the second side)
  tm.t[4] = tm.t[0]; tm.t[5] = tm.t[1];
  GemmEpilogue epi{EPI_ACCUM, C0, ldc0, nullptr, 0, 0.f, nullptr, 0, 0};
  epi.n_split = split; epi.n_live = N0; epi.Cn = C1; epi.ldcn = ldc1;
  tm.sa = only_if;
  const double flops = 2.0 * M * (double)(N0 + N1) * A.K, sms = (double)ctx->sm_count, t_kb = bn == 64 ? 0.40 : 0.66;
  // one tile per CTA (in waves: 2816 x (704 + 704) over 35 columns 22 us, 29 as work items of the persistent kernel), or clusters of S splits
  // that are all resident, at least eight k-blocks each.  Two k-blocks end hardly sooner on an idle GPU and hold several times the SMs; us with
  // two / with eight: a flush of 1024 x (128 + 256) over 300 columns 20.5 / 22.2, 800 20.9 / 20.5, 1600 21.2 / 20.8; a step of a language model of
  // 256 units alone 222 / 226, three on three streams 134 / 119; a tagger of 16 sentences alone 532 / 524, three 256 / 237.
  uint32_t Sc = 0;
  double cost = 1e30;
  for (uint32_t S = 1; S <= (only_if ? 1u : 8u) && (S == 1 || kb / S >= 8); ++S) {
    if (S > 1 && ((kb + (kb + S - 1) / S - 1) / ((kb + S - 1) / S) != S || !cluster_fits(ctx, bn, S, tiles))) continue;
    const double t = (S == 1 ? ceil(tiles / sms) : 1.0) * (((kb + S - 1) / S) * t_kb + 9.0);
    if (t < cost) { cost = t; Sc = S; }
  }
  // work items of the persistent kernel, as partial products and one sum per side (512 x (32 + 128) over 10560 columns: 19 us and 2 x 4, two
  // launches 29 and 35; 1024 x (128 + 256) over 107000: 369 us and 2 x 3, two launches 537)
  uint32_t Sp = 0;
  for (uint32_t S = 2; S <= 64 && kb / S >= 16 && !only_if; ++S) {
    if ((kb + (kb + S - 1) / S - 1) / ((kb + S - 1) / S) != S) continue;   // (no empty split)
    const double t = ceil((double)tiles * S / sms) * (((kb + S - 1) / S) * t_kb + 3.0) + 6.0 + (S + 2) * 4.0e-6 * M * N / 5.0 + 5.0;
    if (t < 0.97 * cost) { cost = t; Sp = S; }
  }
  const dim3 grid(tiles_m, (N + bn - 1) / bn, 1);
  const bool through_memory = Sp == 0 && Sc > 1 && !ctx->cluster_splitk;   // (dyb200_ctx_cluster_splitk: the clusters' splits, the same partial tiles)
  if (through_memory) Sp = Sc;
  void* pw = nullptr;
  if (Sp && dyb200_scratch(ctx, (size_t)Sp * M * N * sizeof(float), &pw) != DYB200_OK) {   // (no room for partial products)
    Sp = 0;
    if (!ctx->cluster_splitk) Sc = 1;
  }
  TcKernel kern;
  if (Sp == 0) {
    if ((rc = tc_kernel(ctx, bn, Sc > 1, TC_TWO, &kern))) return rc;
    GemmProfScope scope(ctx, only_if ? 0.0 : flops, 1, M, N0 + N1, kb * 32, (uint32_t)EPI_ACCUM);   // (under a condition: the products on pairs have been counted)
    if (Sc == 1) {
      dyb_launch_as(true, kern, grid, kThreads, SMEM_BYTES, ctx, tm, M, N, kb, 0u, kb, epi, ctx->dev_flags);
    } else {
      cudaLaunchConfig_t cfg;
      memset(&cfg, 0, sizeof(cfg));
      cfg.gridDim = dim3(grid.x, grid.y, Sc); cfg.blockDim = dim3(kThreads, 1, 1); cfg.dynamicSmemBytes = SMEM_BYTES; cfg.stream = ctx->stream;
      cudaLaunchAttribute attr[2];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = Sc;
      attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[1].val.programmaticStreamSerializationAllowed = 1;
      cfg.attrs = attr; cfg.numAttrs = ctx->pdl ? 2 : 1;
      cudaLaunchKernelEx(&cfg, kern, tm, M, N, kb, 0u, (kb + Sc - 1) / Sc, epi, ctx->dev_flags);
    }
    DYB_LAUNCHED(ctx);
    return DYB200_OK;
  }
  // partial products over the columns of both sides
  float* const part = (float*)pw;
  const GemmEpilogue pepi{EPI_STORE, part, M, nullptr, 0, 0.f, nullptr, 0, 0};
  if (through_memory) {
    if ((rc = tc_kernel(ctx, bn, false, TC_TWO, &kern))) return rc;
    GemmProfScope scope(ctx, flops, 1, M, N0 + N1, kb * 32, (uint32_t)EPI_ACCUM);
    dyb_launch_as(true, kern, dim3(grid.x, grid.y, Sp), kThreads, SMEM_BYTES, ctx, tm, M, N, kb, 0u,
               (kb + Sp - 1) / Sp, pepi, ctx->dev_flags);
    DYB_LAUNCHED(ctx);
  } else {
    tm.store_map = M % 4 == 0;
    if (tm.store_map && (rc = dyb200_tc_make_store_map(ctx, &tm.t[4], part, M, N, Sp, M, 64))) return rc;
    PersistKernel persist;
    if ((rc = persist_kernel(ctx, bn, false, &persist))) return rc;
    GemmProfScope scope(ctx, flops, 1, M, N0 + N1, kb * 32, (uint32_t)EPI_ACCUM);
    dyb_launch(persist, dim3(ctx->sm_count), kThreads, SMEM_PERSIST_BYTES, ctx, tm, M, N, kb, 0u, tiles_m, tiles, tiles_m > 16 ? 16u : 0u,
               Sp, pepi, ctx->dev_flags);
    DYB_LAUNCHED(ctx);
  }
  const GemmEpilogue e0{EPI_ACCUM, C0, ldc0, nullptr, 0, 0.f, nullptr, 0, 0}, e1{EPI_ACCUM, C1, ldc1, nullptr, 0, 0.f, nullptr, 0, 0};
  if ((rc = dyb200_splitk_reduce(ctx, part, Sp, M, N0, e0, (size_t)M * N))) return rc;
  return dyb200_splitk_reduce(ctx, part + (size_t)M * split, Sp, M, N1, e1, (size_t)M * N);
}

bool dyb200_tc_eligible(uint32_t M, uint32_t N, double flops) {
  // Small products stay on the CUDA-core kernel: packing + a 128x128 tile would mostly move padding.  A product with few
  // rows but many columns or a long reduction (the tag layer of a tagger: 32 or 45 rows times 100 000 tokens) is still far
  // better off here - most of a tile's rows are padding, but the work is bound by reading the long operand once.
  // (Between 2 and 8 MFLOP the CUDA-core kernel is slow when its grid is one or two CTAs - 190 us for the 128 x 21 x 1024
  // products of a tagger batch's last time steps - but it is plain fp32: a lower limit here was measured to cost accuracy
  // margin in small-batch recurrences (1.5e-4 of a row's scale after 100 steps of 3xTF32 products), so the limit stays.)
  return !(flops < 8.0e6 || M < 16 || (M + BM - 1) / BM > 65535u || (N + BN - 1) / BN > 65535u);
}

int dyb200_gemm_tc(dyb200_ctx* ctx, uint32_t M, uint32_t N, int npairs, const GemmPair* pairs, const GemmEpilogue& epi,
                   int* handled) {
  *handled = 0;
  if (M == 0 || N == 0 || npairs < 1 || npairs > 2) return DYB200_OK;
  double flops = 0;
  for (int p = 0; p < npairs; ++p) flops += 2.0 * M * N * pairs[p].K;
  if (!dyb200_tc_eligible(M, N, flops)) return DYB200_OK;
  for (int p = 0; p < npairs; ++p) if (pairs[p].K == 0) return DYB200_OK;
  *handled = 1;
  PackedOp A[2], B[2];
  if (npairs == 1 && !pairs[0].maskB && dyb200_f16_takes(flops, pairs[0].K)) {
    // Both operands as they lie: lines are rows of a K-major operand (A transposed / B not), or k of an MN-major one.
    const GemmPair& g = pairs[0];
    const bool a_mn = g.transA == 0, b_mn = g.transB != 0;
    F16Jobs jobs;
    F16Job ja, jb;
    int rc;
    jobs.n = 0;
    if (g.a_is_param) rc = dyb200_f16_param(ctx, g.A, g.lda, a_mn ? g.K : M, a_mn ? M : g.K, a_mn ? F16_ELEM : F16_LINE, &ja);
    else if (!(rc = dyb200_f16_planes(ctx, g.A, g.lda, a_mn ? g.K : M, a_mn ? M : g.K, a_mn ? F16_ELEM : F16_LINE, &ja))) jobs.job[jobs.n++] = ja;
    if (rc) return rc;
    if ((rc = dyb200_f16_planes(ctx, g.B, g.ldb, b_mn ? g.K : N, b_mn ? N : g.K, b_mn ? F16_ELEM : F16_LINE, &jb))) return rc;
    jobs.job[jobs.n++] = jb;
    if ((rc = dyb200_f16_pack(ctx, &jobs))) return rc;
    A[0] = dyb200_f16_op(ja, a_mn); B[0] = dyb200_f16_op(jb, b_mn);
    return dyb200_tc_gemm_packed(ctx, M, N, 1, A, B, epi);
  }
  PackJobs batch;   // all operands that need packing go out in one launch
  dyb200_tc_pack_begin(&batch);
  int rcp = DYB200_OK;
  for (int p = 0; p < npairs && !rcp; ++p) {
    const GemmPair& g = pairs[p];
    // A: rows = m. op(A)(m,k) = transA ? A[k + lda*m] : A[m + lda*k]  -> k is fast iff transA.  An operand whose rows are
    // the fast index is split as it lies (K rows of M values) and read MN-major (single products only): no transposing
    // pass, and a parameter then has ONE set of planes for this product and for the one that uses it transposed.
    const bool a_mn = npairs == 1 && g.transA == 0, b_mn = npairs == 1 && g.transB != 0;
    int& rc = rcp;
    if (a_mn) {
      rc = g.a_is_param ? dyb200_tc_param(ctx, g.A, g.lda, true, g.K, M, &A[p], &batch)
                        : dyb200_tc_pack(ctx, g.A, g.lda, true, g.K, M, nullptr, 0, 0, &A[p], &batch);
      A[p].rows = M; A[p].K = g.K; A[p].mn_major = 1;
    } else {
      rc = g.a_is_param ? dyb200_tc_param(ctx, g.A, g.lda, g.transA != 0, M, g.K, &A[p], &batch)
                        : dyb200_tc_pack(ctx, g.A, g.lda, g.transA != 0, M, g.K, nullptr, 0, 0, &A[p], &batch);
    }
    if (rc) break;
    // B: rows = n. op(B)(k,n) = transB ? B[n + ldb*k] : B[k + ldb*n]  -> k is fast iff !transB
    if (b_mn) {
      rc = dyb200_tc_pack(ctx, g.B, g.ldb, true, g.K, N, g.maskB, g.mask_ld, g.mask_full, &B[p], &batch);
      B[p].rows = N; B[p].K = g.K; B[p].mn_major = 1;
    } else {
      rc = dyb200_tc_pack(ctx, g.B, g.ldb, g.transB == 0, N, g.K, g.maskB, g.mask_ld, g.mask_full, &B[p], &batch);
    }
  }
  if (!rcp) rcp = dyb200_tc_pack_flush(ctx, &batch);
  if (rcp) {   // (planes of a parameter that were queued count as packed, and were not: nothing that is cached does any more)
    ctx->param_version++;
    return rcp;
  }
  return dyb200_tc_gemm_packed(ctx, M, N, npairs, A, B, epi);
}

// ---- deferred parameter-gradient products ---------------------------------------------------------
// dW = sum_t A_t * B_t^T (A_t: M x k_t, B_t: N x k_t, both column-major) arises once per time step for
// a parameter shared by all steps (dWx, dWh of an LSTM layer, dR of the output projection).  Instead of
// T small products with K = batch, the packed K-major planes of every step are appended along K and ONE
// product with K = sum k_t runs at the end: the tensor pipe sees a long reduction and C is read and
// written once.  One A operand can serve two B operands (dWx and dWh share the gate gradient).
// All planes are MN-major for that product: one row per COLUMN of the accumulator - Mp = M rounded up to 32 floats in A,
// Np[j] in B[j] - element (m, col) at plane[col * Mp + m].  For an LSTM layer these are the layouts the recurrence reads
// K-major: A = the gate-gradient planes, right operand of dx / dh = [Wx; Wh]^T dgates in the backward pass; B[0] = x .*
// mask_x and B[1] = h_tm1 .* mask_h, right operands of the gate product in the forward pass.  So every set of planes is
// written once, by whoever produces the values (a packing launch, the LSTM epilogue, the cell pass), serves both products,
// and no transposed copy exists.
struct dyb200_wgrad {
  uint32_t M, Mp, N[2], Np[2], Kcap;
  uint32_t k;    // columns of A filled so far (the product at flush time runs over [0, k))
  uint32_t kb;   // columns of the B operands filled so far
  PackedOp A, B[2];
  // Pre-split sequence inputs (dyb200_wgrad_pack_inputs): x_cols = columns of B[0] that hold a whole sequence's x .* mask_x
  // (0: none); rows [c, c + batch) of B[1] are the h input of the step that starts at column c, written by the LSTM
  // epilogue of the step before; h_col = the column whose B[1] rows the last forward call wrote; step = columns per step
  // of that sequence (0: varying).
  uint32_t x_cols, h_col, step;
};
// Whether the flush makes fp16 pairs of the TF32 planes first: 16 bytes moved per value (a pass for the scales over the hi planes, one
// that reads both planes and writes the pairs) against products at 490 instead of 190 TFLOP/s, so it is the multiply-adds per
// value, M N / (M + N), that decide.  us with TF32 / fp16 pairs: 4096 x (1024 + 1024), K = 17920 1285 / 887, K = 2240 243 / 144, K = 560
// 112 / 71; 4096 x (512 + 1024) x 2240 185 / 134; 2048 x (512 + 512) (683 per value) x 4480 120 / 123; 1024 x (128 + 256) (279) x 107000
// 536 / 664.  The error is no larger (max / rms of |row| |column|, 4096 x 1024 x 17920: 9.5e-8 / 1.4e-8 and 9.2e-8 / 1.1e-8).
static bool wgrad_on_f16(const dyb200_wgrad* w) {
  const double N = (double)w->N[0] + w->N[1];
  return w->k >= 256 && w->M * N >= 800.0 * (w->M + N);
}
// A pair of halves has the 22 bits of a TF32 pair within 2^28 of its scale, the largest value of a row over ALL columns.  Gradients that fade over
// the steps leave that range, and dWx of a feature that is there in the first steps only would be made of what is left of them.  So the
// passes that make the pairs also look at each row's blocks of eight columns: where one that is not all zero lies more than 2^kF16Span below
// the row's largest value, a device word sends the flush back to the TF32 planes - the products of pairs end at once, and the grouped
// product, which otherwise ends at once, adds its result.  So no element is further off than 2^-26 of the largest of its block.
// The words and the empty launch cost 4 us of 66 (4096 x (1024 + 1024), K = 560) or 888 (K = 17920).
static int wgrad_f16_planes(dyb200_ctx* ctx, const dyb200_wgrad* w, const PackedOp* ops, const bool* side, PackedOp* pairs, const uint32_t** wide) {
  F16Jobs jobs;
  jobs.n = 0;
  size_t halves = 0, words = 0;
  for (int q = 0; q < 3; ++q) {
    if (q && !side[q - 1]) continue;
    halves += 2 * (size_t)w->k * round_up(ops[q].rows, 64);
    words += 2 * (size_t)round_up(ops[q].rows, 4);
  }
  void* p;   // (one block: there is room for all or nothing is taken; the planes are whole 128-byte lines)
  int rc;
  if ((rc = dyb200_scratch(ctx, halves * sizeof(__half) + (words + 1) * sizeof(uint32_t), &p))) return rc;
  __half* h = (__half*)p;
  uint32_t* s = (uint32_t*)(h + halves);
  jobs.words = s; jobs.n_words = words + 1; jobs.wide = s + words;
  for (int q = 0; q < 3; ++q) {
    if (q && !side[q - 1]) continue;
    const uint32_t n = ops[q].rows, pitch = round_up(n, 64), wn = round_up(n, 4);
    F16Job& j = jobs.job[jobs.n++];
    j = F16Job{ops[q].hi, ops[q].pitch, w->k, n, pitch, F16_ELEM, s, h, h + (size_t)w->k * pitch};
    j.src_lo = ops[q].lo;
    j.low = s + wn;
    h += 2 * (size_t)w->k * pitch; s += 2 * (size_t)wn;
    pairs[q] = dyb200_f16_op(j, true);
  }
  *wide = jobs.wide;
  return dyb200_f16_pack(ctx, &jobs);
}
// natural pack of the k columns [col, col + k) of operand j (b is N[j] x k column-major; the mask is indexed like b)
static int pack_b_rows(dyb200_ctx* ctx, dyb200_wgrad* w, int j, uint32_t col, uint32_t k, const float* b, uint32_t ldb, const float* mask,
                       int mask_full, PackJobs* batch) {
  return pack(ctx, b, ldb, 1, k, w->N[j], mask, ldb, mask_full, w->B[j].hi + (size_t)col * w->Np[j], w->B[j].lo + (size_t)col * w->Np[j],
              w->Np[j], batch);
}

// Same as dyb200_wgrad_push, but the packing work is queued in `batch` (the caller launches it).
int dyb200_wgrad_push_batched(dyb200_wgrad* w, uint32_t k, const float* a, uint32_t lda, const float* b0, uint32_t ldb0,
                              const float* mask0, int mask0_full, const float* b1, uint32_t ldb1, const float* mask1,
                              int mask1_full, dyb200_ctx* ctx, PackJobs* batch) {
  DYB_CHECK_ARG(ctx, w && a && b0 && (w->N[1] == 0 || b1), "wgrad_push: null argument");
  DYB_CHECK_ARG(ctx, w->k + k <= w->Kcap, "wgrad_push: %u + %u columns exceed the capacity %u", w->k, k, w->Kcap);
  if (k == 0) return DYB200_OK;
  // (a is M x k column-major: the k rows of the MN-major planes, each M contiguous values)
  int rc = pack(ctx, a, lda, true, k, w->M, nullptr, 0, 0, w->A.hi + (size_t)w->k * w->Mp, w->A.lo + (size_t)w->k * w->Mp, w->Mp, batch);
  if (rc) return rc;
  rc = pack_b_rows(ctx, w, 0, w->k, k, b0, ldb0, mask0, mask0_full, batch);
  if (rc) return rc;
  if (w->N[1]) {
    rc = pack_b_rows(ctx, w, 1, w->k, k, b1, ldb1, mask1, mask1_full, batch);
    if (rc) return rc;
  }
  w->k += k;
  w->kb = w->k;
  return DYB200_OK;
}

// For a producer that writes the A planes of the next k columns itself: where they go (k rows of `pitch` floats: row =
// column of the accumulator, M values each), and the B operands queued as in dyb200_wgrad_push_batched.  The accumulator
// advances by k.
int dyb200_wgrad_reserve(dyb200_wgrad* w, uint32_t k, float** a_hi, float** a_lo, uint32_t* pitch, const float* b0, uint32_t ldb0,
                         const float* mask0, int mask0_full, const float* b1, uint32_t ldb1, const float* mask1, int mask1_full,
                         dyb200_ctx* ctx, PackJobs* batch) {
  DYB_CHECK_ARG(ctx, w && b0 && (w->N[1] == 0 || b1), "wgrad_reserve: null argument");
  DYB_CHECK_ARG(ctx, w->k + k <= w->Kcap, "wgrad_reserve: %u + %u columns exceed the capacity %u", w->k, k, w->Kcap);
  *a_hi = w->A.hi + (size_t)w->k * w->Mp; *a_lo = w->A.lo + (size_t)w->k * w->Mp; *pitch = w->Mp;
  int rc = pack_b_rows(ctx, w, 0, w->k, k, b0, ldb0, mask0, mask0_full, batch);
  if (rc) return rc;
  if (w->N[1]) {
    rc = pack_b_rows(ctx, w, 1, w->k, k, b1, ldb1, mask1, mask1_full, batch);
    if (rc) return rc;
  }
  w->k += k;
  w->kb = w->k;
  return DYB200_OK;
}
void dyb200_wgrad_unreserve(dyb200_wgrad* w, uint32_t k) { w->k -= k; w->kb = w->k; }
// Explicit column positions, for callers that fill the B operands (the layer inputs) during the forward pass and the A
// operand (the gate gradient) during the backward pass: step t of a sequence uses columns [t * k, (t + 1) * k) both times.
int dyb200_wgrad_push_b_at(dyb200_wgrad* w, uint32_t col, uint32_t k, const float* b0, uint32_t ldb0, const float* mask0, int mask0_full,
                           const float* b1, uint32_t ldb1, const float* mask1, int mask1_full, dyb200_ctx* ctx, PackJobs* batch) {
  // (b0 == nullptr: the first operand's columns are already in place, see dyb200_wgrad_pack_inputs)
  DYB_CHECK_ARG(ctx, w && (w->N[1] == 0 || b1), "wgrad_push_b_at: null argument");
  DYB_CHECK_ARG(ctx, (uint64_t)col + k <= w->Kcap, "wgrad_push_b_at: columns [%u, %u) exceed the capacity %u", col, col + k, w->Kcap);
  int rc = b0 ? pack_b_rows(ctx, w, 0, col, k, b0, ldb0, mask0, mask0_full, batch) : DYB200_OK;
  if (rc) return rc;
  if (w->N[1]) {
    rc = pack_b_rows(ctx, w, 1, col, k, b1, ldb1, mask1, mask1_full, batch);
    if (rc) return rc;
  }
  if (col + k > w->kb) w->kb = col + k;
  return DYB200_OK;
}
int dyb200_wgrad_reserve_a_at(dyb200_wgrad* w, uint32_t col, uint32_t k, float** a_hi, float** a_lo, uint32_t* pitch, dyb200_ctx* ctx) {
  DYB_CHECK_ARG(ctx, w && (uint64_t)col + k <= w->Kcap, "wgrad_reserve_a_at: columns [%u, %u) exceed the capacity", col, col + k);
  *a_hi = w->A.hi + (size_t)col * w->Mp; *a_lo = w->A.lo + (size_t)col * w->Mp; *pitch = w->Mp;
  if (col + k > w->k) w->k = col + k;
  return DYB200_OK;
}
int dyb200_wgrad_pack_a_at(dyb200_wgrad* w, uint32_t col, uint32_t k, const float* a, uint32_t lda, dyb200_ctx* ctx, PackJobs* batch) {
  DYB_CHECK_ARG(ctx, w && a && (uint64_t)col + k <= w->Kcap, "wgrad_pack_a_at: columns [%u, %u) exceed the capacity", col, col + k);
  int rc = pack(ctx, a, lda, 1, k, w->M, nullptr, 0, 0, w->A.hi + (size_t)col * w->Mp, w->A.lo + (size_t)col * w->Mp, w->Mp, batch);
  if (rc) return rc;
  if (col + k > w->k) w->k = col + k;
  return DYB200_OK;
}
bool dyb200_wgrad_x_planes(const dyb200_wgrad* w, uint32_t col, uint32_t k, PackedOp* out) {
  if (!w || (w->step && k != w->step) || (uint64_t)col + k > w->x_cols) return false;
  *out = w->B[0];
  out->rows = k; out->K = w->N[0]; out->mn_major = 0;
  out->hi += (size_t)col * w->Np[0]; out->lo += (size_t)col * w->Np[0];
  return true;
}
bool dyb200_wgrad_h_planes(const dyb200_wgrad* w, uint32_t col, uint32_t k, PackedOp* out) {
  if (!w || w->N[1] == 0 || (w->step && k != w->step) || w->h_col != col || (uint64_t)col + k > w->x_cols) return false;
  *out = w->B[1];
  out->rows = k; out->K = w->N[1]; out->mn_major = 0;
  out->hi += (size_t)col * w->Np[1]; out->lo += (size_t)col * w->Np[1];
  return true;
}
bool dyb200_wgrad_next_h(dyb200_wgrad* w, uint32_t col, uint32_t k, GemmEpilogue* epi) {
  // (all k columns of h_t are written at the next step's position; with steps of varying width the next step may use fewer)
  if (!w || w->N[1] == 0 || w->x_cols == 0 || (w->step && k != w->step) || (uint64_t)col + 2 * (uint64_t)k > w->x_cols) return false;
  const uint32_t next = col + k;
  epi->hn_hi = w->B[1].hi + (size_t)next * w->Np[1]; epi->hn_lo = w->B[1].lo + (size_t)next * w->Np[1]; epi->hn_pitch = w->Np[1];
  w->h_col = next;
  if (next + k > w->kb) w->kb = next + k;
  return true;
}
// ---- sequence kernels (lstm_seq.cu): the operand planes the accumulator holds for a whole sequence ----
bool dyb200_wgrad_seq_planes(const dyb200_wgrad* w, uint32_t steps, uint32_t step, SeqPlanes* out) {
  if (!w || w->N[1] == 0 || w->x_cols == 0 || w->step != step || w->x_cols != (uint64_t)steps * step) return false;
  out->X = w->B[0]; out->X.rows = w->x_cols; out->X.K = w->N[0]; out->X.mn_major = 0;
  out->Hs = w->B[1]; out->Hs.rows = w->x_cols; out->Hs.K = w->N[1]; out->Hs.mn_major = 0;
  return true;
}
// h of the first step (h0 .* mask_h): operand planes of columns [0, step).  The same values
// dyb200_vanilla_lstm_fwd_fused_at splits at deferred_col = 0.
int dyb200_wgrad_seq_h0(dyb200_wgrad* w, const float* h0, const float* mh, int mh_full, dyb200_ctx* ctx, PackJobs* batch) {
  return pack_b_rows(ctx, w, 1, 0, w->step, h0, w->N[1], mh, mh_full, batch);
}
void dyb200_wgrad_seq_done(dyb200_wgrad* w) {
  w->h_col = w->x_cols - w->step;   // the planes of the last step's h input are the most recent ones
  if (w->x_cols > w->kb) w->kb = w->x_cols;
}
bool dyb200_wgrad_column_planes(const dyb200_wgrad* w, uint32_t columns, PackedOp* D, PackedOp* X, PackedOp* Hs) {
  if (!w || columns > w->Kcap || (X && columns > w->x_cols) || (Hs && w->N[1] == 0)) return false;
  if (D) { *D = w->A; D->rows = columns; D->K = w->M; D->mn_major = 0; }
  if (X) { *X = w->B[0]; X->rows = columns; X->K = w->N[0]; X->mn_major = 0; }
  if (Hs) { *Hs = w->B[1]; Hs->rows = columns; Hs->K = w->N[1]; Hs->mn_major = 0; }
  return true;
}
bool dyb200_wgrad_b_planes(const dyb200_wgrad* w, uint32_t col, uint32_t k, PackedOp* X, PackedOp* Hs) {
  if (!w || w->N[1] == 0 || (uint64_t)col + k > w->Kcap) return false;
  PackedOp* o[2] = {X, Hs};
  for (int j = 0; j < 2; ++j) {
    *o[j] = w->B[j];
    o[j]->rows = k; o[j]->K = w->N[j]; o[j]->mn_major = 0;
    o[j]->hi += (size_t)col * w->Np[j]; o[j]->lo += (size_t)col * w->Np[j];
  }
  return true;
}
void dyb200_wgrad_h_done(dyb200_wgrad* w) {
  w->h_col = 0xffffffffu;           // (no single step's planes are the latest)
  if (w->x_cols > w->kb) w->kb = w->x_cols;
}
int dyb200_tc_make_tmap(dyb200_ctx* ctx, void* map, float* plane, uint32_t rows, uint32_t K, uint32_t pitch, uint32_t box_rows) {
  EncodeTiledFn enc;
  int rc = get_encoder(ctx, &enc);
  if (rc) return rc;
  return make_map(ctx, enc, (CUtensorMap*)map, plane, rows, K, pitch, box_rows);
}
int dyb200_tc_make_tmap_f16(dyb200_ctx* ctx, void* map, __half* plane, uint32_t rows, uint32_t K, uint32_t pitch, uint32_t box_rows, bool mn_major) {
  EncodeTiledFn enc;
  int rc = get_encoder(ctx, &enc);
  if (rc) return rc;
  return mn_major ? make_map_mn(ctx, enc, (CUtensorMap*)map, (float*)plane, rows, K, pitch, box_rows, true)
                  : make_map(ctx, enc, (CUtensorMap*)map, (float*)plane, rows, K, pitch, box_rows, true);
}
int dyb200_tc_make_store_map(dyb200_ctx* ctx, void* map, float* C, uint32_t M, uint32_t N, uint32_t S, uint32_t ldc, uint32_t box_cols) {
  EncodeTiledFn enc;
  int rc = get_encoder(ctx, &enc);
  if (rc) return rc;
  cuuint64_t dims[3] = {M, N, S}, strides[2] = {(cuuint64_t)ldc * 4, (cuuint64_t)ldc * N * 4};
  cuuint32_t box[3] = {BM, box_cols, 1}, estr[3] = {1, 1, 1};
  CUresult r = enc((CUtensorMap*)map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, C, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return dyb200_fail(ctx, DYB200_ECUDA, "cuTensorMapEncodeTiled failed with code %d (output %u x %u, ld %u)", (int)r, M, N, ldc);
  return DYB200_OK;
}
uint32_t dyb200_tc_tile_cols(uint32_t N) { return tile_cols(N); }
uint32_t dyb200_wgrad_rows(const dyb200_wgrad* w) { return w->M; }
uint32_t dyb200_wgrad_fill(const dyb200_wgrad* w) { return w->k; }

extern "C" {

int dyb200_wgrad_create(dyb200_ctx* ctx, uint32_t M, uint32_t N0, uint32_t N1, uint32_t Kcap, dyb200_wgrad** out) {
  DYB_CHECK_ARG(ctx, out && M > 0 && N0 > 0 && Kcap > 0, "wgrad_create: bad shape");
  dyb200_wgrad* w = (dyb200_wgrad*)calloc(1, sizeof(dyb200_wgrad));
  if (!w) return dyb200_fail(ctx, DYB200_ENOMEM, "wgrad_create: host allocation failed");
  w->M = M; w->Mp = round_up(M, 32); w->N[0] = N0; w->N[1] = N1; w->Np[0] = round_up(N0, 32); w->Np[1] = round_up(N1, 32);
  w->Kcap = round_up(Kcap, 32); w->k = 0; w->kb = 0;
  w->x_cols = 0; w->h_col = 0xffffffffu; w->step = 0;
  auto alloc = [&](PackedOp* p, uint32_t rows) -> bool {
    p->rows = rows; p->K = 0; p->pitch = w->Kcap;
    size_t bytes = (size_t)rows * w->Kcap * sizeof(float);
    if (cudaMalloc((void**)&p->hi, bytes) != cudaSuccess) { cudaGetLastError(); p->hi = nullptr; return false; }
    if (cudaMalloc((void**)&p->lo, bytes) != cudaSuccess) { cudaGetLastError(); p->lo = nullptr; return false; }
    return true;
  };
  // (Kcap rows of Mp / Np floats, the same bytes as Mp / Np rows of Kcap; zeroed once so that the padding beyond M / N stays
  // finite)
  bool ok = alloc(&w->A, w->Mp) && alloc(&w->B[0], w->Np[0]) && (N1 == 0 || alloc(&w->B[1], w->Np[1]));
  if (ok) {
    w->A.rows = M; w->A.pitch = w->Mp; w->A.mn_major = 1;
    for (int j = 0; j < 2; ++j) { w->B[j].rows = w->N[j]; w->B[j].pitch = w->Np[j]; w->B[j].mn_major = 1; }
    PackedOp* ps[3] = {&w->A, &w->B[0], &w->B[1]};
    for (int q = 0; q < 3 && ok; ++q) {
      if (!ps[q]->hi) continue;
      const size_t bytes = (size_t)ps[q]->pitch * w->Kcap * sizeof(float);
      // (on the context's stream: the legacy default stream's clear could land on planes that a non-blocking stream had filled by then)
      ok = cudaMemsetAsync(ps[q]->hi, 0, bytes, ctx->stream) == cudaSuccess && cudaMemsetAsync(ps[q]->lo, 0, bytes, ctx->stream) == cudaSuccess;
    }
    if (!ok) cudaGetLastError();
  }
  if (!ok) {
    for (PackedOp* p : {&w->A, &w->B[0], &w->B[1]}) { if (p->hi) cudaFree(p->hi); if (p->lo) cudaFree(p->lo); }
    free(w);
    return dyb200_fail(ctx, DYB200_ENOMEM, "wgrad_create: cudaMalloc failed for M %u, N %u + %u, K %u", M, N0, N1, Kcap);
  }
  *out = w;
  return DYB200_OK;
}

int dyb200_wgrad_destroy(dyb200_wgrad* w) {
  if (!w) return DYB200_OK;
  for (PackedOp* p : {&w->A, &w->B[0], &w->B[1]}) { if (p->hi) cudaFree(p->hi); if (p->lo) cudaFree(p->lo); }
  free(w);
  return DYB200_OK;
}

// Appends one step: a = A_t (M x k, leading dimension lda), b0 / b1 = B_t operands (N x k) with optional
// multiplicative masks indexed like b (mask[r + (full ? ld * c : 0)]).
int dyb200_wgrad_push(dyb200_wgrad* w, uint32_t k, const float* a, uint32_t lda, const float* b0, uint32_t ldb0,
                      const float* mask0, int mask0_full, const float* b1, uint32_t ldb1, const float* mask1,
                      int mask1_full, dyb200_ctx* ctx) {
  PackJobs batch;
  dyb200_tc_pack_begin(&batch);
  int rc = dyb200_wgrad_push_batched(w, k, a, lda, b0, ldb0, mask0, mask0_full, b1, ldb1, mask1, mask1_full, ctx, &batch);
  if (rc) return rc;
  return dyb200_tc_pack_flush(ctx, &batch);
}

// C0 += A * B0^T (and C1 += A * B1^T) over everything pushed since the last flush; empties the accumulator.
int dyb200_wgrad_pack_inputs(dyb200_wgrad* w, const dyb200_tensor* x_all, const dyb200_tensor* mask_x, uint32_t step, dyb200_ctx* ctx) {
  { int rc0__ = dyb200_scratch_begin(ctx); if (rc0__) return rc0__; }
  DYB_CHECK_ARG(ctx, w && x_all && x_all->v, "wgrad_pack_inputs: null argument");
  DYB_CHECK_ARG(ctx, step > 0 || !mask_x, "wgrad_pack_inputs: steps of varying width (step = 0) take no mask");
  const uint32_t I = t_rows(x_all), n = x_all->bd;
  DYB_CHECK_ARG(ctx, t_cols(x_all) == 1 && I == w->N[0] && w->N[1] > 0 && n <= w->Kcap && (step == 0 || n % step == 0),
                "wgrad_pack_inputs: x is %u x %u, the accumulator expects %u rows, at most %u columns, whole steps of %u", I, n, w->N[0], w->Kcap, step);
  DYB_CHECK_ARG(ctx, !mask_x || (t_rows(mask_x) == I && (mask_x->bd == step || mask_x->bd == 1)), "wgrad_pack_inputs: mask shape mismatch");
  const float* mk = mask_x ? mask_x->v : nullptr;
  const int full = mask_x ? mask_x->bd == step : 0;
  PackJobs batch;
  dyb200_tc_pack_begin(&batch);
  // row = column of the sequence, reduction index of the forward product = input feature
  int rc = pack(ctx, x_all->v, I, 1, n, I, mk, I, full, w->B[0].hi, w->B[0].lo, w->Np[0], &batch, step ? step : n);
  if (!rc) rc = pack_flush_impl(ctx, &batch);
  if (rc) return rc;
  w->x_cols = n; w->step = step; w->h_col = 0xffffffffu;
  if (n > w->kb) w->kb = n;
  return DYB200_OK;
}

// Whether the two results share an element (M x N0 and M x N1, column-major): one weight read at both places, say.  Rows of one matrix side by
// side (the same leading dimension, row ranges that do not meet) do not.
static bool wgrad_results_meet(const dyb200_wgrad* w, const float* C0, uint32_t ldc0, const float* C1, uint32_t ldc1) {
  const uintptr_t a = (uintptr_t)C0, b = (uintptr_t)C1;
  const size_t na = 4 * ((size_t)ldc0 * (w->N[0] - 1) + w->M), nb = 4 * ((size_t)ldc1 * (w->N[1] - 1) + w->M);
  if (a + na <= b || b + nb <= a) return false;
  if (ldc0 != ldc1 || ldc0 < w->M || (a - b) % 4 != 0) return true;
  const uint32_t gap = (uint32_t)((a > b ? a - b : b - a) / 4 % ldc0);
  return gap < w->M || ldc0 - gap < w->M;
}
int dyb200_wgrad_flush(dyb200_wgrad* w, float* C0, uint32_t ldc0, float* C1, uint32_t ldc1, dyb200_ctx* ctx) {
  { int rc0__ = dyb200_scratch_begin(ctx); if (rc0__) return rc0__; }
  DYB_CHECK_ARG(ctx, w && C0 && (w->N[1] == 0 || C1), "wgrad_flush: null argument");
  // (pre-split inputs belong to one sequence: the next one has to call dyb200_wgrad_pack_inputs again)
  const uint32_t kb_seen = w->kb;
  w->x_cols = 0; w->h_col = 0xffffffffu;
  if (w->k == 0) { w->kb = 0; return DYB200_OK; }
  DYB_CHECK_ARG(ctx, kb_seen >= w->k, "wgrad_flush: the B operands cover %u columns, the A operand %u", kb_seen, w->k);
  PackedOp ops[3] = {w->A, w->B[0], w->B[1]};   // (MN-major: one plane row per column)
  for (PackedOp& o : ops) o.K = w->k;
  float* const C[2] = {C0, C1};
  const uint32_t ldc[2] = {ldc0, ldc1};
  int rc;
  bool done[2] = {false, w->N[1] == 0}, pairs_fit = false;
  // (results that meet are added to by one product after the other, not by the tiles of one launch)
  const bool apart = w->N[1] && wgrad_results_meet(w, C0, ldc0, C1, ldc1);
  PackedOp pairs[3];
  const uint32_t* wide;
  const bool side[2] = {w->N[0] > (uint32_t)BN, w->N[1] > (uint32_t)BN};
  if (wgrad_on_f16(w)) {
    rc = wgrad_f16_planes(ctx, w, ops, side, pairs, &wide);
    if (rc && rc != DYB200_ENOMEM) return rc;
    pairs_fit = rc == DYB200_OK;   // (without room for them the planes in hand serve)
  }
  if (pairs_fit) {
    // (a side of one tile is no product of the pair kernel and stays on the TF32 planes; by the rule at least one side is wider)
    PackedOp sides[2];
    int n = 0, at[2] = {0, 0};
    for (int j = 0; j < 2; ++j)
      if (side[j]) { done[j] = true; at[n] = j; sides[n++] = ops[1 + j]; }
    for (int q = 0; q < n; ++q) {
      const GemmEpilogue e{EPI_ACCUM, C[at[q]], ldc[at[q]], nullptr, 0, 0.f, nullptr, 0, 0};
      if ((rc = dyb200_tc_gemm_packed(ctx, w->M, sides[q].rows, 1, &pairs[0], &pairs[1 + at[q]], e, 0, wide))) return rc;
    }
    for (int q = 0; q < n; q += apart ? 1 : 2) {
      PackedOp two[2] = {sides[q], sides[1]};
      if (n == 1 || apart) two[1].rows = 0;
      if ((rc = dyb200_tc_gemm_packed2(ctx, w->M, ops[0], two, C[at[q]], ldc[at[q]], C[at[1]], ldc[at[1]], wide))) return rc;
    }
  } else if (w->N[1] && !apart) {
    if ((rc = dyb200_tc_gemm_packed2(ctx, w->M, ops[0], ops + 1, C0, ldc0, C1, ldc1))) return rc;
    done[0] = done[1] = true;
  }
  for (int j = 0; j < 2; ++j) {
    if (done[j]) continue;
    const GemmEpilogue e{EPI_ACCUM, C[j], ldc[j], nullptr, 0, 0.f, nullptr, 0, 0};
    if ((rc = dyb200_tc_gemm_packed(ctx, w->M, w->N[j], 1, &ops[0], &ops[1 + j], e))) return rc;
  }
  w->k = 0;
  w->kb = 0;
  return DYB200_OK;
}

}  // extern "C"
