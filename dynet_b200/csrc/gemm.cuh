// Internal GEMM interface shared by the LSTM nodes and dyb200_gemm.
//   C[M x N] = epilogue( sum_p op(A_p)[M x K_p] * (op(B_p) .* mask_p)[K_p x N] )
// All matrices are column-major fp32.  Up to two (A, B) pairs accumulate into the same
// tile, which is how the gate pre-activation Wx*x + Wh*h is formed in one kernel.
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"

struct GemmPair {
  const float* A; uint32_t lda; int transA;   // op(A)(m,k) = transA ? A[k + lda*m] : A[m + lda*k]
  const float* B; uint32_t ldb; int transB;   // op(B)(k,n) = transB ? B[n + ldb*k] : B[k + ldb*n]
  uint32_t K;
  // optional multiplicative mask on B, indexed like B's storage: element at (row r, col c)
  // of the stored matrix uses mask[r + (mask_full ? mask_ld * c : 0)]  (dropout masks, bd 1 or B)
  const float* maskB; uint32_t mask_ld; int mask_full;
  int a_is_param;   // A is a parameter matrix: its packed form may be kept in the context's parameter cache
};

enum GemmEpiMode {
  EPI_STORE = 0,      // C = acc
  EPI_ACCUM = 1,      // C += acc
  EPI_GATES = 2,      // C = act(acc + bias[m] + (H <= m < 2H ? forget_bias : 0)); sigmoid for m < 3H, tanh above
  EPI_ACCUM_MASK = 3, // C += acc * maskC[m + (maskc_full ? maskc_ld * n : 0)]
  EPI_BIAS = 4,       // C = acc + bias[m]   (column vector broadcast over the N columns)
  // The A operand was packed with interleaved gate rows (dyb200_tc_param_gates): tile t, row 32 q + l is gate q
  // (i, f, o, g) of hidden unit u = 32 t + l.  gates[q H + u, n] = act(acc + bias + forget bias) as in EPI_GATES,
  // then c_out[u, n] = i g + f c_prev[u, n] and h_out[u, n] = o tanh(c) (VanillaLSTMC / VanillaLSTMH forward).
  EPI_LSTM_CELL = 5
};

struct GemmEpilogue {
  int mode;
  float* C; uint32_t ldc;
  const float* bias; uint32_t H; float forget_bias;
  const float* maskC; uint32_t maskc_ld; int maskc_full;
  // Optional second destination: rows m >= split_m go to C2 (row m - split_m) with their own leading dimension and
  // mask; split_m = 0 disables it.  Lets one product with stacked A operands ([Wx; Wh]^T) feed two tensors.
  uint32_t split_m = 0;
  float* C2 = nullptr; uint32_t ldc2 = 0;
  const float* maskC2 = nullptr; uint32_t maskc2_ld = 0; int maskc2_full = 0;
  // EPI_LSTM_CELL only: previous cell state and the two outputs, all H x N with leading dimension H
  const float* c_prev = nullptr; float* c_out = nullptr; float* h_out = nullptr;
  // EPI_LSTM_CELL, optional: h .* hmask also goes out as split operand planes (row = batch column, H values each): the
  // K-major right operand of the next time step's gate product and, read MN-major, the right operand of the layer's
  // weight-gradient product.  16-byte aligned, H % 4 == 0.
  float* hn_hi = nullptr; float* hn_lo = nullptr; uint32_t hn_pitch = 0;
  const float* hmask = nullptr; uint32_t hmask_ld = 0; int hmask_full = 0;
  // Two right operands side by side (TmapPack::n_split): columns [0, n_live) belong to C, those from n_split on to Cn, the ones between do not exist.
  uint32_t n_split = 0, n_live = 0; float* Cn = nullptr; uint32_t ldcn = 0;
};
#ifdef __CUDACC__
// The destination of a tile whose first column is n0 (a tile lies on one side): C, n0 and the end of its columns N.
__device__ __forceinline__ void epi_side(GemmEpilogue& e, uint32_t& n0, uint32_t& N) {
  if (!e.n_split) return;
  if (n0 >= e.n_split) { e.C = e.Cn; e.ldc = e.ldcn; n0 -= e.n_split; N -= e.n_split; }
  else N = e.n_live;
}
#endif
#ifdef __CUDACC__
// h .* mask of four hidden units [u, u + 4) of batch column n, written as operand planes (see GemmEpilogue::hn_hi).
__device__ __forceinline__ void epi_emit_h(const GemmEpilogue& epi, uint32_t u, uint32_t n, float4 h) {
  if (epi.hmask) {
    const float4 mk = *reinterpret_cast<const float4*>(epi.hmask + u + (epi.hmask_full ? (size_t)epi.hmask_ld * n : 0));
    h.x *= mk.x; h.y *= mk.y; h.z *= mk.z; h.w *= mk.w;
  }
  float4 hi, lo;
  split_tf32(h.x, hi.x, lo.x); split_tf32(h.y, hi.y, lo.y); split_tf32(h.z, hi.z, lo.z); split_tf32(h.w, hi.w, lo.w);
  *reinterpret_cast<float4*>(epi.hn_hi + (size_t)n * epi.hn_pitch + u) = hi;
  *reinterpret_cast<float4*>(epi.hn_lo + (size_t)n * epi.hn_pitch + u) = lo;
}
#endif
#ifdef __CUDACC__
// ---- 2 x 11 bits in fp16 ---------------------------------------------------------------------------------------------------
// A TF32 hi / lo pair carries 2 x 11 significand bits.  fp16 has the same 11, at twice the rate of the tensor pipe and half the
// bytes, with 5 bits of exponent.  So an operand row is scaled by a power of two that brings its largest
// element to [2^14, 2^15), hi = fp16(x s), lo = fp16((x s - hi) 2^11): elements down to 2^-28 of the row's largest keep all
// 2 x 11 bits, smaller ones an absolute error below 2^-50 of it.  Per k step: A_hi x [B_hi | B_lo] as ONE instruction of twice
// the columns (B_lo lies right behind B_hi in shared memory), whose halves are the accumulators D1 (hi hi) and D2, then
// A_lo x B_hi into D2; the result is (D1 + 2^-11 D2) / (s_a s_b).  A chain of D1 is one third of the accumulations of the TF32
// chain for the same K (the tensor core truncates at each), so chains are cut every 1024 of K here.
// A scale word is the bit pattern of the row's largest finite |x|: the scale is 2^(141 - E), E its exponent field.
__device__ __forceinline__ int scale_field(uint32_t word) {   // E, kept where both the scale and its inverse are normal numbers
  const int e = (int)(word >> 23);
  return e < 27 ? 27 : e;
}
// |v| as the word that maxima are taken of: bit pattern, infinities and NaNs (which come through a split as they are) count as 0
__device__ __forceinline__ uint32_t finite_mag(float v) {
  const uint32_t u = __float_as_uint(v) & 0x7fffffffu;
  return u < 0x7f800000u ? u : 0u;
}
// Whether a magnitude loses bits to the scale of its row: it is not zero and lies 2^28 below the largest one.
__device__ __forceinline__ bool pair_loses(uint32_t mag, uint32_t word) { return mag && (int)(mag >> 23) + 28 <= scale_field(word); }
__device__ __forceinline__ float scale_of(uint32_t word) { return __int_as_float((268 - scale_field(word)) << 23); }
__device__ __forceinline__ float inv_scale_of(uint32_t word) { return __int_as_float((scale_field(word) - 14) << 23); }   // 2^(E - 141)
// v 2^(Ea + Eb - 282): in two factors, so that nothing overflows on the way to a result that does not
__device__ __forceinline__ float unscale(float v, int t) {
  const int h = t >> 1;
  return (v * __int_as_float((h + 127) << 23)) * __int_as_float((t - h + 127) << 23);
}
constexpr float kLoScale = 1.0f / 2048.0f;
__device__ __forceinline__ void split_f16(float xs, __half& hi, __half& lo) {
  hi = __float2half_rn(xs);
  lo = __float2half_rn((xs - __half2float(hi)) * 2048.0f);
}
#endif
// Row m of the product -> destination pointer of column 0, leading dimension and mask of that row.
struct EpiRow { float* c; uint32_t ldc; const float* mask; uint32_t mask_ld; int mask_full; };
__host__ __device__ inline EpiRow epi_row(const GemmEpilogue& e, uint32_t m) {
  if (e.split_m && m >= e.split_m) {
    const uint32_t r = m - e.split_m;
    return EpiRow{e.C2 + r, e.ldc2, e.maskC2 ? e.maskC2 + r : nullptr, e.maskc2_ld, e.maskc2_full};
  }
  return EpiRow{e.C + m, e.ldc, e.maskC ? e.maskC + m : nullptr, e.maskc_ld, e.maskc_full};
}

// fp32 CUDA-core path: any shape, any alignment.
int dyb200_gemm_simt(dyb200_ctx* ctx, uint32_t M, uint32_t N, int npairs, const GemmPair* pairs, const GemmEpilogue& epi);
// fp32 path for products of few columns (gemm_thin.cu): whether the dispatcher gives it a product, the product itself, and the
// LSTM step built on it (gates, c and h; pre_in_gates: epi.C holds Wx x + b of the step and only Wh h is added).
bool dyb200_thin_columns(uint32_t M, uint32_t N, uint32_t K);
bool dyb200_thin_takes(uint32_t M, uint32_t N, int npairs, const GemmPair* pairs, const GemmEpilogue& epi);
int dyb200_gemm_thin(dyb200_ctx* ctx, uint32_t M, uint32_t N, int npairs, const GemmPair* pairs, const GemmEpilogue& epi);
int dyb200_lstm_thin(dyb200_ctx* ctx, uint32_t H, uint32_t B, int npairs, const GemmPair* pairs, int pre_in_gates, const GemmEpilogue& epi);
// fp32 path for products with a narrow side and a long one (gemm_narrow.cu).
bool dyb200_narrow_takes(uint32_t M, uint32_t N, int npairs, const GemmPair* pairs, const GemmEpilogue& epi);
int dyb200_gemm_narrow(dyb200_ctx* ctx, uint32_t M, uint32_t N, const GemmPair& p, const GemmEpilogue& epi);
// 3xTF32 tensor-pipe path (tcgen05 + TMEM + TMA); returns DYB200_ERUNTIME with *handled = 0
// when the shape/alignment is outside what it supports.
int dyb200_gemm_tc(dyb200_ctx* ctx, uint32_t M, uint32_t N, int npairs, const GemmPair* pairs, const GemmEpilogue& epi,
                   int* handled);
// Dispatcher: tensor path when eligible, else the CUDA-core path.
int dyb200_gemm_fused(dyb200_ctx* ctx, uint32_t M, uint32_t N, int npairs, const GemmPair* pairs, const GemmEpilogue& epi);

// ---- pieces of the tensor path, for entry points that reuse one packed operand in several products ----
// TF32 hi / lo planes of an operand: `rows` rows (m or n) of K values.  K-major (mn_major = 0): element (r, k) at
// plane[r * pitch + k].  MN-major (left operands of dyb200_tc_gemm_packed only): element (r, k) at plane[k * pitch + r] -
// the K-major planes of the transposed matrix, used as they are.
// f16: the planes hold scaled fp16 pairs instead (below; hi / lo then point at halves, K-blocks are 64 wide) and `scale` the
// scale words of the rows.
struct PackedOp {
  float* hi; float* lo; uint32_t rows, K, pitch; uint32_t mn_major = 0;
  uint32_t f16 = 0; const uint32_t* scale = nullptr;
};
// ---- fp16 operand planes ----
// One operand as `lines` lines of n contiguous values (line i at src + ld i), its planes laid out alike.  Every ROW of the operand has
// a scale of its own: one word per line (F16_LINE: lines are rows of a K-major operand) or per position in the line (F16_ELEM:
// positions are rows of an MN-major operand).  A matrix that is read both ways needs both sets of planes: with one scale for all of
// it, rows 2^28 below its largest value would lose their bits.
enum F16Scale { F16_LINE = 0, F16_ELEM = 1 };
// src_lo: the source is a pair of TF32 planes, src the hi one (null: plain fp32).
constexpr int kF16MaxJobs = 3;
constexpr uint32_t kF16PadMax = 16384;
struct F16Job { const float* src; uint32_t ld, lines, n, pitch; int mode; uint32_t* scale; __half* hi; __half* lo; const float* src_lo = nullptr;
  uint32_t perm_H = 0;        // (F16_ELEM) positions are gate rows q perm_H + u, written interleaved as dyb200_tc_param_gates does
  uint32_t mark = 0;          // (F16_LINE) 1: four values side by side that all lose bits to their line's scale (pair_loses) become zeros, bit 0 of its word says so
  uint32_t pad_H = 0;         // (F16_LINE, lines of at most kF16PadMax values) values are gate units q pad_H + u, written at q (pad_H rounded up to 64) + u, zeros between
  uint32_t* low = nullptr; };   // (F16_ELEM) a word per position, see F16Jobs::wide
// wide: becomes 1 where the values of a position span more than a pair holds: of its blocks of eight lines that are not all zero, one's largest
// value lies more than 2^kF16Span below the position's (jobs with `low` words).  words: scale and low words and the flag of all
// jobs, cleared at once (null: each job's scale words by themselves).
constexpr int kF16Span = 24;
struct F16Jobs { F16Job job[kF16MaxJobs]; int n; uint32_t start[kF16MaxJobs + 1];   // start: units of work before each job (set for a launch)
  uint32_t* wide = nullptr; uint32_t* words = nullptr; size_t n_words = 0; };
// Planes and scale words for a job from the scratch arena; dyb200_f16_pack fills those of up to three jobs in one pass each.
int dyb200_f16_planes(dyb200_ctx* ctx, const float* src, uint32_t ld, uint32_t lines, uint32_t n, int mode, F16Job* job, uint32_t pad_H = 0);
int dyb200_f16_pack(dyb200_ctx* ctx, F16Jobs* jobs);
// The same for a parameter, from the parameter cache when it is on.
int dyb200_f16_param(dyb200_ctx* ctx, const float* src, uint32_t ld, uint32_t lines, uint32_t n, int mode, F16Job* job, uint32_t pad_H = 0, uint32_t mark = 0);
PackedOp dyb200_f16_op(const F16Job& j, bool mn_major);
// The gate weights of a layer, Wx (4H x I) and Wh (4H x H), as MN-major planes with interleaved rows (lines = their columns, 128 rows per 32 units) and one
// scale word per row of Wx and one per row of Wh (4H words each, not interleaved); from the parameter cache when it is on.
struct F16Gates { __half *x_hi, *x_lo, *h_hi, *h_lo; const uint32_t* scale; };
int dyb200_f16_gates(dyb200_ctx* ctx, const float* Wx, const float* Wh, uint32_t I, uint32_t H, F16Gates* out);
// Products that use fp16 pairs, by useful flops.  Finding the scales adds a clear and a pass over the operands; us with TF32 / fp16 pairs,
// splitting included: 1500^3 (6.8 GFLOP) 43 / 45, 1024 x 256 x 13000 (6.8) 77 / 75, 2000 x 2000 x 1000 (8.0) 50 / 39, 4096 x 512 x 2240 (9.4)
// 74 / 68, 10000 x 512 x 1024 (10.5) 89 / 74, 2048^3 (17) 96 / 61, 10000 x 1024 x 1120 (23) 192 / 99.  A short reduction is bound by its result
// either way (1024 x 107000 x 128, 28 GFLOP: 200 / 217); from 24 GFLOP on it takes the pairs for their smaller error.
inline bool dyb200_f16_takes(double flops, uint32_t K) { return flops >= 24.0e9 || (flops >= 8.0e9 && K >= 256); }
// A queue of packing work that one kernel launch executes (several small operands per launch).
constexpr int kMaxPackJobs = 8;
constexpr int kLayoutGates = 2, kLayoutF16 = 3, kLayoutGatesF16 = 5, kLayoutPadF16 = 6, kLayoutMarkF16 = 7;   // (kLayoutF16 + F16_LINE or F16_ELEM; the last two: F16Job::pad_H, mark)
struct PackJob {
  const float* src; const float* mask; float* hi; float* lo;
  uint32_t ld, rows, K, mask_ld, pitch, gx, perm_H;
  uint32_t mask_period;   // > 0: a full mask repeats every mask_period batch columns (one mask for every time step of a sequence)
  int k_is_fast, mask_full, vec;
};
struct PackJobs { PackJob job[kMaxPackJobs]; uint32_t start[kMaxPackJobs + 1]; int n; };
inline void dyb200_tc_pack_begin(PackJobs* b) { b->n = 0; b->start[0] = 0; }
int dyb200_tc_pack_flush(dyb200_ctx* ctx, PackJobs* batch);
// Packs `rows x K` (element (r, k) at src[k + ld*r] when k_is_fast, else src[r + ld*k]) times an optional mask
// into planes taken from the scratch arena (valid until the current entry point returns).  With a batch the work is
// only queued: the planes are filled when the batch is flushed.
int dyb200_tc_pack(dyb200_ctx* ctx, const float* src, uint32_t ld, bool k_is_fast, uint32_t rows, uint32_t K,
                   const float* mask, uint32_t mask_ld, int mask_full, PackedOp* out, PackJobs* batch = nullptr);
// Same for a parameter matrix: served from the parameter cache when it is on.
int dyb200_tc_param(dyb200_ctx* ctx, const float* src, uint32_t ld, bool k_is_fast, uint32_t rows, uint32_t K, PackedOp* out,
                    PackJobs* batch = nullptr);   // (batch: a caller that cannot launch it increments ctx->param_version)
// A gate weight matrix (rows = 4H, element (r, k) at src[r + ld * k]) with its rows interleaved for EPI_LSTM_CELL.
int dyb200_tc_param_gates(dyb200_ctx* ctx, const float* src, uint32_t ld, uint32_t rows, uint32_t K, PackedOp* out);
// Number of K splits dyb200_tc_gemm_packed will use for this shape (1 = the epilogue runs in the MMA kernel).
uint32_t dyb200_tc_splits(const dyb200_ctx* ctx, uint32_t M, uint32_t N, uint32_t kb_total);
// Two parameter matrices with the same K and leading dimension stacked along the rows: rows [0, rows) from src,
// rows [rows, rows + rows2) from src2.
int dyb200_tc_param2(dyb200_ctx* ctx, const float* src, uint32_t rows, const float* src2, uint32_t rows2, uint32_t ld,
                     bool k_is_fast, uint32_t K, PackedOp* out);
// force_splits > 0: that many K splits (normalised so that no split is empty) instead of the cost model's choice.
// unless (products of the pair kernel): a device word; where it is not zero the product is left out.
int dyb200_tc_gemm_packed(dyb200_ctx* ctx, uint32_t M, uint32_t N, int npairs, const PackedOp* A, const PackedOp* B,
                          const GemmEpilogue& epi, uint32_t force_splits = 0, const uint32_t* unless = nullptr);
int dyb200_splitk_reduce(dyb200_ctx* ctx, const float* part, uint32_t S, uint32_t M, uint32_t N, const GemmEpilogue& epi, size_t split_stride = 0,
                         const uint32_t* unless = nullptr);
// C0 += A B0^T and C1 += A B1^T in one launch (TF32 planes, all MN-major; dWx and dWh of a layer).  only_if: a device word; where it is zero
// the launch does nothing (then B[1].rows may be 0, and the launch is one tile per CTA).
int dyb200_tc_gemm_packed2(dyb200_ctx* ctx, uint32_t M, const PackedOp& A, const PackedOp* B, float* C0, uint32_t ldc0, float* C1, uint32_t ldc1,
                           const uint32_t* only_if = nullptr);
// Tiling of the backward recurrence of an LSTM layer (dx_t, dh_{t-1} += [Wx; Wh]^T dgates_t), shared by the per-step call
// and the sequence kernel so that both add the same partial sums: tile width, batch-column blocks per CTA of the sequence
// kernel (1 or 2) and K splits.  False when the shape does not suit the sequence kernel (the per-step call then lets the
// cost model choose).
struct LstmBwdTiling { uint32_t bn, ncb, S; };
bool dyb200_lstm_bwd_tiling(const dyb200_ctx* ctx, uint32_t I, uint32_t H, uint32_t B, LstmBwdTiling* out);
bool dyb200_tc_eligible(uint32_t M, uint32_t N, double flops);
// Planes of `rows x K` taken from the scratch arena, left for the caller's kernel to fill.
int dyb200_tc_planes(dyb200_ctx* ctx, uint32_t rows, uint32_t K, PackedOp* out);
struct dyb200_wgrad;
// The accumulator's A planes (dgates of all columns) are MN-major: one row of `pitch` floats per column, M values each.  The
// reserve calls hand out the rows of k columns for the caller's kernel to fill (a_hi / a_lo point at the first of them);
// the same rows are a K-major right operand (rows = columns, K = M) for the caller's own products.
int dyb200_wgrad_reserve(dyb200_wgrad* w, uint32_t k, float** a_hi, float** a_lo, uint32_t* pitch, const float* b0, uint32_t ldb0,
                         const float* mask0, int mask0_full, const float* b1, uint32_t ldb1, const float* mask1, int mask1_full,
                         dyb200_ctx* ctx, PackJobs* batch);
void dyb200_wgrad_unreserve(dyb200_wgrad* w, uint32_t k);   // takes the last k columns back (dyb200_wgrad_reserve)
int dyb200_wgrad_push_b_at(dyb200_wgrad* w, uint32_t col, uint32_t k, const float* b0, uint32_t ldb0, const float* mask0, int mask0_full,
                           const float* b1, uint32_t ldb1, const float* mask1, int mask1_full, dyb200_ctx* ctx, PackJobs* batch);
int dyb200_wgrad_reserve_a_at(dyb200_wgrad* w, uint32_t col, uint32_t k, float** a_hi, float** a_lo, uint32_t* pitch, dyb200_ctx* ctx);
int dyb200_wgrad_pack_a_at(dyb200_wgrad* w, uint32_t col, uint32_t k, const float* a, uint32_t lda, dyb200_ctx* ctx, PackJobs* batch);
uint32_t dyb200_wgrad_rows(const dyb200_wgrad* w);
// Pre-split sequence inputs (dyb200_wgrad_pack_inputs): the forward operand planes of the step that starts at column `col`,
// when they are available.  x: rows [col, col + k) of the planes filled by dyb200_wgrad_pack_inputs; h: the planes the
// previous step's LSTM epilogue wrote for this column.  Return false when the caller has to split that input itself.
bool dyb200_wgrad_x_planes(const dyb200_wgrad* w, uint32_t col, uint32_t k, PackedOp* out);
bool dyb200_wgrad_h_planes(const dyb200_wgrad* w, uint32_t col, uint32_t k, PackedOp* out);
// Destinations for the split planes of the NEXT step's h input (the step that starts at column col + k), or false when
// there is no next step or the inputs were not pre-split.  Marks those planes as the h input of column col + k.
bool dyb200_wgrad_next_h(dyb200_wgrad* w, uint32_t col, uint32_t k, GemmEpilogue* epi);
uint32_t dyb200_wgrad_fill(const dyb200_wgrad* w);
int dyb200_wgrad_push_batched(dyb200_wgrad* w, uint32_t k, const float* a, uint32_t lda, const float* b0, uint32_t ldb0,
                              const float* mask0, int mask0_full, const float* b1, uint32_t ldb1, const float* mask1,
                              int mask1_full, dyb200_ctx* ctx, PackJobs* batch);

// ---- sequence kernels (lstm_seq.cu) ----
// Operand planes of a whole sequence held by an accumulator after dyb200_wgrad_pack_inputs: X = x .* mask_x (row = column
// of the sequence, K = I), Hs = h_tm1 .* mask_h (row = column, K = H; rows [c, c + step) are the input of the step that
// starts at column c).  False when they are not in place for `steps` steps of `step` columns.
struct SeqPlanes { PackedOp X, Hs; };
bool dyb200_wgrad_seq_planes(const dyb200_wgrad* w, uint32_t steps, uint32_t step, SeqPlanes* out);
int dyb200_wgrad_seq_h0(dyb200_wgrad* w, const float* h0, const float* mh, int mh_full, dyb200_ctx* ctx, PackJobs* batch);
void dyb200_wgrad_seq_done(dyb200_wgrad* w);
// For kernels that run a whole sequence of equal or ragged steps (lstm_rec.cu): the first `columns` columns as K-major right
// operands - D = dgates (K = M), X = inputs of dyb200_wgrad_pack_inputs (K = I), Hs = h inputs (K = H); null: not asked for.
// False when X is asked for and the inputs of that many columns are not in place.  dyb200_wgrad_h_done: all Hs rows are written.
bool dyb200_wgrad_column_planes(const dyb200_wgrad* w, uint32_t columns, PackedOp* D, PackedOp* X, PackedOp* Hs);
void dyb200_wgrad_h_done(dyb200_wgrad* w);
// The planes of columns [col, col + k) of both right operands, filled or to be filled.
bool dyb200_wgrad_b_planes(const dyb200_wgrad* w, uint32_t col, uint32_t k, PackedOp* X, PackedOp* Hs);
// The forward product of a layer on fp16 pairs (lstm_seq.cu): T steps of B columns, or a single one driven from outside - the same kernel, so
// the same bits.  Whether a shape takes it, with its tile width and K splits; the call, whose inputs are planes of the accumulator.
bool dyb200_seq_f16_plan(dyb200_ctx* ctx, uint32_t I, uint32_t H, uint32_t B, uint32_t* bn, uint32_t* S);
struct SeqF16Call {
  uint32_t I, H, B, T;
  const float *Wx, *Wh, *b, *h0, *c0, *mh; int mh_full; float forget_bias;
  float *gates, *c, *h;
  PackedOp X, Hs;          // TF32 planes of the columns' inputs (X without lo: the inputs themselves); rows [0, B) of Hs are filled here unless h0_done, the later
                           // ones by the kernel (without hi: not wanted)
  int h0_done, emit_last;  // emit_last: rows [T B, (T + 1) B) of Hs receive the last step's h
};
int dyb200_seq_f16(dyb200_ctx* ctx, const SeqF16Call& q);
// The backward pass of a wide layer on fp16 pairs (lstm_bwd_wide.cu): T steps of B columns, or a single one driven from outside - the same kernels, so
// the same bits.  Whether a layer takes it, with the column blocks per CTA and K splits of its recurrence; the call.
bool dyb200_bwd_wide_plan(dyb200_ctx* ctx, uint32_t H, uint32_t B, uint32_t* ncb, uint32_t* S);
struct BwdWideCall {
  uint32_t I, H, B, T;
  const float *Wx, *Wh, *gates, *c, *c0;
  float *dh, *dc;                // of all steps; a single step without dE/dc has none
  float *dh_prev, *dc_prev;      // of the step before the first, or null
  float* dx; const float* mx; int mx_full; const float* mh; int mh_full;   // (dx null: not wanted)
  float* db;
  float *dn_hi, *dn_lo; uint32_t dn_pitch;   // TF32 planes of the columns' dgates, to be filled
  int fresh_dx, fresh_dc;        // dx is written, whatever it holds; dc holds nothing yet: zeros from outside
};
int dyb200_bwd_wide(dyb200_ctx* ctx, const BwdWideCall& q);
// db += row sums of dgates, part = [step][tile][G], tiles in order and then the steps (at most kDbMaxSteps); clears the counters at `done`, if any
constexpr uint32_t kDbMaxSteps = 256;
int dyb200_seq_db(dyb200_ctx* ctx, const float* part, uint32_t steps, uint32_t tiles, uint32_t G, float* db, uint32_t* done);
// A 2-D tensor map (CUtensorMap, 128 bytes at `map`) over a K-major plane: box = 32 floats of K x box_rows rows, 128-byte swizzle.
int dyb200_tc_make_tmap(dyb200_ctx* ctx, void* map, float* plane, uint32_t rows, uint32_t K, uint32_t pitch, uint32_t box_rows);
// The same over a plane of halves (64 of K), and over an MN-major one (K lines of `rows` halves).
int dyb200_tc_make_tmap_f16(dyb200_ctx* ctx, void* map, __half* plane, uint32_t rows, uint32_t K, uint32_t pitch, uint32_t box_rows, bool mn_major);
// A 3-D tensor map over S matrices side by side (M x N each, leading dimension ldc, 16-byte aligned): box = 128 rows x box_cols columns.
int dyb200_tc_make_store_map(dyb200_ctx* ctx, void* map, float* C, uint32_t M, uint32_t N, uint32_t S, uint32_t ldc, uint32_t box_cols);
// Products of fp16 pairs on pairs of SMs (gemm_pair.cu).
bool dyb200_pair_takes(const dyb200_ctx* ctx, uint32_t M, uint32_t N, const GemmEpilogue& epi);
uint32_t dyb200_tc_tile_cols(uint32_t N);   // width of the output tile the tensor path uses for N columns (64 or 128)
