/* Internal interface between the kernel library and the C++ drivers (host/).  The LSTM recurrence of one or two directions over
 * ragged batches in one launch per pass, with its products over all columns formed outside.  Not part of the public C ABI.
 *
 * Columns are laid out step after step: step t has the columns [prefix[t], prefix[t + 1]), and the widths never grow.  The
 * inputs of all columns must have been split into the accumulator w by dyb200_wgrad_pack_inputs (step 0 or equal steps). */
#pragma once
#include "../../include/dyb200.h"
#ifdef __cplusplus
extern "C" {
#endif
typedef struct {
  const float *Wh, *h0, *c0, *mask_h;   /* h0 / c0 / mask_h may be NULL: zeros / none */
  float *gates, *c, *h;
  float *dh, *dc;                       /* backward only; dc may be NULL (zero from outside, not kept) */
  float *db;
  struct dyb200_wgrad* w;               /* may be NULL in the forward pass (no operand planes wanted) */
} dyb200i_rec_dir;

/* Steps from which a sequence is worth the fixed costs of the recurrence kernels: reading Wh into registers (3 - 5 us), the
 * separate input product and the separate dx product.  Shorter ones stay on the per-step calls. */
enum { kRecMinSteps = 8 };
/* 1 when the kernels take a layer of H units and N columns (of the widest step) on this device, and T steps are worth it. */
int dyb200i_rec_takes(dyb200_ctx* ctx, uint32_t H, uint32_t T, uint32_t N, int ndir);
/* gates = Wx x + b over the first `columns` columns, x = the input planes of w. */
int dyb200i_rec_inputs(dyb200_ctx* ctx, struct dyb200_wgrad* w, const float* Wx, const float* b, uint32_t I, uint32_t H, uint32_t columns,
                       float* gates);
int dyb200i_rec_fwd(dyb200_ctx* ctx, int ndir, const dyb200i_rec_dir* dirs, uint32_t H, uint32_t T, uint32_t N, const uint32_t* prefix_dev,
                    int mask_full, float forget_bias);
/* columns = all of them: marks the gate-gradient planes of w as filled. */
int dyb200i_rec_bwd(dyb200_ctx* ctx, int ndir, const dyb200i_rec_dir* dirs, uint32_t H, uint32_t T, uint32_t N, const uint32_t* prefix_dev,
                    int mask_full, uint32_t columns);
/* dx += Wx^T dgates (.* mask_x, which repeats every `period` columns when mask_full), dgates = the planes left in w by rec_bwd; overwrite: dx = that. */
int dyb200i_rec_dx(dyb200_ctx* ctx, struct dyb200_wgrad* w, const float* Wx, uint32_t I, uint32_t H, uint32_t columns, const float* mask_x,
                   int mask_full, uint32_t period, float* dx, int overwrite);

/* A driver whose gradient buffers hold nothing yet says so instead of clearing them: the clear is a pass of writes, and adding to zeros one of reads.
 * dyb200_affine_transform_bwd and dyb200_softmax_output_bwd_fused with `overwrite`: dEdxi, or dh alone, is written, whatever it holds. */
int dyb200i_affine_transform_bwd(const dyb200_tensor* xs, int nxs, const dyb200_tensor* fx, const dyb200_tensor* dEdf, unsigned i, dyb200_tensor* dEdxi,
                                 const void* attrs, void* aux_mem, int overwrite, dyb200_ctx* ctx);
int dyb200i_softmax_output_bwd_fused(const dyb200_tensor* x, const dyb200_tensor* h, const dyb200_tensor* R, const dyb200_tensor* dEdf, const void* aux_mem,
                                     dyb200_tensor* dR, dyb200_tensor* db, dyb200_tensor* dh, dyb200_tensor* dx_scratch, uint32_t flags, int overwrite,
                                     dyb200_ctx* ctx);
/* dyb200_vanilla_lstm_seq_bwd with `fresh` bits: dx_all is written, whatever it holds; dE/dc is zero from outside and not wanted (dc_all: scratch memory). */
enum { DYB200I_FRESH_DX = 1, DYB200I_FRESH_DC = 2 };
int dyb200i_lstm_seq_bwd(const dyb200_tensor* x_all, const dyb200_tensor* h0, const dyb200_tensor* c0, const dyb200_tensor* Wx, const dyb200_tensor* Wh,
                         const dyb200_tensor* mask_x, const dyb200_tensor* mask_h, const dyb200_lstm_gates_attrs* attrs, const dyb200_tensor* gates_all,
                         const dyb200_tensor* c_all, const dyb200_tensor* h_all, dyb200_tensor* dh_all, dyb200_tensor* dc_all, dyb200_tensor* dx_all,
                         dyb200_tensor* dWx, dyb200_tensor* dWh, dyb200_tensor* db, struct dyb200_wgrad* deferred, uint32_t steps, unsigned fresh,
                         dyb200_ctx* ctx);

/* The dependent-launch setting in force.  set >= 0 changes it, unless the caller of the library has chosen one. */
int dyb200i_dependent_launch(dyb200_ctx* ctx, int set);
#ifdef __cplusplus
}
/* A driver's own launches are ordinary ones (or what it says) unless the caller has chosen otherwise; the context is left as it was found. */
struct dyb200i_ordinary_launches {
  dyb200_ctx* ctx;
  int was;
  explicit dyb200i_ordinary_launches(dyb200_ctx* c, int dependent = 0) : ctx(c), was(dyb200i_dependent_launch(c, dependent)) {}
  ~dyb200i_ordinary_launches() { dyb200i_dependent_launch(ctx, was); }
  dyb200i_ordinary_launches(const dyb200i_ordinary_launches&) = delete;
};
/* The same for a driver with a second context of its own beside the caller's: what is in force on the caller's - its choice, or else `dependent` - holds for both. */
struct dyb200i_both_launches {
  dyb200i_ordinary_launches first, second;
  dyb200i_both_launches(dyb200_ctx* caller, dyb200_ctx* own, int dependent)
      : first(caller, dependent), second(own, dyb200i_dependent_launch(caller, -1)) {}
};
#endif
