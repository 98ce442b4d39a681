// The recurrence of an LSTM layer of moderate width over a whole sequence (equal or shrinking batches), one launch per pass for
// one or two directions: lstm_rec.cu.  The input product Wx x + b of all steps is formed beforehand by one GEMM, and
// dx / dWx / dWh of all steps follow as one GEMM each, so that only Wh h_{t-1} (forward) and Wh^T dgates_t (backward) remain
// in the chain.
#pragma once
#include "common.cuh"

struct RecDirF {
  const float* Wh;       // 4H x H, column-major
  float* gates;          // 4H x columns: Wx x + b on entry, gate activations on exit
  float *c, *h;          // H x columns
  const float *h0, *c0;  // H x N (null: zeros)
  const float* mask;     // dropout mask of h_{t-1} (null: none)
  float *hn_hi, *hn_lo;  // TF32 planes of h_{t-1} .* mask, one row per column (null: not wanted)
};
struct RecFwd {
  RecDirF d[2];
  uint32_t H, U, T, N, G, ncap, hn_pitch;
  uint32_t first, step, cap;   // (lstm_rec.cu) cluster g has the columns first * g + step * i, i < cap
  uint32_t ndir;   // directions in the grid of lstm_rec_tc.cu, whose groups take neighbouring columns
  int mask_full;
  float fb;
  const uint32_t* prefix;   // device, T + 1 entries: step t has the columns [prefix[t], prefix[t + 1]), widths never grow (null: N each)
  uint32_t* flags;
};
struct RecDirB {
  const float* Wh;
  const float *gates, *c, *c0;
  float* dh;             // H x columns: dE/dh_t from outside on entry, complete on exit
  float* dc;             // the same for dE/dc_t (null: zero from outside, not kept)
  const float* mask;
  float *dn_hi, *dn_lo;  // TF32 planes of dgates, one row of 4H per column
  float* dbpart;         // [G][4H] row sums of dgates per cluster
};
struct RecBwd {
  RecDirB d[2];
  uint32_t H, U, T, N, G, ncap, dn_pitch;
  uint32_t first, step, cap;
  uint32_t ndir;
  int mask_full;
  const uint32_t* prefix;
  uint32_t* flags;
};

// lstm_rec_tc.cu: clusters per direction.
struct RecTcPlan { uint32_t G; };
// U hidden units per CTA, C CTAs per cluster, KD / KD2 = reduction elements per lane, G clusters per direction, room for ncap
// columns per cluster (forward, backward).  tcf / tcb: the pass runs on the tensor pipe.
struct RecPlan { uint32_t U, C, KD, KD2, Gf, Gb, ncapf, ncapb; bool tcf, tcb; RecTcPlan tf, tb; };
// False when the width is outside what the registers of a cluster hold, or N columns are more than the clusters can carry.
bool dyb200_rec_plan(dyb200_ctx* ctx, uint32_t H, uint32_t N, int ndir, RecPlan* out);
// ndir directions (1 or 2) share T, N and prefix.  U, G, ncap, the dealing of the columns and flags are filled in here.
int dyb200_rec_fwd(dyb200_ctx* ctx, const RecPlan& p, RecFwd* a, int ndir);
// db[dir] (4H) += row sums of dgates over all columns (partial sums in scratch memory).
int dyb200_rec_bwd(dyb200_ctx* ctx, const RecPlan& p, RecBwd* a, int ndir, float* const* db);
int dyb200_rec_launch_cfg(dyb200_ctx* ctx, const void* kernel, cudaLaunchConfig_t* cfg, cudaLaunchAttribute* attr, dim3 grid, uint32_t threads, size_t smem);
bool dyb200_rec_tc_plan(dyb200_ctx* ctx, bool bwd, uint32_t H, uint32_t N, int ndir, RecTcPlan* out);
int dyb200_rec_tc_fwd(dyb200_ctx* ctx, const RecTcPlan& p, RecFwd* a, int ndir);
int dyb200_rec_tc_bwd(dyb200_ctx* ctx, const RecTcPlan& p, RecBwd* a, int ndir);
