// The forward recurrence of a wide layer over a sequence of few columns (lstm_wide.cu).
#pragma once
#include "common.cuh"

struct WideFwd {
  const float* Wh;                 // 4H x H, column-major
  float* gates;                    // 4H x B per step: Wx x + b on entry, gate activations on exit
  float *c, *h;                    // H x B per step
  const float *h0, *c0, *mask;     // mask of h_{t-1}: null, H or H x B
  float *hn_hi, *hn_lo;            // TF32 planes of h_{t-1} .* mask, one row per column, from the second step on (null: not wanted)
  uint32_t hn_pitch, H, B, T;
  int mask_full;
  float fb;
  unsigned long long* xchg;        // [2][B][H]: value and step number (filled in here)
  uint32_t* flags;
};
bool dyb200_wide_takes(const dyb200_ctx* ctx, uint32_t H, uint32_t B);
// *launched = false: the driver refused the launch, nothing has run.
int dyb200_wide_fwd(dyb200_ctx* ctx, WideFwd a, bool* launched);
