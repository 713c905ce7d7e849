// The decode step as the mixer's window call launches it.
#pragma once
#include <cuda_runtime.h>

#include <initializer_list>

#include "../../include/m3scan.h"

namespace m3 {

// What surrounds the recurrence of a decoding step in the mixer: the projection's row, the convolution and its
// carried inputs, the B / C bias and norm, dt / lambda, the gate.
struct MixerStep {
  const void* proj;              // [batch, width]
  int width, d_inner, bc, conv_channels, K, PG;   // PG: heads per group
  int off_dt, off_lam, off_theta;                 // columns of the projection
  int has_norm;
  int vec4;                      // set by mixer_step: channels move four at a time
  float eps;
  const void* conv_in;           // [batch, K-1, conv_channels]
  void* conv_out;
  const float *conv_w, *conv_b, *dt_bias, *b_bias, *c_bias, *norm_w;
  void* out;                     // gated output; NULL: the ungated y goes to m3_step_out::y
};

// Whether the row kernels serve a shape and these (16-byte aligned) state tensors.
bool step_rows_supported(int head_dim, int d_state, int rank, std::initializer_list<const void*> state);
// One decoding step of the whole mixer as one launch.  Of the step's inputs only the state, a_log and d_skip are read
// from `d`; the rest comes from the projection.
cudaError_t mixer_step(const m3_ctx* ctx, const m3_step_desc& d, const m3_step_out& o, const MixerStep& m);

}  // namespace m3
