// The mixer's steps in front of the scan as one launch each way (m3_front.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include "../../include/m3scan.h"

namespace m3 {

// x | B C of the projection -> convolution + SiLU -> x, and B, C with bias and RMS norm in the scan's layout; dt and
// lambda.  Everything by column bands of the projection (row stride `width`).
struct Front {
  int B, T, H, N, R, K;          // heads == groups
  int di, bc, width;             // d_inner, heads * d_state * rank, the projection's width
  int off_dt, off_lam;           // columns of dt and lambda
  int reverse;                   // the second half of x, of B and of C runs right to left
  int has_norm;
  float eps;
  const void* proj;
  const void* hist;              // [B, K-1, di + 2 bc] or NULL
  const float *conv_w, *conv_b, *b_bias, *c_bias, *gain, *dt_bias;
};
struct FrontOut {
  void *x, *b, *c, *dt, *lam;    // lam NULL: lambda is not learned
  void* hist;                    // new history, or NULL
};
// Gradients: of the scan's inputs in, of the projection's x | B C, dt and lambda bands out.
struct FrontGrads {
  const void *dx, *db, *dc, *ddt, *dlam;
  void* dproj;
  float *dconv_w, *dconv_b, *db_bias, *dc_bias, *dgain, *ddt_bias;   // NULL: not wanted
  float* part;                   // front_part_floats() floats of scratch
};

bool front_supported(int dtype, const Front& f, const void* x, const void* b, const void* c);
cudaError_t front_forward(cudaStream_t st, int dtype, const Front& f, const FrontOut& o, uint64_t* launches);
size_t front_part_floats(const Front& f);
cudaError_t front_backward(cudaStream_t st, int dtype, const Front& f, const FrontGrads& g, uint64_t* launches);

}  // namespace m3
