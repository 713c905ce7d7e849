// Host-side interface of the tensor-core kernel family.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/m3scan.h"

namespace m3 {

// Shapes the family serves: bf16, head_dim 64, d_state 128, rank 1, 2 or 4.
// 16-byte alignment: the kernels move rows as 16-byte vectors and bulk tensor copies.
inline bool tc_aligned(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline bool tc_supported(const m3_scan_desc& s) {
  return s.dtype == M3_BF16 && s.head_dim == 64 && s.d_state == 128 && (s.rank == 1 || s.rank == 2 || s.rank == 4) &&
         s.seq > 0 && tc_aligned(s.x) && tc_aligned(s.b) && tc_aligned(s.c) && tc_aligned(s.theta) && s.theta_stride % 8 == 0;
}
// Time steps per 128-row tile and tiles per stripe.
inline int tc_tile_steps(int rank) { return 128 / rank; }
inline int tc_tiles(int seq, int rank) { return (seq + tc_tile_steps(rank) - 1) / tc_tile_steps(rank); }

// A tensor map over the rows of a dense [B, T, H, cols] bf16 tensor as the caller stores them:
// dimensions (cols, H, T, B), box (64, 1, steps, 1), so 64 columns of `steps` consecutive time steps of
// one (batch, head) land as a dense [steps][128 bytes] panel (one request per 64 columns), rows past
// either end of the sequence arriving as zeros.  With `swizzle` the 16-byte chunks of a panel row are
// XOR-swizzled by row & 7 (the 128-byte swizzle; the panel must then start on a 1024-byte boundary).
// cols a multiple of 64; needs a 16-byte aligned base.
// `tok_stride`: elements between consecutive tokens (0: dense, H * cols; else a multiple of 8 for a band of a wider row).
bool tc_make_row_map(CUtensorMap* map, const void* base, int B, int T, int H, int cols, int steps, bool swizzle, int tok_stride = 0);

struct TcFwdParams {
  alignas(64) CUtensorMap tm_b, tm_c;         // row maps of b and c
  alignas(64) CUtensorMap tm_th;              // row map of theta (rotational dynamics)
  alignas(64) CUtensorMap tm_y;               // row map of y: its tiles leave by bulk tensor stores when out_maps
  int out_maps;
  const __nv_bfloat16 *x, *b, *c, *dt, *lam, *theta;
  const float *a_log, *d_skip, *h0, *lu0, *angle0;
  __nv_bfloat16* y;
  float *h_out, *lu_out, *angle_out;
  __nv_bfloat16* ckpt_h;  // [BH, tiles, 64 x 128 operand tile] bf16 state entering each tile, or NULL
  float* ckpt_angle;  // [BH, tiles, 64] angle entering each tile, or NULL
  int* err;           // device flag set when a bounded wait gave up
  int B, T, H, R, disc;
  int rev;            // the last `rev` heads walk time right to left
  int ths;            // elements between consecutive tokens of theta
  uint32_t wait_limit; // iteration limit of the bounded waits (m3_ctx_set_wait_limit)
  // time segments of a stripe (work distribution in m3_tc_roles.cuh): nseg == 1 hands nothing over
  int nseg, tps, grid;
  int ahead;          // 1: seg_state and seg_angle hold every boundary's state before the launch (m3_tc_ahead.cu)
  float *seg_state, *seg_angle;
  int* seg_flag;
};

// What a 128-row tile takes inside a stripe, microseconds measured on a B200: what plans weigh cuts by.
inline float tc_tile_us(bool backward, bool rot, int rank) {
  if (backward) return !rot ? 10.0f : (rank == 1 ? 14.2f : 13.2f);
  return rank == 1 ? (rot ? 5.3f : 4.6f) : (rot ? 4.5f : 3.8f);
}

// How a launch of the stripe kernels cuts its stripes in time (m3_tc_fwd.cu).  Returns segments per stripe, tiles per
// segment and the grid; bytes of hand-over scratch (state, angle, flags) through *scratch_bytes.
void tc_segment_plan(int BH, int tiles, bool allow_split, bool backward, bool rot, int rank, int* nseg, int* tps, int* grid,
                     size_t* scratch_bytes);

// Segments that run side by side (m3_tc_ahead.cu): the state and angle at every boundary are worked out first, in the
// seg_state / seg_angle the stripe kernels read, and nothing is handed over.
struct Dims;
struct TcAhead {
  int nseg, tps;                  // segments of a stripe, tiles of a segment
  int gps, gt;                    // groups of a segment, tiles of a group
  float *hs, *asum, *cd;          // per group
  float *seg_state, *seg_angle;   // per segment
};
bool tc_ahead_plan(int BH, int tiles, bool backward, bool rot, int rank, int* nseg, int* tps);
// nseg and tps given: fills in the rest; bytes of scratch.
size_t tc_ahead_bytes(int BH, TcAhead* a, char* base);
// dy NULL: forward; else the gradient of the state (dh: the one reaching the returned state, or NULL).  full_angle: the
// forward pass of a training step.
cudaError_t tc_ahead(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const void* dy, const float* dh,
                     const float* ckpt_angle, const TcAhead& a, bool full_angle, uint64_t* launches);

cudaError_t tc_forward(cudaStream_t st, const TcFwdParams& p, bool rotational);
// load_kernels of every kernel that a forward pass may launch.
cudaError_t tc_load();
cudaError_t tc_ahead_load();
struct TcBwdParams {
  alignas(64) CUtensorMap tm_b, tm_c, tm_x, tm_dy, tm_th;  // row maps of the inputs and dy
  alignas(64) CUtensorMap tm_dx, tm_db, tm_dc; // row maps of the gradients asked for: their tiles leave by bulk tensor stores when out_maps
  int out_maps;
  const __nv_bfloat16 *x, *b, *c, *dt, *lam, *theta, *dy;
  const float *a_log, *d_skip, *h0, *lu0;
  const float *dh, *dlu, *dangle;        // gradients reaching the returned state, or NULL
  const __nv_bfloat16* ckpt_h;           // written by the forward pass
  const float* ckpt_angle;
  __nv_bfloat16 *dx, *db, *dc, *dtheta;  // NULL skips the store
  float *da, *dg, *dw, *ddt_rot;         // [BH, tiles * steps] per-token scalars for the final pass
  float *partA, *partD;                  // [BH, tiles] partial sums of d a_log / d d_skip
  float *ip0;                            // [BH] <dH_0, last_u0>
  float *dh0, *dlu0, *dangle0;           // NULL skips the store
  int* err;
  int B, T, H, R, disc;
  int rev;            // the last `rev` heads walk time right to left
  int ths;            // elements between consecutive tokens of theta and d theta
  uint32_t wait_limit;
  int nseg, tps, grid;   // as in TcFwdParams; the gradient of the state and the running sum of d phi are handed over
  int ahead;             // with it, the sums of d phi stay within a segment: dphi [BH, tiles * steps, 64] receives them and
  float *dphi, *dpsum;   // dpsum [BH, nseg, 64] the segments' totals, for k_rows_final to finish
  float *seg_state, *seg_angle;
  int* seg_flag;
};

cudaError_t tc_backward(cudaStream_t st, const TcBwdParams& p, bool rotational);

}  // namespace m3
