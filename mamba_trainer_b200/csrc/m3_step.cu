// One decoding step of the Mamba-3 recurrence (the reference's mamba3_step,
// src/ssm/scan.rs:649-712, with its three fused helpers ssm_coefficients / ssm_angle /
// ssm_state_update, src/tensor/ops/fused.rs:1338-1806, folded into one launch):
//   alpha = exp(dt A), beta = (1 - lambda) dt alpha, gamma = lambda dt
//   phi   = wrap(angle + dt theta);  B^, C^ = B, C rotated by -phi
//   u     = sum_r x^(r) (x) B^^(r);  h' = alpha h + beta last_u + gamma u
//   y^(r) = C^^(r) . h' (over d_state) + D x^(r)
// Two kernels: k_step_rows for the shapes models have (d_state 64 or 128, rank 1, 2 or 4, aligned state), on its own
// or with the whole mixer step around it (m3_mixer_window); k_step, one CTA per (batch, head), for every other shape.
// The fp32 state streams through once (read h and last_u, write h' and u), which is all the traffic that matters.
#include <type_traits>

#include "m3_internal.h"
#include "m3_step.h"
#include "m3_tc_common.cuh"

namespace m3 {

constexpr int kStepMaxRank = 8;
constexpr int kStepMaxRows = 64;

// ---- the step over rows of the state ----------------------------------------------------------------------
// A CTA owns `rows` consecutive rows p of one (batch, head)'s state, which are contiguous: h and last_u arrive by two
// bulk copies requested before anything else, the prologue (the mixer's convolution, norms and activations when
// FUSED, the rotation) runs while they are under way, the update happens in place in shared memory and the new state
// leaves by two bulk copies.  No register holds state in flight, so the number of bytes in flight is that of the
// resident CTAs' buffers (the first version, with the state prefetched into registers, had 103 registers per thread
// and 25 % occupancy and ran at 2.5 TB/s; batch 64 x 32 heads x 64 x 128, rank 2: 94 us -> 64 us; 57 us with
// the prefetch of step_ahead: 77 % of the measured copy bandwidth).
// A step is latency bound while the grid is small (rows per CTA go down to 8: more CTAs) and HBM bound once it is
// large (64 rows per CTA: the prologue is shared by all of them); see step_rows_per_cta.
struct StepRows {
  m3_step_desc d;
  m3_step_out o;
  int rows;       // state rows of a CTA
  unsigned ahead; // a CTA brings into L2 what the one this many places later will read; 0: none
  int* err;       // raised when the wait for the copies gives up
  uint32_t wait_limit;
  MixerStep mx;
};

// v[V] per lane -> the sum over the L lanes of a row of v[i], i = *index, on every lane whose low bits (those below
// the halving steps) are zero: a butterfly that halves the values while it has more than one (V - 1 shuffles and
// log2(L) - log2(V) more, instead of V log2(L)).
template <int V, int L>
__device__ __forceinline__ float row_reduce(float (&v)[V], int& index, bool& writer) {
  const int lane = threadIdx.x & 31;
  int nv = V;
  index = 0;
  writer = true;
#pragma unroll
  for (int o = L / 2; o >= 1; o >>= 1) {
    if (nv > 1) {
      nv >>= 1;
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < V / 2; ++i) {
        if (i < nv) {
          const float send = up ? v[i] : v[i + nv];
          const float keep = up ? v[i + nv] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      }
      if (up) index += nv;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
      if (lane & o) writer = false;
    }
  }
  return v[0];
}

template <class T, int V>
struct alignas(V * sizeof(T)) StepVec {
  T v[V];
  __device__ __forceinline__ void load(const T* p) {
    if constexpr (V * sizeof(T) == 16) *reinterpret_cast<uint4*>(v) = __ldg(reinterpret_cast<const uint4*>(p));
    else if constexpr (V * sizeof(T) == 8) *reinterpret_cast<uint2*>(v) = __ldg(reinterpret_cast<const uint2*>(p));
    else v[0] = p[0];
  }
  __device__ __forceinline__ void store(T* p) const {
    if constexpr (V * sizeof(T) == 16) *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(v);
    else if constexpr (V * sizeof(T) == 8) *reinterpret_cast<uint2*>(p) = *reinterpret_cast<const uint2*>(v);
    else p[0] = v[0];
  }
};

// V neighbouring channels of the convolution for a single new position: the K - 1 carried inputs, then the new one;
// its SiLU, rounded to the element type.  Writes the channels' new history when `keep`.  Every load is issued before
// the first is used: in a step that fills the memory pipe a load takes microseconds, so what counts is how many of
// them a CTA waits for one after the other (a channel per thread and three rounds of them cost 35 us of a step whose
// state takes 50 us).
template <class T, int V, int KT>
__device__ __forceinline__ void conv_step(const MixerStep& m, int b, int c, const T* proj_row, bool keep, float (&out)[V]) {
  const size_t h0 = (size_t)b * (m.K - 1) * m.conv_channels + c;
  const T* hist = static_cast<const T*>(m.conv_in) + h0;
  T* next = static_cast<T*>(m.conv_out) + h0;
  StepVec<T, V> xk[KT];
  StepVec<float, V> wk[KT], acc;
#pragma unroll
  for (int k = 0; k < KT; ++k)
    if (k < m.K) {
      wk[k].load(m.conv_w + (size_t)k * m.conv_channels + c);
      xk[k].load(k < m.K - 1 ? hist + (size_t)k * m.conv_channels : proj_row + c);
    }
  if (m.conv_b) acc.load(m.conv_b + c);
  else
#pragma unroll
    for (int i = 0; i < V; ++i) acc.v[i] = 0.0f;
#pragma unroll
  for (int k = 0; k < KT; ++k)
    if (k < m.K) {
#pragma unroll
      for (int i = 0; i < V; ++i) acc.v[i] = fmaf(wk[k].v[i], ldf(xk[k].v, i), acc.v[i]);
      if (keep && k > 0) xk[k].store(next + (size_t)(k - 1) * m.conv_channels);
    }
#pragma unroll
  for (int i = 0; i < V; ++i) out[i] = round_to(proj_row, __fdividef(acc.v[i], 1.0f + __expf(-acc.v[i])));
}

// Called by one warp: requests into L2 the state of the CTA `ahead` places later in the grid and, eight regions of four
// 128-byte lines, what its prologue reads of its own (a longer region's rest is left; B, C and the parameters are shared by
// CTAs and in L2 anyway).  Hints only, of addresses that the later CTA does read.
template <class T, int N, int R, bool FUSED>
__device__ __forceinline__ void prefetch_later(const StepRows& a) {
  const m3_step_desc& d = a.d;
  const MixerStep& mx = a.mx;
  const unsigned at = blockIdx.x + blockIdx.y * gridDim.x + a.ahead;
  if (at >= gridDim.x * gridDim.y) return;
  constexpr int NH = N / 2, kElt = (int)sizeof(T);
  const int P = d.head_dim, bh = (int)(at % gridDim.x), p_lo = (int)(at / gridDim.x) * a.rows, nrows = min(P - p_lo, a.rows);
  const int lane = threadIdx.x & 31, region = lane >> 2, byte = (lane & 3) * 128;
  if (lane < 2) m3tc::bulk_prefetch((lane ? d.last_u : d.h) + ((size_t)bh * P + p_lo) * N, (uint32_t)(nrows * N * 4));
  const void* p = nullptr;
  int bytes = 0;
  if (region == 7) {
    if (d.dynamics == M3_ROTATIONAL && d.angle) p = d.angle + (size_t)bh * NH, bytes = NH * 4;
  } else if (FUSED) {
    const int h = bh % d.heads, b = bh / d.heads, col = (h * P + p_lo) * R;
    const T* pr = static_cast<const T*>(mx.proj) + (size_t)b * mx.width;
    bytes = nrows * R * kElt;
    if (region == 6) {
      p = pr + mx.off_theta + h * NH, bytes = d.dynamics == M3_ROTATIONAL ? NH * kElt : 0;
    } else if (region >= 2) {   // the carried inputs of x's channels
      p = static_cast<const T*>(mx.conv_in) + ((size_t)b * (mx.K - 1) + region - 2) * mx.conv_channels + col;
      if (region - 2 >= mx.K - 1) bytes = 0;
    } else {
      p = pr + col + (region ? mx.d_inner : 0);   // z, x
    }
  } else if (region == 0) {
    p = static_cast<const T*>(d.x) + ((size_t)bh * P + p_lo) * R, bytes = nrows * R * kElt;
  } else if (region < 3) {
    p = static_cast<const T*>(region == 1 ? d.b : d.c) + (size_t)bh * N * R, bytes = N * R * kElt;
  } else if (region == 3 && d.dynamics == M3_ROTATIONAL) {
    p = static_cast<const T*>(d.theta) + (size_t)bh * NH, bytes = NH * kElt;
  }
  if (byte < bytes) asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const char*>(p) + byte));
}

template <class T, int N, int R, int RPT, bool FUSED>
__global__ void __launch_bounds__(256, 3) k_step_rows(const __grid_constant__ StepRows a) {
  after_predecessor();
  constexpr int LPR = N / 4, RPW = 32 / LPR, PASS = 8 * RPW * RPT, NH = N / 2, JN = N / 32;
  const m3_step_desc& d = a.d;
  const m3_step_out& o = a.o;
  const MixerStep& mx = a.mx;
  __shared__ float s_b[R * N], s_c[R * N], s_cs[NH], s_sn[NH];
  __shared__ uint64_t bar;
  extern __shared__ __align__(128) float s_dyn[];   // h [rows][N], last_u [rows][N], x [rows][R], z likewise
  float *s_h = s_dyn, *s_u = s_dyn + a.rows * N, *s_x = s_u + a.rows * N, *s_z = s_x + a.rows * R;
  const int bh = blockIdx.x, h = bh % d.heads, b = bh / d.heads;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int P = d.head_dim, p_lo = blockIdx.y * a.rows, nrows = min(P - p_lo, a.rows);
  const size_t slab = ((size_t)bh * P + p_lo) * N;   // first state element of the CTA's rows
  const uint32_t slab_bytes = (uint32_t)(nrows * N * 4);
  if (tid == 224) {   // a thread of the last warp: the convolution's work items start at the first
    m3tc::mbar_init(&bar, 1);
    m3tc::fence_async_smem();
    m3tc::mbar_expect_tx(&bar, 2 * slab_bytes);
    m3tc::bulk_load(s_h, d.h + slab, slab_bytes, &bar);
    m3tc::bulk_load(s_u, d.last_u + slab, slab_bytes, &bar);
  }
  if (a.ahead && warp == 7) prefetch_later<T, N, R, FUSED>(a);
  // ---- scalars, angles -------------------------------------------------------------------------------------
  const T* pr = FUSED ? static_cast<const T*>(mx.proj) + (size_t)b * mx.width : nullptr;
  float dt, lam;
  if (FUSED) {
    dt = round_to(pr, softplus(ldf(pr, mx.off_dt + h) + (mx.dt_bias ? mx.dt_bias[h] : 0.0f)));
    lam = d.discretization == M3_LEARNED_TRAPEZOID ? round_to(pr, sigmoid(ldf(pr, mx.off_lam + h)))
                                                   : lambda_at(static_cast<const T*>(nullptr), d.discretization, 0);
  } else {
    dt = ldf(static_cast<const T*>(d.dt), bh);
    lam = lambda_at(static_cast<const T*>(d.lambda), d.discretization, bh);
  }
  // everything later steps need from memory is requested here, behind the state
  const float a_log = d.a_log[h], dsk = d.d_skip ? d.d_skip[h] : 0.0f;
  float bias[JN], gain[JN];
  if (FUSED) {
    const float* bp = warp % (2 * R) < R ? mx.b_bias : mx.c_bias;
#pragma unroll
    for (int j = 0; j < JN; ++j) {
      bias[j] = bp ? bp[(size_t)h * N + lane + 32 * j] : 0.0f;
      gain[j] = mx.has_norm && mx.norm_w ? mx.norm_w[lane + 32 * j] : 1.0f;
    }
    if (mx.out)
      for (int e = tid; e < nrows * R; e += 256) s_z[e] = ldf(pr, ((size_t)h * P + p_lo) * R + e);
  }
  const bool rot = d.dynamics == M3_ROTATIONAL;
  if (rot && tid < NH) {
    const float th = FUSED ? ldf(pr, mx.off_theta + h * NH + tid) : ldf(static_cast<const T*>(d.theta), (size_t)bh * NH + tid);
    const float a0 = d.angle ? d.angle[(size_t)bh * NH + tid] : 0.0f;
    const float ph = wrap_angle(a0 + dt * th);
    if (o.angle && blockIdx.y == 0) o.angle[(size_t)bh * NH + tid] = ph;
    sincosf(ph, &s_sn[tid], &s_cs[tid]);
  }
  // ---- x of the CTA's rows, B and C of the head ----------------------------------------------------------------
  const int nx = nrows * R;
  if (FUSED) {
    const int g = h / mx.PG;
    const bool first = blockIdx.y == 0 && h % mx.PG == 0;   // one CTA keeps the history of B's and C's channels
    const T* xband = pr + mx.d_inner;                       // the convolved band x | B C of the projection
    auto channels = [&](auto vec, auto taps) {
      constexpr int V = decltype(vec)::value, KT = decltype(taps)::value;   // KT >= K
      for (int e = V * tid; e < 2 * R * N + nx; e += V * 256) {
        float v[V], *dst;
        if (e < 2 * R * N) {
          const int which = e / (R * N), j = e - which * R * N;   // j = r * N + n, as the projection stores it
          conv_step<T, V, KT>(mx, b, mx.d_inner + which * mx.bc + g * R * N + j, xband, first, v);
          dst = (which ? s_c : s_b) + j;
        } else {
          const int j = e - 2 * R * N;
          conv_step<T, V, KT>(mx, b, (h * P + p_lo) * R + j, xband, true, v);
          dst = s_x + j;
        }
#pragma unroll
        for (int i = 0; i < V; ++i) dst[i] = v[i];
      }
    };
    if (mx.vec4 && mx.K <= 4) channels(std::integral_constant<int, 4>{}, std::integral_constant<int, 4>{});
    else channels(std::integral_constant<int, 1>{}, std::integral_constant<int, 8>{});
  } else {
    const T* bm = static_cast<const T*>(d.b) + (size_t)bh * N * R;
    const T* cm = static_cast<const T*>(d.c) + (size_t)bh * N * R;
    for (int e = tid; e < N * R; e += 256) {
      const int n = e / R, r = e % R;
      s_b[r * N + n] = ldf(bm, e);
      s_c[r * N + n] = ldf(cm, e);
    }
    const T* x = static_cast<const T*>(d.x) + ((size_t)bh * P + p_lo) * R;
    for (int e = tid; e < nx; e += 256) s_x[e] = ldf(x, e);
  }
  __syncthreads();
  // ---- bias, RMS norm, rotation: a warp per (tensor, rank), columns n = lane + 32 j, so a plane's two columns sit in
  //      one thread -------------------------------------------------------------------------------------------
  if (const int i = warp; i < 2 * R) {   // R <= 4: one row per warp at most
    float* row = (i < R ? s_b : s_c) + (i % R) * N;
    float v[JN];
#pragma unroll
    for (int j = 0; j < JN; ++j) v[j] = row[lane + 32 * j];
    if (FUSED) {
      float ss = 0.0f;
#pragma unroll
      for (int j = 0; j < JN; ++j) {
        v[j] += bias[j];
        ss = fmaf(v[j], v[j], ss);
      }
      if (mx.has_norm) {
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, s);
        const float scale = rsqrtf(ss * (1.0f / N) + mx.eps);
#pragma unroll
        for (int j = 0; j < JN; ++j) v[j] = v[j] * scale * gain[j];
      }
#pragma unroll
      for (int j = 0; j < JN; ++j) v[j] = round_to(pr, v[j]);
    }
    if (rot) {
#pragma unroll
      for (int j = 0; j < JN / 2; ++j) {
        const float cs = s_cs[lane + 32 * j], sn = s_sn[lane + 32 * j];
        const float v1 = v[j], v2 = v[j + JN / 2];
        v[j] = v1 * cs + v2 * sn;
        v[j + JN / 2] = v2 * cs - v1 * sn;
      }
    }
#pragma unroll
    for (int j = 0; j < JN; ++j) row[lane + 32 * j] = v[j];
  }
  __syncthreads();
  // ---- the state --------------------------------------------------------------------------------------------
  const float alpha = expf(dt * -expf(a_log));
  const float beta = (1.0f - lam) * dt * alpha, gamma = lam * dt;
  const int n0 = 4 * (lane % LPR), prow = warp * RPW + lane / LPR;   // this thread's columns; its row in a group of 8 RPW
  float4 bv[R], cv[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    bv[r] = *reinterpret_cast<const float4*>(&s_b[r * N + n0]);
    cv[r] = *reinterpret_cast<const float4*>(&s_c[r * N + n0]);
  }
  const bool ok = m3tc::mbar_wait(&bar, 0, a.wait_limit);
  if (!ok && a.err) m3tc::raise_flag(a.err);
  for (int p0 = 0; p0 < nrows; p0 += PASS) {
    float acc[RPT * R];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
      const int p = p0 + prow + i * 8 * RPW;
#pragma unroll
      for (int r = 0; r < R; ++r) acc[i * R + r] = 0.0f;
      if (p < nrows) {
        float4* hp = reinterpret_cast<float4*>(s_h + p * N + n0);
        float4* up = reinterpret_cast<float4*>(s_u + p * N + n0);
        const float4 hv = *hp, uv = *up;
        float u[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const float xv = s_x[p * R + r];
          u[0] += xv * bv[r].x; u[1] += xv * bv[r].y; u[2] += xv * bv[r].z; u[3] += xv * bv[r].w;
        }
        float4 hn;
        hn.x = alpha * hv.x + beta * uv.x + gamma * u[0];
        hn.y = alpha * hv.y + beta * uv.y + gamma * u[1];
        hn.z = alpha * hv.z + beta * uv.z + gamma * u[2];
        hn.w = alpha * hv.w + beta * uv.w + gamma * u[3];
        *hp = hn;
        *up = make_float4(u[0], u[1], u[2], u[3]);
#pragma unroll
        for (int r = 0; r < R; ++r) acc[i * R + r] = cv[r].x * hn.x + cv[r].y * hn.y + cv[r].z * hn.z + cv[r].w * hn.w;
      }
    }
    int idx;
    bool writer;
    const float v = row_reduce<RPT * R, LPR>(acc, idx, writer);
    const int p = p0 + prow + (idx / R) * 8 * RPW;
    if (writer && p < nrows) {
      const int r = idx % R;
      const float yv = v + dsk * s_x[p * R + r];
      const size_t oi = (size_t)(p_lo + p) * R + r;
      if (FUSED && mx.out) {
        const float z = s_z[p * R + r];
        stf(static_cast<T*>(mx.out), (size_t)bh * P * R + oi, round_to(pr, yv) * (z * sigmoid(z)));
      } else {
        stf(static_cast<T*>(o.y), (size_t)bh * P * R + oi, yv);
      }
    }
  }
  m3tc::fence_async_smem();
  __syncthreads();
  if (!ok) {  // results are invalid and reported; the copies must not outlive the CTA
    m3tc::mbar_wait(&bar, 0);
    return;
  }
  if (tid == 0) {
    m3tc::bulk_store(o.h + slab, s_h, slab_bytes);
    m3tc::bulk_store(o.last_u + slab, s_u, slab_bytes);
    m3tc::bulk_commit();
    m3tc::bulk_wait_all();
  }
}

// State rows per CTA: at most 64 (64 KB of state at d_state 128, three CTAs per SM), and as many fewer as it takes to
// have about four CTAs per SM: a small step is all latency, and the chain inside a CTA grows with its rows.
inline int step_rows_per_cta(int bh, int head_dim, int pass1) {
  int rows = head_dim < kStepMaxRows ? head_dim : kStepMaxRows;
  while (rows > pass1 && (long long)bh * ((head_dim + rows - 1) / rows) < 4 * sm_count()) rows = (rows + 1) / 2;
  return (rows + pass1 - 1) / pass1 * pass1;
}

// A grid of several waves (three CTAs per SM) is bound by the chain inside a CTA as much as by bytes: its small loads wait
// behind the state of its neighbours.  Each CTA therefore requests into L2 what the CTA one per SM later needs.
// Mixer steps, d_state 128, bf16, behind a flushed L2, us: 64 sequences x 32 heads of rank 1 / 2 / 4: 65.5 / 69.6 / 79.9 -> 59.4 / 63.5
// / 75.8; 128 x 32: 114.8 -> 100.4; 256 x 24: 170 -> 137; 24 x 24: 28.7 -> 26.6. The state alone gives half of it or less (128 x 32:
// 110.8); half a CTA per SM later is as good, two per SM 3 % worse and three 10 %: the requests take bandwidth from what is waited for.
inline unsigned step_ahead(unsigned ctas) { return ctas > 3u * sm_count() ? (unsigned)sm_count() : 0u; }

inline uint32_t step_wait_limit(const m3_ctx* ctx) { return ctx->wait_limit ? ctx->wait_limit : (1u << 18); }

template <class T, int N, int R, bool FUSED>
cudaError_t step_rows_launch(cudaStream_t st, StepRows a) {
  constexpr int kPass1 = 8 * (128 / N);   // rows of a pass with one row per thread
  a.rows = step_rows_per_cta(a.d.batch * a.d.heads, a.d.head_dim, kPass1);
  const dim3 grid(a.d.batch * a.d.heads, (a.d.head_dim + a.rows - 1) / a.rows);
  a.ahead = step_ahead(grid.x * grid.y);
  const int smem = (int)sizeof(float) * a.rows * (2 * N + 2 * R);
  auto kern = a.rows > kPass1 ? k_step_rows<T, N, R, 2, FUSED> : k_step_rows<T, N, R, 1, FUSED>;
  if (smem > 44 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
  }
  launch(kern, grid, 256, smem, st, a);
  return cudaGetLastError();
}
template <class T, int N, bool FUSED>
cudaError_t step_rows_rank(cudaStream_t st, const StepRows& a) {
  switch (a.d.rank) {
    case 1: return step_rows_launch<T, N, 1, FUSED>(st, a);
    case 2: return step_rows_launch<T, N, 2, FUSED>(st, a);
    default: return step_rows_launch<T, N, 4, FUSED>(st, a);
  }
}
template <bool FUSED>
cudaError_t step_rows(cudaStream_t st, const StepRows& a) {
  if (a.d.dtype == M3_BF16)
    return a.d.d_state == 64 ? step_rows_rank<__nv_bfloat16, 64, FUSED>(st, a) : step_rows_rank<__nv_bfloat16, 128, FUSED>(st, a);
  return a.d.d_state == 64 ? step_rows_rank<float, 64, FUSED>(st, a) : step_rows_rank<float, 128, FUSED>(st, a);
}

bool step_rows_supported(int head_dim, int d_state, int rank, std::initializer_list<const void*> state) {
  if ((d_state != 64 && d_state != 128) || (rank != 1 && rank != 2 && rank != 4)) return false;
  for (const void* p : state)
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;   // the state moves by bulk copies
  return true;
}

cudaError_t mixer_step(const m3_ctx* ctx, const m3_step_desc& d, const m3_step_out& o, const MixerStep& mixer) {
  // four channels per access (up to four taps: more would not fit the registers) where every row of the projection, the history and the parameters allows it (16-byte
  // aligned float32, 8- or 16-byte aligned elements; a head's x and the slices of it start at multiples of 8 channels)
  MixerStep m = mixer;
  const size_t es = d.dtype == M3_BF16 ? 2 : 4;
  auto ok = [](const void* p, size_t a) { return reinterpret_cast<uintptr_t>(p) % a == 0; };
  m.vec4 = m.width % 4 == 0 && m.d_inner % 4 == 0 && m.bc % 4 == 0 && (d.head_dim * d.rank) % 4 == 0 && ok(m.proj, 4 * es) &&
           ok(m.conv_in, 4 * es) && ok(m.conv_out, 4 * es) && ok(m.conv_w, 16) && ok(m.conv_b, 16);
  return step_rows<true>(ctx->stream, StepRows{d, o, 0, 0, ctx->dev_err, step_wait_limit(ctx), m});
}

template <class T>
__global__ void __launch_bounds__(256) k_step(m3_step_desc d, m3_step_out o) {
  extern __shared__ float sm[];
  const int P = d.head_dim, N = d.d_state, R = d.rank, NH = N / 2;
  float* s_b = sm;               // [R][N] rotated B
  float* s_c = s_b + R * N;      // [R][N] rotated C
  float* s_x = s_c + R * N;      // [R][P]
  const int bh = blockIdx.x, h = bh % d.heads;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const T* x = static_cast<const T*>(d.x) + (size_t)bh * P * R;
  const T* bm = static_cast<const T*>(d.b) + (size_t)bh * N * R;
  const T* cm = static_cast<const T*>(d.c) + (size_t)bh * N * R;
  const float dt = ldf(static_cast<const T*>(d.dt), bh);
  const float lam = lambda_at(static_cast<const T*>(d.lambda), d.discretization, bh);
  const float alpha = expf(dt * -expf(d.a_log[h]));
  const float beta = (1.0f - lam) * dt * alpha, gamma = lam * dt;
  const bool rot = d.dynamics == M3_ROTATIONAL;
  if (rot) {
    const T* th = static_cast<const T*>(d.theta) + (size_t)bh * NH;
    for (int m = tid; m < NH; m += 256) {
      const float a0 = d.angle ? d.angle[(size_t)bh * NH + m] : 0.0f;
      const float ph = wrap_angle(a0 + dt * ldf(th, m));
      if (o.angle) o.angle[(size_t)bh * NH + m] = ph;
      float sn, cs;
      sincosf(ph, &sn, &cs);
      for (int r = 0; r < R; ++r) {
        const float b1 = ldf(bm, (size_t)m * R + r), b2 = ldf(bm, (size_t)(m + NH) * R + r);
        const float c1 = ldf(cm, (size_t)m * R + r), c2 = ldf(cm, (size_t)(m + NH) * R + r);
        s_b[r * N + m] = b1 * cs + b2 * sn;  s_b[r * N + m + NH] = b2 * cs - b1 * sn;
        s_c[r * N + m] = c1 * cs + c2 * sn;  s_c[r * N + m + NH] = c2 * cs - c1 * sn;
      }
    }
  } else {
    for (int e = tid; e < N * R; e += 256) {
      const int n = e / R, r = e % R;
      s_b[r * N + n] = ldf(bm, e);
      s_c[r * N + n] = ldf(cm, e);
    }
  }
  for (int e = tid; e < P * R; e += 256) s_x[(e % R) * P + e / R] = ldf(x, e);
  __syncthreads();
  const float dsk = d.d_skip ? d.d_skip[h] : 0.0f;
  const float* hin = d.h + (size_t)bh * P * N;
  const float* uin = d.last_u + (size_t)bh * P * N;
  float* hout = o.h + (size_t)bh * P * N;
  float* uout = o.last_u + (size_t)bh * P * N;
  T* y = static_cast<T*>(o.y) + (size_t)bh * P * R;
  // 128-bit path: each lane owns 4 consecutive state columns per pass; it needs rows of whole float4s
  // and 16-byte aligned state tensors (a caller may hand over an offset view), else the scalar loop
  const bool vec4 = (N & 3) == 0 &&
                    !((reinterpret_cast<uintptr_t>(d.h) | reinterpret_cast<uintptr_t>(d.last_u) |
                       reinterpret_cast<uintptr_t>(o.h) | reinterpret_cast<uintptr_t>(o.last_u)) & 15);
  if (vec4) {
    for (int p = warp; p < P; p += 8) {
      float acc[kStepMaxRank];
#pragma unroll
      for (int r = 0; r < kStepMaxRank; ++r) acc[r] = 0.0f;
      for (int n = 4 * lane; n < N; n += 128) {
        const size_t i = (size_t)p * N + n;
        const float4 hv = __ldg(reinterpret_cast<const float4*>(hin + i));
        const float4 uv = __ldg(reinterpret_cast<const float4*>(uin + i));
        float u[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (int r = 0; r < R; ++r) {
          const float xv = s_x[r * P + p];
          const float4 bv = *reinterpret_cast<const float4*>(&s_b[r * N + n]);
          u[0] += xv * bv.x; u[1] += xv * bv.y; u[2] += xv * bv.z; u[3] += xv * bv.w;
        }
        float4 hn;
        hn.x = alpha * hv.x + beta * uv.x + gamma * u[0];
        hn.y = alpha * hv.y + beta * uv.y + gamma * u[1];
        hn.z = alpha * hv.z + beta * uv.z + gamma * u[2];
        hn.w = alpha * hv.w + beta * uv.w + gamma * u[3];
        *reinterpret_cast<float4*>(hout + i) = hn;
        *reinterpret_cast<float4*>(uout + i) = make_float4(u[0], u[1], u[2], u[3]);
#pragma unroll
        for (int r = 0; r < kStepMaxRank; ++r)
          if (r < R) {
            const float4 cv = *reinterpret_cast<const float4*>(&s_c[r * N + n]);
            acc[r] += cv.x * hn.x + cv.y * hn.y + cv.z * hn.z + cv.w * hn.w;
          }
      }
#pragma unroll
      for (int r = 0; r < kStepMaxRank; ++r) {
        if (r < R) {
          float v = acc[r];
#pragma unroll
          for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
          if (lane == 0) stf(y, (size_t)p * R + r, v + dsk * s_x[r * P + p]);
        }
      }
    }
    return;
  }
  for (int p = warp; p < P; p += 8) {
    float acc[kStepMaxRank];
#pragma unroll
    for (int r = 0; r < kStepMaxRank; ++r) acc[r] = 0.0f;
    for (int n = lane; n < N; n += 32) {
      float u = 0.0f;
      for (int r = 0; r < R; ++r) u += s_x[r * P + p] * s_b[r * N + n];
      const size_t i = (size_t)p * N + n;
      const float hn = alpha * hin[i] + beta * uin[i] + gamma * u;
      hout[i] = hn;
      uout[i] = u;
#pragma unroll
      for (int r = 0; r < kStepMaxRank; ++r)
        if (r < R) acc[r] += s_c[r * N + n] * hn;
    }
#pragma unroll
    for (int r = 0; r < kStepMaxRank; ++r) {
      if (r < R) {
        float v = acc[r];
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
        if (lane == 0) stf(y, (size_t)p * R + r, v + dsk * s_x[r * P + p]);
      }
    }
  }
}

}  // namespace m3

extern "C" int m3_step_forward(m3_ctx* ctx, const m3_step_desc* d, const m3_step_out* o) {
  if (!ctx) return M3_ERR_NULL;
  if (!d || !o) return m3::fail(ctx, M3_ERR_NULL, "descriptor and outputs are required");
  if (d->batch <= 0 || d->heads <= 0 || d->head_dim <= 0 || d->d_state <= 0 || d->rank <= 0)
    return m3::fail(ctx, M3_ERR_SHAPE, "extents must be positive");
  if (d->rank > m3::kStepMaxRank) return m3::fail(ctx, M3_ERR_UNSUPPORTED, "rank %d > %d in the decode step", d->rank, m3::kStepMaxRank);
  if (d->dtype != M3_F32 && d->dtype != M3_BF16) return m3::fail(ctx, M3_ERR_UNSUPPORTED, "dtype %d", d->dtype);
  if (d->dynamics == M3_ROTATIONAL && (d->d_state % 2)) return m3::fail(ctx, M3_ERR_CONFIG, "rotational dynamics require an even d_state");
  if (!d->x || !d->b || !d->c || !d->dt || !d->a_log || !d->h || !d->last_u || !o->y || !o->h || !o->last_u)
    return m3::fail(ctx, M3_ERR_NULL, "x, b, c, dt, a_log, the state and the outputs are required");
  if (d->discretization == M3_LEARNED_TRAPEZOID && !d->lambda) return m3::fail(ctx, M3_ERR_NULL, "learned trapezoid needs lambda");
  if (d->dynamics == M3_ROTATIONAL && !d->theta) return m3::fail(ctx, M3_ERR_NULL, "rotational dynamics need theta");
  if (const int rc = m3::take_device_flag(ctx, "in an earlier call, seen on entry to m3_step_forward")) return rc;
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return m3::cuda_fail(ctx, e, "cudaSetDevice");
  if (m3::step_rows_supported(d->head_dim, d->d_state, d->rank, {d->h, d->last_u, o->h, o->last_u})) {
    e = m3::step_rows<false>(ctx->stream, m3::StepRows{*d, *o, 0, 0, ctx->dev_err, m3::step_wait_limit(ctx), {}});
    if (e != cudaSuccess) return m3::cuda_fail(ctx, e, "decode step");
    ctx->launches += 1;
    return M3_OK;
  }
  const size_t smem = sizeof(float) * ((size_t)2 * d->rank * d->d_state + (size_t)d->rank * d->head_dim);
  if (smem > 200 * 1024) return m3::fail(ctx, M3_ERR_UNSUPPORTED, "decode step: rank * (2 d_state + head_dim) too large");
  const int grid = d->batch * d->heads;
  if (d->dtype == M3_BF16) {
    e = cudaFuncSetAttribute(m3::k_step<__nv_bfloat16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) m3::k_step<__nv_bfloat16><<<grid, 256, smem, ctx->stream>>>(*d, *o);
  } else {
    e = cudaFuncSetAttribute(m3::k_step<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) m3::k_step<float><<<grid, 256, smem, ctx->stream>>>(*d, *o);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return m3::cuda_fail(ctx, e, "decode step");
  ctx->launches += 1;
  return M3_OK;
}
