// The mixer's steps between its input projection and the scan, fused (src/models/mamba3.rs:340-446): depthwise causal
// convolution + SiLU over x | B C (src/nn/conv.rs:143-213), B / C bias + RMS norm + rank-last layout, dt and lambda.
// One launch forward; backward one launch and one that adds the parameter gradients' partial sums.
//
// HBM bound streaming: the projection's band is read once and x, B, C written once (backward: the band, the three
// gradients, and the band's gradient).  As separate kernels the convolution wrote its B C half for the B / C kernels to
// read back, twice in the backward pass, and both recomputed each other's values.  A warp owns 128 neighbouring
// channels of the convolution - a whole (group, rank) row of B or C at d_state 128, two at d_state 64 - four per lane,
// and walks a run of time steps with the taps' window in registers and the rows of the next four steps already
// requested; the norm's row sums are shuffles.  The warps of a block are neighbours in time (and, for ranks 2 and 4, the
// ranks of one group, whose results are interleaved through shared memory on their way out).
// bf16, 8 x 2048 tokens, 12 heads, d_state 128: forward 184 -> 100 us, backward 343 -> 270 us.
#include <cuda_bf16.h>

#include <type_traits>

#include "m3_front.h"
#include "m3_internal.h"

namespace m3 {
namespace {

constexpr int KT = 4;    // taps the kernels are compiled for: a shorter convolution has leading zero taps
constexpr int kWarps = 8;

template <class T>
struct Four;   // four neighbouring elements
template <>
struct Four<float> {
  float4 v;
  __device__ __forceinline__ void load(const float* p) { v = __ldg(reinterpret_cast<const float4*>(p)); }
  __device__ __forceinline__ void clear() { v = make_float4(0.0f, 0.0f, 0.0f, 0.0f); }
  __device__ __forceinline__ void get(float (&f)[4]) const { f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w; }
  __device__ __forceinline__ void set(const float (&f)[4]) { v = make_float4(f[0], f[1], f[2], f[3]); }
  __device__ __forceinline__ void store(float* p) const { *reinterpret_cast<float4*>(p) = v; }
};
template <>
struct Four<__nv_bfloat16> {
  uint2 v;
  __device__ __forceinline__ void load(const __nv_bfloat16* p) { v = __ldg(reinterpret_cast<const uint2*>(p)); }
  __device__ __forceinline__ void clear() { v = make_uint2(0u, 0u); }
  __device__ __forceinline__ void get(float (&f)[4]) const {
    f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xffff0000u);
    f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xffff0000u);
  }
  __device__ __forceinline__ void set(const float (&f)[4]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(f[0], f[1]), b = __floats2bfloat162_rn(f[2], f[3]);
    v.x = *reinterpret_cast<const uint32_t*>(&a);
    v.y = *reinterpret_cast<const uint32_t*>(&b);
  }
  __device__ __forceinline__ void store(__nv_bfloat16* p) const { *reinterpret_cast<uint2*>(p) = v; }
};

__device__ __forceinline__ void fma4(const float (&a)[4], const float (&b)[4], float (&c)[4]) {   // packed pairs
  const float2 lo = __ffma2_rn(make_float2(a[0], a[1]), make_float2(b[0], b[1]), make_float2(c[0], c[1]));
  const float2 hi = __ffma2_rn(make_float2(a[2], a[3]), make_float2(b[2], b[3]), make_float2(c[2], c[3]));
  c[0] = lo.x; c[1] = lo.y; c[2] = hi.x; c[3] = hi.y;
}

// Sum over the lanes of a row (N / 4 of them), on all of them.
template <int N>
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
  for (int o = N / 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The warp's place: 128 channels of the convolution from `c0 - 4 lane`, a run of time steps.
template <int N, int R>
struct Place {
  static constexpr int WR = R * N > 128 ? R * N / 128 : 1;   // warps that hold one group's ranks
  bool bc;          // B or C (else x)
  int which;        // 0: B, 1: C
  int c0;           // this lane's first channel of the convolution
  int j;            // and of its band (x, B or C)
  bool live;        // the channel exists
  bool rev;         // and runs right to left
  int tl, run, t0;  // the warp's place in time within the block, its steps, the first of them
};
template <int N, int R>
__device__ __forceinline__ Place<N, R> place(const Front& f, int bx, int nx, int nb, int run) {
  using P = Place<N, R>;
  P p;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  p.bc = bx >= nx;
  if (!p.bc) {
    p.which = 0;
    p.tl = w; p.run = run;
    p.j = bx * 128 + 4 * lane;
    p.live = p.j < f.di;
    p.c0 = p.j;
    p.rev = f.reverse && p.j >= f.di / 2;
  } else {
    const int i = bx - nx;
    p.which = i / nb;
    p.tl = w / P::WR; p.run = run * P::WR;
    p.j = ((i - p.which * nb) * P::WR + w % P::WR) * 128 + 4 * lane;
    p.live = p.j < f.bc;
    p.c0 = f.di + p.which * f.bc + p.j;
    p.rev = f.reverse && p.j >= f.bc / 2;
  }
  if (!p.live) { p.j = 0; p.c0 = p.bc ? f.di : 0; }
  p.t0 = blockIdx.y * (kWarps * run) + p.tl * p.run;
  return p;
}

// Row of scan position t of the band (the carried history for t < 0, zero where nothing is).
template <class T>
__device__ __forceinline__ void load_band(Four<T>& v, const Front& f, int b, int t, int c0, bool rev) {
  const T* proj = static_cast<const T*>(f.proj);
  const T* hist = static_cast<const T*>(f.hist);
  if (t >= 0 && t < f.T) v.load(proj + ((size_t)b * f.T + (rev ? f.T - 1 - t : t)) * f.width + f.di + c0);
  else if (t < 0 && hist && t + f.K - 1 >= 0) v.load(hist + ((size_t)b * (f.K - 1) + t + f.K - 1) * (f.di + 2 * f.bc) + c0);
  else v.clear();
}
__device__ __forceinline__ void load_taps(const Front& f, int c0, float (&wt)[KT][4], float (&bs)[4]) {
  Four<float> q;
#pragma unroll
  for (int k = 0; k < KT; ++k) {
    const int kk = k - (KT - f.K);
    if (kk >= 0) q.load(f.conv_w + (size_t)kk * (f.di + 2 * f.bc) + c0); else q.clear();
    q.get(wt[k]);
  }
  if (f.conv_b) q.load(f.conv_b + c0); else q.clear();
  q.get(bs);
}

// dt = softplus(dt_raw + bias), lambda = sigmoid(lambda_raw) of the block's steps.
template <class T>
__device__ __forceinline__ void act_forward(const Front& f, const FrontOut& o, int b, int t0, int steps) {
  const T* proj = static_cast<const T*>(f.proj);
  const int n = min(steps, f.T - t0) * f.H;
  for (int i = threadIdx.x; i < n; i += kWarps * 32) {
    const int l = i / f.H, h = i - l * f.H;
    const size_t tok = (size_t)b * f.T + t0 + l;
    const T* row = proj + tok * f.width;
    stf(static_cast<T*>(o.dt), tok * f.H + h, softplus(ldf(row, f.off_dt + h) + (f.dt_bias ? f.dt_bias[h] : 0.0f)));
    if (o.lam) stf(static_cast<T*>(o.lam), tok * f.H + h, sigmoid(ldf(row, f.off_lam + h)));
  }
}

template <class T, int N, int R, int RUN>
__global__ void __launch_bounds__(kWarps * 32) k_front_fwd(Front f, FrontOut o, int nx, int nb) {
  using P = Place<N, R>;
  constexpr int kStage = R > 1 ? kWarps * 4 * 128 : 1;
  __shared__ __align__(16) T stage[kStage];   // ranks > 1: four steps of every warp's rows, [time lane][step][n * R + r]
  const int b = blockIdx.z, lane = threadIdx.x & 31, bx = blockIdx.x;
  if (bx == nx + 2 * nb) {
    act_forward<T>(f, o, b, blockIdx.y * (kWarps * RUN), kWarps * RUN);
    return;
  }
  const P p = place<N, R>(f, bx, nx, nb, RUN);
  float wt[KT][4], bs[4], bias[4] = {0.0f, 0.0f, 0.0f, 0.0f}, gain[4] = {1.0f, 1.0f, 1.0f, 1.0f};
  load_taps(f, p.c0, wt, bs);
  const int g = p.j / (R * N), r = (p.j / N) % R, n = p.j % N;
  if (p.bc) {
    Four<float> q;
    const float* bp = p.which ? f.c_bias : f.b_bias;
    if (bp) { q.load(bp + (size_t)g * N + n); q.get(bias); }
    if (f.has_norm && f.gain) { q.load(f.gain + n); q.get(gain); }
  }
  Four<T> next[4];
  float win[KT - 1 + 4][4];   // rows t - 3 .. t + 3 of the current four steps
  {
    Four<T> v;
#pragma unroll
    for (int k = 0; k < KT - 1; ++k) {
      load_band<T>(v, f, b, p.t0 - (KT - 1) + k, p.c0, p.rev);
      v.get(win[k]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) load_band<T>(next[i], f, b, p.t0 + i, p.c0, p.rev);
  }
  for (int s = 0; s < p.run; s += 4) {
#pragma unroll
    for (int i = 0; i < 4; ++i) next[i].get(win[KT - 1 + i]);
    if (s + 4 < p.run) {
#pragma unroll
      for (int i = 0; i < 4; ++i) load_band<T>(next[i], f, b, p.t0 + s + 4 + i, p.c0, p.rev);
    }
    float y[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int e = 0; e < 4; ++e) y[i][e] = bs[e];
#pragma unroll
      for (int k = 0; k < KT; ++k) fma4(wt[k], win[i + k], y[i]);
#pragma unroll
      for (int e = 0; e < 4; ++e) y[i][e] = __fdividef(y[i][e], 1.0f + __expf(-y[i][e]));   // SiLU
    }
    if (p.bc) {
      float ss[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        ss[i] = 0.0f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          y[i][e] = round_to(static_cast<const T*>(nullptr), y[i][e]) + bias[e];
          ss[i] = fmaf(y[i][e], y[i][e], ss[i]);
        }
      }
      if (f.has_norm) {
#pragma unroll
        for (int i = 0; i < 4; ++i) ss[i] = row_sum<N>(ss[i]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float scale = rsqrtf(ss[i] * (1.0f / N) + f.eps);
#pragma unroll
          for (int e = 0; e < 4; ++e) y[i][e] = y[i][e] * scale * gain[e];
        }
      }
    }
    Four<T> q;
    if (!p.bc || R == 1) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = p.t0 + s + i;
        if (!p.live || t >= f.T) continue;
        const size_t tok = (size_t)b * f.T + (p.rev ? f.T - 1 - t : t);
        T* dst = p.bc ? static_cast<T*>(p.which ? o.c : o.b) + tok * f.bc : static_cast<T*>(o.x) + tok * f.di;
        q.set(y[i]);
        q.store(dst + p.j);
      }
    } else {
      T* st = stage + p.tl * (P::WR * 4 * 128);
      __syncthreads();   // the previous four steps have left
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) stf(st, i * (P::WR * 128) + (n + e) * R + r, y[i][e]);
      __syncthreads();
      const int e0 = 4 * ((threadIdx.x >> 5) % P::WR * 32 + lane);   // this thread's four elements of every step
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int t = p.t0 + s + i;
        if (t >= f.T) continue;
        const size_t tok = (size_t)b * f.T + (p.rev ? f.T - 1 - t : t);
        q = *reinterpret_cast<const Four<T>*>(st + i * (P::WR * 128) + e0);
        q.store(static_cast<T*>(p.which ? o.c : o.b) + (tok * f.H + g) * N * R + e0);
      }
    }
#pragma unroll
    for (int k = 0; k < KT - 1; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) win[k][e] = win[4 + k][e];
  }
  // the K - 1 inputs the next window continues from, by the warp that has the last step
  if (o.hist && p.live && p.t0 < f.T && p.t0 + p.run >= f.T) {
    Four<T> v;
    for (int k = 0; k < f.K - 1; ++k) {
      load_band<T>(v, f, b, f.T - (f.K - 1) + k, p.c0, false);
      v.store(static_cast<T*>(o.hist) + ((size_t)b * (f.K - 1) + k) * (f.di + 2 * f.bc) + p.c0);
    }
  }
}

// ---- backward ----------------------------------------------------------------------------------------------------
// Partial sums of a block (blockIdx.y, blockIdx.z): taps and bias of its channels, [K + 1][di + 2 bc]; for its B / C
// channels the gradients of the bias [bc-channel] (summed over ranks afterwards) and of the gain; dt's bias [H].
struct PartLayout {
  size_t conv, bias, gain, act, total;   // offsets within a block's floats
};
__host__ __device__ inline PartLayout part_layout(const Front& f) {
  PartLayout l;
  const size_t C = (size_t)f.di + 2 * f.bc;
  l.conv = 0;
  l.bias = (KT + 1) * C;
  l.gain = l.bias + 2 * (size_t)f.bc;
  l.act = l.gain + 2 * (size_t)f.bc;
  l.total = (l.act + f.H + 3) / 4 * 4;   // blocks store 16 bytes at a time
  return l;
}

// d dt_raw, d lambda_raw and the dt bias's partial sums of the block's steps: thread (head, time lane).
template <class T>
__device__ __forceinline__ void act_backward(const Front& f, const FrontGrads& g, int b, int t0, int steps, float* part, float* red) {
  const T* proj = static_cast<const T*>(f.proj);
  T* dproj = static_cast<T*>(g.dproj);
  constexpr int kThreads = kWarps * 32;
  for (int h0 = 0; h0 < f.H; h0 += kThreads) {
    const int nh = min(f.H - h0, kThreads), lanes = kThreads / nh, tl = threadIdx.x / nh, h = h0 + threadIdx.x % nh;
    float s = 0.0f;
    if (tl < lanes) {
      const float bias = f.dt_bias ? f.dt_bias[h] : 0.0f;
#pragma unroll 4
      for (int l = tl; l < steps; l += lanes) {
        if (t0 + l >= f.T) break;
        const size_t tok = (size_t)b * f.T + t0 + l, row = tok * f.width;
        const float v = ldf(static_cast<const T*>(g.ddt), tok * f.H + h) * sigmoid(ldf(proj, row + f.off_dt + h) + bias);
        stf(dproj, row + f.off_dt + h, v);
        s += v;
        if (g.dlam) {
          const float lam = sigmoid(ldf(proj, row + f.off_lam + h));
          stf(dproj, row + f.off_lam + h, ldf(static_cast<const T*>(g.dlam), tok * f.H + h) * lam * (1.0f - lam));
        }
      }
    }
    __syncthreads();
    red[threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.x < nh) {
      float tot = 0.0f;
      for (int i = 0; i < lanes; ++i) tot += red[i * nh + threadIdx.x];
      part[h0 + threadIdx.x] = tot;
    }
  }
}

template <class T, int N, int R, int RUN>
__global__ void __launch_bounds__(kWarps * 32, 2) k_front_bwd(Front f, FrontGrads gr, int nx, int nb) {
  using P = Place<N, R>;
  __shared__ __align__(16) float ahead[kWarps][KT - 1][128];   // g of every warp's first three steps, for the warp before it
  __shared__ __align__(16) float red[kWarps][128];
  const int b = blockIdx.z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, bx = blockIdx.x;
  const PartLayout pl = part_layout(f);
  float* part = gr.part + ((size_t)b * gridDim.y + blockIdx.y) * pl.total;
  if (bx == nx + 2 * nb) {
    act_backward<T>(f, gr, b, blockIdx.y * (kWarps * RUN), kWarps * RUN, part + pl.act, &red[0][0]);
    return;
  }
  const P p = place<N, R>(f, bx, nx, nb, RUN);
  float wt[KT][4], bs[4], bias[4] = {0.0f, 0.0f, 0.0f, 0.0f}, gain[4] = {1.0f, 1.0f, 1.0f, 1.0f};
  load_taps(f, p.c0, wt, bs);
  const int grp = p.j / (R * N), r = (p.j / N) % R, n = p.j % N;
  if (p.bc) {
    Four<float> q;
    const float* bp = p.which ? f.c_bias : f.b_bias;
    if (bp) { q.load(bp + (size_t)grp * N + n); q.get(bias); }
    if (f.has_norm && f.gain) { q.load(f.gain + n); q.get(gain); }
  }
  const T* gin = static_cast<const T*>(!p.bc ? gr.dx : (p.which ? gr.dc : gr.db));
  // the gradient of a step's four channels as the scan left it: x dense; B, C with the ranks interleaved
  auto load_grad = [&](Four<T> (&v)[R], int t) {
    if (t >= f.T) {
#pragma unroll
      for (int i = 0; i < R; ++i) v[i].clear();
      return;
    }
    const size_t tok = (size_t)b * f.T + (p.rev ? f.T - 1 - t : t);
    if (!p.bc) {
      v[0].load(gin + tok * f.di + p.j);
    } else {
      const T* src = gin + (tok * f.H + grp) * N * R + (size_t)n * R;
#pragma unroll
      for (int i = 0; i < R; ++i) v[i].load(src + 4 * i);
    }
  };
  auto pick = [&](const Four<T> (&v)[R], float (&o)[4]) {
    if (R == 1 || !p.bc) {
      v[0].get(o);
    } else {
      float all[R][4];
#pragma unroll
      for (int i = 0; i < R; ++i) v[i].get(all[i]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o[e] = 0.0f;
#pragma unroll
        for (int rr = 0; rr < R; ++rr) o[e] = rr == r ? all[(e * R + rr) / 4][(e * R + rr) % 4] : o[e];
      }
    }
  };
  float pw[KT][4], pb[4], pbias[4], pgain[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    pb[e] = pbias[e] = pgain[e] = 0.0f;
#pragma unroll
    for (int k = 0; k < KT; ++k) pw[k][e] = 0.0f;
  }
  // go = d pre of one step, from its taps' window and its gradient; own: the step feeds the parameter gradients
  auto step = [&](const float (&w0)[4], const float (&w1)[4], const float (&w2)[4], const float (&w3)[4], const Four<T> (&gv)[R],
                  bool own, float (&go)[4]) {
    float pre[4], gy[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) pre[e] = bs[e];
    fma4(wt[0], w0, pre);
    fma4(wt[1], w1, pre);
    fma4(wt[2], w2, pre);
    fma4(wt[3], w3, pre);
    pick(gv, gy);
    const float mine = own ? 1.0f : 0.0f;
    float sg[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) sg[e] = __fdividef(1.0f, 1.0f + __expf(-pre[e]));
    if (p.bc) {
      float v[4], ss = 0.0f, dot = 0.0f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[e] = round_to(static_cast<const T*>(nullptr), pre[e] * sg[e]) + bias[e];
        ss = fmaf(v[e], v[e], ss);
        dot = fmaf(gy[e] * gain[e], v[e], dot);
      }
      if (f.has_norm) {
#pragma unroll
        for (int o = N / 8; o > 0; o >>= 1) {
          ss += __shfl_xor_sync(0xffffffffu, ss, o);
          dot += __shfl_xor_sync(0xffffffffu, dot, o);
        }
        const float rstd = rsqrtf(ss * (1.0f / N) + f.eps), md = dot * rstd * (1.0f / N);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float xh = v[e] * rstd;
          pgain[e] = fmaf(mine * gy[e], xh, pgain[e]);
          gy[e] = rstd * (gy[e] * gain[e] - xh * md);
        }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) pbias[e] = fmaf(mine, gy[e], pbias[e]);
    }
    float og[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      go[e] = gy[e] * (sg[e] * (1.0f + pre[e] * (1.0f - sg[e])));   // gradients past T are zero, so go is too
      og[e] = mine * go[e];
      pb[e] += og[e];
    }
    fma4(og, w0, pw[0]);
    fma4(og, w1, pw[1]);
    fma4(og, w2, pw[2]);
    fma4(og, w3, pw[3]);
  };
  T* dband = static_cast<T*>(gr.dproj) + f.di + p.c0;
  // dx[t] = sum_delay w[K-1-delay] g[t + delay], from gw[j] = g[t + j]
  auto emit = [&](int t, const float (&g0)[4], const float (&g1)[4], const float (&g2)[4], const float (&g3)[4]) {
    if (!p.live || t < p.t0 || t >= f.T) return;
    float o[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    fma4(wt[3], g0, o);
    fma4(wt[2], g1, o);
    fma4(wt[1], g2, o);
    fma4(wt[0], g3, o);
    Four<T> q;
    q.set(o);
    q.store(dband + ((size_t)b * f.T + (p.rev ? f.T - 1 - t : t)) * f.width);
  };
  Four<T> nx_[2], ng[2][R];          // the rows of the next two steps
  float win[KT][4], gw[KT - 1][4];   // x[t-3 .. t]; g[t-3 .. t-1]
  {
    Four<T> v;
#pragma unroll
    for (int k = 0; k < KT - 1; ++k) {
      load_band<T>(v, f, b, p.t0 - (KT - 1) + k, p.c0, p.rev);
      v.get(win[k]);
#pragma unroll
      for (int e = 0; e < 4; ++e) gw[k][e] = 0.0f;
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      load_band<T>(nx_[i], f, b, p.t0 + i, p.c0, p.rev);
      load_grad(ng[i], p.t0 + i);
    }
  }
  const int last_tl = kWarps / (p.bc ? P::WR : 1) - 1, stride = p.bc ? P::WR : 1;
  // the run, then - to finish the last three rows - a few more steps by the warp that is last in time; the others take
  // the three g they need from the warp behind them
  const int total = p.tl == last_tl ? p.run + 4 : p.run;
#pragma unroll 1
  for (int s = 0; s < total; s += 2) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = p.t0 + s + i;
      nx_[i].get(win[KT - 1]);
      Four<T> gv[R];
#pragma unroll
      for (int j = 0; j < R; ++j) gv[j] = ng[i][j];
      load_band<T>(nx_[i], f, b, t + 2, p.c0, p.rev);
      load_grad(ng[i], t + 2);
      float go[4];
      step(win[0], win[1], win[2], win[3], gv, s < p.run, go);
      if (s + i < KT - 1)   // for the warp before this one in time
        *reinterpret_cast<float4*>(&ahead[warp][s + i][4 * lane]) = make_float4(go[0], go[1], go[2], go[3]);
      if (t - 3 < p.t0 + p.run) emit(t - 3, gw[0], gw[1], gw[2], go);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        gw[0][e] = gw[1][e]; gw[1][e] = gw[2][e]; gw[2][e] = go[e];
        win[0][e] = win[1][e]; win[1][e] = win[2][e]; win[2][e] = win[3][e];
      }
    }
  }
  __syncthreads();
  if (p.tl != last_tl) {
    float h[KT - 1][4];
#pragma unroll
    for (int k = 0; k < KT - 1; ++k) {
      const float4 q = *reinterpret_cast<const float4*>(&ahead[warp + stride][k][4 * lane]);
      h[k][0] = q.x; h[k][1] = q.y; h[k][2] = q.z; h[k][3] = q.w;
    }
    const int t = p.t0 + p.run - 3;
    emit(t, gw[0], gw[1], gw[2], h[0]);
    emit(t + 1, gw[1], gw[2], h[0], h[1]);
    emit(t + 2, gw[2], h[0], h[1], h[2]);
  }
  // the block's partial sums: its warps in time order, one quantity after the other (a fixed order)
  const int C = f.di + 2 * f.bc;
  auto reduce = [&](const float (&v)[4], float* dst) {
    __syncthreads();
    *reinterpret_cast<float4*>(&red[warp][4 * lane]) = make_float4(v[0], v[1], v[2], v[3]);
    __syncthreads();
    if (p.tl == 0 && p.live) {
      float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      for (int w = warp; w < kWarps; w += stride) {
        const float4 q = *reinterpret_cast<const float4*>(&red[w][4 * lane]);
        s.x += q.x; s.y += q.y; s.z += q.z; s.w += q.w;
      }
      *reinterpret_cast<float4*>(dst) = s;
    }
  };
#pragma unroll
  for (int k = 0; k < KT; ++k) reduce(pw[k], part + pl.conv + (size_t)k * C + p.c0);
  reduce(pb, part + pl.conv + (size_t)KT * C + p.c0);
  if (p.bc) {
    reduce(pbias, part + pl.bias + (size_t)p.which * f.bc + p.j);
    reduce(pgain, part + pl.gain + (size_t)p.which * f.bc + p.j);
  }
}

// out[c] = sum over blocks (for the B / C bias over the ranks too) of the partial sums, in a fixed order: block (32, 32)
// owns 32 columns, thread row y every 32nd term, the 32 row sums are added in order.  blockIdx.y: which gradient; the
// gain's columns are summed row by row of B and C here and over the rows by k_front_gain.
__global__ void __launch_bounds__(1024) k_front_sums(Front f, FrontGrads g, int nblk) {
  __shared__ float red[32][33];
  const PartLayout pl = part_layout(f);
  const int C = f.di + 2 * f.bc, c = blockIdx.x * 32 + threadIdx.x;
  float* out = nullptr;
  int ncols = 0, inner = 1, istride = 0;
  size_t off = 0;
  switch (blockIdx.y) {
    case 0: out = g.dconv_w; ncols = f.K * C; off = pl.conv + (size_t)(KT - f.K) * C + c; break;
    case 1: out = g.dconv_b; ncols = C; off = pl.conv + (size_t)KT * C + c; break;
    case 2:
    case 3:
      out = blockIdx.y == 2 ? g.db_bias : g.dc_bias;
      ncols = f.H * f.N; inner = f.R; istride = f.N;
      off = pl.bias + (blockIdx.y == 3 ? f.bc : 0) + (size_t)(c / f.N) * f.R * f.N + c % f.N;
      break;
    case 4: out = g.dgain ? g.part + (size_t)nblk * pl.total : nullptr; ncols = 2 * f.bc; off = pl.gain + c; break;
    default: out = g.ddt_bias; ncols = f.H; off = pl.act + c; break;
  }
  if (!out || blockIdx.x * 32 >= ncols) return;
  float s = 0.0f;
  if (c < ncols) {
    const int n = nblk * inner;
#pragma unroll 4
    for (int t = threadIdx.y; t < n; t += 32) {
      const int blk = inner == 1 ? t : t / inner;
      s += g.part[(size_t)blk * pl.total + off + (size_t)(t - blk * inner) * istride];
    }
  }
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < ncols) {
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; ++i) tot += red[i][threadIdx.x];
    out[c] = tot;
  }
}

__global__ void __launch_bounds__(1024) k_front_gain(const float* __restrict__ rows, int nrows, int N, float* __restrict__ out) {
  __shared__ float red[32][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  float s = 0.0f;
  for (int t = threadIdx.y; t < nrows; t += 32) s += rows[(size_t)t * N + c];
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0) {
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; ++i) tot += red[i][threadIdx.x];
    out[c] = tot;
  }
}

// Steps per warp: sixteen amortise the window's start and the warp's parameters; a grid of fewer than four blocks per SM
// is cut finer so that every SM has work.
int front_run(const Front& f, int tiles) {
  const long long blocks = (long long)tiles * f.B * ((f.T + kWarps * 16 - 1) / (kWarps * 16));
  return blocks >= 4 * 148 ? 16 : 4;
}
template <int N, int R>
void front_tiles(const Front& f, int* nx, int* nb) {
  constexpr int kCh = 128 * Place<N, R>::WR;
  *nx = (f.di + 127) / 128;
  *nb = (f.bc + kCh - 1) / kCh;
}

template <class T, int N, int R>
cudaError_t forward_t(cudaStream_t st, const Front& f, const FrontOut& o) {
  int nx, nb;
  front_tiles<N, R>(f, &nx, &nb);
  const int run = front_run(f, nx + 2 * nb);
  const dim3 grid(nx + 2 * nb + 1, (f.T + kWarps * run - 1) / (kWarps * run), f.B);
  if (run == 16) k_front_fwd<T, N, R, 16><<<grid, kWarps * 32, 0, st>>>(f, o, nx, nb);
  else k_front_fwd<T, N, R, 4><<<grid, kWarps * 32, 0, st>>>(f, o, nx, nb);
  return cudaGetLastError();
}
template <class T, int N, int R>
cudaError_t backward_t(cudaStream_t st, const Front& f, const FrontGrads& g) {
  int nx, nb;
  front_tiles<N, R>(f, &nx, &nb);
  const int run = front_run(f, nx + 2 * nb), C = f.di + 2 * f.bc;
  const dim3 grid(nx + 2 * nb + 1, (f.T + kWarps * run - 1) / (kWarps * run), f.B);
  if (run == 16) k_front_bwd<T, N, R, 16><<<grid, kWarps * 32, 0, st>>>(f, g, nx, nb);
  else k_front_bwd<T, N, R, 4><<<grid, kWarps * 32, 0, st>>>(f, g, nx, nb);
  k_front_sums<<<dim3((f.K * C + 31) / 32, 6), dim3(32, 32), 0, st>>>(f, g, (int)(grid.y * grid.z));
  if (g.dgain)
    k_front_gain<<<N / 32, dim3(32, 32), 0, st>>>(g.part + part_layout(f).total * grid.y * grid.z, 2 * f.H * R, N, g.dgain);
  return cudaGetLastError();
}

template <class F>
auto dispatch(int dtype, const Front& f, F fn) {
  auto with_rank = [&](auto t, auto n) {
    if (f.R == 1) return fn(t, n, std::integral_constant<int, 1>{});
    if (f.R == 2) return fn(t, n, std::integral_constant<int, 2>{});
    return fn(t, n, std::integral_constant<int, 4>{});
  };
  auto with_n = [&](auto t) {
    return f.N == 64 ? with_rank(t, std::integral_constant<int, 64>{}) : with_rank(t, std::integral_constant<int, 128>{});
  };
  return dtype == M3_BF16 ? with_n(__nv_bfloat16{}) : with_n(float{});
}

}  // namespace

// Four elements per access: every row and column offset a multiple of four, every base aligned to four elements, the
// float32 parameters to 16 bytes; a direction change must not fall inside a lane's four channels.
bool front_supported(int dtype, const Front& f, const void* x, const void* b, const void* c) {
  if ((f.N != 64 && f.N != 128) || (f.R != 1 && f.R != 2 && f.R != 4) || f.K < 1 || f.K > KT) return false;
  if (f.B > 65535 || (f.T + 31) / 32 > 65535) return false;
  if (f.width % 4 || f.di % (f.reverse ? 8 : 4) || f.bc % (f.reverse ? 8 : 4)) return false;
  const uintptr_t a = dtype == M3_BF16 ? 7 : 15;
  for (const void* p : {f.proj, f.hist, x, b, c})
    if (reinterpret_cast<uintptr_t>(p) & a) return false;
  for (const float* p : {f.conv_w, f.conv_b, f.b_bias, f.c_bias, f.gain})
    if (reinterpret_cast<uintptr_t>(p) & 15) return false;
  return true;
}

cudaError_t front_forward(cudaStream_t st, int dtype, const Front& f, const FrontOut& o, uint64_t* launches) {
  if (launches) *launches += 1;
  return dispatch(dtype, f, [&](auto t, auto n, auto r) { return forward_t<decltype(t), n.value, r.value>(st, f, o); });
}

size_t front_part_floats(const Front& f) {
  int nx, nb;
  dispatch(M3_F32, f, [&](auto, auto n, auto r) { front_tiles<n.value, r.value>(f, &nx, &nb); return 0; });
  const int run = front_run(f, nx + 2 * nb);
  return part_layout(f).total * f.B * ((f.T + kWarps * run - 1) / (kWarps * run)) + 2 * (size_t)f.bc;
}

cudaError_t front_backward(cudaStream_t st, int dtype, const Front& f, const FrontGrads& g, uint64_t* launches) {
  if (launches) *launches += g.dgain ? 3 : 2;
  return dispatch(dtype, f, [&](auto t, auto n, auto r) { return backward_t<decltype(t), n.value, r.value>(st, f, g); });
}

}  // namespace m3
