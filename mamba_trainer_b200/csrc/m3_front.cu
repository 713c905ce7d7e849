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
// bf16, 8 x 2048 tokens, 12 heads, d_state 128, device time: forward 184 -> 69 us, backward 343 -> 174 us (and 12 us of sums).
#include <cuda_bf16.h>

#include <type_traits>

#include "m3_front.h"
#include "m3_internal.h"

namespace m3 {
namespace {

constexpr int KT = 4;    // taps the kernels are compiled for: a shorter convolution has leading zero taps
constexpr int kWarps = 8;    // of a block of the forward kernel
constexpr int kBwdWarps = 4; // and of the backward one, whose threads need up to 170 registers: three blocks per SM

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

// Two floats per instruction (packed fp32): of all resources these kernels use instruction issue most (64 % of the slots
// forward, 47 % backward, where the chains of a step take the rest; DRAM 38 and 26 %).
__device__ __forceinline__ void mul4(const float (&a)[4], const float (&b)[4], float (&c)[4]) {
  const float2 lo = __fmul2_rn(make_float2(a[0], a[1]), make_float2(b[0], b[1]));
  const float2 hi = __fmul2_rn(make_float2(a[2], a[3]), make_float2(b[2], b[3]));
  c[0] = lo.x; c[1] = lo.y; c[2] = hi.x; c[3] = hi.y;
}
__device__ __forceinline__ void add4(const float (&a)[4], const float (&b)[4], float (&c)[4]) {
  const float2 lo = __fadd2_rn(make_float2(a[0], a[1]), make_float2(b[0], b[1]));
  const float2 hi = __fadd2_rn(make_float2(a[2], a[3]), make_float2(b[2], b[3]));
  c[0] = lo.x; c[1] = lo.y; c[2] = hi.x; c[3] = hi.y;
}
__device__ __forceinline__ float dot4(const float (&a)[4], const float (&b)[4]) {
  const float2 s = __ffma2_rn(make_float2(a[2], a[3]), make_float2(b[2], b[3]),
                              __fmul2_rn(make_float2(a[0], a[1]), make_float2(b[0], b[1])));
  return s.x + s.y;
}
// sigmoid of four values by the special-function unit (2 ulp each step, denormals flushed: without that every
// exponential and reciprocal carries three more instructions).
__device__ __forceinline__ void sigmoid4(const float (&v)[4], float (&s)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    float x, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(x) : "f"(v[e] * -1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.0f + x));
    s[e] = r;
  }
}
// Rounded to the element type, four at a time.
__device__ __forceinline__ void round4(const float*, float (&)[4]) {}
__device__ __forceinline__ void round4(const __nv_bfloat16*, float (&v)[4]) {
  Four<__nv_bfloat16> q;
  q.set(v);
  q.get(v);
}

__device__ __forceinline__ void fma4(const float (&a)[4], const float (&b)[4], float (&c)[4]) {   // packed pairs
  const float2 lo = __ffma2_rn(make_float2(a[0], a[1]), make_float2(b[0], b[1]), make_float2(c[0], c[1]));
  const float2 hi = __ffma2_rn(make_float2(a[2], a[3]), make_float2(b[2], b[3]), make_float2(c[2], c[3]));
  c[0] = lo.x; c[1] = lo.y; c[2] = hi.x; c[3] = hi.y;
}

// Sums over the lanes of a row (N / 4 of them) of V = 2 or 4 values, on all of them: the halves of the row first split the
// values between them, and the totals come back by V shuffles - 7 or 10 instead of 10 or 20.
template <int N, int V>
__device__ __forceinline__ void row_sums(float (&v)[V]) {
  constexpr int L = N / 4;
  const int lane = threadIdx.x & 31;
  int nv = V;
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) {
    if (nv > 1) {
      nv >>= 1;
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < V / 2; ++i)
        if (i < nv) {
          const float send = up ? v[i] : v[i + nv], keep = up ? v[i + nv] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  const float mine = v[0];   // lane bits L/2 (and L/4): which value
#pragma unroll
  for (int i = 0; i < V; ++i) v[i] = __shfl_sync(0xffffffffu, mine, (lane & ~(L - 1)) | (i * (L / V)));
}

// The warp's place: 128 channels of the convolution from `c0 - 4 lane`, a run of time steps.
template <int N, int R>
struct Place {
  static constexpr int WR = R * N > 128 ? R * N / 128 : 1;   // warps that hold one group's ranks
  bool bc;          // B or C (else x)
  int which;        // 0: B, 1: C
  int base;         // the block's first channel of its band (x, B or C)
  int c0;           // this lane's first channel of the convolution
  int j;            // and of its band
  bool live;        // the channel exists (a lane past the band's end reads the band's first channels and stores nothing)
  bool rev;         // and runs right to left
  int tl, run, t0;  // the warp's place in time within the block, its steps, the first of them
};
template <int N, int R, int WARPS>
__device__ __forceinline__ Place<N, R> place(const Front& f, int bx, int nx, int nb, int run) {
  using P = Place<N, R>;
  P p;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  p.bc = bx >= nx;
  if (!p.bc) {
    p.which = 0;
    p.tl = w; p.run = run;
    p.base = bx * 128;
    p.j = p.base + 4 * lane;
  } else {
    const int i = bx - nx;
    p.which = i / nb;
    p.tl = w / P::WR; p.run = run * P::WR;
    p.base = (i - p.which * nb) * P::WR * 128;
    p.j = p.base + w % P::WR * 128 + 4 * lane;
  }
  const int width = p.bc ? f.bc : f.di;
  p.live = p.j < width;
  if (!p.live) p.j = 0;
  p.c0 = (p.bc ? f.di + p.which * f.bc : 0) + p.j;
  p.rev = f.reverse && p.j >= width / 2;
  p.t0 = blockIdx.y * (WARPS * run) + p.tl * p.run;
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
__global__ void __launch_bounds__(kWarps * 32, 3) k_front_fwd(Front f, FrontOut o, int nx, int nb) {
  after_predecessor();
  using P = Place<N, R>;
  constexpr int kStage = R > 1 ? kWarps * 4 * 128 : 1;
  __shared__ __align__(16) T stage[kStage];   // ranks > 1: four steps of every warp's rows, [time lane][step][n * R + r]
  const int b = blockIdx.z, lane = threadIdx.x & 31, bx = blockIdx.x;
  if (bx == nx + 2 * nb) {
    act_forward<T>(f, o, b, blockIdx.y * (kWarps * RUN), kWarps * RUN);
    return;
  }
  const P p = place<N, R, kWarps>(f, bx, nx, nb, RUN);
  float wt[KT][4], bs[4], bias[4] = {0.0f, 0.0f, 0.0f, 0.0f}, gain[4] = {1.0f, 1.0f, 1.0f, 1.0f};
  load_taps(f, p.c0, wt, bs);
  const int g = p.j / (R * N), r = (p.j / N) % R, n = p.j % N;
  if (p.bc) {
    Four<float> q;
    const float* bp = p.which ? f.c_bias : f.b_bias;
    if (bp) { q.load(bp + (size_t)g * N + n); q.get(bias); }
    if (f.has_norm && f.gain) { q.load(f.gain + n); q.get(gain); }
  }
  // `inside`: every row this warp touches is one of the sequence's, so rows are reached by adding a stride
  auto walk = [&](auto inside) {
    constexpr bool IN = decltype(inside)::value;
    const ptrdiff_t xs = p.rev ? -(ptrdiff_t)f.width : (ptrdiff_t)f.width;
    const T* px = static_cast<const T*>(f.proj) + ((ptrdiff_t)b * f.T + (p.rev ? f.T - 1 - p.t0 : p.t0)) * f.width + f.di + p.c0;
    auto row = [&](Four<T>& v, int s) {   // x of step t0 + s
      if (IN) v.load(px + s * xs); else load_band<T>(v, f, b, p.t0 + s, p.c0, p.rev);
    };
    const size_t ow = p.bc ? f.bc : f.di;
    T* out = p.bc ? static_cast<T*>(p.which ? o.c : o.b) : static_cast<T*>(o.x);
    out += ((size_t)b * f.T + (p.rev ? f.T - 1 - p.t0 : p.t0)) * ow;
    const ptrdiff_t os = p.rev ? -(ptrdiff_t)ow : (ptrdiff_t)ow;
    Four<T> next[4];
    float win[KT - 1 + 4][4];   // rows t - 3 .. t + 3 of the current four steps
    {
      Four<T> v;
#pragma unroll
      for (int k = 0; k < KT - 1; ++k) {
        row(v, k - (KT - 1));
        v.get(win[k]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) row(next[i], i);
    }
#pragma unroll 1
    for (int s = 0; s < p.run; s += 4) {
#pragma unroll
      for (int i = 0; i < 4; ++i) next[i].get(win[KT - 1 + i]);
      if (s + 4 < p.run) {
#pragma unroll
        for (int i = 0; i < 4; ++i) row(next[i], s + 4 + i);
      }
      float y[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float sg[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) y[i][e] = bs[e];
#pragma unroll
        for (int k = 0; k < KT; ++k) fma4(wt[k], win[i + k], y[i]);
        sigmoid4(y[i], sg);
        mul4(y[i], sg, y[i]);   // SiLU
      }
      if (p.bc) {
        float ss[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          round4(static_cast<const T*>(nullptr), y[i]);
          add4(y[i], bias, y[i]);
          ss[i] = dot4(y[i], y[i]);
        }
        if (f.has_norm) {
          row_sums<N, 4>(ss);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float r_ = rsqrtf(ss[i] * (1.0f / N) + f.eps);
            const float scale[4] = {r_, r_, r_, r_};
            mul4(y[i], scale, y[i]);
            mul4(y[i], gain, y[i]);
          }
        }
      }
      Four<T> q;
      if (!p.bc || R == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (!IN && (!p.live || p.t0 + s + i >= f.T)) continue;
          q.set(y[i]);
          q.store(out + (s + i) * os + p.j);
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
          if (!IN && p.t0 + s + i >= f.T) continue;
          q = *reinterpret_cast<const Four<T>*>(st + i * (P::WR * 128) + e0);
          q.store(out + (s + i) * os + g * N * R + e0);
        }
      }
#pragma unroll
      for (int k = 0; k < KT - 1; ++k)
#pragma unroll
        for (int e = 0; e < 4; ++e) win[k][e] = win[4 + k][e];
    }
  };
  // (the ranks of a group meet at block barriers in there, and the walk of inside blocks stores without asking for `live`:
  // the choice is the block's)
  const int blk = blockIdx.y * (kWarps * RUN), ch = p.bc ? 128 * P::WR : 128;
  if (blk >= KT - 1 && blk + kWarps * RUN <= f.T && p.base + ch <= (p.bc ? f.bc : f.di)) walk(std::true_type{});
  else walk(std::false_type{});
  // the K - 1 inputs the next window continues from, by the warp that has the last step
  if (o.hist && p.live && p.t0 < f.T && p.t0 + p.run >= f.T) {
    Four<T> v;
    for (int k = 0; k < f.K - 1; ++k) {
      load_band<T>(v, f, b, f.T - (f.K - 1) + k, p.c0, false);
      v.store(static_cast<T*>(o.hist) + ((size_t)b * (f.K - 1) + k) * (f.di + 2 * f.bc) + p.c0);
    }
  }
}

constexpr int kAhead = 8;   // steps by which the backward walk's rows are brought into L2 before they are loaded
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

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

// Behind the blocks' sums: the gain's columns row by row of B and C, and how many of them k_front_sums has finished.
__host__ __device__ inline unsigned* gain_count(const Front& f, const FrontGrads& g, size_t nblk) {
  return reinterpret_cast<unsigned*>(g.part + part_layout(f).total * nblk + 2 * (size_t)f.bc);
}

// d dt_raw, d lambda_raw and the dt bias's partial sums of the block's steps: thread (head, time lane).
template <class T>
__device__ __forceinline__ void act_backward(const Front& f, const FrontGrads& g, int b, int t0, int steps, float* part, float* red) {
  const T* proj = static_cast<const T*>(f.proj);
  T* dproj = static_cast<T*>(g.dproj);
  constexpr int kThreads = kBwdWarps * 32;
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
__global__ void __launch_bounds__(kBwdWarps * 32, 3) k_front_bwd(Front f, FrontGrads gr, int nx, int nb) {
  after_predecessor();
  using P = Place<N, R>;
  __shared__ __align__(16) float ahead[kBwdWarps][KT - 1][128];   // g of every warp's first three steps, for the warp before it
  __shared__ __align__(16) float red[kBwdWarps][128];
  const int b = blockIdx.z, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, bx = blockIdx.x;
  const PartLayout pl = part_layout(f);
  float* part = gr.part + ((size_t)b * gridDim.y + blockIdx.y) * pl.total;
  if (bx == 0 && blockIdx.y == 0 && b == 0 && threadIdx.x == 0) *gain_count(f, gr, (size_t)gridDim.y * gridDim.z) = 0u;
  if (bx == nx + 2 * nb) {
    act_backward<T>(f, gr, b, blockIdx.y * (kBwdWarps * RUN), kBwdWarps * RUN, part + pl.act, &red[0][0]);
    return;
  }
  const P p = place<N, R, kBwdWarps>(f, bx, nx, nb, RUN);
  float wt[KT][4], bs[4], bias[4] = {0.0f, 0.0f, 0.0f, 0.0f}, gain[4] = {1.0f, 1.0f, 1.0f, 1.0f};
  load_taps(f, p.c0, wt, bs);
  const int grp = p.j / (R * N), r = (p.j / N) % R, n = p.j % N;
  if (p.bc) {
    Four<float> q;
    const float* bp = p.which ? f.c_bias : f.b_bias;
    if (bp) { q.load(bp + (size_t)grp * N + n); q.get(bias); }
    if (f.has_norm && f.gain) { q.load(f.gain + n); q.get(gain); }
  }
  const T* gin = static_cast<const T*>(!p.bc ? gr.dx : (p.which ? gr.dc : gr.db)) + (p.bc ? (grp * N + n) * R : p.j);
  const size_t gwid = p.bc ? (size_t)f.bc : (size_t)f.di;
  T* dband = static_cast<T*>(gr.dproj) + f.di + p.c0;
  // this lane's rank of four neighbouring columns, out of the 4 R elements that the scan's layout interleaves
  auto pick = [&](const Four<T> (&v)[R], float (&o)[4]) {
    if (R == 1 || !p.bc) {
      v[0].get(o);
    } else if constexpr (sizeof(T) == 2) {
      const uint32_t sel = (r & 1) ? 0x3244u : 0x1044u;   // the high or the low half of a word, as a float
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(v);
        const uint32_t x = R == 2 ? w[e] : ((r & 2) ? w[(2 * e + 1) % (2 * R)] : w[(2 * e) % (2 * R)]);
        o[e] = __uint_as_float(__byte_perm(x, 0u, sel));
      }
    } else {
      const float* w = reinterpret_cast<const float*>(v);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        o[e] = w[e * R];
#pragma unroll
        for (int rr = 1; rr < R; ++rr) o[e] = rr == r ? w[e * R + rr] : o[e];
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
  // go[u] = d pre of two consecutive steps, from the five rows of their taps' windows and their gradients; OWN: the steps
  // feed the parameter gradients.  Two at a time: a step is one chain (exponential, reciprocal, row sums by shuffles,
  // reciprocal root), twelve warps do not cover it, and four row sums share their shuffles.
  auto two_steps = [&](auto own, const float (&r0)[4], const float (&r1)[4], const float (&r2)[4], const float (&r3)[4],
                       const float (&r4)[4], const Four<T> (&g0)[R], const Four<T> (&g1)[R], float (&go)[2][4]) {
    constexpr bool OWN = decltype(own)::value;
    float v[2][4], ds[2][4], gy[2][4];
    pick(g0, gy[0]);
    pick(g1, gy[1]);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float pre[4], sg[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) pre[e] = bs[e];
      fma4(wt[0], u ? r1 : r0, pre);
      fma4(wt[1], u ? r2 : r1, pre);
      fma4(wt[2], u ? r3 : r2, pre);
      fma4(wt[3], u ? r4 : r3, pre);
      sigmoid4(pre, sg);
      mul4(pre, sg, v[u]);   // SiLU; its derivative is sg + v (1 - sg)
      const float nv[4] = {-v[u][0], -v[u][1], -v[u][2], -v[u][3]};
      add4(sg, v[u], ds[u]);
      fma4(nv, sg, ds[u]);
    }
    if (p.bc) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        round4(static_cast<const T*>(nullptr), v[u]);
        add4(v[u], bias, v[u]);
      }
      if (f.has_norm) {
        float sums[4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          float dxh[4];
          mul4(gy[u], gain, dxh);
          sums[2 * u] = dot4(v[u], v[u]);
          sums[2 * u + 1] = dot4(dxh, v[u]);
        }
        row_sums<N, 4>(sums);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const float rstd = rsqrtf(sums[2 * u] * (1.0f / N) + f.eps), md = -sums[2 * u + 1] * rstd * (1.0f / N);
          const float rs4[4] = {rstd, rstd, rstd, rstd}, md4[4] = {md, md, md, md};
          float dxh[4];
          mul4(gy[u], gain, dxh);
          mul4(v[u], rs4, v[u]);   // normalised
          if (OWN) fma4(gy[u], v[u], pgain);
          fma4(v[u], md4, dxh);
          mul4(dxh, rs4, gy[u]);
        }
      }
      if (OWN) {
        add4(pbias, gy[0], pbias);
        add4(pbias, gy[1], pbias);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      mul4(gy[u], ds[u], go[u]);   // gradients past T are zero, so go is too
      if (OWN) {
        add4(pb, go[u], pb);
        fma4(go[u], u ? r1 : r0, pw[0]);
        fma4(go[u], u ? r2 : r1, pw[1]);
        fma4(go[u], u ? r3 : r2, pw[2]);
        fma4(go[u], u ? r4 : r3, pw[3]);
      }
    }
  };
  // dx[t] = sum_delay w[K-1-delay] g[t + delay], from gj = g[t + j]
  const ptrdiff_t xs = p.rev ? -(ptrdiff_t)f.width : (ptrdiff_t)f.width;
  T* const d0 = dband + ((ptrdiff_t)b * f.T + (p.rev ? f.T - 1 - p.t0 : p.t0)) * f.width;
  auto emit = [&](int s, const float (&g0)[4], const float (&g1)[4], const float (&g2)[4], const float (&g3)[4]) {
    if (!p.live || s < 0 || p.t0 + s >= f.T) return;
    float o[4];
    mul4(wt[3], g0, o);
    fma4(wt[2], g1, o);
    fma4(wt[1], g2, o);
    fma4(wt[0], g3, o);
    Four<T> q;
    q.set(o);
    q.store(d0 + s * xs);
  };
  const int last_tl = kBwdWarps / (p.bc ? P::WR : 1) - 1, stride = p.bc ? P::WR : 1;
  float gw[4][4];   // g of the last four steps; step s in slot s & 3 (every loop over steps is unrolled by four)
  auto walk = [&](auto inside) {
    constexpr bool IN = decltype(inside)::value;
    const T* px = static_cast<const T*>(f.proj) + ((ptrdiff_t)b * f.T + (p.rev ? f.T - 1 - p.t0 : p.t0)) * f.width + f.di + p.c0;
    const ptrdiff_t gs = p.rev ? -(ptrdiff_t)gwid : (ptrdiff_t)gwid;
    const T* pg = gin + ((ptrdiff_t)b * f.T + (p.rev ? f.T - 1 - p.t0 : p.t0)) * (ptrdiff_t)gwid;
    auto row = [&](Four<T>& v, int s) {
      if (IN) v.load(px + s * xs); else load_band<T>(v, f, b, p.t0 + s, p.c0, p.rev);
    };
    auto grad = [&](Four<T> (&v)[R], int s) {   // the gradient of a step as the scan left it
#pragma unroll
      for (int i = 0; i < R; ++i) {
        if (!IN) v[i].clear();
        if ((i == 0 || p.bc) && (IN || p.t0 + s < f.T)) v[i].load(pg + s * gs + 4 * i);
      }
    };
    Four<T> nxt[2], ng[2][R];   // the rows of the next two steps
    float win[4][4];            // x of the last four steps, in rotation like gw
    {
      Four<T> v;
#pragma unroll
      for (int k = 1; k < KT; ++k) {
        row(v, k - KT);
        v.get(win[k]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        row(nxt[i], i);
        grad(ng[i], i);
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) gw[k][e] = 0.0f;
    auto four = [&](auto own, int s0) {
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        const int s = s0 + i;
        float x3[4], x4[4], go[2][4];
        nxt[0].get(x3);
        nxt[1].get(x4);
        Four<T> g0[R], g1[R];
#pragma unroll
        for (int j = 0; j < R; ++j) { g0[j] = ng[0][j]; g1[j] = ng[1][j]; }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          row(nxt[u], s + 2 + u);
          grad(ng[u], s + 2 + u);
          if (IN && s + u + kAhead < p.run) {
            prefetch_l2(px + (s + u + kAhead) * xs);
            prefetch_l2(pg + (s + u + kAhead) * gs);
          }
        }
        two_steps(own, win[(i + 1) & 3], win[(i + 2) & 3], win[(i + 3) & 3], x3, x4, g0, g1, go);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int c = i + u;
          if (s0 == 0 && c < KT - 1)   // for the warp before this one in time
            *reinterpret_cast<float4*>(&ahead[warp][c][4 * lane]) = make_float4(go[u][0], go[u][1], go[u][2], go[u][3]);
          if (s + u - 3 < p.run) emit(s + u - 3, gw[(c + 1) & 3], gw[(c + 2) & 3], gw[(c + 3) & 3], go[u]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            gw[c][e] = go[u][e];
            win[c][e] = u ? x4[e] : x3[e];
          }
        }
      }
    };
#pragma unroll 1
    for (int s = 0; s < p.run; s += 4) four(std::true_type{}, s);
    // the last three rows need three more g: the last warp in time works them out, the others take them from the warp
    // behind them
    if (p.tl == last_tl) four(std::false_type{}, p.run);
  };
  const int end = p.t0 + p.run + (p.tl == last_tl ? 6 : 2);   // rows are requested two steps ahead
  if (p.t0 >= KT - 1 && end <= f.T) walk(std::true_type{});
  else walk(std::false_type{});
  __syncthreads();
  if (p.tl != last_tl) {
    float h[KT - 1][4];
#pragma unroll
    for (int k = 0; k < KT - 1; ++k) {
      const float4 q = *reinterpret_cast<const float4*>(&ahead[warp + stride][k][4 * lane]);
      h[k][0] = q.x; h[k][1] = q.y; h[k][2] = q.z; h[k][3] = q.w;
    }
    emit(p.run - 3, gw[1], gw[2], gw[3], h[0]);
    emit(p.run - 2, gw[2], gw[3], h[0], h[1]);
    emit(p.run - 1, gw[3], h[0], h[1], h[2]);
  }
  // the block's partial sums: its warps in time order, one quantity after the other (a fixed order)
  const int C = f.di + 2 * f.bc;
  auto reduce = [&](const float (&v)[4], float* dst) {
    __syncthreads();
    *reinterpret_cast<float4*>(&red[warp][4 * lane]) = make_float4(v[0], v[1], v[2], v[3]);
    __syncthreads();
    if (p.tl == 0 && p.live) {
      float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      for (int w = warp; w < kBwdWarps; w += stride) {
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

// out[c] = sum over blocks (for the B / C bias over the ranks too) of the partial sums, in a fixed order: block (32, 8)
// owns 32 columns, thread row y every 8th term, the 8 row sums are added in order.  The blocks of the gradients follow one
// another (a grid with a row per gradient is mostly blocks with nothing to do).  The gain's columns are summed row by row of
// B and C, and over the rows by whichever of their blocks finishes last (in a fixed order; k_front_bwd clears the count): as
// a launch of its own that took 2 us and 3.5 us of the host's time.
constexpr int kSumRows = 8;
struct SumRange {
  float* out;
  size_t off;          // first column within a block's floats
  int ncols, inner, istride, first_block;
};
struct SumPlan {
  SumRange r[6];
  int n, blocks;
  float *gain_rows, *gain;   // gain NULL: none
  unsigned* gain_count;
  int gain_blocks, nrows;
};
__global__ void __launch_bounds__(32 * kSumRows) k_front_sums(SumPlan plan, const float* __restrict__ part, size_t pitch, int nblk,
                                                             int N) {
  after_predecessor();
  __shared__ float red[kSumRows][33];
  int i = 0;
  while (i + 1 < plan.n && (int)blockIdx.x >= plan.r[i + 1].first_block) ++i;
  const SumRange q = plan.r[i];
  const int c = ((int)blockIdx.x - q.first_block) * 32 + threadIdx.x;
  float s = 0.0f;
  if (c < q.ncols) {
    // a bias column (head, n) is the sum over the head's ranks, N apart
    const float* src = part + q.off + (q.inner > 1 ? (size_t)(c / N) * q.inner * N + c % N : c);
    const int n = nblk * q.inner;
#pragma unroll 8
    for (int t = threadIdx.y; t < n; t += kSumRows) {
      const int blk = q.inner == 1 ? t : t / q.inner;
      s += src[(size_t)blk * pitch + (size_t)(t - blk * q.inner) * q.istride];
    }
  }
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < q.ncols) {
    float tot = 0.0f;
#pragma unroll
    for (int j = 0; j < kSumRows; ++j) tot += red[j][threadIdx.x];
    q.out[c] = tot;
  }
  if (!plan.gain || q.out != plan.gain_rows) return;
  __shared__ unsigned last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0 && threadIdx.y == 0) last = atomicAdd(plan.gain_count, 1u);
  __syncthreads();
  if (last != (unsigned)plan.gain_blocks - 1u) return;
  __threadfence();
  for (int c0 = 0; c0 < N; c0 += 32) {
    float v = 0.0f;
#pragma unroll 8
    for (int t = threadIdx.y; t < plan.nrows; t += kSumRows) v += __ldcg(plan.gain_rows + (size_t)t * N + c0 + threadIdx.x);
    red[threadIdx.y][threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.y == 0) {
      float tot = 0.0f;
#pragma unroll
      for (int j = 0; j < kSumRows; ++j) tot += red[j][threadIdx.x];
      plan.gain[c0 + threadIdx.x] = tot;
    }
    __syncthreads();
  }
}
SumPlan sum_plan(const Front& f, const FrontGrads& g, int nblk) {
  const PartLayout pl = part_layout(f);
  const int C = f.di + 2 * f.bc;
  SumPlan p{};
  auto add = [&](float* out, size_t off, int ncols, int inner, int istride) {
    if (!out) return;
    p.r[p.n++] = SumRange{out, off, ncols, inner, istride, p.blocks};
    p.blocks += (ncols + 31) / 32;
  };
  add(g.dconv_w, pl.conv + (size_t)(KT - f.K) * C, f.K * C, 1, 0);
  add(g.dconv_b, pl.conv + (size_t)KT * C, C, 1, 0);
  add(g.db_bias, pl.bias, f.H * f.N, f.R, f.N);
  add(g.dc_bias, pl.bias + f.bc, f.H * f.N, f.R, f.N);
  if (g.dgain) {
    p.gain = g.dgain;
    p.gain_rows = g.part + (size_t)nblk * pl.total;
    p.gain_count = gain_count(f, g, nblk);
    p.gain_blocks = (2 * f.bc + 31) / 32;
    p.nrows = 2 * f.bc / f.N;
    add(p.gain_rows, pl.gain, 2 * f.bc, 1, 0);
  }
  add(g.ddt_bias, pl.act, f.H, 1, 0);
  return p;
}

// Steps per warp: a block of 128 steps amortises the window's start and the warps' parameters; a grid of fewer than four
// such blocks per SM is cut finer so that every SM has work.
bool front_long(const Front& f, int tiles) { return (long long)tiles * f.B * ((f.T + 127) / 128) >= 4 * sm_count(); }
int bwd_steps(const Front& f, int tiles) { return kBwdWarps * (front_long(f, tiles) ? 32 : 8); }
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
  const int run = front_long(f, nx + 2 * nb) ? 16 : 4;
  const dim3 grid(nx + 2 * nb + 1, (f.T + kWarps * run - 1) / (kWarps * run), f.B);
  if (run == 16) launch(k_front_fwd<T, N, R, 16>, grid, kWarps * 32, 0, st, f, o, nx, nb);
  else launch(k_front_fwd<T, N, R, 4>, grid, kWarps * 32, 0, st, f, o, nx, nb);
  return cudaGetLastError();
}
template <class T, int N, int R>
cudaError_t backward_t(cudaStream_t st, const Front& f, const FrontGrads& g) {
  int nx, nb;
  front_tiles<N, R>(f, &nx, &nb);
  const int steps = bwd_steps(f, nx + 2 * nb);
  const dim3 grid(nx + 2 * nb + 1, (f.T + steps - 1) / steps, f.B);
  if (steps == kBwdWarps * 32) launch(k_front_bwd<T, N, R, 32>, grid, kBwdWarps * 32, 0, st, f, g, nx, nb);
  else launch(k_front_bwd<T, N, R, 8>, grid, kBwdWarps * 32, 0, st, f, g, nx, nb);
  const int nblk = (int)(grid.y * grid.z);
  const SumPlan plan = sum_plan(f, g, nblk);
  if (plan.blocks)
    launch(k_front_sums, plan.blocks, dim3(32, kSumRows), 0, st, plan, g.part, part_layout(f).total, nblk, N);
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
  const int steps = bwd_steps(f, nx + 2 * nb);
  return part_layout(f).total * f.B * ((f.T + steps - 1) / steps) + 2 * (size_t)f.bc + 4;
}

cudaError_t front_backward(cudaStream_t st, int dtype, const Front& f, const FrontGrads& g, uint64_t* launches) {
  if (launches) *launches += 2;
  return dispatch(dtype, f, [&](auto t, auto n, auto r) { return backward_t<decltype(t), n.value, r.value>(st, f, g); });
}

}  // namespace m3
