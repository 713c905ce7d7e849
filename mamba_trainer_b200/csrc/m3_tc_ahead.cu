// States at segment boundaries, ahead of the tensor-core stripe kernels: what lets the segments of ONE stripe run side by
// side.  The stripe kernels keep the state in TMEM and walk a stripe tile by tile, so a launch of fewer stripes than SMs
// leaves SMs idle however long the sequence is (16 stripes of 14 tiles: 94 us on 16 of 148 SMs).  Two short launches
// come first here:
//   k_tile_state  per half tile (64 rows), all of all stripes at once: its own contribution to the state,
//                 X~^T diag(sw) B^ (backward, to its gradient: (exp(acum) dY~)^T C^), its decay and its angle
//   k_tile_pass   sequential over half tiles, parallel over state elements: the state (and the angle) at every segment
//                 boundary, in the place where the stripe kernels expect what the segment before handed over
// after which the segments are independent.  The contraction is mma.sync on operands rounded to bf16, like the stripe
// kernels' own; accumulation and states are float32.  The price is one more reading of B and x (C and dy) and a state per
// half tile; tc_ahead_plan weighs it.  (Whole tiles, two halves one after the other in a block, took 31 us for 224 tiles of
// rank 1 where half tiles take 25: there are few blocks, so what counts is the chain inside one.)
#include "m3_rows.cuh"
#include "m3_tc.h"

namespace m3 {
namespace rows {
namespace {

constexpr int kN = 128, kNH = 64, kPN = kP * kN;

template <int R>
struct TileSmem {
  float b[kRows * kN];
  union {   // the angles are spent when x (from registers) takes their place: four blocks share an SM
    float x[kRows * kP];
    float phi[(kRows / R) * kNH];
  };
  float q[256], base[kNH];
  Scal<R> s;
};

// This thread's words of a half tile's rows of x or dy, and what load_rows makes of them.
template <int R>
struct RawRows {
  static constexpr int PER = kP * R / 4, NI = (kRows / R) * PER / 256;
  uint2 w[NI];
  __device__ __forceinline__ void load(const __nv_bfloat16* src, const Dims& d, const Chunk& c) {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int it = threadIdx.x + i * 256, l = it / PER, e = 4 * (it - l * PER), t = c.t0 + l;
      w[i] = make_uint2(0u, 0u);
      if (t < d.T) w[i] = __ldg(reinterpret_cast<const uint2*>(src + tok_index(d, c.b, t, c.h) * kP * R + e));
    }
  }
  __device__ __forceinline__ void store(float* dst) const {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const int it = threadIdx.x + i * 256, l = it / PER, e = 4 * (it - l * PER);
      const float f[4] = {__uint_as_float(w[i].x << 16), __uint_as_float(w[i].x & 0xffff0000u), __uint_as_float(w[i].y << 16),
                          __uint_as_float(w[i].y & 0xffff0000u)};
      if (R == 1) {
        *reinterpret_cast<float4*>(dst + at<kP>(l, e)) = make_float4(f[0], f[1], f[2], f[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) dst[at<kP>(l * R + (e + j) % R, (e + j) / R)] = f[j];
      }
    }
  }
};

// Forward: rows rotated by the angle since the half tile's start.  Backward: by the absolute angle; the forward pass left
// the one entering every whole tile, so the second half adds up the first one's.
template <int R, bool ROT, bool BWD>
__global__ void __launch_bounds__(256, 4) k_tile_state(Dims d, m3_scan_desc in, const __nv_bfloat16* __restrict__ dy,
                                                       const float* __restrict__ ckpt_angle, float* __restrict__ hs,
                                                       float* __restrict__ asum, float* __restrict__ cd_out) {
  using T = __nv_bfloat16;
  extern __shared__ __align__(16) unsigned char smem[];
  TileSmem<R>& sm = *reinterpret_cast<TileSmem<R>*>(smem);
  constexpr int LT = kRows / R;
  const Chunk c = this_chunk(d);
  const size_t slot = (size_t)c.bh * d.C + c.k;
  const int tid = threadIdx.x;
  RawRows<R> raw;
  raw.load(BWD ? dy : static_cast<const T*>(in.x), d, c);
  if (ROT && BWD) {
    const int q = tid >> 6, m = tid & 63;
    float s = q == 0 ? ckpt_angle[((size_t)c.bh * ((d.C + 1) / 2) + c.k / 2) * kNH + m] : 0.0f;
    if (c.k & 1) {
#pragma unroll
      for (int i = 0; i < LT / 4; ++i) {
        const int t = c.t0 - LT + q * (LT / 4) + i;   // the half before this one is whole
        s += ldf(static_cast<const T*>(in.dt), tok_index(d, c.b, t, c.h)) *
             ldf(static_cast<const T*>(in.theta), theta_index(d, c.b, t, c.h) + m);
      }
    }
    sm.q[tid] = s;
  }
  chunk_scalars<T, R>(sm.s, d, c, in);   // (its barriers also complete q)
  if (tid == 0) cd_out[slot] = sm.s.ac[LT - 1];
  const float* scale = BWD ? sm.s.eac : sm.s.sw;
  const T* rows_in = static_cast<const T*>(BWD ? in.c : in.b);
  if constexpr (ROT) {
    if (tid < kNH) sm.base[tid] = BWD ? wrap_angle(sm.q[tid] + sm.q[tid + 64] + sm.q[tid + 128] + sm.q[tid + 192]) : 0.0f;
    __syncthreads();
    chunk_angles<T, kN, R, 256>(sm.phi, sm.q, sm.s, d, c, static_cast<const T*>(in.theta), sm.base,
                                [&](int m, float sum) { if (!BWD) asum[slot * kNH + m] = sum; });
    __syncthreads();
    float* const to[1] = {sm.b};
    const T* const from[1] = {rows_in};
    load_rotated<T, kN, R, 256, 1, true>(to, from, sm.phi, scale, d, c);
    __syncthreads();
  } else {
    load_scaled<T, kN, R, 256, true>(sm.b, rows_in, scale, d, c);
  }
  raw.store(sm.x);
  __syncthreads();
  const int warp = tid >> 5, m0 = 32 * (warp & 1), n0 = 32 * (warp >> 1);
  float acc[2][4][4];
  zero(acc);
  warp_mma<2, 4, false, false, true, true, kP, kN>(acc, sm.x, m0, sm.b, n0, 0, kRows);
  store_acc<kN>(acc, m0, n0, hs + slot * kPN);
}

// A thread owns planes (m, m + 64) of rows p, p + 32 and walks the half tiles in time (backward: against it); U of them
// are requested before the first is used; tps is in half tiles here.  seg_state / seg_angle of segment s: what leaves it towards the next one walked.
template <bool ROT, bool BWD>
__global__ void __launch_bounds__(256) k_tile_pass(Dims d, m3_scan_desc in, const float* __restrict__ dh,
                                                   const float* __restrict__ hs, const float* __restrict__ asum,
                                                   const float* __restrict__ cd, int tps, int nseg,
                                                   float* __restrict__ seg_state, float* __restrict__ seg_angle) {
  using T = __nv_bfloat16;
  constexpr int U = 8;
  const int bh = blockIdx.y, b = bh / d.H, h = bh - b * d.H;
  const int id = blockIdx.x * 256 + threadIdx.x, m = id % kNH, p = id / kNH;
  const int o[4] = {at<kN>(p, m), at<kN>(p, m) + kNH, at<kN>(p + 32, m), at<kN>(p + 32, m) + kNH};
  const int plain[4] = {p * kN + m, p * kN + m + kNH, (p + 32) * kN + m, (p + 32) * kN + m + kNH};
  float carry[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  float ang = 0.0f;
  if (BWD) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (dh) carry[i] = dh[(size_t)bh * kPN + plain[i]];
  } else {
    if (in.h0) {   // the seed of scan.rs:524-535
      const size_t i0 = tok_index(d, b, 0, h);
      const float first = (1.0f - lambda_at(static_cast<const T*>(in.lambda), d.disc, i0)) * ldf(static_cast<const T*>(in.dt), i0);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        carry[i] = in.h0[(size_t)bh * kPN + plain[i]] + first * in.last_u0[(size_t)bh * kPN + plain[i]];
    }
    if (ROT && in.angle0) ang = in.angle0[(size_t)bh * kNH + m];
  }
  // the last segment walked hands nothing over: stop at its first tile
  const int tiles = d.C, count = BWD ? tiles - tps : (nseg - 1) * tps;
  for (int i0 = 0; i0 < count; i0 += U) {
    float s[U][4], e[U], da[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = min(i0 + u, count - 1), k = BWD ? tiles - 1 - i : i;
      const size_t slot = (size_t)bh * tiles + k;
#pragma unroll
      for (int j = 0; j < 4; ++j) s[u][j] = __ldg(hs + slot * kPN + o[j]);
      e[u] = cd[slot];
      da[u] = ROT && !BWD ? asum[slot * kNH + m] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i0 + u >= count) break;
      const int k = BWD ? tiles - 1 - (i0 + u) : i0 + u;
      float sn = 0.0f, cs = 1.0f;
      if (ROT && !BWD) {
        sincosf(ang, &sn, &cs);
        ang = wrap_angle(ang + da[u]);
      }
      const float ec = exp_decay(e[u]);
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        const float s1 = s[u][j], s2 = s[u][j + 1];
        carry[j] = fmaf(ec, carry[j], ROT && !BWD ? s1 * cs + s2 * sn : s1);
        carry[j + 1] = fmaf(ec, carry[j + 1], ROT && !BWD ? s2 * cs - s1 * sn : s2);
      }
      if (BWD ? k % tps == 0 : (k + 1) % tps == 0) {
        const size_t seg = (size_t)bh * nseg + k / tps;
#pragma unroll
        for (int j = 0; j < 4; ++j) seg_state[seg * kPN + plain[j]] = carry[j];
        if (ROT && !BWD && p == 0) seg_angle[seg * kNH + m] = ang;
      }
    }
  }
}

template <int R, bool ROT, bool BWD>
cudaError_t ahead_t(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const void* dy, const float* dh, const float* ckpt_angle,
                    const TcAhead& a) {
  auto kern = k_tile_state<R, ROT, BWD>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TileSmem<R>));
  if (e != cudaSuccess) return e;
  kern<<<dim3(d.C, d.B * d.H), 256, sizeof(TileSmem<R>), st>>>(d, in, static_cast<const __nv_bfloat16*>(dy), ckpt_angle, a.hs,
                                                              a.asum, a.cd);
  k_tile_pass<ROT, BWD><<<dim3(32 * kNH / 256, d.B * d.H), 256, 0, st>>>(d, in, dh, a.hs, a.asum, a.cd, 2 * a.tps, a.nseg, a.seg_state,
                                                                        a.seg_angle);
  return cudaGetLastError();
}

}  // namespace
}  // namespace rows

// Whether to cut `BH` stripes of `tiles` tiles into segments that run side by side, and into how many.  Microseconds,
// measured on a B200: a tile takes about 5.5 forward and 15 backward inside a stripe, an item costs about one more to
// start and finish; the tile states take 1.3 per tile and SM after 5 for the launch, the pass 5 + 0.15 per tile.  Beyond a
// third of the SMs too little is idle to pay for it.
bool tc_ahead_plan(int BH, int tiles, bool backward, int* nseg, int* tps) {
  constexpr int kSms = 148;
  if (BH > kSms / 3 || tiles < 3 || (size_t)BH * tiles > (1u << 14)) return false;   // at most 1 GB of states
  const float c = backward ? 15.0f : 5.5f;
  const float pre = 10.0f + 1.3f * (float)((BH * (long long)tiles + kSms - 1) / kSms) + 0.15f * tiles;
  float best = 0.9f * tiles * c;
  bool found = false;
  for (int n = 2; n <= tiles && n <= 4 * kSms; ++n) {
    const int per = (tiles + n - 1) / n, segs = (tiles + per - 1) / per;
    const int rounds = (BH * segs + kSms - 1) / kSms;
    const float t = pre + rounds * (per + 1) * c;
    if (t < best) {
      best = t;
      found = true;
      *nseg = segs;
      *tps = per;
    }
  }
  return found;
}

size_t tc_ahead_bytes(int BH, int tiles, int nseg, TcAhead* a, char* base) {
  size_t off = 0;
  auto take = [&](size_t n) {
    float* p = base ? reinterpret_cast<float*>(base + off) : nullptr;
    off += (n * sizeof(float) + 255) / 256 * 256;
    return p;
  };
  TcAhead t{};
  t.hs = take((size_t)BH * 2 * tiles * rows::kPN);
  t.asum = take((size_t)BH * 2 * tiles * rows::kNH);
  t.cd = take((size_t)BH * 2 * tiles);
  t.seg_state = take((size_t)BH * nseg * rows::kPN);
  t.seg_angle = take((size_t)BH * nseg * rows::kNH);
  if (a) {
    t.nseg = a->nseg;
    t.tps = a->tps;
    *a = t;
  }
  return off;
}

cudaError_t tc_ahead(cudaStream_t st, Dims d, const m3_scan_desc& in, const void* dy, const float* dh, const float* ckpt_angle,
                     const TcAhead& a) {
  d.L = tc_tile_steps(d.R) / 2;
  d.C = (d.T + d.L - 1) / d.L;   // (an odd number when the last tile has one half only)
  auto go = [&](auto r, auto rot) {
    return dy ? rows::ahead_t<r.value, rot.value, true>(st, d, in, dy, dh, ckpt_angle, a)
              : rows::ahead_t<r.value, rot.value, false>(st, d, in, nullptr, nullptr, nullptr, a);
  };
  auto with_rot = [&](auto r) { return d.rot ? go(r, std::true_type{}) : go(r, std::false_type{}); };
  switch (d.R) {
    case 1: return with_rot(std::integral_constant<int, 1>{});
    case 2: return with_rot(std::integral_constant<int, 2>{});
    default: return with_rot(std::integral_constant<int, 4>{});
  }
}

}  // namespace m3
