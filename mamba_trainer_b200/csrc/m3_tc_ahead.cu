// States at segment boundaries, ahead of the tensor-core stripe kernels: what lets the segments of ONE stripe run side by
// side.  The stripe kernels keep the state in TMEM and walk a stripe tile by tile, so a launch of fewer stripes than SMs
// leaves SMs idle however long the sequence is (16 stripes of 14 tiles: 94 us on 16 of 148 SMs).  Two short launches
// come first here (three in a training step with rotation: k_group_angle):
//   k_group_state  per group of tiles, all groups of all stripes at once: what the group adds to the state,
//                  (sw X~)^T B^ decayed to its end (backward, to the state's gradient: (exp(acum) dY~)^T C^ from its
//                  start), its decay and its angle
//   k_group_pass   sequential over groups, parallel over state elements: the state (and the angle) at every segment
//                  boundary, in the place where the stripe kernels expect what the segment before handed over
// after which the segments are independent.  The last segment's groups (backward: the first one's) are needed by nobody and
// not worked out.  Operands are rounded to bf16 where the stripe kernels' are - x or dY with its weight, the rotated B or C;
// accumulation and states are float32.  (B is rotated by the angle since the group's start, unless a backward pass will
// follow: k_group_angle.)
//
// k_group_state walks its group in half tiles (64 rows) with the rows of the next one in registers, the sum in registers
// too, and leaves one state per group.  Its products are warp-level (mma.sync on bf16, operands by ldmatrix): a half tile
// has one product of 1 MFLOP between two conversions, which is what it spends its time on.  An earlier form, a block per
// half tile in TF32 with nothing requested ahead, took as long per tile as the whole forward kernel and a state per half
// tile through memory: prefill of 1777 tokens, 16 heads: 25 + 12 us -> 14 + 9 us.
#include <cuda_fp16.h>

#include "m3_rows.cuh"
#include "m3_tc.h"
#include "m3_tc_common.cuh"

namespace m3 {
namespace {

using m3tc::bf16_hi;
using m3tc::bf16_lo;
using m3tc::pack_bf16;
using rows::kP;
using rows::kRows;

constexpr int kN = 128, kNH = 64, kPN = kP * kN, kThreads = 256;

// Operands [row][COLS] bf16, 16-byte chunks XOR-swizzled by row & 7: ldmatrix reads eight bank groups.
template <int COLS>
__device__ __forceinline__ uint32_t off(int row, int chunk) {
  return (uint32_t)(row * COLS * 2) + (uint32_t)((chunk ^ (row & 7)) << 4);
}
__device__ __forceinline__ void ldm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// A work item of a conversion: a step and 32 bytes of its row (16 for one rank) - 8 columns of one or two ranks, 4 of four.
template <int R>
struct Item {
  static constexpr int LT = kRows / R, CW = R == 4 ? 4 : 8, W = R == 1 ? 4 : 8;
  static constexpr int GROUPS = 64 / CW, PER = LT * GROUPS / kThreads;
  int l, col;
  __device__ __forceinline__ explicit Item(int i) {
    const int it = threadIdx.x + i * kThreads;
    l = it / GROUPS;
    col = (it % GROUPS) * CW;
  }
};
template <int R>
__device__ __forceinline__ float item_el(const uint32_t (&w)[Item<R>::W], int j, int r) {   // column j of rank r
  if (R == 1) return (j & 1) ? bf16_hi(w[j >> 1]) : bf16_lo(w[j >> 1]);
  if (R == 2) return r ? bf16_hi(w[j]) : bf16_lo(w[j]);
  const uint32_t v = w[(2 * j + (r >> 1)) % Item<R>::W];
  return (r & 1) ? bf16_hi(v) : bf16_lo(v);
}
template <int R>
__device__ __forceinline__ void get(uint32_t (&w)[Item<R>::W], const __nv_bfloat16* p, bool live) {
#pragma unroll
  for (int i = 0; i < Item<R>::W / 4; ++i) {
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (live) v = __ldg(reinterpret_cast<const uint4*>(p) + i);
    w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
  }
}
template <int R, int COLS>
__device__ __forceinline__ void put(uint8_t* buf, int row, int col, const float (&v)[Item<R>::CW]) {
  uint8_t* p = buf + off<COLS>(row, col >> 3) + (col & 7) * 2;
  if constexpr (Item<R>::CW == 8)
    *reinterpret_cast<uint4*>(p) = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
  else
    *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]));
}

// What the kernel keeps per half tile: dt, and exp(cd - ac) w (backward: exp(ac)) of its steps, its decay.
template <int R>
struct HalfScal {
  static constexpr int LT = kRows / R;
  float dt[LT], scale[LT], cd, pad[3];
};
// dt and lambda (raw: a conversion would wait for the load) for the warp that works the scalars out.
template <int R>
struct HalfLoads {
  static constexpr int LT = kRows / R, EPL = LT >= 32 ? LT / 32 : 1;
  uint16_t dtw[EPL + 1], lamw[EPL + 1];
  __device__ __forceinline__ void load(const m3_scan_desc& in, const Dims& d, int b, int h, int t0) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i <= EPL; ++i) {
      const int t = t0 + lane * EPL + i;
      dtw[i] = 0;
      lamw[i] = d.disc == 1 ? 0x3f00 : 0x3f80;   // one half, one
      if (t < d.T) {
        const size_t o = tok_index(d, b, t, h);
        dtw[i] = __ldg(static_cast<const unsigned short*>(in.dt) + o);
        if (d.disc == 2) lamw[i] = __ldg(static_cast<const unsigned short*>(in.lambda) + o);
      }
    }
  }
  template <bool BWD>
  __device__ __forceinline__ void work_out(HalfScal<R>& s, float A, int T, int t0) const {   // one whole warp
    const int lane = threadIdx.x & 31;
    float dt[EPL + 1], lam[EPL + 1], loc[EPL], wv[EPL], run = 0.0f;
#pragma unroll
    for (int i = 0; i <= EPL; ++i) {
      dt[i] = __uint_as_float((uint32_t)dtw[i] << 16);
      lam[i] = __uint_as_float((uint32_t)lamw[i] << 16);
    }
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
      const int l = lane * EPL + i, t = t0 + l;
      wv[i] = 0.0f;
      if (l < LT && t < T) {
        wv[i] = lam[i] * dt[i] + (t + 1 < T ? (1.0f - lam[i + 1]) * dt[i + 1] : 0.0f);
        run += dt[i] * A;
      }
      loc[i] = run;
    }
    float tot = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float n = __shfl_up_sync(0xffffffffu, tot, o);
      if (lane >= o) tot += n;
    }
    const float base = tot - run, cd = __shfl_sync(0xffffffffu, tot, 31);
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
      const int l = lane * EPL + i;
      if (l < LT) {
        const float ac = base + loc[i];
        s.dt[l] = dt[i];
        s.scale[l] = BWD ? exp_decay(ac) : exp_decay(cd - ac) * wv[i];
      }
    }
    if (lane == 0) s.cd = cd;
  }
};

template <int R>
struct GroupSmem {
  static constexpr int LT = kRows / R;
  uint8_t b[kRows * kN * 2], x[kRows * kP * 2];
  float phi[LT * kNH];       // wrapped angle of (step, plane)
  float2 q[8 * 32], carry[2][32];
  HalfScal<R> s[3];
};

// Cumulative angles: warp o takes the o-th eighth of a half tile's steps, lane m2 planes 2 m2 and 2 m2 + 1.
template <int R>
struct HalfAngles {
  static constexpr int LT = kRows / R, LO = LT / 8;
  uint32_t th[LO];
  __device__ __forceinline__ void load(const __nv_bfloat16* theta, const Dims& d, int b, int h, int t0) {
    const int o = threadIdx.x >> 5, m2 = threadIdx.x & 31;
#pragma unroll
    for (int i = 0; i < LO; ++i) {
      const int t = t0 + o * LO + i;
      th[i] = t < d.T ? __ldg(reinterpret_cast<const uint32_t*>(theta + theta_index(d, b, t, h)) + m2) : 0u;
    }
  }
  __device__ __forceinline__ void partial(float2* q, const float* dt) const {
    const int o = threadIdx.x >> 5, m2 = threadIdx.x & 31;
    float2 s = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < LO; ++i) {
      s.x = fmaf(dt[o * LO + i], bf16_lo(th[i]), s.x);
      s.y = fmaf(dt[o * LO + i], bf16_hi(th[i]), s.y);
    }
    q[o * 32 + m2] = s;
  }
  __device__ __forceinline__ void finish(float* phi, const float2* q, const float* dt, const float2* in, float2* out) const {
    const int o = threadIdx.x >> 5, m2 = threadIdx.x & 31;
    float2 run = in[m2];
#pragma unroll
    for (int j = 0; j < 7; ++j) {
      const float2 v = q[j * 32 + m2];
      run.x += j < o ? v.x : 0.0f;
      run.y += j < o ? v.y : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < LO; ++i) {
      const int l = o * LO + i;
      run.x = fmaf(dt[l], bf16_lo(th[i]), run.x);
      run.y = fmaf(dt[l], bf16_hi(th[i]), run.y);
      const float2 w = make_float2(wrap_angle(run.x), wrap_angle(run.y));
      *reinterpret_cast<float2*>(phi + l * kNH + 2 * m2) = w;
      if (l == LT - 1) out[m2] = w;
    }
  }
};

// FULL_ANGLE forward pass (one whose backward pass will follow): every group's angle ahead of k_group_state, so that B^ is
// rotated by the angle since the start of the sequence and rounded as the stripe kernel's is.  A d theta sums the d phi of all
// later steps, where the two sides of every pair of steps cancel - if both see the same B^ and C^: with B rotated by the angle
// since the group's start, rounded there, and the weights rounded with it, d theta was 1.4 to 1.5 times as far from 64-bit
// results as that of whole stripes (4 stripes of 1670 steps, rank 1; 6 of 1072, rank 2); it is at most 1.07 times now.  One
// launch of 4 us (forward + backward of a 2 x 509-token mixer, 8 heads, rank 2: 168.6 -> 173.1 us); the pass then has nothing
// to rotate.
template <int R>
__global__ void __launch_bounds__(kThreads) k_group_angle(Dims d, m3_scan_desc in, TcAhead a, int tiles) {
  after_predecessor();
  __shared__ float2 part[8][32];
  constexpr int LT = 2 * kRows / R;   // steps of a tile
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bh = blockIdx.y, b = bh / d.H, h = bh - b * d.H;
  const int seg = (int)blockIdx.x / a.gps, k0 = seg * a.tps + ((int)blockIdx.x % a.gps) * a.gt;
  const int k1 = min(min(k0 + a.gt, (seg + 1) * a.tps), tiles), t1 = min(k1 * LT, d.T);
  float2 s = make_float2(0.0f, 0.0f);
#pragma unroll 4
  for (int t = k0 * LT + warp; t < t1; t += 8) {
    const float dt = ldf(static_cast<const __nv_bfloat16*>(in.dt), tok_index(d, b, t, h));
    const uint32_t th = __ldg(reinterpret_cast<const uint32_t*>(static_cast<const __nv_bfloat16*>(in.theta) + theta_index(d, b, t, h)) + lane);
    s.x = fmaf(dt, bf16_lo(th), s.x);
    s.y = fmaf(dt, bf16_hi(th), s.y);
  }
  part[warp][lane] = s;
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int w = 1; w < 8; ++w) { s.x += part[w][lane].x; s.y += part[w][lane].y; }
    *reinterpret_cast<float2*>(a.asum + ((size_t)bh * gridDim.x + blockIdx.x) * kNH + 2 * lane) =
        make_float2(wrap_angle(s.x), wrap_angle(s.y));
  }
}

template <int R, bool ROT, bool BWD, bool FULL_ANGLE>
__global__ void __launch_bounds__(kThreads, 2) k_group_state(Dims d, m3_scan_desc in, const __nv_bfloat16* __restrict__ dy,
                                                             const float* __restrict__ ckpt_angle, TcAhead a, int tiles) {
  after_predecessor();
  extern __shared__ __align__(128) unsigned char smem[];
  GroupSmem<R>& sm = *reinterpret_cast<GroupSmem<R>*>(smem);
  using IT = Item<R>;
  constexpr int LT = kRows / R;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bh = blockIdx.y, b = bh / d.H, h = bh - b * d.H;
  // group blockIdx.x: of segment seg (backward: the first segment has none), tiles [k0, k1)
  const int seg = (int)blockIdx.x / a.gps + (BWD ? 1 : 0), k0 = seg * a.tps + ((int)blockIdx.x % a.gps) * a.gt;
  const int k1 = min(min(k0 + a.gt, (seg + 1) * a.tps), tiles);
  const int j0 = 2 * k0, j1 = min(2 * max(k1, k0), (d.T + LT - 1) / LT);   // half tiles; none for an empty group
  const size_t slot = (size_t)bh * gridDim.x + blockIdx.x;
  const __nv_bfloat16* rows_in = static_cast<const __nv_bfloat16*>(BWD ? in.c : in.b);
  const __nv_bfloat16* px = BWD ? dy : static_cast<const __nv_bfloat16*>(in.x);
  const __nv_bfloat16* theta = static_cast<const __nv_bfloat16*>(in.theta);
  const float A = -expf(in.a_log[h]);
  uint32_t r1[IT::PER][IT::W], r2[IT::PER][IT::W], xr[IT::PER][IT::W];
  auto load_rows = [&](int j) {
#pragma unroll
    for (int i = 0; i < IT::PER; ++i) {
      const Item<R> it(i);
      const int t = j * LT + it.l;
      const bool live = t < d.T;
      const size_t tok = live ? tok_index(d, b, t, h) : 0;
      get<R>(r1[i], rows_in + tok * kN * R + it.col * R, live);
      get<R>(r2[i], rows_in + tok * kN * R + (it.col + kNH) * R, live);
      get<R>(xr[i], px + tok * kP * R + it.col * R, live);
    }
  };
  HalfLoads<R> hl;
  HalfAngles<R> ha;
  if (j0 < j1) load_rows(j0);
  if (warp < 2) {   // scalars of the first two half tiles
    hl.load(in, d, b, h, (j0 + warp) * LT);
    hl.template work_out<BWD>(sm.s[warp], A, d.T, (j0 + warp) * LT);
  }
  if (warp == 0) hl.load(in, d, b, h, (j0 + 2) * LT);
  if (ROT) {
    ha.load(theta, d, b, h, j0 * LT);
    if constexpr (FULL_ANGLE) {   // the angles of the groups before this one, a warp every eighth
      const float* as = a.asum + (size_t)bh * gridDim.x * kNH + 2 * lane;
      float2 v = make_float2(0.0f, 0.0f);
      if (warp == 0 && in.angle0) v = make_float2(in.angle0[(size_t)bh * kNH + 2 * lane], in.angle0[(size_t)bh * kNH + 2 * lane + 1]);
#pragma unroll 4
      for (int g = warp; g < (int)blockIdx.x; g += 8) {
        const float2 w = *reinterpret_cast<const float2*>(as + (size_t)g * kNH);
        v = make_float2(wrap_angle(v.x + w.x), wrap_angle(v.y + w.y));
      }
      sm.q[warp * 32 + lane] = v;
      __syncthreads();
      if (warp == 0) {
#pragma unroll
        for (int w = 1; w < 8; ++w) v = make_float2(v.x + sm.q[w * 32 + lane].x, v.y + sm.q[w * 32 + lane].y);
        sm.carry[0][lane] = make_float2(wrap_angle(v.x), wrap_angle(v.y));
      }
    } else if (tid < 32) {
      sm.carry[0][tid] = BWD && j0 < j1 ? *reinterpret_cast<const float2*>(ckpt_angle + ((size_t)bh * tiles + k0) * kNH + 2 * tid)
                                        : make_float2(0.0f, 0.0f);
    }
  }
  __syncthreads();
  if (ROT) {
    ha.partial(sm.q, sm.s[0].dt);
    __syncthreads();
    ha.finish(sm.phi, sm.q, sm.s[0].dt, sm.carry[0], sm.carry[1]);
    ha.load(theta, d, b, h, (j0 + 1) * LT);
    __syncthreads();
  }
  float acc[8][4];
#pragma unroll
  for (int t = 0; t < 8; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[t][e] = 0.0f;
  // products: warp (p strip of 16, half of the columns); both operands are stored across the contraction
  const int p0 = 16 * (warp & 3), n0 = 64 * (warp >> 2), l7 = lane & 7, b3 = (lane >> 3) & 1, b4 = lane >> 4;
  const uint32_t ax = (uint32_t)__cvta_generic_to_shared(sm.x) + (l7 + 8 * b4) * (kP * 2), bx = (uint32_t)__cvta_generic_to_shared(sm.b) + (l7 + 8 * b3) * (kN * 2);
  float total = 0.0f;   // log decay of the half tiles gone by
  for (int j = j0, n = 0; j < j1; ++j, ++n) {
    const HalfScal<R>& s = sm.s[n % 3];
    const float before = BWD ? exp_decay(total) : 1.0f;
#pragma unroll
    for (int i = 0; i < IT::PER; ++i) {
      const Item<R> it(i);
      const float sc = s.scale[it.l] * before;
      float cs[IT::CW], sn[IT::CW];
#pragma unroll
      for (int c = 0; c < IT::CW; ++c) { cs[c] = 1.0f; sn[c] = 0.0f; }
      if (ROT) {
#pragma unroll
        for (int c = 0; c < IT::CW; c += 4) {
          const float4 v = *reinterpret_cast<const float4*>(sm.phi + it.l * kNH + it.col + c);
          const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            cs[c + k] = __cosf(f[k]);
            sn[c + k] = __sinf(f[k]);
            if (BWD || FULL_ANGLE) {   // as in the stripe kernel's table, so that C^ (B^) is the one it has
              const float2 h = __half22float2(__floats2half2_rn(cs[c + k], sn[c + k]));
              cs[c + k] = h.x;
              sn[c + k] = h.y;
            }
          }
        }
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float o1[IT::CW], o2[IT::CW], ox[IT::CW];
#pragma unroll
        for (int c = 0; c < IT::CW; ++c) {
          const float v1 = item_el<R>(r1[i], c, r), v2 = item_el<R>(r2[i], c, r);
          o1[c] = ROT ? v1 * cs[c] + v2 * sn[c] : v1;
          o2[c] = ROT ? v2 * cs[c] - v1 * sn[c] : v2;
          ox[c] = item_el<R>(xr[i], c, r) * sc;
        }
        put<R, kN>(sm.b, it.l * R + r, it.col, o1);
        put<R, kN>(sm.b, it.l * R + r, it.col + kNH, o2);
        put<R, kP>(sm.x, it.l * R + r, it.col, ox);
      }
    }
    if (j + 1 < j1) {
      load_rows(j + 1);
      if (ROT) ha.partial(sm.q, sm.s[(n + 1) % 3].dt);
    }
    __syncthreads();
    if (!BWD) {
      const float e = exp_decay(s.cd);
#pragma unroll
      for (int t = 0; t < 8; ++t)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[t][c] *= e;
    }
#pragma unroll
    for (int k = 0; k < kRows; k += 16) {
      uint32_t fa[4], fb[4];
      ldm4t(fa, ax + k * (kP * 2) + ((((p0 >> 3) + b3) ^ l7) << 4));
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        ldm4t(fb, bx + k * (kN * 2) + (((((n0 >> 3) + 2 * t) + b4) ^ l7) << 4));
        mma16(acc[2 * t], fa, fb[0], fb[1]);
        mma16(acc[2 * t + 1], fa, fb[2], fb[3]);
      }
    }
    total += s.cd;
    if (j + 1 < j1) {
      if (ROT) {
        ha.finish(sm.phi, sm.q, sm.s[(n + 1) % 3].dt, sm.carry[(n + 1) & 1], sm.carry[n & 1]);
        ha.load(theta, d, b, h, (j + 2) * LT);
      }
      if (warp == 0) {
        hl.template work_out<BWD>(sm.s[(n + 2) % 3], A, d.T, (j + 2) * LT);
        hl.load(in, d, b, h, (j + 3) * LT);
      }
    }
    __syncthreads();
  }
  float* dst = a.hs + slot * kPN;
  const int g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int t = 0; t < 8; ++t)
#pragma unroll
    for (int e = 0; e < 4; e += 2)
      *reinterpret_cast<float2*>(dst + rows::at<kN>(p0 + g + 4 * e, n0 + 8 * t + 2 * q)) = make_float2(acc[t][e], acc[t][e + 1]);
  if (tid == 0) a.cd[slot] = total;
  if (ROT && !BWD && !FULL_ANGLE && tid < 32)
    *reinterpret_cast<float2*>(a.asum + slot * kNH + 2 * tid) = j0 < j1 ? sm.carry[(j1 - j0) & 1][tid] : make_float2(0.0f, 0.0f);
}

// A thread owns planes (m, m + 64) of rows p, p + 32 and walks the groups in time (backward: against it); U of them are
// requested before the first is used.  seg_state / seg_angle of segment s: what leaves it towards the next one walked.
// ROT: the groups have angles; LOCAL: their states are those of B rotated by the angle since the group's start.
template <bool ROT, bool BWD, bool LOCAL>
__global__ void __launch_bounds__(256) k_group_pass(Dims d, m3_scan_desc in, const float* __restrict__ dh, TcAhead a, int count) {
  after_predecessor();
  using T = __nv_bfloat16;
  constexpr int U = 8;
  const int bh = blockIdx.y, b = bh / d.H, h = bh - b * d.H;
  const int id = blockIdx.x * 256 + threadIdx.x, m = id % kNH, p = id / kNH;
  const int o[4] = {rows::at<kN>(p, m), rows::at<kN>(p, m) + kNH, rows::at<kN>(p + 32, m), rows::at<kN>(p + 32, m) + kNH};
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
    if (ROT && in.angle0) ang = wrap_angle(in.angle0[(size_t)bh * kNH + m]);
  }
  for (int i0 = 0; i0 < count; i0 += U) {
    float s[U][4], e[U], da[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = min(i0 + u, count - 1), k = BWD ? count - 1 - i : i;
      const size_t slot = (size_t)bh * count + k;
#pragma unroll
      for (int j = 0; j < 4; ++j) s[u][j] = __ldg(a.hs + slot * kPN + o[j]);
      e[u] = a.cd[slot];
      da[u] = ROT && !BWD ? a.asum[slot * kNH + m] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (i0 + u >= count) break;
      const int k = BWD ? count - 1 - (i0 + u) : i0 + u;
      float sn = 0.0f, cs = 1.0f;
      if (ROT && !BWD) {
        if (LOCAL) sincosf(ang, &sn, &cs);
        ang = wrap_angle(ang + da[u]);
      }
      const float ec = exp_decay(e[u]);
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        const float s1 = s[u][j], s2 = s[u][j + 1];
        carry[j] = fmaf(ec, carry[j], LOCAL ? s1 * cs + s2 * sn : s1);
        carry[j + 1] = fmaf(ec, carry[j + 1], LOCAL ? s2 * cs - s1 * sn : s2);
      }
      if (BWD ? k % a.gps == 0 : (k + 1) % a.gps == 0) {
        const size_t seg = (size_t)bh * a.nseg + k / a.gps + (BWD ? 1 : 0);
#pragma unroll
        for (int j = 0; j < 4; ++j) a.seg_state[seg * kPN + plain[j]] = carry[j];
        if (ROT && !BWD && p == 0) a.seg_angle[seg * kNH + m] = ang;
      }
    }
  }
}

template <int R, bool ROT, bool BWD, bool FULL_ANGLE>
cudaError_t ahead_t(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const void* dy, const float* dh, const float* ckpt_angle,
                    const TcAhead& a) {
  auto kern = k_group_state<R, ROT, BWD, FULL_ANGLE>;
  const int count = (a.nseg - 1) * a.gps;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GroupSmem<R>));
  if (e != cudaSuccess) return e;
  if (FULL_ANGLE) launch(k_group_angle<R>, dim3(count, d.B * d.H), kThreads, 0, st, d, in, a, tc_tiles(d.T, R));
  launch(kern, dim3(count, d.B * d.H), kThreads, sizeof(GroupSmem<R>), st, d, in, static_cast<const __nv_bfloat16*>(dy),
         ckpt_angle, a, tc_tiles(d.T, R));
  launch(k_group_pass<ROT, BWD, ROT && !BWD && !FULL_ANGLE>, dim3(32 * kNH / 256, d.B * d.H), 256, 0, st, d, in, dh, a, count);
  return cudaGetLastError();
}

}  // namespace

template <int R>
static cudaError_t load_r() {
  return load_kernels(k_group_state<R, true, false, false>, k_group_state<R, false, false, false>);
}
cudaError_t tc_ahead_load() {
  cudaError_t e = load_kernels(k_group_pass<true, false, true>, k_group_pass<false, false, false>);
  for (cudaError_t (*f)() : {load_r<1>, load_r<2>, load_r<4>})
    if (e == cudaSuccess) e = f();
  return e;
}

// Whether to cut `BH` stripes of `tiles` tiles into segments that run side by side, and into how many.  Microseconds,
// measured on a B200: a tile takes tc_tile_us inside a stripe, an item about one more to start and finish; working out what
// a tile adds to the state takes about 4 per tile and SM, and the two launches and the pass some 12 more.  Beyond a third of
// the SMs it takes long stripes to gain anything (96 stripes of 16 tiles: nothing; 64 of 248: forward + backward 3.47 -> 2.06 ms).
bool tc_ahead_plan(int BH, int tiles, bool backward, bool rot, int rank, int* nseg, int* tps) {
  const int sms = sm_count();
  if (BH > sms || tiles < (BH > sms / 3 ? 24 : 3)) return false;
  const float c = tc_tile_us(backward, rot, rank);
  float best = 0.92f * tiles * c;
  bool found = false;
  for (int n = 2; n <= tiles && n <= 4 * sms; ++n) {
    const int per = (tiles + n - 1) / n, segs = (tiles + per - 1) / per;
    if (segs != n) continue;
    const int rounds = (BH * segs + sms - 1) / sms;
    const float work = 4.0f * BH * (segs - 1) * per / sms;
    const float t = 12.0f + (work > 8.0f ? work : 8.0f) + rounds * (per + 1) * c;
    if (t < best) {
      best = t;
      found = true;
      *nseg = segs;
      *tps = per;
    }
  }
  return found;
}

// Groups of a segment: as long as there are some two blocks per SM, as a group's state goes through memory once; single
// tiles where there are fewer.
static void ahead_groups(int BH, TcAhead* a) {
  a->gt = a->tps;
  while (a->gt > 1 && (long long)BH * (a->nseg - 1) * ((a->tps + a->gt - 1) / a->gt) < 2 * sm_count()) a->gt = (a->gt + 1) / 2;
  a->gps = (a->tps + a->gt - 1) / a->gt;
}

size_t tc_ahead_bytes(int BH, TcAhead* a, char* base) {
  size_t at = 0;
  auto take = [&](size_t n) {
    float* p = base ? reinterpret_cast<float*>(base + at) : nullptr;
    at += (n * sizeof(float) + 255) / 256 * 256;
    return p;
  };
  ahead_groups(BH, a);
  const size_t groups = (size_t)BH * (a->nseg - 1) * a->gps;
  a->hs = take(groups * kPN);
  a->asum = take(groups * kNH);
  a->cd = take(groups);
  a->seg_state = take((size_t)BH * a->nseg * kPN);
  a->seg_angle = take((size_t)BH * a->nseg * kNH);
  return at;
}

cudaError_t tc_ahead(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const void* dy, const float* dh,
                     const float* ckpt_angle, const TcAhead& a, bool full_angle, uint64_t* launches) {
  const bool known = full_angle && d.rot && !dy;
  *launches += known ? 3 : 2;
  auto go = [&](auto r, auto rot) {
    if (dy) return ahead_t<r.value, rot.value, true, false>(st, d, in, dy, dh, ckpt_angle, a);
    if constexpr (rot.value)
      if (known) return ahead_t<r.value, true, false, true>(st, d, in, nullptr, nullptr, nullptr, a);
    return ahead_t<r.value, rot.value, false, false>(st, d, in, nullptr, nullptr, nullptr, a);
  };
  auto with_rot = [&](auto r) { return d.rot ? go(r, std::true_type{}) : go(r, std::false_type{}); };
  switch (d.R) {
    case 1: return with_rot(std::integral_constant<int, 1>{});
    case 2: return with_rot(std::integral_constant<int, 2>{});
    default: return with_rot(std::integral_constant<int, 4>{});
  }
}

}  // namespace m3
