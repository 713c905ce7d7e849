// Shared device code of the chunk-parallel family (m3_rows_fwd.cu, m3_rows_bwd.cu): float32 arithmetic for head_dim 64,
// d_state 64 or 128, rank 1, 2 or 4 - every float32 model shape, and bf16 at d_state 64.
//
// A CTA works on one chunk of 64 rows rho = (t, r) (64 / R time steps) of one (batch, head); all chunks of all stripes
// run at once and only the pass over chunk states is sequential (m3_rows_fwd.cu says which kernels there are).
//
// Contractions run on the tensor cores in split TF32: an operand x is hi + lo, hi = x rounded to TF32's 11 significant bits,
// lo = the rest cut to as many, and a product is lo hi + hi lo + hi hi; what is dropped (lo lo, and what is cut from lo) is
// below 2^-22 of it.  For float32 tensors the sum over the contraction is kept by the float32 units (warp_mma says why): with
// hi cut and the whole sum left to the tensor core, y, d x, d B and d C were 2.7 to 4.6 times as far from 64-bit results as
// the generic family's, now 0.6 to 0.9 times, for 2 % of the time (8 x 1024 tokens x 16 heads, d_state 128, mixer forward +
// backward: 1125 -> 1149 us; the double sums of the log decay, SumOf, and the skip's place in d x: 1165 us).  mma.sync m16n8k8
// runs 278 TFLOP/s on a B200, so 93 after the threefold product, against 51 measured for float32 FMAs from registers (and half
// of that in the 64 x 64 block products of the generic family).  Fragments come four words at a time by ldmatrix where the
// operand is stored along the contraction.  tcgen05's kind::tf32 would be faster still, but wants every operand K-major in
// shared memory: half of the operands here are contracted along their rows.  An operand whose values are bf16 already is its
// own hi part and needs no lo product.
//
// Operands lie in shared memory as [row][col] floats with leading dimension N or 64, columns XOR-swizzled by fsw(row),
// so that fragments along either index come without bank conflicts: eight rows x four columns (an operand contracted
// along its columns) and four rows x eight columns (along its rows) both touch 32 different banks.
#pragma once
#include <type_traits>

#include "m3_internal.h"

namespace m3 {
namespace rows {

constexpr int kP = 64, kRows = 64;

__host__ __device__ __forceinline__ constexpr int fsw(int row) { return ((row & 1) << 4) | ((row & 2) << 2) | (row & 4); }
template <int LD>
__device__ __forceinline__ int at(int row, int col) { return row * LD + (col ^ fsw(row)); }

// hi is x rounded to the 19 bits that the tensor core reads of a TF32 operand, lo the rest (exact; the tensor core reads its
// upper 19 bits, which cuts it below 2^-23 of x).  Rounding hi makes lo's sign independent of x's, so that neither what is
// cut from lo nor the dropped lo lo pulls a sum one way.
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
  hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  lo = __float_as_uint(x - __uint_as_float(hi));
}
// Four 8-row x 4-column pieces of float32 by one instruction: word q of row g of each is this lane's.
__device__ __forceinline__ void ldm4f(uint32_t (&r)[4], const float* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(p))
               : "memory");
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// The same into registers that need not be cleared first.
__device__ __forceinline__ void mma_tf32_new(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.0f));
}

// acc[mt][nt] += A[m0 + 16 mt.., k] B[k, n0 + 8 nt..] over k in [k0, k1) (multiples of 8), by one warp.
// AKC: A is stored [m][k], else [k][m]; BKC: B is stored [n][k], else [k][n].  AEX / BEX: that operand's values are
// exact in TF32.  Accumulator layout: element e of a tile is row g + 8 (e >> 1), column 2 q + (e & 1), with g = lane / 4,
// q = lane % 4.
// SUM: the products of every eight k are summed in the tensor core and added to acc by the float32 units, whose additions
// round to nearest; the tensor core's own cut, which over a sum of 64 to 128 would be most of the error (float32).  Tensors of
// bf16 leave the whole sum to the tensor core.
template <int MT, int NT, bool AKC, bool BKC, bool AEX, bool BEX, int LDA, int LDB, bool SUM>
__device__ __forceinline__ void warp_mma(float (&acc)[MT][NT][4], const float* sA, int m0, const float* sB, int n0, int k0,
                                         int k1) {
  static_assert(!BKC || NT % 2 == 0, "a load brings two column tiles");
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  const int fq = fsw(q), fq4 = fq ^ 4, f7 = fsw(lane & 7);
  // this lane's row and column group in a load of four pieces (operands stored along k)
  const float* pa = sA + (m0 + (lane & 15)) * LDA;
  const float* pb = sB + (n0 + (lane & 7) + ((lane >> 4) << 3)) * LDB;
  const int ka = (lane >> 4) << 2, kb = ((lane >> 3) & 1) << 2;
#pragma unroll 2
  for (int k = k0; k < k1; k += 8) {
    uint32_t ah[MT][4], al[MT][4], bh[NT][2], bl[NT][2];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      if (AKC) {
        ldm4f(ah[mt], pa + 16 * mt * LDA + ((k + ka) ^ f7));
      } else {
        const int m = m0 + 16 * mt + g;
        const float* r0 = sA + (k + q) * LDA;
        const float* r1 = r0 + 4 * LDA;
        ah[mt][0] = __float_as_uint(r0[m ^ fq]); ah[mt][1] = __float_as_uint(r0[(m + 8) ^ fq]);
        ah[mt][2] = __float_as_uint(r1[m ^ fq4]); ah[mt][3] = __float_as_uint(r1[(m + 8) ^ fq4]);
      }
      if (!AEX) {
#pragma unroll
        for (int i = 0; i < 4; ++i) split_tf32(__uint_as_float(ah[mt][i]), ah[mt][i], al[mt][i]);
      }
    }
    if (BKC) {
#pragma unroll
      for (int np = 0; np < NT / 2; ++np) {
        uint32_t r[4];
        ldm4f(r, pb + 16 * np * LDB + ((k + kb) ^ f7));
        bh[2 * np][0] = r[0]; bh[2 * np][1] = r[1];
        bh[(2 * np + 1) % NT][0] = r[2]; bh[(2 * np + 1) % NT][1] = r[3];
      }
    } else {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int n = n0 + 8 * nt + g;
        const float* r0 = sB + (k + q) * LDB;
        bh[nt][0] = __float_as_uint(r0[n ^ fq]); bh[nt][1] = __float_as_uint(r0[4 * LDB + (n ^ fq4)]);
      }
    }
    if (!BEX) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int i = 0; i < 2; ++i) split_tf32(__uint_as_float(bh[nt][i]), bh[nt][i], bl[nt][i]);
    }
    if constexpr (SUM) {
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          float t[4];
          if (!AEX) mma_tf32_new(t, al[mt], bh[nt]); else if (!BEX) mma_tf32_new(t, ah[mt], bl[nt]); else mma_tf32_new(t, ah[mt], bh[nt]);
          if (!AEX && !BEX) mma_tf32(t, ah[mt], bl[nt]);
          if (!AEX || !BEX) mma_tf32(t, ah[mt], bh[nt]);
          if constexpr (MT * NT <= 4) {   // two sums per instruction (with more tiles the pairs cost spills: 88 -> 89 us of states)
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
              const float2 v = __fadd2_rn(make_float2(acc[mt][nt][e], acc[mt][nt][e + 1]), make_float2(t[e], t[e + 1]));
              acc[mt][nt][e] = v.x;
              acc[mt][nt][e + 1] = v.y;
            }
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[mt][nt][e] += t[e];
          }
        }
    } else {
      if (!AEX) {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) mma_tf32(acc[mt][nt], al[mt], bh[nt]);
      }
      if (!BEX) {
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) mma_tf32(acc[mt][nt], ah[mt], bl[nt]);
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) mma_tf32(acc[mt][nt], ah[mt], bh[nt]);
    }
  }
}
template <int MT, int NT>
__device__ __forceinline__ void zero(float (&acc)[MT][NT][4]) {
#pragma unroll
  for (int a = 0; a < MT; ++a)
#pragma unroll
    for (int b = 0; b < NT; ++b)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[a][b][e] = 0.0f;
}
// f(row, col, pair of accumulators in columns col, col + 1) over a warp's accumulators.
template <int MT, int NT, class F>
__device__ __forceinline__ void for_acc(float (&acc)[MT][NT][4], int m0, int n0, F f) {
  const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int hh = 0; hh < 2; ++hh)
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
        f(m0 + 16 * mt + 8 * hh + g, n0 + 8 * nt + 2 * q, acc[mt][nt][2 * hh], acc[mt][nt][2 * hh + 1]);
}
// Accumulators into a swizzled [row][col] buffer.
template <int LD, int MT, int NT>
__device__ __forceinline__ void store_acc(float (&acc)[MT][NT][4], int m0, int n0, float* dst) {
  for_acc(acc, m0, n0, [&](int row, int col, float& a, float& b) {
    *reinterpret_cast<float2*>(dst + at<LD>(row, col)) = make_float2(a, b);
  });
}

// Four consecutive elements of a tensor as floats (16-byte aligned float32, 8-byte aligned bf16), and back.
__device__ __forceinline__ float4 load4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 w = __ldg(reinterpret_cast<const uint2*>(p));
  return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16),
                     __uint_as_float(w.y & 0xffff0000u));
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  uint2 w;
  w.x = *reinterpret_cast<const uint32_t*>(&a);
  w.y = *reinterpret_cast<const uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = w;
}

// What a kernel knows about its chunk.
struct Chunk {
  int k, bh, b, h, t0;   // chunk, stripe, batch row, head, first scan position
};
__device__ __forceinline__ Chunk this_chunk(const Dims& d) {
  Chunk c;
  c.k = blockIdx.x; c.bh = blockIdx.y;
  c.b = c.bh / d.H; c.h = c.bh - c.b * d.H; c.t0 = c.k * d.L;
  return c;
}

// Per-token scalars of a chunk in shared memory: dt, lambda (one step of look-ahead), cumulative log decay, weights,
// exp(ac), exp(cd - ac) and that times w.
template <int R>
struct Scal {
  static constexpr int LT = kRows / R;
  float dt[LT + 1], lam[LT + 1], ac[LT], g[LT], w[LT], eac[LT], dte[LT], sw[LT];
};
// What the sums of the log decay and of its gradient over a chunk are kept in.  Sums by a tree do not share their roundings
// as sequential ones do, and the differences of two of them near the chunk's end, which weigh most, would carry those of the
// whole sum: double for float32 tensors.  (Far below the rounding of bf16 tensors.)
template <class T>
using SumOf = std::conditional_t<sizeof(T) == 4, double, float>;
// Inclusive prefix sum over the lanes (SUFFIX: over this lane and those behind it).
template <bool SUFFIX, class S>
__device__ __forceinline__ S lane_scan(S v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const S n = SUFFIX ? __shfl_down_sync(0xffffffffu, v, o) : __shfl_up_sync(0xffffffffu, v, o);
    if (SUFFIX ? lane + o < 32 : lane >= o) v += n;
  }
  return v;
}
// Contains two block barriers; complete after the caller's next one.
template <class T, int R>
__device__ __forceinline__ void chunk_scalars(Scal<R>& s, const Dims& d, const Chunk& c, const m3_scan_desc& in) {
  constexpr int LT = kRows / R;
  const int tid = threadIdx.x;
  if (tid <= LT) {
    const int t = c.t0 + tid;
    float vdt = 0.0f, vl = 1.0f;
    if (t < d.T && !d.raw) {
      const size_t i = tok_index(d, c.b, t, c.h);
      vdt = ldf(static_cast<const T*>(in.dt), i);
      vl = lambda_at(static_cast<const T*>(in.lambda), d.disc, i);
    }
    s.dt[tid] = vdt;
    s.lam[tid] = vl;
  }
  __syncthreads();
  if (tid < 32) {
    constexpr int EPL = LT >= 32 ? LT / 32 : 1;
    const float A = d.raw ? 0.0f : -expf(in.a_log[c.h]);
    SumOf<T> loc[EPL], run = 0;
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
      const int l = tid * EPL + i, t = c.t0 + l;
      float gv = 0.0f, wv = 0.0f;
      SumOf<T> av = 0;
      if (l < LT && t < d.T) {
        if (d.raw) {  // scan.rs:116-126: the caller's own a, g, w
          const size_t o = tok_index(d, c.b, t, c.h);
          av = ldf(static_cast<const T*>(in.a_raw), o);
          gv = ldf(static_cast<const T*>(in.g_raw), o);
          wv = ldf(static_cast<const T*>(in.w_raw), o);
        } else {
          av = (SumOf<T>)s.dt[l] * A;
          gv = s.lam[l] * s.dt[l];
          wv = gv + (t + 1 < d.T ? (1.0f - s.lam[l + 1]) * s.dt[l + 1] : 0.0f);
        }
      }
      if (l < LT) { s.g[l] = gv; s.w[l] = wv; }
      run += av;
      loc[i] = run;
    }
    const SumOf<T> tot = lane_scan<false>(run), base = tot - run, cd = __shfl_sync(0xffffffffu, tot, 31);
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
      const int l = tid * EPL + i;
      if (l < LT) {
        const SumOf<T> ac = base + loc[i];
        s.ac[l] = (float)(l == LT - 1 ? cd : ac);
        s.eac[l] = exp_decay((float)ac);
        s.dte[l] = exp_decay((float)(cd - ac));
        s.sw[l] = s.dte[l] * s.w[l];
      }
    }
  }
  __syncthreads();
}

// Cumulative angle of a chunk, phi[l * NH + m] = base[m] + sum_{l' <= l} dt theta (wrapped), by THREADS threads;
// s_q: THREADS floats.  total(m, sum): called once per plane with the chunk's sum.  Needs s.dt; contains a barrier,
// complete after the caller's next one.
template <class T, int N, int R, int THREADS, class F>
__device__ __forceinline__ void chunk_angles(float* phi, float* s_q, const Scal<R>& s, const Dims& d, const Chunk& c,
                                             const T* theta, const float* base, F total) {
  constexpr int NH = N / 2, LT = kRows / R, NQ = THREADS / NH < LT ? THREADS / NH : LT, LQ = LT / NQ;
  const int q = threadIdx.x / NH, m = threadIdx.x % NH;
  float loc[LQ], run = 0.0f;
  if (q < NQ) {
    float th[LQ];
#pragma unroll
    for (int i = 0; i < LQ; ++i) {
      const int t = c.t0 + q * LQ + i;
      th[i] = t < d.T ? ldf(theta, theta_index(d, c.b, t, c.h) + m) : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < LQ; ++i) {
      run += s.dt[q * LQ + i] * th[i];
      loc[i] = run;
    }
    s_q[q * NH + m] = run;
  }
  __syncthreads();
  if (q < NQ) {
    float off = base ? base[m] : 0.0f;
    float before = 0.0f;
    for (int j = 0; j < q; ++j) before += s_q[j * NH + m];
#pragma unroll
    for (int i = 0; i < LQ; ++i) {
      // wrap_angle without its division: for the sines only, where a whole turn more or less at the ends does not matter
      const float v = off + before + loc[i];
      phi[(q * LQ + i) * NH + m] = fmaf(rintf(v * 0.15915494309189535f), -kTwoPi, v);
    }
    if (q == NQ - 1) total(m, before + run);
  }
}

// Rows of a [.., cols, R] tensor of the caller into a swizzled [64][cols] buffer (rank de-interleaved, zero past T).
template <class T, int R, int COLS, int THREADS>
__device__ __forceinline__ void load_rows(float* dst, const T* src, const Dims& d, const Chunk& c) {
  constexpr int LT = kRows / R, PER = COLS * R / 4;
  static_assert(LT * PER % THREADS == 0, "whole rounds");
#pragma unroll
  for (int i = 0; i < LT * PER / THREADS; ++i) {
    const int it = threadIdx.x + i * THREADS, l = it / PER, e = 4 * (it - l * PER), t = c.t0 + l;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (t < d.T) v = load4(src + tok_index(d, c.b, t, c.h) * COLS * R + e);
    if (R == 1) {
      *reinterpret_cast<float4*>(dst + at<COLS>(l, e)) = v;
    } else {
      const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) dst[at<COLS>(l * R + (e + j) % R, (e + j) / R)] = f[j];
    }
  }
}

// sin and cos of an angle in [-pi, pi], by the function that takes it in units of pi: no branch for large arguments, whose
// code and stack sincosf carries; the scaling moves the angle by less than its own last bit.
__device__ __forceinline__ void sincos_wrapped(float phi, float* sn, float* cs) { sincospif(phi * 0.31830988618379067f, sn, cs); }

// Rows of B or C (two tensors at once share the sines), rotated by -phi; `scale` (per step, or NULL) multiplies them.
template <class T, int N, int R, int THREADS, int NTENS>
__device__ __forceinline__ void load_rotated(float* const (&dst)[NTENS], const T* const (&src)[NTENS], const float* phi,
                                             const float* scale, const Dims& d, const Chunk& c) {
  constexpr int LT = kRows / R, NH = N / 2, PER = NH * R / 4, NA = R == 1 ? 4 : (R == 2 ? 2 : 1);
#pragma unroll
  for (int i = 0; i < LT * PER / THREADS; ++i) {
    const int it = threadIdx.x + i * THREADS, l = it / PER, e = 4 * (it - l * PER), t = c.t0 + l;
    float4 v1[NTENS], v2[NTENS];
#pragma unroll
    for (int w = 0; w < NTENS; ++w) {
      v1[w] = v2[w] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (t < d.T) {
        const T* p = src[w] + tok_index(d, c.b, t, c.h) * N * R + e;
        v1[w] = load4(p);
        v2[w] = load4(p + NH * R);
      }
    }
    float cs[NA], sn[NA];
    const float sc = scale ? scale[l] : 1.0f;
#pragma unroll
    for (int j = 0; j < NA; ++j) {
      sincos_wrapped(phi[l * NH + e / R + j], &sn[j], &cs[j]);
      cs[j] *= sc;
      sn[j] *= sc;
    }
#pragma unroll
    for (int w = 0; w < NTENS; ++w) {
      const float a[4] = {v1[w].x, v1[w].y, v1[w].z, v1[w].w}, b[4] = {v2[w].x, v2[w].y, v2[w].z, v2[w].w};
      float o1[4], o2[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        o1[j] = a[j] * cs[j / R] + b[j] * sn[j / R];
        o2[j] = b[j] * cs[j / R] - a[j] * sn[j / R];
      }
      if (R == 1) {
        *reinterpret_cast<float4*>(dst[w] + at<N>(l, e)) = make_float4(o1[0], o1[1], o1[2], o1[3]);
        *reinterpret_cast<float4*>(dst[w] + at<N>(l, e + NH)) = make_float4(o2[0], o2[1], o2[2], o2[3]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int row = l * R + (e + j) % R, n = (e + j) / R;
          dst[w][at<N>(row, n)] = o1[j];
          dst[w][at<N>(row, n + NH)] = o2[j];
        }
      }
    }
  }
}
// The same without a rotation.
template <class T, int N, int R, int THREADS>
__device__ __forceinline__ void load_scaled(float* dst, const T* src, const float* scale, const Dims& d, const Chunk& c) {
  constexpr int LT = kRows / R, PER = N * R / 4;
#pragma unroll
  for (int i = 0; i < LT * PER / THREADS; ++i) {
    const int it = threadIdx.x + i * THREADS, l = it / PER, e = 4 * (it - l * PER), t = c.t0 + l;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (t < d.T) v = load4(src + tok_index(d, c.b, t, c.h) * N * R + e);
    const float sc = scale[l];
    const float f[4] = {v.x * sc, v.y * sc, v.z * sc, v.w * sc};
    if (R == 1) {
      *reinterpret_cast<float4*>(dst + at<N>(l, e)) = make_float4(f[0], f[1], f[2], f[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) dst[at<N>(l * R + (e + j) % R, (e + j) / R)] = f[j];
    }
  }
}

// A swizzled [64][COLS] buffer out to rows of a [.., COLS, R] tensor (rank interleaved again), 16 (8) bytes a thread.
template <class T, int R, int COLS, int THREADS>
__device__ __forceinline__ void store_rows(T* dst, const float* src, const Dims& d, const Chunk& c) {
  constexpr int LT = kRows / R, PER = COLS * R / 4;
#pragma unroll
  for (int i = 0; i < LT * PER / THREADS; ++i) {
    const int it = threadIdx.x + i * THREADS, l = it / PER, e = 4 * (it - l * PER), t = c.t0 + l;
    if (t >= d.T) continue;
    float4 v;
    if (R == 1) {
      v = *reinterpret_cast<const float4*>(src + at<COLS>(l, e));
    } else {
      float f[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) f[j] = src[at<COLS>(l * R + (e + j) % R, (e + j) / R)];
      v = make_float4(f[0], f[1], f[2], f[3]);
    }
    store4(dst + tok_index(d, c.b, t, c.h) * COLS * R + e, v);
  }
}

// Sum over the lanes of a quad (the columns of a row), and over the eight lanes of equal q (the rows of a column).
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ float group_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  v += __shfl_xor_sync(0xffffffffu, v, 8);
  return v + __shfl_xor_sync(0xffffffffu, v, 16);
}

// Scratch of a forward pass that a backward pass may need (floats).  States are kept [p][n] with the columns swizzled
// by p as in shared memory, so that they move as they are.
struct RowsWs {
  float* hs;     // [BH, C, P, N] local chunk state, then the state entering the chunk
  float* asum;   // [BH, C, NH] the chunk's angle
  float* abase;  // [BH, C, NH] the angle entering it
  float* cd;     // [BH, C] its log decay
};
struct RowsBwdWs {
  float* dhs;    // [BH, C + 1, P, N] local dH, then dS_k; slot C: the gradient of the seed state
  float* dphi;   // [BH, Tp, NH] sum of d phi over the rest of the chunk
  float* dpsum;  // [BH, C, NH] over the chunk
};

// f(element type, N, R, rotational) as compile-time constants for a shape the family serves.
template <class F>
cudaError_t dispatch(const Dims& d, const m3_scan_desc& in, F f) {
  auto with_rot = [&](auto t, auto n, auto r) {
    return d.rot ? f(t, n, r, std::true_type{}) : f(t, n, r, std::false_type{});
  };
  auto with_rank = [&](auto t, auto n) {
    if (d.R == 1) return with_rot(t, n, std::integral_constant<int, 1>{});
    if (d.R == 2) return with_rot(t, n, std::integral_constant<int, 2>{});
    return with_rot(t, n, std::integral_constant<int, 4>{});
  };
  auto with_n = [&](auto t) {
    return d.N == 64 ? with_rank(t, std::integral_constant<int, 64>{}) : with_rank(t, std::integral_constant<int, 128>{});
  };
  return in.dtype == M3_BF16 ? with_n(__nv_bfloat16{}) : with_n(float{});
}

cudaError_t dh_local(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const void* dy, const RowsWs& ws, float* dhs);

}  // namespace rows

// Whether the family serves a descriptor (its y included).
bool rows_supported(const m3_scan_desc& s, const void* y);
// The extents with this family's chunk.
Dims rows_dims(Dims d);
size_t rows_ws_layout(const Dims& d, rows::RowsWs* ws, char* base);
cudaError_t rows_forward(cudaStream_t st, const Dims& d, const m3_scan_desc& desc, const m3_scan_out& out,
                         const rows::RowsWs& ws, uint64_t* launches);
cudaError_t rows_load(int dtype);   // load_kernels of every kernel a forward pass of the element type may launch
// The last pass over tokens for the tensor-core family's side-by-side segments (bf16, d_state 128, rotational): d.L steps
// per tile, `per_seg` tiles per segment.
cudaError_t rows_final(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const float* dphi, const float* dpsum, int per_seg,
                       int nseg, const GenericBwdWs& bw, void* ddt, void* dlam, void* dtheta, float* dangle0, const HeadSums& hs);
size_t rows_bwd_ws_layout(const Dims& d, rows::RowsBwdWs* rw, GenericBwdWs* bw, char* base);
cudaError_t rows_backward(cudaStream_t st, const Dims& d, const m3_scan_desc& desc, const rows::RowsWs& ws,
                          const rows::RowsBwdWs& rw, const GenericBwdWs& bw, const m3_scan_bwd_in& in, uint32_t mask,
                          const m3_scan_grads& grads, uint64_t* launches);

}  // namespace m3
