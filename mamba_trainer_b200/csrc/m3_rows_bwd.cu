// Backward of the chunk-parallel family (m3_rows.cuh), the hand adjoint of m3_rows_fwd.cu.  Launches:
//   k_rows_state     (m3_rows_fwd.cu) local dH_k = (exp(acum) dY~)^T C^ of every chunk
//   k_rows_pass_rev  sequential over chunks: dS_k = dH_{k+1}, dH_k = exp(cd_k) dH_{k+1} + Rot(local)
//   k_rows_adjoint   per chunk, everything that needs its rows: d x, d B, d C, the band adjoint, the per-token
//                    scalars' gradients, d phi summed backwards within the chunk
//   k_rows_final     per chunk: the later chunks' d phi on top -> d theta, d dt, d lambda
// (plus the seed state's gradients and the per-head sums).  The generic family took 15 launches and wrote dX~, dB^, dC^,
// d band and d phi to global memory in between: 1.96 ms for float32, batch 8 x 1024 tokens x 16 heads, d_state 128.
#include "m3_rows.cuh"

namespace m3 {
namespace rows {
namespace {

template <int N, bool ROT>
__global__ void __launch_bounds__(256) k_rows_pass_rev(Dims d, const float* __restrict__ dh, RowsWs ws, RowsBwdWs rw) {
  after_predecessor();
  constexpr int NH = N / 2, PN = kP * N, U = 4;
  const int bh = blockIdx.y;
  const int id = blockIdx.x * 256 + threadIdx.x, m = id % NH, p = id / NH;   // planes (m, m + NH) of rows p, p + 32
  const int o[4] = {at<N>(p, m), at<N>(p, m) + NH, at<N>(p + 32, m), at<N>(p + 32, m) + NH};
  const int plain[4] = {p * N + m, p * N + m + NH, (p + 32) * N + m, (p + 32) * N + m + NH};
  float carry[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) carry[i] = dh ? dh[(size_t)bh * PN + plain[i]] : 0.0f;
  float* hs = rw.dhs + (size_t)bh * (d.C + 1) * PN;
  for (int k1 = d.C - 1; k1 >= 0; k1 -= U) {
    float s[U][4], ecd[U], ang[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const size_t k = max(k1 - u, 0);
#pragma unroll
      for (int i = 0; i < 4; ++i) s[u][i] = hs[k * PN + o[i]];
      ecd[u] = ws.cd[(size_t)bh * d.C + k];
      ang[u] = ROT ? ws.abase[((size_t)bh * d.C + k) * NH + m] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (k1 - u < 0) break;
      const size_t k = k1 - u;
      float sn = 0.0f, cs = 1.0f;
      if (ROT) sincosf(ang[u], &sn, &cs);
      const float e = exp_decay(ecd[u]);
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        hs[k * PN + o[i]] = carry[i];
        hs[k * PN + o[i + 1]] = carry[i + 1];
        const float s1 = s[u][i], s2 = s[u][i + 1];
        carry[i] = fmaf(e, carry[i], ROT ? s1 * cs + s2 * sn : s1);
        carry[i + 1] = fmaf(e, carry[i + 1], ROT ? s2 * cs - s1 * sn : s2);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) hs[(size_t)d.C * PN + o[i]] = carry[i];
}

// Gradients of the seed state: dh0 = dH_0, dlast_u0 = (1 - lambda_0) dt_0 dH_0, and <dH_0, last_u0> for d dt_0, d lambda_0.
template <class T, int N>
__global__ void __launch_bounds__(256) k_rows_seed(Dims d, m3_scan_desc in, RowsBwdWs rw, float* __restrict__ ip0,
                                                   float* __restrict__ dh0, float* __restrict__ dlu0) {
  after_predecessor();
  __shared__ float red[8];
  constexpr int PN = kP * N;
  const int bh = blockIdx.x, b = bh / d.H, h = bh - b * d.H;
  const float* g = rw.dhs + ((size_t)bh * (d.C + 1) + d.C) * PN;
  float first = 0.0f;
  if (!d.raw) {
    const size_t i0 = tok_index(d, b, 0, h);
    first = (1.0f - lambda_at(static_cast<const T*>(in.lambda), d.disc, i0)) * ldf(static_cast<const T*>(in.dt), i0);
  }
  float s = 0.0f;
  for (int e = threadIdx.x; e < PN; e += 256) {
    const float v = g[at<N>(e / N, e % N)];
    const size_t o = (size_t)bh * PN + e;
    if (dh0) dh0[o] = v;
    if (dlu0) dlu0[o] = first * v;
    if (in.last_u0 && !d.raw) s += v * in.last_u0[o];
  }
  s = block_sum_256(s, red);
  if (threadIdx.x == 0) ip0[bh] = s;
}

// Threads of k_rows_adjoint.  d_state 128: 16 warps, one CTA per SM (177 KB of shared memory).  d_state 64: 8 warps with
// tiles twice as wide, so that two CTAs share an SM and one's products run beside the other's loads and epilogues
// (bf16, 4 x 1500 tokens x 8 heads: 120 -> 93 us).
template <int N>
constexpr int kAdjThreads = N == 64 ? 256 : 512;
template <int N, int R>
struct AdjSmem {
  static constexpr int kThreads = kAdjThreads<N>, WC = kThreads / 128, WN = kThreads / 64;   // warp columns: see the kernel
  float c[kRows * N], b[kRows * N], x[kRows * kP], dy[kRows * kP];
  float hs[2 * kRows * N];   // H_k and dS_k; then M and dG; then dB and dC on their way out
  float phi[(kRows / R) * (N / 2)];
  float row[WC][kRows], col[4][kRows], dw[4][kRows], dg[WC][kRows], q[WC][kRows], t1[WN][kRows];   // partial sums per warp column / row
  float sq[kThreads], red[16], dac[kRows / R], dast[kRows / R];
  Scal<R> s;
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// Sum over the block; complete for every thread.
template <int kAdj>
__device__ __forceinline__ float adj_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < kAdj / 32; ++i) s += red[i];
  return s;
}

static_assert(sizeof(AdjSmem<64, 1>) <= 115712, "two CTAs share an SM");

template <class T>
struct AdjOut {
  T *dx, *db, *dc;                  // NULL skips the store
  float *da, *dg, *dw;              // [BH, Tp]
  float *part_a, *part_d;           // [BH, C]
  const float *dlu, *dangle;        // gradients that reach the returned state, or NULL
};

template <class T, int N, int R, bool ROT>
__global__ void __launch_bounds__(kAdjThreads<N>, N == 64 ? 2 : 1) k_rows_adjoint(Dims d, m3_scan_desc in, const T* __restrict__ dy, RowsWs ws,
                                                          RowsBwdWs rw, AdjOut<T> out) {
  after_predecessor();
  extern __shared__ __align__(16) unsigned char smem[];
  AdjSmem<N, R>& sm = *reinterpret_cast<AdjSmem<N, R>*>(smem);
  constexpr int NH = N / 2, PN = kP * N, LT = kRows / R, kAdj = kAdjThreads<N>;
  constexpr bool EX = sizeof(T) == 2;   // x and dy of a bf16 tensor are exact in TF32
  const Chunk c = this_chunk(d);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q4 = lane & 3;
  float *sH = sm.hs, *sS = sm.hs + PN, *sM = sm.hs, *sG = sm.hs + kRows * kRows, *sDB = sm.hs, *sDC = sm.hs + kRows * N;
  // ---- the chunk's rows and states ------------------------------------------------------------------------
  {
    const float* h = ws.hs + ((size_t)c.bh * d.C + c.k) * PN;
    const float* s = rw.dhs + ((size_t)c.bh * (d.C + 1) + c.k) * PN;
    for (int i = 4 * tid; i < PN; i += 4 * kAdj) {
      cp_async16(sH + i, h + i);
      cp_async16(sS + i, s + i);
    }
  }
  load_rows<T, R, kP, kAdj>(sm.x, static_cast<const T*>(in.x), d, c);
  load_rows<T, R, kP, kAdj>(sm.dy, dy, d, c);
  chunk_scalars<T, R>(sm.s, d, c, in);
  if constexpr (ROT) {
    chunk_angles<T, N, R, kAdj>(sm.phi, sm.sq, sm.s, d, c, static_cast<const T*>(in.theta),
                                ws.abase + ((size_t)c.bh * d.C + c.k) * NH, [](int, float) {});
    __syncthreads();
    float* const to[2] = {sm.b, sm.c};
    const T* const from[2] = {static_cast<const T*>(in.b), static_cast<const T*>(in.c)};
    load_rotated<T, N, R, kAdj, 2>(to, from, sm.phi, nullptr, d, c);
  } else {
    load_rows<T, R, N, kAdj>(sm.b, static_cast<const T*>(in.b), d, c);
    load_rows<T, R, N, kAdj>(sm.c, static_cast<const T*>(in.c), d, c);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const Scal<R>& ts = sm.s;
  // ---- products that need the states ------------------------------------------------------------------------
  constexpr int WC = AdjSmem<N, R>::WC, WN = AdjSmem<N, R>::WN;
  constexpr int NT = N / (8 * WN);   // [64 x N] results: warps 2 (32 rows) x WN
  const int wm = warp & 1, wn = warp >> 1, M0 = 32 * wm, N0 = 8 * NT * wn;
  constexpr int NX = 8 / WC;         // [64 x 64] results: warps 4 (16 rows) x WC
  const int m0 = 16 * (warp & 3), n0 = 8 * NX * (warp >> 2);
  float dc[2][NT][4], db[2][NT][4], dx[1][NX][4];
  const float dsk = in.d_skip ? in.d_skip[c.h] : 0.0f;
  zero(dc);
  zero(db);
  zero(dx);
  warp_mma<2, NT, true, false, EX, false, kP, N, !EX>(dc, sm.dy, M0, sH, N0, 0, kP);   // T1 = dY~ H_k
  warp_mma<2, NT, true, false, EX, false, kP, N, !EX>(db, sm.x, M0, sS, N0, 0, kP);    // X~ dS_k
  warp_mma<1, NX, true, true, false, false, N, N, !EX>(dx, sm.b, m0, sS, n0, 0, N);     // U = B^ dS_k^T
  {
    float t1[2][2] = {{0.0f, 0.0f}, {0.0f, 0.0f}};   // <T1, C^> of the rows
    for_acc(dc, M0, N0, [&](int row, int col, float& a, float& b) {
      const float2 cv = *reinterpret_cast<const float2*>(sm.c + at<N>(row, col));
      const int i = (row - M0 - g) >> 3;
      t1[i >> 1][i & 1] += a * cv.x + b * cv.y;
      const float e = ts.eac[row / R];
      a *= e;
      b *= e;
    });
    for_acc(db, M0, N0, [&](int row, int, float& a, float& b) {
      const float e = ts.sw[row / R];
      a *= e;
      b *= e;
    });
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float v = quad_sum(t1[i >> 1][i & 1]);
      if (q4 == 0) sm.t1[wn][M0 + 8 * i + g] = v;
    }
    float qs[2] = {0.0f, 0.0f};   // q = <U, x> of the rows; dX~ starts as sw U (+ D dy)
    for_acc(dx, m0, n0, [&](int row, int col, float& a, float& b) {
      const float2 xv = *reinterpret_cast<const float2*>(sm.x + at<kP>(row, col));
      qs[(row - m0 - g) >> 3] += a * xv.x + b * xv.y;
      const float e = ts.sw[row / R];
      a *= e;
      b *= e;
      if (EX) {
        const float2 gv = *reinterpret_cast<const float2*>(sm.dy + at<kP>(row, col));
        a = fmaf(dsk, gv.x, a);
        b = fmaf(dsk, gv.y, b);
      }
    });
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float v = quad_sum(qs[i]);
      if (q4 == 0) sm.q[warp >> 2][m0 + 8 * i + g] = v;
    }
  }
  float dcd = 0.0f, dD = 0.0f;
  for (int i = 4 * tid; i < PN; i += 4 * kAdj) {
    const float4 a = *reinterpret_cast<const float4*>(sH + i), b = *reinterpret_cast<const float4*>(sS + i);
    dcd += a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w;
  }
  if (in.d_skip) {
    for (int i = 4 * tid; i < kRows * kP; i += 4 * kAdj) {
      const float4 a = *reinterpret_cast<const float4*>(sm.x + i), b = *reinterpret_cast<const float4*>(sm.dy + i);
      dD += a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w;
    }
  }
  // ---- the band: G = C^ B^^T, dM = dY~ X~^T below the diagonal ------------------------------------------------
  float gm[1][NX][4], dm[1][NX][4];
  zero(gm);
  zero(dm);
  const bool below = n0 < m0 + 16;
  if (below) {
    warp_mma<1, NX, true, true, false, false, N, N, !EX>(gm, sm.c, m0, sm.b, n0, 0, N);
    warp_mma<1, NX, true, true, EX, EX, kP, kP, !EX>(dm, sm.dy, m0, sm.x, n0, 0, kP);
  }
  dcd = adj_sum<kAdj>(dcd, sm.red);   // the states have been read by everyone: M and dG take their place
  dD = adj_sum<kAdj>(dD, sm.red);
  {
    float rowE[2] = {0.0f, 0.0f}, dgp[2] = {0.0f, 0.0f};
    float colE[NX][2], dwE[NX][2];
#pragma unroll
    for (int nt = 0; nt < NX; ++nt) colE[nt][0] = colE[nt][1] = dwE[nt][0] = dwE[nt][1] = 0.0f;
#pragma unroll
    for (int nt = 0; nt < NX; ++nt)
#pragma unroll
      for (int hh = 0; hh < 2; ++hh) {
        const int row = m0 + 8 * hh + g, l = row / R;
        const float ac = ts.ac[l];
        float mv[2], gv[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int s = (n0 + 8 * nt + 2 * q4 + j) / R;
          const float gg = gm[0][nt][2 * hh + j], dd = dm[0][nt][2 * hh + j];
          mv[j] = gv[j] = 0.0f;
          if (s < l) {
            const float raw = ac - ts.ac[s], dec = exp_decay(raw), w = ts.w[s];
            const float e = dd * gg * dec, ei = e * w * clamp_inside(raw);
            mv[j] = gg * w * dec;
            gv[j] = dd * w * dec;
            rowE[hh] += ei;
            colE[nt][j] += ei;
            dwE[nt][j] += e;
          } else if (s == l) {
            mv[j] = gg * ts.g[s];
            gv[j] = dd * ts.g[s];
            dgp[hh] += dd * gg;
          }
        }
        *reinterpret_cast<float2*>(sM + at<kRows>(row, n0 + 8 * nt + 2 * q4)) = make_float2(mv[0], mv[1]);
        *reinterpret_cast<float2*>(sG + at<kRows>(row, n0 + 8 * nt + 2 * q4)) = make_float2(gv[0], gv[1]);
      }
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const float r = quad_sum(rowE[hh]), v = quad_sum(dgp[hh]);
      if (q4 == 0) {
        sm.row[warp >> 2][m0 + 8 * hh + g] = r;
        sm.dg[warp >> 2][m0 + 8 * hh + g] = v;
      }
    }
#pragma unroll
    for (int nt = 0; nt < NX; ++nt)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const float a = group_sum(colE[nt][j]), b = group_sum(dwE[nt][j]);
        if (g == 0) {
          sm.col[warp & 3][n0 + 8 * nt + 2 * q4 + j] = a;
          sm.dw[warp & 3][n0 + 8 * nt + 2 * q4 + j] = b;
        }
      }
  }
  __syncthreads();
  // ---- dX~ += M^T dY~, dB^ += dG^T C^, dC^ += dG B^ (only the triangle's half of each sum) ---------------------
  warp_mma<1, NX, false, false, false, EX, kRows, kP, !EX>(dx, sM, m0, sm.dy, n0, m0, kRows);
  warp_mma<2, NT, false, false, false, false, kRows, N, !EX>(db, sG, M0, sm.c, N0, M0, kRows);
  warp_mma<2, NT, true, false, false, false, kRows, N, !EX>(dc, sG, M0, sm.b, N0, 0, M0 + 32);
  __syncthreads();   // M and dG are spent, and dY~ but for the words that a thread's own share of dX~ replaces
  if constexpr (EX) {
    store_acc<kP>(dx, m0, n0, sm.dy);
  } else {   // float32: the skip's share last, as all that is added behind it is rounded at its size
    for_acc(dx, m0, n0, [&](int row, int col, float& a, float& b) {
      float2* const to = reinterpret_cast<float2*>(sm.dy + at<kP>(row, col));
      *to = make_float2(fmaf(dsk, to->x, a), fmaf(dsk, to->y, b));
    });
  }
  store_acc<N>(db, M0, N0, sDB);
  store_acc<N>(dc, M0, N0, sDC);
  __syncthreads();
  const bool last = c.k == d.C - 1;
  const int l_end = d.T - 1 - c.t0;
  if (last && out.dlu) {   // gradient through last_u = sum_r x (x) B^ at the final token
    const float* gl = out.dlu + (size_t)c.bh * PN;
    for (int e = tid; e < R * (kP + N); e += kAdj) {
      const int r = e / (kP + N), i = e - r * (kP + N), row = l_end * R + r;
      float v = 0.0f;
      if (i < kP) {
        for (int n = 0; n < N; ++n) v += gl[i * N + n] * sm.b[at<N>(row, n)];
        sm.dy[at<kP>(row, i)] += v;
      } else {
        for (int p = 0; p < kP; ++p) v += gl[p * N + i - kP] * sm.x[at<kP>(row, p)];
        sDB[at<N>(row, i - kP)] += v;
      }
    }
    __syncthreads();
  }
  // ---- out: d x; d B, d C rotated back by +phi, and d phi (src/tensor/ops/fused.rs:627-672) ----------------------
  if (out.dx) store_rows<T, R, kP, kAdj>(out.dx, sm.dy, d, c);
  if constexpr (ROT) {
    float* dphi = sm.x;   // [LT][NH]; x is spent (the barrier above)
    constexpr int PER = NH * R / 4, NA = R == 1 ? 4 : (R == 2 ? 2 : 1);
#pragma unroll
    for (int i = 0; i < LT * PER / kAdj; ++i) {
      const int it = tid + i * kAdj, l = it / PER, e = 4 * (it - l * PER), t = c.t0 + l;
      float cs[NA], sn[NA], dp[NA];
#pragma unroll
      for (int j = 0; j < NA; ++j) {
        sincos_wrapped(sm.phi[l * NH + e / R + j], &sn[j], &cs[j]);
        dp[j] = 0.0f;
      }
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const float* gr = w ? sDC : sDB;
        const float* op = w ? sm.c : sm.b;
        float u1[4], u2[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int a1 = at<N>(l * R + (e + j) % R, (e + j) / R), a2 = a1 + NH;   // the swizzle leaves NH's bit alone
          const float g1 = gr[a1], g2 = gr[a2];
          dp[j / R] += g1 * op[a2] - g2 * op[a1];
          u1[j] = g1 * cs[j / R] - g2 * sn[j / R];
          u2[j] = g1 * sn[j / R] + g2 * cs[j / R];
        }
        T* dst = w ? out.dc : out.db;
        if (dst && t < d.T) {
          dst += tok_index(d, c.b, t, c.h) * N * R + e;
          store4(dst, make_float4(u1[0], u1[1], u1[2], u1[3]));
          store4(dst + NH * R, make_float4(u2[0], u2[1], u2[2], u2[3]));
        }
      }
#pragma unroll
      for (int j = 0; j < NA; ++j) {
        const int m = e / R + j;
        float v = t < d.T ? dp[j] : 0.0f;
        if (last && l == l_end && out.dangle) v += out.dangle[(size_t)c.bh * NH + m];
        dphi[l * NH + m] = v;
      }
    }
    __syncthreads();
    // sums over the rest of the chunk, plane by plane
    constexpr int NQ = kAdj / NH < LT ? kAdj / NH : LT, LQ = LT / NQ;
    const int qq = tid / NH, m = tid % NH;
    float loc[LQ], run = 0.0f;
    if (qq < NQ) {
#pragma unroll
      for (int i = LQ - 1; i >= 0; --i) {
        run += dphi[(qq * LQ + i) * NH + m];
        loc[i] = run;
      }
      sm.sq[qq * NH + m] = run;
    }
    __syncthreads();
    if (qq < NQ) {
      float off = 0.0f;
      for (int j = NQ - 1; j > qq; --j) off += sm.sq[j * NH + m];
#pragma unroll
      for (int i = 0; i < LQ; ++i) rw.dphi[((size_t)c.bh * d.Tp + c.t0 + qq * LQ + i) * NH + m] = off + loc[i];
      if (qq == 0) rw.dpsum[((size_t)c.bh * d.C + c.k) * NH + m] = off + run;
    }
  } else {
    if (out.db) store_rows<T, R, N, kAdj>(out.db, sDB, d, c);
    if (out.dc) store_rows<T, R, N, kAdj>(out.dc, sDC, d, c);
  }
  // ---- the scalars' gradients: band, carry-out, chunk-state and chunk-decay terms -----------------------------------
  const float cd = ts.ac[LT - 1];
  if (tid < LT) {
    const int l = tid;
    float rows_ = 0.0f, t1 = 0.0f, q = 0.0f, dgv = 0.0f, col = 0.0f, dwv = 0.0f;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int ro = l * R + r;
#pragma unroll
      for (int i = 0; i < WC; ++i) {
        rows_ += sm.row[i][ro];
        dgv += sm.dg[i][ro];
        q += sm.q[i][ro];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        col += sm.col[i][ro];
        dwv += sm.dw[i][ro];
      }
#pragma unroll
      for (int i = 0; i < WN; ++i) t1 += sm.t1[i][ro];
    }
    const float ac = ts.ac[l], raw = cd - ac, sg = ts.dte[l];
    const float dast = sg * ts.w[l] * q * clamp_inside(raw);
    sm.dac[l] = rows_ - col + ts.eac[l] * clamp_inside(ac) * t1 - dast;
    sm.dast[l] = dast;
    const size_t o = (size_t)c.bh * d.Tp + c.t0 + l;
    out.dw[o] = dwv + sg * q;
    out.dg[o] = dgv;
  }
  __syncthreads();
  if (warp == 0) {   // reverse cumulative sum of d acum, the chunk-decay terms on its last step
    constexpr int EPL = LT >= 32 ? LT / 32 : 1;
    float tail = 0.0f;
    for (int i = lane; i < LT; i += 32) tail += sm.dast[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tail += __shfl_xor_sync(0xffffffffu, tail, o);
    tail += exp_decay(cd) * clamp_inside(cd) * dcd;
    SumOf<T> loc[EPL], run = 0;
#pragma unroll
    for (int i = EPL - 1; i >= 0; --i) {
      const int l = lane * EPL + i;
      if (l < LT) run += (SumOf<T>)sm.dac[l] + (l == LT - 1 ? tail : 0.0f);
      loc[i] = run;
    }
    const SumOf<T> tot = lane_scan<true>(run);
    float pa = 0.0f;
#pragma unroll
    for (int i = 0; i < EPL; ++i) {
      const int l = lane * EPL + i;
      if (l < LT) {
        const float da = (float)(tot - run + loc[i]);
        out.da[(size_t)c.bh * d.Tp + c.t0 + l] = da;
        pa += da * ts.dt[l];
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) pa += __shfl_xor_sync(0xffffffffu, pa, o);
    if (lane == 0) {
      out.part_a[(size_t)c.bh * d.C + c.k] = pa;
      out.part_d[(size_t)c.bh * d.C + c.k] = dD;
    }
  }
}

// ---- rotational dynamics: the later chunks' d phi on top, then per token d theta, d dt and d lambda (the arithmetic of
// kb_final).  A warp per step, lanes over planes; a block per d.L steps, `per_seg` blocks to a segment whose sums of d phi
// are complete within it, `nseg` of those (here the chunks; the tensor-core family's segments are longer).
// Ahead of these rows of blocks (`head_rows`), one block per head for its sums.  A warp requests its next four steps before
// it uses the first (as a loop over steps it waited for each pair of loads), and what the per-token part needs with them:
// float32, 8 x 1024 tokens x 16 heads, d_state 128, 42 -> 25 us; its bytes take 15.  (Eight steps, fewer blocks: 35.)
template <class T, int N>
__global__ void __launch_bounds__(256) k_rows_final(Dims d, m3_scan_desc in, RowsBwdWs rw, GenericBwdWs bw, int has_state,
                                                    T* __restrict__ ddt, T* __restrict__ dlam, T* __restrict__ dtheta,
                                                    float* __restrict__ dangle0, int per_seg, int nseg, HeadSums hs, int head_rows) {
  after_predecessor();
  constexpr int NH = N / 2, NQ = 256 / NH, PL = NH / 32, U = 4;
  __shared__ float s_off[NQ][NH], s_rot[128], red[8];
  if (blockIdx.z || (int)blockIdx.y < head_rows) {
    const int h = (int)blockIdx.y * (int)gridDim.x + (int)blockIdx.x;
    if (h < d.H) head_sums(d, h, hs, bw, red);
    return;
  }
  Chunk c;
  c.k = blockIdx.x; c.bh = blockIdx.y - head_rows;
  c.b = c.bh / d.H; c.h = c.bh - c.b * d.H; c.t0 = c.k * d.L;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const T* dt = static_cast<const T*>(in.dt);
  const T* theta = static_cast<const T*>(in.theta);
  float v[U][PL], th[U][PL], vdt[U];
  auto load = [&](int l0) {   // steps l0, l0 + 8, ...
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int l = l0 + 8 * u, t = c.t0 + l;
      const bool live = l < d.L && t < d.T;
      const size_t ti = live ? theta_index(d, c.b, t, c.h) : 0, o = ((size_t)c.bh * d.Tp + (live ? t : c.t0)) * NH;
      vdt[u] = live ? ldf(dt, tok_index(d, c.b, t, c.h)) : 0.0f;
#pragma unroll
      for (int i = 0; i < PL; ++i) {
        v[u][i] = live ? rw.dphi[o + lane + 32 * i] : 0.0f;
        th[u][i] = live ? ldf(theta, ti + lane + 32 * i) : 0.0f;
      }
    }
  };
  load(warp);
  // what the per-token part at the end needs, requested with the rest
  const int t_own = c.t0 + tid;
  const bool own = tid < d.L && t_own < d.T && (ddt || dlam);
  const size_t o_own = (size_t)c.bh * d.Tp + (own ? t_own : c.t0), i_own = own ? tok_index(d, c.b, t_own, c.h) : 0;
  float own_da = 0.0f, own_gw = 0.0f, own_dwm1 = 0.0f, own_dt = 0.0f, own_lam = 0.0f;
  if (own) {
    own_da = bw.da[o_own];
    own_gw = bw.dg[o_own] + bw.dw[o_own];
    own_dwm1 = t_own > 0 ? bw.dw[o_own - 1] : 0.0f;
    own_dt = ldf(dt, i_own);
    own_lam = lambda_at(static_cast<const T*>(in.lambda), d.disc, i_own);
  }
  {
    const int q = tid / NH, m = tid % NH;
    float s = 0.0f;
#pragma unroll 4
    for (int k = c.k / per_seg + 1 + q; k < nseg; k += NQ) s += rw.dpsum[((size_t)c.bh * nseg + k) * NH + m];
    s_off[q][m] = s;
  }
  __syncthreads();
  float off[PL];
#pragma unroll
  for (int i = 0; i < PL; ++i) {
    off[i] = 0.0f;
#pragma unroll
    for (int q = 0; q < NQ; ++q) off[i] += s_off[q][lane + 32 * i];
    if (c.k == 0 && warp == 0 && dangle0)
      dangle0[(size_t)c.bh * NH + lane + 32 * i] = off[i] + rw.dpsum[(size_t)c.bh * nseg * NH + lane + 32 * i];
  }
  for (int l0 = warp; l0 < d.L; l0 += 8 * U) {
    if (l0 != warp) load(l0);
    float s[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int l = l0 + 8 * u, t = c.t0 + l;
      s[u] = 0.0f;
#pragma unroll
      for (int i = 0; i < PL; ++i) {
        const float g = v[u][i] + off[i];
        s[u] += g * th[u][i];
        if (dtheta && l < d.L && t < d.T) stf(dtheta, theta_index(d, c.b, t, c.h) + lane + 32 * i, g * vdt[u]);
      }
    }
    const float sum = warp_sums<U>(s);
    const int l = l0 + 8 * (lane / (32 / U));
    if (lane % (32 / U) == 0 && l < d.L) s_rot[l] = sum;
  }
  __syncthreads();
  if (own) {
    const float A = -expf(in.a_log[c.h]);
    float vdl = own_gw * own_dt - own_dwm1 * own_dt;
    float vdd = own_da * A + own_gw * own_lam + own_dwm1 * (1.0f - own_lam) + s_rot[tid];
    if (has_state && t_own == 0) {
      const float ip = bw.ip0[c.bh];
      vdl -= own_dt * ip;
      vdd += (1.0f - own_lam) * ip;
    }
    if (ddt) stf(ddt, i_own, vdd);
    if (dlam) stf(dlam, i_own, vdl);
  }
}

template <class T, int N>
cudaError_t final_t(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const RowsBwdWs& rw, const GenericBwdWs& bw, void* ddt,
                    void* dlam, void* dtheta, float* dangle0, int per_seg, int nseg, const HeadSums& hs) {
  const int nx = (d.T + d.L - 1) / d.L, BH = d.B * d.H;
  int rows = hs.any() ? (d.H + nx - 1) / nx : 0;
  const bool layer = BH + rows > 65535;   // (the heads' blocks in a layer of their own where the rows are used up)
  if (layer) rows = 0;
  const dim3 grid(nx, BH + rows, layer ? 2 : 1);
  launch(k_rows_final<T, N>, grid, 256, 0, st, d, in, rw, bw, in.h0 ? 1 : 0, static_cast<T*>(ddt), static_cast<T*>(dlam),
         static_cast<T*>(dtheta), dangle0, per_seg, nseg, hs, rows);
  return cudaGetLastError();
}

template <class T, int N, int R, bool ROT>
cudaError_t backward_t(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const RowsWs& ws, const RowsBwdWs& rw,
                       const GenericBwdWs& bw, const m3_scan_bwd_in& up, uint32_t mask, const m3_scan_grads& g,
                       uint64_t* launches) {
  auto want = [&](uint32_t bit, void* p) { return (mask & bit) ? p : nullptr; };
  const dim3 grid(d.C, d.B * d.H);
  const bool has_state = in.h0 != nullptr;
  uint64_t n = 3;
  cudaError_t e = dh_local(st, d, in, up.dy, ws, rw.dhs);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_rows_adjoint<T, N, R, ROT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(AdjSmem<N, R>));
  if (e != cudaSuccess) return e;
  launch(k_rows_pass_rev<N, ROT>, dim3(32 * (N / 2) / 256, d.B * d.H), 256, 0, st, d, up.dh, ws, rw);
  const AdjOut<T> out{static_cast<T*>(want(M3_GRAD_X, g.dx)), static_cast<T*>(want(M3_GRAD_B, g.db)),
                      static_cast<T*>(want(M3_GRAD_C, g.dc)), bw.da, bw.dg, bw.dw, bw.partA, bw.partD,
                      d.raw ? nullptr : up.dlast_u, up.dangle};
  launch(k_rows_adjoint<T, N, R, ROT>, grid, kAdjThreads<N>, sizeof(AdjSmem<N, R>), st, d, in,
         static_cast<const T*>(up.dy), ws, rw, out);
  if (has_state) {
    launch(k_rows_seed<T, N>, d.B * d.H, 256, 0, st, d, in, rw, bw.ip0, static_cast<float*>(want(M3_GRAD_H0, g.dh0)),
           d.raw ? nullptr : static_cast<float*>(want(M3_GRAD_LAST_U0, g.dlast_u0)));
    n += 1;
  }
  void* ddt = want(M3_GRAD_DT, g.ddt);
  void* dlam = d.disc == M3_LEARNED_TRAPEZOID ? want(M3_GRAD_LAMBDA, g.dlambda) : nullptr;
  float* dalog = d.raw ? nullptr : static_cast<float*>(want(M3_GRAD_A_LOG, g.da_log));
  float* ddsk = in.d_skip ? static_cast<float*>(want(M3_GRAD_D_SKIP, g.dd_skip)) : nullptr;
  if (launches) *launches += n + (ROT ? 1 : 0);
  if (!ROT) return finalize_scalars(st, d, in, bw, ddt, dlam, dalog, ddsk, launches, &g);
  return final_t<T, N>(st, d, in, rw, bw, ddt, dlam, want(M3_GRAD_THETA, g.dtheta),
                       in.angle0 ? static_cast<float*>(want(M3_GRAD_ANGLE0, g.dangle0)) : nullptr, 1, d.C, HeadSums{in.a_log, dalog, ddsk});
}

}  // namespace
}  // namespace rows

cudaError_t rows_final(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const float* dphi, const float* dpsum, int per_seg,
                       int nseg, const GenericBwdWs& bw, void* ddt, void* dlam, void* dtheta, float* dangle0, const HeadSums& hs) {
  const rows::RowsBwdWs rw{nullptr, const_cast<float*>(dphi), const_cast<float*>(dpsum)};
  return rows::final_t<__nv_bfloat16, 128>(st, d, in, rw, bw, ddt, dlam, dtheta, dangle0, per_seg, nseg, hs);
}

size_t rows_bwd_ws_layout(const Dims& d, rows::RowsBwdWs* rw, GenericBwdWs* bw, char* base) {
  size_t off = 0;
  auto take = [&](size_t n) {
    float* p = base ? reinterpret_cast<float*>(base + off) : nullptr;
    off += (n * sizeof(float) + 255) / 256 * 256;
    return p;
  };
  const size_t BH = (size_t)d.B * d.H;
  rows::RowsBwdWs r;
  GenericBwdWs b{};
  r.dhs = take(BH * (d.C + 1) * d.P * d.N);
  r.dphi = take(BH * d.Tp * d.NH);
  r.dpsum = take(BH * d.C * d.NH);
  b.da = take(BH * d.Tp);
  b.dg = take(BH * d.Tp);
  b.dw = take(BH * d.Tp);
  b.partA = take(BH * d.C);
  b.partD = take(BH * d.C);
  b.ip0 = take(BH);
  if (rw) *rw = r;
  if (bw) *bw = b;
  return off;
}

cudaError_t rows_backward(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const rows::RowsWs& ws,
                          const rows::RowsBwdWs& rw, const GenericBwdWs& bw, const m3_scan_bwd_in& up, uint32_t mask,
                          const m3_scan_grads& grads, uint64_t* launches) {
  return rows::dispatch(d, in, [&](auto t, auto n, auto r, auto rot) {
    return rows::backward_t<decltype(t), n.value, r.value, rot.value>(st, d, in, ws, rw, bw, up, mask, grads, launches);
  });
}

}  // namespace m3
