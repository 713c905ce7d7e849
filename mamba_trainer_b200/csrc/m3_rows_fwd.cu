// Forward of the chunk-parallel family (m3_rows.cuh): three launches.
//   k_rows_state  per chunk: scalars, angles within the chunk, S_k = X~^T diag(sw) B^ with B rotated by the angle
//                 since the chunk's start
//   k_rows_pass   sequential over chunks, parallel over state elements: H_{k+1} = exp(cd_k) H_k + Rot(S_k); the state
//                 and the angle entering every chunk (a rotation by the entering angle commutes with the sum over the
//                 chunk's rows, so no pass over the sequence is needed before the states are built)
//   k_rows_out    per chunk: Y = (C~ B~^T o band) X~ + exp(acum) C~ H_k^T + D x
// Nothing but the chunk states (N * 64 floats per 64 rows) goes through global memory in between: rows of B, C and x
// are read and rotated where they are used.  float32, batch 8 x 1024 tokens x 16 heads, d_state 128, rotational: the
// generic family's seven launches took 1.20 ms.
// References: src/ssm/scan.rs:458-618 over :116-291, as restated in m3_generic_fwd.cu.
#include "m3_rows.cuh"

namespace m3 {
namespace rows {
namespace {

// ---- S_k (forward) or the local part of dH_k (backward: (exp(acum) dY~)^T C^, the same product with other rows) ---
template <int N, int R>
struct StateSmem {
  float b[kRows * N], x[kRows * kP], phi[(kRows / R) * (N / 2)], q[256];
  Scal<R> s;
};
template <class T, int N, int R, bool ROT, bool BWD>
__global__ void __launch_bounds__(256, N == 64 ? 4 : 3) k_rows_state(Dims d, m3_scan_desc in, const T* __restrict__ dy, RowsWs ws,
                                                    float* __restrict__ dst) {
  after_predecessor();
  extern __shared__ __align__(16) unsigned char smem[];
  StateSmem<N, R>& sm = *reinterpret_cast<StateSmem<N, R>*>(smem);
  constexpr int NH = N / 2;
  const Chunk c = this_chunk(d);
  load_rows<T, R, kP, 256>(sm.x, BWD ? dy : static_cast<const T*>(in.x), d, c);
  chunk_scalars<T, R>(sm.s, d, c, in);
  const float* scale = BWD ? sm.s.eac : sm.s.sw;
  const T* rows_in = static_cast<const T*>(BWD ? in.c : in.b);
  if constexpr (ROT) {
    chunk_angles<T, N, R, 256>(sm.phi, sm.q, sm.s, d, c, static_cast<const T*>(in.theta), nullptr, [&](int m, float sum) {
      if (!BWD) ws.asum[((size_t)c.bh * d.C + c.k) * NH + m] = sum;
    });
    __syncthreads();
    float* const to[1] = {sm.b};
    const T* const from[1] = {rows_in};
    load_rotated<T, N, R, 256, 1>(to, from, sm.phi, scale, d, c);
  } else {
    load_scaled<T, N, R, 256>(sm.b, rows_in, scale, d, c);
  }
  if (!BWD && threadIdx.x == 0) ws.cd[(size_t)c.bh * d.C + c.k] = sm.s.ac[kRows / R - 1];
  __syncthreads();
  constexpr bool EX = sizeof(T) == 2;   // x and dy of a bf16 tensor are exact in TF32
  constexpr int NT = N / 32;
  const int warp = threadIdx.x >> 5, m0 = 32 * (warp & 1), n0 = 8 * NT * (warp >> 1);
  float acc[2][NT][4];
  zero(acc);
  warp_mma<2, NT, false, false, EX, false, kP, N, !EX>(acc, sm.x, m0, sm.b, n0, 0, kRows);
  store_acc<N>(acc, m0, n0, dst + ((size_t)c.bh * (BWD ? d.C + 1 : d.C) + c.k) * kP * N);
}

// ---- the pass over chunk states: a thread owns planes (m, m + NH) of two rows p, p + 32 --------------------------
template <class T, int N, bool ROT>
__global__ void __launch_bounds__(256) k_rows_pass(Dims d, m3_scan_desc in, RowsWs ws, float* h_out) {   // (h_out may be h0)
  after_predecessor();
  constexpr int NH = N / 2, PN = kP * N, U = 4;
  const int bh = blockIdx.y, b = bh / d.H, h = bh - b * d.H;
  const int id = blockIdx.x * 256 + threadIdx.x, m = id % NH, p = id / NH;   // p < 32
  const int o[4] = {at<N>(p, m), at<N>(p, m) + NH, at<N>(p + 32, m), at<N>(p + 32, m) + NH};
  const int plain[4] = {p * N + m, p * N + m + NH, (p + 32) * N + m, (p + 32) * N + m + NH};
  float carry[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  if (in.h0) {
    float first = 0.0f;
    if (in.last_u0 && !d.raw) {   // the seed of scan.rs:524-535
      const size_t i0 = tok_index(d, b, 0, h);
      first = (1.0f - lambda_at(static_cast<const T*>(in.lambda), d.disc, i0)) * ldf(static_cast<const T*>(in.dt), i0);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      carry[i] = in.h0[(size_t)bh * PN + plain[i]];
      if (in.last_u0 && !d.raw) carry[i] += first * in.last_u0[(size_t)bh * PN + plain[i]];
    }
  }
  float ang = ROT && in.angle0 ? wrap_angle(in.angle0[(size_t)bh * NH + m]) : 0.0f;
  float* hs = ws.hs + (size_t)bh * d.C * PN;
  for (int k0 = 0; k0 < d.C; k0 += U) {
    float s[U][4], ecd[U], da[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {   // U chunks are requested before the first is used: the chain is in the carry only
      const size_t k = min(k0 + u, d.C - 1);
#pragma unroll
      for (int i = 0; i < 4; ++i) s[u][i] = hs[k * PN + o[i]];
      ecd[u] = ws.cd[(size_t)bh * d.C + k];
      da[u] = ROT ? ws.asum[((size_t)bh * d.C + k) * NH + m] : 0.0f;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (k0 + u >= d.C) break;
      const size_t k = k0 + u;
      float sn = 0.0f, cs = 1.0f;
      if (ROT) {
        sincos_wrapped(ang, &sn, &cs);
        if (p == 0) ws.abase[((size_t)bh * d.C + k) * NH + m] = ang;
        ang = wrap_angle(ang + da[u]);
      }
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
  if (h_out) {
#pragma unroll
    for (int i = 0; i < 4; ++i) h_out[(size_t)bh * PN + plain[i]] = carry[i];
  }
}

// ---- outputs of a chunk ------------------------------------------------------------------------------------------
// 97 KB of shared memory at d_state 128, so two CTAs share an SM: the state takes the buffer of B once C B^T is done
// (its loads are in registers meanwhile), M that of the angles, y that of M.
template <int N, int R>
struct OutSmem {
  float c[kRows * N], b[kRows * N], x[kRows * kP];
  union {
    float m[kRows * kP];
    float phi[(kRows / R) * (N / 2)];
  };
  float q[256];
  Scal<R> s;
};
template <class T, int N, int R, bool ROT>
__global__ void __launch_bounds__(256, N == 64 ? 3 : 2) k_rows_out(Dims d, m3_scan_desc in, RowsWs ws, T* __restrict__ y,
                                                     float* __restrict__ last_u, float* __restrict__ angle_out) {
  after_predecessor();
  extern __shared__ __align__(16) unsigned char smem[];
  OutSmem<N, R>& sm = *reinterpret_cast<OutSmem<N, R>*>(smem);
  constexpr int NH = N / 2, PN = kP * N;
  constexpr bool EX = sizeof(T) == 2;
  const Chunk c = this_chunk(d);
  const int tid = threadIdx.x, warp = tid >> 5;
  load_rows<T, R, kP, 256>(sm.x, static_cast<const T*>(in.x), d, c);
  chunk_scalars<T, R>(sm.s, d, c, in);
  if constexpr (ROT) {
    if (angle_out && c.k == d.C - 1 && tid < NH) {   // (not in the pass, whose blocks all read an angle0 it may replace)
      const size_t o = ((size_t)c.bh * d.C + c.k) * NH + tid;
      angle_out[(size_t)c.bh * NH + tid] = wrap_angle(ws.abase[o] + ws.asum[o]);
    }
    chunk_angles<T, N, R, 256>(sm.phi, sm.q, sm.s, d, c, static_cast<const T*>(in.theta),
                               ws.abase + ((size_t)c.bh * d.C + c.k) * NH, [](int, float) {});
    __syncthreads();
    float* const to[2] = {sm.b, sm.c};
    const T* const from[2] = {static_cast<const T*>(in.b), static_cast<const T*>(in.c)};
    load_rotated<T, N, R, 256, 2>(to, from, sm.phi, nullptr, d, c);
  } else {
    load_rows<T, R, N, 256>(sm.b, static_cast<const T*>(in.b), d, c);
    load_rows<T, R, N, 256>(sm.c, static_cast<const T*>(in.c), d, c);
  }
  float4 hreg[PN / 1024];
  const float4* hk = reinterpret_cast<const float4*>(ws.hs + ((size_t)c.bh * d.C + c.k) * PN);
#pragma unroll
  for (int i = 0; i < PN / 1024; ++i) hreg[i] = hk[tid + 256 * i];
  __syncthreads();
  if (last_u && c.k == d.C - 1) {   // sum_r x_{T-1}^(r) (x) B^_{T-1}^(r)   (scan.rs:621-638)
    const int l = d.T - 1 - c.t0;
    for (int e = tid; e < PN; e += 256) {
      const int p = e / N, n = e % N;
      float v = 0.0f;
#pragma unroll
      for (int r = 0; r < R; ++r) v += sm.x[at<kP>(l * R + r, p)] * sm.b[at<N>(l * R + r, n)];
      last_u[(size_t)c.bh * PN + e] = v;
    }
  }
  // G = C~ B~^T below the diagonal, M = G o band
  const int m0 = 32 * (warp & 1), n0 = 16 * (warp >> 1);
  {
    float g[2][2][4];
    zero(g);
    if (n0 < m0 + 32) warp_mma<2, 2, true, true, false, false, N, N, !EX>(g, sm.c, m0, sm.b, n0, 0, N);
    for_acc(g, m0, n0, [&](int row, int col, float& a, float& b) {
      const int l = row / R;
      const float ac = sm.s.ac[l];
      float v[2] = {a, b};
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int s = (col + j) / R;
        v[j] *= s < l ? sm.s.w[s] * exp_decay(ac - sm.s.ac[s]) : (s == l ? sm.s.g[s] : 0.0f);
      }
      *reinterpret_cast<float2*>(sm.m + at<kP>(row, col)) = make_float2(v[0], v[1]);
    });
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < PN / 1024; ++i) reinterpret_cast<float4*>(sm.b)[tid + 256 * i] = hreg[i];
  __syncthreads();
  // Y = exp(acum) C~ H^T + M X~
  float acc[2][2][4];
  zero(acc);
  warp_mma<2, 2, true, true, false, false, N, N, !EX>(acc, sm.c, m0, sm.b, n0, 0, N);
  for_acc(acc, m0, n0, [&](int row, int, float& a, float& b) {
    const float e = sm.s.eac[row / R];
    a *= e;
    b *= e;
  });
  warp_mma<2, 2, true, false, false, EX, kP, kP, !EX>(acc, sm.m, m0, sm.x, n0, 0, m0 + 32);
  __syncthreads();   // M is spent: its buffer stages y
  const float dsk = in.d_skip ? in.d_skip[c.h] : 0.0f;
  for_acc(acc, m0, n0, [&](int row, int col, float& a, float& b) {
    const float2 xv = *reinterpret_cast<const float2*>(sm.x + at<kP>(row, col));
    *reinterpret_cast<float2*>(sm.m + at<kP>(row, col)) = make_float2(fmaf(dsk, xv.x, a), fmaf(dsk, xv.y, b));
  });
  __syncthreads();
  store_rows<T, R, kP, 256>(y, sm.m, d, c);
}

template <class K>
cudaError_t smem_limit(K kern, size_t bytes) {
  return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <class T, int N, int R, bool ROT>
cudaError_t forward_t(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const m3_scan_out& out, const RowsWs& ws) {
  const dim3 grid(d.C, d.B * d.H);
  cudaError_t e = smem_limit(k_rows_state<T, N, R, ROT, false>, sizeof(StateSmem<N, R>));
  if (e == cudaSuccess) e = smem_limit(k_rows_out<T, N, R, ROT>, sizeof(OutSmem<N, R>));
  if (e != cudaSuccess) return e;
  launch(k_rows_state<T, N, R, ROT, false>, grid, 256, sizeof(StateSmem<N, R>), st, d, in, nullptr, ws, ws.hs);
  launch(k_rows_pass<T, N, ROT>, dim3(32 * (N / 2) / 256, d.B * d.H), 256, 0, st, d, in, ws,
         in.want_state ? out.h : nullptr);
  launch(k_rows_out<T, N, R, ROT>, grid, 256, sizeof(OutSmem<N, R>), st, d, in, ws, static_cast<T*>(out.y),
         in.want_state && !d.raw ? out.last_u : nullptr, in.want_state ? out.angle : nullptr);
  return cudaGetLastError();
}

template <class T, int N, int R>
cudaError_t load_t() {
  return load_kernels(k_rows_state<T, N, R, true, false>, k_rows_state<T, N, R, false, false>, k_rows_pass<T, N, true>,
                      k_rows_pass<T, N, false>, k_rows_out<T, N, R, true>, k_rows_out<T, N, R, false>);
}
template <class T>
cudaError_t load_all() {
  cudaError_t e = cudaSuccess;
  for (cudaError_t (*f)() : {load_t<T, 64, 1>, load_t<T, 64, 2>, load_t<T, 64, 4>, load_t<T, 128, 1>, load_t<T, 128, 2>, load_t<T, 128, 4>})
    if (e == cudaSuccess) e = f();
  return e;
}

template <class T, int N, int R, bool ROT>
cudaError_t dh_local_t(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const void* dy, const RowsWs& ws, float* dhs) {
  cudaError_t e = smem_limit(k_rows_state<T, N, R, ROT, true>, sizeof(StateSmem<N, R>));
  if (e != cudaSuccess) return e;
  launch(k_rows_state<T, N, R, ROT, true>, dim3(d.C, d.B * d.H), 256, sizeof(StateSmem<N, R>), st, d, in,
         static_cast<const T*>(dy), ws, dhs);
  return cudaGetLastError();
}

}  // namespace

// First launch of the backward pass: local dH_k of every chunk into slot k of dhs.
cudaError_t dh_local(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const void* dy, const RowsWs& ws, float* dhs) {
  return dispatch(d, in, [&](auto t, auto n, auto r, auto rot) {
    return dh_local_t<decltype(t), n.value, r.value, rot.value>(st, d, in, dy, ws, dhs);
  });
}

}  // namespace rows

// Vector accesses of 4 elements: every tensor and theta-free row start aligned to that.  A caller who names the generic family
// gets it.
bool rows_supported(const m3_scan_desc& s, const void* y) {
  if (s.path == M3_PATH_GENERIC) return false;
  if (s.head_dim != rows::kP || (s.d_state != 64 && s.d_state != 128) || (s.rank != 1 && s.rank != 2 && s.rank != 4)) return false;
  const uintptr_t a = s.dtype == M3_F32 ? 15 : 7;
  for (const void* p : {s.x, s.b, s.c, y})
    if (reinterpret_cast<uintptr_t>(p) & a) return false;
  return s.seq > 0;
}

Dims rows_dims(Dims d) {
  d.L = rows::kRows / d.R;
  d.C = (d.T + d.L - 1) / d.L;
  d.Tp = d.C * d.L;
  d.LR = rows::kRows;
  return d;
}

size_t rows_ws_layout(const Dims& d, rows::RowsWs* ws, char* base) {
  size_t off = 0;
  auto take = [&](size_t n) {
    float* p = base ? reinterpret_cast<float*>(base + off) : nullptr;
    off += (n * sizeof(float) + 255) / 256 * 256;
    return p;
  };
  const size_t chunks = (size_t)d.B * d.H * d.C;
  rows::RowsWs t;
  t.hs = take(chunks * d.P * d.N);
  t.asum = take(chunks * d.NH);
  t.abase = take(chunks * d.NH);
  t.cd = take(chunks);
  if (ws) *ws = t;
  return off;
}

cudaError_t rows_load(int dtype) { return dtype == M3_BF16 ? rows::load_all<__nv_bfloat16>() : rows::load_all<float>(); }

cudaError_t rows_forward(cudaStream_t st, const Dims& d, const m3_scan_desc& in, const m3_scan_out& out,
                         const rows::RowsWs& ws, uint64_t* launches) {
  if (launches) *launches += 3;
  return rows::dispatch(d, in, [&](auto t, auto n, auto r, auto rot) {
    return rows::forward_t<decltype(t), n.value, r.value, rot.value>(st, d, in, out, ws);
  });
}

}  // namespace m3
