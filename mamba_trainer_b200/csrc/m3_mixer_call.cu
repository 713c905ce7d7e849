// The mixer between its two projections as ONE call of the library (Mamba3Mixer::project / finish around
// mamba3_scan, src/models/mamba3.rs:340-461, :475-560): the steps of m3_conv.cu, m3_mixer.cu and the scan enqueued
// back to back by native code.  A decoding step used to spend 145 us of host time in Python on seven calls whose
// kernels take 37 us together; a window of one position is one launch now (k_step_rows).
#include "m3_front.h"
#include "m3_internal.h"
#include "m3_step.h"

namespace m3 {
namespace {

// Widths and column offsets of the projection's bands.
struct MixerDims {
  int di, bc, conv, width, off_dt, off_lam, off_th;
  bool learned, rot;
  size_t es, tok;
};

int mixer_dims(m3_ctx* ctx, const m3_mixer_desc* s, MixerDims* m) {
  if (!ctx) return M3_ERR_NULL;
  if (!s) return fail(ctx, M3_ERR_NULL, "a descriptor is required");
  if (s->batch <= 0 || s->seq <= 0 || s->heads <= 0 || s->head_dim <= 0 || s->d_state <= 0 || s->rank <= 0 || s->groups <= 0)
    return fail(ctx, M3_ERR_SHAPE, "mixer: extents must be positive");
  if (s->heads % s->groups) return fail(ctx, M3_ERR_CONFIG, "heads %d not a multiple of groups %d", s->heads, s->groups);
  if (s->dtype != M3_F32 && s->dtype != M3_BF16) return fail(ctx, M3_ERR_UNSUPPORTED, "dtype %d", s->dtype);
  if (!s->proj || !s->conv_weight || !s->a_log) return fail(ctx, M3_ERR_NULL, "proj, conv_weight and a_log are required");
  if (s->conv_kernel < 1 || s->conv_kernel > 8) return fail(ctx, M3_ERR_UNSUPPORTED, "conv_kernel %d outside [1, 8]", s->conv_kernel);
  m->learned = s->discretization == M3_LEARNED_TRAPEZOID;
  m->rot = s->dynamics == M3_ROTATIONAL;
  m->di = s->heads * s->head_dim * s->rank;
  m->bc = s->groups * s->d_state * s->rank;
  m->conv = m->di + 2 * m->bc;
  m->off_dt = 2 * m->di + 2 * m->bc;
  m->off_lam = m->off_dt + s->heads;
  m->off_th = m->off_lam + (m->learned ? s->heads : 0);
  m->width = m->off_th + (m->rot ? s->heads * (s->d_state / 2) : 0);
  m->es = s->dtype == M3_BF16 ? 2 : 4;
  m->tok = (size_t)s->batch * s->seq;
  return M3_OK;
}

const char* at(const void* p, size_t elems, size_t es) { return static_cast<const char*>(p) + elems * es; }

// The steps in front of the scan as one launch (m3_front.cu), where it serves the shape; else the convolution, the
// B / C steps and the activations one after the other, with the convolution's B C half in a buffer of its own.
Front front_of(const m3_mixer_desc* s, const MixerDims& m) {
  Front f{};
  f.B = s->batch; f.T = s->seq; f.H = s->heads; f.N = s->d_state; f.R = s->rank; f.K = s->conv_kernel;
  f.di = m.di; f.bc = m.bc; f.width = m.width; f.off_dt = m.off_dt; f.off_lam = m.off_lam;
  f.reverse = s->reverse_heads ? 1 : 0; f.has_norm = s->has_norm ? 1 : 0; f.eps = s->eps;
  f.proj = s->proj; f.conv_w = s->conv_weight; f.conv_b = s->conv_bias; f.b_bias = s->b_bias; f.c_bias = s->c_bias;
  f.gain = s->norm_weight; f.dt_bias = s->dt_bias;
  return f;
}
bool one_front(const m3_mixer_desc* s, const MixerDims& m, const void* hist = nullptr, const void* new_hist = nullptr) {
  Front f = front_of(s, m);
  f.hist = hist;
  return s->groups == s->heads && front_supported(s->dtype, f, new_hist, nullptr, nullptr);
}

// Intermediate results of a window or of a forward pass, laid out in one workspace.
struct MixerWs {
  char *x, *bcr, *b, *c, *dt, *lam, *y, *theta;
};
// theta is read from its band of the projection - unless the tensor-core family would serve the shape but for the band
// not starting on 16 bytes (it moves theta by bulk tensor copies): then it is copied once.
bool theta_copied(const m3_mixer_desc* s, const MixerDims& m) {
  return m.rot && s->dtype == M3_BF16 && s->head_dim == 64 && s->d_state == 128 && (s->rank == 1 || s->rank == 2 || s->rank == 4) &&
         s->path != M3_PATH_GENERIC && (m.width % 8 || (reinterpret_cast<uintptr_t>(s->proj) + 2 * (size_t)m.off_th) % 16);
}
cudaError_t copy_theta(m3_ctx* ctx, const m3_mixer_desc* s, const MixerDims& m, void* dst, size_t dst_pitch, const void* src,
                       size_t src_pitch) {
  return cudaMemcpy2DAsync(dst, dst_pitch, src, src_pitch, (size_t)s->heads * (s->d_state / 2) * m.es, m.tok,
                           cudaMemcpyDeviceToDevice, ctx->stream);
}
size_t mixer_ws(const m3_mixer_desc* s, const MixerDims& m, MixerWs* w, void* base, const void* hist = nullptr,
                const void* new_hist = nullptr) {
  size_t off = 0;
  auto take = [&](size_t elems) {
    char* p = base ? static_cast<char*>(base) + off : nullptr;
    off += (elems * m.es + 255) / 256 * 256;
    return p;
  };
  const size_t hn = (size_t)s->heads * s->d_state * s->rank;
  MixerWs t;
  t.x = take(m.tok * m.di);
  t.bcr = one_front(s, m, hist, new_hist) ? nullptr : take(m.tok * 2 * m.bc);
  t.b = take(m.tok * hn);
  t.c = take(m.tok * hn);
  t.dt = take(m.tok * s->heads);
  t.lam = m.learned ? take(m.tok * s->heads) : nullptr;
  t.y = take(m.tok * m.di);
  t.theta = theta_copied(s, m) ? take(m.tok * s->heads * (s->d_state / 2)) : nullptr;
  if (w) *w = t;
  return off;
}

// Descriptors of the steps, over the projection's bands and the workspace.
struct MixerSteps {
  m3_conv_desc conv{};
  m3_bc_desc bc{};
  m3_act_desc act{};
  m3_scan_desc scan{};
  m3_gate_desc gate{};
  m3_gate_norm_desc gate_norm{};
};
void mixer_steps(const m3_mixer_desc* s, const MixerDims& m, const MixerWs& w, MixerSteps* t) {
  m3_conv_desc& c = t->conv;
  c.batch = s->batch; c.seq = s->seq; c.channels = m.conv; c.kernel_size = s->conv_kernel; c.dtype = s->dtype; c.activation = 1;
  c.x_stride = m.width; c.y_stride = m.di; c.x = at(s->proj, m.di, m.es);
  c.weight = s->conv_weight; c.bias = s->conv_bias;
  c.split = m.di; c.y2_stride = 2 * m.bc; c.y2 = w.bcr;
  if (s->reverse_heads) {
    // direction-major bands (mamba3.rs:352-370): the second half of x, of B and of C belongs to the heads that walk
    // right to left; their convolution runs right to left as well
    const int lo[3] = {m.di / 2, m.di + m.bc / 2, m.di + m.bc + m.bc / 2}, hi[3] = {m.di, m.di + m.bc, m.di + 2 * m.bc};
    c.n_reversed = 3;
    for (int i = 0; i < 3; ++i) { c.reversed_lo[i] = lo[i]; c.reversed_hi[i] = hi[i]; }
  }
  m3_bc_desc& b = t->bc;
  b.batch = s->batch; b.seq = s->seq; b.heads = s->heads; b.groups = s->groups; b.d_state = s->d_state; b.rank = s->rank;
  b.dtype = s->dtype; b.has_norm = s->has_norm; b.eps = s->eps; b.raw_stride = 2 * m.bc;
  b.b_raw = w.bcr; b.c_raw = w.bcr + (size_t)m.bc * m.es;
  b.b_bias = s->b_bias; b.c_bias = s->c_bias; b.norm_weight = s->norm_weight;
  m3_act_desc& a = t->act;
  a.batch = s->batch; a.seq = s->seq; a.heads = s->heads; a.dtype = s->dtype; a.stride = m.width;
  a.dt_raw = at(s->proj, m.off_dt, m.es);
  a.lambda_raw = m.learned ? at(s->proj, m.off_lam, m.es) : nullptr;
  a.dt_bias = s->dt_bias;
  m3_scan_desc& k = t->scan;
  k.batch = s->batch; k.seq = s->seq; k.heads = s->heads; k.head_dim = s->head_dim; k.d_state = s->d_state; k.rank = s->rank;
  k.chunk = s->chunk; k.dtype = s->dtype; k.discretization = s->discretization; k.dynamics = s->dynamics; k.path = s->path;
  k.reverse_heads = s->reverse_heads;
  k.x = w.x; k.b = w.b; k.c = w.c; k.dt = w.dt; k.lambda = w.lam;
  k.a_log = s->a_log; k.d_skip = s->d_skip;
  if (m.rot) {
    k.theta = w.theta ? w.theta : at(s->proj, m.off_th, m.es);
    k.theta_stride = w.theta ? 0 : m.width;
  }
  m3_gate_desc& g = t->gate;
  g.batch = s->batch; g.seq = s->seq; g.channels = m.di; g.dtype = s->dtype; g.z_stride = m.width; g.y = w.y; g.z = s->proj;
  m3_gate_norm_desc& n = t->gate_norm;
  n.batch = s->batch; n.seq = s->seq; n.channels = m.di; n.dtype = s->dtype; n.z_stride = m.width; n.y = w.y; n.z = s->proj;
  n.weight = s->post_weight; n.eps = s->eps;
}

#define M3_TRY(call)                 \
  do {                               \
    const int rc_ = (call);          \
    if (rc_ != M3_OK) return rc_;    \
  } while (0)

// Everything in front of the scan: x, B, C, dt, lambda into the workspace.
int run_front(m3_ctx* ctx, const m3_mixer_desc* s, const MixerDims& m, const MixerWs& w, MixerSteps& t, const void* hist,
              void* new_hist) {
  if (w.theta) {
    const cudaError_t e = copy_theta(ctx, s, m, w.theta, (size_t)s->heads * (s->d_state / 2) * m.es,
                                     at(s->proj, m.off_th, m.es), (size_t)m.width * m.es);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "theta");
  }
  if (one_front(s, m, hist, new_hist)) {
    cudaError_t e = cudaSetDevice(ctx->device);
    Front f = front_of(s, m);
    f.hist = hist;
    if (e == cudaSuccess) e = front_forward(ctx->stream, s->dtype, f, FrontOut{w.x, w.b, w.c, w.dt, w.lam, new_hist}, &ctx->launches);
    return e == cudaSuccess ? M3_OK : cuda_fail(ctx, e, "mixer front");
  }
  t.conv.history = hist;
  M3_TRY(m3_conv_forward(ctx, &t.conv, w.x, new_hist));
  M3_TRY(m3_bc_forward(ctx, &t.bc, w.b, w.c));
  return m3_dt_lambda_forward(ctx, &t.act, w.dt, w.lam);
}

int run_gate(m3_ctx* ctx, const m3_mixer_desc* s, const MixerSteps& t, void* out) {
  return s->post_norm ? m3_gate_norm_forward(ctx, &t.gate_norm, out) : m3_gate_forward(ctx, &t.gate, out);
}

// Gradients on their way through a backward pass.
struct MixerBwdWs {
  char *dy, *dx, *db, *dc, *ddt, *dlam, *dbcr, *dtheta;
  float* part;
};
size_t mixer_bwd_ws(const m3_mixer_desc* s, const MixerDims& m, MixerBwdWs* w, void* base) {
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* p = base ? static_cast<char*>(base) + off : nullptr;
    off += (bytes + 255) / 256 * 256;
    return p;
  };
  const size_t hn = (size_t)s->heads * s->d_state * s->rank, row = m.tok * m.es;
  const bool front = one_front(s, m);
  MixerBwdWs t;
  t.dy = take(row * m.di);
  t.dx = take(row * m.di);
  t.db = take(row * hn);
  t.dc = take(row * hn);
  t.ddt = take(row * s->heads);
  t.dlam = m.learned ? take(row * s->heads) : nullptr;
  t.dbcr = front ? nullptr : take(row * 2 * m.bc);
  t.dtheta = theta_copied(s, m) ? take(row * s->heads * (s->d_state / 2)) : nullptr;
  t.part = front ? reinterpret_cast<float*>(take(front_part_floats(front_of(s, m)) * sizeof(float))) : nullptr;
  if (w) *w = t;
  return off;
}

bool one_launch(const m3_mixer_desc* s, const m3_mixer_window_io* io) {
  return s->seq == 1 && step_rows_supported(s->head_dim, s->d_state, s->rank,
                                            {io->h_in, io->last_u_in, io->h_out, io->last_u_out});
}

}  // namespace
}  // namespace m3

using namespace m3;

extern "C" {

size_t m3_mixer_window_bytes(const m3_mixer_desc* s, const m3_mixer_window_io* io) {
  MixerDims m;
  m3_ctx scratch;  // messages go nowhere: the call itself reports them
  if (!s || !io || mixer_dims(&scratch, s, &m) != M3_OK) return 0;
  if (one_launch(s, io) && !s->post_norm) return 0;
  return mixer_ws(s, m, nullptr, nullptr, io->conv_in, io->conv_out);
}

int m3_mixer_window(m3_ctx* ctx, const m3_mixer_desc* s, const m3_mixer_window_io* io, void* workspace) {
  MixerDims m;
  M3_TRY(mixer_dims(ctx, s, &m));
  M3_TRY(take_device_flag(ctx, "in an earlier call, seen on entry to m3_mixer_window"));
  if (!io || !io->h_in || !io->last_u_in || !io->out || !io->h_out || !io->last_u_out)
    return fail(ctx, M3_ERR_NULL, "the state, the output and the new state's buffers are required");
  if (s->conv_kernel > 1 && (!io->conv_in || !io->conv_out)) return fail(ctx, M3_ERR_NULL, "the convolution's history is required");
  if (s->reverse_heads) return fail(ctx, M3_ERR_UNSUPPORTED, "a bidirectional mixer has no causal state to carry");
  if (m.rot && !io->angle_out) return fail(ctx, M3_ERR_NULL, "rotational dynamics carry an angle");
  MixerWs w;
  const bool step = one_launch(s, io);
  if (!(step && !s->post_norm) && !workspace) return fail(ctx, M3_ERR_NULL, "a workspace is required");
  mixer_ws(s, m, &w, workspace, io->conv_in, io->conv_out);
  m3_step_desc sd{};
  sd.batch = s->batch; sd.heads = s->heads; sd.head_dim = s->head_dim; sd.d_state = s->d_state; sd.rank = s->rank;
  sd.dtype = s->dtype; sd.discretization = s->discretization; sd.dynamics = s->dynamics;
  sd.a_log = s->a_log; sd.d_skip = s->d_skip; sd.h = io->h_in; sd.last_u = io->last_u_in; sd.angle = m.rot ? io->angle_in : nullptr;
  m3_step_out so{w.y, io->h_out, io->last_u_out, m.rot ? io->angle_out : nullptr};
  MixerSteps t;
  if (step) {
    cudaError_t e = cudaSetDevice(ctx->device);
    if (e == cudaSuccess) {
      MixerStep f{};
      f.proj = s->proj; f.width = m.width; f.d_inner = m.di; f.bc = m.bc; f.conv_channels = m.conv; f.K = s->conv_kernel;
      f.PG = s->heads / s->groups; f.off_dt = m.off_dt; f.off_lam = m.off_lam; f.off_theta = m.off_th;
      f.has_norm = s->has_norm; f.eps = s->eps; f.conv_in = io->conv_in; f.conv_out = io->conv_out;
      f.conv_w = s->conv_weight; f.conv_b = s->conv_bias; f.dt_bias = s->dt_bias; f.b_bias = s->b_bias; f.c_bias = s->c_bias;
      f.norm_w = s->norm_weight;
      f.out = s->post_norm ? nullptr : io->out;
      e = mixer_step(ctx, sd, so, f);
    }
    if (e != cudaSuccess) return cuda_fail(ctx, e, "mixer step");
    ctx->launches += 1;
    if (!s->post_norm) return M3_OK;
    mixer_steps(s, m, w, &t);
    return m3_gate_norm_forward(ctx, &t.gate_norm, io->out);
  }
  mixer_steps(s, m, w, &t);
  M3_TRY(run_front(ctx, s, m, w, t, io->conv_in, io->conv_out));
  if (s->seq == 1) {
    sd.x = w.x; sd.b = w.b; sd.c = w.c; sd.dt = w.dt; sd.lambda = w.lam;
    sd.theta = t.scan.theta;   // one batch row's heads are dense; more than one row would need the band's stride
    float* dense = nullptr;
    if (m.rot && s->batch > 1 && !w.theta) {
      const size_t row = (size_t)s->heads * (s->d_state / 2) * m.es;
      cudaError_t e = scratch_alloc(ctx, reinterpret_cast<void**>(&dense), row * s->batch, ctx->stream);
      if (e == cudaSuccess)
        e = cudaMemcpy2DAsync(dense, row, sd.theta, (size_t)m.width * m.es, row, s->batch, cudaMemcpyDeviceToDevice, ctx->stream);
      if (e != cudaSuccess) {
        if (dense) cudaFreeAsync(dense, ctx->stream);
        return cuda_fail(ctx, e, "theta of the step");
      }
      sd.theta = dense;
    }
    const int rc = m3_step_forward(ctx, &sd, &so);
    if (dense) cudaFreeAsync(dense, ctx->stream);
    if (rc != M3_OK) return rc;
  } else {
    t.scan.want_state = 1;
    t.scan.h0 = io->h_in; t.scan.last_u0 = io->last_u_in; t.scan.angle0 = m.rot ? io->angle_in : nullptr;
    const m3_scan_out out{w.y, io->h_out, io->last_u_out, m.rot ? io->angle_out : nullptr};
    M3_TRY(m3_scan_forward(ctx, &t.scan, &out, nullptr));
  }
  return run_gate(ctx, s, t, io->out);
}

size_t m3_mixer_activation_bytes(const m3_mixer_desc* s) {
  MixerDims m;
  m3_ctx scratch;
  return s && mixer_dims(&scratch, s, &m) == M3_OK ? mixer_ws(s, m, nullptr, nullptr) : 0;
}

size_t m3_mixer_backward_bytes(const m3_mixer_desc* s) {
  MixerDims m;
  m3_ctx scratch;
  return s && mixer_dims(&scratch, s, &m) == M3_OK ? mixer_bwd_ws(s, m, nullptr, nullptr) : 0;
}

int m3_mixer_forward(m3_ctx* ctx, const m3_mixer_desc* s, void* out, void* activations, m3_saved** saved) {
  if (saved) *saved = nullptr;
  MixerDims m;
  M3_TRY(mixer_dims(ctx, s, &m));
  if (!out || !activations) return fail(ctx, M3_ERR_NULL, "the output and the activations' memory are required");
  MixerWs w;
  MixerSteps t;
  mixer_ws(s, m, &w, activations);
  mixer_steps(s, m, w, &t);
  M3_TRY(run_front(ctx, s, m, w, t, nullptr, nullptr));
  const m3_scan_out so{w.y, nullptr, nullptr, nullptr};
  M3_TRY(m3_scan_forward(ctx, &t.scan, &so, saved));
  const int rc = run_gate(ctx, s, t, out);
  if (rc != M3_OK && saved && *saved) {
    m3_saved_free(ctx, *saved);
    *saved = nullptr;
  }
  return rc;
}

int m3_mixer_backward(m3_ctx* ctx, const m3_mixer_desc* s, const m3_saved* saved, const void* activations, const void* dout,
                      const m3_mixer_grads* g, void* workspace) {
  MixerDims m;
  M3_TRY(mixer_dims(ctx, s, &m));
  if (!saved || !activations || !dout || !g || !g->dproj || !workspace)
    return fail(ctx, M3_ERR_NULL, "saved context, activations, dout, dproj and a workspace are required");
  MixerWs w;
  MixerSteps t;
  MixerBwdWs b;
  mixer_ws(s, m, &w, const_cast<void*>(activations));
  mixer_steps(s, m, w, &t);
  mixer_bwd_ws(s, m, &b, workspace);
  auto band = [&](size_t col) { return static_cast<char*>(g->dproj) + col * m.es; };
  // every band of dproj is written exactly once: z by the gate, theta by the scan, x | B C, dt and lambda in front of it
  if (s->post_norm) M3_TRY(m3_gate_norm_backward(ctx, &t.gate_norm, dout, b.dy, g->dproj, g->dpost_weight));
  else M3_TRY(m3_gate_backward(ctx, &t.gate, dout, b.dy, g->dproj));
  m3_scan_bwd_in in{};
  in.dy = b.dy;
  m3_scan_grads sg{};
  sg.dx = b.dx; sg.db = b.db; sg.dc = b.dc; sg.ddt = b.ddt; sg.dlambda = b.dlam;
  sg.dtheta = b.dtheta ? b.dtheta : (m.rot ? band(m.off_th) : nullptr);
  sg.da_log = g->da_log; sg.dd_skip = g->dd_skip;
  M3_TRY(m3_scan_backward_moved(ctx, saved, &t.scan, &in, M3_GRAD_ALL, &sg));
  if (b.dtheta) {
    const cudaError_t e = copy_theta(ctx, s, m, band(m.off_th), (size_t)m.width * m.es, b.dtheta,
                                     (size_t)s->heads * (s->d_state / 2) * m.es);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "d theta");
  }
  if (one_front(s, m)) {
    const FrontGrads fg{b.dx, b.db, b.dc, b.ddt, b.dlam, g->dproj, g->dconv_weight, g->dconv_bias, g->db_bias, g->dc_bias,
                        g->dnorm_weight, g->ddt_bias, b.part};
    const cudaError_t e = front_backward(ctx->stream, s->dtype, front_of(s, m), fg, &ctx->launches);
    return e == cudaSuccess ? M3_OK : cuda_fail(ctx, e, "mixer front backward");
  }
  M3_TRY(m3_dt_lambda_backward(ctx, &t.act, b.ddt, b.dlam, band(m.off_dt), m.learned ? band(m.off_lam) : nullptr, g->ddt_bias));
  M3_TRY(m3_bc_backward(ctx, &t.bc, b.db, b.dc, b.dbcr, b.dbcr + (size_t)m.bc * m.es, g->db_bias, g->dc_bias, g->dnorm_weight));
  t.conv.dy2 = b.dbcr;
  return m3_conv_backward(ctx, &t.conv, b.dx, band(m.di), g->dconv_weight, g->dconv_bias, nullptr);
}

}  // extern "C"
