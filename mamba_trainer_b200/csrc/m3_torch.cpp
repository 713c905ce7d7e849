// PyTorch side of the fused nodes, in native code: the scan and the mixer as autograd nodes over the C ABI, and the
// inference window.  What Python did per call - descriptors through ctypes, a Python autograd function each way, a
// gradient buffer at a time - cost 120 us of a scan's forward + backward whose library calls take 26 us; the small calls
// (a 2 x 256-token scan, a decoding step) were bound by it.
// The arithmetic stays in libm3scan; this extension allocates with torch and enqueues on torch's current stream.
#include <ATen/Context.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/record_function.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include <map>
#include <mutex>
#include <optional>
#include <string>

#include "../../include/m3scan.h"

namespace {

using at::Tensor;
using torch::autograd::variable_list;
using OptTensor = c10::optional<Tensor>;

PyObject* g_from_status = nullptr;   // error.from_status

// A context is shared by the threads of a process (autograd runs backward passes on a thread of its own): binding the
// stream, the calls that use it and the reading of their message go together under its lock.  Python code that calls the
// library takes the same lock (ssm/scan.py) and needs the interpreter's to go on, so nobody waits here holding that; a
// thread may take it again (a finaliser that runs in between).
std::recursive_mutex& lock_of(m3_ctx* ctx) {
  static auto* mu = new std::mutex;   // never destroyed: nodes may outlive the statics of a process on its way out
  static auto* locks = new std::map<m3_ctx*, std::recursive_mutex>;
  std::lock_guard<std::mutex> g(*mu);
  return (*locks)[ctx];
}
struct Status {
  int rc = M3_OK;
  std::string message;
};
// One call of the library on the current stream of `t`'s device.
template <class F>
Status locked(m3_ctx* ctx, const Tensor& t, F call) {
  std::optional<py::gil_scoped_release> nogil;
  if (PyGILState_Check()) nogil.emplace();
  std::lock_guard<std::recursive_mutex> lock(lock_of(ctx));
  m3_ctx_set_stream(ctx, c10::cuda::getCurrentCUDAStream(t.device().index()).stream());
  Status s;
  s.rc = call();
  if (s.rc != M3_OK) s.message = m3_last_error(ctx);
  return s;
}

// The library's error as the package's exception class; rethrown across the autograd engine's threads as it is.
[[noreturn]] void raise_status(const Status& s) {
  py::gil_scoped_acquire gil;
  PyObject* exc = PyObject_CallFunction(g_from_status, "is", s.rc, s.message.c_str());
  if (exc) {
    PyErr_SetObject(reinterpret_cast<PyObject*>(Py_TYPE(exc)), exc);
    Py_DECREF(exc);
  }
  python_error e;
  e.persist();
  throw e;
}

const void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
void* mut(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
const float* fptr(const Tensor& t) { return static_cast<const float*>(ptr(t)); }
float* fmut(const Tensor& t) { return static_cast<float*>(mut(t)); }

// Uninitialised memory for results and scratch of one call, straight from the allocator behind at::empty: these calls are the
// larger part of what a small call costs the host (a decoding step makes five of them).  What at::empty does besides is for those
// who watch the dispatcher (modes, profilers) and for the fill that torch's deterministic algorithms ask for: they get at::empty
// itself.
class Fresh {
 public:
  Fresh()
      : watched_(c10::impl::TorchDispatchModeTLS::any_modes_set() || at::hasCallbacks() ||
                 (at::globalContext().deterministicAlgorithms() && at::globalContext().deterministicFillUninitializedMemory())) {}
  Tensor operator()(at::IntArrayRef sizes, at::ScalarType el, const Tensor& device_of) const {
    if (watched_) return at::empty(sizes, at::TensorOptions().dtype(el).device(device_of.device()));
    return Tensor(at::detail::empty_cuda(sizes, el, device_of.device(), c10::nullopt));
  }
  Tensor like(const Tensor& t) const { return (*this)(t.sizes(), t.scalar_type(), t); }
  Tensor bytes(size_t n, const Tensor& device_of) const { return (*this)({static_cast<int64_t>(n)}, at::kByte, device_of); }

 private:
  bool watched_;
};

Tensor as(const Tensor& t, at::ScalarType el) {
  if (!t.defined()) return t;
  return t.scalar_type() == el && t.is_contiguous() ? t : t.to(el).contiguous();
}
Tensor as(const OptTensor& t, at::ScalarType el) { return t.has_value() ? as(*t, el) : Tensor(); }

// A tensor of the forward pass for the backward pass: saved the way autograd saves one, so saved-tensor hooks (activation
// checkpointing, offloading) may drop it and give back another.  Backward passes take every address from what unpack()
// returns, which has the forward's element type, density and alignment modulo 16 bytes (the library chose kernels and
// layouts by them).
struct Saved {
  torch::autograd::SavedVariable var;
  at::ScalarType el{};
  c10::Device device{c10::kCPU};
  int64_t numel = 0, align = 0;
  bool present = false;

  void set(const Tensor& t) {
    if (!t.defined()) return;
    var = torch::autograd::SavedVariable(t, false);
    el = t.scalar_type(); device = t.device(); numel = t.numel();
    align = reinterpret_cast<uintptr_t>(t.data_ptr()) % 16;
    present = true;
  }
  Tensor unpack(std::shared_ptr<torch::autograd::Node> node) const {   // refuses a second pass unless the graph is retained
    if (!present) return Tensor();
    const Tensor v = var.unpack(std::move(node));
    TORCH_CHECK(v.numel() == numel, "a saved tensor came back with ", v.numel(), " elements instead of ", numel);
    if (fits(v)) return v;
    at::NoGradGuard no_grad;
    const Tensor t = as(v.to(device), el);
    if (fits(t)) return t;
    const int64_t es = t.element_size();   // (an allocation starts on 16 bytes)
    return at::empty({numel + 16 / es}, t.options()).narrow(0, align / es, numel).view(t.sizes()).copy_(t);
  }
  bool fits(const Tensor& t) const {
    return t.scalar_type() == el && t.device() == device && t.is_contiguous() &&
           static_cast<int64_t>(reinterpret_cast<uintptr_t>(t.data_ptr()) % 16) == align;
  }
};
// The nodes have no forward-mode rule: an input with a tangent is refused, as torch refuses it for a Python node without one.
void refuse_tangents(const Tensor* t, int n) {
  for (int i = 0; i < n; ++i)
    TORCH_CHECK_NOT_IMPLEMENTED(!t[i].defined() || !t[i]._fw_grad(0).defined(),
                                "forward-mode AD is not implemented for the fused scan and mixer");
}
int dtype_code(const Tensor& t) { return t.scalar_type() == at::kBFloat16 ? M3_BF16 : M3_F32; }

// ---- the scan -----------------------------------------------------------------------------------------------------
constexpr int kScanInputs = 11;   // x, b, c, dt, a_log, lambda, theta, d_skip, h0, last_u0, angle0: the bits of grad_mask
void scan_inputs(m3_scan_desc& d, const Tensor (&t)[kScanInputs]) {
  d.x = ptr(t[0]); d.b = ptr(t[1]); d.c = ptr(t[2]); d.dt = ptr(t[3]); d.a_log = fptr(t[4]); d.lambda = ptr(t[5]);
  d.theta = ptr(t[6]); d.d_skip = fptr(t[7]); d.h0 = fptr(t[8]); d.last_u0 = fptr(t[9]); d.angle0 = fptr(t[10]);
}
struct ScanNode : public torch::autograd::Node {
  m3_ctx* ctx = nullptr;
  m3_saved* handle = nullptr;
  m3_scan_desc desc{};   // extents and options
  Saved in[kScanInputs];
  bool has_state = false, has_angle = false;

  ~ScanNode() override { free_handle(); }
  void free_handle() {
    if (!handle) return;
    m3_saved_free(ctx, handle);   // (on the stream that the handle remembers: no lock)
    handle = nullptr;
  }
  void release_variables() override {
    for (auto& v : in) v.var.reset_data();
    free_handle();
  }
  std::string name() const override { return "Mamba3ScanBackward"; }

  variable_list apply(variable_list&& up) override {
    Tensor t[kScanInputs], g[kScanInputs];
    for (int i = 0; i < kScanInputs; ++i) t[i] = in[i].unpack(shared_from_this());
    m3_scan_desc d = desc;
    scan_inputs(d, t);
    uint32_t mask = 0;
    const Fresh fresh;
    for (int i = 0; i < kScanInputs; ++i)
      if (in[i].present && task_should_compute_output(i)) {
        g[i] = fresh.like(t[i]);
        mask |= 1u << i;
      }
    auto dense = [](const Tensor& v) { return v.defined() ? v.contiguous() : v; };
    const Tensor dy = up[0].defined() ? up[0].contiguous() : at::zeros_like(t[0]);
    const Tensor dh = has_state ? dense(up[1]) : Tensor(), du = has_state ? dense(up[2]) : Tensor();
    const Tensor da = has_angle ? dense(up[3]) : Tensor();
    const m3_scan_bwd_in bin{ptr(dy), fptr(dh), fptr(du), fptr(da)};
    m3_scan_grads out{};
    out.dx = mut(g[0]); out.db = mut(g[1]); out.dc = mut(g[2]); out.ddt = mut(g[3]); out.da_log = fmut(g[4]);
    out.dlambda = mut(g[5]); out.dtheta = mut(g[6]); out.dd_skip = fmut(g[7]);
    out.dh0 = fmut(g[8]); out.dlast_u0 = fmut(g[9]); out.dangle0 = fmut(g[10]);
    const Status s = locked(ctx, t[0], [&] { return m3_scan_backward_moved(ctx, handle, &d, &bin, mask, &out); });
    if (s.rc != M3_OK) raise_status(s);
    return variable_list(g, g + kScanInputs);
  }
};

// Inputs as the caller has them (checked by the caller): converted to x's element type, parameters and states to float32.
std::vector<OptTensor> scan(uintptr_t handle, const Tensor& x0, const Tensor& b0, const Tensor& c0, const Tensor& dt0,
                            const Tensor& a_log0, const OptTensor& lam0, const OptTensor& theta0, const OptTensor& d_skip0,
                            const OptTensor& h00, const OptTensor& lu00, const OptTensor& ang00, int chunk, int disc, bool want_state,
                            int path, int rev) {
  m3_ctx* ctx = reinterpret_cast<m3_ctx*>(handle);
  const auto el = x0.scalar_type();
  const Tensor t[kScanInputs] = {as(x0, el), as(b0, el), as(c0, el), as(dt0, el), as(a_log0, at::kFloat), as(lam0, el),
                                 as(theta0, el), as(d_skip0, at::kFloat), as(h00, at::kFloat), as(lu00, at::kFloat),
                                 as(ang00, at::kFloat)};
  refuse_tangents(t, kScanInputs);
  const Tensor& x = t[0];
  const int64_t B = x.size(0), T = x.size(1), H = x.size(2), P = x.size(3), R = x.size(4), N = t[1].size(3);
  m3_scan_desc d{};
  d.batch = B; d.seq = T; d.heads = H; d.head_dim = P; d.d_state = N; d.rank = R; d.chunk = chunk; d.dtype = dtype_code(x);
  d.discretization = disc; d.dynamics = t[6].defined() ? M3_ROTATIONAL : M3_REAL; d.want_state = want_state; d.path = path;
  d.reverse_heads = rev;
  scan_inputs(d, t);
  const Fresh fresh;
  Tensor y = fresh.like(x), h, lu, ang;
  if (want_state) {
    h = fresh({B, H, P, N}, at::kFloat, x);
    lu = fresh({B, H, P, N}, at::kFloat, x);
    if (t[6].defined()) ang = fresh({B, H, N / 2}, at::kFloat, x);
  }
  bool track = false;
  if (at::GradMode::is_enabled())
    for (const Tensor& v : t) track = track || (v.defined() && v.requires_grad());
  const m3_scan_out out{mut(y), fmut(h), fmut(lu), fmut(ang)};
  m3_saved* saved = nullptr;
  const Status s = locked(ctx, x, [&] { return m3_scan_forward(ctx, &d, &out, track ? &saved : nullptr); });
  if (s.rc != M3_OK) raise_status(s);
  if (track) {
    std::shared_ptr<ScanNode> node(new ScanNode(), torch::autograd::deleteNode);
    node->ctx = ctx;
    node->handle = saved;
    node->desc = d;
    node->set_next_edges(torch::autograd::collect_next_edges(t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], t[9], t[10]));
    for (int i = 0; i < kScanInputs; ++i) node->in[i].set(t[i]);
    node->has_state = want_state;
    node->has_angle = ang.defined();
    variable_list outs{y};
    if (want_state) { outs.push_back(h); outs.push_back(lu); }
    if (ang.defined()) outs.push_back(ang);
    torch::autograd::set_history(outs, node);
  }
  auto opt = [](const Tensor& v) { return v.defined() ? OptTensor(v) : OptTensor(); };
  return {y, opt(h), opt(lu), opt(ang)};
}

// ---- the mixer ----------------------------------------------------------------------------------------------------
constexpr int kMixerParams = 9, kNormWeight = 7, kPostWeight = 8;   // in the order of m3_mixer_desc
struct Spec {   // the integers of m3_mixer_desc between its extents and its pointers
  int heads, head_dim, d_state, rank, groups, chunk, disc, rotational, has_norm, post_norm, path, reverse_heads;
};
void mixer_inputs(m3_mixer_desc& d, const Tensor& proj, const Tensor* p) {
  d.proj = ptr(proj);
  d.conv_weight = fptr(p[0]); d.conv_bias = fptr(p[1]); d.dt_bias = fptr(p[2]); d.a_log = fptr(p[3]); d.d_skip = fptr(p[4]);
  d.b_bias = fptr(p[5]); d.c_bias = fptr(p[6]); d.norm_weight = fptr(p[7]); d.post_weight = fptr(p[8]);
}
m3_mixer_desc mixer_desc(const Tensor& proj, const Tensor (&p)[kMixerParams], const Spec& s, double eps) {
  m3_mixer_desc d{};
  d.batch = proj.size(0); d.seq = proj.size(1);
  d.heads = s.heads; d.head_dim = s.head_dim; d.d_state = s.d_state; d.rank = s.rank; d.groups = s.groups; d.chunk = s.chunk;
  d.dtype = dtype_code(proj); d.discretization = s.disc; d.dynamics = s.rotational ? M3_ROTATIONAL : M3_REAL;
  d.conv_kernel = p[0].size(0); d.has_norm = s.has_norm; d.post_norm = s.post_norm; d.path = s.path;
  d.reverse_heads = s.reverse_heads; d.eps = static_cast<float>(eps);
  mixer_inputs(d, proj, p);
  return d;
}
Spec spec_of(const std::vector<int64_t>& v) {
  TORCH_CHECK(v.size() == 12, "a mixer is described by 12 integers");
  return Spec{(int)v[0], (int)v[1], (int)v[2], (int)v[3], (int)v[4], (int)v[5],
              (int)v[6], (int)v[7], (int)v[8], (int)v[9], (int)v[10], (int)v[11]};
}

struct MixerNode : public torch::autograd::Node {
  m3_ctx* ctx = nullptr;
  m3_saved* handle = nullptr;
  m3_mixer_desc desc{};    // extents and options
  Tensor act;
  Saved in[1 + kMixerParams];   // proj, then the parameters

  ~MixerNode() override { free_handle(); }
  void free_handle() {
    if (!handle) return;
    m3_saved_free(ctx, handle);   // (on the stream that the handle remembers: no lock)
    handle = nullptr;
  }
  void release_variables() override {
    for (auto& v : in) v.var.reset_data();
    free_handle();
    act = Tensor();
  }
  std::string name() const override { return "Mamba3MixerBackward"; }

  variable_list apply(variable_list&& up) override {
    variable_list g(1 + kMixerParams);
    Tensor t[1 + kMixerParams];
    for (int i = 0; i <= kMixerParams; ++i) t[i] = in[i].unpack(shared_from_this());
    if (!up[0].defined()) return g;
    m3_mixer_desc d = desc;
    mixer_inputs(d, t[0], t + 1);
    const Tensor dout = up[0].contiguous();
    // (a gain whose norm was switched off is read by nothing: no gradient)
    const Fresh fresh;
    for (int i = 0; i <= kMixerParams; ++i)
      if (in[i].present && (i != 1 + kNormWeight || d.has_norm) && (i != 1 + kPostWeight || d.post_norm))
        g[i] = fresh.like(t[i]);
    const m3_mixer_grads out{mut(g[0]), fmut(g[1]), fmut(g[2]), fmut(g[3]), fmut(g[4]), fmut(g[5]),
                             fmut(g[6]), fmut(g[7]), fmut(g[8]), fmut(g[9])};
    const Tensor work = fresh.bytes(m3_mixer_backward_bytes(&d), act);
    const Status s = locked(ctx, t[0], [&] { return m3_mixer_backward(ctx, &d, handle, ptr(act), ptr(dout), &out, mut(work)); });
    if (s.rc != M3_OK) raise_status(s);
    return g;
  }
};

Tensor mixer(uintptr_t handle, const Tensor& proj0, const std::vector<OptTensor>& params, const std::vector<int64_t>& ints,
             double eps, int64_t d_inner) {
  m3_ctx* ctx = reinterpret_cast<m3_ctx*>(handle);
  TORCH_CHECK(params.size() == kMixerParams, "a mixer has ", kMixerParams, " parameters");
  const Tensor proj = proj0.contiguous();
  Tensor p[kMixerParams];
  for (int i = 0; i < kMixerParams; ++i) p[i] = as(params[i], at::kFloat);
  refuse_tangents(&proj, 1);
  refuse_tangents(p, kMixerParams);
  const m3_mixer_desc d = mixer_desc(proj, p, spec_of(ints), eps);
  const Fresh fresh;
  Tensor out = fresh({proj.size(0), proj.size(1), d_inner}, proj.scalar_type(), proj);
  const Tensor act = fresh.bytes(m3_mixer_activation_bytes(&d), proj);
  bool track = false;
  if (at::GradMode::is_enabled()) {
    track = proj.requires_grad();
    for (const Tensor& v : p) track = track || (v.defined() && v.requires_grad());
  }
  m3_saved* saved = nullptr;
  const Status s = locked(ctx, proj, [&] { return m3_mixer_forward(ctx, &d, mut(out), mut(act), track ? &saved : nullptr); });
  if (s.rc != M3_OK) raise_status(s);
  if (track) {
    std::shared_ptr<MixerNode> node(new MixerNode(), torch::autograd::deleteNode);
    node->ctx = ctx;
    node->handle = saved;
    node->desc = d;
    node->act = act;
    node->in[0].set(proj);
    for (int i = 0; i < kMixerParams; ++i) node->in[1 + i].set(p[i]);
    node->set_next_edges(torch::autograd::collect_next_edges(proj, p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], p[8]));
    torch::autograd::set_history(out, node);
  }
  return out;
}

// Inference with a carried cache: (out, new history, h, last_u, angle or None).
std::vector<OptTensor> window(uintptr_t handle, const Tensor& proj0, const std::vector<OptTensor>& params,
                              const std::vector<int64_t>& ints, double eps, int64_t d_inner, const Tensor& conv0, const Tensor& h0,
                              const Tensor& lu0, const OptTensor& ang0) {
  at::NoGradGuard no_grad;
  m3_ctx* ctx = reinterpret_cast<m3_ctx*>(handle);
  TORCH_CHECK(params.size() == kMixerParams, "a mixer has ", kMixerParams, " parameters");
  const Tensor proj = proj0.contiguous();
  Tensor p[kMixerParams];
  for (int i = 0; i < kMixerParams; ++i) p[i] = as(params[i], at::kFloat);
  const Spec s = spec_of(ints);
  const m3_mixer_desc d = mixer_desc(proj, p, s, eps);
  const Tensor conv = as(conv0, proj.scalar_type()), h = as(h0, at::kFloat), lu = as(lu0, at::kFloat);
  const Tensor ang = s.rotational ? as(ang0, at::kFloat) : Tensor();
  const Fresh fresh;
  const Tensor out = fresh({proj.size(0), proj.size(1), d_inner}, proj.scalar_type(), proj), conv2 = fresh.like(conv);
  const Tensor h2 = fresh.like(h), lu2 = fresh.like(lu);
  Tensor ang2;
  if (s.rotational) ang2 = fresh({proj.size(0), s.heads, s.d_state / 2}, at::kFloat, proj);
  const m3_mixer_window_io io{ptr(conv), fptr(h), fptr(lu), fptr(ang), mut(out), mut(conv2), fmut(h2), fmut(lu2), fmut(ang2)};
  const size_t bytes = m3_mixer_window_bytes(&d, &io);
  Tensor work;
  if (bytes) work = fresh.bytes(bytes, proj);
  const Status done = locked(ctx, proj, [&] { return m3_mixer_window(ctx, &d, &io, mut(work)); });
  if (done.rc != M3_OK) raise_status(done);
  return {out, conv2, h2, lu2, ang2.defined() ? OptTensor(ang2) : OptTensor()};
}

}  // namespace

PYBIND11_MODULE(_m3torch, m) {
  m.def("set_from_status", [](py::object f) { g_from_status = f.release().ptr(); });
  auto of = [](uintptr_t handle) -> std::recursive_mutex& { return lock_of(reinterpret_cast<m3_ctx*>(handle)); };
  m.def("lock", [of](uintptr_t handle) { of(handle).lock(); }, py::call_guard<py::gil_scoped_release>());
  m.def("unlock", [of](uintptr_t handle) { of(handle).unlock(); });
  m.def("scan", &scan);
  m.def("mixer", &mixer);
  m.def("window", &window);
}
