"""The autograd nodes around the library (csrc/m3_torch.cpp, ssm/scan.py): what torch may do to a node between its
forward and its backward pass, and to the module that holds the parameters."""
import pytest
import torch

from mamba_trainer_b200.nn import MixerCore, MixerShape
from mamba_trainer_b200.ssm import ScanInputs, mamba3_scan, ssd_chunked

pytestmark = pytest.mark.gpu


def _scan_case(dtype, head_dim, d_state, T=200):
    """(function of leaves, leaves, upstream gradient); the scan's own inputs are intermediate results."""
    g = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    B, H, R = 1, 2, 1
    leaves = [r(B, T, H, head_dim, R).to(dtype), (r(B, T, H, d_state, R) / d_state ** 0.5).to(dtype),
              (r(B, T, H, d_state, R) / d_state ** 0.5).to(dtype), (0.05 + 0.1 * r(B, T, H).abs()).to(dtype), r(H).abs(),
              torch.sigmoid(r(B, T, H)).to(dtype), r(B, T, H, d_state // 2).to(dtype), r(H)]

    def f(*v):
        x, b, c, dt, a_log, lam, theta, d_skip = (t * 0.5 for t in v)
        return mamba3_scan(ScanInputs.new(x, b, c, dt, a_log, lam).with_theta(theta).with_skip(d_skip).with_chunk_size(64)).y
    return f, leaves, r(B, T, H, head_dim, R).to(dtype)


def _ssd_case():
    g = torch.Generator(device="cuda").manual_seed(2)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    leaves = [r(2, 50, 2, 16), r(2, 50, 2, 24), r(2, 50, 2, 24), -r(2, 50, 2).abs(), r(2, 50, 2), r(2, 50, 2), r(2, 2, 16, 24)]
    return (lambda *v: ssd_chunked(*(t * 0.5 for t in v), chunk_size=16)[0]), leaves, r(2, 50, 2, 16)


def _mixer_case(dtype, head_dim=64, d_state=128, T=200):
    shape = MixerShape(2, head_dim, d_state, 1)
    torch.manual_seed(3)
    core = MixerCore(shape, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(4)
    proj = torch.randn(2, T, shape.in_proj_width, device="cuda", generator=g).to(dtype)
    names = [n for n, _ in core.named_parameters()]

    def f(p, *params):
        return torch.func.functional_call(core, {n: q * 0.5 for n, q in zip(names, params)}, (p * 0.5,))
    return f, [proj] + [q.detach().clone() for q in core.parameters()], \
        torch.randn(2, T, shape.d_inner, device="cuda", generator=g).to(dtype)


CASES = {
    "scan_tensor_core": lambda: _scan_case(torch.bfloat16, 64, 128),
    "scan_chunk_parallel": lambda: _scan_case(torch.float32, 64, 64),
    "scan_generic": lambda: _scan_case(torch.float32, 24, 40),
    "ssd": _ssd_case,
    "mixer_bf16": lambda: _mixer_case(torch.bfloat16),
    "mixer_f32": lambda: _mixer_case(torch.float32),
    "mixer_f32_separate_steps": lambda: _mixer_case(torch.float32, 24, 40),
}


def _gradients(f, leaves, dout, around=None, apply=None):
    leaves = [t.clone().requires_grad_(True) for t in leaves]
    if around is None:
        out = (apply or (lambda fn, *a: fn(*a)))(f, *leaves)
    else:
        with around:
            out = f(*leaves)
    # whatever the forward pass let go of is taken over by others before the backward pass runs
    junk = [torch.full((n,), float("nan"), device="cuda") for n in (64, 1024, 16384, 1 << 18, 1 << 20) for _ in range(12)]
    grads = torch.autograd.grad(out, leaves, dout)
    del junk
    return (out.detach(),) + grads


@pytest.mark.parametrize("how", ["checkpoint", "offload", "moved"])
@pytest.mark.parametrize("case", CASES)
def test_gradients_under_saved_tensor_hooks(case, how):
    """Activation checkpointing and offloading drop what a node saved and bring back other tensors - in `moved`, at another
    alignment: the adjoint reads those, and the gradients are the plain run's."""
    from torch.utils.checkpoint import checkpoint
    f, leaves, dout = CASES[case]()
    want = _gradients(f, leaves, dout)
    if how == "checkpoint":
        got = _gradients(f, leaves, dout, apply=lambda fn, *a: checkpoint(fn, *a, use_reentrant=False))
    elif how == "offload":
        got = _gradients(f, leaves, dout, torch.autograd.graph.save_on_cpu())
    else:
        def unpack(t):
            return torch.empty(t.numel() + 3, dtype=t.dtype, device="cuda")[3:].view(t.shape).copy_(t)
        got = _gradients(f, leaves, dout, torch.autograd.graph.saved_tensors_hooks(lambda t: t.detach().cpu().contiguous(), unpack))
    for i, (a, e) in enumerate(zip(got, want)):
        assert torch.equal(a, e), (i, float((a.float() - e.float()).abs().max()))


def test_moved_inputs_are_checked():
    """The C entry that takes the inputs' new addresses refuses another shape, another alignment and an absent input."""
    import ctypes as C
    from mamba_trainer_b200 import _ffi
    from mamba_trainer_b200.ssm import Context
    ctx = Context.for_device(torch.device("cuda"))
    B, T, H, P, N = 1, 70, 2, 24, 40
    n = {"x": B * T * H * P, "b": B * T * H * N, "c": B * T * H * N, "dt": B * T * H, "lambda_": B * T * H, "a_log": H}
    t = {k: torch.rand(v + 4, device="cuda") for k, v in n.items()}
    at = lambda off: {k: C.c_void_p(v.data_ptr() + 4 * off) for k, v in t.items()}
    make = lambda off=0, **kw: _ffi.ScanDesc(**{**dict(batch=B, seq=T, heads=H, head_dim=P, d_state=N, rank=1, chunk=16,
                                                       discretization=2), **at(off), **kw})
    y, saved = torch.empty(n["x"], device="cuda"), C.c_void_p()
    ctx.check(ctx.lib.m3_scan_forward(ctx.handle, C.byref(make()), C.byref(_ffi.ScanOut(y=C.c_void_p(y.data_ptr()))), C.byref(saved)))
    dx = torch.empty_like(y)
    run = lambda d: ctx.lib.m3_scan_backward_moved(ctx.handle, saved, C.byref(d), C.byref(_ffi.ScanBwdIn(dy=C.c_void_p(y.data_ptr()))),
                                                   _ffi.GRAD_X, C.byref(_ffi.ScanGrads(dx=C.c_void_p(dx.data_ptr()))))
    assert run(make()) == _ffi.OK
    assert run(make(heads=1)) == _ffi.ERR_CONFIG
    assert run(make(off=1)) == _ffi.ERR_UNSUPPORTED
    assert run(make(lambda_=None)) == _ffi.ERR_NULL
    ctx.check(ctx.lib.m3_saved_free(ctx.handle, saved))


@pytest.mark.parametrize("head_dim,d_state", [(64, 64), (24, 40)])
def test_switched_off_norms_have_no_gradient(head_dim, d_state):
    """A norm that is switched off on a built module leaves its gain out of the graph: no gradient (not memory that nothing
    wrote), and the other gradients are those of a module built without it."""
    kw = dict(chunk=16, device="cuda")
    shape = MixerShape(2, head_dim, d_state, 1)
    torch.manual_seed(0)
    off, without = MixerCore(shape, post_gate_norm=True, **kw), MixerCore(shape, bc_norm=False, **kw)
    without.load_state_dict({k: v for k, v in off.state_dict().items() if k not in ("norm_w", "post_norm_w")})
    off.use_norm = off.post_gate_norm = False
    proj = torch.randn(2, 50, shape.in_proj_width, device="cuda")
    for core in (off, without):
        core(proj).square().sum().backward()
    assert off.norm_w.grad is None and off.post_norm_w.grad is None
    for n, q in without.named_parameters():
        assert torch.equal(q.grad, getattr(off, n).grad), n


def test_threads_with_streams_of_their_own():
    """Native nodes, with their backward passes on autograd's threads, and the calls that go through ctypes, from threads
    with streams of their own: each call's launches stay on its thread's stream, behind that stream's writes of its inputs."""
    import threading
    from mamba_trainer_b200.nn import causal_conv1d
    from mamba_trainer_b200.ssm import SsmState, mamba3_step
    cases = [_scan_case(torch.bfloat16, 64, 128), _scan_case(torch.float32, 64, 64), _ssd_case(), _mixer_case(torch.float32)]
    g = torch.Generator(device="cuda").manual_seed(5)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    one = [r(4, 2, 64, 1), r(4, 2, 64, 1), r(4, 2, 64, 1), r(4, 2).abs(), torch.sigmoid(r(4, 2)), r(2).abs(), None, None]
    state, img, w = (r(4, 2, 64, 64), r(4, 2, 64, 64)), r(4, 300, 96), r(4, 96)
    step = lambda *v: mamba3_step(*v, None, None, SsmState(*state))[0]
    work = [lambda c=c: _gradients_alone(*c) for c in cases]
    work += [lambda: (step(*(t * 1.0 for t in one[:6])),), lambda: (causal_conv1d(img * 1.0, w),)]
    want = [f() for f in work]
    torch.cuda.synchronize()
    failed = []

    def loop(f, expected):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(40):
                got = f()
                torch.cuda.current_stream().synchronize()
                if not all(torch.equal(a, e) for a, e in zip(got, expected)):
                    failed.append(f)
                    return
    threads = [threading.Thread(target=loop, args=(f, e)) for f, e in zip(work, want)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed


def _gradients_alone(f, leaves, dout):
    leaves = [t.clone().requires_grad_(True) for t in leaves]
    out = f(*leaves)
    return (out.detach(),) + torch.autograd.grad(out, leaves, dout)


@pytest.mark.filterwarnings("ignore")
def test_traced_calls_compute():
    """torch.jit.trace records a call of the node, not the buffers that the traced run happened to fill: other inputs give
    their own results and gradients."""
    for case in ("scan_tensor_core", "scan_chunk_parallel"):
        f, leaves, dout = CASES[case]()
        traced = torch.jit.trace(f, tuple(t.clone().requires_grad_(True) for t in leaves), check_trace=False)
        other = [t * 0.75 for t in leaves]
        for a, e in zip(_gradients_alone(traced, other, dout), _gradients_alone(f, other, dout)):
            assert torch.equal(a, e), case
    shape = MixerShape(2, 64, 128, 1)
    core = MixerCore(shape, device="cuda")
    proj, dout = torch.randn(2, 70, shape.in_proj_width, device="cuda"), torch.randn(2, 70, shape.d_inner, device="cuda")
    traced = torch.jit.trace(core, (proj,), check_trace=False)
    for a, e in zip(_gradients_alone(traced, [proj + 1], dout), _gradients_alone(core, [proj + 1], dout)):
        assert torch.equal(a, e)


@pytest.mark.parametrize("kind,dtype,d_state,T,rank", [
    ("step", torch.bfloat16, 128, 1, 2),       # more than three blocks per SM: with the prefetch of later blocks' inputs
    ("window", torch.bfloat16, 128, 900, 1),   # the front, states of segments side by side, the stripes, the gate
    ("window", torch.float32, 64, 90, 1),
    ("mixer", torch.bfloat16, 128, 500, 2),    # segments side by side each way
    ("mixer", torch.float32, 128, 130, 1),
    ("mixer", torch.bfloat16, 64, 200, 1),
])
def test_captured_calls_replay(kind, dtype, d_state, T, rank):
    """A graph of an inference window or a training step, whose launches are programmatic edges there, computes what the
    calls do - from the values its inputs hold when it is replayed."""
    from mamba_trainer_b200.nn import MixerCache
    from mamba_trainer_b200.ssm import SsmState
    heads, B = (32, 16) if kind == "step" else (4, 2)
    if d_state == 128 and dtype == torch.bfloat16 and T > 1:
        from tests._util import segments
        from tests.test_scan_gpu import tc_workload
        assert max(segments(tc_workload(rank, True, T, B, heads))) < -1
    shape = MixerShape(heads, 64, d_state, rank)
    torch.manual_seed(7)
    core = MixerCore(shape, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(8)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)
    proj, other = (r(B, T, shape.in_proj_width).to(dtype) for _ in range(2))
    if kind == "mixer":
        dout, leaves = r(B, T, shape.d_inner).to(dtype), [proj.requires_grad_(True)] + list(core.parameters())

        def run():
            y = core(proj)
            return (y.detach(),) + torch.autograd.grad(y, leaves, dout)
    else:
        cache = MixerCache(r(B, 3, shape.conv_channels).to(dtype), SsmState(r(B, heads, 64, d_state), r(B, heads, 64, d_state),
                                                                            r(B, heads, d_state // 2)))

        def run():
            y, c = core.forward_cached(proj, cache)
            return y, c.conv, c.ssm.h, c.ssm.last_u, c.ssm.angle
    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = run()
    for values in (other, other * 0.5):
        with torch.no_grad():
            proj.copy_(values)
        graph.replay()
        for i, (a, e) in enumerate(zip([v.clone() for v in out], run())):
            assert torch.equal(a, e), i


@pytest.mark.parametrize("case", ["scan_tensor_core", "mixer_bf16"])
def test_allocations_are_seen_by_those_who_watch(case):
    """Results and scratch come from at::empty when a dispatch mode or a profiler is active: both see them, in the forward pass
    and in the backward pass."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Seen(TorchDispatchMode):
        def __init__(self):
            super().__init__()
            self.names = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.names.append(str(func))
            return func(*args, **(kwargs or {}))
    f, leaves, dout = CASES[case]()
    leaves = [t.clone().requires_grad_(True) for t in leaves]
    out = f(*leaves)
    with Seen() as fwd:
        out = f(*leaves)
    with Seen() as bwd:
        torch.autograd.grad(out, leaves, dout)
    assert any("empty" in n for n in fwd.names) and sum("empty" in n for n in bwd.names) >= len(leaves)
    with torch.autograd.profiler.profile() as prof:
        f(*leaves)
    assert any("aten::empty" == e.key for e in prof.key_averages())
