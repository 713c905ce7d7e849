"""Host-side logic of the mixer-side mirrors: widths, validation and error mapping (no GPU)."""
import pytest
import torch

from mamba_trainer_b200.error import ConfigError, ShapeError, UnsupportedError
from mamba_trainer_b200.nn import CausalConv1d, MixerCore, MixerShape, causal_conv1d
from mamba_trainer_b200.ssm import Discretization


def test_widths_follow_the_reference_config():
    """src/ssm/config.rs:165-200: d_inner = heads * head_dim * rank, bc = groups * d_state * rank, the
    projection is z | x | B | C | dt | lambda | theta."""
    s = MixerShape(heads=12, head_dim=64, d_state=128, rank=2, groups=4)
    assert s.d_inner == 12 * 64 * 2 and s.bc_width == 4 * 128 * 2
    assert s.lambda_width == 12 and s.theta_width == 12 * 128 // 2
    assert s.conv_channels == s.d_inner + 2 * s.bc_width
    assert s.in_proj_width == 2 * s.d_inner + 2 * s.bc_width + 12 + 12 + 768
    plain = MixerShape(heads=4, head_dim=8, d_state=16, learned_lambda=False, rotational=False)
    assert plain.n_groups == 4 and plain.lambda_width == 0 and plain.theta_width == 0
    assert plain.in_proj_width == 2 * 32 + 2 * 64 + 4


def test_mixer_core_rejects_inconsistent_configurations():
    with pytest.raises(ConfigError):
        MixerCore(MixerShape(heads=6, head_dim=4, d_state=8, groups=4))               # heads % groups
    with pytest.raises(ConfigError):
        MixerCore(MixerShape(heads=2, head_dim=4, d_state=7, rotational=True))        # odd d_state with rotation
    with pytest.raises(ConfigError):
        MixerCore(MixerShape(heads=3, head_dim=4, d_state=8), bidirectional=True)     # mamba3.rs:107-108
    with pytest.raises(ConfigError):
        MixerCore(MixerShape(heads=2, head_dim=4, d_state=8, learned_lambda=False),
                  discretization=Discretization.LearnedTrapezoid)
    with pytest.raises(ConfigError):
        MixerCore(MixerShape(heads=2, head_dim=4, d_state=8), bidirectional=True, post_gate_norm=True)   # mamba3.rs:175-179
    assert MixerCore(MixerShape(heads=2, head_dim=4, d_state=8, rank=2), post_gate_norm=True).post_norm_w.shape == (16,)
    core = MixerCore(MixerShape(heads=2, head_dim=4, d_state=8))
    assert core.post_norm_w is None
    assert core.conv_w.shape == (4, 2 * 4 + 2 * 2 * 8) and core.norm_w.shape == (8,)
    with pytest.raises(ShapeError):
        core(torch.zeros(1, 3, core.shape.in_proj_width + 1))
    with pytest.raises(UnsupportedError):
        core(torch.zeros(1, 3, core.shape.in_proj_width, dtype=torch.float16))


def test_conv_validates_before_touching_the_device():
    w = torch.zeros(4, 6)
    with pytest.raises(ShapeError):
        causal_conv1d(torch.zeros(2, 6), w)                       # rank (conv.rs:178-187)
    with pytest.raises(ShapeError):
        causal_conv1d(torch.zeros(1, 5, 7), w)                    # channel count
    with pytest.raises(UnsupportedError):
        causal_conv1d(torch.zeros(1, 5, 6), torch.zeros(9, 6))    # more taps than the kernels serve
    with pytest.raises(ShapeError):
        causal_conv1d(torch.zeros(1, 5, 6), w, history=torch.zeros(1, 2, 6))
    conv = CausalConv1d(6, 4)
    assert conv.empty_history(3).shape == (3, 3, 6) and conv.weight.shape == (4, 6)


def test_mixer_core_takes_parameters_that_are_none_of_its_own():
    """A parametrised or pruned weight, a plain tensor in the place of an absent parameter and functional_call's stand-ins
    reach the native call as the module's attributes have them."""
    import torch.nn.utils.parametrize as parametrize
    import torch.nn.utils.prune as prune
    names = ("conv_w", "conv_b", "dt_bias", "a_log", "d_skip", "b_bias", "c_bias", "norm_w", "post_norm_w")

    class Twice(torch.nn.Module):
        def forward(self, v):
            return 2 * v
    core = MixerCore(MixerShape(heads=2, head_dim=4, d_state=8), d_skip=False)
    assert set(core.state_dict()) == set(names) - {"d_skip", "post_norm_w"}
    before = core.conv_w.detach().clone()
    parametrize.register_parametrization(core, "conv_w", Twice())
    prune.random_unstructured(core, "b_bias", 0.5)
    core.d_skip = torch.ones(2)
    got = dict(zip(names, core._spec()[0]))
    assert torch.equal(got["conv_w"], 2 * before) and got["conv_w"].requires_grad
    assert got["b_bias"] is core.b_bias and got["d_skip"] is core.d_skip and got["post_norm_w"] is None
    assert got["a_log"] is core.a_log
    stand_in = torch.zeros(2)
    seen = []
    core.forward = lambda: seen.append(core._spec()[0][3])
    torch.func.functional_call(core, {"a_log": stand_in}, ())
    assert seen[0] is stand_in


def test_the_contexts_lock_keeps_other_threads_out():
    """What `with ctx:` holds: another thread waits for it without holding the interpreter's lock, and its owner may take it
    again."""
    import threading
    from mamba_trainer_b200 import _ffi
    ext, handle, order = _ffi.extension(), 4096, []   # (a key; nothing is read there)

    def other():
        ext.lock(handle)
        order.append("other")
        ext.unlock(handle)
    ext.lock(handle)
    ext.lock(handle)
    t = threading.Thread(target=other)
    t.start()
    t.join(0.2)
    order.append("owner")
    ext.unlock(handle)
    t.join(0.1)
    assert t.is_alive() and order == ["owner"]
    ext.unlock(handle)
    t.join(10)
    assert order == ["owner", "other"]


@pytest.mark.filterwarnings("ignore")
def test_a_native_node_is_traced_as_a_call():
    """What ssm.scan.native does under torch.jit.trace, with a stand-in whose arithmetic the tracer cannot see either."""
    import numpy as np
    from mamba_trainer_b200.ssm.scan import native

    class Unseen(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x, w):
            ctx.save_for_backward(x, w)
            return torch.from_numpy(np.tanh(x.detach().numpy()) * w.detach().numpy())

        @staticmethod
        def backward(ctx, g):
            x, w = ctx.saved_tensors
            return g * w * (1 - x.tanh() ** 2), g * x.tanh()

    def f(x, w):
        return native(lambda handle, a, b, absent, factor: (factor * Unseen.apply(a, b), None), 0, (x * 0.5, w * 2, None), (2,))[0] * 3
    make = lambda: [torch.randn(3, 4, requires_grad=True) for _ in range(2)]
    traced = torch.jit.trace(f, make(), check_trace=False)
    for _ in range(2):
        v = make()
        assert torch.equal(traced(*v), f(*v))
        for a, e in zip(torch.autograd.grad(traced(*v).sum(), v), torch.autograd.grad(f(*v).sum(), v)):
            assert torch.equal(a, e)


def test_forward_mode_is_refused():
    """A tangent on an input of a native node (of either kind) is refused, not dropped."""
    from torch.autograd import forward_ad
    from mamba_trainer_b200 import _ffi
    ext = _ffi.extension()
    x, b, dt, a = torch.ones(1, 2, 1, 4, 1), torch.ones(1, 2, 1, 4, 1), torch.ones(1, 2, 1), torch.ones(1)
    core = MixerCore(MixerShape(heads=1, head_dim=4, d_state=4))
    proj = torch.ones(1, 2, core.shape.in_proj_width)
    params, *spec = core._spec()
    with forward_ad.dual_level():
        for i, t in enumerate((x, b, b, dt, a)):
            args = [x, b, b, dt, a]
            args[i] = forward_ad.make_dual(t, torch.ones_like(t))
            with pytest.raises(NotImplementedError):
                ext.scan(0, *args, None, None, None, None, None, None, 64, 0, False, 0, 0)
        with pytest.raises(NotImplementedError):
            ext.mixer(0, forward_ad.make_dual(proj, proj), params, *spec)
        dual = [forward_ad.make_dual(params[3].detach(), torch.ones(1)) if i == 3 else p for i, p in enumerate(params)]
        with pytest.raises(NotImplementedError):
            ext.mixer(0, proj, dual, *spec)


def test_options_of_other_number_types_reach_the_native_calls(monkeypatch):
    """A chunk length that is a float or longer than 32 bits hold, and switches that are no bools of Python's own, are taken
    as they have always been."""
    import numpy as np
    from mamba_trainer_b200.ssm import ScanInputs, mamba3_scan, scan
    want = MixerCore(MixerShape(heads=2, head_dim=4, d_state=8), chunk=64)._spec()[1:]
    odd = MixerCore(MixerShape(heads=2, head_dim=4, d_state=8, rotational=np.bool_(True)), chunk=64.0, bc_norm=np.bool_(True))
    assert odd._spec(np.int64(0))[1:] == want and type(odd._spec()[1][5]) is int
    assert MixerCore(MixerShape(heads=2, head_dim=4, d_state=8), chunk=10 ** 12)._spec()[1][5] == 1 << 30
    seen = []
    monkeypatch.setattr(scan, "native", lambda node, handle, t, options: seen.append(options) or (t[0], None, None, None))
    monkeypatch.setattr(scan.Context, "of", lambda device: type("", (), {"handle": type("", (), {"value": 0})}))
    x, dt = torch.ones(1, 2, 1, 4, 1), torch.ones(1, 2, 1)
    for chunk in (64.0, np.int64(64), 10 ** 12):
        mamba3_scan(ScanInputs.new(x, x, x, dt, torch.ones(1), dt).with_chunk_size(chunk).with_state_output(False))
        got = seen.pop()
        assert got[0] == min(int(chunk), 1 << 30) and all(type(v) in (int, bool) for v in got)
