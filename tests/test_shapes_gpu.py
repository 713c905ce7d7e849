"""Kernels that a rule on sizes picks, at the sizes where the rule and the tiles have their edges."""
import pytest
import torch

from _util import norm_rel, ref_metric, segments
from mamba_trainer_b200.ssm import Discretization

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,B,H,P,N,R,groups,K,post,learned", [
    (torch.float32, 1, 3, 64, 128, 1, None, 4, False, True),    # one launch, rows split down to one pass
    (torch.float32, 3, 4, 40, 64, 2, 2, 2, False, True),        # head_dim no multiple of a pass, shared groups
    (torch.float32, 40, 32, 64, 128, 1, None, 4, False, False),  # whole heads per block, fixed lambda
    (torch.float32, 2, 4, 64, 64, 4, 4, 8, True, True),         # the norm behind the gate is a launch of its own
    (torch.bfloat16, 5, 8, 64, 128, 4, 2, 4, False, True),
    (torch.bfloat16, 9, 12, 64, 64, 1, None, 4, True, True),
    (torch.float32, 2, 2, 8, 32, 3, None, 4, False, True),      # a shape the row kernels leave to k_step
])
def test_decode_step_matches_the_parallel_pass(dtype, B, H, P, N, R, groups, K, post, learned):
    """A prefill window, then single positions from the carried cache, against one pass over the whole sequence."""
    from mamba_trainer_b200.nn import MixerCore, MixerShape
    shape = MixerShape(H, P, N, R, groups, learned)
    torch.manual_seed(R)
    core = MixerCore(shape, conv_kernel=K, chunk=8, device="cuda", post_gate_norm=post,
                     discretization=None if learned else Discretization.Trapezoid)
    with torch.no_grad():
        for q in (core.b_bias, core.c_bias, core.conv_b, core.d_skip):
            q.normal_(0, 0.3)
    proj = torch.randn(B, 9, shape.in_proj_width, device="cuda").to(dtype)
    with torch.no_grad():
        whole = core(proj)
    out, cache = core.forward_cached(proj[:, :5])
    outs = [out]
    for t in range(5, 9):
        o, cache = core.forward_cached(proj[:, t:t + 1], cache)
        outs.append(o)
    got = torch.cat(outs, 1)
    assert ref_metric(got.float(), whole.float()) <= (2e-4 if dtype == torch.float32 else 3e-2)


@pytest.mark.parametrize("dtype,H,P,N,R,K,rot,fused", [
    (torch.bfloat16, 16, 64, 128, 2, 4, True, True),
    (torch.bfloat16, 15, 96, 128, 4, 2, True, True),      # two blocks a head, the second of half the rows
    (torch.float32, 15, 72, 64, 1, 8, False, True),       # more taps than are brought in ahead, no angles
    (torch.float32, 16, 64, 128, 4, 4, True, False),
    (torch.bfloat16, 17, 96, 64, 1, 4, False, False),
])
def test_decode_steps_of_several_waves_equal_small_ones(dtype, H, P, N, R, K, rot, fused):
    """Grids of more than three blocks per SM bring later blocks' inputs into L2; three rows of the batch alone do not.  The
    arithmetic is the same up to the order of a row's sums: float32 outputs within N float32 roundings, bf16 within two."""
    from mamba_trainer_b200.nn import MixerCache, MixerCore, MixerShape
    from mamba_trainer_b200.ssm import SsmState, mamba3_step
    B, few = 3 * torch.cuda.get_device_properties(0).multi_processor_count // H + 2, slice(0, 3)
    torch.manual_seed(H)
    r = lambda *s: torch.randn(*s, device="cuda")
    h, u, ang = r(B, H, P, N), r(B, H, P, N), r(B, H, N // 2)
    state = lambda rows: SsmState(h[rows], u[rows], ang[rows] if rot else None)
    if fused:
        core = MixerCore(MixerShape(H, P, N, R, rotational=rot), conv_kernel=K, device="cuda")
        proj, conv = r(B, 1, core.shape.in_proj_width).to(dtype), r(B, K - 1, core.shape.conv_channels).to(dtype)
        run = lambda rows: core.forward_cached(proj[rows], MixerCache(conv[rows], state(rows)))[0]
    else:
        ins = [r(B, H, P, R), r(B, H, N, R), r(B, H, N, R) / N ** 0.5, r(B, H).abs(), torch.sigmoid(r(B, H))]
        theta, a_log = r(B, H, N // 2), r(H)
        run = lambda rows: mamba3_step(*(t[rows].to(dtype) for t in ins), a_log, theta[rows] if rot else None, None, state(rows))[0]
    tol = N * 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -8
    for rows in (few, slice(B - 3, B)):
        assert norm_rel(run(slice(0, B))[rows].float(), run(rows).float()) <= tol


@pytest.mark.parametrize("dtype,B,T,H,N,R,rot,state,rev,disc", [
    (torch.float32, 2, 64, 2, 128, 1, True, False, 0, 2),     # exactly one chunk
    (torch.float32, 1, 1, 3, 64, 1, True, True, 0, 2),        # one token
    (torch.float32, 1, 65, 2, 64, 1, False, True, 0, 2),      # one token past a chunk
    (torch.float32, 2, 321, 2, 128, 2, True, True, 1, 2),     # ragged, a right-to-left head, carried state
    (torch.float32, 1, 150, 2, 128, 4, True, False, 0, 1),
    (torch.float32, 1, 77, 2, 64, 4, False, True, 2, 0),
    (torch.bfloat16, 2, 200, 3, 64, 1, True, True, 0, 2),
    (torch.bfloat16, 1, 333, 2, 64, 2, False, False, 1, 2),
    (torch.bfloat16, 1, 90, 2, 64, 4, True, True, 0, 2),
])
def test_chunk_parallel_family_matches_the_oracle(dtype, B, T, H, N, R, rot, state, rev, disc):
    """Outputs, states and every gradient against the float64 oracle: float32 as tight as the generic family's
    tests, bf16 at 2e-2 (float32 arithmetic on bf16 inputs, so only inputs and outputs are rounded)."""
    from test_scan_gpu import check_bf16, check_f32, compare_all, small_inputs
    t, ds = small_inputs(B, T, H, 64, N, R, rot, state, seed=T + N + R)
    d = Discretization(disc)
    if d is not Discretization.LearnedTrapezoid:
        t["lam"] = torch.full_like(t["lam"], d.fixed_lambda())
    for k in ("b", "c"):
        t[k] = t[k] / N ** 0.5
    for k in ("x", "b", "c", "dt", "lam", "theta", "dy"):
        if t[k] is not None:
            t[k] = t[k].to(dtype)
    compare_all(t, 64, check_f32 if dtype == torch.float32 else check_bf16, True, ds, discretization=d, reverse_heads=rev)


@pytest.mark.parametrize("B,T,H,N,R,rot", [(2, 256, 4, 64, 1, False), (1, 2000, 4, 128, 1, True), (2, 513, 4, 128, 2, True),
                                          (2, 300, 4, 64, 4, False)])
def test_chunk_parallel_float32_is_as_accurate_as_float32_sums(B, T, H, N, R, rot):
    """Split TF32 against float32 multiply-adds, on inputs as models have them: the chunk-parallel family's distance from
    the float64 oracle is at most the generic family's, which an x that starts off 16 bytes takes.  (1.1: the rounding
    noise of the smallest tensors here, a few thousand values.)"""
    from _util import fused_run, oracle_run
    from mamba_trainer_b200 import synthetic
    w = synthetic.Workload("float32", B, T, H, 64, N, 64, R, torch.float32, Discretization.LearnedTrapezoid, rot,
                           "rms" if R == 1 else "scaled")
    t = synthetic.make_inputs(w, seed=T)
    y, _, exact = oracle_run(t, 64, False)
    exact["y"] = y
    dev = {k: v.cuda() if v is not None else None for k, v in t.items()}
    buf = torch.empty(t["x"].numel() + 1, device="cuda")
    off = dict(dev, x=buf[1:].view(t["x"].shape).copy_(t["x"]))
    (y, _, got), (yg, _, generic) = fused_run(dev, 64, False), fused_run(off, 64, False)
    got["y"], generic["y"] = y, yg
    for n in ("y", "x", "b", "c", "dt", "lam") + (("theta",) if rot else ()):
        a, e = norm_rel(got[n], exact[n]), norm_rel(generic[n], exact[n])
        assert a <= 1.1 * e, (n, a, e)


@pytest.mark.parametrize("dtype,N,R,rot", [(torch.float32, 64, 1, True), (torch.float32, 128, 2, False), (torch.bfloat16, 64, 1, True)])
def test_the_generic_path_runs_the_generic_kernels(dtype, N, R, rot):
    """A caller who names the generic family gets it at shapes the chunk-parallel one serves, in the scan and in the mixer:
    the oracle's results, from more launches."""
    from test_scan_gpu import check_bf16, check_f32, compare_all, small_inputs
    from _util import fused_run
    from mamba_trainer_b200 import _ffi
    from mamba_trainer_b200.nn import MixerCore, MixerShape
    from mamba_trainer_b200.ssm import Context
    t, ds = small_inputs(2, 150, 2, 64, N, R, rot, True, seed=N + R)
    for k in ("x", "b", "c", "dt", "lam", "theta", "dy"):
        if t[k] is not None:
            t[k] = (t[k] / (N ** 0.5 if k in "bc" else 1)).to(dtype)
    ctx = Context.for_device(torch.device("cuda"))

    def launches(f):
        before = ctx.lib.m3_launch_count(ctx.handle)
        f()
        return ctx.lib.m3_launch_count(ctx.handle) - before
    check = check_f32 if dtype == torch.float32 else check_bf16
    n = {p: launches(lambda: fused_run(t, 64, True, True, ds, path=p)) for p in (_ffi.PATH_AUTO, _ffi.PATH_GENERIC)}
    assert n[_ffi.PATH_GENERIC] > n[_ffi.PATH_AUTO], n
    compare_all(t, 64, check, True, ds, path=_ffi.PATH_GENERIC)
    shape = MixerShape(2, 64, N, R, None, True, rot)
    torch.manual_seed(1)
    core = MixerCore(shape, device="cuda")
    proj = torch.randn(2, 150, shape.in_proj_width, device="cuda").to(dtype).requires_grad_(True)
    outs = []
    m = {p: launches(lambda: outs.append(core(proj, path=p))) for p in (_ffi.PATH_AUTO, _ffi.PATH_GENERIC)}
    assert m[_ffi.PATH_GENERIC] > m[_ffi.PATH_AUTO], m
    (a,), (b,) = (torch.autograd.grad(o.float().square().sum(), [proj]) for o in outs)
    assert norm_rel(outs[0], outs[1]) <= (1e-5 if dtype == torch.float32 else 2e-2)
    assert norm_rel(a, b) <= (1e-5 if dtype == torch.float32 else 2e-2)


@pytest.mark.parametrize("dtype,B,T,H,N,state", [(torch.float32, 2, 64, 2, 128, True), (torch.float32, 1, 65, 3, 64, False),
                                                (torch.float32, 1, 321, 2, 64, True), (torch.bfloat16, 1, 150, 2, 128, True)])
def test_ssd_chunked_at_chunk_parallel_shapes(dtype, B, T, H, N, state):
    """The entry with the caller's own a, g, w takes the chunk-parallel kernels at head_dim 64: against the oracle."""
    from test_scan_gpu import check_bf16, check_f32
    from mamba_trainer_b200.ssm import ssd_chunked
    from oracle import m3_oracle as O
    g = torch.Generator().manual_seed(T)
    r = lambda *s: torch.randn(*s, generator=g)
    vals = [r(B, T, H, 64), r(B, T, H, N) / N ** 0.5, r(B, T, H, N) / N ** 0.5, -0.3 * r(B, T, H).abs(), r(B, T, H), r(B, T, H)]
    vals = [v.to(dtype) for v in vals] + ([r(B, H, 64, N)] if state else [])
    dy, dh = r(B, T, H, 64).to(dtype), r(B, H, 64, N)
    cpu = [v.double().requires_grad_(True) for v in vals]
    ey, eh = O.ssd_chunked(*cpu[:6], cpu[6] if state else None, 64, True)
    eg = torch.autograd.grad((ey * dy.double()).sum() + (eh * dh.double()).sum(), cpu)
    dev = [v.cuda().requires_grad_(True) for v in vals]
    y, h = ssd_chunked(*dev[:6], dev[6] if state else None, 64, True)
    gg = torch.autograd.grad((y.float() * dy.float().cuda()).sum() + (h * dh.cuda()).sum(), dev)
    check = check_f32 if dtype == torch.float32 else check_bf16
    check("y", y, ey.detach())
    check("h", h, eh.detach())
    for n, a, e in zip(("x", "b", "c", "a", "g", "w", "h0"), gg, eg):
        check("d" + n, a, e)


def test_chunk_parallel_backward_takes_unaligned_gradients():
    """dy and the gradient buffers of the C ABI may start anywhere; aligned ones give the same bits."""
    import ctypes as C
    from mamba_trainer_b200 import _ffi, synthetic
    from mamba_trainer_b200.ssm import Context
    w = synthetic.WORKLOADS[0].scaled(batch=1, heads=2, seq=100)
    t = {k: v.cuda() if v is not None else None for k, v in synthetic.make_inputs(w, seed=3).items()}
    ctx = Context.for_device(torch.device("cuda"))
    p = lambda v: C.c_void_p(v.data_ptr()) if v is not None else None
    desc = _ffi.ScanDesc(batch=1, seq=100, heads=2, head_dim=64, d_state=64, rank=1, chunk=64, dtype=_ffi.F32,
                         discretization=2, x=p(t["x"]), b=p(t["b"]), c=p(t["c"]), dt=p(t["dt"]), lambda_=p(t["lam"]),
                         a_log=p(t["a_log"]), d_skip=p(t["d_skip"]))
    y, saved = torch.empty_like(t["x"]), C.c_void_p()
    out = _ffi.ScanOut(y=p(y))
    ctx.check(ctx.lib.m3_scan_forward(ctx.handle, C.byref(desc), C.byref(out), C.byref(saved)))
    got = []
    for off in (0, 1):
        at = lambda v: torch.empty(v.numel() + 8, device="cuda")[off:off + v.numel()].view_as(v)
        dy, dx, db, dc = at(t["dy"]), at(t["x"]), at(t["b"]), at(t["c"])
        dy.copy_(t["dy"])
        g = _ffi.ScanGrads(dx=p(dx), db=p(db), dc=p(dc))
        ctx.check(ctx.lib.m3_scan_backward(ctx.handle, saved, C.byref(_ffi.ScanBwdIn(dy=p(dy))), _ffi.GRAD_ALL, C.byref(g)))
        got.append((dx, db, dc))
    ctx.check(ctx.lib.m3_saved_free(ctx.handle, saved))
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype,B,T,H,N,R,K,norm,learned,bidir", [
    (torch.float32, 1, 1, 2, 128, 1, 4, True, True, False),      # one step, most of a block dead
    (torch.float32, 2, 33, 3, 64, 1, 2, True, True, False),      # odd heads: no row of four, the separate steps both times
    (torch.float32, 1, 131, 2, 64, 2, 3, False, False, False),   # no norm: the plain bias
    (torch.float32, 2, 150, 4, 128, 2, 4, True, True, True),     # both directions
    (torch.float32, 1, 70, 2, 64, 4, 1, True, True, False),
    (torch.float32, 3, 600, 8, 128, 4, 4, True, True, False),    # long runs per warp
])
def test_mixer_front_matches_the_separate_steps(dtype, B, T, H, N, R, K, norm, learned, bidir):
    """The fused launches in front of the scan against the convolution, B / C and activation steps of the C ABI run one
    by one: a projection that starts off a 16-byte boundary takes those."""
    from mamba_trainer_b200.nn import MixerCore, MixerShape
    shape = MixerShape(H, 64, N, R, None, learned)
    torch.manual_seed(T)
    core = MixerCore(shape, conv_kernel=K, chunk=16, bc_norm=norm, norm_gain=norm, bidirectional=bidir, device="cuda")
    with torch.no_grad():
        for q in (core.b_bias, core.c_bias, core.conv_b, core.d_skip):
            q.normal_(0, 0.3)
    W = shape.in_proj_width
    raw = torch.randn(B * T * W + 1, device="cuda")
    dout = torch.randn(B, T, shape.d_inner, device="cuda")
    res = []
    for off in (0, 1):
        buf = torch.empty(B * T * W + 8, device="cuda")
        proj = buf[off:off + B * T * W].copy_(raw[:-1]).view(B, T, W).requires_grad_(True)
        out = core(proj)
        res.append((out,) + torch.autograd.grad(out, [proj] + list(core.parameters()), dout))
    names = ["out", "proj"] + [n for n, _ in core.named_parameters()]
    for n, a, e in zip(names, *res):
        scale = max(1.0, float(e.abs().max()))
        assert ((a - e).abs() <= 2e-5 * scale + 1e-4 * e.abs()).all(), (n, float((a - e).abs().max()), scale)


@pytest.mark.parametrize("dtype,B,T,H,P,N,R,bidir", [
    (torch.float32, 2, 64, 6, 32, 128, 1, True),      # d_inner 192: the second tile of x is half dead, no block inside
    (torch.float32, 1, 131, 6, 32, 64, 1, True),      # the same with blocks whose every step is inside the sequence
    (torch.float32, 2, 131, 2, 32, 64, 1, False),     # one direction, d_inner 64
    (torch.float32, 12, 1290, 6, 32, 64, 1, True),    # blocks of 128 steps
    (torch.bfloat16, 1, 131, 6, 32, 64, 1, True),
    (torch.bfloat16, 2, 99, 6, 32, 128, 2, True),
    (torch.bfloat16, 1, 200, 6, 16, 64, 4, True),     # d_inner 384: whole tiles, a direction change inside one
    (torch.bfloat16, 1, 70, 4, 24, 64, 1, False),     # d_inner 96
])
def test_mixer_front_tiles_past_the_bands_end(dtype, B, T, H, P, N, R, bidir):
    """Bands that do not fill the front's 128-channel tiles: no lane past a band's end writes anything, whichever way its
    blocks run.  Against the separate steps, and the launch counts say that one run took each form."""
    from mamba_trainer_b200.nn import MixerCore, MixerShape
    from mamba_trainer_b200.ssm import Context
    shape = MixerShape(H, P, N, R, None, True)
    torch.manual_seed(T)
    core = MixerCore(shape, chunk=64, bidirectional=bidir, device="cuda")
    with torch.no_grad():
        for q in (core.b_bias, core.c_bias, core.conv_b, core.d_skip):
            q.normal_(0, 0.3)
    W = shape.in_proj_width
    raw = torch.randn(B * T * W, device="cuda").to(dtype)
    dout = torch.randn(B, T, shape.d_inner, device="cuda").to(dtype)
    ctx = Context.for_device(torch.device("cuda"))
    res, launches = [], []
    for off in (0, 1):
        buf = torch.empty(B * T * W + 8, device="cuda", dtype=dtype)
        proj = buf[off:off + B * T * W].copy_(raw).view(B, T, W).requires_grad_(True)
        before = ctx.lib.m3_launch_count(ctx.handle)
        out = core(proj)
        res.append((out,) + torch.autograd.grad(out, [proj] + list(core.parameters()), dout))
        launches.append(ctx.lib.m3_launch_count(ctx.handle) - before)
    assert launches[0] < launches[1], launches
    names = ["out", "proj"] + [n for n, _ in core.named_parameters()]
    for n, a, e in zip(names, *res):
        a, e = a.float(), e.float()
        scale = max(1.0, float(e.abs().max()))
        if dtype == torch.float32:
            assert ((a - e).abs() <= 2e-5 * scale + 1e-4 * e.abs()).all(), (n, float((a - e).abs().max()), scale)
        else:   # a flipped rounding of x, B or C is 2^-8 of the value and travels on: the bound of the other bf16 tests
            assert norm_rel(a, e) <= 2e-2 and ref_metric(a, e) <= 2e-2 * scale, (n, norm_rel(a, e), ref_metric(a, e), scale)


@pytest.mark.parametrize("B,H,R,rot,T,state,rev", [
    (2, 2, 1, True, 385, True, 0),      # four tiles, the last one a single step: cut in the backward pass only
    (2, 2, 1, True, 769, True, 0),      # seven tiles: the fewest that are cut both ways
    (2, 2, 1, False, 1000, True, 0),    # real dynamics of rank 1
    (2, 2, 2, True, 1000, True, 1),     # a right-to-left head, carried state and angle
    (2, 2, 2, True, 449, False, 0),     # the second half of the last tile is padding
    (2, 2, 4, True, 321, True, 0),
    (2, 2, 4, False, 160, False, 1),    # five tiles: the fewest of real dynamics that the backward pass cuts
    (2, 2, 4, False, 256, False, 1),    # eight: the forward pass too
    (5, 8, 4, True, 999, True, 0),       # 32 tiles of 40 stripes: states of groups of several tiles, the last one shorter
])
def test_side_by_side_segments_match_the_oracle(B, H, R, rot, T, state, rev):
    """Few stripes of the tensor-core family: segments of a stripe run at once from states worked out ahead of them."""
    from test_scan_gpu import check_bf16, compare_all, small_inputs, tc_workload
    fwd, bwd = segments(tc_workload(R, rot, T, B, H))
    assert bwd < -1 and (fwd < -1) == ((R, T) not in ((1, 385), (4, 160))), (fwd, bwd)
    t, ds = small_inputs(B, T, H, 64, 128, R, rot, state, seed=T + R)
    for k in ("b", "c"):
        t[k] = t[k] / 128 ** 0.5
    t["dt"] = t["dt"] * 0.2
    if rot:
        t["theta"] = t["theta"] * 0.3
    for k in ("x", "b", "c", "dt", "lam", "theta", "dy"):
        if t[k] is not None:
            t[k] = t[k].to(torch.bfloat16)

    def check(name, a, e):   # d theta: as in the tests of the stripe kernels, amplified by cancellation
        if name == "dtheta":
            assert float((a.double().cpu() - e).norm() / e.norm()) <= 3e-2, name
        else:
            check_bf16(name, a, e)
    compare_all(t, 64, check, True, ds, path=2, reverse_heads=rev)


@pytest.mark.parametrize("T,H,R,copies", [(1670, 4, 1, 40), (1072, 6, 2, 27)])
def test_cut_stripes_lose_no_accuracy(T, H, R, copies):
    """Few stripes, cut into segments that run side by side, against the same stripes among copies of themselves, which run
    whole or cut one segment after another (bit for bit the same): d theta, where the two sides of every pair of steps have
    to cancel, is as close to the float64 oracle (1.08: what the segments' own float32 sums may move)."""
    from _util import fused_run, oracle_run
    from mamba_trainer_b200 import synthetic
    from mamba_trainer_b200.ssm import Context
    w = synthetic.Workload("cut", 1, T, H, 64, 128, 64, R, torch.bfloat16, Discretization.LearnedTrapezoid, True,
                           "rms" if R == 1 else "scaled")
    ctx = Context.for_device(torch.device("cuda"))

    def run(v):
        before = ctx.lib.m3_launch_count(ctx.handle)
        _, _, g = fused_run(v, 64, False, path=2)
        return g["theta"], ctx.lib.m3_launch_count(ctx.handle) - before
    assert max(segments(w)) < -1 and min(segments(w, batch=copies)) >= 1
    errors = []
    for seed in range(3):
        t = synthetic.make_inputs(w, seed=seed)
        _, _, exact = oracle_run(t, 64, False)
        many = {k: v.repeat(copies, *[1] * (v.dim() - 1)) if v.dim() >= 3 else v for k, v in t.items() if v is not None}
        (cut, n_cut), (whole, n_whole) = run(t), run(many)
        assert n_cut > n_whole, (n_cut, n_whole)
        errors.append((norm_rel(cut.float(), exact["theta"]), norm_rel(whole[:1].float(), exact["theta"])))
    a, e = (sum(v) for v in zip(*errors))
    assert a <= 1.08 * e, errors


@pytest.mark.parametrize("T,H,R", [(8200, 2, 1), (9001, 3, 2)])
def test_long_cut_stripes_match_the_oracle(T, H, R):
    """Stripes of some hundred tiles cut into segments, inputs as models have them.  d theta, a difference of sums over the
    sequence, is held to the reference's own bf16 matmul mode on the same inputs, as in the tests of whole stripes."""
    from test_scan_gpu import check_bf16
    from _util import fused_run, oracle_run, reference_mode_error
    from mamba_trainer_b200 import synthetic
    from mamba_trainer_b200.ssm import Context
    w = synthetic.Workload("long", 1, T, H, 64, 128, 64, R, torch.bfloat16, Discretization.LearnedTrapezoid, True,
                           "rms" if R == 1 else "scaled")
    assert max(segments(w)) < -1
    t = synthetic.make_inputs(w, seed=R)
    ctx = Context.for_device(torch.device("cuda"))
    before = ctx.lib.m3_launch_count(ctx.handle)
    y, _, got = fused_run(t, 64, False, path=2)
    # group states, pass and stripe kernel each way, the angles of the forward pass, the joined sums of d phi
    assert ctx.lib.m3_launch_count(ctx.handle) - before >= 7
    ey, _, exact = oracle_run(t, 64, False)
    mode = reference_mode_error(t, 64, exact, ("theta",))
    check_bf16("y", y, ey)
    for n, e in exact.items():
        if n == "theta":
            assert norm_rel(got[n].float(), e) <= max(2e-2, mode[n]), (n, norm_rel(got[n].float(), e), mode)
        else:
            check_bf16("d" + n, got[n], e)


@pytest.mark.parametrize("dtype,H,N,R,T,rot", [(torch.float32, 40, 128, 1, 700, True), (torch.bfloat16, 40, 64, 2, 300, True),
                                              (torch.bfloat16, 2, 128, 1, 1000, True), (torch.bfloat16, 3, 128, 2, 700, False),
                                              (torch.bfloat16, 2, 128, 1, 1000, False), (torch.float32, 3, 40, 1, 90, True)])
def test_a_state_replaced_in_place(dtype, H, N, R, T, rot):
    """The C entry's returned state in the buffers of the one carried in gives what separate buffers give."""
    import ctypes as C
    from test_scan_gpu import small_inputs
    from mamba_trainer_b200 import _ffi
    from mamba_trainer_b200.ssm import Context
    P = 24 if N == 40 else 64
    t, _ = small_inputs(2, T, H, P, N, R, rot, True, seed=T)
    for k in ("x", "b", "c", "dt", "lam", "theta"):
        if t[k] is not None:
            t[k] = (t[k] / (N ** 0.5 if k in "bc" else 1)).to(dtype)
    t = {k: v.cuda() if v is not None else None for k, v in t.items()}
    p = lambda v: C.c_void_p(v.data_ptr()) if v is not None else None
    ctx, res = Context.for_device(torch.device("cuda")), []
    for in_place in (False, True):
        st = [v.clone() if v is not None else None for v in (t["h0"], t["last_u0"], t["angle0"])]
        new = st if in_place else [torch.empty_like(v) if v is not None else None for v in st]
        y = torch.empty_like(t["x"])
        d = _ffi.ScanDesc(batch=2, seq=T, heads=H, head_dim=P, d_state=N, rank=R, chunk=64, discretization=2, want_state=1,
                          dtype=_ffi.F32 if dtype == torch.float32 else _ffi.BF16, dynamics=int(rot), x=p(t["x"]), b=p(t["b"]),
                          c=p(t["c"]), dt=p(t["dt"]), lambda_=p(t["lam"]), theta=p(t["theta"]), a_log=p(t["a_log"]),
                          h0=p(st[0]), last_u0=p(st[1]), angle0=p(st[2]))
        out = _ffi.ScanOut(y=p(y), h=p(new[0]), last_u=p(new[1]), angle=p(new[2]))
        ctx.check(ctx.lib.m3_scan_forward(ctx.handle, C.byref(d), C.byref(out), None))
        res.append([y] + [v for v in new if v is not None])
    # (a tensor-core stripe runs whole in place and cut otherwise: bf16 operands either way)
    tol = 2e-2 if dtype == torch.bfloat16 and N == 128 else 0.0
    for n, a, e in zip(("y", "h", "last_u", "angle"), *res):
        if n == "angle":
            assert float((torch.sin(a) - torch.sin(e)).abs().max()) <= (2e-3 if tol else 0.0)
        else:
            assert norm_rel(a.float(), e.float()) <= tol, n


def test_real_dynamics_of_rank_1_match_the_oracle_at_multiples_of_eight():
    """Sequences a multiple of eight, whole stripes: more heads than are cut side by side."""
    from test_scan_gpu import check_bf16, compare_all, small_inputs
    t, ds = small_inputs(6, 264, 10, 64, 128, 1, False, True, seed=3)
    for k in ("b", "c"):
        t[k] = t[k] / 128 ** 0.5
    t["dt"] = t["dt"] * 0.2
    for k in ("x", "b", "c", "dt", "lam", "dy"):
        t[k] = t[k].to(torch.bfloat16)
    compare_all(t, 64, check_bf16, True, ds, path=2)


def test_per_head_sums_where_the_grid_has_no_row_left():
    """65535 stripes: the heads' blocks of the last launch, which lie ahead of the stripes' rows, get a layer of their own.
    The sums equal those of the two halves (float32 sums of 65535 terms: 1e-4)."""
    from _util import fused_run
    from mamba_trainer_b200 import synthetic
    w = synthetic.Workload("rows", 65535, 2, 1, 64, 64, 64, 1, torch.float32, Discretization.LearnedTrapezoid, True, "rms")
    t = synthetic.make_inputs(w, seed=7)
    _, _, g = fused_run(t, 64, False, True)
    sums = {}
    for lo, hi in ((0, 30000), (30000, 65535)):
        part = {k: v if v is None or k in ("a_log", "d_skip") else v[lo:hi] for k, v in t.items()}
        _, _, gp = fused_run(part, 64, False, True)
        for n, v in gp.items():
            if n in ("a_log", "d_skip"):
                sums[n] = sums.get(n, 0) + v.double()
            else:
                assert torch.equal(g[n][lo:hi], v), n
    for n, v in sums.items():
        assert torch.allclose(g[n].double(), v, rtol=1e-4, atol=1e-3), (n, g[n], v)
