"""m3_scan_forward_noalloc, called straight through the C ABI.

The entry point serves hosts that may not allocate device memory while running (an
arena-owning server, a latency-bound decode loop): it must give what m3_scan_forward
gives, call after call, out of the scratch block built into the library.  This file is
collected last so that a run stopping at the first failure has already run the rest.
"""
import ctypes as C

import pytest
import torch

from mamba_trainer_b200 import _ffi, synthetic

pytestmark = pytest.mark.gpu


def _desc(t, w, want_state=True):
    p = lambda v: C.c_void_p(v.data_ptr()) if v is not None else None
    return _ffi.ScanDesc(
        batch=w.batch, seq=w.seq, heads=w.heads, head_dim=w.head_dim, d_state=w.d_state, rank=w.rank,
        chunk=w.chunk, dtype=_ffi.F32 if w.dtype == torch.float32 else _ffi.BF16, discretization=2,
        dynamics=1 if t["theta"] is not None else 0, want_state=int(want_state),
        path=_ffi.PATH_GENERIC,   # overridden per case
        x=p(t["x"]), b=p(t["b"]), c=p(t["c"]), dt=p(t["dt"]), lambda_=p(t["lam"]), theta=p(t["theta"]),
        a_log=p(t["a_log"]), d_skip=p(t["d_skip"]), h0=None, last_u0=None, angle0=None)


def _outputs(t, w):
    y = torch.full_like(t["x"], float("nan"))
    st = lambda *s: torch.full(s, float("nan"), device="cuda")
    h, lu = st(w.batch, w.heads, w.head_dim, w.d_state), st(w.batch, w.heads, w.head_dim, w.d_state)
    ang = st(w.batch, w.heads, w.d_state // 2) if t["theta"] is not None else None
    p = lambda v: C.c_void_p(v.data_ptr()) if v is not None else None
    return (y, h, lu, ang), _ffi.ScanOut(y=p(y), h=p(h), last_u=p(lu), angle=p(ang))


def _free_bytes():
    free, _ = torch.cuda.mem_get_info()
    return free


@pytest.mark.parametrize("idx,kw,path", [(0, dict(), _ffi.PATH_GENERIC),
                                         (3, dict(batch=1, heads=2, seq=300), _ffi.PATH_GENERIC),
                                         (3, dict(batch=1, heads=2, seq=300), _ffi.PATH_AUTO)])
def test_noalloc_forward_matches_the_allocating_one_twice(idx, kw, path):
    """Two calls in a row must both give what m3_scan_forward gives.  Between them a call of ANOTHER shape
    runs on the same built-in block, so that what the first call left there is not what the second would
    write anyway; the second call must not change the device's free memory (nothing is allocated once the
    library's kernels and the block have been touched); and one case is checked against the oracle itself,
    not only against the allocating entry point.  PATH_AUTO takes the tensor-core family, which needs no
    scratch when nothing is kept for a backward pass."""
    from tests._util import oracle_run, norm_rel
    lib = _ffi.load()
    ctx = C.c_void_p()
    assert lib.m3_ctx_create(0, C.byref(ctx)) == _ffi.OK
    try:
        w = synthetic.WORKLOADS[idx].scaled(**kw) if kw else synthetic.WORKLOADS[idx]
        t = {k: (v.cuda() if v is not None else None) for k, v in synthetic.make_inputs(w, seed=4).items()}
        desc = _desc(t, w)
        desc.path = path
        assert lib.m3_scan_scratch_bytes(C.byref(desc), 0) <= _ffi.NOALLOC_SCRATCH_BYTES
        want, out = _outputs(t, w)
        assert lib.m3_scan_forward(ctx, C.byref(desc), C.byref(out), None) == _ffi.OK, lib.m3_last_error(ctx)
        assert lib.m3_sync(ctx) == _ffi.OK
        # the other shape that runs in between (generic family, so it does use the block)
        w2 = synthetic.WORKLOADS[0].scaled(batch=1, heads=3, seq=150)
        t2 = {k: (v.cuda() if v is not None else None) for k, v in synthetic.make_inputs(w2, seed=9).items()}
        desc2 = _desc(t2, w2)
        for call in range(2):
            got, out2 = _outputs(t, w)
            torch.cuda.synchronize()
            before = _free_bytes()
            rc = lib.m3_scan_forward_noalloc(ctx, C.byref(desc), C.byref(out2))
            assert rc == _ffi.OK, lib.m3_last_error(ctx).decode()
            assert lib.m3_sync(ctx) == _ffi.OK
            if call == 1:
                assert _free_bytes() == before, "the second call changed the device's free memory"
            tight = path == _ffi.PATH_GENERIC
            for name, a, e in zip(("y", "h", "last_u", "angle"), got, want):
                if e is None:
                    continue
                a, e = a.float(), e.float()
                assert torch.isfinite(a).all(), f"{name} (call {call})"
                if tight:   # same kernels on different scratch: the float32 tolerance of the parity tests
                    assert ((a - e).abs() <= 1e-5 * max(1.0, float(e.abs().max())) + 1e-4 * e.abs()).all(), \
                        f"{name} (call {call})"
                else:       # the same tensor-core kernels: bit for bit
                    assert torch.equal(a, e), f"{name} (call {call})"
            if call == 0:
                _, out3 = _outputs(t2, w2)
                assert lib.m3_scan_forward_noalloc(ctx, C.byref(desc2), C.byref(out3)) == _ffi.OK
                assert lib.m3_sync(ctx) == _ffi.OK
        if idx == 3 and path == _ffi.PATH_GENERIC:   # against the float64 oracle (bf16 inputs: 2e-2)
            ey, est, _ = oracle_run({k: v for k, v in t.items() if v is not None}, w.chunk, True, torch.float64, False)
            assert norm_rel(got[0].float(), ey) <= 2e-2
            assert norm_rel(got[1].float(), est.h) <= 2e-2
    finally:
        lib.m3_ctx_destroy(ctx)


def test_noalloc_refuses_what_does_not_fit():
    lib = _ffi.load()
    ctx = C.c_void_p()
    assert lib.m3_ctx_create(0, C.byref(ctx)) == _ffi.OK
    try:
        w = synthetic.WORKLOADS[1].scaled(batch=2)   # ~300 MB of scratch
        dummy = torch.zeros(1, device="cuda")
        p = C.c_void_p(dummy.data_ptr())
        desc = _ffi.ScanDesc(batch=w.batch, seq=w.seq, heads=w.heads, head_dim=w.head_dim, d_state=w.d_state,
                             rank=1, chunk=64, dtype=_ffi.BF16, discretization=2, dynamics=0, want_state=0,
                             path=_ffi.PATH_GENERIC,   # the family that needs the block (nothing is launched: refused first)
                             x=p, b=p, c=p, dt=p, lambda_=p, theta=None, a_log=p, d_skip=None)
        assert lib.m3_scan_scratch_bytes(C.byref(desc), 0) > _ffi.NOALLOC_SCRATCH_BYTES
        out = _ffi.ScanOut(y=p, h=None, last_u=None, angle=None)
        assert lib.m3_scan_forward_noalloc(ctx, C.byref(desc), C.byref(out)) == _ffi.ERR_UNSUPPORTED
        assert b"scratch" in lib.m3_last_error(ctx)
    finally:
        lib.m3_ctx_destroy(ctx)


def test_noalloc_calls_of_two_streams_keep_off_each_other():
    """Few long stripes of the tensor-core family put segment states into the shared block: calls of two streams are put one
    behind the other, and give what each gives alone; a call that is captured into a graph, whose launches cannot be, runs
    whole stripes as one launch without the block."""
    from tests._util import norm_rel
    lib = _ffi.load()
    ctxs = [C.c_void_p(), C.c_void_p()]
    for c in ctxs:
        assert lib.m3_ctx_create(0, C.byref(c)) == _ffi.OK
    try:
        w = synthetic.WORKLOADS[3].scaled(batch=1, heads=2, seq=1500)
        ts = [{k: (v.cuda() if v is not None else None) for k, v in synthetic.make_inputs(w, seed=s).items()} for s in (5, 6)]
        descs = [_desc(t, w) for t in ts]
        for d in descs:
            d.path = _ffi.PATH_AUTO

        def call(i):
            got, out = _outputs(ts[i], w)
            torch.cuda.synchronize()
            return got, lambda: lib.m3_scan_forward_noalloc(ctxs[i], C.byref(descs[i]), C.byref(out)), out
        alone = []
        for i in (0, 1):
            got, run, _keep = call(i)
            before = lib.m3_launch_count(ctxs[i])
            assert run() == _ffi.OK, lib.m3_last_error(ctxs[i]).decode()
            assert lib.m3_sync(ctxs[i]) == _ffi.OK
            assert lib.m3_launch_count(ctxs[i]) - before > 1      # cut into segments
            alone.append(got)
        calls = [(i, call(i)) for _ in range(8) for i in (0, 1)]
        for i, (_, run, _keep) in calls:
            assert run() == _ffi.OK, lib.m3_last_error(ctxs[i]).decode()
        for c in ctxs:
            assert lib.m3_sync(c) == _ffi.OK
        for i, (got, _, _keep) in calls:
            for a, e in zip(got[:3], alone[i][:3]):
                assert torch.equal(a, e)
        got, run, _keep = call(0)
        graph, side, before = torch.cuda.CUDAGraph(), torch.cuda.Stream(), lib.m3_launch_count(ctxs[0])
        assert lib.m3_ctx_set_stream(ctxs[0], side.cuda_stream) == _ffi.OK
        with torch.cuda.graph(graph, stream=side):
            assert run() == _ffi.OK, lib.m3_last_error(ctxs[0]).decode()
        assert lib.m3_launch_count(ctxs[0]) - before == 1
        graph.replay()
        torch.cuda.synchronize()
        for a, e in zip(got[:3], alone[0][:3]):   # bf16 operands either way
            assert norm_rel(a.float(), e.float()) <= 2e-2
    finally:
        for c in ctxs:
            lib.m3_ctx_destroy(c)


def test_noalloc_with_a_misaligned_y_allocates_nothing():
    """A y that the tensor-core family cannot write goes to a family that needs scratch: the block, not the pool."""
    from tests._util import norm_rel
    lib = _ffi.load()
    ctx = C.c_void_p()
    assert lib.m3_ctx_create(0, C.byref(ctx)) == _ffi.OK
    try:
        w = synthetic.WORKLOADS[3].scaled(batch=1, heads=2, seq=300)
        t = {k: (v.cuda() if v is not None else None) for k, v in synthetic.make_inputs(w, seed=7).items()}
        desc = _desc(t, w)
        desc.path = _ffi.PATH_AUTO
        (y, *_rest), out = _outputs(t, w)
        off = torch.zeros(y.numel() + 8, device="cuda", dtype=y.dtype)[4:4 + y.numel()]   # 8 bytes
        out2 = _ffi.ScanOut(y=C.c_void_p(off.data_ptr()), h=out.h, last_u=out.last_u, angle=out.angle)
        assert lib.m3_scan_forward_noalloc(ctx, C.byref(desc), C.byref(out)) == _ffi.OK   # warm-up
        assert lib.m3_sync(ctx) == _ffi.OK
        torch.cuda.synchronize()
        before = _free_bytes()
        assert lib.m3_scan_forward_noalloc(ctx, C.byref(desc), C.byref(out2)) == _ffi.OK, lib.m3_last_error(ctx).decode()
        assert lib.m3_sync(ctx) == _ffi.OK
        assert _free_bytes() == before
        assert norm_rel(off.view(y.shape).float(), y.float()) <= 2e-2   # bf16 operands on one side
        desc.path = _ffi.PATH_TENSOR
        assert lib.m3_scan_forward_noalloc(ctx, C.byref(desc), C.byref(out2)) == _ffi.ERR_UNSUPPORTED
    finally:
        lib.m3_ctx_destroy(ctx)


def test_one_warm_up_call_loads_every_kernel():
    """In a process of its own: after one call per element type, calls of shapes that take other kernels (another rank,
    d_state, dynamics, few long stripes) leave the device's free memory as it is."""
    import subprocess
    import sys
    from pathlib import Path
    code = """
import ctypes as C, torch
from mamba_trainer_b200 import _ffi, synthetic
from mamba_trainer_b200.ssm import Discretization
from tests.test_zz_no_alloc import _desc, _outputs
lib, ctx = _ffi.load(), C.c_void_p()
assert lib.m3_ctx_create(0, C.byref(ctx)) == _ffi.OK
def make(dtype, heads, seq, n, rank, rot, p=64):
    w = synthetic.Workload('w', 1, seq, heads, p, n, 64, rank, dtype, Discretization.LearnedTrapezoid, rot, 'scaled')
    t = {k: (v.cuda() if v is not None else None) for k, v in synthetic.make_inputs(w, seed=1).items()}
    d = _desc(t, w)
    d.path = _ffi.PATH_AUTO
    return t, d, _outputs(t, w)
warm = [make(torch.float32, 2, 100, 64, 1, True), make(torch.bfloat16, 2, 100, 128, 1, True)]
other = [make(torch.float32, 2, 70, 128, 2, False), make(torch.float32, 2, 50, 40, 1, True, 24), make(torch.float32, 1, 90, 64, 4, True),
         make(torch.bfloat16, 2, 256, 128, 1, False), make(torch.bfloat16, 2, 900, 128, 2, True), make(torch.bfloat16, 2, 90, 64, 2, True),
         make(torch.bfloat16, 150, 64, 128, 4, False), make(torch.bfloat16, 2, 1000, 128, 4, False)]
def run(c):
    assert lib.m3_scan_forward_noalloc(ctx, C.byref(c[1]), C.byref(c[2][1])) == _ffi.OK, lib.m3_last_error(ctx)
    assert lib.m3_sync(ctx) == _ffi.OK
for c in warm: run(c)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
for c in other: run(c)
assert torch.cuda.mem_get_info()[0] == free, (free, torch.cuda.mem_get_info()[0])
"""
    root = Path(__file__).resolve().parent.parent
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_stripes_stay_whole_where_memory_has_run_out():
    """In a process of its own: with no room left for the scratch that cut stripes hand their state over in, a forward pass
    runs whole stripes, to the same results bit for bit."""
    import subprocess
    import sys
    from pathlib import Path
    code = """
import ctypes as C, torch
from mamba_trainer_b200 import _ffi, synthetic
from mamba_trainer_b200.ssm import Discretization
from tests.test_zz_no_alloc import _desc, _outputs
lib, ctx = _ffi.load(), C.c_void_p()
assert lib.m3_ctx_create(0, C.byref(ctx)) == _ffi.OK
def make(batch, seq):
    w = synthetic.Workload('w', batch, seq, 32, 64, 128, 64, 1, torch.bfloat16, Discretization.LearnedTrapezoid, False, 'rms')
    t = {k: (v.cuda() if v is not None else None) for k, v in synthetic.make_inputs(w, seed=1).items()}
    d = _desc(t, w)
    d.path = _ffi.PATH_AUTO
    return t, d, _outputs(t, w)
def run(c):
    rc = lib.m3_scan_forward(ctx, C.byref(c[1]), C.byref(c[2][1]), None)
    assert rc == _ffi.OK, lib.m3_last_error(ctx)
    assert lib.m3_sync(ctx) == _ffi.OK
    return [v.clone() for v in c[2][0] if v is not None]
small, big = make(2, 300), make(5, 2900)
assert lib.m3_scan_segments(C.byref(small[1]), 0) == 1 and lib.m3_scan_segments(C.byref(big[1]), 0) > 1
run(small)                                  # loads the kernel of whole stripes
torch.cuda.synchronize()
torch.cuda.empty_cache()
MiB = 1 << 20
fill = torch.empty((torch.cuda.mem_get_info()[0] // (2 * MiB) - 3) * 2 * MiB, dtype=torch.uint8, device='cuda')
assert torch.cuda.mem_get_info()[0] < 15 * MiB                        # the scratch takes 15.9
rc = lib.m3_scan_forward(ctx, C.byref(big[1]), C.byref(big[2][1]), None)
assert rc == _ffi.OK, lib.m3_last_error(ctx)
assert lib.m3_sync(ctx) == _ffi.OK
del fill
torch.cuda.empty_cache()
whole = [v.clone() for v in big[2][0] if v is not None]
for a, e in zip(run(big), whole): assert torch.equal(a, e)
"""
    root = Path(__file__).resolve().parent.parent
    r = subprocess.run([sys.executable, "-c", code], cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
