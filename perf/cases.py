"""Workloads of the fused Mamba-3 scan and its mixer, as a training or serving program calls them.

Three kinds of call, each through the package's public entry points:

  scan    `mamba3_scan` forward and its gradient with respect to every input (one layer's scan in training)
  mixer   `MixerCore` forward and its gradient with respect to the projection and every parameter
          (the stretch of a layer between its two projections, in training)
  window  `MixerCore.forward_cached`: inference with a carried cache - a prefill window, or with seq 1 a
          decoding step

`listed` has the sizes of the five benchmark configurations (the largest one as the shard that one of eight
GPUs gets), the layer widths that go with them, and the small and ragged calls around them; `draw` picks from
the ranges those stand for.
"""
import math
import random

import torch

from mamba_trainer_b200 import synthetic
from mamba_trainer_b200.nn.mixer import MixerCache, MixerCore, MixerShape
from mamba_trainer_b200.ssm import Discretization, ScanInputs, SsmState, mamba3_scan

HEAD_DIM = 64
CONV_KERNEL = 4


def _case(kind, batch, seq, heads, d_state=128, rank=1, dtype="bf16", rotational=True, learned=True, chunk=64):
    return {"kind": kind, "batch": batch, "seq": seq, "heads": heads, "d_state": d_state, "rank": rank,
            "dtype": dtype, "rotational": rotational, "learned": learned, "chunk": chunk}


def listed():
    return [
        # One user decoding on a 768-wide layer: the smallest call there is, all latency.
        dict(_case("window", 1, 1, 12), name="decode_b1_h12"),
        # A full serving batch decoding on a 2048-wide MIMO layer: the state streams through once.
        dict(_case("window", 64, 1, 32, rank=2), name="decode_b64_h32_r2"),
        # One prompt of a length nobody rounded, before decoding starts: few stripes, long in time.
        dict(_case("window", 1, 1777, 16), name="prefill_b1_t1777_h16"),
        # Configuration 0: the small float32 scan that parity work and tests run all day.
        dict(_case("scan", 2, 256, 4, d_state=64, dtype="f32", rotational=False, learned=False), name="scan_f32_cfg0"),
        # A float32 training step of a 1024-wide layer (float32 is the reference's own element type).
        dict(_case("mixer", 8, 1024, 16, dtype="f32"), name="mixer_f32_h16"),
        # bf16 with the smaller state of configuration 0, on a ragged sequence.
        dict(_case("scan", 4, 1500, 8, d_state=64), name="scan_bf16_n64_t1500"),
        # Configurations 1 to 3 in training: SISO real, SISO rotational, MIMO of rank 4.
        dict(_case("scan", 8, 2048, 12, rotational=False), name="scan_cfg1"),
        dict(_case("scan", 8, 4096, 16), name="scan_cfg2"),
        dict(_case("scan", 16, 4096, 32, rank=4), name="scan_cfg3"),
        # Configuration 4, the scaling workload: the shard of one of eight GPUs.
        dict(_case("scan", 8, 16384, 32, rank=2, chunk=128), name="scan_cfg4_shard"),
        # A bf16 training step of the 768-wide layer, and a short ragged MIMO one (fine-tuning).
        dict(_case("mixer", 8, 2048, 12), name="mixer_h12"),
        dict(_case("mixer", 2, 509, 8, rank=2), name="mixer_r2_t509"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    """One more case.  Heads are those of layers 256 to 2048 wide; sequence lengths, window lengths and batches are
    spread over their logarithm and mostly odd; two thirds or more are bf16, rotational, d_state 128, which is what
    models are trained and served with."""
    kind = rng.choice(["scan", "scan", "mixer", "mixer", "window", "window"])
    dtype = "f32" if rng.random() < 0.3 else "bf16"
    heads = rng.choice([4, 8, 12, 16, 24, 32])
    d_state = 64 if rng.random() < 0.25 else 128
    rank = rng.choice([1, 1, 2, 4])
    rotational = rng.random() < 0.75
    learned = rng.random() < 0.8
    chunk = rng.choice([64, 64, 128])
    # token-heads times ranks of one call, at most those of the largest listed case of the element type; bf16 with the
    # small state is used for small models
    most = (1 << 17) if dtype == "f32" else (1 << 18) if d_state == 64 else (1 << 23)
    if kind == "window":
        if rng.random() < 0.5:
            seq, batch = 1, _log_int(rng, 1, 256)
        else:
            seq, batch = _log_int(rng, 16, 8192), _log_int(rng, 1, 8)
    else:
        seq, batch = _log_int(rng, 128, 16384), _log_int(rng, 1, 16)
    while batch > 1 and batch * seq * heads * rank > most:
        batch = (batch + 1) // 2
    if batch * seq * heads * rank > most:
        seq = most // (batch * heads * rank)
    return _case(kind, batch, seq, heads, d_state, rank, dtype, rotational, learned, chunk)


def _dtype(case):
    return torch.float32 if case["dtype"] == "f32" else torch.bfloat16


def _disc(case):
    return Discretization.LearnedTrapezoid if case["learned"] else Discretization.Euler


def _shape(case):
    return MixerShape(case["heads"], HEAD_DIM, case["d_state"], case["rank"], None, case["learned"], case["rotational"])


def prepare(case, seed):
    if case["kind"] == "scan":
        return _prepare_scan(case, seed)
    return _prepare_mixer(case, seed)


def _prepare_scan(case, seed):
    # rank 1 models normalise B and C before the scan, MIMO ones scale them by 1 / sqrt(d_state)
    w = synthetic.Workload("case", case["batch"], case["seq"], case["heads"], HEAD_DIM, case["d_state"], case["chunk"],
                           case["rank"], _dtype(case), _disc(case), case["rotational"],
                           "rms" if case["rank"] == 1 else "scaled")
    t = synthetic.make_inputs_chunked(w, seed=seed, device="cuda", chunk=4)
    if not case["learned"]:
        t["lam"] = None
    names = [k for k in ("x", "b", "c", "dt", "a_log", "lam", "theta", "d_skip") if t[k] is not None]
    for k in names:
        t[k].requires_grad_(True)
    inputs = ScanInputs.new(t["x"], t["b"], t["c"], t["dt"], t["a_log"], t["lam"]).with_skip(t["d_skip"])
    inputs = inputs.with_chunk_size(case["chunk"]).with_discretization(_disc(case)).with_state_output(False)
    if t["theta"] is not None:
        inputs = inputs.with_theta(t["theta"])
    return {"kind": "scan", "inputs": inputs, "names": names, "leaves": [t[k] for k in names], "dy": t["dy"]}


def _prepare_mixer(case, seed):
    dev, el, shape = torch.device("cuda"), _dtype(case), _shape(case)
    B, T, H, N = case["batch"], case["seq"], case["heads"], case["d_state"]
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    randn = lambda *s: torch.randn(*s, device=dev, generator=gen)
    with torch.random.fork_rng(devices=[]):
        torch.manual_seed(seed)
        core = MixerCore(shape, conv_kernel=CONV_KERNEL, chunk=case["chunk"], discretization=_disc(case), device=dev)
    with torch.no_grad():  # a trained layer's biases and skips are not all zeros and ones
        core.conv_b.add_(0.1 * randn(*core.conv_b.shape))
        core.b_bias.add_(0.02 * randn(H, N))
        core.c_bias.add_(0.02 * randn(H, N))
        core.norm_w.add_(0.1 * randn(N))
        core.d_skip.add_(0.2 * randn(H))
    proj = torch.empty((B, T, shape.in_proj_width), device=dev, dtype=el).normal_(generator=gen)
    if case["kind"] == "window":
        cache = MixerCache(randn(B, CONV_KERNEL - 1, shape.conv_channels).to(el),
                           SsmState(0.1 * randn(B, H, HEAD_DIM, N), 0.1 * randn(B, H, HEAD_DIM, N),
                                    math.pi * (2.0 * torch.rand(B, H, N // 2, device=dev, generator=gen) - 1.0)
                                    if case["rotational"] else None))
        return {"kind": "window", "core": core, "proj": proj, "cache": cache}
    proj.requires_grad_(True)
    params = dict(core.named_parameters())
    dout = torch.empty((B, T, shape.d_inner), device=dev, dtype=el).normal_(generator=gen)
    return {"kind": "mixer", "core": core, "proj": proj, "dout": dout, "names": ["proj"] + list(params),
            "leaves": [proj] + list(params.values())}


def run(state):
    if state["kind"] == "window":
        out, cache = state["core"].forward_cached(state["proj"], state["cache"])
        res = {"out": out, "conv": cache.conv, "h": cache.ssm.h, "last_u": cache.ssm.last_u}
        if cache.ssm.angle is not None:
            res["angle"] = cache.ssm.angle
        return res
    if state["kind"] == "scan":
        y = mamba3_scan(state["inputs"]).y
        grads = torch.autograd.grad(y, state["leaves"], state["dy"])
    else:
        y = state["core"](state["proj"])
        grads = torch.autograd.grad(y, state["leaves"], state["dout"])
    return {"y": y.detach(), **{"d_" + k: g for k, g in zip(state["names"], grads)}}


def work(case):
    es = 4 if case["dtype"] == "f32" else 2
    B, T, H, N, R, P = case["batch"], case["seq"], case["heads"], case["d_state"], case["rank"], HEAD_DIM
    tok, passes = B * T, 1 if case["kind"] == "window" else 3
    n_theta = N // 2 if case["rotational"] else 0
    if case["kind"] == "scan":
        inputs = H * (P * R + 2 * N * R + n_theta + 1 + (1 if case["learned"] else 0))
        nbytes = tok * es * 2 * (inputs + H * P * R)         # inputs and dy in, gradients and y out
    else:
        s = _shape(case)
        nbytes = tok * es * (s.in_proj_width + s.d_inner)    # projection in, gated output out
        if case["kind"] == "mixer":
            nbytes *= 2                                      # d out in, d projection out
        else:                                                # the cache, in and out
            nbytes += 2 * B * (es * (CONV_KERNEL - 1) * s.conv_channels + 4 * H * (2 * P * N + n_theta))
    # Products of the scan: the causal half of C B^T and of its product with x over a chunk, the chunk state and its
    # read-out (a window of one token has only the state's); the backward pass has two for each of the forward's.
    L = min(case["chunk"], T)
    flops = tok * H * passes * (L * R * R * (N + P) + 4 * R * P * N)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["dtype"] == "f32":
        # 32-bit sums; d theta is a difference of sums over the whole sequence, which costs it about a digit
        return {"rel": 2e-5, "max": 2e-3}
    # bf16 operands; the same cancellation makes d theta the loosest output where there is a rotation
    return {"rel": 3e-2 if case["rotational"] and case["kind"] != "window" else 1e-2, "max": 0.5}
