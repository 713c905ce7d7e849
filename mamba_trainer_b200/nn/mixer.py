"""The stretch of the Mamba-3 mixer between its input and output projections, as one call of the library each way.

Mirrors Mamba3Mixer::project + mamba3_scan + finish of the reference (src/models/mamba3.rs:340-461,
:475-484, :540-556; one direction or bidirectional, with or without post_gate_norm): the projection's output
[batch, seq, width] is cut into z | x B C | dt | lambda | theta WITHOUT copies (the kernels read
column bands of it and the backward pass writes the bands of one gradient buffer), then

    convolution + SiLU over x|B|C  ->  B/C bias + RMS norm + layout  ->  softplus / sigmoid
    ->  scan  ->  y * silu(z)        (rms_norm(y) * gain * silu(z) with post_gate_norm)

Every step runs in libm3scan (m3_mixer_forward, m3_mixer_backward, m3_mixer_window), which enqueues the whole stretch.
"""
from __future__ import annotations

import ctypes as C
from dataclasses import dataclass
from functools import cached_property
from typing import Optional

import torch

from .. import _ffi
from ..error import ConfigError, ShapeError, UnsupportedError
from ..ssm.config import Discretization
from ..ssm.scan import Context, SsmState, _DTYPES, _Saved


def _f32(t: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """t as a dense float32 tensor outside the tape; itself when it is one already."""
    if t is None or (t.dtype is torch.float32 and t.is_contiguous()):
        return t
    return t.detach().to(torch.float32).contiguous()


# The parameters in the order of m3_mixer_desc.
_PARAMS = ("conv_w", "conv_b", "dt_bias", "a_log", "d_skip", "b_bias", "c_bias", "norm_w", "post_norm_w")


@dataclass(frozen=True)
class MixerShape:
    """The widths of SsmConfig (src/ssm/config.rs:165-200)."""
    heads: int
    head_dim: int
    d_state: int
    rank: int = 1
    groups: Optional[int] = None
    learned_lambda: bool = True
    rotational: bool = True

    @cached_property
    def n_groups(self) -> int:
        return self.groups or self.heads

    @cached_property
    def d_inner(self) -> int:
        return self.heads * self.head_dim * self.rank

    @cached_property
    def bc_width(self) -> int:
        return self.n_groups * self.d_state * self.rank

    @cached_property
    def lambda_width(self) -> int:
        return self.heads if self.learned_lambda else 0

    @cached_property
    def theta_width(self) -> int:
        return self.heads * self.d_state // 2 if self.rotational else 0

    @cached_property
    def conv_channels(self) -> int:
        return self.d_inner + 2 * self.bc_width

    @cached_property
    def in_proj_width(self) -> int:
        return 2 * self.d_inner + 2 * self.bc_width + self.heads + self.lambda_width + self.theta_width


@dataclass
class MixerCache:
    """What a layer carries from one window to the next (MixerCache, src/models/mamba3.rs:62-80): the
    convolution's last K-1 inputs and the scan's state."""
    conv: torch.Tensor      # [batch, K-1, conv_channels]
    ssm: SsmState


class _MixerCore(torch.autograd.Function):
    """The node: forward = m3_mixer_forward, backward rule = m3_mixer_backward.  `o` is the m3_mixer_desc of the call with
    the gated output's width; the tensors it points into are the other arguments (float32, dense)."""

    @staticmethod
    def forward(fctx, o, proj, *par):
        desc, width = o
        ctx = Context.for_device(proj.device)
        lib = ctx.lib
        B, T, _ = proj.shape
        out = torch.empty((B, T, width), device=proj.device, dtype=proj.dtype)
        act = torch.empty(lib.m3_mixer_activation_bytes(desc), device=proj.device, dtype=torch.uint8)
        track = any(fctx.needs_input_grad)
        saved = C.c_void_p()
        rc = lib.m3_mixer_forward(ctx.handle, desc, out.data_ptr(), act.data_ptr(), C.byref(saved) if track else None)
        if rc:
            ctx.check(rc)
        if track:
            fctx.m3, fctx.desc = ctx, desc
            fctx.saved = _Saved(ctx, saved)
            fctx.keep = (proj, act) + par
        return out

    @staticmethod
    def backward(fctx, dout):
        ctx, desc = fctx.m3, fctx.desc
        ctx.bind_current_stream()
        proj, act = fctx.keep[:2]
        dev = proj.device
        dout = dout.contiguous()
        dproj = torch.empty_like(proj)
        grads = [None if t is None else torch.empty_like(t) for t in fctx.keep[2:]]
        work = torch.empty(ctx.lib.m3_mixer_backward_bytes(desc), device=dev, dtype=torch.uint8)
        rc = ctx.lib.m3_mixer_backward(
            ctx.handle, desc, fctx.saved.handle, act.data_ptr(), dout.data_ptr(),
            _ffi.PACK_MIXER_GRADS.pack(dproj.data_ptr(), *[0 if t is None else t.data_ptr() for t in grads]), work.data_ptr())
        if rc:
            ctx.check(rc)
        return (None, dproj, *grads)


class MixerCore(torch.nn.Module):
    """Parameters and forward of the mixer between its projections (src/models/mamba3.rs:140-270 for
    the parameters; float32 masters, activations float32 or bfloat16)."""

    def __init__(self, shape: MixerShape, conv_kernel: int = 4, chunk: int = 64, conv_bias: bool = True,
                 bc_bias: bool = True, bc_norm: bool = True, norm_gain: bool = True, d_skip: bool = True,
                 eps: float = 1e-5, discretization: Optional[Discretization] = None, bidirectional: bool = False,
                 post_gate_norm: bool = False, device=None):
        super().__init__()
        if shape.heads % shape.n_groups:
            raise ConfigError(f"heads {shape.heads} not a multiple of groups {shape.n_groups}")
        if shape.rotational and shape.d_state % 2:
            raise ConfigError("rotational dynamics require an even d_state")
        if bidirectional and (shape.heads % 2 or shape.n_groups % 2):
            raise ConfigError("a bidirectional mixer needs even heads and groups")      # mamba3.rs:107-108
        if bidirectional and post_gate_norm:                                            # mamba3.rs:175-179
            raise ConfigError("post_gate_norm would normalise across both directions at once; use bc_norm with a "
                              "bidirectional mixer")
        self.shape, self.chunk, self.eps, self.use_norm = shape, chunk, eps, bc_norm
        self.bidirectional = bidirectional
        self.disc = Discretization(discretization) if discretization is not None else (
            Discretization.LearnedTrapezoid if shape.learned_lambda else Discretization.Euler)
        if shape.learned_lambda != self.disc.needs_lambda_projection():
            raise ConfigError("learned_lambda and the discretization disagree")
        par = lambda t: torch.nn.Parameter(t.to(device) if device is not None else t)
        Cc, H, N = shape.conv_channels, shape.heads, shape.d_state
        self.conv_w = par((torch.rand(conv_kernel, Cc) * 2 - 1) / conv_kernel ** 0.5)
        self.conv_b = par(torch.zeros(Cc)) if conv_bias else None
        self.dt_bias = par(torch.log(torch.expm1(torch.exp(torch.empty(H).uniform_(-6.9, -2.3)))))  # softplus^-1
        self.a_log = par(torch.empty(H).uniform_(0.0, 2.77))
        self.d_skip = par(torch.ones(H)) if d_skip else None
        self.b_bias = par(torch.zeros(H, N)) if bc_bias else None
        self.c_bias = par(torch.zeros(H, N)) if bc_bias else None
        self.norm_w = par(torch.ones(N)) if (bc_norm and norm_gain) else None
        # RmsNormConfig::new(d_inner) (mamba3.rs:245-247): a gain of ones over the scan's flattened output
        self.post_gate_norm = post_gate_norm
        self.post_norm_w = par(torch.ones(shape.d_inner)) if post_gate_norm else None
        for name in _PARAMS:   # absent parameters are named all the same
            if name not in self._parameters:
                delattr(self, name)
                self.register_parameter(name, None)

    def empty_cache(self, batch: int, device, dtype=torch.float32) -> MixerCache:
        s = self.shape
        return MixerCache(torch.zeros((batch, self.conv_w.shape[0] - 1, s.conv_channels), device=device, dtype=dtype),
                          SsmState.zeros(batch, s.heads, s.head_dim, s.d_state, s.rotational, device))

    def _pack_desc(self, proj: torch.Tensor, par, path: int = _ffi.PATH_AUTO) -> bytes:
        """The library's description (m3_mixer_desc) of this mixer on `proj`, with parameters `par` (in _PARAMS' order)."""
        s = self.shape
        B, T, _ = proj.shape
        return _ffi.PACK_MIXER_DESC.pack(
            B, T, s.heads, s.head_dim, s.d_state, s.rank, s.n_groups, self.chunk, _DTYPES[proj.dtype], self.disc,
            s.rotational, self._parameters["conv_w"].shape[0], self.use_norm, self.post_gate_norm, path,
            s.heads // 2 if self.bidirectional else 0, self.eps, 0,
            proj.data_ptr(), *[0 if t is None else t.data_ptr() for t in par])

    def forward_cached(self, proj: torch.Tensor, cache: Optional[MixerCache] = None):
        """Inference with a carried state (Mamba3Mixer::apply_with_state, src/models/mamba3.rs:486-560):
        a prefill window or a single decoding step.  Returns (gated output, new MixerCache).  A window
        of one position runs the decode kernel, longer ones the scan; either way it is one call of the library."""
        s = self.shape
        if proj.dim() != 3 or proj.shape[2] != s.in_proj_width:
            raise ShapeError(f"expected [batch, seq, {s.in_proj_width}], got {tuple(proj.shape)}")
        if self.bidirectional:
            raise UnsupportedError("a bidirectional mixer has no causal state to carry")   # mamba3.rs:494-499
        proj = proj.detach() if proj.is_contiguous() else proj.detach().contiguous()
        dev, el = proj.device, proj.dtype
        ctx = Context.for_device(dev)
        B, T, _ = proj.shape
        H, P, N = s.heads, s.head_dim, s.d_state
        if cache is None:
            cache = self.empty_cache(B, dev, el)
        st = cache.ssm
        conv = cache.conv
        if conv.dtype is not el or not conv.is_contiguous():
            conv = conv.to(el).contiguous()
        h, lu = _f32(st.h), _f32(st.last_u)
        ang = _f32(st.angle) if s.rotational else None
        K = self._parameters["conv_w"].shape[0]
        if conv.shape != (B, K - 1, s.conv_channels):
            raise ShapeError(f"the cache's convolution history has shape {tuple(conv.shape)}, expected "
                             f"{(B, K - 1, s.conv_channels)}")
        if h.shape != (B, H, P, N) or lu.shape != (B, H, P, N) or (ang is not None and ang.shape != (B, H, N // 2)):
            raise ShapeError(f"the cache's state does not match batch {B}, heads {H}, head_dim {P}, d_state {N}")
        par = [_f32(self._parameters[n]) for n in _PARAMS]
        desc = self._pack_desc(proj, par)
        out = torch.empty((B, T, s.d_inner), device=dev, dtype=el)
        conv2 = torch.empty_like(conv)
        h2, lu2 = torch.empty_like(h), torch.empty_like(lu)
        ang2 = torch.empty((B, H, N // 2), device=dev, dtype=torch.float32) if s.rotational else None
        io = _ffi.PACK_MIXER_WINDOW_IO.pack(
            conv.data_ptr(), h.data_ptr(), lu.data_ptr(), 0 if ang is None else ang.data_ptr(), out.data_ptr(),
            conv2.data_ptr(), h2.data_ptr(), lu2.data_ptr(), 0 if ang2 is None else ang2.data_ptr())
        lib = ctx.lib
        n = lib.m3_mixer_window_bytes(desc, io)
        work = torch.empty(n, device=dev, dtype=torch.uint8) if n else None
        rc = lib.m3_mixer_window(ctx.handle, desc, io, work.data_ptr() if n else None)
        if rc:
            ctx.check(rc)
        return out, MixerCache(conv2, SsmState(h2, lu2, ang2))

    def forward(self, proj: torch.Tensor, path: int = _ffi.PATH_AUTO) -> torch.Tensor:
        """proj: the input projection's output [batch, seq, in_proj_width]; returns the gated scan
        output [batch, seq, d_inner], the input of the output projection."""
        s = self.shape
        if proj.dim() != 3 or proj.shape[2] != s.in_proj_width:
            raise ShapeError(f"expected [batch, seq, {s.in_proj_width}], got {tuple(proj.shape)}")
        if proj.dtype not in _DTYPES:
            raise UnsupportedError(f"element type {proj.dtype}: float32 and bfloat16 are served")
        # Bidirectional (mamba3.rs:97-112): every piece of the projection is direction-major; the second
        # half of the heads walks right to left inside the convolution and the scan, and nothing is
        # reversed in memory.
        if proj.shape[1] == 0:                      # nothing to scan (scan.rs:134-144)
            return proj.new_zeros((proj.shape[0], 0, s.d_inner)) + 0.0 * proj.sum()
        proj = proj.contiguous()
        p = self._parameters
        par = [t if t is None or (t.dtype is torch.float32 and t.is_contiguous()) else t.to(torch.float32).contiguous()
               for t in (p[n] for n in _PARAMS)]
        return _MixerCore.apply((self._pack_desc(proj, par, path), s.d_inner), proj, *par)
