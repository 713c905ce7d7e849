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

from dataclasses import dataclass
from functools import cached_property
from typing import Optional

import torch

from .. import _ffi
from ..error import ConfigError, ShapeError, UnsupportedError
from ..ssm.config import Discretization
from ..ssm.scan import Context, SsmState, _DTYPES, native


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

    def empty_cache(self, batch: int, device, dtype=torch.float32) -> MixerCache:
        s = self.shape
        return MixerCache(torch.zeros((batch, self.conv_w.shape[0] - 1, s.conv_channels), device=device, dtype=dtype),
                          SsmState.zeros(batch, s.heads, s.head_dim, s.d_state, s.rotational, device))

    def _spec(self, path: int = _ffi.PATH_AUTO):
        """The parameters in _PARAMS' order, the integers of m3_mixer_desc, eps and d_inner: what the native node takes."""
        s, p = self.shape, self._parameters
        chunk = self.chunk
        if type(chunk) is not int or chunk > 1 << 30:   # (the native call takes integers of 32 bits)
            chunk = min(int(chunk), 1 << 30)
        # (what is no parameter of the module: absent, or parametrised, pruned, assigned, a view of a flattened one)
        return ([p[n] if n in p else getattr(self, n) for n in _PARAMS],
                (s.heads, s.head_dim, s.d_state, s.rank, s.n_groups, chunk, self.disc, 1 if s.rotational else 0,
                 1 if self.use_norm else 0, 1 if self.post_gate_norm else 0, path, s.heads // 2 if self.bidirectional else 0),
                self.eps, s.d_inner)

    def forward_cached(self, proj: torch.Tensor, cache: Optional[MixerCache] = None):
        """Inference with a carried state (Mamba3Mixer::apply_with_state, src/models/mamba3.rs:486-560):
        a prefill window or a single decoding step.  Returns (gated output, new MixerCache).  A window
        of one position runs the decode kernel, longer ones the scan; either way it is one call of the library."""
        s = self.shape
        if proj.dim() != 3 or proj.shape[2] != s.in_proj_width:
            raise ShapeError(f"expected [batch, seq, {s.in_proj_width}], got {tuple(proj.shape)}")
        if self.bidirectional:
            raise UnsupportedError("a bidirectional mixer has no causal state to carry")   # mamba3.rs:494-499
        if proj.dtype not in _DTYPES:
            raise UnsupportedError(f"element type {proj.dtype}: float32 and bfloat16 are served")
        B = proj.shape[0]
        H, P, N = s.heads, s.head_dim, s.d_state
        if cache is None:
            cache = self.empty_cache(B, proj.device, proj.dtype)
        st = cache.ssm
        spec = self._spec()
        K = spec[0][0].shape[0]
        if cache.conv.shape != (B, K - 1, s.conv_channels):
            raise ShapeError(f"the cache's convolution history has shape {tuple(cache.conv.shape)}, expected "
                             f"{(B, K - 1, s.conv_channels)}")
        if st.h.shape != (B, H, P, N) or st.last_u.shape != (B, H, P, N) or (
                s.rotational and st.angle is not None and st.angle.shape != (B, H, N // 2)):
            raise ShapeError(f"the cache's state does not match batch {B}, heads {H}, head_dim {P}, d_state {N}")
        out, conv, h, last_u, angle = _ffi.extension().window(
            Context.of(proj.device).handle.value, proj, *spec, cache.conv, st.h, st.last_u, st.angle)
        return out, MixerCache(conv, SsmState(h, last_u, angle))

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
        mixer, handle, (params, *spec) = _ffi.extension().mixer, Context.of(proj.device).handle.value, self._spec(path)
        if not torch._C._is_tracing():
            return mixer(handle, proj, params, *spec)
        return native(lambda h, x, *p: (mixer(h, x, p, *spec),), handle, (proj, *params), ())[0]
