"""Kernels that a rule on sizes picks, at the sizes where the rule and the tiles have their edges."""
import pytest
import torch

from _util import ref_metric
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
