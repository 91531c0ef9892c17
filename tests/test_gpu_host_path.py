"""What the native host path must leave to the general one, or return just like it."""
import pytest
import torch
from torch.autograd import forward_ad

from helpers import make_problem

pytestmark = pytest.mark.gpu


def _problem():
    return make_problem(91, [100, 60], [100, 60], 2, 1, 64, 64, 64, True, torch.bfloat16, 0.7, "diag")


@pytest.mark.parametrize("which", ["q", "k", "v"])
@pytest.mark.parametrize("grad_mode", [torch.enable_grad, torch.no_grad])
def test_forward_mode_is_refused_whatever_the_grad_mode(which, grad_mode):
    """There is no forward-mode derivative: a dual input raises, it never loses its tangent."""
    import hbsattn_b200 as hb
    pr = _problem()
    with forward_ad.dual_level(), grad_mode():
        t = {n: pr[n] for n in "qkv"}
        t[which] = forward_ad.make_dual(t[which], torch.ones_like(t[which]))
        with pytest.raises((NotImplementedError, RuntimeError)):
            hb.HBSAttention(t["q"], t["k"], t["v"], pr["cu_q"], pr["cu_k"], pr["mask"], 64, 64, True, None)
