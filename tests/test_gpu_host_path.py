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


@pytest.mark.parametrize("d", [64, 18])
def test_backward_takes_an_lse_of_any_strides(d):
    import hbsattn_b200 as hb
    pr = make_problem(92, [100, 60], [100, 60], 2, 1, d, 64, 64, True, torch.bfloat16 if d == 64 else torch.float32, 0.7, "diag")
    rest = (pr["cu_q"], pr["cu_k"], pr["mask"], 64, 64, True)
    out, lse = hb.HBSAttention_with_lse(pr["q"], pr["k"], pr["v"], *rest)
    d_out = torch.ones_like(out)
    want = hb.attention_backward(pr["q"], pr["k"], pr["v"], out, lse, d_out, *rest)
    turned = lse.t().contiguous().t()                # the same values, heads first in memory
    assert not turned.is_contiguous()
    torch.cuda.empty_cache()                         # small blocks come one behind the other out of one segment
    for _ in range(3):
        got = hb.attention_backward(pr["q"], pr["k"], pr["v"], out, turned, d_out, *rest)
        for a, b in zip(got, want):
            assert (a.float() - b.float()).abs().max().item() <= 1e-4 * b.float().abs().max().item()      # fp32: atomics in any order


@pytest.mark.parametrize("lens,block", [([1], 16), ([30, 500, 0, 7], 64), ([70000], 16)])
def test_block_tables_own_their_bytes_only(lens, block, tmp_path):
    import hbsattn_b200 as hb
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device="cuda")
    num, *tables = hb.calculate_blocks(cu, block)
    assert num == sum(-(-n // block) for n in lens)
    for t, size in zip(tables, (num + 1, num, len(lens) + 1)):
        assert t.numel() == size and t.untyped_storage().nbytes() == 4 * size
    torch.save(tables, tmp_path / "tables.pt")
    for a, b in zip(tables, torch.load(tmp_path / "tables.pt")):
        assert torch.equal(a, b)
