"""What a gradient may depend on: rows of another sample, rows of the packed tensors that belong to no sample, and rows that see no
key take part in no pair, so whatever they hold (NaN and Inf included) the gradients of the other rows keep their bits.
The sizes make the backward's tiles ragged: q-blocks and k-blocks that end inside a tile, with the other rows right behind."""
import pytest
import torch

from helpers import make_problem

pytestmark = pytest.mark.gpu

LAYOUTS = [
    # hq, hk, d, qbs, kbs, causal
    (2, 2, 128, 128, 128, True),
    (8, 2, 64, 80, 48, False),
    (3, 1, 96, 48, 144, True),
    (8, 1, 32, 16, 16, True),
    (2, 1, 128, 80, 80, True),            # blocks that end inside a tile of their sample
    (32, 1, 64, 16, 80, True),            # tiles of two tokens, 32 heads each
]


def _gradients(pr, q, k, v, d_out):
    import hbsattn_b200 as hb
    rest = (pr["cu_q"], pr["cu_k"], pr["mask"], pr["qbs"], pr["kbs"], pr["causal"])
    out, lse = hb.HBSAttention_with_lse(q, k, v, *rest)
    grads = hb.attention_backward(q, k, v, out, lse, d_out, *rest)
    assert hb.last_status()[0] == 0
    return out, grads


def _with(t, rows, value):
    t = t.clone()
    t[rows] = value
    return t


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("layout", LAYOUTS, ids=[f"d{x[2]}_{x[3]}x{x[4]}" for x in LAYOUTS])
def test_rows_of_another_sample_and_behind_the_last(layout, dtype, value):
    hq, hk, d, qbs, kbs, causal = layout
    pr = make_problem(71, [203, 150, 77], [203, 150, 77], hq, hk, d, qbs, kbs, causal, dtype, 0.6, "diag" if causal else "first")
    d_out = torch.randn(pr["q"].shape, generator=torch.Generator().manual_seed(7)).to(dtype).cuda()
    behind = 70                                       # rows behind the last sample, as in a buffer that is larger than the batch
    q, k, v, d_out = (torch.cat([t, torch.zeros(behind, *t.shape[1:], dtype=dtype, device="cuda")]) for t in (pr["q"], pr["k"], pr["v"], d_out))
    out0, clean = _gradients(pr, q, k, v, d_out)
    second, end = slice(203, 353), slice(430, 500)
    own = slice(0, 203), slice(353, 430)              # samples 0 and 2
    for bad in ((_with(q, second, value), k, d_out), (q, _with(k, second, value), d_out), (q, k, _with(d_out, second, value))):
        out, grads = _gradients(pr, bad[0], bad[1], v, bad[2])
        for rows in own:
            assert torch.equal(out[rows], out0[rows])
            for got, want in zip(grads, clean):
                assert torch.equal(got[rows], want[rows])
    for bad in ((_with(q, end, value), k, d_out), (q, _with(k, end, value), d_out), (q, k, _with(d_out, end, value))):
        _, grads = _gradients(pr, bad[0], bad[1], v, bad[2])
        for got, want in zip(grads, clean):
            assert torch.equal(got, want) and got[end].abs().max().item() == 0.0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_rows_without_keys(dtype):
    """Causal with more queries than keys: the first rows of the sample see no key, but share tiles with rows that do."""
    pr = make_problem(72, [230], [100], 4, 2, 128, 64, 64, True, dtype, 1.0, None)
    d_out = torch.randn(pr["q"].shape, generator=torch.Generator().manual_seed(7)).to(dtype).cuda()
    rows = slice(0, 130)
    _, clean = _gradients(pr, pr["q"], pr["k"], pr["v"], d_out)
    assert clean[0][rows].abs().max().item() == 0.0
    for q, g in ((_with(pr["q"], rows, float("nan")), d_out), (pr["q"], _with(d_out, rows, float("nan")))):
        _, grads = _gradients(pr, q, pr["k"], pr["v"], g)
        for got, want in zip(grads, clean):
            assert torch.equal(got, want)
