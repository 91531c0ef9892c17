"""Tensor-core backward at the sizes where its tiles can go wrong, against torch.autograd through the fp32 oracle: blocks that
are split unevenly (80, 144), smaller than a tile (16, 48) and larger than one (256), GQA groups that do not pack into a
tile, padded head dimensions, one-row samples, and fp16 gradients far outside fp16's own comfortable range.
Tolerance as in test_gpu_backward.py: the products carry 16 bits or more, so what is left is the 8 or 11 bits of the inputs, of
the forward's output (it enters delta) and of the gradients themselves: 2e-2 of the largest magnitude, 1e-2 on average."""
import numpy as np
import pytest
import torch

from helpers import make_lengths, make_problem
from oracle import oracle_forward

pytestmark = pytest.mark.gpu

CASES = [
    # name, q lengths, k lengths (None: the same), hq, hk, d, qbs, kbs, causal, dtype
    ("one_row", [1], [1], 1, 1, 128, 128, 128, True, torch.bfloat16),
    ("tile_edges", [63, 64, 65, 127, 128, 129], None, 2, 1, 64, 64, 64, True, torch.bfloat16),
    ("blocks_of_16", (40, 300), None, 3, 1, 128, 16, 16, True, torch.bfloat16),
    ("uneven_80x144", (100, 500), (50, 700), 6, 2, 96, 80, 144, False, torch.float16),
    ("wide_256", (100, 600), None, 8, 1, 128, 256, 256, True, torch.bfloat16),
    ("group_of_64", (30, 90), (200, 400), 64, 1, 32, 48, 48, True, torch.float16),
    ("q_longer_than_k", (200, 300), (40, 120), 4, 4, 40, 144, 80, True, torch.bfloat16),
    ("many_items", (900, 1500), None, 16, 8, 128, 128, 128, True, torch.bfloat16),
]


def _grads(pr, d_out):
    q, k, v = (pr[n].float().detach().clone().requires_grad_(True) for n in ("q", "k", "v"))
    out = oracle_forward(q, k, v, pr["cu_q_list"], pr["cu_k_list"], pr["mask"], pr["qbs"], pr["kbs"], pr["causal"], None)
    out.backward(d_out.float())
    return q.grad, k.grad, v.grad


def _compare(got, want, what, pr, d_out):
    # Where a gradient cancels (a row that sees one key has dP = delta exactly), the two fp32 dot products that are subtracted are
    # each off by at most d 2^-24 of max|dO| max|V| d, and dS meets K or Q of at most max(|q|, |k|): the bound of what is left.
    d = pr["q"].shape[2]
    rest = 2 * d * 2.0 ** -24 * d * d_out.abs().max().item() * pr["v"].abs().max().item() * max(pr["q"].abs().max().item(), pr["k"].abs().max().item()) * d ** -0.5
    for nm, g, w in zip(("dq", "dk", "dv"), got, want):
        assert torch.isfinite(g).all(), (what, nm)
        err = (g.float() - w).abs()
        top, mean = w.abs().max().item(), w.abs().mean().item()
        if top <= rest:
            assert err.max().item() <= rest, (what, nm, err.max().item(), rest)
            continue
        assert err.max().item() <= 2e-2 * top and err.mean().item() <= 1e-2 * mean, (what, nm, err.max().item() / max(top, 1e-30), err.mean().item() / max(mean, 1e-30))


def _problem(case, seed=61):
    name, ql, kl, hq, hk, d, qbs, kbs, causal, dtype = case
    rng = np.random.default_rng(len(name))
    ql = ql if isinstance(ql, list) else make_lengths(rng, 3, *ql)
    kl = ql if kl is None else kl if isinstance(kl, list) else make_lengths(rng, 3, *kl)
    return make_problem(seed, ql, kl, hq, hk, d, qbs, kbs, causal, dtype, 0.5, "diag" if causal else "first")


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_matches_autograd_and_repeats(case):
    import hbsattn_b200 as hb
    pr = _problem(case)
    d_out = torch.randn(pr["q"].shape, generator=torch.Generator().manual_seed(7)).to(case[-1]).cuda()
    out, lse = hb.HBSAttention_with_lse(pr["q"], pr["k"], pr["v"], pr["cu_q"], pr["cu_k"], pr["mask"], pr["qbs"], pr["kbs"], pr["causal"])

    def run():
        return hb.attention_backward(pr["q"], pr["k"], pr["v"], out, lse, d_out, pr["cu_q"], pr["cu_k"], pr["mask"], pr["qbs"], pr["kbs"], pr["causal"])
    got = run()
    assert hb.last_status()[0] == 0
    _compare(got, _grads(pr, d_out), case[0], pr, d_out)
    for a, b in zip(got, run()):                      # one writer per element: the same bits every time
        assert torch.equal(a, b)


@pytest.mark.parametrize("magnitude", [2.0 ** -14, 2.0 ** 8])
def test_fp16_gradients_of_any_magnitude(magnitude):
    """dS is scaled by a power of two inside: a gradient of 2^-14 (whose dS is subnormal in fp16) and one of 2^8 (whose
    dO V^T exceeds fp16) come out as the scaled gradient of an ordinary one, to the rounding of the result."""
    import hbsattn_b200 as hb
    pr = _problem(("fp16", [200, 90], [300, 90], 4, 2, 128, 64, 64, True, torch.float16))
    pr["v"] = pr["v"] * 4.0                            # dO V^T of order 4 sqrt(128) |dO|; the products stay inside fp16's range in the result
    d_out = (torch.randn(pr["q"].shape, generator=torch.Generator().manual_seed(7)) * magnitude).half().cuda()
    out, lse = hb.HBSAttention_with_lse(pr["q"], pr["k"], pr["v"], pr["cu_q"], pr["cu_k"], pr["mask"], 64, 64, True)
    got = hb.attention_backward(pr["q"], pr["k"], pr["v"], out, lse, d_out, pr["cu_q"], pr["cu_k"], pr["mask"], 64, 64, True)
    assert hb.last_status()[0] == 0
    _compare(got, _grads(pr, d_out), magnitude, pr, d_out)
