"""K/V tiles strung together from 16-key pieces across block boundaries: every block size that is no multiple of 64 in its
own way (smaller than a tile, larger, with a remainder of one, two or three pieces), rows whose last tile is partly empty, samples that
end inside a piece, blocks cut by the causal reach, and one-block rows, against the fp32 oracle and the CUDA-core kernel."""
import numpy as np
import pytest
import torch

from helpers import make_lengths, make_problem
from oracle import oracle_forward

pytestmark = pytest.mark.gpu

CASES = [
    # name, q lengths, k lengths (None: the same), hq, hk, d, qbs, kbs, causal, dtype, density
    ("one_key", [1, 1], [1, 17], 1, 1, 64, 16, 16, True, torch.bfloat16, 1.0),
    ("blocks_of_16", (40, 300), None, 8, 2, 128, 64, 16, True, torch.bfloat16, 0.4),
    ("blocks_of_32", (40, 300), (1, 400), 4, 4, 64, 32, 32, False, torch.float16, 0.5),
    ("blocks_of_48", [47, 48, 49, 95, 97, 191, 193], None, 4, 1, 128, 80, 48, True, torch.bfloat16, 0.7),
    ("blocks_of_80", (100, 700), None, 6, 2, 96, 64, 80, True, torch.float16, 0.5),
    ("blocks_of_112", (1, 40), (200, 900), 4, 2, 256, 16, 112, True, torch.bfloat16, 0.6),
    ("blocks_of_144", (300, 600), (100, 200), 2, 2, 40, 128, 144, True, torch.float16, 0.8),
    ("blocks_of_208", (100, 900), None, 2, 1, 80, 48, 208, False, torch.bfloat16, 1.0),
]


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_matches_oracle_and_generic(case):
    import hbsattn_b200 as hb
    name, ql, kl, hq, hk, d, qbs, kbs, causal, dtype, keep = case
    rng = np.random.default_rng(len(name))
    ql = ql if isinstance(ql, list) else make_lengths(rng, 3, *ql)
    kl = ql if kl is None else kl if isinstance(kl, list) else make_lengths(rng, 3, *kl)
    pr = make_problem(71, ql, kl, hq, hk, d, qbs, kbs, causal, dtype, keep, None)
    args = (pr["q"], pr["k"], pr["v"], pr["cu_q"], pr["cu_k"], pr["mask"], qbs, kbs, causal)
    out = {}
    for family in ("sm100", "generic"):
        hb.set_kernel_family(family)
        try:
            out[family] = hb.HBSAttention_with_lse(*args)
        finally:
            hb.set_kernel_family("auto")
        assert hb.last_status()[0] == 0
    gold, gold_lse = oracle_forward(pr["q"].cpu().float(), pr["k"].cpu().float(), pr["v"].cpu().float(), pr["cu_q_list"], pr["cu_k_list"],
                                    pr["mask"].cpu(), qbs, kbs, causal, None, return_lse=True)
    # 16-bit probabilities and results: 2^-8 (bfloat16) of values of order 1 each
    for family, (o, lse) in out.items():
        err = (o.cpu().float() - gold).abs()
        assert err.max().item() <= 2e-2 * max(1.0, gold.abs().max().item()) and err.mean().item() <= 1e-3, (family, err.max().item(), err.mean().item())
        dead = torch.isinf(gold_lse)
        assert torch.equal(torch.isinf(lse.cpu()), dead)
        assert (lse.cpu()[~dead] - gold_lse[~dead]).abs().max().item() <= 2e-3 if (~dead).any() else True


def test_neighbours_do_not_leak():
    """Samples whose last piece is cut: the rows of the next sample behind it and what follows the last one are masked, and a
    tile's empty pieces hold zeros rather than what an earlier tile left there."""
    import hbsattn_b200 as hb
    pr = make_problem(72, [70, 50], [41, 90], 2, 2, 64, 64, 48, False, torch.bfloat16, 1.0, None)
    args = (pr["cu_q"], pr["cu_k"], pr["mask"], 64, 48, False, None)
    out = hb.HBSAttention(pr["q"], pr["k"], pr["v"], *args)
    k, v = pr["k"].clone(), pr["v"].clone()
    k[41:] = 3e4                                       # the second sample's keys and values: the first must not see them
    v[41:] = -3e4
    got = hb.HBSAttention(pr["q"], k, v, *args)
    assert torch.equal(got[:70], out[:70])
