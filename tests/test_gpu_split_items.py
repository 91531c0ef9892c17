"""Work items shared by a cluster of CTAs (few rows, long contexts): one token and a few, parts without a tile of their own, rows with fewer
active tiles than there are parts, rows without any key, tiles of gathered pieces, every head-dimension tile, and the schedule
entry point, against the fp32 oracle and the CUDA-core kernel."""
import pytest
import torch

from helpers import make_problem
from oracle import oracle_forward

pytestmark = pytest.mark.gpu

CASES = [
    # name, q lengths, k lengths, hq, hk, d, qbs, kbs, causal, dtype, density
    ("one_token", [1, 1, 1], [4000, 9000, 16384], 16, 2, 64, 16, 128, True, torch.bfloat16, 0.2),
    ("one_item", [3], [13000], 1, 1, 128, 16, 128, True, torch.float16, 0.5),
    ("few_tokens_80_keys", [5, 33, 20], [7001, 3500, 5003], 6, 2, 96, 16, 80, True, torch.bfloat16, 0.3),
    ("wide_heads", [17, 1], [3200, 6401], 4, 2, 256, 32, 64, False, torch.bfloat16, 0.2),
    ("fewer_tiles_than_parts", [20, 40], [6000, 9000], 4, 4, 64, 16, 64, True, torch.float16, 0.02),
    ("short_beside_long", [128, 128, 100], [12000, 100, 60], 2, 1, 40, 128, 48, True, torch.bfloat16, 0.6),
    ("prompt", [700], [6200], 2, 2, 128, 128, 128, True, torch.bfloat16, 0.4),
]


@pytest.mark.parametrize("case", CASES, ids=[c[0] for c in CASES])
def test_matches_oracle_and_generic(case):
    import hbsattn_b200 as hb
    name, ql, kl, hq, hk, d, qbs, kbs, causal, dtype, keep = case
    pr = make_problem(81, ql, kl, hq, hk, d, qbs, kbs, causal, dtype, keep, None)
    args = (pr["q"], pr["k"], pr["v"], pr["cu_q"], pr["cu_k"], pr["mask"], qbs, kbs, causal)
    out = {}
    for family in ("sm100", "generic"):
        hb.set_kernel_family(family)
        try:
            out[family] = hb.HBSAttention_with_lse(*args)
        finally:
            hb.set_kernel_family("auto")
        assert hb.last_status()[0] == 0
    gold, gold_lse = oracle_forward(pr["q"].float(), pr["k"].float(), pr["v"].float(), pr["cu_q_list"], pr["cu_k_list"],
                                    pr["mask"], qbs, kbs, causal, None, return_lse=True)
    dead = torch.isinf(gold_lse)
    if name == "fewer_tiles_than_parts":
        assert dead.any() and not dead.all()
    # 16-bit probabilities and results: 2^-8 (bfloat16) of values of order 1 each
    for family, (o, lse) in out.items():
        err = (o.float() - gold).abs()
        assert err.max().item() <= 2e-2 * max(1.0, gold.abs().max().item()) and err.mean().item() <= 1e-3, (family, err.max().item(), err.mean().item())
        assert torch.equal(torch.isinf(lse), dead), family
        assert (o[dead] == 0).all()
        assert (lse[~dead] - gold_lse[~dead]).abs().max().item() <= 2e-3
    schedule = hb.build_schedule(pr["q"], pr["k"], pr["cu_q"], pr["cu_k"], pr["mask"], qbs, kbs, causal)
    for _ in range(2):
        assert torch.equal(hb.attention_with_schedule(pr["q"], pr["k"], pr["v"], schedule), out["sm100"][0])


def test_parts_with_different_maxima():
    """Scores that grow along the context: every part has another reference maximum, the last one outweighs the others."""
    import hbsattn_b200 as hb
    pr = make_problem(82, [2], [8192], 4, 1, 64, 16, 64, True, torch.bfloat16, 1.0, None)
    pr["k"] = (pr["k"].float() * torch.linspace(0.1, 6.0, 8192, device="cuda")[:, None, None]).to(torch.bfloat16)
    out = hb.HBSAttention(pr["q"], pr["k"], pr["v"], pr["cu_q"], pr["cu_k"], pr["mask"], 16, 64, True, None)
    gold = oracle_forward(pr["q"].float(), pr["k"].float(), pr["v"].float(), pr["cu_q_list"], pr["cu_k_list"], pr["mask"], 16, 64, True, None)
    assert (out.float() - gold).abs().max().item() <= 2e-2 * max(1.0, gold.abs().max().item())
