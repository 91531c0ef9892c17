"""Rows that a q-block lacks: warps of the tensor-core kernel whose rows do not exist (they answer for tiles without computing
them), in launches with more items than resident CTAs, and thread groups of the CUDA-core kernel with two rows, one or none,
against the fp32 oracle."""
import pytest
import torch

from helpers import make_problem
from oracle import oracle_forward

pytestmark = pytest.mark.gpu

WARP_CASES = [
    # name, q lengths, hq, hk, d, qbs, kbs, causal, dtype
    ("blocks_of_16", [700, 333], 4, 4, 64, 16, 64, True, torch.bfloat16),
    ("blocks_of_80_by_3", [900, 401], 6, 2, 128, 80, 128, True, torch.float16),
    ("blocks_of_80_by_4", [640, 97, 1], 8, 2, 64, 80, 48, False, torch.bfloat16),
    ("ragged_128", [129, 160, 161, 192, 193, 224, 225, 33], 2, 2, 128, 128, 64, True, torch.bfloat16),
    ("wide", [300, 95], 2, 1, 256, 48, 64, True, torch.float16),
]


@pytest.mark.parametrize("case", WARP_CASES, ids=[c[0] for c in WARP_CASES])
def test_warps_without_rows(case):
    import hbsattn_b200 as hb
    name, ql, hq, hk, d, qbs, kbs, causal, dtype = case
    pr = make_problem(91, ql, ql, hq, hk, d, qbs, kbs, causal, dtype, 0.5, None)
    out = hb.HBSAttention(pr["q"], pr["k"], pr["v"], pr["cu_q"], pr["cu_k"], pr["mask"], qbs, kbs, causal, None)
    gold = oracle_forward(pr["q"].float(), pr["k"].float(), pr["v"].float(), pr["cu_q_list"], pr["cu_k_list"], pr["mask"], qbs, kbs, causal, None)
    err = (out.float() - gold).abs()
    # 16-bit probabilities and results: 2^-8 (bfloat16) of values of order 1 each
    assert err.max().item() <= 2e-2 * max(1.0, gold.abs().max().item()) and err.mean().item() <= 1e-3
    big = (pr["q"].float() * 200.0).to(dtype)            # scores of which raw words read as 16-bit numbers are infinities and NaNs
    assert torch.isfinite(hb.HBSAttention(big, pr["k"], pr["v"], pr["cu_q"], pr["cu_k"], pr["mask"], qbs, kbs, causal, None)).all()


PAIR_CASES = [
    # name, q lengths, k lengths, hq, hk, d, qbs, kbs, causal
    ("one_row", [1, 33], [1, 40], 2, 1, 18, 48, 16, True),
    ("half_a_pair", [48, 95, 49], None, 4, 2, 32, 48, 32, True),
    ("two_chunks", [160, 81, 65], None, 2, 2, 64, 80, 48, False),
    ("four_chunks", [200, 256], [150, 300], 4, 1, 96, 256, 80, True),
    ("widest_pair", [130, 64], None, 2, 1, 128, 128, 128, True),
    ("above_pairs", [70, 31], None, 2, 2, 200, 64, 64, True),
    ("blocks_of_32", [70, 31], None, 2, 2, 40, 32, 64, False),
]


@pytest.mark.parametrize("case", PAIR_CASES, ids=[c[0] for c in PAIR_CASES])
def test_rows_in_pairs(case):
    import hbsattn_b200 as hb
    name, ql, kl, hq, hk, d, qbs, kbs, causal = case
    pr = make_problem(92, ql, kl or ql, hq, hk, d, qbs, kbs, causal, torch.float32, 0.6, None)
    out, lse = hb.HBSAttention_with_lse(pr["q"], pr["k"], pr["v"], pr["cu_q"], pr["cu_k"], pr["mask"], qbs, kbs, causal)
    gold, gold_lse = oracle_forward(pr["q"], pr["k"], pr["v"], pr["cu_q_list"], pr["cu_k_list"], pr["mask"], qbs, kbs, causal, None, return_lse=True)
    dead = torch.isinf(gold_lse)
    assert torch.equal(torch.isinf(lse), dead) and (out[dead] == 0).all()
    # sums of at most 300 terms of order 1 in 32 bits, the oracle's own included: a few hundred units of 2^-24
    assert (out - gold).abs().max().item() <= 3e-5
    if (~dead).any():
        assert (lse - gold_lse)[~dead].abs().max().item() <= 3e-5
