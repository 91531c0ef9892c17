"""Forms of a launch that few calls reach: batches above 1024 samples, whose schedule is made by three kernels instead of one, and
packed units beside an unsharded call where only one of the two shares its items among CTAs."""
import numpy as np
import pytest
import torch

from helpers import make_lengths, make_problem
from oracle import oracle_block_decisions, oracle_forward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,causal,dtype", [(1025, True, torch.bfloat16), (1500, False, torch.float16), (4100, True, torch.float16)])
def test_many_samples(batch, causal, dtype):
    """1025: the first batch size of that schedule; 4100: beyond the sizes whose samples are ordered by length."""
    import hbsattn_b200 as hb
    rng = np.random.default_rng(batch)
    lens = make_lengths(rng, batch, 1, 40)
    pr = make_problem(95, lens, lens, 4, 2, 64, 16, 16, causal, dtype, 0.6, "diag" if causal else "first")
    rest = (pr["cu_q"], pr["cu_k"], pr["mask"], 16, 16, causal)
    decisions, counts = hb.block_decisions(pr["q"], pr["k"], *rest)
    want = oracle_block_decisions(pr["cu_q_list"], pr["cu_k_list"], pr["mask"], 16, 16, causal)
    np.testing.assert_array_equal(decisions.cpu().numpy(), want)
    np.testing.assert_array_equal(counts.cpu().numpy(), want.sum(axis=2))
    q, k, v = (pr[n].float().requires_grad_(True) for n in "qkv")
    gold = oracle_forward(q, k, v, pr["cu_q_list"], pr["cu_k_list"], pr["mask"], 16, 16, causal, None)
    d_out = torch.randn(pr["q"].shape, generator=torch.Generator().manual_seed(7)).to(dtype).cuda()
    gold.backward(d_out.float())
    for family in ("sm100", "generic"):
        hb.set_kernel_family(family)
        try:
            out, lse = hb.HBSAttention_with_lse(pr["q"], pr["k"], pr["v"], *rest)
            assert hb.last_status()[0] == 0
            grads = hb.attention_backward(pr["q"], pr["k"], pr["v"], out, lse, d_out, *rest)
            assert hb.last_status()[0] == 0
        finally:
            hb.set_kernel_family("auto")
        # rows with few keys: values of order 1 to 4, rounded to 2^-8 of themselves at least twice
        err = (out.float() - gold.detach()).abs()
        assert err.max().item() <= 4e-2 and err.mean().item() <= 2e-3, (family, err.max().item(), err.mean().item())
        for g, w in zip(grads, (q.grad, k.grad, v.grad)):
            assert (g.float() - w).abs().max().item() <= 2e-2 * w.abs().max().item(), family


@pytest.mark.parametrize("heads,tokens,blocks", [((16, 16), 40, (64, 128)), ((8, 2), 20, (16, 80))])
def test_packed_units_where_only_the_part_is_shared(heads, tokens, blocks):
    """One long-context sample: all heads together fill more of the chip than one unit does, so the unit alone is split into more parts
    (or at all), its sums are taken in another order, and it equals the unsharded call up to the rounding of P and of the result."""
    import hbsattn_b200 as hb
    from hbsattn_b200.shard import pack_units, unpack_output
    ql, kl = [tokens] * 12, [5000] * 12
    pr = make_problem(96, ql, kl, *heads, 64, *blocks, True, torch.bfloat16, 0.4, "diag")
    rest = (pr["cu_q"], pr["cu_k"], pr["mask"], pr["qbs"], pr["kbs"], True)
    full = hb.HBSAttention(pr["q"], pr["k"], pr["v"], *rest, None)
    got = torch.full_like(full, float("nan"))
    units = [(b, h) for b in range(12) for h in range(heads[1])]
    for i in range(0, len(units), 3):
        pk = pack_units(units[i:i + 3], pr["q"], pr["k"], pr["v"], *rest[:5])
        out = hb.HBSAttention_csr(pk.q, pk.k, pk.v, pk.cu_q_seqlens, pk.cu_k_seqlens, pk.csr_row_ptr, pk.csr_col_idx, pk.num_q_block,
                                  pk.num_k_block, pr["qbs"], pr["kbs"], True)
        assert hb.last_status()[0] == 0
        unpack_output(pk, out, got)
    gold = oracle_forward(pr["q"].float(), pr["k"].float(), pr["v"].float(), pr["cu_q_list"], pr["cu_k_list"], pr["mask"], pr["qbs"], pr["kbs"], True, None)
    # P and the result are rounded to 2^-9 of themselves on either side; the outputs are means over a few hundred keys and more
    for o in (full, got):
        assert ((o.float() - gold).norm() / gold.norm()).item() <= 5e-3
    assert ((got.float() - full.float()).norm() / gold.norm()).item() <= 5e-3
