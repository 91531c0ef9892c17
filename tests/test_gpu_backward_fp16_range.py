"""fp16 gradients whose P and dS lie far below what fp16 itself resolves: long flat rows, attention sinks under a loss-scaled dO,
rows and samples whose dO differ by orders of magnitude.  Compared with a float64 evaluation of the same formulas on the GPU, part by
part (the keys beside the sink, the small rows), not against the largest gradient.
Tolerance: an fp16 result is rounded to 2^-11 of itself, 2^-11 / sqrt(3) = 2.8e-4 in the 2-norm at most, and O and lse, which the
backward starts from, carry 2^-11 and 2^-24; 6e-4 covers the sum of the roundings.  Gradients below fp16's normal range (2^-14) are
avoided by the choice of dO."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gold(q, k, v, d_out, out, causal):
    """dq, dk, dv in float64 of one sample, one kv-head per q-head group; delta from the rounded output, as the backward takes it."""
    group = q.shape[1] // k.shape[1]
    grads = [torch.zeros(t.shape, dtype=torch.float64, device="cuda") for t in (q, k, v)]
    scale = q.shape[2] ** -0.5
    for h in range(q.shape[1]):
        Q, K, V, G, O = (t.double() for t in (q[:, h], k[:, h // group], v[:, h // group], d_out[:, h], out[:, h]))
        s = Q @ K.T * scale
        if causal:
            s.masked_fill_(torch.ones_like(s, dtype=torch.bool).triu(1 + k.shape[0] - q.shape[0]), float("-inf"))
        p = torch.softmax(s, dim=1)
        ds = p * (G @ V.T - (G * O).sum(1, keepdim=True)) * scale
        grads[0][:, h] = ds @ K
        grads[1][:, h // group] += ds.T @ Q
        grads[2][:, h // group] += p.T @ G
    return grads


def _run(q, k, v, d_out, cu, causal, blocks=(128, 128)):
    import hbsattn_b200 as hb
    cu = torch.tensor(cu, dtype=torch.int32, device="cuda")
    n = [sum(-(-int(x) // b) for x in cu.diff().tolist()) for b in blocks]
    mask = torch.ones(k.shape[1], n[0], n[1], dtype=torch.bool, device="cuda")
    out, lse = hb.HBSAttention_with_lse(q, k, v, cu, cu, mask, *blocks, causal)
    grads = hb.attention_backward(q, k, v, out, lse, d_out, cu, cu, mask, *blocks, causal)
    assert hb.last_status()[0] == 0
    return out, grads


def _rel(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, dtype=torch.float32).cuda()


@pytest.mark.parametrize("blocks", [(128, 128), (80, 48)], ids=["128x128", "80x48"])
@pytest.mark.parametrize("tokens,height,grad", [(16384, 0.0, 16.0), (8192, 16.0, 256.0), (4096, 20.0, 1024.0), (16384, 22.0, 8192.0)])
def test_long_rows_and_sinks(tokens, height, grad, blocks):
    """One key whose logit stands `height` above the others for every query (0: nearly flat attention over all of the keys)."""
    g = torch.Generator().manual_seed(int(height) + tokens)
    d = 64
    q, k, v = (_normal(g, tokens, 1, d) for _ in range(3))
    q *= 0.1
    if height:
        u = torch.nn.functional.normalize(_normal(g, d), dim=0)
        q = q + 8.0 * u
        k = k - (k @ u)[..., None] * u                # no other key along the sink's direction
        k[7] = u * (height * d ** 0.5 / 8.0)
    q, k, v = q.half(), k.half(), v.half()
    d_out = (_normal(g, tokens, 1, d) * grad).half()
    out, got = _run(q, k, v, d_out, [0, tokens], False, blocks)
    want = _gold(q, k, v, d_out, out, False)
    others = torch.arange(tokens, device="cuda") != 7
    for name, a, b in zip(("dq", "dk", "dv"), got, want):
        if name == "dq" and height > 16.0:            # dS of the sink cancels to the last bits of fp32 there, with P and dS of any precision
            continue
        rows = slice(None) if name == "dq" else others
        assert _rel(a[rows], b[rows]) <= 6e-4, (name, _rel(a[rows], b[rows]))


@pytest.mark.parametrize("causal", [False, True])
def test_rows_and_samples_of_different_magnitude(causal):
    """dO of a row in three, and of one sample, 10^-4 of the others'; each group of rows within the tolerance of its own."""
    g = torch.Generator().manual_seed(5)
    cu, hq, hk, d = [0, 700, 1500], 4, 2, 128
    q, k, v, d_out = (_normal(g, cu[-1], h, d) for h in (hq, hk, hk, hq))
    d_out[::3] *= 1e-4
    d_out[cu[1]:] *= 1e-4
    d_out *= 4096.0
    q, k, v, d_out = (t.half() for t in (q, k, v, d_out))
    out, got = _run(q, k, v, d_out, cu, causal, (64, 64))
    for b in (0, 1):
        s = slice(cu[b], cu[b + 1])
        dq, dk, dv = _gold(q[s], k[s], v[s], d_out[s], out[s], causal)
        small = torch.arange(cu[b], cu[b + 1], device="cuda") % 3 == 0
        first = 8 if causal else 0                    # rows that see a few keys only: dS is what is left of cancelling numbers
        small[:first] = False
        big = ~small
        big[:first] = False
        # a sample of small dO: the small rows of it are below fp16's normal range; its large rows are what is looked at
        for rows in (big, small) if b == 0 else (big,):
            assert _rel(got[0][s][rows], dq[rows]) <= 6e-4, (b, "dq", _rel(got[0][s][rows], dq[rows]))
        assert _rel(got[1][s], dk) <= 6e-4 and _rel(got[2][s], dv) <= 6e-4, (b, _rel(got[1][s], dk), _rel(got[2][s], dv))


def test_a_gradient_does_not_depend_on_the_other_samples():
    """The scales are taken from the sample alone: another sample's dO, 2^12 times larger, changes no bit."""
    g = torch.Generator().manual_seed(6)
    cu = [0, 300, 700]
    q, k, v, d_out = (_normal(g, cu[-1], h, 96).half() for h in (4, 2, 2, 4))
    _, first = _run(q, k, v, d_out, cu, True, (64, 80))
    d_out[cu[1]:] *= 4096.0
    _, second = _run(q, k, v, d_out, cu, True, (64, 80))
    for a, b in zip(first, second):
        assert torch.equal(a[:cu[1]], b[:cu[1]])
