"""Which kernels a backward runs on: the family that set_kernel_family selects, and what the tensor-core backward leaves to the CUDA cores
(head dimensions above 128, odd strides).  Both against torch.autograd through the fp32 oracle and against each other; block masks in
CSR form, which only the C ABI takes for a backward, against the dense mask.
Tolerance as in test_gpu_backward.py: 2e-2 of the largest magnitude, 1e-2 on average."""
import ctypes

import pytest
import torch

from helpers import make_problem
from oracle import oracle_forward

pytestmark = pytest.mark.gpu


def _oracle_grads(pr, d_out):
    q, k, v = (pr[n].float().detach().clone().requires_grad_(True) for n in ("q", "k", "v"))
    out = oracle_forward(q, k, v, pr["cu_q_list"], pr["cu_k_list"], pr["mask"], pr["qbs"], pr["kbs"], pr["causal"], None)
    out.backward(d_out.float())
    return q.grad, k.grad, v.grad


def _close(got, want):
    for name, g, w in zip(("dq", "dk", "dv"), got, want):
        err = (g.float() - w.float()).abs()
        assert torch.isfinite(g).all() and err.max().item() <= 2e-2 * w.abs().max().item(), (name, err.max().item(), w.abs().max().item())
        assert err.mean().item() <= 1e-2 * w.float().abs().mean().item(), (name, err.mean().item(), w.float().abs().mean().item())


def _setup(d, dtype, qbs=64, kbs=80, causal=True):
    pr = make_problem(81, [150, 260], [150, 260], 4, 2, d, qbs, kbs, causal, dtype, 0.6, "diag" if causal else "first")
    return pr, torch.randn(pr["q"].shape, generator=torch.Generator().manual_seed(7)).to(dtype).cuda()


def _grads(pr, d_out, q=None, k=None, v=None):
    import hbsattn_b200 as hb
    q, k, v = (pr[n] if t is None else t for n, t in zip("qkv", (q, k, v)))
    rest = (pr["cu_q"], pr["cu_k"], pr["mask"], pr["qbs"], pr["kbs"], pr["causal"])
    out, lse = hb.HBSAttention_with_lse(q, k, v, *rest)
    grads = hb.attention_backward(q, k, v, out, lse, d_out, *rest)
    assert hb.last_status()[0] == 0
    return grads


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d", [64, 128])
def test_selected_family_runs(d, dtype):
    import hbsattn_b200 as hb
    pr, d_out = _setup(d, dtype)
    want = _oracle_grads(pr, d_out)
    rest = (pr["cu_q"], pr["cu_k"], pr["mask"], pr["qbs"], pr["kbs"], pr["causal"])
    out, lse = hb.HBSAttention_with_lse(pr["q"], pr["k"], pr["v"], *rest)
    auto = hb.attention_backward(pr["q"], pr["k"], pr["v"], out, lse, d_out, *rest)
    hb.set_kernel_family("generic")
    try:
        generic = hb.attention_backward(pr["q"], pr["k"], pr["v"], out, lse, d_out, *rest)
        q = pr["q"].detach().clone().requires_grad_(True)
        hb.HBSAttention(q, pr["k"], pr["v"], pr["cu_q"], pr["cu_k"], pr["mask"], pr["qbs"], pr["kbs"], pr["causal"], None).backward(d_out)
    finally:
        hb.set_kernel_family("auto")
    _close(auto, want)
    _close(generic, want)
    _close([q.grad], want[:1])
    # the same forward, sums in another order: some of the roundings of tens of thousands of elements differ, if these are other kernels
    assert not all(torch.equal(a, b) for a, b in zip(auto, generic))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("d", [200, 256])
@pytest.mark.parametrize("family", ["auto", "sm100"])
def test_wide_heads(d, dtype, family):
    """A forward that the tensor-core kernel takes, a backward that it does not: accepted with either family."""
    import hbsattn_b200 as hb
    pr, d_out = _setup(d, dtype)
    hb.set_kernel_family(family)
    try:
        got = _grads(pr, d_out)
    finally:
        hb.set_kernel_family("auto")
    _close(got, _oracle_grads(pr, d_out))


def _strided(t, how):
    if how == "heads_first":                          # [heads, tokens, d] in memory: rows stay 16-byte aligned
        return t.transpose(0, 1).contiguous().transpose(0, 1)
    wide = torch.zeros(*t.shape[:2], t.shape[2] + (8 if how == "padded" else 1), dtype=t.dtype, device=t.device)
    wide[..., :t.shape[2]] = t                        # "odd": rows 2 bytes apart from alignment, for the CUDA cores
    return wide[..., :t.shape[2]]


@pytest.mark.parametrize("how", ["heads_first", "padded", "odd"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_strided_inputs(how, dtype):
    pr, d_out = _setup(64, dtype)
    got = _grads(pr, _strided(d_out, how), *(_strided(pr[n], how) for n in "qkv"))
    _close(got, _oracle_grads(pr, d_out))


@pytest.mark.parametrize("impl", ["generic", "sm100"])
@pytest.mark.parametrize("causal", [True, False])
def test_csr_mask(impl, causal):
    import hbsattn_b200 as hb
    from hbsattn_b200 import _lib, hbsa_interface
    from hbsattn_b200.shard import csr_of_mask
    pr, d_out = _setup(64, torch.float16, causal=causal)
    q, k, v = pr["q"], pr["k"], pr["v"]
    out, lse = hb.HBSAttention_with_lse(q, k, v, pr["cu_q"], pr["cu_k"], pr["mask"], pr["qbs"], pr["kbs"], causal)
    lib = _lib.load()
    nhk, nqb, nkb = pr["mask"].shape
    csr = csr_of_mask(pr["mask"])

    def run(mask, csr):
        grads = [torch.empty_like(t) for t in (q, k, v)]
        ws = hbsa_interface.alloc_workspace(nhk, nqb, nkb, 2, q.device)
        nbytes = lib.hbsa_backward_workspace_bytes(q.shape[0], k.shape[0], q.shape[1], k.shape[1], q.shape[2])
        space = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        b = _lib.BackwardArgs()
        b.struct_bytes = ctypes.sizeof(_lib.BackwardArgs)
        b.fwd = hbsa_interface.make_args(q, k, v, out, pr["cu_q"], pr["cu_k"], mask, pr["qbs"], pr["kbs"], causal, None, nqb, nkb, ws,
                                         {"generic": _lib.HBSA_IMPL_GENERIC, "sm100": _lib.HBSA_IMPL_SM100}[impl], lse=lse, csr=csr)
        b.d_o = d_out.data_ptr()
        for i in range(3):
            b.do_stride[i] = d_out.stride(i)
        b.dq, b.dk, b.dv = (g.data_ptr() for g in grads)
        b.grad_workspace, b.grad_workspace_bytes = space.data_ptr(), nbytes
        assert lib.hbsa_backward(ctypes.byref(b), torch.cuda.current_stream().cuda_stream) == 0, _lib.last_error()
        assert hbsa_interface.read_status(ws)[0] == 0
        return grads
    dense, listed = run(pr["mask"], None), run(None, csr)
    _close(listed, _oracle_grads(pr, d_out))
    if impl == "sm100":                               # one writer per element: the same tiles, the same bits
        for a, b in zip(dense, listed):
            assert torch.equal(a, b)
