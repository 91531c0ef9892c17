"""Runs one benchmark workload through HBSAttention, or VARIANTS through the forward or the backward, a number of times and
stores a fingerprint of every output (run as a script by tests/test_gpu_strict_order.py; which build of the library is
loaded is decided by the HBSATTN_B200_LIBRARY environment variable of the process).

    python tests/fingerprint_worker.py <workload, or "variants" for all of VARIANTS> <repeats> <out.pt>

The fingerprint of an output [total_q, nhead_q, headdim] is one int64 per token: the 16-bit patterns of the token's
values weighted with fixed odd numbers and summed, so that two outputs have equal fingerprints only if they are
bit-identical (up to collisions of a 64-bit checksum)."""
import os
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "tests"))

import torch

# The forms of the kernels that the benchmark workloads do not reach: rings of four stages (d <= 64), tiles gathered across block
# boundaries, items shared by a cluster, the widest tile, and the backward (fp16 with and without items that are done again).
VARIANTS = {
    # name: (backward, q lengths, k lengths, hq, hk, d, qbs, kbs, causal, dtype, density)
    "four_stages": (False, [4096, 3000, 5001], None, 16, 16, 64, 128, 128, True, torch.bfloat16, 0.4),
    "gathered_d128": (False, [4096, 3000, 5001], None, 16, 4, 128, 80, 48, False, torch.bfloat16, 0.3),
    "gathered_d64": (False, [4096, 3000, 5001], None, 16, 16, 64, 64, 80, True, torch.float16, 0.3),
    "shared_d64": (False, [1] * 8, [16384, 30000] * 4, 32, 4, 64, 16, 128, True, torch.bfloat16, 0.3),
    "shared_gathered_d128": (False, [17] * 4, [9000, 16001] * 2, 8, 4, 128, 32, 80, True, torch.bfloat16, 0.5),
    "wide_d256": (False, [2000, 3001], None, 8, 8, 256, 128, 128, True, torch.bfloat16, 0.4),
    "backward_bf16_d128": (True, [4096, 3001], None, 8, 4, 128, 128, 128, True, torch.bfloat16, 0.3),
    "backward_bf16_d64": (True, [1200, 700, 999], None, 16, 4, 64, 80, 48, False, torch.bfloat16, 0.4),
    "backward_fp16_d128": (True, [4096, 3001], None, 8, 8, 128, 128, 128, True, torch.float16, 0.3),
    "backward_fp16_d64": (True, [1200, 700, 999], None, 16, 4, 64, 80, 48, False, torch.float16, 0.4),
    "backward_fp16_again": (True, [2048, 1500], None, 8, 4, 64, 128, 128, True, torch.float16, 1.0),
}


def fingerprint(out: torch.Tensor) -> torch.Tensor:
    flat = out.reshape(out.shape[0], -1)
    g = torch.Generator(device="cpu").manual_seed(1234)
    w = (torch.randint(1, 2 ** 31, (flat.shape[1],), generator=g, dtype=torch.int64) * 2 + 1).to(out.device)
    parts = []
    for r0 in range(0, flat.shape[0], 8192):
        bits = flat[r0:r0 + 8192].view(torch.int16).to(torch.int64)
        parts.append((bits * w).sum(dim=1))
    return torch.cat(parts).cpu()


def variant(name, repeats):
    import hbsattn_b200 as hb
    from helpers import make_problem
    backward, ql, kl, hq, hk, d, qbs, kbs, causal, dtype, keep = VARIANTS[name]
    pr = make_problem(61, ql, ql if kl is None else kl, hq, hk, d, qbs, kbs, causal, dtype, keep, "diag" if causal else "first")
    rest = (pr["cu_q"], pr["cu_k"], pr["mask"], qbs, kbs, causal)
    d_out = torch.randn(pr["q"].shape, generator=torch.Generator().manual_seed(7)).to(dtype).cuda()
    if name == "backward_fp16_again":                   # a sink 20 above the other keys: every item of dK/dV is left to the second launch
        pr["q"][..., 0] = 8.0
        pr["k"][..., 0] = 0.0
        pr["k"][pr["cu_k_list"][:-1]] = torch.tensor([20.0] + [0.0] * (d - 1), dtype=dtype, device="cuda")
    prints = []
    for _ in range(repeats):
        out, lse = hb.HBSAttention_with_lse(pr["q"], pr["k"], pr["v"], *rest)
        outputs = (out,) + (hb.attention_backward(pr["q"], pr["k"], pr["v"], out, lse, d_out, *rest) if backward else ())
        assert hb.last_status()[0] == 0
        prints.append(torch.cat([fingerprint(t) for t in outputs]))
    return prints


def main():
    workload, repeats, out_path = sys.argv[1], int(sys.argv[2]), sys.argv[3]
    if workload == "variants":
        prints = {name: variant(name, repeats) for name in VARIANTS}
        from hbsattn_b200 import _lib
        torch.save({"prints": prints, "library": _lib.LIB_PATH}, out_path)
        return
    import bench
    import hbsattn_b200 as hb
    dev = torch.device("cuda", 0)
    wl = bench.make_workload(workload, 0, dev)
    w = wl["w"]
    hb.set_kernel_family("sm100")
    prints = []
    for _ in range(repeats):
        out = hb.HBSAttention(wl["q"], wl["k"], wl["v"], wl["cu_q_t"], wl["cu_k_t"], wl["mask"], w["qbs"], w["kbs"], w["causal"], None)
        assert hb.last_status()[0] == 0
        prints.append(fingerprint(out))
        del out
    from hbsattn_b200 import _lib
    torch.save({"prints": prints, "library": _lib.LIB_PATH}, out_path)


if __name__ == "__main__":
    main()
