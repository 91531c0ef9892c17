"""The calls whose speed counts, as users of this package make them.

``listed()`` holds a dozen of them, from one small example batch to long-context prefill and a training step; ``draw(rng)``
gives further ones from the same ranges.  A case is a flat dict:

  call          which public entry points a pass goes through (see ``run``)
  dtype         of q, k, v
  batch, q_min, q_max, k_min, k_max, round_to, len_seed
                samples and their lengths: uniform in [min, max], rounded down to a multiple of ``round_to``, fixed by
                ``len_seed``; k_max = 0 means every k_len equals its q_len
  heads_q, heads_k, head_dim, q_block, k_block, causal
  keep          Bernoulli density of the block mask; under a causal mask the last k-block that a q-block may see is always
                kept, so that no row is empty
"""
import numpy as np
import torch

import hbsattn_b200 as hb
from hbsattn_b200.shard import csr_of_mask

DTYPES = {"bfloat16": torch.bfloat16, "float16": torch.float16, "float32": torch.float32}


def _case(call, batch, q_len, k_len, heads, head_dim, blocks, causal, keep, dtype="bfloat16", round_to=1, len_seed=0, **more):
    k_len = k_len or (0, 0)
    return dict(call=call, dtype=dtype, batch=batch, q_min=q_len[0], q_max=q_len[1], k_min=k_len[0], k_max=k_len[1], round_to=round_to,
                len_seed=len_seed, heads_q=heads[0], heads_k=heads[1], head_dim=head_dim, q_block=blocks[0], k_block=blocks[1],
                causal=causal, keep=keep, **more)


def listed():
    return [
        # the example batch of the package's first user: five short samples, ten positional arguments; pure call latency
        _case("forward", 5, (32, 32), (23, 39), (8, 2), 32, (32, 16), True, 0.7, name="example_batch"),
        # a serving loop over small ragged batches: the block tables are made for every new batch, then passed on
        _case("tables", 8, (30, 500), None, (16, 4), 64, (64, 64), True, 0.5, name="small_new_batches"),
        # one decoding step of a long-context batch: one new token per sample, the schedule shared by the layers of the model
        _case("schedule", 16, (1, 1), (16384, 32768), (64, 8), 64, (16, 128), True, 0.2, name="decode_step"),
        # a chunk of new tokens against a long context (bottom-right causal, ragged key ends)
        _case("forward", 16, (128, 512), (16384, 32768), (64, 8), 64, (16, 128), True, 0.2, round_to=16, name="chunk_on_context"),
        # the headline workload: eight samples of 8192 tokens, 0.9 sparse, block tables kept by the caller
        _case("kept", 8, (8192, 8192), None, (32, 32), 128, (128, 128), True, 0.1, name="prefill_8k"),
        # prompts of unequal length, GQA, block sizes that are no powers of two, bidirectional
        _case("kept", 8, (1024, 16384), None, (32, 8), 128, (80, 48), False, 0.3, round_to=16, len_seed=1, name="varlen_gqa_80x48"),
        # long prompts at 0.7 sparsity, where the tensor cores set the pace
        _case("kept", 8, (16384, 16384), None, (32, 32), 128, (128, 128), True, 0.3, name="prefill_16k"),
        # half precision, a head dimension between the tile sizes, odd lengths, and the log-sum-exp wanted beside the output
        _case("lse", 6, (301, 3001), None, (24, 8), 96, (64, 80), True, 0.4, dtype="float16", len_seed=2, name="fp16_d96_with_lse"),
        # one rank's share of a sharded forward: (sample, kv-head) units packed as samples, block mask in CSR form
        _case("csr", 32, (8192, 8192), None, (1, 1), 128, (128, 128), True, 0.3, name="packed_units_csr"),
        # single precision, as used to check results
        _case("forward", 4, (200, 1500), None, (8, 2), 64, (64, 64), True, 0.5, dtype="float32", len_seed=3, name="fp32_check"),
        # one attention layer of a training step, forward and backward
        _case("train", 2, (8192, 8192), None, (16, 16), 128, (128, 128), True, 0.1, name="train_8k"),
        # the same for ragged GQA samples with small heads and uneven blocks
        _case("train", 8, (100, 1200), None, (16, 4), 64, (80, 48), False, 0.3, dtype="float16", len_seed=4, name="train_varlen_gqa"),
    ]


def _most(call, dtype):
    """The dearest listed case of a kind, in FLOPs: what a drawn one may cost at most."""
    return max(work(c)["flops"] for c in listed() if (c["call"] == "train") == (call == "train") and (c["dtype"] == "float32") == (dtype == "float32"))


def draw(rng):
    """One more case: sizes over the whole range of the listed ones (log-uniform), odd ones among them."""

    def log_int(lo, hi):
        return int(round(lo * (hi / lo) ** rng.random()))

    kind = rng.choice(["forward", "tables", "kept", "kept", "schedule", "lse", "csr", "train", "train", "fp32"])
    while True:
        call, dtype = ("forward", "float32") if kind == "fp32" else (kind, rng.choice(["bfloat16", "bfloat16", "float16"]))
        batch = rng.choice([1, 2, 3, 5, 8, 16])
        heads_k = rng.choice([1, 2, 4, 8, 16, 32])
        heads_q = heads_k * rng.choice([1, 1, 2, 3, 4, 8])
        head_dim = rng.choice([32, 64, 64, 96, 128, 128] if call == "train" or kind == "fp32" else [32, 64, 64, 80, 96, 128, 128, 128, 256])
        blocks = (rng.choice([16, 32, 64, 80, 128, 128]), rng.choice([16, 48, 64, 80, 128, 128, 256]))
        causal = rng.random() < 0.7
        keep = rng.choice([0.1, 0.2, 0.3, 0.5, 0.7])
        k_len = None
        if call == "schedule":                                     # a few new tokens on a long context
            n = log_int(1, 64)
            q_len, k_len = (max(1, n // 2), n), tuple(sorted((log_int(1024, 32768), log_int(1024, 32768))))
            causal = True
        elif call == "csr":
            heads_k, batch = 1, rng.choice([4, 8, 16, 32])
            heads_q = rng.choice([1, 1, 2, 4, 8])
            q_len = (log_int(256, 8192),) * 2
        else:
            q_len = tuple(sorted((log_int(16, 16384), log_int(16, 16384))))
            if rng.random() < 0.25 and call != "train":            # new tokens behind a longer context
                k_len = tuple(sorted(n + log_int(64, 16384) for n in q_len))
        case = _case(call, batch, q_len, k_len, (heads_q, heads_k), head_dim, blocks, causal, keep, dtype=dtype,
                     round_to=rng.choice([1, 1, 16]), len_seed=rng.randrange(1 << 30))
        cu_q, cu_k = _lengths(case)
        blocks_q, blocks_k = _blocks(cu_q, case["q_block"])[-1], _blocks(cu_k, case["k_block"])[-1]
        elements = max(int(cu_q[-1]) * heads_q, int(cu_k[-1]) * heads_k) * head_dim
        if work(case)["flops"] <= _most(call, dtype) and heads_k * int(blocks_q) * int(blocks_k) <= 1 << 26 and elements <= 1 << 29:
            return case


def _lengths(case):
    """Cumulative lengths of the samples' queries and keys."""
    rng = np.random.default_rng(case["len_seed"])
    r = case["round_to"]

    def lens(lo, hi):
        return np.maximum(rng.integers(lo, hi + 1, size=case["batch"]) // r * r, min(r, hi))

    q = lens(case["q_min"], case["q_max"])
    k = lens(case["k_min"], case["k_max"]) if case["k_max"] else q
    return np.concatenate([[0], np.cumsum(q)]), np.concatenate([[0], np.cumsum(k)])


def _blocks(cu, size):
    """First block of every sample, and their number at the end."""
    return np.concatenate([[0], np.cumsum((np.diff(cu) + size - 1) // size)])


def _last_seen(case, b, cu_q, cu_k):
    """Per q-block of sample b: the last in-sample k-block that a row of it may see (negative: none)."""
    ql, kl = int(cu_q[b + 1] - cu_q[b]), int(cu_k[b + 1] - cu_k[b])
    n = -(-ql // case["q_block"])
    last = -(-kl // case["k_block"]) - 1
    if not case["causal"]:
        return np.full(n, last)
    row = np.minimum((np.arange(n) + 1) * case["q_block"], ql) - 1 + (kl - ql)
    return np.where(row < 0, -1, np.minimum(row // case["k_block"], last))


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    dtype = DTYPES[case["dtype"]]
    cu_q, cu_k = _lengths(case)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device=dev, dtype=dtype)

    s = dict(case=case)
    s["q"] = normal(int(cu_q[-1]), case["heads_q"], case["head_dim"])
    s["k"] = normal(int(cu_k[-1]), case["heads_k"], case["head_dim"])
    s["v"] = normal(int(cu_k[-1]), case["heads_k"], case["head_dim"])
    s["cu_q"] = torch.as_tensor(cu_q, dtype=torch.int32, device=dev)
    s["cu_k"] = torch.as_tensor(cu_k, dtype=torch.int32, device=dev)
    first_q, first_k = _blocks(cu_q, case["q_block"]), _blocks(cu_k, case["k_block"])
    mask = torch.rand(case["heads_k"], int(first_q[-1]), int(first_k[-1]), generator=g, device=dev) < case["keep"]
    if case["causal"]:
        seen = [_last_seen(case, b, cu_q, cu_k) for b in range(case["batch"])]
        rows = np.concatenate([first_q[b] + np.flatnonzero(x >= 0) for b, x in enumerate(seen)])
        cols = np.concatenate([first_k[b] + x[x >= 0] for b, x in enumerate(seen)])
        mask[:, torch.as_tensor(rows, device=dev), torch.as_tensor(cols, device=dev)] = True
    s["mask"] = mask
    if case["call"] in ("kept", "train"):
        s["tables"] = hb.calculate_blocks(s["cu_q"], case["q_block"]) + hb.calculate_blocks(s["cu_k"], case["k_block"])
    elif case["call"] == "schedule":
        s["schedule"] = hb.build_schedule(s["q"], s["k"], s["cu_q"], s["cu_k"], mask, case["q_block"], case["k_block"], case["causal"])
    elif case["call"] == "csr":                                     # pairs of different samples are not listed
        of_q = torch.as_tensor(np.repeat(np.arange(case["batch"]), np.diff(first_q)), device=dev)
        of_k = torch.as_tensor(np.repeat(np.arange(case["batch"]), np.diff(first_k)), device=dev)
        s["csr"] = csr_of_mask(mask & (of_q[:, None] == of_k[None, :]))
        s["blocks"] = int(first_q[-1]), int(first_k[-1])
        del s["mask"]
    if case["call"] == "train":
        s["d_out"] = normal(*s["q"].shape)
        for n in "qkv":
            s[n].requires_grad_(True)
    return s


def run(s):
    case, call = s["case"], s["case"]["call"]
    data = s["q"], s["k"], s["v"]
    blocks = case["q_block"], case["k_block"], case["causal"]
    if call == "forward":
        return hb.HBSAttention(*data, s["cu_q"], s["cu_k"], s["mask"], *blocks, None)
    if call == "kept":
        return hb.HBSAttention(*data, s["cu_q"], s["cu_k"], s["mask"], *blocks, None, "auto", *s["tables"])
    if call == "tables":
        tables = hb.calculate_blocks(s["cu_q"], case["q_block"]) + hb.calculate_blocks(s["cu_k"], case["k_block"])
        return hb.HBSAttention(*data, s["cu_q"], s["cu_k"], s["mask"], *blocks, None, "auto", *tables), tables
    if call == "schedule":
        return hb.attention_with_schedule(*data, s["schedule"])
    if call == "lse":
        return hb.HBSAttention_with_lse(*data, s["cu_q"], s["cu_k"], s["mask"], *blocks)
    if call == "csr":
        return hb.HBSAttention_csr(*data, s["cu_q"], s["cu_k"], *s["csr"], *s["blocks"], *blocks)
    out = hb.HBSAttention(*data, s["cu_q"], s["cu_k"], s["mask"], *blocks, None, "auto", *s["tables"])
    return (out,) + torch.autograd.grad(out, data, s["d_out"])


def work(case):
    """Expected over the mask's draw.  FLOPs of the active block pairs (a pair on the causal diagonal counts in
    full, as the package's benchmark counts it): two products forward, five more backward.  Bytes: q, out and their gradients
    whole, k and v where at least one q-block of the head attends to them, and the mask inside the samples."""
    cu_q, cu_k = _lengths(case)
    size = 4 if case["dtype"] == "float32" else 2
    pairs, touched, mask = 0.0, 0.0, 0.0
    for b in range(case["batch"]):
        ql, kl = int(cu_q[b + 1] - cu_q[b]), int(cu_k[b + 1] - cu_k[b])
        last = _last_seen(case, b, cu_q, cu_k)
        rows_q = np.minimum(case["q_block"], ql - np.arange(len(last)) * case["q_block"])
        n_k = -(-kl // case["k_block"])
        rows_k = np.minimum(case["k_block"], kl - np.arange(n_k) * case["k_block"]).astype(np.float64)
        upto = np.concatenate([[0.0], np.cumsum(rows_k)])
        keys = case["keep"] * upto[last + 1]
        if case["causal"]:
            keys = keys + np.where(last >= 0, (1.0 - case["keep"]) * rows_k[np.maximum(last, 0)], 0.0)
        pairs += float((rows_q * keys).sum())
        seen_by = (last[None, :] >= np.arange(n_k)[:, None]).sum(axis=1)
        forced = (last[None, :] == np.arange(n_k)[:, None]).any(axis=1) & case["causal"]
        touched += float((rows_k * np.where(forced, 1.0, 1.0 - (1.0 - case["keep"]) ** seen_by)).sum())
        mask += float((last + 1).sum())
    train = case["call"] == "train"
    flops = pairs * case["heads_q"] * case["head_dim"] * (14.0 if train else 4.0)
    rows = int(cu_q[-1]) * case["heads_q"] * case["head_dim"] * size
    keys = touched * case["heads_k"] * case["head_dim"] * size
    data = 4.0 * rows + 4.0 * keys if train else 2.0 * rows + 2.0 * keys
    mask_bytes = mask * case["heads_k"] if case["call"] not in ("schedule", "csr") else 4.0 * case["keep"] * mask * case["heads_k"]
    lse = 4.0 * int(cu_q[-1]) * case["heads_q"] if case["call"] == "lse" else 0.0
    return {"bytes": data + mask_bytes + lse, "flops": flops}


def tolerance(case):
    """Results carry the rounding of their type: sums are taken in 32 bits whatever it is, 16-bit results and probabilities are
    rounded to 8 (bfloat16) or 11 (float16) bits."""
    return {"rel": {"float32": 1e-5, "bfloat16": 1e-2, "float16": 2e-3}[case["dtype"]]}
