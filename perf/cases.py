"""The work whose time matters to users of this engine, as a list of measurable cases.

A case is one call of the public API as a program makes it: an attention forward
(`moba_forward`, inference and prefill) or a training step of the op (`moba_attention` and
its gradients). `listed()` names the fixed cases, `draw()` gives further ones from the same
ranges: sequences of 256 to 524 288 tokens with odd lengths among them, batches of one to
four, packed batches of ragged sequences, plain and grouped-query heads, head_dim 64 and
128, bfloat16 and float16 with blocks of 128 keys, smaller blocks, float32, and two to
twelve blocks per query.
"""

import math
import random

import torch

import moba_triton_b200 as moba

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def _case(name, op, *, seq, hq, hkv, d, dtype="bf16", batch=1, block=128, top_k=8, n_seq=0, lengths_seed=0,
          shortest=0, longest=0, align=1, skew=False):
    """`seq` is the length of each batch row; with `n_seq` sequences packed it is the token
    total, and their lengths are log-uniform between `shortest` and `longest` before scaling."""
    c = dict(op=op, batch=batch, seq=seq, hq=hq, hkv=hkv, d=d, dtype=dtype, block=block, top_k=top_k,
             n_seq=n_seq, lengths_seed=lengths_seed, shortest=shortest, longest=longest, align=align, skew=skew)
    return dict(c, name=name) if name else c


def listed():
    return [
        # The smallest training step: a short sequence whose last block is cut short, two query
        # heads to a KV head. Launches and host work are what it costs.
        _case("step_1k", "train", seq=1000, hq=4, hkv=2, d=64, top_k=4),
        # A short grouped-query prompt, forward only: time to first token of a small request.
        _case("prefill_2k_gqa", "forward", seq=2048, hq=8, hkv=2, d=128),
        # A prompt of ordinary length, forward only.
        _case("prefill_8k", "forward", seq=8192, hq=4, hkv=4, d=64),
        # A serving batch: sixteen prompts of ragged, unaligned lengths packed into one call, in
        # float16, with the head layout of a grouped-query model.
        _case("prefill_packed_f16", "forward", seq=40000, hq=32, hkv=8, d=128, dtype="f16",
              n_seq=16, lengths_seed=3, shortest=300, longest=9000),
        # A long prompt with a wider selection: twelve blocks per query.
        _case("prefill_64k_top12", "forward", seq=65536, hq=4, hkv=4, d=64, top_k=12),
        # float32, forward: what a numerical check of a model runs.
        _case("forward_4k_f32", "forward", seq=4096, hq=4, hkv=4, d=64, dtype="f32"),
        # Finer blocks of 64 keys on a batch of two, training.
        _case("step_8k_block64", "train", batch=2, seq=8192, hq=4, hkv=4, d=128, block=64),
        # The benchmark's own shape: long-context training, one sequence.
        _case("step_128k", "train", seq=131072, hq=4, hkv=4, d=64),
        # Long-context training with a whole layer's grouped-query heads.
        _case("step_128k_gqa", "train", seq=131072, hq=32, hkv=8, d=128),
        # Packed training batch: 32 sequences of 1k to 32k tokens.
        _case("step_256k_packed", "train", seq=262144, hq=16, hkv=16, d=128, n_seq=32, lengths_seed=1,
              shortest=1024, longest=32768, align=128),
        # The longest context, with selections that crowd onto the early blocks.
        _case("step_512k_skewed", "train", seq=524288, hq=32, hkv=8, d=128, skew=True),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(("padded", "padded", "padded", "packed", "packed", "small_block", "f32"))
    op = rng.choice(("train", "forward"))
    if kind == "f32":
        hq, hkv = rng.choice(((2, 2), (4, 4), (4, 2), (8, 2)))
        return _case(None, "forward", seq=_log_uniform(rng, 256, 8192), hq=hq, hkv=hkv, d=rng.choice((64, 64, 128)),
                     dtype="f32", top_k=rng.choice((3, 4, 8)))
    if kind == "small_block":
        hq, hkv = rng.choice(((2, 2), (4, 4), (8, 2)))
        return _case(None, op, batch=rng.choice((1, 2)), seq=_log_uniform(rng, 512, 16384), hq=hq, hkv=hkv,
                     d=rng.choice((64, 128)), dtype=rng.choice(("bf16", "bf16", "f16")), block=rng.choice((32, 64, 64)),
                     top_k=rng.choice((4, 8)))
    hq, hkv = rng.choice(((4, 4), (4, 4), (4, 2), (4, 1), (8, 2), (16, 4), (16, 16), (32, 8)))
    d, dtype = rng.choice((64, 128)), rng.choice(("bf16", "bf16", "bf16", "f16"))
    top_k = rng.choice((2, 3, 4, 6, 8, 8, 8, 12))
    if kind == "packed":
        n = rng.choice((2, 4, 8, 16, 32))
        tokens = _log_uniform(rng, 256 * n, min(262144, 16384 * n))
        return _case(None, op, seq=tokens, hq=hq, hkv=hkv, d=d, dtype=dtype, top_k=top_k, n_seq=n,
                     lengths_seed=rng.randrange(1 << 20), shortest=256, longest=8192)
    batch = 1 if top_k == 12 else rng.choice((1, 1, 2, 4))
    seq = _log_uniform(rng, 256, 65536 if top_k == 12 else 131072)
    if rng.random() < 0.5:
        seq = max(256, seq // 128 * 128)
    return _case(None, op, batch=batch, seq=max(256, min(seq, 262144 // batch)), hq=hq, hkv=hkv, d=d, dtype=dtype,
                 top_k=top_k)


def lengths(case):
    """The sequence lengths of a case: fixed by the case, not by the seed of its values."""
    if not case["n_seq"]:
        return [case["seq"]] * case["batch"]
    g = torch.Generator().manual_seed(case["lengths_seed"])
    u = torch.rand(case["n_seq"], generator=g, dtype=torch.float64)
    raw = torch.exp(math.log(case["shortest"]) + u * math.log(case["longest"] / case["shortest"]))
    a = case["align"]
    out = [max(a, int(round(float(x) / a)) * a) for x in raw * (case["seq"] / float(raw.sum()))]
    out[out.index(max(out))] += case["seq"] - sum(out)
    return out


def prepare(case, seed):
    """q, k, v (and the upstream gradient of a training step) i.i.d. N(0, 1), the configuration
    and, for a packed batch, its sequence offsets. A skewed case adds a direction of norm 2 per
    KV head to its queries and to the first tenth of its keys."""
    dev, dt = torch.device("cuda"), DTYPES[case["dtype"]]
    g = torch.Generator(device=dev).manual_seed(seed)
    b, s, hq, hkv, d = case["batch"], case["seq"], case["hq"], case["hkv"], case["d"]
    q = torch.randn((b, s, hq, d), generator=g, device=dev, dtype=dt)
    k = torch.randn((b, s, hkv, d), generator=g, device=dev, dtype=dt)
    v = torch.randn((b, s, hkv, d), generator=g, device=dev, dtype=dt)
    if case["skew"]:
        u = torch.randn((hkv, d), generator=g, device=dev)
        u = (2.0 * u / u.norm(dim=-1, keepdim=True)).to(dt)
        q += u.repeat_interleave(hq // hkv, dim=0)
        k[:, : s // 10] += u
    state = dict(op=case["op"], q=q, k=k, v=v, cfg=moba.MoBAConfig(block_size=case["block"], top_k=case["top_k"], dtype=dt),
                 packing={})
    if case["n_seq"]:
        lens = lengths(case)
        ends = [0]
        for n in lens:
            ends.append(ends[-1] + n)
        state["packing"] = dict(cu_seqlens=torch.tensor(ends, dtype=torch.int32, device=dev), max_seqlen=max(lens))
    if case["op"] == "train":
        state["do"] = torch.randn((b, s, hq, d), generator=g, device=dev, dtype=dt)
        for t in (q, k, v):
            t.requires_grad_(True)
    return state


def run(state):
    q, k, v, cfg = state["q"], state["k"], state["v"], state["cfg"]
    if state["op"] == "forward":
        return moba.moba_forward(q, k, v, cfg, **state["packing"])
    out = moba.moba_attention(q, k, v, cfg, **state["packing"])
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["do"])
    return {"out": out.detach(), "dq": dq, "dk": dk, "dv": dv}


def work(case):
    """Scores of every (query, past block) pair, attention over the (query, key) pairs of the
    selected blocks (4 D flops forward, 2.5 times as much again backward); inputs read once,
    outputs written once."""
    bs, take, d = case["block"], case["top_k"] - 1, case["d"]
    attended = candidates = tokens = 0
    for n in lengths(case):
        tokens += n
        for j in range(-(-n // bs)):
            rows = min(bs, n - j * bs)
            attended += rows * (rows + 1) // 2 + rows * min(j, take) * bs
            candidates += rows * j
    train = case["op"] == "train"
    size = 4 if case["dtype"] == "f32" else 2
    q_bytes, k_bytes = tokens * case["hq"] * d * size, tokens * case["hkv"] * d * size
    return {"flops": case["hq"] * d * (2.0 * candidates + 4.0 * attended * (3.5 if train else 1.0)),
            "bytes": float(q_bytes * (4 if train else 2) + k_bytes * (4 if train else 2))}


def tolerance(case):
    # 16-bit types: probabilities, partial outputs and gradients are rounded to the type, and a
    # query whose last two candidate blocks score within one rounding step of each other may take
    # the other one, which changes that query's rows wholly ("max").
    return {"f32": {"rel": 1e-5}, "bf16": {"rel": 1e-2, "max": 0.9}, "f16": {"rel": 5e-3, "max": 0.9}}[case["dtype"]]
