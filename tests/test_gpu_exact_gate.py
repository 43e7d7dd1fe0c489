"""The exact tensor-core gate against float64 scores where its rounding is decided by its error
bound: scores a little off the middle between two values of the input type, hidden behind terms
that cancel; signed zeros; infinities, NaN and numbers whose squares leave the range of float32.

Keys are constant within a block, so the block means are the keys themselves. The gate runs inside
the whole op only; which blocks it selected is read off the output, with one-hot values per block."""

import pytest
import torch

import moba_triton_b200 as moba

pytestmark = pytest.mark.gpu

BS = 32


def selected_by_the_op(q, kb, cfg):
    """[S, H, blocks]: does the output of row (s, h) hold block b's value. q [S,H,D]; kb [blocks,1,D]."""
    s, h, d = q.shape
    nb = kb.shape[0]
    k = kb.repeat_interleave(cfg.block_size, dim=0)[None, :s].contiguous()
    out = []
    for b0 in range(0, nb, d):
        v = torch.zeros(nb, 1, d, device=q.device, dtype=q.dtype)
        n = min(d, nb - b0)
        v[b0:b0 + n, 0, :n] = torch.eye(n, device=q.device, dtype=q.dtype)
        v = v.repeat_interleave(cfg.block_size, dim=0)[None, :s].contiguous()
        out.append(moba.moba_forward(q[None], k, v, cfg)[0, :, :, :n])
    return torch.cat(out, -1)


def selected_by_exact_scores(q, kb, cfg):
    """The rule itself: float64 scores, rounded to float32 and to the type; ties to the lower id;
    NaN and -inf are never selected; the own block always is."""
    s, nb = q.shape[0], kb.shape[0]
    dots = torch.einsum("shd,nd->shn", q.double(), kb[:, 0].double())
    scores = dots.float().to(q.dtype).double() + 0.0
    own = torch.arange(s, device=q.device) // cfg.block_size
    ids = torch.arange(nb, device=q.device)
    scores[(ids[None, :] >= own[:, None])[:, None].expand_as(scores)] = -float("inf")
    scores = torch.where(torch.isnan(scores), -float("inf"), scores)
    order = torch.sort(scores, dim=-1, descending=True, stable=True)     # stable: ties stay in order of id
    mask = torch.zeros_like(scores, dtype=torch.bool)
    take = min(cfg.top_k - 1, nb)
    mask.scatter_(-1, order.indices[..., :take], order.values[..., :take] > -float("inf"))
    mask |= (ids[None, :] == own[:, None])[:, None]
    return mask


def check(q, kb, cfg, unseen=()):
    """`unseen`: blocks without a finite key, whose share of the output cannot be read."""
    got, want = selected_by_the_op(q, kb, cfg) > 0, selected_by_exact_scores(q, kb, cfg)
    for b in unseen:
        got[..., b] = want[..., b]
    assert torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("d,top_k", [(64, 4), (64, 12), (64, 17), (128, 9), (128, 13)])
@pytest.mark.parametrize("blocks", [20, 64, 150])
def test_scores_beside_a_rounding_boundary(blocks, d, top_k, dtype, device):
    """Scores (n + 1/2) steps of the type plus or minus a trace, with B - B added to them: a sum in
    float32 that keeps 24 bits of its largest term loses the trace for most of the B drawn."""
    g = torch.Generator().manual_seed(blocks * 7 + d)
    bits = 8 if dtype == torch.bfloat16 else 11              # significant bits: steps of 2^(1 - bits) in [1, 2)
    s = blocks * BS - 3
    ints = lambda lo, hi, *shape: torch.randint(lo, hi + 1, shape, generator=g).double()
    q = torch.zeros(s, 1, d, dtype=torch.float64)
    kb = torch.zeros(blocks, 1, d, dtype=torch.float64)
    q[:, 0, 0] = 2.0 ** ints(0, 10, s)                       # B = q0 k0, -B = q0 k1 and q0 k17 (another step of 16)
    kb[:, 0, 0] = 1.0
    near = torch.rand(blocks, generator=g) < 0.5
    kb[:, 0, 1] = torch.where(near, -1.0, 0.0)
    kb[:, 0, 17] = torch.where(near, 0.0, -1.0)
    q[:, 0, 1] = q[:, 0, 17] = q[:, 0, 0]
    q[:, 0, 2:5] = 1.0
    kb[:, 0, 2] = 1.0 + ints(0, 3, blocks) * 2.0 ** (1 - bits)
    kb[:, 0, 3] = 2.0 ** -bits * ints(0, 1, blocks)          # half a step, or none
    kb[:, 0, 4] = ints(-1, 1, blocks) * 2.0 ** -ints(12, 14, blocks)   # the trace
    q *= 2.0 ** ints(-1, 1, s)[:, None, None] if dtype == torch.bfloat16 else 1.0
    q, kb = q.to(dtype).to(device), kb.to(dtype).to(device)
    check(q, kb, moba.MoBAConfig(BS, top_k, dtype=dtype))


@pytest.mark.parametrize("case", ["zero_rows", "tiny", "huge", "same_head"])
@pytest.mark.parametrize("blocks", [20, 60])
def test_rows_without_a_finite_bound(blocks, case, device):
    """zero_rows: query rows of zeros (padding) beside another head whose keys hold an infinity.
    tiny / huge: squares below / above the range of float32. same_head: the infinity, and a NaN,
    among the candidates themselves."""
    dtype, d = torch.bfloat16, 64
    cfg = moba.MoBAConfig(BS, 6, dtype=dtype)
    g = torch.Generator().manual_seed(blocks)
    s = blocks * BS - 7
    q = torch.randint(-3, 4, (s, 1, d), generator=g).to(dtype).to(device)
    kb = torch.randint(-1, 2, (blocks, 1, d), generator=g).to(dtype).to(device)
    if case == "tiny":
        return check(q * 2.0 ** -80, kb * 2.0 ** 20, cfg)
    if case == "huge":
        return check(q * 2.0 ** 80, kb * 2.0 ** -80, cfg)
    if case == "same_head":
        kb[blocks // 2, 0, 5] = float("inf")
        kb[blocks // 3, 0, 6] = float("nan")
        q[::3] = 0
        return check(q, kb, cfg, unseen=(blocks // 2, blocks // 3))
    q[::2] = 0
    want = selected_by_exact_scores(q, kb, cfg)
    # two KV heads: the first as drawn, the second with an infinite key at its start
    k = kb.repeat_interleave(BS, dim=0)[None, :s]
    k2 = k.clone()
    k2[0, 3, 0, 0] = float("inf")
    v = torch.zeros(blocks, 1, d, device=device, dtype=dtype)
    v[:, 0, :blocks] = torch.eye(blocks, device=device, dtype=dtype)
    v = v.repeat_interleave(BS, dim=0)[None, :s]
    out = moba.moba_forward(torch.cat([q[None], q[None]], 2), torch.cat([k, k2], 2), torch.cat([v, v], 2), cfg)
    assert torch.equal(out[0, :, :1, :blocks] > 0, want)


@pytest.mark.parametrize("block", [32, 128], ids=["exact", "plain"])
@pytest.mark.parametrize("rows", ["tiny", "zero"])
def test_a_negative_zero_ties_with_zero(block, rows, device):
    """float16 scores that round to zero from either side are one score: the lower id wins. Rows of
    zeros score zero everywhere and select the first blocks."""
    dtype, d, blocks = torch.float16, 64, 60
    cfg = moba.MoBAConfig(block, 5, dtype=dtype)
    g = torch.Generator().manual_seed(3)
    s = blocks * block
    q = (torch.randint(-1, 2, (s, 1, d), generator=g) * 2.0 ** -14).to(dtype).to(device)
    kb = (torch.randint(-1, 2, (blocks, 1, d), generator=g) * 2.0 ** -14).to(dtype).to(device)
    if rows == "zero":
        q[::2] = 0
    check(q, kb, cfg)


def selected_by_the_packed_op(qs, kbs, cfg):
    """As `selected_by_the_op`, for sequences packed into one call: a list of [S_i, H, blocks_i]."""
    d, lens = qs[0].shape[2], [q.shape[0] for q in qs]
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device=qs[0].device)
    keys = lambda rows: torch.cat([r.repeat_interleave(cfg.block_size, dim=0)[:n] for r, n in zip(rows, lens)])[None]
    out = [[] for _ in qs]
    for b0 in range(0, max(kb.shape[0] for kb in kbs), d):
        v = [torch.eye(kb.shape[0], device=kb.device, dtype=kb.dtype)[:, b0:b0 + d] for kb in kbs]
        v = [torch.nn.functional.pad(x, (0, d - x.shape[1]))[:, None] for x in v]
        got = moba.moba_forward(torch.cat(qs)[None], keys(kbs), keys(v), cfg, cu_seqlens=cu, max_seqlen=max(lens))
        for i, o in enumerate(got[0].split(lens)):
            out[i].append(o)
    return [torch.cat(o, -1)[..., :kb.shape[0]] for o, kb in zip(out, kbs)]


def ladder(blocks, rows, d, dtype, tiles, g):
    """Queries and block means whose every score lies on the middle between two values of the type, or a trace
    beside it: any of them is unsure, and passes or not by its whole part, of which the rows have five kinds. They
    are spread over the rows by tiles of 128, so that all of a warp's lists fill up together, or row by row."""
    ids = torch.arange(blocks)
    half, span = (0.5, 128) if dtype == torch.bfloat16 else (0.0625, 64)       # half a step of the type in [128, 256)
    whole = torch.stack([ids % span,                          # rising: all enter the list
                         span - 1 - ids % span,               # falling: none after the first
                         torch.full_like(ids, 7),             # equal: the trace and the id decide
                         torch.where(ids < 256, ids % 3, span // 2 + ids % 5),   # high past the first 256
                         torch.randint(0, span, (blocks,), generator=g)])
    kb = torch.zeros(blocks, 1, d, dtype=torch.float64)
    q = torch.zeros(rows, 2, d, dtype=torch.float64)
    for h in range(2):
        kind = (torch.arange(rows) // (128 if tiles else 1) + h) % 5
        q[:, h] = torch.nn.functional.one_hot(3 * kind, d) + torch.nn.functional.one_hot(3 * kind + 1, d) + torch.nn.functional.one_hot(3 * kind + 2, d)
    for p in range(5):
        kb[:, 0, 3 * p] = 128.0 + whole[p]
        kb[:, 0, 3 * p + 1] = half
        kb[:, 0, 3 * p + 2] = torch.randint(-1, 2, (blocks,), generator=g) * 2.0 ** -10
    return q.to(dtype), kb.to(dtype)


@pytest.mark.parametrize("tiles", [True, False], ids=["by-tiles", "by-rows"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("d,top_k", [(64, 4), (64, 12), (64, 17), (128, 13)])
@pytest.mark.parametrize("blocks", [255, 256, 257, 321, 577])
def test_unsure_scores_past_the_bounding_pass(blocks, d, top_k, dtype, tiles, device):
    """More candidates than the 256 that bound the rest; every score is taken again in float64, so the
    lists of those that wait fill up in the middle of a window, with lanes that lag a window behind."""
    g = torch.Generator().manual_seed(blocks + d + top_k)
    q, kb = ladder(blocks, blocks * BS - 11, d, dtype, tiles, g)
    check(q.to(device), kb.to(device), moba.MoBAConfig(BS, top_k, dtype=dtype))


@pytest.mark.parametrize("block,d,top_k", [(32, 64, 12), (64, 128, 5), (128, 64, 17), (128, 128, 13)])
def test_unsure_scores_in_packed_sequences(block, d, top_k, device):
    """Odd and even numbers of query tiles, sequences of one row and of less than a block, starts anywhere."""
    g = torch.Generator().manual_seed(block + d)
    cfg = moba.MoBAConfig(block, top_k)
    qs, kbs = [], []
    for n in (1, 300 * block - 5, 127, 3 * 128, 40 * block + 1, 2 * 128 - 1, 259 * block, 17):
        q, kb = ladder(-(-n // block), n, d, torch.bfloat16, n % 2 == 0, g)
        qs.append(q.to(device))
        kbs.append(kb.to(device))
    for q, kb, got in zip(qs, kbs, selected_by_the_packed_op(qs, kbs, cfg)):
        assert torch.equal(got > 0, selected_by_exact_scores(q, kb, cfg))
