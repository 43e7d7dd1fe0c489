"""The tensor-core gates against float64 scores where floating-point details decide: signed zeros.

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
