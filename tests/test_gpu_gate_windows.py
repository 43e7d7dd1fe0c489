"""The tensor-core gate where its bookkeeping has edges: candidate counts around a window of 64 scores,
around the bounding pass (more than 16 candidates; 128 at either end bound) and odd numbers of query tiles,
with score patterns that let every candidate pass its bar, or none after the first.

Scores are whole numbers that both 16-bit types hold, so the rule decides alone: score descending,
ties to the lower id, then the own block; the result is the same, bit for bit."""

import pytest
import torch

import moba_triton_b200 as moba

pytestmark = pytest.mark.gpu

BS = 128


def patterns(blocks, d, g):
    """Block means [blocks, d]: column c is the score of every block for a query that is one-hot in c."""
    ids = torch.arange(blocks)
    kb = torch.randint(-120, 121, (blocks, d), generator=g)
    kb[:, 0] = ids % 241 - 120                                # rising: every candidate enters the list
    kb[:, 1] = 120 - ids % 241                                # falling: none after the first few
    kb[:, 2] = 7                                              # all equal: the lowest ids
    kb[:, 3] = torch.where(ids % 64 >= 32, 100, -100)         # one half of every window
    kb[:, 4] = torch.where(ids % 32 == 31, ids % 100, -5)     # the last column of either half
    kb[:, 5] = -(ids // 64)                                   # ties in windows, falling
    return kb


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("d,top_k", [(64, 8), (64, 3), (128, 8), (128, 9)])
@pytest.mark.parametrize("blocks", [1, 2, 17, 18, 33, 64, 65, 66, 129, 257, 258, 321, 386, 449, 641])
def test_selection_is_the_rule(blocks, d, top_k, dtype, device):
    g = torch.Generator().manual_seed(blocks * 3 + d)
    kb = patterns(blocks, d, g)
    s = blocks * BS - 37
    hot = torch.randint(0, d, (s,), generator=g)
    hot[::5] = torch.arange(0, s, 5) // 5 % 6
    q = torch.nn.functional.one_hot(hot, d)[:, None].to(dtype)
    cfg = moba.MoBAConfig(BS, top_k, dtype=dtype)
    got = moba.gate_select(q[None].to(device), kb[None, None].to(dtype).to(device), cfg).cpu()[0, 0]

    scores = kb.t()[hot].double()                             # [s, blocks]
    own = torch.arange(s) // BS
    ids = torch.arange(blocks)
    scores[ids[None] >= own[:, None]] = -float("inf")
    order = torch.sort(scores, dim=-1, descending=True, stable=True)
    take = min(top_k - 1, blocks)
    best = torch.where(order.values[:, :take] > -float("inf"), order.indices[:, :take], blocks)
    want = torch.full((s, top_k), blocks)
    want[:, :take] = best
    want[:, top_k - 1] = own
    want = want.sort(dim=-1).values
    want = torch.where(want == blocks, -1, want).to(got.dtype)
    assert torch.equal(got, want)
