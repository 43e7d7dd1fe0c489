"""Work items that the CTAs claim from a counter, in groups of rows, against the fixed deal that the calls with
an index keep: O and dQ do not depend on who runs an item, so they are the same bits; dK and dV are sums over
items that may be cut elsewhere. Sizes are the smallest that claim (tiles per SM), with a last group that is
short, sequences of less than a block beside long ones, and blocks that nobody selects."""

import pytest
import torch

import moba_triton_b200 as moba
from helpers import max_abs_error

pytestmark = pytest.mark.gpu

CASES = [
    # lengths, q heads, kv heads, head_dim, top_k, own block always selected
    ([9000, 100, 7000, 5001, 8000, 6400, 300, 9100, 4000, 6000, 5099], 16, 16, 128, 8, True),   # groups of 32 of 176 rows
    ([30000, 77, 9923], 8, 2, 128, 8, True),                                                    # one group of six rows
    ([24000, 24000], 16, 2, 64, 8, False),                                                      # blocks without a query
]


@pytest.mark.parametrize("lens,hq,hkv,d,top_k,own", CASES, ids=["groups", "one-group", "no-own-block"])
def test_claimed_items_equal_dealt_ones(lens, hq, hkv, d, top_k, own, device):
    tokens = sum(lens)
    assert tokens * hq * top_k / 128 / 148 >= (192 if d == 64 else 96)
    cfg = moba.MoBAConfig(128, top_k, always_select_current=own)
    g = torch.Generator(device=device).manual_seed(tokens)
    q, k, v, do = (torch.randn((1, tokens, h, d), generator=g, device=device, dtype=torch.bfloat16) for h in (hq, hkv, hkv, hq))
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device=device)
    kw = dict(cu_seqlens=cu, max_seqlen=max(lens))
    index = moba.build_csc_fused(q, k, cfg, **kw)
    got = []
    for args in (dict(index=index), kw):
        leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
        out = moba.moba_attention(*leaves, cfg, **args)
        out.backward(do)
        got.append([out.detach()] + [t.grad for t in leaves])
    dealt, claimed = got
    live = ~torch.isnan(dealt[0])                             # no own block: the first rows select nothing
    assert torch.equal(live, ~torch.isnan(claimed[0])) and (own == bool(live.all()))
    assert torch.equal(dealt[0][live], claimed[0][live])
    assert torch.equal(dealt[1], claimed[1])
    for a, b in zip(dealt[2:], claimed[2:]):
        # float32 sums of the same terms in other groups, rounded to bfloat16: a step of the largest sum
        assert max_abs_error(a, b) <= 2.0 ** -7 * float(a.float().abs().max())
        assert torch.equal(a == 0, b == 0)
