"""Work items that the CTAs claim from a counter, in groups of rows, against the fixed deal that the calls with
an index keep: results do not depend on who runs an item, and both cut the columns alike, so they are the same
bits. Sizes are above the lines from which on items are claimed (tiles per SM), with a last group that is short,
sequences of less than a block beside long ones, and blocks that nobody selects, whose gradients are zeros that
have to be written."""

import pytest
import torch

import moba_triton_b200 as moba
from helpers import max_abs_error
from moba_triton_b200 import _lib
from moba_triton_b200.tuning import launch_plan

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


CLAIMED = [
    # lengths, q heads, kv heads, head_dim, top_k, own block always selected
    ([9000, 100, 7000, 5001, 8000, 6400, 300, 9100, 4000, 6000, 5099], 16, 16, 128, 8, True),   # groups of 32 of 176 rows
    ([30000, 77, 9923], 8, 2, 128, 8, True),                                                    # one group of six rows
    ([29000, 29000], 16, 2, 64, 8, False),                                                      # blocks without a query
    ([40, 300, 129, 50000, 128, 1, 500, 77, 256], 16, 2, 64, 8, False),                         # ... whose rows are mostly padding
    ([40000, 64, 1000, 130], 8, 2, 128, 8, False),
]


@pytest.mark.parametrize("lens,hq,hkv,d,top_k,own", CLAIMED, ids=["groups", "one-group", "no-own-block", "short-beside-long", "short-beside-long-128"])
def test_gradients_of_claimed_items_are_the_same_bits(lens, hq, hkv, d, top_k, own, device):
    tokens = sum(lens)
    line = 192 if d == 64 else 96
    assert tokens * hq * top_k / 128 / 148 >= (max(line, 6 * hq // hkv * top_k) if len(lens) <= 2 else line)
    cfg = moba.MoBAConfig(128, top_k, always_select_current=own)
    g = torch.Generator(device=device).manual_seed(tokens)
    q, k, v, do = (torch.randn((1, tokens, h, d), generator=g, device=device, dtype=torch.bfloat16) for h in (hq, hkv, hkv, hq))
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device=device)
    kw = dict(cu_seqlens=cu, max_seqlen=max(lens))
    index = moba.build_csc_fused(q, k, cfg, **kw)
    assert index.chunk_tiles == launch_plan(q.shape, hkv, q.dtype, cfg, **kw)["chunk_tiles"]
    got = []
    for args in (dict(index=index), kw):
        leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
        out = moba.moba_attention(*leaves, cfg, **args)
        del_me = [torch.full_like(t, float("nan")) for t in (q, k, v)]     # the memory that the gradients will get
        del del_me
        out.backward(do)
        got.append([out.detach()] + [t.grad for t in leaves])
    dealt, claimed = got
    live = ~torch.isnan(dealt[0])                             # no own block: the first rows select nothing
    assert torch.equal(live, ~torch.isnan(claimed[0])) and (own == bool(live.all()))
    assert torch.equal(dealt[0][live], claimed[0][live])
    assert torch.equal(dealt[1], claimed[1])
    starts = cu[:-1].tolist()
    for a, b in zip(dealt[2:], claimed[2:]):
        assert torch.equal(a, b)
        assert not torch.isnan(b).any()
        if not own:                                           # nobody selects the last block of a sequence
            for lo, n in zip(starts, lens):
                assert not b[0, lo + (n - 1) // 128 * 128:lo + n].any()


@pytest.mark.parametrize("lens,hq,hkv,top_k,tc", [([5000, 1, 0, 777, 128], 4, 2, 4, 3), ([9000], 8, 1, 8, 1), ([300000], 1, 1, 8, 1), ([6000], 2, 2, 3, 0)],
                         ids=["packed", "cut", "many-cut-columns", "uncut"])
def test_the_padding_of_a_row_counts_its_pieces(lens, hq, hkv, top_k, tc, device):
    """A row of the item table: its full pieces and an item for each block, with tiles in front, then padding (at
    least one entry) that names the number of the former."""
    tokens, nb = sum(lens), -(-max(lens) // 128)
    g = torch.Generator(device=device).manual_seed(tokens)
    q, k = (torch.randn((1, tokens, h, 64), generator=g, device=device, dtype=torch.bfloat16) for h in (hq, hkv))
    cu = torch.tensor([0, *torch.tensor(lens).cumsum(0).tolist()], dtype=torch.int32, device=device)
    old = _lib.set_chunk_tiles(tc)
    try:
        index = moba.build_csc_fused(q, k, moba.MoBAConfig(128, top_k), cu_seqlens=cu, max_seqlen=max(lens))
    finally:
        _lib.set_chunk_tiles(old)
    tiles = (index.col_nnz.cpu() + 127) // 128                # [n_seq, Hkv, blocks]
    full = ((tiles - 1).clamp(min=0) // index.chunk_tiles).sum(-1)
    assert tc == 0 or int(full.max()) > 0
    for items, n in zip(index.work_items.cpu().flatten(0, 1), full.flatten().tolist()):
        padding = items[:, 3] == -2
        assert int((~padding).sum()) == n + nb and bool(padding[n + nb:].all()) and bool(padding[-1])
        assert bool((items[padding] == torch.tensor([0, n, 0, -2], dtype=torch.int32)).all())
        has = items[:n + nb, 2] > 0
        assert bool((has[:-1] >= has[1:]).all())


@pytest.mark.parametrize("s,h,d,chunk", [(60000, 16, 64, 30000), (76000, 16, 128, 38000)], ids=["one-group", "groups"])
def test_windows_that_claim(s, h, d, chunk, device):
    """Query windows above the lines (the backward of a window claims): O and dQ are the bits of the whole call.
    dK and dV are sums over two windows, each rounded to bfloat16 (2^-9 of it) and their sum once more."""
    assert chunk * h * 8 / 128 / 148 >= (192 if d == 64 else 256)
    cfg = moba.MoBAConfig(128, 8)
    g = torch.Generator(device=device).manual_seed(s)
    q, k, v, do = (torch.randn((1, s, h, d), generator=g, device=device, dtype=torch.bfloat16) for _ in range(4))
    got = []
    for kw in ({}, dict(query_chunk=chunk)):
        leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
        out = moba.moba_attention(*leaves, cfg, **kw)
        out.backward(do)
        got.append([out.detach()] + [t.grad for t in leaves])
        del out, leaves
    whole, windows = got
    assert torch.equal(windows[0], whole[0]) and torch.equal(windows[1], whole[1])
    for a, b in zip(windows[2:], whole[2:]):
        for a_part, b_part in zip(a.split(12800, dim=1), b.split(12800, dim=1)):
            assert (a_part.float() - b_part.float()).norm() <= 2.0 ** -7 * b_part.float().norm()
