"""The whole-op entry points (`moba_b200_op_forward` / `_op_backward`, what `moba_attention` and
`moba_forward` call when no index is given) against the staged ones with an explicit index. The
selections are the same, so where both run the same attention kernels O and dQ are the same bits;
dK/dV may be cut into other work items and are compared within the engine's tolerance. Sizes lie on
both sides of the line between the one-launch transpose and the five-pass one, and of the finer cut
of small problems. Blocks finer than 128 keys run on columns of 128 in the whole op (other kernels
than the staged calls: compared within the tolerance), and more than eight ranked blocks, like the
finer blocks, on the exact tensor-core gate, whose selections must be those of the float64 one."""

import pytest
import torch

import moba_triton_b200 as moba
from moba_triton_b200 import _lib
from moba_triton_b200.kernels.moba_fwd import op_plan
from moba_triton_b200.tuning import launch_plan

from conftest import make_qkv
from helpers import max_abs_error

pytestmark = pytest.mark.gpu

CASES = [
    # B, S, Hq, Hkv, D, block, top_k, dtype, cu_seqlens
    (1, 100, 2, 1, 64, 128, 3, torch.bfloat16, None),            # one short block
    (1, 1000, 4, 2, 64, 128, 4, torch.bfloat16, None),
    (3, 900, 2, 2, 128, 128, 8, torch.float16, None),            # batch rows end inside a block
    (1, 16384, 1, 1, 64, 128, 8, torch.bfloat16, None),          # the last row length of the one-launch transpose
    (1, 16512, 1, 1, 64, 128, 8, torch.bfloat16, None),          # the first beyond it
    (1, 13000, 1, 1, 64, 128, 10, torch.bfloat16, None),         # nine ids per lane of a cluster of sixteen
    (1, 5000, 5, 5, 64, 128, 4, torch.bfloat16, None),           # five rows: clusters of eight
    (1, 8192, 2, 2, 64, 16, 2, torch.bfloat16, None),            # 512 columns
    (1, 8208, 2, 2, 64, 16, 2, torch.bfloat16, None),            # 513
    (1, 6144, 5, 5, 64, 16, 3, torch.float32, None),             # 384 columns: 48 KB of counters beside static memory
    (1, 45000, 1, 1, 64, 128, 2, torch.bfloat16, None),          # 352
    (1, 1500, 4, 2, 64, 128, 4, torch.bfloat16, [0, 1, 130, 700, 1500]),
    (1, 700, 2, 2, 64, 32, 5, torch.float32, [0, 333, 700]),
    (2, 1000, 4, 2, 128, 64, 8, torch.bfloat16, None),           # a column's second block cut short
    (1, 3000, 2, 2, 64, 32, 6, torch.float16, [0, 31, 33, 1500, 3000]),
    (1, 9000, 4, 1, 64, 64, 8, torch.bfloat16, None),            # 141 candidates: past the first chunk of block means
    (1, 6000, 2, 2, 64, 128, 12, torch.bfloat16, None),          # eleven ranked blocks
    (1, 20000, 2, 1, 128, 128, 13, torch.float16, None),         # twelve, two chunks, head_dim 128
    (1, 6000, 2, 2, 64, 128, 17, torch.bfloat16, None),          # sixteen: the last the exact gate takes
    (1, 4000, 2, 2, 64, 128, 18, torch.bfloat16, None),          # seventeen: the portable gate
]


@pytest.mark.parametrize("b,s,hq,hkv,d,bs,top_k,dtype,cu", CASES, ids=[f"s{c[1]}-h{c[2]}kv{c[3]}-blk{c[5]}" for c in CASES])
def test_whole_op_equals_the_staged_calls(b, s, hq, hkv, d, bs, top_k, dtype, cu, device):
    cfg = moba.MoBAConfig(bs, top_k, dtype=dtype)
    q, k, v, do = (t.to(device) for t in make_qkv((b, s, hq, d), hkv, dtype=dtype, seed=61, with_do=True))
    kw = {} if cu is None else dict(cu_seqlens=torch.tensor(cu, dtype=torch.int32, device=device),
                                    max_seqlen=max(y - x for x, y in zip(cu[:-1], cu[1:])))
    index = moba.build_csc_fused(q, k, cfg, **kw)
    got = []
    for args in (dict(index=index), kw):
        leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
        out = moba.moba_attention(*leaves, cfg, **args)
        out.backward(do)
        got.append([out.detach()] + [t.grad for t in leaves])
    staged, whole = got
    same_kernels = bs == 128 or dtype == torch.float32
    for i, (a, w) in enumerate(zip(whole, staged)):
        if same_kernels and i < 2:
            assert torch.equal(a, w)
        assert max_abs_error(a, w) <= (1e-5 if dtype == torch.float32 else 2e-2)
    assert torch.equal(moba.moba_forward(q, k, v, cfg, **kw), whole[0])


@pytest.mark.parametrize("flags", [dict(causal=False), dict(always=False), dict(includes=False)], ids=["noncausal", "noown", "extra"])
def test_finer_blocks_with_the_other_options(flags, device):
    cfg = moba.MoBAConfig(32, 4, always_select_current=flags.get("always", True), top_k_includes_current=flags.get("includes", True))
    q, k, v, do = (t.to(device) for t in make_qkv((1, 1100, 4, 64), 2, dtype=torch.bfloat16, seed=62, with_do=True))
    index = moba.build_csc_fused(q, k, cfg)
    got = []
    for ix in (index, None):
        leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
        out = moba.moba_attention(*leaves, cfg, index=ix, causal=flags.get("causal", True))
        out.backward(do)
        got.append([out.detach()] + [t.grad for t in leaves])
    for staged, whole in zip(*got):
        assert torch.equal(torch.isnan(staged), torch.isnan(whole))          # no own block: the first rows select nothing
        assert max_abs_error(staged.nan_to_num(), whole.nan_to_num()) <= 2e-2


def gradients(q, k, v, do, cfg, **kw):
    leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
    out = moba.moba_attention(*leaves, cfg, **kw)
    out.backward(do)
    return [out.detach()] + [t.grad for t in leaves]


@pytest.mark.parametrize("block,top_k,d,dtype", [(64, 4, 64, torch.bfloat16), (32, 6, 128, torch.float16), (16, 3, 64, torch.bfloat16),
                                                 (128, 12, 64, torch.bfloat16), (48, 4, 64, torch.bfloat16), (64, 4, 64, torch.float32)])
def test_query_windows_run_the_kernels_of_the_whole_op(block, top_k, d, dtype, device):
    """O and dQ bit for bit whatever the block size; windows that end inside a block, and one of a row."""
    cfg = moba.MoBAConfig(block, top_k, dtype=dtype)
    q, k, v, do = (t.to(device) for t in make_qkv((2, 1201, 4, d), 2, dtype=dtype, seed=64, with_do=True))
    whole = gradients(q, k, v, do, cfg)
    for chunk in (400, 333, 5000):
        got = gradients(q, k, v, do, cfg, query_chunk=chunk)
        assert torch.equal(got[0], whole[0]) and torch.equal(got[1], whole[1])
        for a, w in zip(got[2:], whole[2:]):                 # sums over the windows: rounded once more
            assert max_abs_error(a, w) <= (1e-5 if dtype == torch.float32 else 2e-2)
        assert torch.equal(moba.moba_forward(q, k, v, cfg, query_chunk=chunk), whole[0])


@pytest.mark.parametrize("block,top_k,d,dtype", [(64, 4, 64, torch.bfloat16), (16, 3, 128, torch.float16), (128, 12, 64, torch.bfloat16),
                                                 (64, 4, 64, torch.float32)])
def test_passes_over_kv_heads_run_the_kernels_of_the_whole_op(block, top_k, d, dtype, device):
    cfg = moba.MoBAConfig(block, top_k, dtype=dtype)
    q, k, v = (t.to(device) for t in make_qkv((2, 1201, 6, d), 3, dtype=dtype, seed=65))
    whole = moba.moba_forward(q, k, v, cfg)
    for n in (1, 2):
        assert torch.equal(moba.moba_forward(q, k, v, cfg, kv_heads_per_pass=n), whole)


@pytest.mark.parametrize("s,hkv,group", [(1024, 16, 1), (2048, 12, 2), (8192, 8, 1)], ids=["cut4", "cut8", "cut8-long"])
def test_passes_over_kv_heads_cut_columns_like_the_whole_call(s, hkv, group, device):
    """1 024, 3 072 and 4 096 tiles as a whole, at most half of that in a pass: by itself a pass would
    cut its columns into finer items and sum dK and dV in other groups."""
    cfg = moba.MoBAConfig(128, 8)
    q, k, v, do = (t.to(device) for t in make_qkv((1, s, hkv * group, 64), hkv, dtype=torch.bfloat16, seed=66, with_do=True))
    whole = gradients(q, k, v, do, cfg)
    for n in (1, hkv // 2):
        for a, w in zip(gradients(q, k, v, do, cfg, kv_heads_per_pass=n), whole):
            assert torch.equal(a, w)


@pytest.mark.parametrize("s,hkv,group,d,block,cuts", [(14208, 4, 1, 64, 128, (14, 8)), (18944, 2, 2, 64, 128, (16, 8)),
                                                      (37888, 4, 1, 128, 128, (24, 16)), (14300, 2, 2, 64, 32, (15, 8)), (7104, 2, 4, 64, 128, (12, 8))],
                         ids=["shortest", "passes", "longest", "finer", "long-columns"])
def test_a_forward_alone_is_cut_finer_than_the_forward_of_a_step(s, hkv, group, d, block, cuts, device):
    """24 to 64 tiles per SM: one workspace holds either table of work items. O is the same bits for both, all
    four results are those of staged calls with the step's cut, and (up to 32 tiles per SM) of passes."""
    cfg = moba.MoBAConfig(block, 8)
    q, k, v, do = (t.to(device) for t in make_qkv((1, s, hkv * group, d), hkv, dtype=torch.bfloat16, seed=68, with_do=True))
    step, alone = (launch_plan(q.shape, hkv, q.dtype, cfg, gradients=g) for g in (True, False))
    assert (step["chunk_tiles"], alone["chunk_tiles"]) == cuts
    assert step["work_items_per_row"] < alone["work_items_per_row"]
    whole = gradients(q, k, v, do, cfg)
    assert torch.equal(moba.moba_forward(q, k, v, cfg), whole[0])
    if block == 128:
        old = _lib.set_chunk_tiles(step["chunk_tiles"])
        try:
            staged = gradients(q, k, v, do, cfg, index=moba.build_csc_fused(q, k, cfg))
        finally:
            _lib.set_chunk_tiles(old)
        for a, w in zip(staged, whole):
            assert torch.equal(a, w)
    for a, w in zip(gradients(q, k, v, do, cfg, kv_heads_per_pass=1), whole if cuts[0] <= 16 else whole[:2]):
        assert torch.equal(a, w)


def test_the_function_of_a_given_index_builds_one_if_there_is_none(device):
    cfg = moba.MoBAConfig(128, 4)
    q, k, v, do = (t.to(device) for t in make_qkv((1, 1000, 4, 64), 2, dtype=torch.bfloat16, seed=67, with_do=True))
    cu = torch.tensor([0, 300, 1000], dtype=torch.int32, device=device)
    for kw in ({}, dict(cu_seqlens=cu, max_seqlen=700)):
        leaves = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
        out = moba.MoBAAttentionFunction.apply(*leaves, cfg, None, True, kw.get("cu_seqlens"), kw.get("max_seqlen"))
        out.backward(do)
        index = moba.build_csc_fused(q, k, cfg, **kw)
        for a, w in zip([out] + [t.grad for t in leaves], gradients(q, k, v, do, cfg, index=index)):
            assert torch.equal(a, w)


class OpenConfig:
    """A configuration object of a caller's own: hashable by identity, and mutable."""
    block_size, top_k, always_select_current = 128, 2, True
    slots_per_query = property(lambda self: self.top_k)

    def num_blocks(self, n):
        return -(-n // self.block_size)

    def past_blocks_selected(self, nb):
        return min(self.top_k - 1, nb)


def test_a_call_is_told_from_an_earlier_one_by_values(device):
    q, k, v = (t.to(device) for t in make_qkv((1, 1000, 2, 64), 2, dtype=torch.bfloat16, seed=63))
    cfg = OpenConfig()
    for top_k, block in ((2, 128), (4, 128), (4, 64)):
        cfg.top_k, cfg.block_size = top_k, block
        want = moba.moba_forward(q, k, v, moba.MoBAConfig(block, top_k))
        assert torch.equal(moba.moba_forward(q, k, v, cfg), want)
        assert torch.equal(moba.moba_attention(q, k, v, cfg), want)
    # a length that is a tensor, changed in place
    longest, frozen = torch.tensor(1000, device=device), moba.MoBAConfig(128, 4)
    for cu in ([0, 300, 1000], [0, 400, 1000]):
        longest.fill_(max(b - a for a, b in zip(cu[:-1], cu[1:])))
        cu = torch.tensor(cu, dtype=torch.int32, device=device)
        assert op_plan(q, k, v, frozen, True, cu, longest).problem.max_seqlen == int(longest)


@pytest.mark.parametrize("d,top_k", [(64, 8), (64, 3), (128, 9)])
@pytest.mark.parametrize("blocks", [32, 33, 34, 64, 65, 66, 129, 258])
def test_gate_at_its_bounds(blocks, d, top_k, device):
    """Candidate counts around the lines between no bounding pass, one half's bar and both halves' bar.
    Scores are whole numbers, exact in every precision; rounded to bfloat16 many of them tie."""
    cfg = moba.MoBAConfig(128, top_k, dtype=torch.bfloat16)
    s = (blocks - 1) * 128 + 5
    g = torch.Generator().manual_seed(blocks)
    q = torch.randint(-7, 8, (1, s, 2, d), generator=g).to(torch.bfloat16).to(device)
    kbar = moba.pool_blocks(q[:, :, :1].contiguous(), cfg)
    kbar = torch.randint(-7, 8, kbar.shape, generator=g).to(kbar.dtype).to(device)
    got = moba.gate_select(q, kbar, cfg).reshape(2, s, -1)
    scores = torch.einsum("shd,nd->hsn", q[0].double(), kbar.reshape(blocks, d).double()).to(torch.bfloat16).double()
    own = torch.arange(s, device=device) // 128
    ids = torch.arange(blocks, device=device)
    key = scores * 1024 - ids                                # score descending, ties to the lower id
    key[:, ids[None, :] >= own[:, None]] = -float("inf")
    best = key.topk(min(top_k - 1, blocks), dim=-1)
    want = torch.where(best.values > -float("inf"), best.indices, blocks)
    want = torch.cat([want, own[None, :, None].expand(2, -1, 1)], -1).sort(-1).values
    have = torch.where(got < 0, blocks, got.long()).sort(-1).values
    assert torch.equal(have, want)


@pytest.mark.parametrize("top_k", [2, 9, 33, 34])
@pytest.mark.parametrize("blocks", [20, 33, 34, 100])
def test_portable_gate_lists(blocks, top_k, device):
    """The list over a warp's lanes (up to 32 ranked blocks) and the one in shared memory, with ties."""
    cfg = moba.MoBAConfig(16, top_k, dtype=torch.float32)
    s = blocks * 16 - 3
    g = torch.Generator().manual_seed(blocks)
    q = torch.randint(-2, 3, (1, s, 2, 64), generator=g).float().to(device)
    kbar = torch.randint(-2, 3, (1, 1, blocks, 64), generator=g).float().to(device)
    got = moba.gate_select(q, kbar, cfg).reshape(2, s, -1)
    scores = torch.einsum("shd,nd->hsn", q[0].double(), kbar.reshape(blocks, 64).double())
    own = torch.arange(s, device=device) // 16
    ids = torch.arange(blocks, device=device)
    key = scores * 1024 - ids
    key[:, ids[None, :] >= own[:, None]] = -float("inf")
    best = key.topk(min(top_k - 1, blocks), dim=-1)
    want = torch.where(best.values > -float("inf"), best.indices, blocks)
    want = torch.cat([want, own[None, :, None].expand(2, -1, 1)], -1).sort(-1).values
    have = torch.where(got < 0, blocks, got.long()).sort(-1).values[..., :want.shape[-1]]
    assert torch.equal(have, want)


@pytest.mark.parametrize("blocks,top_k,d", [(896, 2, 64), (897, 2, 64), (1792, 9, 64), (1793, 9, 64), (2816, 17, 64), (2817, 17, 64), (2945, 18, 64), (1100, 5, 128)])
def test_portable_gate_lists_of_long_rows(blocks, top_k, d, device):
    """Either side of the line between the rows of a warp sorted in step and row by row; the last rows, with ties."""
    cfg = moba.MoBAConfig(16, top_k, dtype=torch.float32)
    s, n = blocks * 16 - 3, 500
    g = torch.Generator().manual_seed(blocks)
    q = torch.randint(-2, 3, (1, s, 1, d), generator=g).float().to(device)
    kbar = torch.randint(-2, 3, (1, 1, blocks, d), generator=g).float().to(device)
    got = moba.gate_select(q, kbar, cfg).reshape(s, -1)[-n:]
    scores = q[0, -n:, 0].double() @ kbar.reshape(blocks, d).double().t()
    own = torch.arange(s - n, s, device=device) // 16
    ids = torch.arange(blocks, device=device)
    key = scores * 4096 - ids
    key[ids[None, :] >= own[:, None]] = -float("inf")
    want = torch.cat([key.topk(top_k - 1, dim=-1).indices, own[:, None]], -1).sort(-1).values
    assert torch.equal(got.long(), want)
