"""Decode attention whose splits merge in thread-block clusters (and a single split inside its block), against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("nh, nkv, hd", [(9, 3, 64), (16, 1, 64), (32, 32, 64), (5, 5, 128), (24, 2, 128), (12, 4, 32), (6, 6, 16), (14, 2, 96)])
@pytest.mark.parametrize("splits", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("block_keys, warps, window", [(16, 8, None), (0, 8, None), (16, 4, None), (0, 4, 100)])
def test_splits_merge_in_a_cluster(nh, nkv, hd, splits, block_keys, warps, window):
    from glassbox_b200 import kernels
    if warps == 8 and hd != 64:
        pytest.skip("eight warps are built for head size 64")
    contexts, page = [1, 16, 17, 130, 700, 0], 16                      # (blocks without keys among the splits; the last is a padding row)
    gen = torch.Generator(device=DEV).manual_seed(nh * splits)
    rand = lambda *shape: torch.randn(shape, generator=gen, device=DEV).bfloat16()
    need = [-(-c // page) for c in contexts]
    order = torch.randperm(sum(need) + 1, generator=torch.Generator().manual_seed(2)).tolist()
    tables = torch.full((len(contexts), 64), -1, dtype=torch.int32)
    at = 0
    for i, m in enumerate(need):
        tables[i, :m] = torch.tensor(order[at:at + m], dtype=torch.int32)
        at += m
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    n, tables = len(contexts), tables.to(DEV)
    q, k, v = rand(n, nh * hd), rand(sum(need) + 1, nkv, page, hd), rand(sum(need) + 1, nkv, page, hd)
    out, status = torch.full((n, nh * hd), 7.0, device=DEV, dtype=torch.bfloat16), i32([0])
    part, ml, counters = torch.empty(n * nh * warps * splits * hd, device=DEV), torch.empty(n * nh * warps * splits * 2, device=DEV), i32([0] * (n * nkv))
    for _ in range(2):                                                # (counters, where a launch uses them, are left zero)
        kernels.attention_decode_mma(q, out, k, v, tables, i32(range(n)), i32([c - 1 for c in contexts]), nh, nkv, hd, page, hd ** -0.5, window, splits,
                                     part, ml, counters, status, block_keys, warps)
    assert int(status) == 0 and not counters.any() and not out[-1].any()
    for i, c in enumerate(contexts[:-1]):
        lo = max(0, c - window) if window else 0
        keys, values = (t[tables[i, :need[i]].long()].transpose(1, 2).flatten(0, 1)[lo:c].double().repeat_interleave(nh // nkv, dim=1) for t in (k, v))
        s = torch.einsum("hd,khd->hk", q[i].double().view(nh, hd), keys) * hd ** -0.5
        want = torch.einsum("hk,khd->hd", torch.softmax(s, -1), values)
        # weights and result in bfloat16: 2^-8 of values of a few
        assert (out[i].double().view(nh, hd) - want).abs().max() < 2.0 ** -8 * 4, i


@pytest.mark.parametrize("nh, nkv, hd, warps", [(9, 3, 64, 8), (16, 1, 64, 8), (24, 2, 128, 4), (32, 4, 96, 4), (16, 1, 16, 4), (5, 1, 64, 4)])
@pytest.mark.parametrize("splits, many", [(2, 100), (6, 64), (8, 64), (3, 160), (13, 3), (30, 3)])
def test_both_ways_of_merging_give_the_same_bits(nh, nkv, hd, warps, splits, many):
    """A few rows merge on the chip, as many as find no room there through global memory (whose scratch may take a large group's heads in
    several passes), as do more splits than a cluster has blocks: the same order of sums, so the same bits."""
    from glassbox_b200 import kernels
    gen = torch.Generator(device=DEV).manual_seed(nh + splits)
    rand = lambda *shape: torch.randn(shape, generator=gen, device=DEV).bfloat16()
    context, page = 1500, 16
    pages = -(-context // page)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    k, v, q = rand(pages, nkv, page, hd), rand(pages, nkv, page, hd), rand(many, nh * hd)
    tables = i32([list(range(pages))] * many)
    scratch = lambda n: (torch.full((n * nh * warps * splits * hd,), float("nan"), device=DEV), torch.full((n * nh * warps * splits * 2,), float("nan"), device=DEV))
    status, counters = i32([0]), i32([0] * (many * nkv))
    positions = i32([(context - 1 - 37 * i) % context for i in range(many)])

    def run(n, keys):
        out = torch.full((n, nh * hd), 7.0, device=DEV, dtype=torch.bfloat16)
        part, ml = scratch(n)
        kernels.attention_decode_mma(q[:n], out, k, v, tables[:n], i32(range(n)), positions[:n], nh, nkv, hd, page, hd ** -0.5, None, splits, part, ml,
                                     counters, status, keys, warps)
        return out
    keys = 16 if warps == 8 else 0
    all_rows = run(many, keys)
    assert int(status) == 0 and not counters.any()
    assert torch.equal(all_rows[:2], run(2, keys))
    for i in range(min(many, 3)):
        c = int(positions[i]) + 1
        kk, vv = (t.transpose(1, 2).flatten(0, 1)[:c].double().repeat_interleave(nh // nkv, dim=1) for t in (k, v))
        want = torch.einsum("hk,khd->hd", torch.softmax(torch.einsum("hd,khd->hk", q[i].double().view(nh, hd), kk) * hd ** -0.5, -1), vv)
        assert (all_rows[i].double().view(nh, hd) - want).abs().max() < 2.0 ** -8 * 4, i
