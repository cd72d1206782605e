"""Prompt attention with two blocks a pair of row tiles (one request of many tiles, or of one tile behind a long context)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("nh, nkv, rows, past, window, page", [
    (9, 3, 1153, 0, 0, 16), (9, 3, 1280, 0, 0, 16), (2, 1, 1281, 0, 0, 64), (3, 1, 1409, 37, 0, 16), (4, 2, 2048, 0, 0, 128), (1, 1, 2047, 1000, 0, 16),
    (3, 3, 1500, 300, 300, 16), (2, 2, 1300, 700, 65, 8), (2, 1, 1400, 0, -512, 16), (9, 3, 128, 1990, 0, 16), (5, 5, 1, 1920, 0, 16), (3, 1, 77, 1025, 600, 32)])
def test_pairs_of_row_tiles(nh, nkv, rows, past, window, page):
    from glassbox_b200 import kernels
    gen = torch.Generator(device=DEV).manual_seed(rows + past)
    rand = lambda *shape: torch.randn(shape, generator=gen, device=DEV).bfloat16()
    total = rows + past
    used = -(-total // page)
    width = max(-(-2048 // page), used + 1)                       # (a table that reaches 2,048 keys: one tile takes the pairs too)
    order = torch.randperm(used + 3, generator=torch.Generator().manual_seed(1))[:used].to(torch.int32)
    table = torch.full((1, width), -1, dtype=torch.int32)
    table[0, :used] = order
    k, v, q = rand(used + 3, nkv, page, 64), rand(used + 3, nkv, page, 64), rand(rows, nh * 64)
    out, status = torch.full((rows, nh * 64), 7.0, device=DEV, dtype=torch.bfloat16), torch.zeros(1, dtype=torch.int32, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    kernels.attention_prefill_tc(q, out, k, v, table.to(DEV), i32([0, rows]), i32([past]), rows, nh, nkv, 64, page, 0.125, window, status)
    assert int(status) == 0
    keys, values = (t[order.long().to(DEV)].transpose(1, 2).flatten(0, 1)[:total].double() for t in (k, v))
    at, pos = torch.arange(total, device=DEV)[None], past + torch.arange(rows, device=DEV)[:, None]
    seen = at <= pos
    if window > 0:
        seen &= at > pos - window
    elif window < 0:
        seen &= at >= pos - pos % -window
    for h in range(nh):
        s = (q[:, h * 64:h * 64 + 64].double() @ keys[:, h // (nh // nkv)].T * 0.125).masked_fill(~seen, float("-inf"))
        want = torch.softmax(s, -1) @ values[:, h // (nh // nkv)]
        # weights in bfloat16 (2^-9 each, of either sign) and one rounding of the result: 2^-8 of values of a few
        assert (out[:, h * 64:h * 64 + 64].double() - want).abs().max() < 2.0 ** -8 * 4, h


@pytest.mark.parametrize("nh, nkv, rows, past", [(9, 3, 1409, 0), (9, 3, 2048, 0), (4, 2, 1600, 0), (2, 1, 1700, 40)])
def test_second_items_of_one_key_tile_repeat_their_bits(nh, nkv, rows, past):
    """The first row tile of a fresh prompt sees one key tile: one softmax group has none there and must not post that item's row
    statistics before the other group has read the first item's. What orders them is `merged` in the kernel; a late reader would
    lose half of a share, so every launch has to give the same bits."""
    from glassbox_b200 import kernels
    gen = torch.Generator(device=DEV).manual_seed(rows)
    rand = lambda *shape: torch.randn(shape, generator=gen, device=DEV).bfloat16()
    pages = -(-(rows + past) // 16)
    k, v, q = rand(pages, nkv, 16, 64), rand(pages, nkv, 16, 64), rand(rows, nh * 64)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    table, first, start, status = i32([list(range(pages))]), i32([0, rows]), i32([past]), i32([0])
    outs = [torch.empty_like(q) for _ in range(50)]
    for out in outs:
        kernels.attention_prefill_tc(q, out, k, v, table, first, start, rows, nh, nkv, 64, 16, 0.125, 0, status)
    assert int(status) == 0 and all(torch.equal(out, outs[0]) for out in outs)


@pytest.mark.parametrize("nh, nkv, rows, past, page", [(9, 3, 1409, 0, 16), (2, 1, 1537, 0, 64), (9, 3, 1600, 0, 16), (2, 2, 1665, 700, 8), (2, 1, 1800, 0, 16)])
def test_odd_and_even_counts_of_row_tiles(nh, nkv, rows, past, page):
    """The tile in the middle of an odd count has no partner; the last tile may have one row."""
    test_pairs_of_row_tiles(nh, nkv, rows, past, 0, page)


@pytest.mark.parametrize("pairs, num_seqs, rows, nh, window, reach", [
    (1, 1, 2048, 9, 0, 2048), (1, 1, 1409, 9, 0, 1409), (0, 1, 1408, 9, 0, 2048), (0, 2, 2048, 9, 0, 2048), (0, 1, 2176, 9, 0, 4096),
    # a window or chunk that ends within what the rows see: tiles see about the same
    (0, 1, 2048, 9, 300, 2048), (0, 1, 2048, 9, 1300, 2048), (0, 1, 2048, 9, -1024, 2048), (1, 1, 2048, 9, 2048, 2048), (1, 1, 2048, 9, 4096, 2048),
    (0, 1, 2048, 9, 2048, 4096), (0, 1, 1500, 9, 2000, 2500),
    # one tile: behind a context that may be long
    (1, 1, 128, 9, 0, 1025), (0, 1, 128, 9, 0, 1024), (0, 1, 129, 9, 0, 4096), (0, 1, 77, 3, 300, 4096), (1, 1, 77, 3, 600, 4096),
    (0, 1, 77, 3, -512, 4096), (1, 1, 1, 148, 0, 2048), (0, 1, 1, 149, 0, 2048)])
def test_which_launches_take_pairs(pairs, num_seqs, rows, nh, window, reach):
    from glassbox_b200 import kernels
    assert kernels.lib().gb_attention_prefill_tc_pairs(num_seqs, rows, nh, window, reach) == pairs
