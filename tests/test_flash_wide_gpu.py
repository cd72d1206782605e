"""The tcgen05 flash kernel with wide values (talking heads, latent cache) against float64 attention over the same bfloat16 numbers, at
the edges of its 128 x 128 tiles. Scores are spread so far that a few keys carry a row: a key, page or column read in another's
place moves the result by the size of a value."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

BATCHES = [  # page size, window, [(cached tokens, new rows) or None for a padding sequence, ...]
    (16, None, [(0, 200), (0, 128), None, (0, 1), (0, 129)]),
    (8, None, [(100, 31), (640, 140), (127, 127)]),
    (32, 100, [(0, 300), (250, 77)]),
    (64, 37, [(500, 130)]),
    (128, None, [(1000, 300)]),
]


def _layout(page, batch, seed):
    """Scattered pages: (slots of every request's tokens, block tables, rows' first, start, number of pages)."""
    g = torch.Generator().manual_seed(seed)
    need = [-(-(c + n) // page) if b else 0 for b in batch for c, n in [b or (0, 0)]]
    order = torch.randperm(sum(need) + 2, generator=g).tolist()
    width = max(need) + 1
    tables, first, start, at = torch.full((len(batch), width), -1, dtype=torch.int32), [0], [], 0
    for i, b in enumerate(batch):
        tables[i, :need[i]] = torch.tensor(order[at:at + need[i]], dtype=torch.int32)
        at += need[i]
        first.append(first[-1] + (b[1] if b else 2))
        start.append(b[0] if b else -1)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    return tables.to(DEV), i32(first), i32(start), sum(need) + 2, max(b[1] for b in batch if b)


def _dense(pool, table, page, length):
    """[length, heads, dim] of one request; pool [pages, heads, page, dim]."""
    pages = table[:-(-length // page)].long()
    return pool[pages].transpose(1, 2).flatten(0, 1)[:length].double()


def _weights(scores, pos, window, sink):
    key = torch.arange(scores.shape[-1], device=scores.device)
    seen = (key <= pos[:, None]) & ((key > pos[:, None] - window) if window else True)
    s = scores.masked_fill(~seen, -math.inf)
    if sink is not None:
        s = torch.cat([s, torch.full_like(s[:, :1], sink)], -1)
    w = torch.softmax(s, -1)
    return w[:, :-1] if sink is not None else w


@pytest.mark.parametrize("page, window, batch", BATCHES)
@pytest.mark.parametrize("H, G, V, cap, unit", [(4, 4, 64, 30.0, True), (6, 2, 64, None, False), (4, 2, 128, 5.0, True), (8, 8, 64, None, True)])
def test_talking_heads(page, window, batch, H, G, V, cap, unit):
    from glassbox_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(page + H)
    tables, first, start, pages, longest = _layout(page, batch, 3)
    n = int(first[-1])
    q = torch.randn(n, H * 64, generator=g, device=DEV).bfloat16()
    k, v = (torch.randn(pages, G, page, d, generator=g, device=DEV).bfloat16() for d in (64, V))
    out = torch.full((n, H * G * V), 7.0, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    kernels.talking_attention_flash(q, out, k, v, tables, first, start, longest, H, G, 64, V, G, page, 0.5, cap, unit, window, status)
    assert int(status) == 0
    got = out.double().view(n, H, G, V)
    for i, b in enumerate(batch):
        a, z = int(first[i]), int(first[i + 1])
        if b is None:
            assert torch.all(got[a:z] == 7.0)
            continue
        pos = b[0] + torch.arange(b[1], device=DEV)
        kk, vv = _dense(k, tables[i], page, b[0] + b[1]), _dense(v, tables[i], page, b[0] + b[1])
        for h in range(H):
            s = q.view(n, H, 64)[a:z, h].double() @ kk[:, h // (H // G)].T * 0.5
            s = cap * torch.tanh(s / cap) if cap else s
            want = torch.einsum("rk,kgv->rgv", _weights(s, pos, window, 0.0 if unit else None), vv)
            # weights rounded to bfloat16, 2^-8 of each at most, in the sum and in its denominator: 2^-8 (sum w |v| + |result|); a few
            # keys share the weight, so half of that
            assert (got[a:z, h] - want).abs().max() <= 2 ** -9 * 2 * vv.abs().max(), (i, h, float((got[a:z, h] - want).abs().max()))


@pytest.mark.parametrize("page, window, batch", BATCHES)
@pytest.mark.parametrize("H, r, sink", [(3, 64, True), (2, 32, False), (1, 16, True)])
def test_latent_cache(page, window, batch, H, r, sink):
    from glassbox_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(page + r)
    tables, first, start, pages, longest = _layout(page, batch, 4)
    n = int(first[-1])
    q = torch.randn(n, H * (128 + r), generator=g, device=DEV).bfloat16()
    cache = torch.randn(pages, page, 128 + r, generator=g, device=DEV).bfloat16()
    sinks = torch.randn(H, generator=g, device=DEV) * 5 if sink else None
    out = torch.full((n, H * 128), 7.0, dtype=torch.bfloat16, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    kernels.latent_flash(q, out, cache, tables, first, start, sinks, H, 128, r, page, 0.4, window, status, longest)
    assert int(status) == 0
    got = out.double().view(n, H, 128)
    for i, b in enumerate(batch):
        a, z = int(first[i]), int(first[i + 1])
        if b is None:
            assert torch.all(got[a:z] == 0.0)       # (as the other kernels over this cache leave them)
            continue
        pos = b[0] + torch.arange(b[1], device=DEV)
        rows = _dense(cache[:, None], tables[i], page, b[0] + b[1])[:, 0]
        for h in range(H):
            s = q.view(n, H, 128 + r)[a:z, h].double() @ rows.T * 0.4
            want = _weights(s, pos, window, float(sinks[h]) if sink else None) @ rows[:, :128]
            # weights rounded to bfloat16 (as above), and the result
            assert (got[a:z, h] - want).abs().max() <= 2 ** -9 * 3 * rows[:, :128].abs().max(), (i, h, float((got[a:z, h] - want).abs().max()))


def test_positions_beyond_the_table_and_missing_pages_are_reported():
    from glassbox_b200 import kernels
    tables, first, start, pages, longest = _layout(16, [(0, 40)], 5)
    q = torch.randn(40, 2 * 160, device=DEV).bfloat16()
    cache = torch.randn(pages, 16, 160, device=DEV).bfloat16()
    for bad, bit in ((tables[:, :2].contiguous(), 4), (tables.clone().index_fill_(1, torch.tensor([1], device=DEV), -1), 2)):
        out, status = torch.full((40, 256), 7.0, dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        kernels.latent_flash(q, out, cache, bad, first, start, None, 2, 128, 32, 16, 0.1, None, status, longest)
        assert int(status) == bit and not (out == 7.0).any()
        assert bit == 2 or not out.any()           # a request beyond its table reads as zeros


@pytest.mark.parametrize("rows", [72, 129, 256, 300])
def test_every_launch_ends_by_itself(rows):
    """Blocks of one to three key tiles, whose last products overlap their warps' last looks at the barriers in every order: launches
    behind one another, beside work that takes multiprocessors away, must all finish (no wait that gives up) with the same result."""
    from glassbox_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(rows)
    tables, first, start, pages, longest = _layout(16, [(0, rows)] * 6, rows)
    n, H = int(first[-1]), 8
    q = torch.randn(n, H * 192, generator=g, device=DEV).bfloat16()
    cache = torch.randn(pages, 16, 192, generator=g, device=DEV).bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    busy, side = torch.randn(4096, 4096, device=DEV), torch.cuda.Stream()
    outs = [torch.full((n, H * 128), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(60)]
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        for _ in range(20):
            busy.mul_(1.0001)
    for out in outs:
        kernels.latent_flash(q, out, cache, tables, first, start, None, H, 128, 64, 16, 0.1, None, status, longest)
    torch.cuda.synchronize()
    assert int(status) == 0
    assert all(torch.equal(outs[0], out) for out in outs[1:])


@pytest.mark.parametrize("cap", [None, 30.0])
def test_a_nan_query_gives_nan(cap):
    """A NaN in one row's query of one head makes that row's results of that head NaN, and no other number changes."""
    from glassbox_b200 import kernels
    if cap is None:
        tables, first, start, pages, longest = _layout(16, [(30, 200)], 6)
        n, H = int(first[-1]), 3
        q = torch.randn(n, H, 160, device=DEV).bfloat16()
        cache = torch.randn(pages, 16, 160, device=DEV).bfloat16()
        run = lambda q, out, st: kernels.latent_flash(q.view(n, -1), out, cache, tables, first, start, None, H, 128, 32, 16, 0.2, None, st, longest)
        make = lambda: torch.zeros(n, H * 128, dtype=torch.bfloat16, device=DEV)
        _nan_row(run, make, q, n, H)
    tables, first, start, pages, longest = _layout(16, [(30, 200)], 7)
    n, H, G = int(first[-1]), 4, 2
    q = torch.randn(n, H, 64, device=DEV).bfloat16()
    k, v = (torch.randn(pages, G, 16, 64, device=DEV).bfloat16() for _ in range(2))
    run = lambda q, out, st: kernels.talking_attention_flash(q.view(n, -1), out, k, v, tables, first, start, longest, H, G, 64, 64, G, 16, 0.5,
                                                             cap, True, None, st)
    _nan_row(run, lambda: torch.zeros(n, H * G * 64, device=DEV), q, n, H)


def _nan_row(run, make, q, n, H):
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    clean, spoiled = make(), make()
    run(q, clean, status)
    bad = q.clone()
    bad[77, 1, 5] = float("nan")
    run(bad, spoiled, status)
    assert int(status) == 0
    a, b = clean.view(n, H, -1), spoiled.view(n, H, -1)
    assert torch.isnan(b[77, 1]).all() and torch.isfinite(a).all()
    b[77, 1] = a[77, 1]
    assert torch.equal(a, b)


@pytest.mark.parametrize("cap", [0.5, 5.0, 50.0])
def test_the_cap_is_as_exact_as_float32_allows(cap):
    """The first token of a request sees one key: beside the unit of score 0 in the denominator its result is value * sigmoid(capped
    score), and a single product makes the score exact, so what is off is the cap (and the last exponential and division)."""
    from glassbox_b200 import kernels
    S = 400
    q = torch.zeros(S, 64, device=DEV)
    q[:, 3] = torch.cat([torch.linspace(-16, 16, S // 2), torch.linspace(-60, 60, S // 2)]).to(DEV)
    q = q.bfloat16()
    k = torch.zeros(S, 1, 8, 64, dtype=torch.bfloat16, device=DEV)
    k[:, 0, 0, 3] = 1.0
    v = torch.full((S, 1, 8, 128), 1.0, dtype=torch.bfloat16, device=DEV)
    i32 = lambda x: torch.as_tensor(x, dtype=torch.int32).to(DEV)
    out, status = torch.zeros(S, 128, device=DEV), i32([0])
    kernels.talking_attention_flash(q, out, k, v, i32(range(S))[:, None].contiguous(), i32(range(S + 1)), i32([0] * S), 1, 1, 1, 64, 128, 1, 8,
                                    0.25, cap, True, None, status)
    s = cap * torch.tanh(q[:, 3].double() * 0.25 / cap)
    want = torch.sigmoid(s)
    # relative: the tanh's two units in the last place (2^-23), its input's and the cap's roundings (3 * 2^-24), all times |s| (1 - sigmoid);
    # the hardware's exponential (2^-22, times 1 - sigmoid) of a rounded difference (|s| log2(e) 2^-24) and the division (2^-23)
    bound = want * ((1 - want) * (s.abs() * (5 * 2 ** -24 + 2 ** -24) + 2 ** -22) + 2 ** -22)
    assert int(status) == 0
    assert ((out.double() - want[:, None]).abs() <= bound[:, None]).all(), float(((out.double() - want[:, None]).abs() / bound[:, None]).max())


@pytest.mark.parametrize("window, G", [(None, 2), (50, 2), (None, 4), (50, 4)])
def test_what_no_row_sees_reaches_no_result(window, G):
    """Pages hold what earlier requests left: past the last row, in front of a window, and in every page the table does not name.
    Infinities and NaN there change no result."""
    from glassbox_b200 import kernels
    batch = [(130, 75), (0, 200), (300, 140), (100, 20), (0, 3)]        # of one to four key tiles
    tables, first, start, pages, longest = _layout(16, batch, 8)
    n = int(first[-1])
    seen = torch.zeros(pages, 16, dtype=torch.bool, device=DEV)
    for i, (c, r) in enumerate(batch):
        for t in range(max(c + 1 - window, 0) if window else 0, c + r):
            seen[int(tables[i, t // 16]), t % 16] = True
        if window:                                          # pages wholly in front of the window may be gone
            tables[i, :max(c + 1 - window, 0) // 16] = -1
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    spoil = lambda t, dim: torch.where(seen.view(seen.shape + (1,) * (t.dim() - 2)), t, torch.tensor(dim, device=DEV, dtype=t.dtype))
    H = 4
    q = torch.randn(n, H * 64, device=DEV).bfloat16()
    k, v = (torch.randn(pages, 16, G, d, device=DEV).bfloat16() for d in (64, 64))
    outs = []
    for bad in (0.0, float("inf"), float("nan")):
        out = torch.zeros(n, H * G * 64, device=DEV)
        kk, vv = (spoil(t, bad).transpose(1, 2).contiguous() for t in (k, v))
        kernels.talking_attention_flash(q, out, kk, vv, tables, first, start, longest, H, G, 64, 64, G, 16, 0.5, 30.0, True, window, status)
        outs.append(out)
    assert int(status) == 0 and torch.isfinite(outs[0]).all() and torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    q = torch.randn(n, H * 192, device=DEV).bfloat16()
    cache = torch.randn(pages, 16, 192, device=DEV).bfloat16()
    outs = []
    for bad in (0.0, float("inf"), float("nan")):
        out = torch.zeros(n, H * 128, dtype=torch.bfloat16, device=DEV)
        kernels.latent_flash(q, out, spoil(cache, bad), tables, first, start, None, H, 128, 64, 16, 0.2, window, status, longest)
        outs.append(out)
    assert int(status) == 0 and torch.isfinite(outs[0]).all() and torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])


def test_a_mixed_step_of_the_latent_mixer_equals_one_kernel_over_all_rows():
    """Leading single tokens (two padding sequences among them) to the decode kernel and the portions behind them to the flash kernel,
    against the tiles of tokens x heads over the whole step."""
    from types import SimpleNamespace
    from glassbox_b200 import kernels
    from glassbox_b200.parts.latent_attention import LatentAttention
    H, c, r, page = 32, 128, 64, 16
    singles = [(60 + 97 * i % 900, 1) for i in range(22)] + [None, None]
    portions = [(40, 300), (0, 200)]
    tables, _, start, pages, longest = _layout(page, [s or (0, 1) for s in singles] + portions, 9)
    lead = len(singles)
    start = torch.tensor([s[0] if s else -1 for s in singles] + [p for p, _ in portions], dtype=torch.int32, device=DEV)
    first = torch.tensor([*range(lead + 1), lead + 300, lead + 500], dtype=torch.int32, device=DEV)
    positions = torch.tensor([s[0] if s else -1 for s in singles] + [p + i for p, n in portions for i in range(n)], dtype=torch.int32, device=DEV)
    n = lead + 500
    g = torch.Generator(device=DEV).manual_seed(5)
    q = torch.randn(n, H * (c + r), generator=g, device=DEV).bfloat16()
    pool = torch.randn(pages, 1, page, c + r, generator=g, device=DEV).bfloat16()
    sink = torch.randn(H, generator=g, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    taken = []
    ctx = SimpleNamespace(decode_only=False, leading_single=lead, max_context=1024, max_rows_per_seq=longest, status=status, seq_first_row=first,
                          seq_start_pos=start, positions=positions,
                          scratch=lambda name, shape, dtype, grow: taken.append(name) or torch.empty(shape, dtype=dtype, device=DEV))
    part = SimpleNamespace(H=H, c=c, r=r, params={"sink": sink}, spec=SimpleNamespace(scale=0.1, window=None))
    part._attend_decode = lambda *a: LatentAttention._attend_decode(part, *a)
    assert kernels.latent_flash_chosen(500, 2, H, 1024)
    got, want = (torch.full((n, H * c), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    LatentAttention.attend(part, ctx, q, got, SimpleNamespace(k=pool, page_size=page, block_tables=tables))
    kernels.latent_attention_mma(q, want, pool, tables, first, start, positions, sink, H, c, r, page, 0.1, None, status, max_rows_per_seq=longest)
    assert int(status) == 0
    # both round their weights and results to bfloat16, 2^-8 of the largest value at most each (see test_latent_cache)
    live = positions >= 0
    assert (got[live].float() - want[live].float()).abs().max() <= 2 ** -9 * 3 * 2 * pool[..., :c].float().abs().max()
    assert torch.isfinite(got.float()).all()
