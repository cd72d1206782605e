"""Decoding of talking-heads attention on the tensor cores, at the edges of its steps and shares, against float64 sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(H, G, D, V, contexts, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    ps, width = 16, max(contexts) // 16 + 2
    tables = [[-1] * width for _ in contexts]
    order = iter(torch.randperm(sum(-(-c // ps) for c in contexts), generator=torch.Generator().manual_seed(seed)).tolist())
    for i, c in enumerate(contexts):
        for j in range(-(-c // ps)):
            tables[i][j] = next(order)
    pages = sum(-(-c // ps) for c in contexts)
    rand = lambda *shape: torch.randn(shape, generator=gen, device=DEV).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    return dict(q=rand(len(contexts), H * D), k=rand(pages, G, ps, D), v=rand(pages, G, ps, V), tables=i32(tables), positions=i32([c - 1 for c in contexts]),
                row_seq=i32(list(range(len(contexts)))))


def _run(kernels, c, H, G, D, V, shares, cap, unit, window):
    n, wide_cols, status = c["q"].shape[0], H * G * V, torch.zeros(1, dtype=torch.int32, device=DEV)
    wide, ml = torch.full((shares * n, wide_cols), float("nan"), device=DEV), torch.full((shares * n, H * 2), float("nan"), device=DEV)
    kernels.talking_attention_decode(c["q"], wide, c["k"], c["v"], c["tables"], c["row_seq"], c["positions"], heads=H, kv_heads=G, dim=D, vdim=V,
                                     value_heads=G, page_size=16, scale=D ** -0.5, softcap=cap, unit_sink=unit, window=window, status=status,
                                     shares=shares, ml=ml)
    talk = torch.randn(H, H, device=DEV, generator=torch.Generator(device=DEV).manual_seed(1))
    att = torch.full((n, H * V), 7.0, device=DEV)
    kernels.talk_combine(wide, talk, att, c["positions"], H, G, V, G, shares=shares, ml=ml, unit_sink=unit)
    return att, talk, int(status)


def _exact(c, H, G, D, V, talk, cap, unit, window):
    out = torch.zeros(c["q"].shape[0], H, V, dtype=torch.float64, device=DEV)
    for i, pos in enumerate(c["positions"].tolist()):
        if pos < 0:
            continue
        lo, pages = max(0, pos + 1 - window) if window else 0, c["tables"][i][: pos // 16 + 1].long()
        k, v = (t[pages].transpose(1, 2).flatten(0, 1)[lo:pos + 1].double() for t in (c["k"], c["v"]))
        s = torch.einsum("gpd,kgd->gpk", c["q"][i].double().view(G, H // G, D), k).reshape(H, -1) * D ** -0.5
        s = cap * torch.tanh(s / cap) if cap else s
        w = torch.exp(s - s.amax(-1, keepdim=True))
        w = w / (w.sum(-1, keepdim=True) + (torch.exp(-s.amax(-1, keepdim=True)) if unit else 0.0))
        mixed = talk.double() @ w
        out[i] = torch.einsum("hk,khv->hv", mixed, v.repeat_interleave(H // G, dim=1))
    return out.view(out.shape[0], -1)


@pytest.mark.parametrize("H, G, D, V", [(16, 4, 64, 64), (32, 8, 64, 64), (8, 2, 128, 64), (5, 1, 64, 128), (24, 4, 64, 128), (18, 2, 128, 128), (40, 8, 64, 16)])
@pytest.mark.parametrize("shares, cap, unit, window", [(1, 30.0, True, None), (1, None, False, 33), (3, 2.0, True, None), (16, None, True, 200)])
def test_decoding_on_the_tensor_cores(H, G, D, V, shares, cap, unit, window):
    from glassbox_b200 import kernels
    assert kernels.lib().gb_talking_decode_mma_heads(H, G, D, V, G)
    c = _case(H, G, D, V, [1, 31, 32, 33, 64, 65, 127, 128, 129, 257, 700], H * 100 + D)
    c["positions"][4] = -1
    att, talk, status = _run(kernels, c, H, G, D, V, shares, cap, unit, window)
    assert status == 0 and (att[4] == 7.0).all()
    att[4] = 0.0
    want = _exact(c, H, G, D, V, talk, cap, unit, window)
    # float32 scores, weights and sums: each some 1e-7 of a weighted sum of H standard normal mixes (weights' sum at most 1)
    assert (att.double() - want).abs().max() < 2e-6 * H ** 0.5 * 4 and (att.double() - want).norm() < 5e-7 * want.norm()


def test_numbers_that_are_not_finite_stay_where_they_are_seen():
    """An infinite value reaches its channel and value head alone (and keeps its sign, though a weight is worked as three terms); keys that
    a row does not see reach nothing; a page that does not exist is recorded and weighs nothing."""
    from glassbox_b200 import kernels
    H, G, D, V = 16, 4, 64, 64
    c = _case(H, G, D, V, [40, 130, 300, 90], 5)
    clean, _, _ = _run(kernels, c, H, G, D, V, 2, 30.0, True, None)
    page = lambda i, pos: (int(c["tables"][i][pos // 16]), pos % 16)
    p, o = page(0, 7)
    c["v"][p, 2, o, 5] = float("inf")
    p, o = page(1, 129)
    c["v"][p, 1, min(o + 1, 15)] = float("nan")                      # (behind the row's own position: never seen)
    c["k"][p, 1, min(o + 1, 15)] = float("inf")
    got, talk, status = _run(kernels, c, H, G, D, V, 2, 30.0, True, None)
    assert status == 0 and torch.equal(got[1:], clean[1:])
    hit = torch.zeros(H, V, dtype=torch.bool, device=DEV)
    hit[8:12, 5] = True
    assert torch.equal(got[0].view(H, V)[~hit], clean[0].view(H, V)[~hit]) and not got[0].view(H, V)[hit].isfinite().any()
    positive = torch.zeros(1, H * G * V, device=DEV)                 # before the mix: +inf for every head
    one = {k: (t[:1] if k in ("q", "tables", "positions", "row_seq") else t) for k, t in c.items()}
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    args = dict(heads=H, kv_heads=G, dim=D, vdim=V, value_heads=G, page_size=16, scale=D ** -0.5, softcap=30.0, unit_sink=True, window=None, status=st)
    kernels.talking_attention_decode(one["q"], positive, one["k"], one["v"], one["tables"], one["row_seq"], one["positions"], **args)
    cell = positive.view(H, G, V)
    assert (cell[:, 2, 5] == float("inf")).all() and cell.isinf().sum() == H and not cell.isnan().any()
    c["tables"][3, 1] = 10 ** 6
    got, _, status = _run(kernels, c, H, G, D, V, 2, 30.0, True, None)
    assert status == 2 and torch.equal(got[1:3], clean[1:3]) and got[3].isfinite().all()


@pytest.mark.parametrize("shares, cap, unit, window", [(1, 2.0, True, None), (2, 2.0, False, None), (3, 3.0, True, 200), (1, 30.0, False, 17)])
def test_scores_of_minus_infinity_take_the_cap(shares, cap, unit, window):
    """A key that is seen is capped whatever its score: an infinite key weighs exp(+-cap) as in every other kernel, and is not taken for a
    masked one where its score is -infinity."""
    from glassbox_b200 import kernels
    H, G, D, V = 16, 4, 64, 64
    c = _case(H, G, D, V, [1, 40, 130, 300], 8)
    for i, pos, g, channel in ((0, 0, 1, 3), (1, 39, 0, 0), (1, 30, 3, 5), (2, 129, 2, 63), (2, 120, 2, 1), (3, 170, 1, 9), (3, 299, 0, 33)):
        c["k"][int(c["tables"][i][pos // 16]), g, pos % 16, channel] = float("inf")       # (the sign of a score is the query's)
    att, talk, status = _run(kernels, c, H, G, D, V, shares, cap, unit, window)
    want = _exact(c, H, G, D, V, talk, cap, unit, window)
    assert status == 0 and want.isfinite().all()
    # as above; a score of 30 in float32 adds 30 units of 6e-8 to a weight's relative error
    assert (att.double() - want).abs().max() < 4e-6 * H ** 0.5 * 4 and (att.double() - want).norm() < 2e-6 * want.norm()


def _merge(kernels, H, V, shares, launches=1):
    gen = torch.Generator(device=DEV).manual_seed(V)
    rand = lambda *shape: torch.randn(shape, generator=gen, device=DEV)
    wide, ml, talk = rand(shares * 1, H * V), rand(shares * 1, H * 2), rand(H, H)
    ml[:, 1::2] = ml[:, 1::2].abs() + 1.0
    att, positions = torch.zeros(1, H * V, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    for _ in range(launches):
        kernels.talk_combine(wide, talk, att, positions, H, 1, V, 1, shares=shares, ml=ml, unit_sink=False)
    return wide, ml, talk, att


def test_merges_of_any_size_in_several_threads():
    """The merging kernel's limit of shared memory is one for all threads: 64 heads of 252 channels beside 64 heads of 508."""
    import threading
    from glassbox_b200 import kernels
    failures = []

    def work(V):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                wide, ml, talk, att = _merge(kernels, 64, V, 2, launches=2000)
                torch.cuda.current_stream().synchronize()
                m, l = ml.double().view(2, 64, 2).unbind(-1)
                f = torch.exp(m - m.amax(0))
                rows = (wide.double().view(2, 64, V) * f[..., None]).sum(0) / (l * f).sum(0)[:, None]
                want = talk.double() @ rows
                # float32 sums of 64 products
                assert (att.double().view(64, V) - want).norm() < 2e-6 * want.norm()
        except Exception as e:      # noqa: BLE001 (reported by the thread that asserts)
            failures.append(repr(e))
    threads = [threading.Thread(target=work, args=(V,)) for V in (252, 508, 252, 508)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def test_a_merge_that_no_block_can_hold_says_so():
    from glassbox_b200 import kernels
    with pytest.raises(kernels.KernelError, match="do not fit a block's shared memory"):
        _merge(kernels, 64, 1020, 2)
