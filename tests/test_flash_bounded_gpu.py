"""Capped scores in the wide flash kernel: from the second key tile on no maximum is formed, so scores that climb from one end of the cap to the
other must still give finite weights and the right ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("cap", [0.5, 8.0, 30.0, 32.0, 33.0, 50.0])
@pytest.mark.parametrize("low, high, window", [(-1.0, 1.0, None), (1.0, -1.0, None), (-0.5, 0.2, None), (-1.0, 1.0, 300)])
@pytest.mark.parametrize("G, page", [(4, 16), (2, 16), (4, 128)])
def test_scores_that_climb_across_the_cap(cap, low, high, window, G, page):
    _climb(cap, low, high, window, G, page, 1e6)


@pytest.mark.parametrize("size", [1e27, 1e-15, 1e-18])
@pytest.mark.parametrize("cap, low, high", [(8.0, -1.0, 1.0), (30.0, -1.0, 1.0), (32.0, -1.0, 1.0), (30.0, 1.0, -1.0), (32.0, -0.1, 1.0)])
def test_values_keep_their_range_whatever_the_scores_do(cap, low, high, size):
    """Large values meet no weight that makes their sums overflow and small ones none that the sums could lose, wherever in the cap the
    first keys lie."""
    _climb(cap, low, high, None, 4, 16, size)


def _climb(cap, low, high, window, G, page, size):
    from glassbox_b200 import kernels
    H, rows = 4, 700
    gen = torch.Generator(device=DEV).manual_seed(int(cap))
    used = -(-rows // page)
    table = torch.randperm(used, generator=torch.Generator().manual_seed(3)).to(torch.int32)[None].to(DEV)
    q = torch.zeros(rows, H, 64, device=DEV)
    q[..., 0] = 4.0 * cap                                                # (scores of four times the cap: its ends, to the last bit or two)
    q[..., 1:] = 0.1 * torch.randn(rows, H, 63, device=DEV, generator=gen)
    q = q.view(rows, -1).bfloat16()
    dense = torch.randn(rows, G, 64, device=DEV, generator=gen)
    dense[..., 0] = torch.linspace(low, high, rows, device=DEV)[:, None]
    v = torch.randn(rows, G, 64, device=DEV, generator=gen) * size
    pool = lambda t: torch.cat([t, torch.zeros(used * page - rows, G, 64, device=DEV)]).view(used, page, G, 64).transpose(1, 2)
    k, vals = torch.zeros(used, G, page, 64, device=DEV, dtype=torch.bfloat16), torch.zeros(used, G, page, 64, device=DEV, dtype=torch.bfloat16)
    k[table[0].long()], vals[table[0].long()] = pool(dense).bfloat16(), pool(v).bfloat16()
    out, status = torch.full((rows, H * G * 64), 7.0, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    kernels.talking_attention_flash(q, out, k, vals, table, i32([0, rows]), i32([0]), rows, heads=H, kv_heads=G, dim=64, vdim=64, value_heads=G,
                                    page_size=page, scale=1.0, softcap=cap, unit_sink=True, window=window, status=status)
    assert int(status) == 0 and out.isfinite().all()
    at, pos = torch.arange(rows, device=DEV)[None], torch.arange(rows, device=DEV)[:, None]
    seen = (at <= pos) & (at > pos - (window or rows))
    values = v.bfloat16().double().view(rows, -1)
    for h in range(H):
        s = q.double().view(rows, H, 64)[:, h] @ dense.bfloat16().double()[:, h // (H // G)].T
        s = (cap * torch.tanh(s / cap)).masked_fill(~seen, float("-inf"))
        top = s.amax(-1, keepdim=True).clamp(min=0.0)
        w = torch.exp(s - top)
        w = w / (w.sum(-1, keepdim=True) + torch.exp(-top))
        # every weight is rounded to bfloat16 (2^-9 of it) and its capped score is off by a few 2^-24 of the cap: the sum of |weight| |value|
        # times 2^-8 bounds both
        err = (out.view(rows, H, -1)[:, h].double() - w @ values).abs()
        assert (err <= 2.0 ** -8 * (w @ values.abs()) + 1e-26 * size).all(), h
