"""The experts' grouped products at the edges of their tiles: experts with 0, 1, 127, 128, 129 and many pairs, outputs and widths
that are no multiple of a tile, against float64 products of the same bfloat16 numbers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _case(E, top, d, ff, unit, counts, seed):
    """Rows whose choices give expert e exactly counts[e] pairs (top distinct experts a row), a padding row among them."""
    g = torch.Generator().manual_seed(seed)
    left, rows = list(counts), []
    while sum(left):
        order = sorted(range(E), key=lambda e: -left[e])[:top]
        rows.append([e if left[e] else -1 for e in order])
        for e in order:
            left[e] -= 1 if left[e] else 0
    pad = len(rows) // 2
    rows.insert(pad, list(range(top)))
    n = len(rows)
    positions = torch.arange(n, dtype=torch.int32)
    positions[pad] = -1
    up_rows = 2 * ff if unit else ff
    h = torch.randn(n, d, generator=g).bfloat16()
    w_up, w_down = (torch.randn(E * up_rows, d, generator=g) / d ** 0.5).bfloat16(), (torch.randn(E * d, ff, generator=g) / ff ** 0.5).bfloat16()
    return h, w_up, w_down, torch.tensor(rows, dtype=torch.int32), positions


@pytest.mark.parametrize("E, top, d, ff, unit, counts", [
    (5, 2, 64, 64, None, [129, 0, 128, 1, 127]),
    (4, 1, 72, 264, None, [300, 5, 0, 64]),
    (3, 2, 136, 40, "silu", [200, 130, 90]),
    (16, 4, 256, 512, "clamped", [128] * 8 + [7] * 8),
    (40, 2, 512, 136, None, [3] * 39 + [40]),
])
def test_grouped_products(E, top, d, ff, unit, counts):
    from glassbox_b200 import kernels
    h, w_up, w_down, choice, positions = _case(E, top, d, ff, unit, counts, d + ff)
    n = h.shape[0]
    pair_unit = {None: None, "silu": kernels.SILU_UNIT, "clamped": (7.0, 1.702)}[unit]
    tables = torch.zeros(E + 1 + n * top, dtype=torch.int32, device=DEV)
    act = torch.full((n, top * ff), float("nan"), dtype=torch.bfloat16, device=DEV)
    pair = torch.full((n, top * d), 7.0, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    kernels.moe_experts_grouped(h.to(DEV), w_up.to(DEV), w_down.to(DEV), E, choice.to(DEV), positions.to(DEV), tables, act, pair, unit=pair_unit,
                                status=status)
    assert int(status) == 0
    got = pair.cpu().double().view(n, top, d)
    up, down = w_up.double().view(E, -1, d), w_down.double().view(E, d, ff)
    for r in range(n):
        for k in range(top):
            e = int(choice[r, k])
            if positions[r] < 0 or e < 0:
                assert torch.all(got[r, k] == 7.0)
                continue
            x = up[e] @ h[r].double()
            if unit == "silu":
                x = x[0::2] / (1 + torch.exp(-x[0::2])) * x[1::2]
            elif unit == "clamped":
                g = x[0::2].clamp(max=7.0)
                x = g / (1 + torch.exp(-1.702 * g)) * (x[1::2].clamp(-7.0, 7.0) + 1)
            else:
                x = x.clamp(min=0) ** 2
            want = down[e] @ x
            # the activations are rounded to bfloat16 (2^-9 each) in front of a sum of ff products with weights of size ff^-1/2
            # (four of its standard deviations, and a quarter for the largest of some thousand sums)
            assert (got[r, k] - want).abs().max() <= 2 ** -9 * 5 * float(x.norm()) / ff ** 0.5 + 1e-5, (r, k, e)


def test_the_unit_divides_as_float32_does():
    """Gates near -87.5, whose denominators lie above 2^126: the quotients, some -1e-36, come out as numbers (times an up sum of 2^100)."""
    from glassbox_b200 import kernels
    n, d, ff = 40, 64, 64
    h = torch.zeros(n, d)
    h[:, 0] = 1.0
    gates = -torch.linspace(86, 88, ff).bfloat16().float()
    w_up, w_down = torch.zeros(ff, 2, d), torch.eye(d, ff)
    w_up[:, 0, 0], w_up[:, 1, 0] = gates, 2.0 ** 100
    dev = lambda t: t.bfloat16().to(DEV).contiguous()
    i32 = lambda *shape: torch.zeros(*shape, dtype=torch.int32, device=DEV)
    pair, status = torch.zeros(n, d, device=DEV), i32(1)
    kernels.moe_experts_grouped(dev(h), dev(w_up.view(2 * ff, d)), dev(w_down), 1, i32(n, 1), torch.arange(n, dtype=torch.int32, device=DEV),
                                i32(2 + n), torch.zeros(n, ff, dtype=torch.bfloat16, device=DEV), pair, unit=kernels.SILU_UNIT, status=status)
    want = gates.double() / (1 + torch.exp(-gates.double())) * 2.0 ** 100
    # float32: the exponential's argument is exact, its value and the quotient a few 2^-23 off; then one rounding to bfloat16
    assert int(status) == 0
    assert ((pair.double().cpu() - want).abs() <= 2 ** -8 * want.abs()).all()


@pytest.mark.parametrize("E, top, d, ff, unit, counts", [
    (3, 2, 72, 40, "silu", [129, 0, 64]),
    (2, 1, 264, 136, None, [1, 255]),
    (4, 3, 1032, 64, None, [128, 127, 65, 3]),
])
def test_rows_gathered_before_the_product(E, top, d, ff, unit, counts):
    """The input rows brought into the pairs' order by a pass of their own: the bits of the product that fetches them row by row."""
    from glassbox_b200 import kernels
    h, w_up, w_down, choice, positions = (t.to(DEV) for t in _case(E, top, d, ff, unit, counts, d))
    n, out = h.shape[0], []
    for gathered in (None, torch.full((n, top * d), float("nan"), dtype=torch.bfloat16, device=DEV)):
        tables, status = torch.zeros(E + 1 + n * top, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        act, pair = torch.zeros((n, top * ff), dtype=torch.bfloat16, device=DEV), torch.full((n, top * d), 7.0, device=DEV)
        kernels.moe_experts_grouped(h, w_up, w_down, E, choice, positions, tables, act, pair, unit=kernels.SILU_UNIT if unit else None,
                                    status=status, gathered=gathered)
        assert int(status) == 0
        out.append(pair)
    assert torch.equal(*out)
