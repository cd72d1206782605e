"""The router's products of many bfloat16 rows on the tensor cores: the choice and the weights of a float64 router, and logits as exact as
sums by FMA."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("n, d, E, top, gate", [(257, 64, 16, 4, False), (300, 1032, 20, 3, True), (272, 200, 128, 8, True), (260, 8, 3, 1, False)])
def test_choice_and_weights(n, d, E, top, gate):
    from glassbox_b200 import kernels
    g = torch.Generator().manual_seed(n)
    h = torch.randn(n, d, generator=g).bfloat16().to(DEV)
    w = (torch.randn(E, d, generator=g) / d ** 0.5).to(DEV)
    wg = (torch.randn(1, d, generator=g) / d ** 0.5).to(DEV) if gate else None
    positions = torch.arange(n, dtype=torch.int32, device=DEV)
    positions[n // 2] = -1
    choice = torch.full((n, top), 77, dtype=torch.int32, device=DEV)
    weight, gates = torch.full((n, top), 5.0, device=DEV), torch.full((n, 1), 5.0, device=DEV) if gate else None
    kernels.moe_route(h, w, None, wg, positions, top, 1, 1, 1.0, choice, weight, gates)
    score = torch.sigmoid(h.double() @ w.double().T)
    live = positions >= 0
    ranked = score.sort(dim=1, descending=True)
    # (a tie of float32 may fall either way: rows whose neighbours in rank differ by less than 1e-6 are left out)
    clear = live & ((ranked.values[:, :top] - ranked.values[:, 1:top + 1]).amin(1) > 1e-6 if E > top else live)
    assert int(clear.sum()) > n // 2
    assert torch.equal(choice[clear].long(), ranked.indices[clear, :top])
    # logits of size one to some 2^-22, halved at most by the sigmoid's slope of a quarter
    assert (weight[clear].double() - ranked.values[clear, :top]).abs().max() <= 2 ** -22
    assert torch.all(choice[~live] == 77) and torch.all(weight[~live] == 5.0)
    if gate:
        assert (gates[live].double() - torch.sigmoid(h.double() @ wg.double().T)[live]).abs().max() <= 2 ** -22
        assert torch.all(gates[~live] == 5.0)


def test_an_infinite_row_is_routed_as_by_fma():
    from glassbox_b200 import kernels
    n, d, E = 270, 64, 8
    g = torch.Generator().manual_seed(1)
    h, w = torch.randn(n, d, generator=g).bfloat16().to(DEV), torch.randn(E, d, generator=g).to(DEV)
    h[5, 7] = float("inf")
    out = []
    for rows in (h, h[5:6].contiguous()):                   # among many, and alone (by FMA)
        choice, weight = torch.zeros(rows.shape[0], 2, dtype=torch.int32, device=DEV), torch.zeros(rows.shape[0], 2, device=DEV)
        kernels.moe_route(rows, w, None, None, torch.arange(rows.shape[0], dtype=torch.int32, device=DEV), 2, 1, 1, 1.0, choice, weight, None)
        out.append((choice, weight))
    assert torch.equal(out[0][0][5], out[1][0][0]) and torch.equal(out[0][1][5], out[1][1][0])
