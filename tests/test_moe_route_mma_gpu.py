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


def _route64(z, top, groups, keep, correction, scoring, best):
    """The chosen experts of one row by float64 logits, the scores, and the smallest difference on which a choice rested."""
    score = torch.sigmoid(z) if scoring == "sigmoid" else torch.softmax(z, 0) if scoring == "softmax" else z
    c, margin = score + correction, float("inf")
    if groups > 1:
        runs = c.view(groups, -1)
        run = runs.amax(1) if best else runs.topk(2, 1).values.sum(1)
        order = run.sort(descending=True)
        margin = float(order.values[keep - 1] - order.values[keep])
        c = torch.where(torch.isin(torch.arange(len(z)) // runs.shape[1], order.indices[:keep]), c, -float("inf"))
    order = c.sort(descending=True)
    margin = min(margin, float((order.values[:top] - order.values[1:top + 1]).min()))
    return order.indices[:top], score, margin


@pytest.mark.parametrize("E, top, d, scoring, groups, keep, options", [
    (16, 4, 1024, "sigmoid", 4, 2, dict(correction=True, gate=True, renorm_eps=1e-20)),
    (32, 3, 136, "softmax", 1, 1, dict(gate=True)),                       # (the gate is the first column of a turn of its own)
    (40, 6, 72, "softmax", 8, 3, dict(group_best=True, renorm_eps=0.0)),
    (128, 8, 520, "chosen", 1, 1, dict(bias=True)),
    (31, 2, 2056, "chosen", 1, 1, dict(bias=True, gate=True)),
])
def test_both_forms_choose_alike(E, top, d, scoring, groups, keep, options):
    """The same rows among 256 (by FMA) and among 257 and more (on the tensor cores): their sums are taken in another order, so that a
    logit's low bits and with them the choice between all but equal experts differ; nothing else does."""
    from glassbox_b200 import kernels
    options, g, n = dict(options), torch.Generator().manual_seed(E), 272
    h, w = torch.randn(n, d, generator=g).bfloat16().to(DEV), (torch.randn(E, d, generator=g) / d ** 0.5).to(DEV)
    extra = torch.randn(E, generator=g) / 4
    correction = extra.to(DEV) if options.pop("correction", False) else None
    bias = extra.to(DEV) if options.pop("bias", False) else None
    wg = (torch.randn(1, d, generator=g) / d ** 0.5).to(DEV) if options.pop("gate", False) else None
    out = []
    for step in (n, 257, 256):
        parts = []
        for at in range(0, n, step):
            rows = h[at:at + step].contiguous()
            m = rows.shape[0]
            choice, weight, gate = torch.zeros(m, top, dtype=torch.int32, device=DEV), torch.zeros(m, top, device=DEV), torch.zeros(m, 1, device=DEV)
            kernels.moe_route(rows, w, correction, wg, torch.arange(m, dtype=torch.int32, device=DEV), top, groups, keep, 1.0, choice, weight,
                              gate if wg is not None else None, router_bias=bias, softmax_chosen=scoring == "chosen", softmax=scoring == "softmax", **options)
            parts.append((choice.cpu(), weight.double().cpu(), gate.double().cpu()))
        out.append([torch.cat(x) for x in zip(*parts)])
    z = (h.double() @ w.double().T).cpu() + (extra.double() if bias is not None else 0.0)
    clear = 0
    for r in range(n):
        want, score, margin = _route64(z[r], top, groups, keep, extra.double() if correction is not None else 0.0, scoring, options.get("group_best", False))
        if margin < 2 ** -18:                               # (logits of up to four are off by some 2^-21 in either form)
            continue
        clear += 1
        weight = torch.softmax(score[want], 0) if scoring == "chosen" else score[want]
        if "renorm_eps" in options:
            weight = weight / weight.sum()
        for choice, weights, _ in out:
            assert torch.equal(choice[r].long(), want), r
            assert (weights[r] - weight).abs().max() <= 2 ** -20, r
    assert clear > 0.9 * n
    assert torch.equal(out[0][0][:257], out[1][0][:257]) and torch.equal(out[0][1][:257], out[1][1][:257])      # (one form: the same bits)
    if wg is not None:
        assert max(float((o[2] - torch.sigmoid(h.double() @ wg.double().T).cpu()).abs().max()) for o in out) <= 2 ** -20
