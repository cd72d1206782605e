"""Float32 decode attention: its splits come together in a cluster where the rule lets them and through global memory where not; a
grid has no more blocks than a row can have rounds of 256 (head size 64) or 128 keys."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("lens, nh, nkv, hd, ps, window", [
    ([1], 9, 3, 64, 16, None),                         # one block: a cluster of one
    ([256, 257], 9, 3, 64, 16, None),                  # a round, and one key more: blocks of the cluster without keys
    ([2048], 15, 5, 64, 16, None),                     # eight blocks, all of them busy
    ([2049], 9, 3, 64, 16, None),                      # more than a cluster holds
    ([700, 0, 3, 511, 512, 513], 9, 3, 64, 8, None),   # more rows than clusters find room, a padding row
    ([700, 0, 3], 9, 3, 64, 8, None),                  # a padding row in a cluster
    ([1000, 129], 20, 4, 128, 16, None),               # a group in two parts (four heads and one)
    ([900, 40], 4, 4, 64, 16, 300),                    # a window: two rounds, whatever the table's width
    ([900] * 40, 8, 2, 128, 16, 100),                  # a window of one round: no partner
])
@pytest.mark.parametrize("splits", [1, 2, 25])
def test_splits_give_the_softmax(lens, nh, nkv, hd, ps, window, splits):
    from glassbox_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(len(lens) + lens[0])
    needs = [-(-n // ps) for n in lens]
    width = 1 << (max(needs) - 1).bit_length()
    pages = sum(needs)
    k = torch.randn(pages, nkv, ps, hd, generator=g, device=DEV)
    v = torch.randn(pages, nkv, ps, hd, generator=g, device=DEV)
    tables = torch.full((len(lens), width), -1, dtype=torch.int32, device=DEV)
    at = 0
    for i, n in enumerate(needs):
        tables[i, :n] = torch.arange(at, at + n, device=DEV, dtype=torch.int32).flip(0)
        at += n
    n = len(lens)
    positions = torch.tensor([x - 1 for x in lens], dtype=torch.int32, device=DEV)
    q = torch.randn(n, nh * hd, generator=g, device=DEV)
    acc = torch.full((n * nh * splits * hd,), float("nan"), device=DEV)
    ml = torch.full((n * nh * splits * 2,), float("nan"), device=DEV)
    counters = torch.zeros(n * nh, dtype=torch.int32, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    for _ in range(2):                                 # the counters are left at zero
        out = torch.full((n, nh * hd), 7.0, device=DEV)
        kernels.attention_decode(q, out, k, v, tables, torch.arange(n, dtype=torch.int32, device=DEV), positions, nh, nkv, hd, ps,
                                 hd ** -0.5, window, splits, acc, ml, counters, status)
        assert int(status) == 0 and int(counters.abs().max()) == 0
        for i, length in enumerate(lens):
            if length == 0:
                assert int(out[i].count_nonzero()) == 0
                continue
            rows = tables[i, :needs[i]].long()
            first = max(0, length - window) if window else 0
            kk = k[rows].permute(1, 0, 2, 3).reshape(nkv, -1, hd)[:, first:length].double()
            vv = v[rows].permute(1, 0, 2, 3).reshape(nkv, -1, hd)[:, first:length].double()
            qq = q[i].reshape(nkv, nh // nkv, hd).double()
            p = torch.softmax(torch.einsum("kgd,ktd->kgt", qq, kk) * hd ** -0.5, -1)
            want = torch.einsum("kgt,ktd->kgd", p, vv).reshape(-1)
            # a score (some hundred products in float32, up to 8 in size) is off by 1e-5 at most and an expf by 2 ulp: a weight by
            # 2e-5 of itself, the output by that times the largest value (5)
            assert float((out[i] - want).abs().max()) <= 1e-4
