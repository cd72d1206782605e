"""Rotation with the cache write, and SwiGLU, four channels at a time: odd sizes, rows with no place, channels that are not rotated, and
operands that the four-channel forms do not take."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
#: three float32 roundings (two products and their sum) of numbers up to 5 in size; one bfloat16 rounding of a result up to 8
TOL = {torch.float32: 2e-6, torch.bfloat16: 3.2e-2}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh, nkv, hd, rot, shift", [
    (9, 3, 64, 64, 0),     # 144 units a row: one round of the block
    (32, 32, 64, 64, 0),   # 1,024 units: four rounds
    (4, 2, 32, 16, 0),     # half of the channels rotated
    (3, 1, 24, 8, 0),      # one unit of pairs, four plain
    (2, 1, 64, 0, 0),      # nothing rotated
    (2, 1, 64, 12, 0),     # pairs in no whole units: single channels
    (2, 1, 64, 64, 1),     # rows that start off a piece: single channels
])
def test_rotation_and_cache_write(dtype, nh, nkv, hd, rot, shift):
    from glassbox_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(hd + rot)
    n, ps, max_pos = 5, 8, 40
    wide = (nh + 2 * nkv) * hd
    room = torch.randn(n * wide + shift, generator=g, device=DEV).to(dtype)
    qkv = room[shift:].view(n, wide)
    before = qkv.double()
    table = torch.randn(max_pos, max(rot, 2) // 2, 2, generator=g, device=DEV) if rot else None
    positions = torch.tensor([0, 39, -1, 7, 40], dtype=torch.int32, device=DEV)      # a padding row, a position beyond the table
    slots = torch.tensor([5, 23, 1, 24, 8], dtype=torch.int32, device=DEV)           # a slot beyond the cache
    k, v = torch.full((3, nkv, ps, hd), 9.0, device=DEV).to(dtype), torch.full((3, nkv, ps, hd), 9.0, device=DEV).to(dtype)
    want_k, want_v = k.double(), v.double()
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    kernels.rope_kv_write(qkv, table, positions, slots, k, v, nh, nkv, hd, rot, ps, True, status)
    want = before.clone()
    for r in range(n):
        p, s = int(positions[r]), int(slots[r])
        if p < 0:
            continue
        heads = before[r, :(nh + nkv) * hd].reshape(-1, hd).clone()
        if rot and p < max_pos:
            c, sn = table[p, :, 0].double(), table[p, :, 1].double()
            a, b = heads[:, :rot // 2].clone(), heads[:, rot // 2:rot].clone()
            heads[:, :rot // 2], heads[:, rot // 2:rot] = a * c - b * sn, b * c + a * sn
        want[r, :(nh + nkv) * hd] = heads.reshape(-1)
        if s < 24:
            want_k[s // ps, :, s % ps] = heads[nh:]
            want_v[s // ps, :, s % ps] = before[r, (nh + nkv) * hd:].reshape(nkv, hd)
    scale = max(1.0, float(want.abs().max()) / 8)
    assert int(status) == (2 | (4 if rot else 0))       # a slot, and a position, out of range
    for got, ref in ((qkv, want), (k, want_k), (v, want_v)):
        assert float((got.double() - ref).abs().max()) <= TOL[dtype] * scale


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n, inter", [(1, 4), (8, 1536), (3, 2052), (600, 1028), (593, 2816), (5, 30)])
def test_swiglu(dtype, n, inter):
    from glassbox_b200 import kernels
    g = torch.Generator(device=DEV).manual_seed(inter)
    gu = torch.randn(n, 2 * inter, generator=g, device=DEV).to(dtype)
    act = torch.full((n, inter), 9.0, device=DEV).to(dtype)
    kernels.swiglu(gu, act)
    a, b = gu.double()[:, :inter], gu.double()[:, inter:]
    want = a * torch.sigmoid(a) * b
    # expf within 2 ulp, a division and a product: 5 roundings of 2^-24; bfloat16 rounds the result once more
    rel = (5 * 2 ** -24) if dtype == torch.float32 else 2 ** -8
    assert float(((act.double() - want).abs() - rel * want.abs()).max()) <= 1e-7
