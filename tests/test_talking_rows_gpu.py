"""The many-row forms of the talking-heads mixer's elementwise kernels against their general forms."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n, H, G, V", [(1024, 4, 1, 4), (257, 16, 4, 64), (513, 9, 9, 20), (350, 6, 3, 36), (1030, 24, 3, 128), (512, 2, 2, 8)])
def test_the_mix_of_many_rows_gives_the_bits_of_the_mix_of_few(n, H, G, V, dt):
    from glassbox_b200 import kernels
    torch.manual_seed(n)
    wide = torch.randn(n * H, G * V, device=DEV)
    talk = torch.randn(H, H, device=DEV)
    pos = torch.randint(0, 50, (n,), dtype=torch.int32, device=DEV)
    pos[::7] = -1
    got, ref = (torch.full((n, H * V), 7.0, dtype=dt, device=DEV) for _ in range(2))
    assert n * G >= 1024
    kernels.talk_combine(wide, talk, got, pos, H, G, V, G)
    for r in range(0, n, 100):                                   # (few rows take the block per pair)
        kernels.talk_combine(wide[r * H:(r + 100) * H], talk, ref[r:r + 100], pos[r:r + 100], H, G, V, G)
    assert torch.equal(got, ref)
    assert (got[::7] == 7).all() and (got[1] != 7).any()


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n, H, G, D, V, rot, biased, write", [(1, 16, 4, 64, 64, 64, True, True), (37, 16, 4, 64, 64, 32, False, True), (5, 3, 1, 20, 12, 8, True, True),
                                                               (300, 8, 8, 128, 96, 0, True, True), (9, 6, 2, 32, 36, 24, True, False)])
def test_four_channels_a_thread_write_what_one_channel_a_thread_writes(n, H, G, D, V, rot, biased, write, dt):
    from glassbox_b200 import kernels
    torch.manual_seed(n + D)
    ps, pages, cols = 16, 24, (H + G) * D + G * V
    outs = []
    wide = torch.randn(n, cols + 8, device=DEV)
    bias = torch.randn(cols, device=DEV) if biased else None
    table = torch.randn(40, rot // 2, 2, device=DEV) if rot else None
    pos = torch.randint(0, 40, (n,), dtype=torch.int32, device=DEV)
    if n > 4:
        pos[3] = -1
    slots = torch.randperm(ps * pages, device=DEV)[:n].to(torch.int32)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    for shift in (0, 1):                                         # a row that starts off a 16-byte boundary takes the general form
        rows = torch.zeros(n, cols + 8, device=DEV)
        rows[:, shift:shift + cols] = wide[:, :cols]
        q = torch.full((n, H * D), 7.0, dtype=dt, device=DEV)
        k, v = torch.zeros(pages, G, ps, D, dtype=dt, device=DEV), torch.zeros(pages, G, ps, V, dtype=dt, device=DEV)
        kernels.bias_rope_write(rows[:, shift:shift + cols], bias, table, pos, slots, q, k, v, H, G, D, V, rot, ps, write, st)
        outs.append((q, k, v))
    assert int(st) == 0
    eps = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -23
    for a, b in zip(*outs):
        # the two forms may contract u cos - v sin to different fused products: an ulp of terms below 32 (normals), once rounded
        assert ((a.double() - b.double()).abs() <= eps * b.double().abs() + 32 * 2.0 ** -23).all()
    assert write or not outs[0][1].any()
