"""The latent mixer's small kernels with eight numbers a thread against their general forms (rows off a 16-byte boundary)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("n, H, dq, r, c, rot, half, write", [
    (1, 1, 8, 8, 8, 8, False, True), (37, 32, 64, 64, 128, 64, False, True), (300, 16, 64, 32, 128, 32, True, False), (9, 5, 16, 24, 64, 16, True, True),
    (66, 3, 0, 40, 1024, 24, False, True), (5, 2, 8, 16, 96, 0, True, True), (130, 40, 64, 64, 128, 48, True, True)])
def test_cache_write_of_eight_numbers_a_thread(n, H, dq, r, c, rot, half, write):
    from glassbox_b200 import kernels
    torch.manual_seed(n + H)
    cols, page = H * (dq + r) + c + r, 16
    proj = torch.randn(n, cols, device=DEV).bfloat16()
    gain, freqs = torch.randn(c, device=DEV), torch.rand(max(rot // 2, 1), device=DEV)
    positions = torch.randint(0, 5000, (n,), dtype=torch.int32, device=DEV)
    slots = torch.randperm(n + 20, device=DEV)[:n].to(torch.int32)
    if n > 4:
        positions[3], slots[4] = -1, 10 ** 6
    outs = []
    for shift in (0, 1):
        wide = torch.zeros(n, cols + 8, device=DEV, dtype=torch.bfloat16)
        wide[:, shift:shift + cols] = proj
        q = torch.full((n, H * (c + r)), 7.0, device=DEV, dtype=torch.bfloat16)
        cache = torch.full(((n + 35) // page, 1, page, c + r), 7.0, device=DEV, dtype=torch.bfloat16)
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        kernels.latent_kv_write(wide[:, shift:shift + cols], H * (dq + r), q, cache, gain, freqs, positions, slots, H, dq, r, c, rot, 1e-5, write, status,
                                half_pairs=half, magnitude=1.25)
        outs.append((q, cache, status))
    assert int(outs[0][2]) == int(outs[1][2]) == (2 if n > 4 and write else 0)
    for x, y in zip(outs[0][:2], outs[1][:2]):
        # u cos - v sin may contract to one fused product or the other, the latent's sum of squares runs in another order: an ulp of float32
        # terms below 16 (normals by 1.25), then a rounding to bfloat16 that may fall the other way (2^-8 of the number)
        assert ((x.double() - y.double()).abs() <= 2.0 ** -7 * y.double().abs() + 16 * 2.0 ** -23).all()
    assert write == bool((outs[0][1] != 7.0).any()) and (outs[0][0][:, c:] != 7.0).any()


@pytest.mark.parametrize("n, H, dq, r, c, rot, half, write", [
    (1, 96, 8, 8, 128, 8, False, True), (33, 127, 16, 8, 8, 8, False, True), (9, 40, 16, 32, 64, 16, True, True), (5, 30, 8, 40, 96, 0, True, True),
    (300, 40, 64, 32, 128, 32, True, False), (7, 1, 0, 1024, 1024, 1024, False, True)])
def test_the_smallest_rows_that_take_eight_numbers_a_thread(n, H, dq, r, c, rot, half, write):
    test_cache_write_of_eight_numbers_a_thread(n, H, dq, r, c, rot, half, write)


@pytest.mark.parametrize("n, heads, N, K, gated", [(1, 1, 8, 16, False), (65, 3, 128, 64, False), (200, 2, 64, 128, True), (63, 5, 72, 16, True), (17, 4, 136, 256, False),
                                                   (130, 2, 192, 48, True)])
def test_per_head_product_with_whole_rows_stored(n, heads, N, K, gated):
    from glassbox_b200 import kernels
    torch.manual_seed(N + K)
    a, w = torch.randn(n, heads * K, device=DEV).bfloat16(), torch.randn(heads, N, K, device=DEV).bfloat16()
    gate = torch.randn(n, heads * N, device=DEV) if gated else None
    outs = []
    for pad in (8, 2):                                                # (heads off a 16-byte boundary: pairs of columns)
        out = torch.full((n, heads * (N + pad)), 7.0, device=DEV, dtype=torch.bfloat16)
        kernels.head_linear(a, w, out, K, N + pad, gate=gate)
        outs.append(out.view(n, heads, N + pad))
    assert torch.equal(outs[0][..., :N], outs[1][..., :N]) and (outs[0][..., N:] == 7.0).all() and (outs[1][..., N:] == 7.0).all()
    want = torch.einsum("nhk,hok->nho", a.double().view(n, heads, K), w.double())
    if gated:
        want = want * torch.sigmoid(gate.double().view(n, heads, N))
    assert (outs[0][..., :N].double() - want).abs().max() <= 2.0 ** -8 * want.abs().max() + 1e-3
