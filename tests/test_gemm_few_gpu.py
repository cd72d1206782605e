"""The tcgen05 product for few rows against float64 products of the same bfloat16 numbers: every epilogue, sizes at the edges of its
tiles, row counts around the sixteens, K of one block to a cluster of eight."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SIZES = [(1, 128, 128), (9, 140, 264), (16, 2048, 8192), (17, 264, 2048), (33, 6144, 2048), (40, 576, 1536), (48, 72, 72), (63, 2048, 2048),
         (64, 16384, 512)]


def _operands(M, N, K, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed + M + N)
    x = torch.randn(M, K + 8, generator=g, device=DEV).bfloat16()[:, :K]                  # rows inside a wider buffer
    w = (torch.randn(N, K, generator=g, device=DEV) / K ** 0.5).bfloat16()
    return x, w, x.double() @ w.double().T


def _close(got, want, rounds):
    # sums of K products of unit size in all: float32 partial sums (1e-6), then `rounds` roundings to bfloat16 (2^-8 each at most)
    assert ((got.double() - want).abs() <= 2e-5 + rounds * 2 ** -8 * want.abs()).all(), float((got.double() - want).abs().max())


@pytest.mark.parametrize("M, N, K", SIZES)
def test_products_and_activations(M, N, K):
    from glassbox_b200 import kernels
    x, w, want = _operands(M, N, K)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    out32, added = torch.full((M, N), 7.0, device=DEV), torch.randn(M, N, device=DEV)
    base = added.clone()
    out16, relu, gelu = (torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(3))
    assert kernels.gemm_few_supported(x, w, out32)
    kernels.gemm_few(x, w, out32, st)
    kernels.gemm_few(x, w, added, st, accumulate=True)
    kernels.gemm_few(x, w, out16, st)
    kernels.gemm_few(x, w, relu, st, relu2=True)
    kernels.gemm_few(x, w, gelu, st, gelu=True)
    _close(out32, want, 0)
    _close(added, base.double() + want, 0)
    _close(out16, want, 1)
    _close(relu, want.clamp(min=0) ** 2, 1.1)
    _close(gelu, torch.nn.functional.gelu(want), 1.1)
    again = torch.empty_like(out32)
    kernels.gemm_few(x, w, again, st)
    assert torch.equal(out32, again) and int(st) == 0                       # the same sums in the same order


@pytest.mark.parametrize("M, N, K", SIZES)
def test_gated_unit(M, N, K):
    from glassbox_b200 import kernels
    x, w, sums = _operands(M, 2 * N, K, 1)
    out = torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    kernels.gemm_few(x, w, out, st, gated=True)
    gate, up = sums[:, :N], sums[:, N:]
    _close(out, gate / (1 + torch.exp(-gate)) * up, 1.1)
    assert int(st) == 0


@pytest.mark.parametrize("nh, nkv, hd, page, M, K", [(3, 1, 64, 16, 10, 576), (32, 32, 64, 16, 64, 2048), (4, 2, 128, 8, 33, 256), (5, 1, 64, 5, 17, 264)])
def test_qkv_with_rotation_and_cache_write(nh, nkv, hd, page, M, K):
    from glassbox_b200 import kernels
    N = (nh + 2 * nkv) * hd
    x, w, sums = _operands(M, N, K, 2)
    g = torch.Generator().manual_seed(1)
    pages = M // page + 4
    slots = torch.randperm(pages * page, generator=g)[:M].to(torch.int32)
    positions = torch.randint(0, 90, (M,), generator=g, dtype=torch.int32)
    positions[M // 2] = -1                                                   # a padding row: nothing of it is stored
    angle = torch.rand(100, hd // 2, generator=g) * 6.28
    table = torch.stack([torch.cos(angle), torch.sin(angle)], -1).to(DEV)
    for rope in (table, None):
        k, v = (torch.full((pages, nkv, page, hd), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        q = torch.full((M, nh * hd + 8), 7.0, dtype=torch.bfloat16, device=DEV)
        st = torch.zeros(1, dtype=torch.int32, device=DEV)
        assert kernels.gemm_few_qkv_supported(x, w, hd, q, k)
        kernels.gemm_few_qkv(x, w, q, rope, positions.to(DEV), slots.to(DEV), k, v, nh, nkv, hd, page, True, st)
        assert int(st) == 0
        heads = sums.view(M, nh + 2 * nkv, hd).clone()
        if rope is not None:
            cs = table.double()[positions.clamp(min=0).long().to(DEV)][:, None]
            a, b = heads[..., :hd // 2].clone(), heads[..., hd // 2:].clone()
            turned = torch.cat([a * cs[..., 0] - b * cs[..., 1], b * cs[..., 0] + a * cs[..., 1]], -1)
            heads[:, :nh + nkv] = turned[:, :nh + nkv]
        live = positions >= 0
        _close(q[live, :nh * hd], heads[live, :nh].flatten(1), 1)
        assert torch.all(q[~live] == 7.0) and torch.all(q[:, nh * hd:] == 7.0)
        at = slots[live].long().to(DEV)
        _close(k[at // page, :, at % page], heads[live, nh:nh + nkv], 1)
        _close(v[at // page, :, at % page], heads[live, nh + nkv:], 1)
        assert int((k != 7.0).any(-1).sum()) == int(live.sum()) * nkv
    positions[0], slots[1] = 100, pages * page
    kernels.gemm_few_qkv(x, w, q, table, positions.to(DEV), slots.to(DEV), k, v, nh, nkv, hd, page, True, st)
    assert int(st) == 6                                                      # beyond the table; beyond the pool


def test_a_long_kernel_before_it_is_no_timeout():
    """The kernel may start while the one before it runs; the limits of its waits (0.2 s) must not count that one's time: a walk of
    the delta rule over a million tokens."""
    from glassbox_b200 import kernels
    n, D, V = 1_000_000, 32, 8
    f32 = lambda *s: torch.zeros(*s, device=DEV)
    i32 = lambda *v: torch.tensor(v, dtype=torch.int32, device=DEV)
    qkv, beta, a, state, out = f32(n, 2 * D + V), f32(n, 1), f32(n, 1), f32(1, D * V), f32(n, V)
    x, w, want = _operands(40, 6144, 2048)
    c, st = torch.empty(40, 6144, device=DEV), i32(0)
    args = (qkv, beta, a, f32(1), f32(1), state, out, i32(0, n), i32(0), i32(0), 1, 1, D, V, True, st)
    kernels.gemm_few(x, w, c, st)
    kernels.channel_delta(*args, decay_per_head=True)
    torch.cuda.synchronize()
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    kernels.channel_delta(*args, decay_per_head=True)
    kernels.gemm_few(x, w, c, st)
    end.record()
    torch.cuda.synchronize()
    assert start.elapsed_time(end) > 210, "the walk is shorter than the limit: this test would say nothing"
    assert int(st) == 0
    _close(c, want, 0)
