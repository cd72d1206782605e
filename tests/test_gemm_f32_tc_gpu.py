"""The product of float32 rows on the tensor cores at the edges of its tiles and steps, against float64; its error beside that of FMA."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _operands(M, N, K, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    a, w = torch.randn(M, K, generator=g).to(DEV), (torch.randn(N, K, generator=g) / K ** 0.5).to(dtype).to(DEV)
    return a, w, a.double() @ w.double().T


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M, N, K", [(9, 8, 64), (128, 64, 68), (129, 65, 96), (300, 130, 100), (20, 1000, 36), (257, 19000, 64), (2047, 960, 72)])
def test_product_of_float32_rows(M, N, K, dtype):
    from glassbox_b200 import kernels
    a, w, ref = _operands(M, N, K, dtype, M + N)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    for pad, add in ((0, False), (3, True)):            # (three columns beside the output: its rows then start anywhere)
        buf = torch.full((M, N + pad), 2.0, device=DEV)
        kernels.gemm_f32_tc(a, w, buf[:, :N], accumulate=add, status=status)
        # sums of K products of size K^-1/2 each: K / 32 roundings of 2^-24 of up to the largest sum seen, and one of the addition
        assert (buf[:, :N].double() - ref - (2.0 if add else 0.0)).abs().max() <= 2 ** -24 * (K / 32 + 4) * (float(ref.abs().max()) + 2.0)
        assert torch.all(buf[:, N:] == 2.0)
    wide = torch.zeros(M, K + 8, device=DEV)
    wide[:, 4:K + 4] = a
    out = torch.empty(M, N, device=DEV)
    kernels.gemm_f32_tc(wide[:, 4:K + 4], w, out, status=status)
    part = torch.empty(9, N, device=DEV)
    kernels.gemm_f32_tc(a[-9:], w, part, status=status)
    assert torch.equal(part, out[-9:]) and int(status) == 0                  # a row's bits do not depend on the rows beside it


@pytest.mark.parametrize("K", [64, 576, 1536])
@pytest.mark.parametrize("kind", ["normal", "positive", "spread"])
def test_as_exact_as_fma(K, kind):
    from glassbox_b200 import kernels
    a, w, _ = _operands(256, 256, K, torch.float32, K)
    if kind == "positive":
        a, w = a.abs(), w.abs()
    elif kind == "spread":
        a = a * torch.exp(3 * torch.randn(a.shape, device=DEV, generator=torch.Generator(DEV).manual_seed(1)))
    ref, out = a.double() @ w.double().T, []
    for product in (kernels.gemm_f32_tc, kernels.gemm_simt):
        c = torch.empty(256, 256, device=DEV)
        product(a, w, c)
        out.append(float((c.double() - ref).norm()))
    assert out[0] <= out[1], out


@pytest.mark.parametrize("numbers", [1, 2, 8])
@pytest.mark.parametrize("N", [64, 4000])                   # (both tile widths)
def test_rows_of_few_numbers_are_as_exact_as_by_fma(numbers, N):
    from glassbox_b200 import kernels
    a, w, _ = _operands(512, N, 576, torch.float32, numbers)
    g = torch.Generator().manual_seed(numbers)
    keep = torch.zeros(512, 576).scatter_(1, torch.rand(512, 576, generator=g).argsort(1)[:, :numbers], 1.0).to(DEV)
    a *= keep
    a[:64] = torch.where(keep[:64] > 0, torch.tensor(0x3F80FFFF, dtype=torch.int32).view(torch.float32).item(), 0.0)
    w[:32] = a.max() if numbers == 1 else w[:32]
    ref, error = a.double() @ w.double().T, []
    for product in (kernels.gemm_f32_tc, kernels.gemm_simt):
        c = torch.empty(512, N, device=DEV)
        product(a, w, c)
        error.append((c.double() - ref).abs())
    if numbers == 1:                                        # one product: 2^-24 for its rounding, a few 2^-32 for terms left out and cut
        assert (error[0] <= 2 ** -24 * (1 + 2 ** -6) * ref.abs()).all()
    assert float(error[0].norm()) <= float(error[1].norm()) * (1 + 2 ** -6)


def test_what_is_not_finite_is_as_by_fma():
    """Infinities, NaN and sums that overflow, in their own rows and columns alone."""
    from glassbox_b200 import kernels
    a, w, _ = _operands(200, 96, 64, torch.float32, 3)
    a[3, 5], a[150, 63], a[77, 0] = float("inf"), float("nan"), -float("inf")
    w[9, 5], w[95, 0] = 0.0, float("inf")
    a[100], w[20] = 3e38, 2.0
    got, want = torch.empty(200, 96, device=DEV), torch.empty(200, 96, device=DEV)
    kernels.gemm_f32_tc(a, w, got)
    kernels.gemm_simt(a, w, want)
    # (row 100: a sum of 64 numbers up to 4e37 may pass 3.4e38 on the way in one order and not in another; with w[20] it ends there)
    assert got[100, 20] == want[100, 20] == float("inf")
    got[100], want[100] = 0.0, 0.0
    finite = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), finite) and torch.equal(got[~finite].nan_to_num(7.0, 8.0, 9.0), want[~finite].nan_to_num(7.0, 8.0, 9.0))
    rows = torch.tensor([r for r in range(200) if r not in (3, 77, 100, 150)], device=DEV)
    clean = (a[rows].double() @ w[:95].double().T)
    assert (got[rows][:, :95].double() - clean).abs().max() <= 1e-5 * float(clean.abs().max())
