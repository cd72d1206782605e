"""The quotient of the sigmoid's epilogues against the division itself, number for number: compiled here from the header."""
import ctypes
import os
import subprocess

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
SOURCE = """
#include "common.cuh"
__global__ void compare(const float* v, const float* d, float* ours, float* theirs, long long n) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i < n) { ours[i] = gb_quotient(v[i], d[i]); theirs[i] = __fdiv_rn(v[i], d[i]); }
}
GB_EXPORT int run(const float* v, const float* d, float* ours, float* theirs, long long n, cudaStream_t stream) {
    compare<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(v, d, ours, theirs, n);
    return (int)cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def both(tmp_path_factory):
    from glassbox_b200.csrc import build
    folder = tmp_path_factory.mktemp("quotient")
    src, lib = str(folder / "quotient.cu"), str(folder / "quotient.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build._nvcc(), *build.ARCH_FLAGS, *build.NVCC_FLAGS, "-I", build.HERE, "-shared", src, "-o", lib], check=True)
    run = ctypes.CDLL(lib).run
    run.argtypes = [ctypes.c_void_p] * 4 + [ctypes.c_longlong, ctypes.c_void_p]

    def call(v, d):
        v, d = v.contiguous(), d.contiguous()
        ours, theirs = torch.empty_like(v), torch.empty_like(v)
        assert run(v.data_ptr(), d.data_ptr(), ours.data_ptr(), theirs.data_ptr(), v.numel(), torch.cuda.current_stream().cuda_stream) == 0
        return ours, theirs
    return call


def _same(ours, theirs):
    return (ours.view(torch.int32) == theirs.view(torch.int32)) | (torch.isnan(ours) & torch.isnan(theirs))


@pytest.mark.parametrize("seed", range(4))
def test_sigmoid_quotients_have_the_bits_of_the_division(both, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = 1 << 26
    v = torch.randn(n, generator=g, device=DEV) * torch.tensor([0.01, 1.0, 10.0, 60.0], device=DEV)[seed]
    ours, theirs = both(v, 1.0 + torch.exp(-v))
    assert _same(ours, theirs).all(), int((~_same(ours, theirs)).sum())
    # any numerator whose remainder is a normal number, any denominator from 1 to 2^125: random significands and exponents
    bits = lambda lo, hi: (torch.randint(lo, hi, (n,), generator=g, device=DEV, dtype=torch.int32) << 23) | \
        torch.randint(0, 1 << 23, (n,), generator=g, device=DEV, dtype=torch.int32)
    d = bits(127, 252).view(torch.float32)
    v = (bits(127, 254).view(torch.float32).view(torch.int32) | (torch.randint(0, 2, (n,), generator=g, device=DEV, dtype=torch.int32) << 31)).view(torch.float32)
    ours, theirs = both(v, d)
    ok = _same(ours, theirs) | (theirs.abs() < 2.0 ** -100)
    assert ok.all(), int((~ok).sum())


def test_the_edges(both):
    inf, nan, big = float("inf"), float("nan"), 3.4e38
    values = [0.0, -0.0, 1.0, -1.0, 1e-30, -88.0, -89.0, 88.0, big, -big, inf, -inf, nan]
    dens = [1.0, 1.0000001, 1.9999999, 2.0, 3.0, 9.9e36, 1.0e37, 1.1e37, 8.5e37, 1.7e38, big, inf, nan]
    v = torch.tensor(values, device=DEV).repeat_interleave(len(dens))
    d = torch.tensor(dens, device=DEV).repeat(len(values))
    ours, theirs = both(v, d)
    # a quotient below the normal numbers is rounded twice at most: half of the smallest subnormal, one more for the estimate's
    ok = _same(ours, theirs) | ((ours - theirs).abs() <= 2.0 ** -148)
    assert ok.all(), [(float(a), float(b), float(x), float(y)) for a, b, x, y, k in zip(v, d, ours, theirs, ok) if not k]


def test_an_infinite_gate_of_the_gated_product():
    """silu(inf) * up is inf * up, as it is with the division."""
    from glassbox_b200 import kernels
    M, K, inter = 200, 64, 64
    a = torch.zeros(M, K, device=DEV).bfloat16()
    a[:, 0] = 1.0
    w = torch.zeros(2 * inter, K, device=DEV).bfloat16()
    w[:inter, 0], w[inter:, 0] = torch.linspace(-3, 3, inter, device=DEV).bfloat16(), 2.0
    w[5, 0], w[9, 0] = float("inf"), float("-inf")
    out = torch.zeros(M, inter, dtype=torch.bfloat16, device=DEV)
    kernels.gemm_tc_gated(a, w, out, torch.zeros(1, dtype=torch.int32, device=DEV))
    g = w[:inter, 0].float()
    want = (g / (1 + torch.exp(-g)) * 2.0).expand(M, inter)
    assert torch.isposinf(out[:, 5]).all() and torch.isnan(out[:, 9]).all()
    keep = [i for i in range(inter) if i not in (5, 9)]
    assert ((out[:, keep].float() - want[:, keep]).abs() <= 2 ** -8 * want[:, keep].abs() + 1e-6).all()
