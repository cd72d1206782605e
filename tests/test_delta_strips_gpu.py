"""The forms of the delta rule's elementwise kernels that take four numbers a thread, against the general forms."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("lengths, C, taps", [([96], 4, 4), ([97, 1], 20, 4), ([131, 2, 60], 1028, 3), ([64, 1, 1, 33], 3072, 2), ([2047, 65], 3072, 4), ([1500, 3, 9], 4100, 4)])
def test_convolution_of_four_channels_a_thread_gives_the_bits_of_one(lengths, C, taps):
    """Requests whose first rows read their slots' last inputs, padding rows, a slot that does not exist; rows that start off a 16-byte
    boundary take the general form."""
    from glassbox_b200 import kernels
    torch.manual_seed(C)
    n, S = sum(lengths), len(lengths)
    x, w = torch.randn(n, C, device=DEV), torch.randn(C, taps, device=DEV)
    state0 = torch.randn(S + 1, 8 + (taps - 1) * C, device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    first = i32([sum(lengths[:i]) for i in range(S + 1)])
    row_seq = i32([i for i, l in enumerate(lengths) for _ in range(l)])
    positions = i32([100 + j for l in lengths for j in range(l)])
    positions[5] = -1
    slots = i32([(i + 1) % (S + 1) for i in range(S - 1)] + [S + 7 if S > 2 else 0])
    outs = []
    for shift in (0, 1):
        wide = torch.zeros(n, C + 4, device=DEV)
        wide[:, shift:shift + C] = x
        y, state, status = torch.full((n, C), 7.0, device=DEV), state0.clone(), torch.zeros(1, dtype=torch.int32, device=DEV)
        kernels.short_conv(wide[:, shift:shift + C], w, y, state, 8, row_seq, positions, first, i32([100] * S), slots, True, status)
        outs.append((y, state, status))
    assert int(outs[0][2]) == (2 if S > 2 else 0)
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("lengths, C, taps", [([96], 4100, 4), ([97, 1], 5380, 4), ([131, 2, 60], 2724, 3), ([64, 1, 1, 33], 5300, 2), ([4096], 96, 4)])
def test_the_smallest_that_take_four_channels(lengths, C, taps):
    test_convolution_of_four_channels_a_thread_gives_the_bits_of_one(lengths, C, taps)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n, heads, v, silu", [(1, 1, 4, False), (7, 3, 60, True), (33, 8, 128, False), (5, 2, 132, True), (129, 3, 256, False)])
def test_head_norm_of_four_numbers_a_lane(n, heads, v, silu, dt):
    from glassbox_b200 import kernels
    torch.manual_seed(v)
    o, gate = torch.randn(n, heads * v, device=DEV), 3.0 * torch.randn(n, heads * v + 4, device=DEV)[:, :heads * v]
    w, out = torch.randn(v, device=DEV), torch.empty(n, heads * v, dtype=dt, device=DEV)
    kernels.gated_head_norm(o, gate, w, out, heads, 1e-5, gate_silu=silu)
    x, g = o.double().view(n, heads, v), gate.double().reshape(n, heads, v)
    want = x / (x.pow(2).mean(-1, keepdim=True) + 1e-5).sqrt() * w.double() * torch.sigmoid(g) * (g if silu else 1.0)
    # a dozen float32 roundings of 2^-24 each (the exponential's argument, up to 12, among them), then one of the result's type
    bound = 32 * 2.0 ** -24 + (2.0 ** -8 if dt == torch.bfloat16 else 0.0)
    assert ((out.double().view(n, heads, v) - want).abs() <= bound * want.abs() + 1e-12).all()
