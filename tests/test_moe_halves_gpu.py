"""The routed experts' halves row by row: four matrix rows a warp, and the form that takes what is not aligned."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("n, top, E, d, ff", [(1, 1, 2, 8, 1), (3, 2, 5, 64, 33), (5, 2, 4, 1032, 34), (8, 4, 16, 264, 1040), (2, 2, 3, 36, 31), (4, 1, 3, 20, 12)])
def test_expert_halves_at_ragged_sizes(n, top, E, d, ff, gated, dt):
    """Rows that are no multiple of a block's 32, K around the 16-byte loads of a warp (1,024 bfloat16, 512 float32) and not in whole
    pieces; a choice that names no expert gives zeros, a padding row is left alone."""
    from glassbox_b200 import kernels
    torch.manual_seed(n * d + ff)
    h = torch.randn(n, d, device=DEV).to(dt)
    up = (torch.randn(E * ff * (2 if gated else 1), d, device=DEV) * d ** -0.5).to(dt)
    down = (torch.randn(E * d, ff, device=DEV) * ff ** -0.5).to(dt)
    choice = torch.randint(0, E, (n, top), dtype=torch.int32, device=DEV)
    positions = torch.zeros(n, dtype=torch.int32, device=DEV)
    if n > 2:
        choice[1, 0], positions[2] = -1, -1
    act, pair = torch.full((n, top * ff), 7.0, device=DEV), torch.full((n, top * d), 7.0, device=DEV)
    kernels.moe_expert_halves(h, up, down, E, choice, positions, act, pair, unit=kernels.SILU_UNIT if gated else None)
    H, U, D = h.double(), up.double().reshape(E, -1, d), down.double().reshape(E, d, ff)
    for r in range(n):
        for t in range(top):
            a, p = act[r, t * ff:(t + 1) * ff].double(), pair[r, t * d:(t + 1) * d].double()
            if int(positions[r]) < 0:
                assert (a == 7).all() and (p == 7).all()
                continue
            e = int(choice[r, t])
            if e < 0:
                assert not a.any() and not p.any()
                continue
            x = U[e] @ H[r]
            ref = x[0::2] * torch.sigmoid(x[0::2]) * x[1::2] if gated else x.clamp(min=0) ** 2
            # float32 sums of d products whose squares sum to about |h|^2 / d, the activation's slope below 4 |x| + 4
            assert (a - ref).abs().max() <= 2.0 ** -22 * d ** 0.5 * (4 * x.abs().max() + 4) ** 2
            assert (p - D[e] @ a).abs().max() <= 2.0 ** -22 * ff ** 0.5 * (1 + a.abs().max())
