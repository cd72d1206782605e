"""float32 prompt attention on the tensor cores: what a row does not see stays away from it whatever it holds, what it sees counts as in
float32, and both forms of the kernel give the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _run(q, k, v, tables, first, start, rows, window=None):
    from glassbox_b200 import kernels
    nkv, ps, hd = k.shape[1:]
    out, status = torch.full_like(q, 7.0), torch.zeros(1, dtype=torch.int32, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    kernels.attention_prefill_f32(q, out, k, v, i32(tables), i32(first), i32(start), rows, q.shape[1] // hd, nkv, hd, ps, hd ** -0.5, window, status)
    assert int(status) == 0
    return out


def _truth(q, keys, values, start, window=None):
    """One head: q [rows, hd], keys and values [context, hd]; what a row does not see is left out of its sums."""
    rows = []
    for r in range(q.shape[0]):
        lo, hi = max(0, start + r + 1 - window) if window else 0, start + r + 1
        s = (q[r].double() * q.shape[1] ** -0.5) @ keys[lo:hi].double().T
        rows.append(torch.softmax(s, 0) @ values[lo:hi].double())
    return torch.stack(rows)


def _pool(n, hd, seed):
    g = torch.Generator().manual_seed(seed)
    pages = -(-n // 16)
    return tuple(torch.randn(pages, 1, 16, hd, generator=g).to(DEV) for _ in range(2)) + (torch.randn(n, hd, generator=g).to(DEV),)


@pytest.mark.parametrize("hd", [16, 32, 64])
@pytest.mark.parametrize("n, start, window", [(1, 0, None), (64, 0, None), (65, 0, 33), (130, 63, None), (257, 127, 100)])
def test_against_float64(hd, n, start, window):
    k, v, _ = _pool(start + n, hd, n)
    q = torch.randn(n, hd, generator=torch.Generator().manual_seed(hd)).to(DEV)
    got = _run(q, k, v, [list(range(k.shape[0]))], [0, n], [start], n, window)
    want = _truth(q, k.reshape(-1, hd), v.reshape(-1, hd), start, window)
    # scores to some 1e-6 and sums of weights and values to 2^-24 times a few: 1e-5 is several of each
    assert (got.double() - want).abs().max() <= 1e-5


@pytest.mark.parametrize("hd", [16, 64])
def test_a_score_of_one_product(hd):
    """Two keys weigh about the same; the first one's score is one product of two numbers with as many bits as they have."""
    k, v, q = (torch.zeros_like(x) for x in _pool(2, hd, 1))
    x = torch.tensor(0x3F80FFFF, dtype=torch.int32).view(torch.float32).item()
    root = hd ** 0.5
    q[:, 0], k[0, 0, 0, 0], k[0, 0, 1, 0] = x * 16, x * root, root * (x * x * 16).__round__() / 16
    v[0, 0, 0], v[0, 0, 1, 0] = 1.0, 3.395e38               # (a value that bfloat16 rounds to infinity)
    got = _run(q, k, v, [[0]], [0, 2], [0], 2)
    want = _truth(q, k.reshape(-1, hd), v.reshape(-1, hd), 0)
    # scores of 16.25, each off by at most 2.25 * 2^-24 of that and the scale's rounding: a weight near a half moves by a quarter of their
    # difference; the exponential, sum and quotient add some 2^-22
    bound = 0.25 * 2 * 16.25 * 3.25 * 2 ** -24 + 2 ** -22
    assert (got[:, 1:].double() - want[:, 1:]).abs().max() <= bound
    assert ((got[:, 0].double() - want[:, 0]).abs() <= 4 * bound * want[:, 0].abs()).all()


def test_numbers_that_are_none_reach_the_rows_that_see_them():
    n, hd = 150, 64
    k, v, q = _pool(n, hd, 2)
    clean = _run(q, k, v, [list(range(k.shape[0]))], [0, n], [0], n)
    k2, v2 = k.clone(), v.clone()
    flat_k, flat_v = k2.view(-1, hd), v2.view(-1, hd)
    flat_v[70, 3], flat_v[101, 9] = float("inf"), float("nan")
    flat_k[40], q2 = 0.0, q.clone()
    flat_k[40, 0] = float("-inf")
    q2[:, 0] = q[:, 0].abs() + 0.1                          # key 40 scores minus infinity with every row: it weighs nothing
    got = _run(q2, k2, v2, [list(range(k.shape[0]))], [0, n], [0], n)
    assert torch.isinf(got[70:, 3]).all() and torch.isnan(got[101:, 9]).all()
    others = [c for c in range(hd) if c not in (3, 9)]
    for r in (39, 41, 69, 70, 149):
        rows = [i for i in range(r + 1) if i != 40]
        s = (q2[r].double() * hd ** -0.5) @ flat_k[rows].double().T
        want = torch.softmax(s, 0) @ flat_v[rows].double()
        assert (got[r, others].double() - want[others]).abs().max() <= 1e-5, r
    assert torch.equal(_run(q, k2, v, [list(range(k.shape[0]))], [0, n], [0], n)[:40], clean[:40])
    assert torch.equal(_run(q, k, v2, [list(range(k.shape[0]))], [0, n], [0], n)[:70], clean[:70])


@pytest.mark.parametrize("start, n, window", [(0, 20, None), (10, 30, None), (300, 64, None), (301, 50, 90)])
def test_a_request_among_many_gives_the_same_bits(start, n, window):
    """Many short portions take a form of one group of warps per block, which walks what four groups share: the bits of a lone request."""
    hd, seqs = 64, 150
    k, v, _ = _pool(start + n, hd, 3)
    q = torch.randn(n, hd, generator=torch.Generator().manual_seed(n)).to(DEV)
    table = list(range(k.shape[0]))
    one = _run(q, k, v, [table], [0, n], [start], n, window)
    many = _run(q.repeat(seqs, 1), k, v, [table] * seqs, [n * i for i in range(seqs + 1)], [start] * seqs, n, window)
    assert torch.equal(many.view(seqs, n, hd), one.expand(seqs, n, hd))


def _portions(lens, starts, nh, seed=5, hd=64):
    """q, keys, values, tables, first rows of requests that bring ``lens`` rows; a start of -1 is a padding sequence."""
    g = torch.Generator().manual_seed(seed)
    need = [-(-(n + max(s, 0)) // 16) for n, s in zip(lens, starts)]
    at, width = [sum(need[:i]) for i in range(len(need))], max(8, max(need))
    tables = [[a + j if j < n and s >= 0 else -1 for j in range(width)] for a, n, s in zip(at, need, starts)]
    k, v = (torch.randn(sum(need), 1, 16, hd, generator=g).to(DEV) for _ in range(2))
    first = [sum(lens[:i]) for i in range(len(lens) + 1)]
    return torch.randn(sum(lens), nh * hd, generator=g).to(DEV), k, v, tables, first


@pytest.mark.parametrize("nh, lens, starts", [
    (1, [300, 1, 0, 65, 64, 2, 128, 20, 16, 16, 16, 16], [0, 3, 0, 0, 7, -1, 0, 0, 5, 0, 0, 0]),       # four groups for all tiles
    (4, [200, 2, 65, 64] + [9] * 40 + [129, 0, 3], [0, -1] + [0] * 45),                                # first tiles apart
    (13, [20] * 20 + [193, 64, 130] + [5] * 20, [300] + [0] * 42),                                     # ... with longer contexts
])
def test_the_bound_of_a_recorded_shape_gives_the_same_bits(nh, lens, starts):
    data = _portions(lens, starts, nh)
    q, first = data[0], data[4]
    want = torch.zeros_like(q)
    for s, (n, p) in enumerate(zip(lens, starts)):          # request by request
        rows = slice(first[s], first[s + 1])
        if n and p >= 0:
            want[rows] = _run(q[rows], data[1], data[2], data[3][s:s + 1], [0, n], [p], n)
    for bound in (max(lens), -(-sum(lens) // 128) * 128):
        got = _run(*data[:4], first, starts, bound)
        assert torch.equal(got, want), bound


def test_the_bound_of_a_recorded_shape_costs_little():
    """150 prompts of 16 tokens, of which a recorded step's shape tells only that no one has more than 2,432."""
    from glassbox_b200 import kernels
    q, k, v, tables, first = _portions([16] * 150, [0] * 150, 32)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    tables, first, start, status, out, times = i32(tables), i32(first), i32([0] * 150), i32([0]), torch.empty_like(q), []
    for bound in (16, 2432):
        spans = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                kernels.attention_prefill_f32(q, out, k, v, tables, first, start, bound, 32, 1, 64, 16, 0.125, None, status)
            b.record()
            torch.cuda.synchronize()
            spans.append(a.elapsed_time(b))
        times.append(min(spans))
    assert times[1] < 2 * times[0], times
