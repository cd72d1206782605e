"""The delta rule in chunks of tokens against the recurrence in float64, and its error beside that of the walk token by token."""
import numpy as np
import pytest
import torch

from plain import zurerax_plain as plain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(lens, H, KH, D, V, per_head, seed):
    rng = np.random.default_rng(seed)
    n, dc = sum(lens), 1 if per_head else D
    qkv = rng.standard_normal((n, 2 * KH * D + H * V))
    beta, a = 2 * rng.standard_normal((n, H)), 2 * rng.standard_normal((n, H * dc))
    # decays from next to none to more than a float32 can hold over a chunk
    dt_bias, a_log = rng.uniform(-6, 1, H * dc), rng.uniform(-3, 3, H)
    states = rng.standard_normal((len(lens), H, D, V))
    return [np.float32(x) for x in (qkv, beta, a, dt_bias, a_log, states)]


def _truth(lens, H, KH, D, V, per_head, qkv, beta, a, dt_bias, a_log, states):
    outs, after, row = [], [], 0
    for s, n in enumerate(lens):
        x = qkv[row:row + n].astype(np.float64)
        q, k = x[:, :KH * D].reshape(n, KH, D), x[:, KH * D:2 * KH * D].reshape(n, KH, D)
        q = q / np.sqrt((q * q).sum(-1, keepdims=True) + 1e-6) * D ** -0.5
        k = k / np.sqrt((k * k).sum(-1, keepdims=True) + 1e-6)
        q, k = np.repeat(q, H // KH, 1), np.repeat(k, H // KH, 1)
        z = plain.softplus(a[row:row + n].astype(np.float64) + dt_bias).reshape(n, H, -1)
        g = np.broadcast_to(np.exp(-np.exp(a_log.astype(np.float64))[None, :, None] * z), (n, H, D))
        b = plain.sigmoid(beta[row:row + n].astype(np.float64))
        v = x[:, 2 * KH * D:].reshape(n, H, V)
        S, o = states[s].astype(np.float64), np.zeros((n, H, V))
        for t in range(n):
            S = g[t][:, :, None] * S
            u = b[t][:, None] * (v[t] - np.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            o[t] = np.einsum("hdv,hd->hv", S, q[t])
        outs.append(o.reshape(n, H * V))
        after.append(S)
        row += n
    return np.concatenate(outs), np.stack(after)


def _run(chunked, lens, H, KH, D, V, per_head, qkv, beta, a, dt_bias, a_log, states, padding=False, room=None, most=None):
    """Requests in slots in reverse order; with ``padding`` a padding sequence of two rows in front. ``room``: the workspace's chunks, if fewer
    than the step needs; ``most``: the bound of a request's rows, if more than they are."""
    from glassbox_b200 import kernels
    f = lambda x: torch.tensor(x.copy(), dtype=torch.float32, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    S, lead = len(lens), [2] if padding else []
    state = torch.full((S + 1, H * D * V + 3), 3.0, device=DEV)
    state[:S, :H * D * V] = f(states[::-1]).reshape(S, -1)
    rows = lead + list(lens)
    pad = lambda x: f(np.concatenate([np.full((sum(lead), x.shape[1]), np.nan, np.float32), x])) if padding else f(x)
    first = i32([0] + list(np.cumsum(rows)))
    start = i32(([-1] if padding else []) + [0] * S)
    slots = i32(([0] if padding else []) + list(range(S - 1, -1, -1)))
    out = torch.zeros((sum(rows), H * V), device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    args = (pad(qkv), pad(beta), pad(a), f(dt_bias), f(a_log), state, out, first, start, slots)
    if chunked:
        work = torch.full((kernels.delta_chunks_needed(sum(rows), len(rows)), H * kernels.delta_chunk_floats()), float("nan"), device=DEV)
        if room is not None:
            work = torch.full((H * (room * kernels.delta_chunk_floats() + kernels.lib().gb_delta_carry_floats()),), float("nan"), device=DEV)
        kernels.channel_delta_chunks(*args, most or max(rows), H, KH, D, V, True, status, work, decay_per_head=per_head)
    else:
        kernels.channel_delta(*args, H, KH, D, V, True, status, decay_per_head=per_head)
    assert int(status) == 0 and torch.all(state[S] == 3.0) and torch.all(state[:, H * D * V:] == 3.0)
    assert torch.all(out[:sum(lead)] == 0)
    return out[sum(lead):].double().cpu().numpy(), state[:S, :H * D * V].reshape(S, H, D, V).double().cpu().numpy()[::-1]


@pytest.mark.parametrize("per_head", [False, True])
@pytest.mark.parametrize("H, KH, D, V, lens", [(2, 1, 128, 128, [31, 32, 33, 1, 96]), (1, 1, 64, 20, [100, 65]), (4, 2, 40, 9, [7, 200])])
def test_chunks_against_the_recurrence(H, KH, D, V, lens, per_head):
    data = _inputs(lens, H, KH, D, V, per_head, D + V)
    want = _truth(lens, H, KH, D, V, per_head, *data)
    for got in (_run(True, lens, H, KH, D, V, per_head, *data), _run(True, lens, H, KH, D, V, per_head, *data, padding=True)):
        for g, w in zip(got, want):
            # sums of up to 128 products of unit vectors with entries near one: 1e-5 is some 80 roundings
            np.testing.assert_allclose(g, w, atol=1e-5 * max(1.0, np.abs(w).max()), rtol=1e-5)


def test_chunks_are_as_exact_as_the_walk():
    lens, H, KH, D, V = [700], 2, 2, 128, 128
    data = _inputs(lens, H, KH, D, V, False, 5)
    want = _truth(lens, H, KH, D, V, False, *data)
    rel = lambda got: [np.linalg.norm(g - w) / np.linalg.norm(w) for g, w in zip(got, want)]
    walk, chunks = rel(_run(False, lens, H, KH, D, V, False, *data)), rel(_run(True, lens, H, KH, D, V, False, *data))
    assert all(c <= 1.2 * w + 1e-7 for c, w in zip(chunks, walk)), (chunks, walk)


def test_a_token_does_not_reach_the_ones_before_it():
    lens, H, KH, D, V = [80], 1, 1, 128, 16
    data = _inputs(lens, H, KH, D, V, False, 6)
    clean, _ = _run(True, lens, H, KH, D, V, False, *data)
    data[0][45] = np.inf
    data[1][45] = np.nan
    spoiled, _ = _run(True, lens, H, KH, D, V, False, *data)
    assert np.array_equal(clean[:45], spoiled[:45]) and not np.isfinite(spoiled[45:]).any()


def test_recorded_prompt_shapes_share_one_workspace(tmp_path_factory):
    """Ten prompt shapes through the engine, each unrecorded, while it is recorded and replayed: the same logits three times, again in
    another order once all are recorded, and one workspace for all of them, none in what a recorded shape keeps for itself."""
    import zurerax_util as zu
    from glassbox_b200.engine.engine import Engine, StepEntry
    cfg = zu.CONFIGS["even"]()
    folder = zu.write_model(str(tmp_path_factory.mktemp("shapes")), cfg, zu.random_weights(cfg, 3))
    eng = Engine(folder, "float32", cache_tokens=1200, page_size=16, max_batch_tokens=1024, max_requests=4)
    tokens = [int(t) for t in np.random.default_rng(4).integers(0, cfg["vocab"], 1024)]
    eng.add_request("r", [])
    step = lambda n: eng.step([StepEntry("r", tokens[:n], [0, n - 1])], commit=False).clone()
    lengths, first = [100 * k for k in range(1, 11)], {}
    for n in lengths:
        # (uncommitted: the request's state slot keeps what the step wrote, so it starts from zero each time)
        for _ in range(3):
            for t in eng.device_cache.state.values():
                t.zero_()
            out = step(n)
            assert torch.equal(first.setdefault(n, out), out), n
    eng.check()
    assert eng.graph_replays >= len(lengths)
    for n in reversed(lengths):
        for t in eng.device_cache.state.values():
            t.zero_()
        assert torch.equal(first[n], step(n)), n
    shared = [b for (name, _), b in eng.scratch._bufs.items() if "delta_chunks" in name]
    own = [name for g in eng._graphs.values() for (name, _) in g["ctx"]._grow._bufs if "delta_chunks" in name]
    heads = {L["mixer"]["heads"] for L in cfg["layers"] if L["type"] == "channel_delta"}
    assert len(shared) == len(heads) and not own


@pytest.mark.parametrize("H, KH, D, V, lens", [(20, 4, 36, 128, [33, 64]), (19, 19, 128, 70, [40]), (2, 1, 64, 128 + 9, [65, 3])])
def test_chunks_of_sixteen_columns_and_of_more_than_a_pass(H, KH, D, V, lens):
    """More blocks of eight columns than multiprocessors (a block then takes sixteen), the last of them past the values' end, and value
    sizes of more than one pass."""
    data = _inputs(lens, H, KH, D, V, False, H)
    for g, w in zip(_run(True, lens, H, KH, D, V, False, *data), _truth(lens, H, KH, D, V, False, *data)):
        np.testing.assert_allclose(g, w, atol=1e-5 * max(1.0, np.abs(w).max()), rtol=1e-5)       # (the bound of the test above)


def test_a_state_of_one_number_per_column():
    """What is left of a sum is one product: it is rounded, and the products of its factors' terms that are left out stay below its rounding.
    A number next to the largest float32 is taken as well."""
    from glassbox_b200 import kernels
    D = V = 64
    rng = np.random.default_rng(1)
    q = np.zeros((2, D), np.float32)
    q[:, 5], q[:, 9] = 3000.0, 4000.0               # (a length of 5,000, next to which 1e-6 is nothing; channel 9 of the state is empty)
    f = np.float32
    unit = f(3000) * (f(1) / np.sqrt(f(25e6)))
    read = float(f(3000) * (f(0.125) / np.sqrt(f(25e6))))
    states = np.zeros((1, 1, D, V), np.float32)
    states[0, 0, 5] = rng.standard_normal(V)
    states[0, 0, 5, :2] = np.array([0x3F80FFFF, 0x7F7F9000], np.uint32).view(np.float32)
    qkv = np.concatenate([q, q, np.zeros((2, V), np.float32)], 1)
    # the first token leaves the state alone (beta 0, no decay) and reads it, the second writes with beta 1
    out, after = _run(True, [2], 1, 1, D, V, True, qkv, np.float32([[-1e4], [1e4]]), np.zeros((2, 1), np.float32), np.zeros(1, np.float32),
                      np.float32([-200.0]), states)
    S, k = states[0, 0, 5].astype(np.float64), float(unit)
    # a product: its rounding and what is left out (2^-24 each), sums of three terms
    assert (np.abs(out[0] - read * S) <= 2.25 * 2 ** -24 * np.abs(read * S)).all()
    # u = -k S, then S + k u: 2.25 of 2^-24 of k S times k, as much of k u, the sum's rounding
    assert (np.abs(after[0, 0, 5] - S * (1 - k * k)) <= 2 ** -24 * (4.5 * k * k + 1) * np.abs(S)).all()


def test_a_short_prompt_is_no_slower_in_chunks():
    """One request of 96 rows, call after call: 28 us in chunks where the walk takes 37. Blocks of the calls to come must not hold the
    multiprocessors that the call at hand needs (37.8 us)."""
    from glassbox_b200 import kernels
    H, D, n = 8, 128, 96
    assert kernels.delta_chunks_chosen(n, 1, D)
    f = lambda *shape: torch.randn(*shape, device=DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    args = (f(n, 3 * H * D), f(n, H), f(n, H * D), f(H * D), f(H), torch.zeros(1, H * D * D, device=DEV), f(n, H * D), i32([0, n]), i32([0]), i32([0]))
    status, times = i32([0]), []
    work = torch.empty(kernels.delta_chunks_needed(n, 1) * H * kernels.delta_chunk_floats(), device=DEV)
    for run in (lambda: kernels.channel_delta_chunks(*args, n, H, H, D, D, True, status, work),
                lambda: kernels.channel_delta(*args, H, H, D, D, True, status)):
        run()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for _ in range(20):
                run()
        spans = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            graph.replay()
            b.record()
            torch.cuda.synchronize()
            spans.append(a.elapsed_time(b))
        times.append(min(spans))
    assert times[0] < 0.9 * times[1], times


@pytest.mark.parametrize("padding", [False, True])
@pytest.mark.parametrize("H, KH, D, V, lens", [(2, 1, 128, 128, [31, 200, 1, 33, 96]), (3, 3, 64, 150, [300]), (1, 1, 40, 24, [5] * 40 + [70, 64])])
def test_passes_and_bounds_give_the_same_bits(H, KH, D, V, lens, padding):
    """A workspace that holds a part of the chunks, down to one, and a bound of the rows that is far above them."""
    data = _inputs(lens, H, KH, D, V, False, V)
    want = _run(True, lens, H, KH, D, V, False, *data, padding=padding)
    for room, most in ((None, 4096), (1, None), (3, 1000), (7, None)):
        got = _run(True, lens, H, KH, D, V, False, *data, padding=padding, room=room, most=most)
        assert all(np.array_equal(g, w) for g, w in zip(got, want)), (room, most)


def test_the_workspace_stays_within_bounds():
    from glassbox_b200 import kernels
    for rows, slots, heads in ((2048, 8, 16), (8192, 64, 16), (1 << 17, 256, 32)):
        floats = kernels.delta_workspace_floats(kernels.delta_chunks_needed(rows, 2 * slots + 8), heads)
        assert floats * 4 <= heads * (24 << 20), (rows, slots)              # 128 chunks of 162 KB and the carried states
