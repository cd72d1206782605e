"""The host-side plans that pick kernel variants from a step's shape (pure Python: no GPU, no library)."""
import pytest

from glassbox_b200 import kernels


@pytest.mark.parametrize("nkv", [1, 3, 5, 32])
@pytest.mark.parametrize("context", [16, 100, 512, 1024, 4096, 8192, 65536])
def test_decode_attention_plan_keeps_its_promises(nkv, context):
    """For every batch size: at least one split; the eight-warp variant never asks for more blocks than SMs (a second
    block of eight warps does not fit beside the first) nor for more partial results per head than its merge holds at
    once; 16 keys per iteration only at head size 64; the plan depends on the shape alone."""
    for rows in list(range(1, 70)) + [128, 500]:
        splits, block_keys, warps = kernels.decode_mma_plan(rows, nkv, 64, context)
        assert splits >= 1 and warps in (4, 8) and block_keys in (0, 16)
        assert (splits, block_keys, warps) == kernels.decode_mma_plan(rows, nkv, 64, context)
        if warps == 4 and block_keys == 16:
            assert splits <= 4                                           # clusters of 5 and 7 place badly
        if warps == 8:
            assert rows * nkv * splits <= 148
            assert splits * warps <= 64
            if block_keys == 16:
                assert context <= 1024 * splits
        assert splits == 1 or splits * 128 <= max(context, 512) * 2      # no split without keys of its own
        # other head sizes have no 16-key or eight-warp variant
        s2, b2, w2 = kernels.decode_mma_plan(rows, nkv, 128, context)
        assert b2 == 0 and w2 == 4 and s2 >= 1


def test_decode_attention_plan_examples():
    """The shapes the benchmark runs (SmolLM2-135M: 3 kv heads, context 4096)."""
    assert kernels.decode_mma_plan(1, 3, 64, 4096) == (8, 16, 8)
    assert kernels.decode_mma_plan(8, 3, 64, 4096) == (6, 16, 8)
    assert kernels.decode_mma_plan(16, 3, 64, 4096) == (3, 0, 8)        # 1,365 keys a block: 32 keys per iteration
    assert kernels.decode_mma_plan(64, 3, 64, 4096) == (2, 16, 4)
    # large batches: the split count whose waves of resident blocks end soonest
    assert kernels.decode_mma_plan(8, 32, 64, 4096) == (3, 16, 4)       # 256 pairs: 2 splits would leave a short second wave
    assert kernels.decode_mma_plan(48, 3, 64, 4096) == (2, 16, 4)       # 144 pairs: 3 splits no longer fit one wave
    assert kernels.decode_mma_plan(13, 32, 64, 4096) == (1, 16, 4)      # 416 pairs fit one wave by themselves
    assert kernels.decode_mma_plan(64, 32, 64, 4096) == (1, 16, 4)
    assert kernels.decode_mma_plan(64, 5, 64, 4096) == (1, 16, 4)


class _DeltaStep:
    """As much of a step context as the delta rule's dispatch reads; the arithmetic is replaced by a record of the route."""

    def __init__(self, scratch, rows, seqs, longest):
        import torch
        from glassbox_b200.engine.context import Scratch, StepContext
        cpu = torch.device("cpu")
        self.own = Scratch(scratch.max_rows, torch.float32, cpu)             # what a recorded context keeps for itself
        self.ctx = StepContext(scratch=scratch, cache=None, status=torch.zeros(1, dtype=torch.int32), dtype=torch.float32, grow_scratch=self.own)
        self.ctx.max_rows_per_seq, self.ctx.seq_start_pos = longest, torch.zeros(seqs, dtype=torch.int32)
        self.qkv, self.state = torch.zeros(rows, 1), torch.zeros(4, 8)

    def route(self, monkeypatch, heads=2, dk=128):
        from glassbox_b200.parts import delta_rule
        taken = []
        monkeypatch.setattr(kernels, "channel_delta", lambda *a, **k: taken.append(("walk", None)))
        monkeypatch.setattr(kernels, "channel_delta_chunks", lambda *a, **k: taken.append(("chunks", a[-1])))
        monkeypatch.setattr(kernels, "delta_chunk_floats", lambda: 6)
        monkeypatch.setattr(kernels, "delta_chunks_needed", lambda n, s: n // 32 + s)
        delta_rule.run_delta(self.ctx, self.qkv, None, None, {"dt_bias": None, "a_log": None}, self.state, None, heads, heads, dk, 128, True)
        return taken[0]


@pytest.mark.parametrize("rows, seqs, longest, dk, want", [
    (64, 1, 128, 128, "walk"),           # a portion of up to 64 rows as a recorded step sees it: 64 rows, a tile of 128
    (128, 1, 128, 128, "chunks"), (2048, 1, 2048, 64, "chunks"), (2048, 1, 2048, 256, "walk"),
    (448, 64, 448, 128, "walk"),         # 36 portions of up to 19 rows, recorded with 64 sequences
    (1024, 64, 1024, 128, "chunks"), (168, 41, 128, 128, "walk"), (2088, 41, 2048, 128, "chunks"),
])
def test_the_delta_rule_is_chosen_by_what_a_recorded_step_knows(monkeypatch, rows, seqs, longest, dk, want):
    import torch
    from glassbox_b200.engine.context import Scratch
    step = _DeltaStep(Scratch(4096, torch.float32, torch.device("cpu")), rows, seqs, longest)
    assert step.route(monkeypatch, dk=dk)[0] == want


def test_recorded_steps_share_the_delta_rules_workspace(monkeypatch):
    """Steps of ten shapes, each with buffers of its own for what depends on the shape, work in one buffer, large enough for the
    largest step of the engine."""
    import torch
    from glassbox_b200.engine.context import Scratch
    shared = Scratch(2048, torch.float32, torch.device("cpu"))
    seen = set()
    for rows, seqs in [(128, 1), (256, 2), (512, 4), (1024, 8), (1536, 8), (2048, 12), (2048, 1), (640, 4), (320, 2), (192, 1)]:
        step = _DeltaStep(shared, rows, seqs, rows)
        how, work = step.route(monkeypatch)
        assert how == "chunks" and work.numel() >= (rows // 32 + seqs) * 2 * 6
        assert not step.own._bufs
        seen.add((work.data_ptr(), work.numel()))
    assert len(seen) == 1 and seen.pop()[1] == (2048 // 32 + 2 * 4 + 8) * 2 * 6


@pytest.mark.parametrize("rows, seqs, heads, context, want", [
    (8, 1, 32, 64, True), (1500, 2, 32, 4096, True), (64, 16, 4, 128, True),      # one round of blocks
    (16 * 64, 16, 32, 128, False), (16 * 96, 16, 32, 128, True),                   # fresh portions in several rounds
    (16 * 32, 16, 32, 2048, False), (16 * 48, 16, 32, 2048, True),                 # behind cached tokens
])
def test_latent_portions_take_the_flash_kernel_where_it_is_the_faster(rows, seqs, heads, context, want):
    assert kernels.latent_flash_chosen(rows, seqs, heads, context) is want


def test_single_tokens_of_a_latent_step_take_the_decode_kernel(monkeypatch):
    """A step of 40 leading single tokens and two portions: rows 0 to 39 to the decode kernel, the portions to the flash kernel, with
    the tables and positions that belong to them."""
    import torch
    from types import SimpleNamespace
    from glassbox_b200.parts.latent_attention import LatentAttention
    taken = []
    monkeypatch.setattr(kernels, "latent_attention_mma_supported", lambda *a: True)
    monkeypatch.setattr(kernels, "latent_flash_supported", lambda *a: True)
    monkeypatch.setattr(kernels, "latent_decode_splits", lambda *a: 1)
    monkeypatch.setattr(kernels, "latent_attention_mma", lambda q, out, cache, tables, first, start, *a, **k: taken.append(
        ("decode" if k.get("decode") else "tiles", q.shape[0], tables.shape[0], first.tolist(), start.tolist())))
    monkeypatch.setattr(kernels, "latent_flash", lambda q, out, cache, tables, first, start, *a, **k: taken.append(
        ("flash", q.shape[0], tables.shape[0], first.tolist(), start.tolist())))
    lead, portions = 40, [300, 500]
    first = list(range(lead + 1)) + [lead + 300, lead + 800]
    start = list(range(100, 100 + lead)) + [7, 9]
    ctx = SimpleNamespace(decode_only=False, leading_single=lead, max_context=2048, max_rows_per_seq=500, status=None,
                          seq_first_row=torch.tensor(first), seq_start_pos=torch.tensor(start), positions=torch.zeros(840))
    part = SimpleNamespace(H=32, c=128, r=64, params={}, spec=SimpleNamespace(scale=1.0, window=None))
    part._attend_decode = lambda *a: LatentAttention._attend_decode(part, *a)
    cache = SimpleNamespace(k=None, page_size=16, block_tables=torch.zeros(42, 8))
    q = torch.zeros(840, 1, dtype=torch.bfloat16)
    LatentAttention.attend(part, ctx, q, q, cache)
    assert taken == [("decode", 40, 40, first[:41], start[:40]), ("flash", 840, 2, first[40:], start[40:])]
    taken.clear()
    ctx.max_context, ctx.seq_first_row = 128, torch.tensor(list(range(lead + 1)) + [lead + 20, lead + 40])      # short portions, many heads
    part.H = 128
    LatentAttention.attend(part, ctx, q[:80], q[:80], cache)
    assert [t[:3] for t in taken] == [("tiles", 80, 42)]


def test_the_few_rows_projection_leaves_unaligned_tables_and_caches_to_the_others(monkeypatch):
    """A rotary table or a cache that does not start on 16 bytes is no error: another kernel takes the step, as ever."""
    import torch
    monkeypatch.setattr(kernels, "gemm_few_supported", lambda *a, **k: True)
    q = torch.zeros(16, 64, dtype=torch.bfloat16)
    cache, table = torch.zeros(1 + 8 * 64, dtype=torch.bfloat16), torch.zeros(1 + 4 * 32 * 2)
    even, odd = cache[:512], cache[1:]
    assert kernels.gemm_few_qkv_supported(q, q, 64, q, even, even, table[:256])
    assert kernels.gemm_few_qkv_supported(q, q, 64, q, even, even, None)
    assert not kernels.gemm_few_qkv_supported(q, q, 64, q, odd, even, None)
    assert not kernels.gemm_few_qkv_supported(q, q, 64, q, even, odd, None)
    assert not kernels.gemm_few_qkv_supported(q, q, 64, q, even, even, table[1:])


def test_talking_decode_shares_are_asked_for_one_kernel():
    """The tensor-core kernel and the one by FMA cut a row's keys by rules of their own: which of them a call takes has to be said."""
    with pytest.raises(TypeError):
        kernels.talking_decode_shares(32, 16, 4, 64, 4, 2048)
