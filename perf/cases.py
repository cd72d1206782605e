"""The work that users of this framework have it do, as cases that can be timed and compared.

Whole steps go through ``Engine.step``; layers and parts go through the parts' own ``forward`` with a ``StepContext``, and
are recorded once as a CUDA graph and replayed, as the engine does with every step of a shape that it meets again.

A case says a batch: ``seqs`` requests that bring ``rows`` tokens in all (``rows == seqs``: single decoded tokens; else
portions of prompts of unequal length), each behind ``past`` tokens of its own that the cache already holds (``ragged``:
between half of that and all of it). Sizes are those of the SmolLM2 shapes and of the models that ``bench.py`` measures.
"""
import math
import os
import random
import tempfile

import torch

from glassbox_b200.cache.device import DeviceCache
from glassbox_b200.config import specs as S
from glassbox_b200.engine.context import Scratch, SeqInfo, StepContext, WeightOrder
from glassbox_b200.parts import build_block, build_part

PAGE = 16
EPS = 1e-5
#: SmolLM2 shapes: width, feed-forward, heads, key/value heads, rope base
LLAMA = {"135m": (576, 1536, 9, 3, 100000.0, 30), "360m": (960, 2560, 15, 5, 100000.0, 32), "1.7b": (2048, 8192, 32, 32, 130000.0, 24)}
VOCAB, HEAD_DIM, MAX_POSITION = 49152, 64, 8192
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}
F64 = torch.float64


def listed():
    return [
        # one user's generation: the smallest call there is, a chain of short kernels
        dict(name="step_decode_135m_b1", kind="step", size="135m", dtype="bfloat16", seqs=1, rows=1, past=1023, ragged=False),
        # a prompt of the benchmark's length, through the whole model
        dict(name="step_prefill_135m_2048", kind="step", size="135m", dtype="bfloat16", seqs=1, rows=2048, past=0, ragged=False),
        # a full decode batch at the benchmark's context: the cache is most of what is read
        dict(name="block_decode_1.7b_b64", kind="block", size="1.7b", dtype="bfloat16", seqs=64, rows=64, past=4095, ragged=False),
        # a service's decode batch of short and middling requests: the matrices are most of what is read
        dict(name="block_decode_1.7b_b40_short", kind="block", size="1.7b", dtype="bfloat16", seqs=40, rows=40, past=600, ragged=True),
        # prompts in the true 32-bit path (three requests whose lengths are no round numbers)
        dict(name="block_prefill_fp32_135m", kind="block", size="135m", dtype="float32", seqs=3, rows=2047, past=0, ragged=False),
        # decoding in the true 32-bit path
        dict(name="block_decode_fp32_135m_b8", kind="block", size="135m", dtype="float32", seqs=8, rows=8, past=2040, ragged=True),
        # a prompt through the delta-rule mixer of Zurerax at width 1024
        dict(name="delta_prefill_2048", kind="delta", d=1024, heads=8, rank=64, dtype="bfloat16", seqs=1, rows=2048, past=0, ragged=False),
        # a prompt through Felovik's routed SwiGLU experts (four of 16, the best two of four groups)
        dict(name="experts_prefill_2048", kind="experts", style="swiglu", d=1024, ff=1024, top=4, dtype="bfloat16", rows=2048),
        # eight decoded tokens through Lonorax's squared-ReLU experts (two of 16) and shared expert at width 2048
        dict(name="experts_decode_8", kind="experts", style="relu2", d=2048, ff=2048, top=2, dtype="bfloat16", rows=8),
        # a prompt through Babotar's talking-heads attention
        dict(name="talking_prefill_2048", kind="talking", d=1024, heads=16, kv=4, dtype="bfloat16", seqs=1, rows=2048, past=0, ragged=False),
        # ... and a decode batch of 32 requests with contexts up to 2,048
        dict(name="talking_decode_32", kind="talking", d=1024, heads=16, kv=4, dtype="bfloat16", seqs=32, rows=32, past=2047, ragged=True),
        # a later portion of a prompt through Zurerax's latent attention at width 2048
        dict(name="latent_prefill_1500", kind="latent", style="sink", d=2048, heads=32, rot=64, dtype="bfloat16", seqs=2, rows=1500, past=900,
             ragged=True),
    ]


def _between(rng, lo, hi):
    """A whole number between lo and hi, even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _batch(rng, decode, most_seqs, most_rows, most_past):
    if decode:
        n = _between(rng, 1, most_seqs)
        return dict(seqs=n, rows=n, past=_between(rng, 100, most_past), ragged=True)
    seqs = rng.randint(1, 3)
    return dict(seqs=seqs, rows=_between(rng, 70, most_rows), past=rng.choice([0, _between(rng, 20, 1000)]), ragged=True)


def draw(rng):
    kind = rng.choice(["step", "block", "block32", "delta", "experts", "talking", "latent"])
    decode = rng.random() < 0.5
    if kind == "step":
        return dict(kind="step", size="135m", dtype="bfloat16", **_batch(rng, decode, 16, 2048, 2000))
    if kind == "block":
        return dict(kind="block", size=rng.choice(sorted(LLAMA)), dtype="bfloat16", **_batch(rng, decode, 64, 2048, 4000))
    if kind == "block32":
        return dict(kind="block", size=rng.choice(["135m", "360m"]), dtype="float32", **_batch(rng, decode, 16, 1200, 2000))
    d = rng.choice([1024, 2048])
    if kind == "delta":
        return dict(kind="delta", d=d, heads=d // 128, rank=d // 16, dtype="bfloat16", **_batch(rng, decode, 64, 2048, 1000))
    if kind == "experts":
        style = rng.choice(["swiglu", "relu2"])
        return dict(kind="experts", style=style, d=d, ff=d, top=4 if style == "swiglu" else 2, dtype="bfloat16",
                    rows=_between(rng, 1, 64) if decode else _between(rng, 70, 2048 if d == 1024 else 1100))
    if kind == "talking":
        return dict(kind="talking", d=d, heads=d // 64, kv=d // 256, dtype="bfloat16",
                    **_batch(rng, decode, 32 if d == 1024 else 12, 2048 if d == 1024 else 1000, 2047))
    style = rng.choice(["sink", "query_latent"])
    return dict(kind="latent", style=style, d=d, heads=d // 64, rot=d // 32, dtype="bfloat16", **_batch(rng, decode, 64, 1800, 2000))


# ------------------------------------------------------------------------------------------------------------- the batch

def _lengths(case):
    """(tokens that each request brings, tokens that its cache holds): the same for every seed."""
    rng = random.Random(case["seqs"] * 7919 + case["rows"])
    n, seqs = case["rows"], case["seqs"]
    if n == seqs:
        rows = [1] * seqs
    else:
        cuts = sorted(rng.sample(range(1, n), seqs - 1)) if seqs > 1 else []
        rows = [b - a for a, b in zip([0] + cuts, cuts + [n])]
    past = [rng.randint(case["past"] // 2, case["past"]) if case["ragged"] else case["past"] for _ in range(seqs)]
    return rows, past


class _Batch:
    """Rows, positions and block tables of a case. The pages that this step writes into have the lowest numbers, the others
    lie scattered over the pool, as in a pool that has been in use for a while."""

    def __init__(self, case):
        self.rows, self.past = _lengths(case) if "seqs" in case else ([case["rows"]], [0])
        rng = random.Random(11)
        self.n, self.seqs = sum(self.rows), len(self.rows)
        self.decode = self.n == self.seqs
        need = [-(-(r + p) // PAGE) for r, p in zip(self.rows, self.past)]
        first_written = [p // PAGE for p in self.past]
        written = [(i, j) for i in range(self.seqs) for j in range(first_written[i], need[i])]
        older = [(i, j) for i in range(self.seqs) for j in range(first_written[i])]
        self.pages, self.written = len(written) + len(older), len(written)
        rng.shuffle(written)
        rng.shuffle(older)
        at = {key: page for page, key in enumerate(written + older)}
        self.width = max(8, 1 << max(max(need) - 1, 0).bit_length())
        self.tables = [[at[(i, j)] if j < need[i] else -1 for j in range(self.width)] for i in range(self.seqs)]
        self.positions = [p + t for r, p in zip(self.rows, self.past) for t in range(r)]
        self.row_seq = [i for i, r in enumerate(self.rows) for _ in range(r)]
        self.slots = [self.tables[i][p // PAGE] * PAGE + p % PAGE for i, p in zip(self.row_seq, self.positions)]
        self.first_row = [sum(self.rows[:i]) for i in range(self.seqs + 1)]


def _context(batch, cache, dtype):
    dev = torch.device("cuda")
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    ctx = StepContext(scratch=Scratch(batch.n + 8, dtype, dev), cache=cache, status=status, dtype=dtype)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=dev)
    ctx.n, ctx.num_wanted, ctx.num_seqs = batch.n, 0, batch.seqs
    ctx.positions, ctx.row_seq = i32(batch.positions), i32(batch.row_seq)
    ctx.seq_first_row, ctx.seq_start_pos = i32(batch.first_row), i32(batch.past)
    ctx.seq_slots = i32(list(range(batch.seqs)))
    ctx.group_slots = [i32(batch.slots) for _ in cache.group_specs]
    ctx.group_tables = [i32(batch.tables) for _ in cache.group_specs]
    ctx.seqs = [SeqInfo(request=i, slot=i, start_pos=batch.past[i], n_rows=batch.rows[i], first_row=batch.first_row[i])
                for i in range(batch.seqs)]
    ctx.max_rows_per_seq = max(batch.rows)
    ctx.max_context = min(MAX_POSITION, batch.width * PAGE) if batch.decode else max(r + p for r, p in zip(batch.rows, batch.past))
    ctx.decode_only, ctx.leading_single = batch.decode, batch.seqs if batch.decode else 0
    ctx.weight_order = WeightOrder()
    return ctx


# --------------------------------------------------------------------------------------------------------- what is built

def _rope(theta, dims, pairing="half"):
    return S.RopeSpec(theta=theta, rotary_dim=dims, max_position=MAX_POSITION, pairing=pairing)


def _build(case):
    """The part of a case."""
    kind = case["kind"]
    if kind == "block":
        d, ff, heads, kv, theta, _ = LLAMA[case["size"]]
        mixer = S.GqaAttentionSpec(num_heads=heads, num_kv_heads=kv, head_dim=HEAD_DIM, scale=HEAD_DIM ** -0.5, position=_rope(theta, HEAD_DIM))
        return build_block(S.LayerSpec(mixer=mixer, ffn=S.SwiGluSpec(ff), mixer_norm=S.RmsNormSpec(EPS), ffn_norm=S.RmsNormSpec(EPS)),
                           hidden_size=d)
    d = case["d"]
    if kind == "delta":
        return build_part("mixer", S.ChannelDeltaSpec(num_heads=case["heads"], num_kv_heads=case["heads"], key_dim=128, value_dim=128, conv_taps=4,
                                                      decay_rank=case["rank"], gate_rank=case["rank"], norm_eps=EPS), hidden_size=d)
    if kind == "talking":
        return build_part("mixer", S.TalkingAttentionSpec(num_heads=case["heads"], num_kv_heads=case["kv"], head_dim=64, value_dim=64, scale=0.125,
                                                          position=_rope(10000.0, 64), softcap=30.0), hidden_size=d)
    if kind == "latent":
        late = case["style"] == "query_latent"
        spec = S.LatentAttentionSpec(num_heads=case["heads"], nope_dim=64, rope_dim=case["rot"], value_dim=64, latent_dim=128,
                                     scale=(64 + case["rot"]) ** -0.5, position=_rope(10000.0, case["rot"], "half" if late else "interleaved"),
                                     latent_eps=EPS, sink=not late, window=1024 if late else None, q_rank=d // 2 if late else None,
                                     output_gate=late)
        return build_part("mixer", spec, hidden_size=d)
    if case["style"] == "swiglu":
        spec = S.RoutedExpertsSpec(num_experts=16, top_k=case["top"], expert_size=case["ff"], num_groups=4, keep_groups=2, correction=False,
                                   scoring="softmax", group_score="best", renormalise=1e-20, activation="swiglu")
    else:
        spec = S.RoutedExpertsSpec(num_experts=16, top_k=case["top"], expert_size=case["ff"], shared_size=case["ff"])
    return build_part("ffn", spec, hidden_size=d)


def _specs_of(part, prefix=""):
    out = {prefix + name: spec for name, spec in part.param_specs().items()}
    for name, sub in part.sub_parts().items():
        out.update(_specs_of(sub, prefix + name + "."))
    return out


def _bind(part, values, prefix=""):
    part.bind({name: values[prefix + name] for name in part.param_specs()})
    for name, sub in part.sub_parts().items():
        _bind(sub, values, prefix + name + ".")


def _values(case, part, seed):
    """The part's parameters: matrices N(0, 0.02) in the activation dtype, gains 1 + N(0, 0.01) or as the part says; the
    delta rule's decays as a trained model has them (time constants of one to a thousand tokens)."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 1000003 + 1)
    dtype, out = DTYPES[case["dtype"]], {}
    for name, spec in sorted(_specs_of(part).items()):
        normal = torch.randn(spec.shape, generator=gen, device="cuda")
        if case["kind"] == "delta" and name == "a_log":
            t = torch.log(1.0 + 15.0 * torch.rand(spec.shape, generator=gen, device="cuda"))
        elif case["kind"] == "delta" and name == "dt_bias":
            step = torch.exp(math.log(1e-3) + math.log(100.0) * torch.rand(spec.shape, generator=gen, device="cuda"))
            t = torch.log(torch.expm1(step))
        elif case["kind"] == "delta" and name == "conv":
            t = 0.3 * normal
        elif spec.init is not None:
            t = spec.init[0] + spec.init[1] * normal
        else:
            t = 1.0 + 0.01 * normal if spec.role == "gain" else 0.02 * normal
        out[name] = t if spec.role == "gain" else t.to(dtype)
    return out


def _inputs(case, seed):
    """Everything that a case's layer works on, made on the GPU: (part, parameters, batch, input rows, cached contents)."""
    part = _build(case)
    values = _values(case, part, seed)
    batch = _Batch(case)
    gen = torch.Generator(device="cuda").manual_seed(seed * 1000003 + 2)
    dtype = DTYPES[case["dtype"]]
    d = LLAMA[case["size"]][0] if case["kind"] == "block" else case["d"]
    x = torch.randn(batch.n, d, generator=gen, device="cuda")
    spec = part.mixer.cache_spec() if case["kind"] == "block" else part.cache_spec() if hasattr(part, "cache_spec") else None
    cached = {}
    if case["kind"] in ("block", "talking"):
        shape = (batch.pages, spec.num_kv_heads, PAGE, 64)
        cached = {"k": torch.randn(shape, generator=gen, device="cuda").to(dtype), "v": torch.randn(shape, generator=gen, device="cuda").to(dtype)}
    elif case["kind"] == "latent":
        cached = {"k": torch.randn((batch.pages, 1, PAGE, spec.head_dim), generator=gen, device="cuda").to(dtype)}
    elif case["kind"] == "delta":
        row = 0.1 * torch.randn((batch.seqs,) + spec.shape, generator=gen, device="cuda")
        fresh = torch.tensor([0.0 if p == 0 else 1.0 for p in batch.past], device="cuda")
        cached = {"state": row * fresh[:, None]}
    return part, values, batch, x if case["kind"] == "block" else x.to(dtype), spec, cached


class _Layer:
    """A layer or part that a program drives itself: its buffers, and its launches recorded as a CUDA graph."""

    def __init__(self, case, seed):
        self.case = case
        self.part, values, self.batch, self.x, spec, cached = _inputs(case, seed)
        _bind(self.part, values)
        dtype = DTYPES[case["dtype"]]
        self.cache = DeviceCache([spec], lambda _: self.batch.pages, PAGE, self.batch.seqs, dtype, torch.device("cuda"))
        if "k" in cached:
            self.cache.k[0][0].copy_(cached["k"])
        if "v" in cached:
            self.cache.v[0][0].copy_(cached["v"])
        self.before = cached.get("state")
        self.ctx = _context(self.batch, self.cache, dtype)
        self.out = torch.empty(self.batch.n, self.x.shape[1], dtype=torch.float32, device="cuda")
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(2):                      # (twice: the order of the weights is learned in the first pass)
                self.launch()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.launch()

    def launch(self):
        ctx, part = self.ctx, self.part
        ctx.next_norm = ctx.norm_after_layer = ctx.prepared_norm = ctx.residual_copy = None
        ctx.weight_order.start_step()
        if self.before is not None:
            self.cache.state[0].copy_(self.before)      # the requests' states as they are before the step
        if self.case["kind"] == "block":
            self.out.copy_(self.x)                      # the residual rows; the layer adds into them
            part.forward(ctx, self.out, ctx.cache_view(0), True)
            return
        ctx.overwrite_output = True
        if self.case["kind"] == "experts":
            part.forward(ctx, self.x, self.out)
        else:
            part.forward(ctx, self.x, self.out, ctx.cache_view(0), True)
        ctx.overwrite_output = False

    def run(self):
        self.graph.replay()
        outs, w = [self.out], self.batch.written
        if self.case["kind"] in ("block", "talking"):
            outs += [self.cache.k[0][0][:w], self.cache.v[0][0][:w]]
        elif self.case["kind"] == "latent":
            outs += [self.cache.k[0][0][:w]]
        elif self.case["kind"] == "delta":
            outs += [self.cache.state[0]]
        return outs


# ------------------------------------------------------------------------------------------------------- whole model steps

_FOLDERS = {}


def _model_tensors(case):
    """The model's tensors by their file names: one model for all seeds."""
    d, ff, heads, kv, _, layers = LLAMA[case["size"]]
    gen = torch.Generator(device="cuda").manual_seed(5)
    matrix = lambda *shape: (0.02 * torch.randn(shape, generator=gen, device="cuda")).to(DTYPES[case["dtype"]])
    gain = lambda: (1.0 + 0.01 * torch.randn(d, generator=gen, device="cuda")).to(DTYPES[case["dtype"]])
    out = {"model.embed_tokens.weight": matrix(VOCAB, d), "model.norm.weight": gain()}
    for i in range(layers):
        p = f"model.layers.{i}."
        out[p + "self_attn.q_proj.weight"] = matrix(heads * HEAD_DIM, d)
        out[p + "self_attn.k_proj.weight"] = matrix(kv * HEAD_DIM, d)
        out[p + "self_attn.v_proj.weight"] = matrix(kv * HEAD_DIM, d)
        out[p + "self_attn.o_proj.weight"] = matrix(d, heads * HEAD_DIM)
        out[p + "mlp.gate_proj.weight"], out[p + "mlp.up_proj.weight"] = matrix(ff, d), matrix(ff, d)
        out[p + "mlp.down_proj.weight"] = matrix(d, ff)
        out[p + "input_layernorm.weight"], out[p + "post_attention_layernorm.weight"] = gain(), gain()
    return out


def _model_folder(case):
    import json
    from glassbox_b200.models.llama import make_llama_raw_config
    from glassbox_b200.weights import write_safetensors
    key = (case["size"], case["dtype"])
    if key not in _FOLDERS:
        d, ff, heads, kv, theta, layers = LLAMA[case["size"]]
        raw = make_llama_raw_config(hidden_size=d, intermediate_size=ff, num_hidden_layers=layers, num_attention_heads=heads,
                                    num_key_value_heads=kv, vocab_size=VOCAB, rope_theta=theta, rms_norm_eps=EPS, tie_word_embeddings=True,
                                    max_position_embeddings=MAX_POSITION)
        folder = tempfile.TemporaryDirectory(prefix="perf_model_")
        with open(os.path.join(folder.name, "config.json"), "w") as f:
            json.dump(raw, f)
        write_safetensors(os.path.join(folder.name, "model.safetensors"), {k: v.cpu() for k, v in _model_tensors(case).items()})
        _FOLDERS[key] = folder
    return _FOLDERS[key].name


def _tokens(case, seed):
    rows, past = _lengths(case)
    rng = random.Random(seed)
    return [[rng.randrange(VOCAB) for _ in range(r + p)] for r, p in zip(rows, past)], past


class _Step:
    """A loaded model whose requests have come as far as the case says. The step is not committed: every pass is the same
    step again."""

    def __init__(self, case, seed):
        from glassbox_b200.engine.engine import Engine, StepEntry
        tokens, past = _tokens(case, seed)
        pages = sum(-(-len(t) // PAGE) + 1 for t in tokens)
        self.engine = Engine(_model_folder(case), case["dtype"], num_pages=pages, page_size=PAGE, max_batch_tokens=2048, max_requests=16)
        self.entries = []
        for i, (t, p) in enumerate(zip(tokens, past)):
            self.engine.add_request(i)
            if p:
                self.engine.step([StepEntry(i, t[:p], [])])
            self.entries.append(StepEntry(i, t[p:], [len(t) - p - 1]))

    def run(self):
        return self.engine.step(self.entries, commit=False)


def prepare(case, seed):
    return _Step(case, seed) if case["kind"] == "step" else _Layer(case, seed)


def run(state):
    return state.run()


# ------------------------------------------------------------------------------------------------ what cannot be done without

def _seen(batch, window=None):
    """(keys that are read from the cache in all, sum over the rows of the keys each sees)."""
    keys = sum(min(p, window) if window else p for p in batch.past)
    pairs = 0
    for r, p in zip(batch.rows, batch.past):
        pairs += sum(min(p + t + 1, window) if window else p + t + 1 for t in range(r))
    return keys, pairs


def work(case):
    b = _Batch(case)
    n, e = b.n, 2 if case["dtype"] == "bfloat16" else 4
    if case["kind"] in ("step", "block"):
        d, ff, heads, kv, _, layers = LLAMA[case["size"]]
        weights = d * HEAD_DIM * (2 * heads + 2 * kv) + 3 * d * ff
        keys, pairs = _seen(b)
        bytes_ = e * (weights + 2 * kv * HEAD_DIM * (keys + n))
        flops = 2 * n * weights + 4 * pairs * heads * HEAD_DIM
        if case["kind"] == "block":
            return {"bytes": bytes_ + 8 * n * d, "flops": flops}
        return {"bytes": layers * bytes_ + e * VOCAB * d + 4 * VOCAB * b.seqs, "flops": layers * flops + 2 * VOCAB * d * b.seqs}
    d = case["d"]
    if case["kind"] == "experts":
        ff, top, gated = case["ff"], case["top"], case["style"] == "swiglu"
        per = (3 if gated else 2) * d * ff
        used = 16 * (1 - (1 - top / 16) ** n)
        shared = 0 if gated else 2 * d * ff
        return {"bytes": int(e * (used * per + shared) + n * d * (e + 4) + 64 * d), "flops": 2 * n * (top * per + shared + 16 * d)}
    if case["kind"] == "delta":
        heads, rank, inner = case["heads"], case["rank"], case["heads"] * 128
        weights = d * (3 * inner + 2 * rank + heads) + 2 * inner * rank + d * inner
        state = 4 * b.seqs * (heads * 128 * 128 + 9 * inner)
        return {"bytes": e * weights + 2 * state + n * d * (e + 4), "flops": 2 * n * weights + 7 * n * heads * 128 * 128}
    heads = case["heads"]
    if case["kind"] == "talking":
        kv = case["kv"]
        weights = d * 64 * (2 * heads + 2 * kv)
        keys, pairs = _seen(b)
        # scores once; mixing before the values or behind them: the cheaper is a product of heads x kv value heads
        return {"bytes": e * weights + e * 128 * kv * (keys + n) + n * d * (e + 4), "flops": 2 * n * weights + 2 * pairs * heads * 64 * (1 + kv)}
    rot, late = case["rot"], case["style"] == "query_latent"
    q_in = d // 2 if late else d
    weights = d * (128 + rot) + q_in * heads * (64 + rot) + (d * d // 2 + d * heads * 64 if late else 0) + 2 * heads * 64 * 128 + d * heads * 64
    keys, pairs = _seen(b, 1024 if late else None)
    return {"bytes": e * weights + e * (128 + rot) * (keys + n) + n * d * (e + 4), "flops": 2 * n * weights + 2 * pairs * heads * (256 + rot)}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 4e-6, "max": 1e-4}
    # bfloat16 operands, activations and caches: one layer rounds a few times; through a whole model it adds up
    return {"rel": 0.03, "max": 0.3} if case["kind"] == "step" else {"rel": 0.015, "max": 0.3}


# ----------------------------------------------------------------------------------------------- the same in plain 64-bit torch

def _rms(x, gain, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * gain


def _silu(x):
    return x * torch.sigmoid(x)


def _angles(positions, theta, dims):
    """The angle of a rotation is defined as a 32-bit product of the position and a frequency rounded to 32 bits."""
    freq = theta ** (-torch.arange(0, dims, 2, dtype=F64, device="cuda") / dims)
    return (torch.tensor(positions, dtype=torch.float32, device="cuda")[:, None] * freq.float()).to(F64)


def _turn(x, positions, theta, dims, pairing="half"):
    """x [rows, heads, D]: the first ``dims`` channels of every head are rotated."""
    ang = _angles(positions, theta, dims)[:, None, :]
    c, s = torch.cos(ang), torch.sin(ang)
    out = x.clone()
    if pairing == "half":
        a, b = x[..., :dims // 2], x[..., dims // 2:dims]
        out[..., :dims // 2], out[..., dims // 2:dims] = a * c - b * s, b * c + a * s
    else:
        a, b = x[..., 0:dims:2], x[..., 1:dims:2]
        out[..., 0:dims:2], out[..., 1:dims:2] = a * c - b * s, b * c + a * s
    return out


def _stored(pool, batch, rows):
    """The pool [pages, heads, PAGE, D] in 64 bits with this step's rows [n, heads, D] in their slots."""
    pool = pool.to(F64)
    slots = torch.tensor(batch.slots, device="cuda")
    pool[slots // PAGE, :, slots % PAGE] = rows
    return pool


def _of_request(pool, batch, i):
    """[context, heads, D] of request i."""
    pages = [p for p in batch.tables[i] if p >= 0]
    flat = pool[torch.tensor(pages, device="cuda")].transpose(1, 2).flatten(0, 1)
    return flat[:batch.past[i] + batch.rows[i]]


def _attention(q, keys, values, past, scale, weigh):
    """q [rows, H, D], keys [context, G, D], values [context, G, V] -> weights by ``weigh(scores, visible)`` [H, rows, context]
    and the values' heads repeated."""
    rows, heads = q.shape[:2]
    keys = keys.repeat_interleave(heads // keys.shape[1], dim=1)
    out = []
    pos = past + torch.arange(rows, device="cuda")[:, None]
    at = torch.arange(keys.shape[0], device="cuda")[None, :]
    for h in range(heads):
        out.append(weigh(q[:, h] @ keys[:, h].T * scale, pos, at, h))
    return torch.stack(out)


def _softmax(s, pos, at, window=None, extra=None):
    seen = at <= pos if window is None else (at <= pos) & (at > pos - window)
    s = s.masked_fill(~seen, -math.inf)
    if extra is None:
        return torch.softmax(s, -1)
    return torch.softmax(torch.cat([s, extra.expand(s.shape[0], 1)], -1), -1)[:, :-1]


def _llama_layer(x, w, batch, pools, shape, theta):
    """One pre-norm layer on rows x [n, d]; ``pools``: (keys, values) before the step, or None where there are none."""
    d, ff, heads, kv = shape
    n, D = x.shape[0], HEAD_DIM
    qkv = _rms(x, w["norm1"]) @ w["wqkv"].T
    q = _turn(qkv[:, :heads * D].view(n, heads, D), batch.positions, theta, D)
    k = _turn(qkv[:, heads * D:(heads + kv) * D].reshape(n, kv, D), batch.positions, theta, D)
    v = qkv[:, (heads + kv) * D:].reshape(n, kv, D)
    keys, values = (_stored(p, batch, r) for p, r in zip(pools, (k, v))) if pools else (k, v)
    att = []
    for i in range(batch.seqs):
        a, b = batch.first_row[i], batch.first_row[i] + batch.rows[i]
        ki, vi = (_of_request(keys, batch, i), _of_request(values, batch, i)) if pools else (k[a:b], v[a:b])
        p = _attention(q[a:b], ki, vi, batch.past[i], D ** -0.5, lambda s, pos, at, h: _softmax(s, pos, at))
        att.append(torch.einsum("hrc,chd->rhd", p, vi.repeat_interleave(heads // kv, dim=1)).reshape(b - a, heads * D))
    x = x + torch.cat(att) @ w["wo"].T
    gu = _rms(x, w["norm2"]) @ w["w_gate_up"].T
    return x + (_silu(gu[:, :ff]) * gu[:, ff:]) @ w["w_down"].T, keys, values


def _exact_step(case, seed):
    """Every request's whole sequence from its start, without a cache."""
    d, ff, heads, kv, theta, layers = LLAMA[case["size"]]
    t = {k: v.to(F64) for k, v in _model_tensors(case).items()}
    logits = []
    for tokens in _tokens(case, seed)[0]:
        batch = _Batch(dict(seqs=1, rows=len(tokens), past=0, ragged=False))
        x = t["model.embed_tokens.weight"][torch.tensor(tokens, device="cuda")]
        for i in range(layers):
            p = f"model.layers.{i}."
            w = {"norm1": t[p + "input_layernorm.weight"], "norm2": t[p + "post_attention_layernorm.weight"],
                 "wqkv": torch.cat([t[p + f"self_attn.{c}_proj.weight"] for c in "qkv"]), "wo": t[p + "self_attn.o_proj.weight"],
                 "w_gate_up": torch.cat([t[p + "mlp.gate_proj.weight"], t[p + "mlp.up_proj.weight"]]), "w_down": t[p + "mlp.down_proj.weight"]}
            x = _llama_layer(x, w, batch, None, (d, ff, heads, kv), theta)[0]
        logits.append(_rms(x[-1:], t["model.norm.weight"]) @ t["model.embed_tokens.weight"].T)
    return torch.cat(logits)


def _exact_block(case, w, batch, x, cached):
    d, ff, heads, kv, theta, _ = LLAMA[case["size"]]
    w = {"norm1": w["mixer_norm.weight"], "norm2": w["ffn_norm.weight"], "wqkv": w["mixer.wqkv"], "wo": w["mixer.wo"],
         "w_gate_up": w["ffn.w_gate_up"], "w_down": w["ffn.w_down"]}
    out, keys, values = _llama_layer(x, w, batch, (cached["k"], cached["v"]), (d, ff, heads, kv), theta)
    return [out, keys[:batch.written], values[:batch.written]]


def _exact_delta(case, w, batch, x, cached):
    H, D, rank = case["heads"], 128, case["rank"]
    inner, taps = H * D, 4
    proj = x @ w["w_in"].T
    conv_in, rest = proj[:, :3 * inner], proj[:, 3 * inner:]
    a = rest[:, :rank] @ w["w_a2"].T + w["dt_bias"]
    gate = torch.sigmoid(rest[:, rank:2 * rank] @ w["w_g2"].T)
    beta = torch.sigmoid(rest[:, 2 * rank:])
    g = torch.exp(-torch.exp(w["a_log"])[:, None] * torch.nn.functional.softplus(a).view(-1, H, D))
    state = cached["state"].to(F64)
    outs, states = [], []
    for i in range(batch.seqs):
        lo, hi = batch.first_row[i], batch.first_row[i + 1]
        Sm = state[i, :H * D * D].view(H, D, D).clone()
        seq = torch.cat([state[i, H * D * D:].view(taps - 1, 3 * inner), conv_in[lo:hi]])
        y = _silu(sum(w["conv"][:, j] * seq[j:j + hi - lo] for j in range(taps)))
        q, k, v = (y[:, j * inner:(j + 1) * inner].view(-1, H, D) for j in range(3))
        q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * D ** -0.5
        k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        o = torch.empty(hi - lo, H, D, dtype=F64, device="cuda")
        for t in range(hi - lo):
            Sm = Sm * g[lo + t, :, :, None]
            u = beta[lo + t, :, None] * (v[t] - torch.einsum("hd,hdv->hv", k[t], Sm))
            Sm = Sm + k[t, :, :, None] * u[:, None, :]
            o[t] = torch.einsum("hd,hdv->hv", q[t], Sm)
        outs.append(o)
        states.append(torch.cat([Sm.flatten(), seq[-(taps - 1):].flatten()]))
    o = _rms(torch.cat(outs), w["out_norm"]) * gate.view(-1, H, D)
    return [o.reshape(-1, inner) @ w["wo"].T, torch.stack(states)]


def _exact_experts(case, w, batch, x, cached):
    E, ff, top, d = 16, case["ff"], case["top"], case["d"]
    logits = x @ w["router"].T
    rows = torch.arange(x.shape[0], device="cuda")[:, None]
    if case["style"] == "swiglu":
        score = torch.softmax(logits, -1)
        best = score.view(-1, 4, 4).amax(-1)
        keep = torch.zeros_like(best).scatter(1, best.topk(2, dim=-1).indices, 1.0).repeat_interleave(4, dim=1) > 0
        chosen = score.masked_fill(~keep, -1.0).topk(top, dim=-1).indices
        weight = score[rows, chosen]
        weight = weight / (weight.sum(-1, keepdim=True) + 1e-20)
        # an expert's gate matrix, then its up matrix
        up = w["w_up"].view(E, 2, ff, d)
    else:
        score = torch.sigmoid(logits)
        chosen = (score + w["correction"]).topk(top, dim=-1).indices
        weight = score[rows, chosen]
        up = w["w_up"].view(E, ff, d)
    down = w["w_down"].view(E, d, ff)
    out = torch.zeros_like(x)
    for e in range(E):
        r, c = (chosen == e).nonzero(as_tuple=True)
        h = x[r]
        act = _silu(h @ up[e, 0].T) * (h @ up[e, 1].T) if case["style"] == "swiglu" else torch.relu(h @ up[e].T) ** 2
        out.index_add_(0, r, (act @ down[e].T) * weight[r, c][:, None])
    if case["style"] != "swiglu":
        out += torch.sigmoid(x @ w["shared_gate"].T) * (torch.relu(x @ w["shared_up"].T) ** 2 @ w["shared_down"].T)
    return [out]


def _exact_talking(case, w, batch, x, cached):
    H, G, n = case["heads"], case["kv"], x.shape[0]
    proj = x @ w["w_in"].T + w["b_in"]
    q = _turn(proj[:, :H * 64].reshape(n, H, 64), batch.positions, 10000.0, 64)
    k = _turn(proj[:, H * 64:(H + G) * 64].reshape(n, G, 64), batch.positions, 10000.0, 64)
    v = proj[:, (H + G) * 64:].reshape(n, G, 64)
    keys, values = _stored(cached["k"], batch, k), _stored(cached["v"], batch, v)
    att, none = [], torch.zeros(1, 1, dtype=F64, device="cuda")
    for i in range(batch.seqs):
        a, b = batch.first_row[i], batch.first_row[i] + batch.rows[i]
        vi = _of_request(values, batch, i)
        p = _attention(q[a:b], _of_request(keys, batch, i), vi, batch.past[i], 0.125,
                       lambda s, pos, at, h: _softmax(30.0 * torch.tanh(s / 30.0), pos, at, extra=none))
        p = torch.einsum("hg,grc->hrc", w["talk"], p)
        att.append(torch.einsum("hrc,chd->rhd", p, vi.repeat_interleave(H // G, dim=1)).reshape(b - a, H * 64))
    return [torch.cat(att) @ w["wo"].T, keys[:batch.written], values[:batch.written]]


def _exact_latent(case, w, batch, x, cached):
    H, r, c, n, d = case["heads"], case["rot"], 128, x.shape[0], case["d"]
    late = case["style"] == "query_latent"
    first = d // 2 if late else H * (64 + r)
    proj = x @ w["w_in"].T
    q = _rms(proj[:, :first], w["q_norm"]) @ w["w_uq"].T if late else proj[:, :first]
    q = q.reshape(n, H, 64 + r)
    pairing = "half" if late else "interleaved"
    q_rot = _turn(q[..., 64:], batch.positions, 10000.0, r, pairing)
    latent = _rms(proj[:, first:first + c], w["latent_norm"])
    key_rot = _turn(proj[:, None, first + c:first + c + r], batch.positions, 10000.0, r, pairing)[:, 0]
    pool = _stored(cached["k"], batch, torch.cat([latent, key_rot], -1)[:, None])
    uk, uv = w["w_uk"].view(H, 64, c), w["w_uv"].view(H, 64, c)
    full = torch.cat([torch.einsum("nhd,hdc->nhc", q[..., :64], uk), q_rot], -1)
    att = []
    for i in range(batch.seqs):
        a, b = batch.first_row[i], batch.first_row[i] + batch.rows[i]
        rows = _of_request(pool, batch, i)
        p = _attention(full[a:b], rows, None, batch.past[i], (64 + r) ** -0.5,
                       lambda s, pos, at, h: _softmax(s, pos, at, 1024 if late else None, None if late else w["sink"][h].view(1, 1)))
        att.append(torch.einsum("hrc,cl,hvl->rhv", p, rows[:, 0, :c], uv).reshape(b - a, H * 64))
    att = torch.cat(att)
    if late:
        att = att * torch.sigmoid(proj[:, first + c + r:])
    return [att @ w["wo"].T, pool[:batch.written]]


def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "step":
            return _exact_step(case, seed)
        _, values, batch, x, _, cached = _inputs(case, seed)
        w = {name: t.to(F64) for name, t in values.items()}
        plain = {"block": _exact_block, "delta": _exact_delta, "experts": _exact_experts, "talking": _exact_talking, "latent": _exact_latent}
        return plain[case["kind"]](case, w, batch, x.to(F64), cached)
