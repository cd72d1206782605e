"""The one model class: an embedding, layers built from parts, an execution order, a final norm
and a head, every one of them a registered part named by the configuration. Which architecture it is
shows only in its ``ModelConfig``.

Forward order follows crates/glassbox-core/src/model.rs:207-362: embed every row, run the layers
(here: the entries of ``config.schedule``), then final norm and head on the wanted rows only.
"""
from __future__ import annotations

from typing import Dict, List

import torch

from .. import kernels
from ..config.specs import ModelConfig
from ..parts import build_block, build_part
from ..parts.block import collapse_streams
from ..parts.base import Part
from ..weights.binding import ParamSpec


def _all_parts(part: Part):
    yield part
    for sub in part.sub_parts().values():
        yield from _all_parts(sub)


def _collect(prefix: str, part: Part, out: Dict[str, ParamSpec], owners: Dict[str, tuple]) -> None:
    for name, spec in part.param_specs().items():
        out[f"{prefix}.{name}"] = spec
        owners[f"{prefix}.{name}"] = (part, name)
    for sub_name, sub in part.sub_parts().items():
        _collect(f"{prefix}.{sub_name}", sub, out, owners)


class DecoderModel:
    def __init__(self, config: ModelConfig):
        config.validate()
        self.config = config
        d = config.hidden_size
        self.embed = build_part("embedding", config.embedding, vocab_size=config.vocab_size, hidden_size=d)
        self.layers = [build_block(spec, hidden_size=d) for spec in config.layers]
        self.final_norm = build_part("norm", config.final_norm, hidden_size=d)
        self.head = build_part("head", config.head, vocab_size=config.vocab_size, hidden_size=d)
        self._owners: Dict[str, tuple] = {}
        self._specs: Dict[str, ParamSpec] = {}
        _collect("embed", self.embed, self._specs, self._owners)
        for i, layer in enumerate(self.layers):
            _collect(f"layers.{i}", layer, self._specs, self._owners)
        _collect("final_norm", self.final_norm, self._specs, self._owners)
        _collect("head", self.head, self._specs, self._owners)
        #: whether a decode step of this model may be recorded as a program for the persistent kernel: only when
        #: no part enqueues device work behind the kernel library's back
        self.program_safe = all(p.launches_through_kernels_only for p in self.parts())

    def param_specs(self) -> Dict[str, ParamSpec]:
        return dict(self._specs)

    def parts(self):
        for top in (self.embed, *self.layers, self.final_norm, self.head):
            yield from _all_parts(top)

    def recordable(self, decode_only: bool) -> bool:
        """Whether every part lets a step of this kind be replayed as a CUDA graph (see ``Part.recordable``)."""
        return all(p.recordable(decode_only) for p in self.parts())

    def bind(self, params: Dict[str, torch.Tensor]) -> None:
        grouped: Dict[int, tuple] = {}
        for path, tensor in params.items():
            part, name = self._owners[path]
            grouped.setdefault(id(part), (part, {}))[1][name] = tensor
        for part, named in grouped.values():
            part.bind(named)
        self.params = dict(params)

    def cache_layer_specs(self) -> List[object]:
        """The cache spec of each cache layer: that of the mixer of the run that writes it."""
        specs: List[object] = [None] * self.config.num_cache_layers

        def needs(layer):
            # a layer that keeps something of its own beside its mixer's cache says so itself
            if hasattr(layer, "cache_spec"):
                return layer.cache_spec()
            mixer = getattr(layer, "mixer", None)
            return mixer.cache_spec() if mixer is not None else None

        for run in self.config.schedule:
            if run.writes_cache:
                specs[run.cache] = needs(self.layers[run.layer])
        for run in self.config.schedule:
            if not run.writes_cache:
                spec = needs(self.layers[run.layer])
                if spec != specs[run.cache]:
                    raise ValueError(f"a run of layer {run.layer} reads cache layer {run.cache}, whose writer keeps "
                                     f"{specs[run.cache]!r}, but needs {spec!r}")
        return specs

    def weight_bytes(self) -> int:
        seen, total = set(), 0
        for t in self.params.values():
            if t.data_ptr() not in seen:
                seen.add(t.data_ptr())
                total += t.numel() * t.element_size()
        return total

    def forward(self, ctx) -> torch.Tensor:
        """Run the rows of ``ctx`` through the model; returns float32 logits [wanted rows, vocab]."""
        n, d = ctx.n, self.config.hidden_size
        if getattr(ctx, "weight_order", None) is not None:
            ctx.weight_order.start_step()
        x = ctx.scratch("x", (n, d), torch.float32)
        program = getattr(ctx, "program", None)
        if program is not None and not (ctx.decode_only and self.program_safe and program.takes_rows(n)):
            program = None
        if program is not None:
            kernels.program_begin(program, ctx.status)
        try:
            return self._forward(ctx, x)
        finally:
            if program is not None:
                kernels.program_end()

    def _forward(self, ctx, x) -> torch.Tensor:
        n, d = ctx.n, self.config.hidden_size
        ctx.next_norm = ctx.norm_after_layer = ctx.prepared_norm = ctx.pending_fold = ctx.residual_copy = None
        self.embed.forward(ctx, ctx.tokens, x)
        streams = self.config.residual_streams
        if streams:
            # the residual is several rows per token, all equal to the embedding's output at the start; the layers
            # work on them and the final norm reads their sum
            embedded, x = x, ctx.scratch("x_streams", (n, streams * d), torch.float32)
            kernels.streams_broadcast(embedded, x, streams)
        schedule = self.config.schedule
        for i, run in enumerate(schedule):
            # which norm reads x after this layer: the next layer's first one, if it says which that is
            entry = getattr(self.layers[schedule[i + 1].layer], "entry_norm", None) if i + 1 < len(schedule) else None
            ctx.norm_after_layer = entry() if entry is not None else None
            self.layers[run.layer].forward(ctx, x, ctx.cache_view(run.cache), run.writes_cache)
        ctx.norm_after_layer = None
        w = ctx.num_wanted
        logits = ctx.scratch("logits", (w, self.config.vocab_size), torch.float32, grow=True)
        if w:
            hs = ctx.scratch("hs", (w, d))
            if streams:
                collapse_streams(ctx, x, streams, self.final_norm, hs, rows=ctx.want_rows)
            else:
                self.final_norm.forward(ctx, x, hs, rows=ctx.want_rows)
            self.head.forward(ctx, hs, logits)
        return logits
