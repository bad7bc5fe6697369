"""The model's two ends: the token embedding and the head that makes logits.

Embedding: row gather times ``scale`` (reference: row fetch
``src/runtime/gpu.rs:420-431``, sqrt(hidden) factor
``src/bin/shimmy_server_gpu/server_inference.rs:603-609``).  Head: row dots
with the head matrix, then the final softcap, logits in float32 (reference:
``src/backend/bindless/sh_head_blob.wgsl:300-334``; tied to the embedding when
no separate matrix exists, ``src/runtime/gpu.rs:763-795``).
"""
from __future__ import annotations

import itertools

import torch

from .. import kernels
from ..weights.loader import WeightDecl
from ..config.base import ConfigError, PartSpec
from .base import Part, build_part, register_part
from .linear import linear


@register_part("embedding", "token_embedding")
class TokenEmbedding(Part):
    """Parameters: ``weight``, ``vocab_size``, ``hidden_size``, ``scale``; optional ``norm`` (a PartSpec of
    category ``norm``): applied to the gathered rows before they become the residual stream."""

    def __init__(self, params, ctx):
        super().__init__(params, ctx)
        self.name = self.param("weight")
        self.vocab = int(self.param("vocab_size"))
        self.hidden = int(self.param("hidden_size"))
        self.scale = float(self.param("scale"))
        self.table = None
        norm = self.params.get("norm")
        self.norm = build_part("norm", norm, ctx) if isinstance(norm, PartSpec) else None

    @property
    def graph_safe(self):
        return self.norm is None or self.norm.graph_safe

    def weight_decls(self):
        return [WeightDecl(self.name, (self.vocab, self.hidden), "table"),
                *(self.norm.weight_decls() if self.norm is not None else [])]

    def load(self, weights):
        self.table = weights[self.name].to(self.ctx.compute_dtype).contiguous()
        if self.norm is not None:
            self.norm.load(weights)

    def decode_bytes(self, lens) -> int:
        return len(lens) * self.hidden * (4 if self.ctx.compute_dtype == torch.float32 else 2)   # the rows it gathers

    def forward(self, ids):
        """ids int32 [T] -> float32 residual stream [T, H]."""
        x = torch.empty(ids.shape[0], self.hidden, dtype=torch.float32, device=ids.device)
        kernels.embed(x, self.table, ids, self.scale)
        return x if self.norm is None else self.norm.forward(x, torch.float32)


@register_part("head", "lm_head")
class LmHead(Part):
    """Parameters: ``vocab_size``, ``hidden_size``, ``softcap`` (0 = off) and
    either ``weight`` or ``tied_to`` (+ ``optional_weight`` that wins when the
    folder holds it); optional ``scale`` (default 1): the logits are multiplied by it
    (before the softcap's place: a design has one or the other)."""
    graph_safe = True


    def __init__(self, params, ctx):
        super().__init__(params, ctx)
        self.vocab = int(self.param("vocab_size"))
        self.hidden = int(self.param("hidden_size"))
        self.softcap = float(self.params.get("softcap") or 0.0)
        self.scale = float(self.params.get("scale", 1.0))
        if self.scale != 1.0 and self.softcap:
            raise ConfigError("lm_head: a scale or a softcap, not both")
        self.w = None
        self._keys = None      # the fused arg-max's key per row (zero between calls)

    def weight_decls(self):
        shape = (self.vocab, self.hidden)
        if "weight" in self.params:
            return [WeightDecl(self.params["weight"], shape, "table")]
        decls = [WeightDecl(self.param("tied_to"), shape, "table")]
        if self.params.get("optional_weight"):
            decls.append(WeightDecl(self.params["optional_weight"], shape, "table", optional=True))
        return decls

    def load(self, weights):
        name = self.params.get("weight") or self.params.get("optional_weight")
        if name is None or name not in weights:
            name = self.param("tied_to")
        self.w = weights[name].to(self.ctx.compute_dtype).contiguous()

    def decode_bytes(self, lens) -> int:
        return self.vocab * self.hidden * (4 if self.ctx.compute_dtype == torch.float32 else 2)

    def logits_flops(self, rows: int) -> int:
        return 2 * rows * self.vocab * self.hidden

    def forward(self, y):
        """y [R, H] compute dtype (after the final norm) -> float32 logits [R, V]."""
        logits = linear(y, self.w, out_dtype=torch.float32, cap=self.softcap)
        if self.scale != 1.0:
            kernels.scale_(logits, self.scale)
        return logits

    SCORE_ROWS = 32      # rows that a sequence wants at least to be scored rather than continued

    def prompt_logits(self, y, counts):
        """:meth:`forward` of a prefill step's rows, ``counts`` of them a sequence, one after the other.  In 32 bits the rows of
        a sequence that wants many go to the product for prompts, those of one that wants a few (its last) to the one for
        few rows: what a sequence asks for decides, not the step, so that its bits do not depend on its neighbours.
        256000 x 2304, one row 365 us against 630 with the prompts' product, 301 rows 7,530 against 1,840."""
        if y.dtype != torch.float32 or max(counts) < self.SCORE_ROWS:
            return self.forward(y)
        logits = torch.empty(y.shape[0], self.vocab, dtype=torch.float32, device=y.device)
        at = 0
        for many, run in itertools.groupby(counts, lambda n: n >= self.SCORE_ROWS):
            n = sum(run)
            if n:
                linear(y[at: at + n], self.w, cap=self.softcap, out=logits[at: at + n], prompt=many)
            at += n
        if self.scale != 1.0:
            kernels.scale_(logits, self.scale)
        return logits

    def forward_argmax(self, y):
        """The token of greedy decoding for every row: int32 [R], the arg-max of
        the (capped) logits over finite values, the lowest id among equals.
        On the tensor-core path the logits never go to memory (the product's
        epilogue keeps the best per row); else logits and the sampler's arg-max."""
        R = y.shape[0]
        tokens = torch.empty(R, dtype=torch.int32, device=y.device)
        if kernels.gemm_tc_supported(y, self.w, None) and self.scale > 0:      # (a positive scale moves no arg-max)
            stride = kernels.argmax_key_stride()
            if self._keys is None or self._keys.numel() < R * stride:
                self._keys = torch.zeros(max(R, 256) * stride, dtype=torch.int64, device=y.device)
            kernels.gemm_tc_argmax(tokens, y, self.w, self.softcap, self._keys)
        else:
            kernels.sample(self.forward(y), tokens, 0.0, 1.0, 1.0)
        return tokens
