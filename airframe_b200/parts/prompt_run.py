"""The layers of a prompt step as one call into the kernel library.

A short prompt's time is the host's: a launch and what stands around it take some 17 us from Python, the kernel behind
it less.  Where all runs of a model are of one kind (``sandwich`` blocks of attention with a rotary encoding, a gated
feed-forward and RMS norms, in bfloat16, of sizes the tensor cores take), their launches are made in the library instead
(``csrc/prompt_layers.cu``): the same kernels with the same arguments, in the same order (a change of what ``SandwichBlock``,
``Attention`` or ``GatedMlp`` launch is made there too).  A prompt of 37 tokens through 26
layers: 3.68 ms part by part, 1.79 ms so (the kernels' own time).  Anything else runs part by part."""
from __future__ import annotations

import struct

import torch

from .. import kernels
from .attention import Attention
from .block import SandwichBlock
from .mlp import GatedMlp
from .norm import RmsNorm
from .rope import Rope

_RUN = struct.Struct("<13Q4q6d")
_STEP = struct.Struct("<13Q14qd")


def _matrix(w, rows: int, cols: int) -> bool:
    """Whether a weight is what its product is told (the bindings, which look at every tensor, are passed by)."""
    return w.dtype == torch.bfloat16 and tuple(w.shape) == (rows, cols) and w.is_contiguous() and w.data_ptr() % 16 == 0 and w.is_cuda


def _vector(w, n: int) -> bool:
    return w.dtype == torch.float32 and w.numel() == n and w.is_contiguous() and w.data_ptr() % 16 == 0 and w.is_cuda


def _alike(block):
    """What the runs of a step have to have in common, or None where a block is not of the kind."""
    m, f = block.mixer, block.feed_forward
    if type(block) is not SandwichBlock or type(m) is not Attention or type(f) is not GatedMlp or type(m.position) is not Rope:
        return None
    norms = [block.norms[r] for r in SandwichBlock.roles]
    rope = m.position
    fits = (block.ctx.compute_dtype == torch.bfloat16 and not (m.packs or m.pad or m.rope_epilogue or m.sinks is not None)
            and m.mask == "window" and f.interleaved and f.w_gu.shape[0] == 2 * f.inter
            and not (m.params.get("wide_output") or f.params.get("wide_output"))
            and all(type(n) is RmsNorm and n.offset == norms[0].offset for n in norms)
            and rope.magnitude == 1.0 and 0 < rope.rotary_dim <= m.hd and m.hidden % 8 == 0 and f.inter % 8 == 0
            and _matrix(m.w_qkv, (m.nq + 2 * m.nkv) * m.hd, m.hidden) and _matrix(m.w_o, m.hidden, m.nq * m.hd)
            and _matrix(f.w_gu, 2 * f.inter, m.hidden) and _matrix(f.w_down, m.hidden, f.inter)
            and all(_vector(n.w, m.hidden) for n in norms) and _vector(rope.inv_freq, rope.rotary_dim // 2)
            and kernels.attn_prefill_tc_supported(m.hd))
    if not fits:
        return None
    return (m.hidden, m.nq, m.nkv, m.hd, f.inter, f.activation, rope.rotary_dim, rope.pairing, norms[0].offset)


def supported(model) -> bool:
    """Whether a loaded model's prompts can run this way."""
    if model.streams != 1 or not model.blocks or any(e.enter is not None for e in model.spec.schedule):
        return False
    kinds = {_alike(model.blocks[e.layer]) for e in model.spec.schedule}
    return len(kinds) == 1 and None not in kinds


def run(model, x, batch, cache) -> bool:
    """All runs of the schedule on the stream ``x`` (float32 [T, H], updated in place).  False: nothing was done (a run's view
    of the cache is not a plain one, or ``kernels.GEMM_TC_PER_SM`` asks for products of another shape)."""
    views = cache.views
    if any(not v.writes or v.keep_step_kv for v in views) or batch.n_seqs > 65535 or kernels.GEMM_TC_PER_SM:
        return False
    blocks = [model.blocks[e.layer] for e in model.spec.schedule]
    first = blocks[0]
    m, f = first.mixer, first.feed_forward
    T, H, W, N = x.shape[0], m.hidden, m.w_qkv.shape[0], m.nq * m.hd
    products = ((W, H), (H, N), (H, f.inter))
    splits = [kernels.gemm_tc_splits(T, rows, K) for rows, K in products]
    h = first.norms["pre_mixer"].forward(x, torch.bfloat16)
    qkv, ctx, mid, a = (torch.empty(T, n, dtype=torch.bfloat16, device=x.device) for n in (W, N, f.inter, H))
    room = max((s * T * rows for (rows, _), s in zip(products, splits) if s > 1), default=0)
    parts = torch.empty(room, dtype=torch.float32, device=x.device) if room else None
    # (the cosines and sines of a step come from its table from so many rows on, as in Rope.encode_and_store)
    tables = T >= kernels.ROPE_TABLE_ROWS and splits[0] == 1
    runs = bytearray()
    for i, (b, view) in enumerate(zip(blocks, views)):
        m, f, n, kv, rope = b.mixer, b.feed_forward, b.norms, view.kv, b.mixer.position
        nxt = blocks[i + 1].norms["pre_mixer"] if i + 1 < len(blocks) else None
        table = rope.rotary_table(batch, m.hd) if tables and rope.rotates_half_pairs(m.hd) else None
        post, pre, last = n["post_mixer"], n["pre_feed_forward"], n["post_feed_forward"]
        runs += _RUN.pack(
            m.w_qkv.data_ptr(), m.w_o.data_ptr(), f.w_gu.data_ptr(), f.w_down.data_ptr(), post.w.data_ptr(), pre.w.data_ptr(),
            last.w.data_ptr(), nxt.w.data_ptr() if nxt is not None else 0, rope.inv_freq.data_ptr(),
            table.data_ptr() if table is not None else 0, kv.k.data_ptr(), kv.v.data_ptr(), kv.page_table.data_ptr(),
            kv.page_table.shape[1], kv.ring_rows, m.window or 0, kernels.kv_keep(kv),
            post.eps, pre.eps, last.eps, nxt.eps if nxt is not None else 0.0, m.scale, m.softcap)
    m, f = first.mixer, first.feed_forward
    step = _STEP.pack(
        *(t.data_ptr() for t in (x, h, qkv, ctx, mid, a)), parts.data_ptr() if room else 0,
        *(t.data_ptr() for t in (batch.positions, batch.seq_of_token, batch.slots, batch.len_after, batch.seq_starts)),
        kernels.error_word(x.device).data_ptr(), T, H, m.nq, m.nkv, m.hd, m.position.rotary_dim,
        kernels.PAIRINGS[m.position.pairing], f.inter, kernels.ACTIVATIONS[f.activation], batch.n_seqs, batch.max_len,
        *splits, first.norms["pre_mixer"].offset)
    kernels.prompt_layers(step, bytes(runs), len(blocks))
    return True
