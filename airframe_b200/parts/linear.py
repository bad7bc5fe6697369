"""y = x W^T for a weight [out, in]: picks the matrix-product kernel.

float32: the plain CUDA-core kernel (true 32-bit), and in a prompt's step, for all
but small weights, the tensor cores with operands in three parts that hold all their
bits; the kind of step and the weight decide, never the number of rows, so that a
row's bits do not depend on the rows beside it.  bfloat16: the tensor-core
kernels where they take the sizes, the plain kernel (bfloat16 operands, 32-bit
accumulators) otherwise.
"""
from __future__ import annotations

import torch

from .. import kernels


def of_prompt(batch) -> bool:
    """Whether a part's rows are a prefill step's (a part called without a batch: no)."""
    return getattr(batch, "is_prefill", False)


def linear(x, w, out_dtype=None, cap: float = 0.0, out=None, prompt: bool = False):
    """x [M, K] (dense rows), w [N, K] -> [M, N] in ``out_dtype`` (x's by default).
    ``cap`` > 0 applies the softcap cap * tanh(y / cap) to the result.  ``prompt``: the
    rows are a prefill step's."""
    M = x.shape[0]
    N = w.shape[0]
    if out is None:
        out = torch.empty(M, N, dtype=out_dtype or x.dtype, device=x.device)
    if kernels.gemm_tc_supported(x, w, out):
        kernels.gemm_tc(out, x, w, cap, checked=True)
    elif prompt and kernels.gemm_f32_tc_supported(x, w, out):
        kernels.gemm_f32_tc(out, x, w, cap)
    else:
        kernels.gemm_plain(out, x, w, cap)
    return out


class PartialSums:
    """The result of a product as float32 split-K partial sums [S, M, N]; the
    consumer (a norm's ``add_normed``, the rotary kernel) adds them in order."""

    def __init__(self, parts):
        self.parts = parts

    @property
    def shape(self):
        return self.parts.shape[1:]


class WeightedSum:
    """A mixer's result as a sum that is still to be taken: ``terms`` is a list
    of (tensor or :class:`PartialSums`, scale).  The consumer (a block's residual
    sum) adds scale * term for every term in 32 bits, so that no term is rounded
    to the compute dtype on its way into the residual stream."""

    def __init__(self, terms):
        self.terms = list(terms)

    @property
    def shape(self):
        return self.terms[0][0].shape


def as_terms(a) -> list:
    """(tensor, scale) pairs of a part's result, whatever form it came in:
    a tensor [T, H], float32 partial sums [S, T, H], or a weighted sum of those."""
    if isinstance(a, WeightedSum):
        return [(t.parts if isinstance(t, PartialSums) else t, float(s)) for t, s in a.terms]
    if isinstance(a, PartialSums):
        return [(a.parts, 1.0)]
    return [(a, 1.0)]


def linear_split(x, w, wide: bool = False, prompt: bool = False):
    """x w^T for few rows and a long K: split-K partial sums when that fills
    the GPU better, else the plain result.  Returns a tensor or PartialSums.
    ``wide``: the plain result is float32 whatever the compute dtype (a
    sublayer's output on its way into the 32-bit residual stream is then not
    rounded to 16 bits in between).  ``prompt``: as in :func:`linear`."""
    M, K = x.shape
    N = w.shape[0]
    out_dtype = torch.float32 if wide else x.dtype
    if kernels.gemm_tc_supported(x, w, None):
        splits = kernels.gemm_tc_splits(M, N, K)
        if splits > 1:
            parts = torch.empty(splits, M, N, dtype=torch.float32, device=x.device)
            kernels.gemm_tc(parts, x, w, splits=splits, checked=True)
            return PartialSums(parts)
        out = torch.empty(M, N, dtype=out_dtype, device=x.device)
        kernels.gemm_tc(out, x, w, checked=True)
        return out
    return linear(x, w, out_dtype=out_dtype, prompt=prompt)


def gated_linear(x, w_gu, inter: int, activation: str, interleaved: bool, prompt: bool = False):
    """act(x w_gate^T) * (x w_up^T).  ``interleaved``: w_gu is in the gated
    tensor-core layout (``kernels.interleave_gate_up``) and one kernel with the
    activation in its epilogue does it all; else w_gu = [gate rows; up rows],
    a product and the activation kernel.  ``prompt``: as in :func:`linear`."""
    M = x.shape[0]
    out = torch.empty(M, inter, dtype=x.dtype, device=x.device)
    if interleaved:
        full = out if w_gu.shape[0] // 2 == inter else torch.empty(M, w_gu.shape[0] // 2, dtype=x.dtype, device=x.device)
        kernels.gemm_tc(full, x, w_gu, gated=True, activation=activation)
        return full if full is out else full[:, :inter].contiguous()
    gu = linear(x, w_gu, prompt=prompt)
    kernels.gated_act(out, gu, activation)
    return out
