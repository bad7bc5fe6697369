"""Kernels that serve the rows of prompts their own way (more values a thread, more tokens a block), against the same call in
pieces that take the other way, or against 64 bits."""
import math
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def K():
    from airframe_b200 import kernels
    return kernels


@pytest.mark.parametrize("nq, nkv, hd, dv", [(6, 2, 64, 64), (2, 1, 8, 8), (3, 3, 24, 24)])
@pytest.mark.parametrize("T, table, bias", [(64, True, False), (130, False, True)])
def test_whole_norm_of_a_prompt(K, nq, nkv, hd, dv, T, table, bias):
    """Against the same rows in steps of up to 63 tokens, whose sums of squares meet in another order (2^-20 of the factor, so
    that a result may round to the neighbouring bfloat16)."""
    g = torch.Generator().manual_seed(T + hd)
    n_q, n_k, n_v = nq * hd, nkv * hd, nkv * dv
    proj = (torch.randn(T, n_q + n_k + n_v, generator=g) * 3).to(DEV)
    wq, wk = torch.randn(n_q, generator=g).to(DEV), torch.randn(n_k, generator=g).to(DEV)
    b = torch.randn(n_q + n_k + n_v, generator=g).to(DEV) if bias else None
    inv = (10000.0 ** (-torch.arange(0, hd, 2) / hd)).float().to(DEV)
    pos = torch.arange(T, dtype=torch.int32, device=DEV)

    def run(lo, hi):
        zeros = torch.zeros(hi - lo, dtype=torch.int32, device=DEV)
        batch = SimpleNamespace(positions=pos[lo:hi], seq_of_token=zeros, slots=zeros[:1],
                                len_after=torch.full((1,), T, dtype=torch.int32, device=DEV), aux={})
        out = torch.empty(hi - lo, n_q + n_k + n_v, dtype=torch.bfloat16, device=DEV)
        K.qk_norm_rope_store(out, proj[lo:hi], batch, nq, nkv, hd, inv, hd, "half", q_weight=wq, k_weight=wk, eps=1e-5, dv=dv,
                             whole_norm=True, bias=b, table=K.rope_table(pos[lo:hi], inv) if table else None)
        return out.double()

    got, want = run(0, T), torch.cat([run(i, min(T, i + 50)) for i in range(0, T, 50)])
    assert ((got - want).abs() <= 2.0 ** -7 * want.abs() + 1e-4).all()
    assert (got == want).double().mean() > 0.99


@pytest.mark.parametrize("width, taps", [(64, 4), (516, 2), (60, 3)])
def test_convolution_of_four_channels_a_thread(K, width, taps):
    """Sequences that begin inside a group of tokens, with and without a history, against rows that cannot be read in fours."""
    g = torch.Generator().manual_seed(width)
    lens, slots = [70, 1, 2, 67, 40], [2, -1, 0, 3, 1]
    T = sum(lens)
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    batch = SimpleNamespace(seq_starts=i32(starts), slots=i32(slots), n_seqs=len(lens), n_tokens=T,
                            seq_of_token=i32([b for b, n in enumerate(lens) for _ in range(n)]))
    proj = torch.randn(T, 2 * width, generator=g).to(DEV)
    odd = torch.zeros(T, 2 * width + 1, device=DEV)
    odd[:, :2 * width] = proj
    bx, cb = torch.randn(width, generator=g).to(DEV), torch.randn(width, generator=g).to(DEV)
    cw, state = torch.randn(taps, width, generator=g).to(DEV), torch.randn(4, taps, width, generator=g).to(DEV)
    u, v = torch.empty(T, width, device=DEV), torch.empty(T, width, device=DEV)
    K.conv_rows(u, proj, width, bx, cw, cb, state, batch)
    K.conv_rows(v, odd[:, :2 * width], width, bx, cw, cb, state, batch)
    assert (u - v).abs().max() < 1e-5
    x = (proj[:, width:] + bx).double().cpu()
    for b, n in enumerate(lens):
        past = state[slots[b], 1:].double().cpu() if slots[b] >= 0 else torch.zeros(taps - 1, width, dtype=torch.float64)
        rows = torch.cat([past, x[starts[b]:starts[b] + n]])
        want = sum(cw[i].double().cpu() * rows[i:i + n] for i in range(taps)) + cb.double().cpu()
        assert (u[starts[b]:starts[b] + n].double().cpu() - want).abs().max() < 1e-5
