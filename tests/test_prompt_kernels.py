"""Kernels of prompt steps at the edges of their tiles, against plain PyTorch in 64 bits."""
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


@pytest.mark.parametrize("N, Kd", [(200, 72), (384, 320), (2304, 1032)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_gemm_tensor_cores_token_tiles(K, N, Kd, out_dtype):
    """Every width of a token tile, on one SM with one accumulator or two and on a pair: the same bits, whatever the tile, as
    the chosen one, and the product in 64 bits within the roundings of its output."""
    gen = torch.Generator().manual_seed(N)
    w = (torch.randn(N, Kd, generator=gen) * 0.05).to(DEV, torch.bfloat16)
    for M in (65, 257, 700):
        x = torch.randn(M, Kd, generator=gen).to(DEV, torch.bfloat16)
        want = x.double() @ w.double().T
        first = torch.full((M, N), float("nan"), device=DEV, dtype=out_dtype)
        K.gemm_tc(first, x, w)
        assert ((first.double() - want).abs() <= (2e-6 if out_dtype == torch.float32 else 2.0 ** -8) * want.abs() + 2e-5).all()
        for n_acc in (1, 2, 4):
            for tile in range(32, 257, 32 if n_acc == 4 else 16):
                out = torch.full((M, N), float("nan"), device=DEV, dtype=out_dtype)
                K.gemm_tc(out, x, w, n_acc=n_acc, token_tile=tile)
                assert torch.equal(out, first), (M, n_acc, tile)


@pytest.mark.parametrize("act", ["gelu_tanh", "silu"])
@pytest.mark.parametrize("inter, Kd", [(200, 72), (448, 320)])
def test_gated_products_of_any_token_tile(K, act, inter, Kd):
    """Every width of a token tile under the gated epilogue, whose halves meet by shuffles: the same bits whatever the tile, and the
    product in 64 bits within the roundings of its output and the activation's."""
    gen = torch.Generator().manual_seed(inter)
    w = (torch.randn(2 * inter, Kd, generator=gen) * 0.05).to(torch.bfloat16)
    wi = K.interleave_gate_up(w[:inter].to(DEV), w[inter:].to(DEV))
    f = {"gelu_tanh": lambda z: torch.nn.functional.gelu(z, approximate="tanh"), "silu": torch.nn.functional.silu}[act]
    for M in (65, 257, 700):
        x = torch.randn(M, Kd, generator=gen).to(torch.bfloat16)
        want = f(x.double() @ w[:inter].double().T) * (x.double() @ w[inter:].double().T)
        x = x.to(DEV)
        first = torch.full((M, wi.shape[0] // 2), float("nan"), device=DEV, dtype=torch.bfloat16)
        K.gemm_tc(first, x, wi, gated=True, activation=act)
        err = (first[:, :inter].double().cpu() - want).abs()
        assert (err <= 2.0 ** -8 * want.abs() + 1e-5).all(), float(err.max())
        for n_acc in (1, 2, 4):
            for tile in range(32, 257, 32 if n_acc == 4 else 16):
                out = torch.full_like(first, float("nan"))
                K.gemm_tc(out, x, wi, gated=True, activation=act, n_acc=n_acc, token_tile=tile)
                assert torch.equal(out[:, :inter], first[:, :inter]), (M, n_acc, tile)
    K.check_device_errors(DEV)


@pytest.mark.parametrize("M, splits", [(129, 3), (300, 2), (520, 4)])
def test_split_products_of_a_prompt(K, M, splits):
    """Partial sums of prompts' rows: equal token tiles, as many as of 256, against tiles of 256 and the sums in 64 bits."""
    N, Kd = 300, 1032
    gen = torch.Generator().manual_seed(M)
    x, w = torch.randn(M, Kd, generator=gen).to(torch.bfloat16), (torch.randn(N, Kd, generator=gen) * 0.05).to(torch.bfloat16)
    out, twin = (torch.full((splits, M, N), float("nan"), device=DEV) for _ in range(2))
    K.gemm_tc(out, x.to(DEV), w.to(DEV), splits=splits)
    K.gemm_tc(twin, x.to(DEV), w.to(DEV), splits=splits, n_acc=1, token_tile=256)
    assert torch.equal(out, twin)
    want = x.double() @ w.double().T
    assert ((out.double().sum(0).cpu() - want).abs() <= 2e-6 * want.abs() + 2e-5).all()
    K.check_device_errors(DEV)


def _attend(q, k, v, scale, cap, seen, slopes, sinks, gate):
    """One sequence in 64 bits: q [n, H, d], k [n, G, d], v [n, G, dv]."""
    n, H = q.shape[:2]
    i, j = torch.arange(n)[:, None], torch.arange(n)[None, :]
    out = []
    for h in range(H):
        g = h * k.shape[1] // H
        s = (q[:, h].double() @ k[:, g].double().T) * scale
        s = cap * torch.tanh(s / cap) if cap else s
        s = (s + (slopes[h].double() * (j - i) if slopes is not None else 0.0)).masked_fill(~seen, -math.inf)
        if sinks is not None:
            s = torch.cat([s, sinks[h].double().expand(n, 1)], 1)
        o = s.softmax(1)[:, :n] @ v[:, g].double()
        out.append(o * torch.sigmoid(gate[:, h].double())[:, None] if gate is not None else o)
    return torch.stack(out, 1)


@pytest.mark.parametrize("hd, dv, nq, nkv", [(64, 64, 2, 1), (40, 24, 4, 2), (128, 128, 3, 3), (96, 256, 2, 1), (130, 30, 2, 2), (256, 256, 4, 2),
                                             (255, 129, 2, 1)])
@pytest.mark.parametrize("mask, window, keep, extras", [("window", 0, 0, False), ("window", 33, 5, True), ("window", 70, 0, True), ("chunk", 50, 70, True)])
def test_attention_prefill_f32(K, hd, dv, nq, nkv, mask, window, keep, extras):
    """Sequences around the tiles of 16 queries and 64 keys; sizes that fill no tile or no 16-byte piece; windows, chunks and first
    tokens that stay visible; slopes, sinks, gates and a cap.  Bound: sums of up to 300 32-bit terms of size one."""
    gen = torch.Generator().manual_seed(hd + dv + window)
    lens, least = [64, 1, 65, 15, 129, 80, 300], 16
    T = sum(lens)
    q, k, v = (torch.randn(T, n, generator=gen) for n in (nq * hd, nkv * hd, nkv * dv))
    slopes, sinks, gate = (torch.rand(nq, generator=gen), torch.randn(nq, generator=gen), torch.randn(T, nq, generator=gen)) if extras else (None,) * 3
    cap = 20.0 if extras else 0.0
    starts = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32)
    out = torch.full((T, nq * dv), 7.0, device=DEV)
    to = [None if t is None else t.to(DEV) for t in (slopes, sinks, gate)]
    K.attn_prefill_f32(out, q.to(DEV), k.to(DEV), v.to(DEV), starts.to(DEV), len(lens), max(lens), nq, nkv, hd, hd ** -0.5, cap, window, to[0], dv,
                       mask, to[1], to[2], keep, least=least)
    at = 0
    for n in lens:
        s, i, j = slice(at, at + n), torch.arange(n)[:, None], torch.arange(n)[None, :]
        at += n
        if n < least:                       # (another kernel's: nothing is written)
            assert bool((out[s] == 7.0).all())
            continue
        seen = j <= i
        if window:
            seen = seen & (((i // window == j // window) if mask == "chunk" else (i - j < window)) | (j < keep))
        want = _attend(q[s].view(n, nq, hd), k[s].view(n, nkv, hd), v[s].view(n, nkv, dv), hd ** -0.5, cap, seen, slopes, sinks,
                       gate[s] if extras else None)
        err = (out[s].double().cpu().view(n, nq, dv) - want).abs().max()
        assert err < 4e-6, (n, float(err))


def test_attention_prefill_f32_of_a_step(K):
    """A step's long and short sequences by two kernels: each sequence has the bits that it has alone, and what is not finite
    reaches only the tokens that see it."""
    gen = torch.Generator().manual_seed(5)
    lens, nq, nkv, hd = [63, 200, 3, 64, 90], 4, 2, 64
    T = sum(lens)
    q, k, v = (torch.randn(T, n * hd, generator=gen).to(DEV) for n in (nq, nkv, nkv))

    def run(q, k, v, lens):
        starts = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
        batch = SimpleNamespace(seq_lens=lens, n_seqs=len(lens), max_len=max(lens), seq_starts=starts,
                                positions=torch.cat([torch.arange(n) for n in lens]).to(DEV, torch.int32),
                                seq_of_token=torch.cat([torch.full((n,), i) for i, n in enumerate(lens)]).to(DEV, torch.int32))
        out = torch.full((sum(lens), nq * hd), 7.0, device=DEV)
        K.attn_prefill(out, q, k, v, batch, nq, nkv, hd, hd ** -0.5, 0.0, 0)
        return out

    together, at = run(q, k, v, lens), 0
    for n in lens:
        assert torch.equal(together[at:at + n], run(q[at:at + n], k[at:at + n], v[at:at + n], [n]))
        at += n
    for bad, t in ((float("nan"), k), (float("inf"), v), (float("nan"), v)):
        u = t.clone()
        u[63 + 70] = bad                                   # (token 70 of the second sequence)
        out = run(q, u if t is k else k, u if t is v else v, lens)
        assert torch.equal(out[:63 + 70], together[:63 + 70]) and torch.equal(out[263:], together[263:])
        assert not out[63 + 70:263].isfinite().any()


def test_attention_prefill_f32_of_many_sequences(K):
    """More sequences than a warp's lanes, long ones between ones that another kernel takes: a block finds its own, and each long
    sequence has the bits that it has alone."""
    gen = torch.Generator().manual_seed(6)
    lens, nq, nkv, hd, least = [3] * 31 + [200] + [63] * 40 + [64, 1, 300] + [80] * 20 + [5], 3, 1, 64, 64
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
    T = starts[-1]
    q, k, v = (torch.randn(T, n * hd, generator=gen).to(DEV) for n in (nq, nkv, nkv))

    def run(lo, hi, own):
        out = torch.full((hi - lo, nq * hd), 7.0, device=DEV)
        at = torch.tensor([sum(own[:i]) for i in range(len(own) + 1)], dtype=torch.int32, device=DEV)
        K.attn_prefill_f32(out, q[lo:hi], k[lo:hi], v[lo:hi], at, len(own), max(own), nq, nkv, hd, hd ** -0.5, 0.0, 0, least=least)
        return out

    out = run(0, T, lens)
    for lo, n in zip(starts, lens):
        if n < least:
            assert bool((out[lo:lo + n] == 7.0).all())
        else:
            assert torch.equal(out[lo:lo + n], run(lo, lo + n, [n]))
