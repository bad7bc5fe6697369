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


def rope_step(K, qkv, pos, nq, nkv, hd, table):
    """Rows turned in place and stored: (rows, key pages, value pages) of one sequence at positions 0 ..."""
    T, pages = qkv.shape[0], (int(pos.max()) + 64) // 64
    inv = (10000.0 ** (-torch.arange(0, hd, 2) / hd)).float().to(DEV)
    zeros = torch.zeros(T, dtype=torch.int32, device=DEV)
    slots, after = zeros[:1], torch.full((1,), int(pos.max()) + 1, dtype=torch.int32, device=DEV)
    kc, vc = (torch.full((pages, nkv, K.PAGE, hd), 7.0, dtype=qkv.dtype, device=DEV) for _ in range(2))
    table = K.rope_table(pos, inv) if table else None
    K.rope_cache_write(qkv, pos, inv, nq, nkv, hd, hd, "half", seq_of_token=zeros, slots=slots, len_after=after, kcache=kc, vcache=vc,
                       page_table=torch.arange(pages, dtype=torch.int32, device=DEV)[None], ring_rows=pages * 64, table=table)
    return qkv, kc, vc


@pytest.mark.parametrize("dtype, T, piece", [(torch.bfloat16, 1001, 500), (torch.float32, 400, 1), (torch.float32, 400, 149), (torch.float32, 7, 3)])
@pytest.mark.parametrize("nq, nkv, hd", [(4, 2, 64), (3, 1, 8), (8, 4, 256)])
def test_rotated_rows(K, dtype, T, piece, nq, nkv, hd):
    """Bits do not depend on how many rows a step has nor on where the angles come from; 64 bits beside them."""
    g = torch.Generator().manual_seed(T + hd)
    rows = torch.randn(T, (nq + 2 * nkv) * hd, generator=g).to(dtype)
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    first = rope_step(K, rows.to(DEV), pos, nq, nkv, hd, True)
    for a, b in zip(first, rope_step(K, rows.to(DEV), pos, nq, nkv, hd, False)):
        assert torch.equal(a, b)
    parts = [rope_step(K, rows[i:i + piece].to(DEV), pos[i:i + piece], nq, nkv, hd, True)[0] for i in range(0, T, piece)]
    assert torch.equal(first[0], torch.cat(parts))
    x = rows[:, :(nq + nkv) * hd].double().view(T, nq + nkv, hd)
    a = torch.arange(T).double()[:, None, None] * (10000.0 ** (-torch.arange(0, hd, 2) / hd)).float().double()
    lo, hi = x[..., :hd // 2], x[..., hd // 2:]
    want = torch.cat([lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()], -1)
    got = first[0].double().cpu()
    # (an angle of up to T, rounded to 32 bits; a result of up to 6 rounded to its type)
    tol = 6 * (T * 2.0 ** -24 + (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -22))
    assert (got[:, :(nq + nkv) * hd].view(T, nq + nkv, hd) - want).abs().max() < tol
    assert torch.equal(got[:, (nq + nkv) * hd:], rows[:, (nq + nkv) * hd:].double())
    k, v = got[:, nq * hd:(nq + nkv) * hd].view(T, nkv, hd), got[:, (nq + nkv) * hd:].view(T, nkv, hd)
    for cache, rows_of in ((first[1], k), (first[2], v)):
        stored = cache.transpose(1, 2).reshape(-1, nkv, hd).double().cpu()
        assert torch.equal(stored[:T], rows_of) and bool((stored[T:] == 7.0).all())


@pytest.mark.parametrize("M, inter", [(1, 4), (3, 1024), (2, 4100), (2 ** 17, 4), (512, 1024), (510, 1028), (128, 4100)])
def test_gated_activation_of_32_bit_rows(K, M, inter):
    """Four values a thread at the edges of a block's 1,024; the same bits as a row that cannot be read in fours."""
    gu = torch.randn(M, 2 * inter, generator=torch.Generator().manual_seed(inter)) * 2
    out = torch.empty(M, inter, device=DEV)
    off = torch.empty(M * inter + 1, device=DEV)[1:].view(M, inter)     # (one value off the 16-byte pieces)
    for act, f in (("gelu_tanh", lambda g: torch.nn.functional.gelu(g, approximate="tanh")), ("silu", torch.nn.functional.silu)):
        K.gated_act(out, gu.to(DEV), act)
        K.gated_act(off, gu.to(DEV), act)
        assert torch.equal(out, off)
        want = f(gu[:, :inter].double()) * gu[:, inter:].double()
        assert (out.double().cpu() - want).abs().max() < 2e-6 * want.abs().max()


@pytest.mark.parametrize("nq, nkv, hd, dv", [(6, 2, 64, 64), (2, 1, 8, 8), (3, 3, 24, 24), (4, 2, 16, 12), (18, 6, 128, 128)])
@pytest.mark.parametrize("T, table, bias", [(64, True, False), (130, False, True)])
def test_whole_norm_of_a_prompt(K, nq, nkv, hd, dv, T, table, bias):
    """The same bits, packed and in the cache, as the rows have in steps of up to 63 tokens."""
    g = torch.Generator().manual_seed(T + hd)
    n_q, n_k, n_v = nq * hd, nkv * hd, nkv * dv
    proj = (torch.randn(T, n_q + n_k + n_v, generator=g) * 3).to(DEV)
    wq, wk = torch.randn(n_q, generator=g).to(DEV), torch.randn(n_k, generator=g).to(DEV)
    b = torch.randn(n_q + n_k + n_v, generator=g).to(DEV) if bias else None
    inv = (10000.0 ** (-torch.arange(0, hd, 2) / hd)).float().to(DEV)
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    pages = (T + 63) // 64 + 1

    def run(cuts):
        kv = SimpleNamespace(k=torch.full((pages, nkv, K.PAGE, hd), 7.0, dtype=torch.bfloat16, device=DEV),
                             v=torch.full((pages, nkv, K.PAGE, dv), 7.0, dtype=torch.bfloat16, device=DEV),
                             page_table=torch.arange(pages, dtype=torch.int32, device=DEV).flip(0)[None].contiguous(), ring_rows=pages * 64)
        rows = []
        for lo, hi in cuts:
            zeros = torch.zeros(hi - lo, dtype=torch.int32, device=DEV)
            batch = SimpleNamespace(positions=pos[lo:hi], seq_of_token=zeros, slots=zeros[:1],
                                    len_after=torch.full((1,), T, dtype=torch.int32, device=DEV), aux={})
            rows.append(torch.empty(hi - lo, n_q + n_k + n_v, dtype=torch.bfloat16, device=DEV))
            K.qk_norm_rope_store(rows[-1], proj[lo:hi], batch, nq, nkv, hd, inv, hd, "half", q_weight=wq, k_weight=wk, eps=1e-5, dv=dv,
                                 whole_norm=True, bias=b, table=K.rope_table(pos[lo:hi], inv) if table else None, kv=kv)
        return torch.cat(rows), kv.k, kv.v

    got, want = run([(0, T)]), run([(i, min(T, i + 50)) for i in range(0, T, 50)])
    for x, y in zip(got, want):
        assert torch.equal(x, y)
    for cache, rows in ((got[1], got[0][:, n_q:n_q + n_k].view(T, nkv, hd)), (got[2], got[0][:, n_q + n_k:].view(T, nkv, dv))):
        stored = cache.flip(0).transpose(1, 2).reshape(pages * 64, nkv, -1)
        assert torch.equal(stored[:T], rows) and bool((stored[T:] == 7.0).all())


@pytest.mark.parametrize("T", [3, 70])
@pytest.mark.parametrize("nq, nkv, hd", [(32, 8, 256), (48, 24, 128), (7, 1, 1360)])
def test_whole_norm_of_the_widest_rows(K, nq, nkv, hd, T):
    """Rows of 48 KB and a little less, which a block's shared memory holds or does not, against 64 bits."""
    g = torch.Generator().manual_seed(nq)
    n = (nq + 2 * nkv) * hd
    proj, wq, wk = torch.randn(T, n, generator=g), torch.randn(nq * hd, generator=g), torch.randn(nkv * hd, generator=g)
    pos = torch.zeros(T, dtype=torch.int32, device=DEV)                   # (position 0: the rotation leaves its rows alone)
    batch = SimpleNamespace(positions=pos, seq_of_token=pos, slots=pos[:1], len_after=pos[:1] + 1, aux={})
    out = torch.empty(T, n, dtype=torch.bfloat16, device=DEV)
    inv = torch.ones(hd // 2, device=DEV)
    K.qk_norm_rope_store(out, proj.to(DEV), batch, nq, nkv, hd, inv, hd, "half", q_weight=wq.to(DEV), k_weight=wk.to(DEV), eps=1e-5, whole_norm=True)
    q, k, v = proj.double().split([nq * hd, nkv * hd, nkv * hd], 1)
    norm = lambda x, w: x / (x.square().mean(1, keepdim=True) + 1e-5).sqrt() * w.double()
    want = torch.cat([norm(q, wq), norm(k, wk), v], 1)
    # (half a unit of a bfloat16 and the sum's roundings)
    assert ((out.double().cpu() - want).abs() <= (2.0 ** -8 + 2.0 ** -18) * want.abs() + 1e-30).all()


@pytest.mark.parametrize("M, H", [(300, 1028), (300, 2308), (5, 4100), (300, 4100), (3, 8188)])
def test_norms_of_widths_one_group_over_a_blocks(K, M, H):
    """Two groups of four values a thread and an odd number of groups: the last one belongs to a row as the others do."""
    g = torch.Generator().manual_seed(M + H)
    x, a, b = (torch.randn(M, H, generator=g) for _ in range(3))
    w1, w2 = torch.randn(H, generator=g), torch.randn(H, generator=g)
    x[:, -4:] *= 40.0
    a[:, -4:] *= 40.0
    norm = lambda t, w: t / (t.square().mean(1, keepdim=True) + 1e-5).sqrt() * w.double()
    x64, a64, b64 = x.double(), a.double(), b.double()

    def check(y, xd, want_x, want_y):
        # (a sum of H squares in 32 bits, a few roundings)
        assert (y.double().cpu() - want_y).abs().max() < 1e-5 * want_y.abs().max()
        assert xd is None or (xd.double().cpu() - want_x).abs().max() < 1e-5 * want_x.abs().max()

    dev = lambda t: t.to(DEV)
    y = torch.full((M, H), float("nan"), device=DEV)
    K.rmsnorm(y, dev(x), dev(w1), 1e-5, 0.0)
    check(y, None, None, norm(x64, w1))
    y, xd = torch.full((M, H), float("nan"), device=DEV), dev(x)
    K.add_rmsnorm(xd, dev(a), dev(w1), 1e-5, 0.0, y=y, w_next=dev(w2), eps_next=1e-5)
    want = x64 + norm(a64, w1)
    check(y, xd, want, norm(want, w2))
    y, xd = torch.full((M, H), float("nan"), device=DEV), dev(x)
    K.add_scaled_rmsnorm(xd, [(dev(a), 0.5), (dev(b), 2.0)], y=y, w_next=dev(w2), eps=1e-5)
    want = x64 + 0.5 * a64 + 2.0 * b64
    check(y, xd, want, norm(want, w2))
    y, xd = torch.full((M, H), float("nan"), device=DEV), dev(x)
    K.add_normed_terms(xd, [(dev(a), 0.5), (dev(b), 2.0)], dev(w1), 1e-5, y=y, w_next=dev(w2), eps_next=1e-5)
    want = x64 + norm(0.5 * a64 + 2.0 * b64, w1)
    check(y, xd, want, norm(want, w2))


@pytest.mark.parametrize("width, taps", [(1024, 4), (2052, 2), (2044, 3), (64, 4)])
def test_convolution_of_four_channels_a_thread(K, width, taps):
    """Sequences that begin inside a group of tokens, with and without a history, against rows that cannot be read in fours."""
    g = torch.Generator().manual_seed(width)
    lens, slots = [270, 1, 2, 267, 140], [2, -1, 0, 3, 1]                 # (170 groups of four tokens: from 512 channels on as many blocks as SMs)
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
    assert torch.equal(u, v)
    x = (proj[:, width:] + bx).double().cpu()
    for b, n in enumerate(lens):
        past = state[slots[b], 1:].double().cpu() if slots[b] >= 0 else torch.zeros(taps - 1, width, dtype=torch.float64)
        rows = torch.cat([past, x[starts[b]:starts[b] + n]])
        want = sum(cw[i].double().cpu() * rows[i:i + n] for i in range(taps)) + cb.double().cpu()
        assert (u[starts[b]:starts[b] + n].double().cpu() - want).abs().max() < 1e-5


def test_rotated_rows_behind_two_to_the_31st_cache_row(K):
    """A cache of more rows than 32 bits with a sign count: heads of 16 elements, the last pages of 64 GB.  (Keys and values share the
    memory, a page apart; nothing but the rows' own places is touched.)"""
    rows, nkv, hd, T = 2 ** 31 + 4 * 64, 1, 16, 64
    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("80 GB of free device memory")
    memory = torch.empty(rows // 64 + 1, nkv, 64, hd, dtype=torch.bfloat16, device=DEV)
    last = rows // 64 - 2
    memory[last - 1:] = 7.0
    qkv = torch.randn(T, 4 * hd).to(torch.bfloat16).to(DEV)                # 2 query heads, 1 of keys, 1 of values
    pos, zeros = torch.arange(T, dtype=torch.int32, device=DEV), torch.zeros(T, dtype=torch.int32, device=DEV)
    K.rope_cache_write(qkv, pos, torch.ones(hd // 2, device=DEV), 2, nkv, hd, hd, "half", seq_of_token=zeros, slots=zeros[:1],
                       len_after=zeros[:1] + T, kcache=memory[:-1], vcache=memory[1:], ring_rows=0,
                       page_table=torch.tensor([[last]], dtype=torch.int32, device=DEV))
    assert last * 64 >= 2 ** 31
    assert torch.equal(memory[last, 0], qkv[:, 2 * hd:3 * hd]) and torch.equal(memory[last + 1, 0], qkv[:, 3 * hd:])
    assert bool((memory[last - 1] == 7.0).all()) and bool((memory[last + 2:] == 7.0).all())


@pytest.mark.parametrize("what, M, piece, H, parts", [("tanh", 260, 100, 1024, 5), ("normed", 900, 300, 2304, 2), ("of_sum", 200, 90, 1024, 9),
                                                    ("of_sum", 70, 64, 4096, 3), ("normed", 70, 64, 4096, 3)])
def test_norms_of_sums_in_steps_of_any_size(K, what, M, piece, H, parts):
    """Rows of a step together and in pieces that other variants take (registers, loads in flight, blocks): the same bits, and 64 bits
    beside them."""
    g = torch.Generator().manual_seed(M)
    x, a, b = torch.randn(M, H, generator=g), torch.randn(parts, M, H, generator=g), torch.randn(M, H, generator=g).to(torch.bfloat16)
    w, w2 = torch.randn(H, generator=g).to(DEV), torch.randn(H, generator=g).to(DEV)

    def run(lo, hi):
        xd, y = x[lo:hi].to(DEV), torch.empty(hi - lo, H, dtype=torch.bfloat16, device=DEV)
        ad, bd = a[:, lo:hi].contiguous().to(DEV), b[lo:hi].to(DEV)
        if what == "tanh":
            K.add_tanh_norm(xd, ad, w, w2, 0.4, y=y, w_next=w2, b_next=w, alpha_next=1.1)
        elif what == "normed":
            K.add_normed_terms(xd, [(ad, 1.0), (bd, 0.5)], w, 1e-5, y=y, w_next=w2, eps_next=1e-6)
        else:
            K.norm_of_sum(xd, [(ad, 1.0), (bd, 0.5)], 2.0, w, w2, 1e-5, y=y)
        return xd, y

    together = run(0, M)
    for whole, pieces in zip(together, zip(*[run(lo, min(M, lo + piece)) for lo in range(0, M, piece)])):
        assert torch.equal(whole, torch.cat(pieces))
    s, w64, v64 = a.double().sum(0), w.double().cpu(), w2.double().cpu()
    if what == "tanh":
        want = x.double() + torch.tanh(0.4 * s) * w64 + v64
    elif what == "normed":
        s = s + 0.5 * b.double()
        want = x.double() + s / (s.square().mean(1, keepdim=True) + 1e-5).sqrt() * w64
    else:
        s = 2.0 * x.double() + s + 0.5 * b.double()
        want = (s - s.mean(1, keepdim=True)) / (s.var(1, keepdim=True, unbiased=False) + 1e-5).sqrt() * w64 + v64
    # (a row's sums of H values in 32 bits, a few roundings)
    assert (together[0].double().cpu() - want).abs().max() < 1e-5 * want.abs().max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads, D, N", [(18, 64, 192), (4, 520, 128), (3, 129, 40), (18, 192, 128)])
def test_products_of_heads_of_few_tokens(K, dtype, heads, D, N):
    """Eight or 32 weights asked for ahead, as the blocks fit one round of the SMs and the inputs are long: the same bits from steps of
    any number of tokens, and the sums in 64 bits."""
    g = torch.Generator().manual_seed(D)
    T = 64
    x, w = torch.randn(T, heads * D, generator=g).to(dtype), torch.randn(heads, D, N, generator=g).to(dtype)

    def run(lo, hi):
        out = torch.full((hi - lo, heads * N), float("nan"), dtype=dtype, device=DEV)
        K.head_project(out, x[lo:hi].to(DEV), w.to(DEV), heads, D, N)
        return out

    whole = run(0, T)
    for piece in (1, 8, 33):
        assert torch.equal(whole, torch.cat([run(lo, min(T, lo + piece)) for lo in range(0, T, piece)]))
    want = torch.einsum("thd,hdn->thn", x.double().view(T, heads, D), w.double()).reshape(T, -1)
    # (sums of D products of size one in 32 bits, and the output's rounding)
    assert (whole.double().cpu() - want).abs().max() < (2e-6 if dtype == torch.float32 else 2.0 ** -7) * D ** 0.5 * 4
