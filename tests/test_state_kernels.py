"""The kernels of the state mixers, of the normed and rotated attention inputs and of the weighted
residual sum, each alone against the plain functions of ``plain_fiferax`` (float64), over sizes that
take every cut of the scan (lanes a column, key channels a lane, columns a block, tokens a chunk)."""
import math
from types import SimpleNamespace

import pytest
import torch

import plain_fiferax as plain

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
PAGE = 64


def batch_of(lens, slots):
    """The fields of a step's batch that the kernels read: sequences packed one after the other."""
    starts = [0]
    for n in lens:
        starts.append(starts[-1] + n)

    def i32(v):
        return torch.tensor(v, dtype=torch.int32, device=DEV)

    return SimpleNamespace(seq_starts=i32(starts), slots=i32(slots), n_seqs=len(lens), n_tokens=starts[-1])


def close(got, ref, tol=2e-5):
    ref = ref.double()
    err = float((got.double().cpu() - ref).abs().max() / ref.abs().max().clamp_min(1e-30))
    assert err < tol, err


@pytest.mark.parametrize("heads,dk,dv", [(2, 8, 8), (3, 24, 40), (1, 32, 32), (2, 64, 16), (2, 100, 36),
                                         (1, 128, 128), (1, 200, 72), (1, 4, 4), (2, 6, 10)])
def test_delta_rule_scan(heads, dk, dv):
    """Two sequences in one step against the plain rule; then the longer one again in three steps of
    unequal sizes down to one token (the state is carried), in a slot that another sequence used before;
    a padding row (slot -1) changes nothing and leaves zeros."""
    from airframe_b200 import kernels
    lens = [37, 5]
    T = sum(lens)
    g = torch.Generator().manual_seed(dk * 131 + dv)
    r, k, v = (torch.randn(T, heads * n, generator=g) for n in (dk, dk, dv))
    w = torch.rand(T, heads * dk, generator=g) * 0.5 + 0.5
    a = torch.rand(T, heads * dk, generator=g)
    u = k.view(T, heads, dk) / torch.sqrt((k.view(T, heads, dk) ** 2).sum(-1, keepdim=True) + 1e-6)
    au = (a.view(T, heads, dk) * u).reshape(T, -1)
    ref, at = [], 0
    for n in lens:
        s = slice(at, at + n)
        o, S = plain.delta_rule(r[s].double().view(n, heads, dk), k[s].double().view(n, heads, dk),
                                v[s].double().view(n, heads, dv), w[s].double().view(n, heads, dk),
                                a[s].double().view(n, heads, dk))
        ref.append((o.reshape(n, -1), S))
        at += n
    state = torch.zeros(4, heads, dv, dk, device=DEV)
    dev = [t.to(DEV) for t in (r, k, v, w, u.reshape(T, -1), au)]
    out = torch.full((T, heads * dv), 7.0, device=DEV)
    kernels.state_scan("delta", out, dev[0], dev[1], dev[2], state, batch_of(lens, [2, 0]), heads, dk, dv,
                       w=dev[3], u=dev[4], au=dev[5])
    close(out[:37], ref[0][0])
    close(out[37:], ref[1][0])
    close(state[2].transpose(1, 2), ref[0][1])
    close(state[0].transpose(1, 2), ref[1][1])
    assert float(state[1].abs().sum()) == 0 and float(state[3].abs().sum()) == 0
    # the first sequence again, in portions, in the slot the second one used; a padding row rides along
    state[0].zero_()
    got = []
    at = 0
    for n in (19, 13, 2, 1, 2):
        rows = [t[at:at + n].contiguous() for t in dev]
        pad = [torch.cat([t, torch.ones(1, t.shape[1], device=DEV)]) for t in rows]
        o = torch.full((n + 1, heads * dv), 7.0, device=DEV)
        before = state.clone()
        kernels.state_scan("delta", o, pad[0], pad[1], pad[2], state, batch_of([n, 1], [0, -1]), heads, dk, dv,
                           w=pad[3], u=pad[4], au=pad[5])
        assert float(o[n].abs().sum()) == 0 and torch.equal(before[1:], state[1:])
        got.append(o[:n])
        at += n
    close(torch.cat(got), ref[0][0])
    close(state[0].transpose(1, 2), ref[0][1])


@pytest.mark.parametrize("heads,dk,dv", [(3, 8, 20), (2, 12, 12), (2, 32, 64), (1, 128, 128), (4, 16, 16), (1, 72, 8)])
def test_decay_scan_with_silu(heads, dk, dv):
    from airframe_b200 import kernels
    lens = [50, 1, 9]
    T = sum(lens)
    g = torch.Generator().manual_seed(dk + 7 * dv)
    q, k, v = (torch.randn(T, heads * n, generator=g) for n in (dk, dk, dv))
    decay = torch.tensor([1.0, 0.5, 0.97, 0.999][:heads])
    state = torch.zeros(3, heads, dv, dk, device=DEV)
    out = torch.empty(T, heads * dv, device=DEV)
    # q, k, v as sections of one wider row, as a packed projection gives them
    packed = torch.cat([q, torch.zeros(T, 3), k, v], dim=1).to(DEV)
    oq, ok, ov = 0, heads * dk + 3, 2 * heads * dk + 3
    kernels.state_scan("decay", out, packed[:, oq:oq + heads * dk], packed[:, ok:ok + heads * dk],
                       packed[:, ov:ov + heads * dv], state, batch_of(lens, [1, 2, 0]), heads, dk, dv,
                       decay=decay.to(DEV), silu=True)
    at = 0
    for n in lens:
        s = slice(at, at + n)
        ref = plain.decay_linear_attention(plain.silu(q[s].double()).view(n, heads, dk),
                                           plain.silu(k[s].double()).view(n, heads, dk),
                                           plain.silu(v[s].double()).view(n, heads, dv), decay.double())
        close(out[s], ref.reshape(n, -1))
        at += n


def test_delta_prep():
    from airframe_b200 import kernels
    T, heads, dk, rank = 9, 3, 20, 7
    n = heads * dk
    g = torch.Generator().manual_seed(1)
    proj = torch.randn(T, 2 * n + rank + 5, generator=g)
    off_k, off_a, off_w1 = 5, 5 + n, 5 + 2 * n
    a_bias, w0 = torch.randn(n, generator=g), torch.randn(n, generator=g)
    w2 = torch.randn(n, rank, generator=g)
    out = torch.empty(T, 3, n, device=DEV)
    kernels.delta_prep(out, proj.to(DEV), off_k, off_a, off_w1, a_bias.to(DEV), w0.to(DEV), w2.t().contiguous().to(DEV), heads, dk,
                       math.exp(-0.5), 1e-6)
    p = proj.double()
    k = p[:, off_k:off_k + n].view(T, heads, dk)
    u = (k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)).reshape(T, n)
    w = torch.exp(-math.exp(-0.5) * plain.sigmoid(torch.tanh(p[:, off_w1:off_w1 + rank]) @ w2.double().T + w0.double()))
    a = plain.sigmoid(p[:, off_a:off_a + n] + a_bias.double())
    close(out[:, 0], w, 1e-6)
    close(out[:, 1], u, 1e-6)
    close(out[:, 2], a * u, 1e-6)


@pytest.mark.parametrize("width", [5, 44, 128, 300])
def test_gated_scan(width):
    from airframe_b200 import kernels
    lens = [23, 1, 6]
    T = sum(lens)
    g = torch.Generator().manual_seed(width)
    proj = torch.randn(T, 3 * width + 2, generator=g) * 2
    bz, bx = torch.randn(width, generator=g), torch.randn(width, generator=g)
    oz, ox, og = 2, 2 + width, 2 + 2 * width
    state = torch.zeros(5, width, device=DEV)
    for dt, tol in ((torch.float32, 2e-6), (torch.bfloat16, 8e-3)):
        state.zero_()
        y = torch.empty(T, width, dtype=dt, device=DEV)
        kernels.gated_scan(y, proj.to(DEV), oz, ox, og, bz.to(DEV), bx.to(DEV), state, batch_of(lens, [4, 0, 2]))
        at = 0
        for n, slot in zip(lens, [4, 0, 2]):
            p = proj[at:at + n].double()
            z = plain.sigmoid(p[:, oz:oz + width] + bz.double())
            c = p[:, ox:ox + width] + bx.double()
            S = plain.gated_recurrence(z, torch.where(c >= 0, c + 0.5, plain.sigmoid(c)))
            close(y[at:at + n], S * plain.silu(p[:, og:og + width]), tol)
            close(state[slot], S[-1], 2e-6)
            at += n


@pytest.mark.parametrize("width", [5, 16, 300])
@pytest.mark.parametrize("lens", [[129], [257, 700, 1], [256], [512, 255]])
def test_gated_scan_of_prompts(width, lens):
    """Steps with prompts: stretches of 256 tokens (of sequences of more than 192) that end inside a run, at its border and at the
    stretch's, shorter sequences beside them; bounds as for short ones (a state is a mean of what entered it: its error does not grow)."""
    from airframe_b200 import kernels
    T = sum(lens)
    g = torch.Generator().manual_seed(width)
    proj = torch.randn(T, 3 * width, generator=g) * 2
    bz, bx = torch.randn(width, generator=g), torch.randn(width, generator=g)
    state = torch.zeros(4, width, device=DEV)
    state[1:] = torch.randn(3, width, generator=g).to(DEV)
    before, slots = state.clone().cpu().double(), [3, 0, 2][:len(lens)]
    y = torch.empty(T, width, device=DEV)
    kernels.gated_scan(y, proj.to(DEV), 0, width, 2 * width, bz.to(DEV), bx.to(DEV), state, batch_of(lens, slots))
    for (s, n), slot in zip(in_order(lens), slots):
        p = proj[s].double()
        z, c = plain.sigmoid(p[:, :width] + bz.double()), p[:, width:2 * width] + bx.double()
        cand, S, out = torch.where(c >= 0, c + 0.5, plain.sigmoid(c)), before[slot], []
        for t in range(n):
            S = (1 - z[t]) * S + z[t] * cand[t]
            out.append(S)
        close(y[s], torch.stack(out) * plain.silu(p[:, 2 * width:]), 2e-6)
        close(state[slot], S, 2e-6)
    assert torch.equal(state[1].cpu().double(), before[1])


@pytest.mark.parametrize("n,group", [(48, 24), (60, 60), (256, 128), (24, 8)])
def test_gated_group_norm(n, group):
    from airframe_b200 import kernels
    T = 7
    g = torch.Generator().manual_seed(n)
    o, w, gate = torch.randn(T, n, generator=g) * 3, torch.randn(n, generator=g), torch.randn(T, n + 4, generator=g)
    y = torch.empty(T, n, device=DEV)
    kernels.gated_group_norm(y, o.to(DEV), w.to(DEV), gate.to(DEV)[:, 4:], group, 1e-5)
    ref = plain.rms(o.double().view(T, n // group, group), 1e-5).reshape(T, n) * w.double() * plain.sigmoid(gate[:, 4:].double())
    close(y, ref, 2e-6)


@pytest.mark.parametrize("nq,nkv,hd,rot,shared_v", [(4, 4, 12, 6, True), (6, 2, 64, 64, True), (2, 1, 20, 0, True),
                                                    (3, 3, 16, 16, False)])
def test_norm_rotate_pack_and_store(nq, nkv, hd, rot, shared_v):
    """q and k heads normed and rotated, v taken from the raw k (or its own heads), rows packed, and k and v
    in the cache: a ring of 64 rows in which, of two tokens that share a row, the later one stays."""
    from airframe_b200 import kernels
    from airframe_b200.cache.sequence_cache import KVView
    from airframe_b200.parts.base import KVNeed
    lens = [70, 3]
    T = sum(lens)
    g = torch.Generator().manual_seed(hd)
    width_in = (nq + nkv + (0 if shared_v else nkv)) * hd
    proj = torch.randn(T, width_in, generator=g)
    qw, kw = torch.randn(hd, generator=g), torch.randn(hd, generator=g)
    inv = torch.tensor([50.0 ** (-2.0 * i / rot) for i in range(rot // 2)], dtype=torch.float32)
    pos = torch.tensor(list(range(70)) + list(range(3)), dtype=torch.int32, device=DEV)
    b = batch_of(lens, [1, 0])
    b.positions = pos
    b.seq_of_token = torch.tensor([0] * 70 + [1] * 3, dtype=torch.int32, device=DEV)
    b.len_after = torch.tensor(lens, dtype=torch.int32, device=DEV)
    kc = torch.zeros(4, nkv, PAGE, hd, device=DEV)
    vc = torch.zeros(4, nkv, PAGE, hd, device=DEV)
    table = torch.tensor([[3], [2]], dtype=torch.int32, device=DEV)            # slot -> its one page
    kv = KVView(kc, vc, table, PAGE, KVNeed(nkv, hd, 40))
    qkv = torch.empty(T, (nq + 2 * nkv) * hd, device=DEV)
    kernels.qk_norm_rope_store(qkv, proj.to(DEV), b, nq, nkv, hd, inv.to(DEV), rot, "half", q_weight=qw.to(DEV),
                               k_weight=kw.to(DEV), eps=1e-5, v_from_k=shared_v, kv=kv)
    p = proj.double()
    q = p[:, :nq * hd].view(T, nq, hd)
    k = p[:, nq * hd:(nq + nkv) * hd].view(T, nkv, hd)
    v = k if shared_v else p[:, (nq + nkv) * hd:].view(T, nkv, hd)
    positions = pos.cpu().long()
    qr = plain.rotate_half(plain.rms(q, 1e-5, qw.double()), positions, 50.0, rot)
    kr = plain.rotate_half(plain.rms(k, 1e-5, kw.double()), positions, 50.0, rot)
    close(qkv[:, :nq * hd], qr.reshape(T, -1), 3e-6)
    close(qkv[:, nq * hd:(nq + nkv) * hd], kr.reshape(T, -1), 3e-6)
    close(qkv[:, (nq + nkv) * hd:], v.reshape(T, -1), 1e-7)
    # sequence 0 (slot 1, page 2): rows 0..5 hold positions 64..69, rows 6..63 positions 6..63
    for row, t in [(0, 64), (5, 69), (6, 6), (63, 63)]:
        close(kc[2, :, row], kr[t], 3e-6)
        close(vc[2, :, row], v[t], 1e-7)
    close(kc[3, :, 2], kr[72], 3e-6)
    assert float(kc[3, :, 3:].abs().sum()) == 0 and float(kc[:2].abs().sum()) == 0


def test_weighted_residual_sum_and_norm():
    from airframe_b200 import kernels
    n, H = 11, 72
    g = torch.Generator().manual_seed(5)
    x0 = torch.randn(n, H, generator=g)
    a = torch.randn(n, H, generator=g).to(torch.bfloat16)
    parts = torch.randn(3, n, H, generator=g)
    w = torch.randn(H, generator=g)
    x = x0.to(DEV)
    y = torch.empty(n, H, device=DEV)
    kernels.add_scaled_rmsnorm(x, [(a.to(DEV), 0.8), (parts.to(DEV), 1.25)], y=y, w_next=w.to(DEV), eps=1e-5, offset=0.0)
    ref = x0.double() + 0.8 * a.double() + 1.25 * parts.double().sum(0)
    close(x, ref, 1e-6)
    close(y, plain.rms(ref, 1e-5, w.double()), 2e-6)
    x = x0.to(DEV)
    kernels.add_scaled_rmsnorm(x, [(parts.to(DEV), 1.0), (a.to(DEV), 1.0), (a.to(DEV), -1.0)])
    close(x, x0.double() + parts.double().sum(0), 1e-6)


CHUNK_LENS = [1, 16, 17, 31, 32, 33, 64, 95, 230]      # tokens at and around the borders of groups of 16 and chunks of 32


def prompt_batch(lens, slots):
    b = batch_of(lens, slots)
    b.seq_lens, b.tokens, b.aux = lens, b.slots, {}
    return b


def in_order(lens):
    at = 0
    for n in lens:
        yield slice(at, at + n), n
        at += n


@pytest.mark.parametrize("at_once", [512, 3])
@pytest.mark.parametrize("heads,dk,dv,rank,scale", [(2, 16, 16, 5, math.exp(-0.5)), (3, 48, 32, 64, 0.01), (1, 64, 80, 128, 2.0),
                                                    (2, 128, 128, 64, math.exp(-0.5)), (1, 112, 16, 1, 200.0)])
def test_general_delta_in_chunks(heads, dk, dv, rank, scale, at_once, monkeypatch):
    """Prompts in chunks against the plain rule in 64 bits and against the token-by-token kernels, then more tokens from the
    states they left; decays from none to (scale 200) all at once; sequences in one launch and in several.  Bounds: the
    recurrence's sums are of up to 128 products of 32 bits, a few thousand roundings of 2^-24 at most: 2e-5 of the largest value."""
    from airframe_b200 import kernels
    assert kernels.state_chunks_supported(dk, dv, rank) and not kernels.state_chunks_supported(dk + 8, dv, rank)
    assert not kernels.state_chunks_supported(dk, dv + 8, rank) and not kernels.state_chunks_supported(dk, dv, 129)
    monkeypatch.setattr(kernels, "STATE_CHUNKS_AT_ONCE", at_once)
    T, n = sum(CHUNK_LENS), heads * dk
    g = torch.Generator().manual_seed(dk + rank)
    widths = {"r": n, "k": n, "v": heads * dv, "a": n, "w1": rank}
    cols, at = {}, 4
    for name, w in widths.items():
        cols[name] = slice(at, at + w)
        at += (w + 3) // 4 * 4
    proj = torch.randn(T, (at + 3) // 4 * 4, generator=g)
    a_bias, w0 = torch.randn(n, generator=g), torch.randn(n, generator=g)
    w2 = torch.randn(n, rank, generator=g) * rank ** -0.5
    slots = [4, 0, 8, 2, 1, 3, 7, 5, 6]
    state = torch.zeros(10, heads, dv, dk, device=DEV)
    p = {name: proj.to(DEV)[:, c] for name, c in cols.items()}
    consts = {"a_bias": a_bias.to(DEV), "w0": w0.to(DEV), "w2t": w2.t().contiguous().to(DEV)}
    out = torch.full((T, heads * dv), 7.0, device=DEV)

    def chunks(rows, o, lens, where):
        kernels.state_chunks("delta", o, p["r"][rows], p["k"][rows], p["v"][rows], state, prompt_batch(lens, where), heads, dk, dv,
                             a=p["a"][rows], low=p["w1"][rows], decay_scale=scale, key_eps=1e-6, **consts)

    chunks(slice(0, T), out, CHUNK_LENS, slots)
    pd = {name: proj.double()[:, c] for name, c in cols.items()}
    w = torch.exp(-scale * plain.sigmoid(torch.tanh(pd["w1"]) @ w2.double().T + w0.double()))
    a = plain.sigmoid(pd["a"] + a_bias.double())
    for (s, length), slot in zip(in_order(CHUNK_LENS), slots):
        o, S = plain.delta_rule(*(t[s].view(length, heads, -1) for t in (pd["r"], pd["k"], pd["v"], w, a)))
        close(out[s], o.reshape(length, -1))
        close(state[slot].transpose(1, 2), S)
    assert float(state[9].abs().sum()) == 0
    # token by token, and the last prompt again in two steps
    pre = torch.empty(T, 3, n, device=DEV)
    kernels.delta_prep(pre, proj.to(DEV), cols["k"].start, cols["a"].start, cols["w1"].start, consts["a_bias"], consts["w0"],
                       consts["w2t"], heads, dk, scale, 1e-6)
    twin, other = torch.empty_like(out), torch.zeros_like(state)
    kernels.state_scan("delta", twin, p["r"], p["k"], p["v"], other, batch_of(CHUNK_LENS, slots), heads, dk, dv, w=pre[:, 0],
                       u=pre[:, 1], au=pre[:, 2])
    close(out, twin.cpu())
    close(state, other.cpu())
    last = list(in_order(CHUNK_LENS))[-1][0]
    whole = out[last].clone()
    state[6].zero_()
    for rows in (slice(last.start, last.start + 77), slice(last.start + 77, last.stop)):
        o = torch.empty(rows.stop - rows.start, heads * dv, device=DEV)
        chunks(rows, o, [len(o)], [6])
        close(o, whole[rows.start - last.start: rows.stop - last.start].cpu())


@pytest.mark.parametrize("heads,dk,dv,silu", [(3, 16, 32, True), (2, 64, 64, False), (4, 128, 128, True), (2, 96, 144, True)])
def test_decay_attention_in_chunks(heads, dk, dv, silu):
    """Prompts in chunks against the plain rule in 64 bits, sections of one wider row; the states go on in a second step."""
    from airframe_b200 import kernels
    T, n = sum(CHUNK_LENS), heads * dk
    g = torch.Generator().manual_seed(dk + 7 * dv)
    proj = torch.randn(T, 8 + 2 * n + heads * dv, generator=g)
    cols = slice(4, 4 + n), slice(4 + n, 4 + 2 * n), slice(8 + 2 * n, None)
    decay = torch.tensor([1.0, 0.0, 0.97, 0.999][:heads])
    slots = [4, 0, 8, 2, 1, 3, 7, 5, 6]
    state = torch.zeros(10, heads, dv, dk, device=DEV)
    out = torch.full((T, heads * dv), 7.0, device=DEV)
    dev = [proj.to(DEV)[:, c] for c in cols]
    act = plain.silu if silu else (lambda x: x)
    ref = [act(proj.double()[:, c]) for c in cols]

    def run(rows, lens, where):
        kernels.state_chunks("decay", out[rows], *(t[rows] for t in dev), state, prompt_batch(lens, where), heads, dk, dv,
                             decay=decay.to(DEV), silu=silu)

    run(slice(0, T), CHUNK_LENS, slots)
    for s, length in in_order(CHUNK_LENS):
        close(out[s], plain.decay_linear_attention(*(t[s].view(length, heads, -1) for t in ref), decay.double()).reshape(length, -1))
    last = list(in_order(CHUNK_LENS))[-1][0]
    whole = out[last].clone()
    state[6].zero_()
    for rows in (slice(last.start, last.start + 77), slice(last.start + 77, last.stop)):
        run(rows, [rows.stop - rows.start], [6])
    close(out[last], whole.cpu())


@pytest.mark.parametrize("what", ["r", "k", "v", "a", "w1"])
@pytest.mark.parametrize("mode", ["delta", "decay"])
def test_chunks_of_values_that_are_not_finite(mode, what):
    """An infinity or a NaN at a token leaves the tokens before it as they are, bit for bit, and reaches the tokens behind it as
    token by token it does: at places within a group of four rows, of 16 tokens and of a chunk of 32."""
    from airframe_b200 import kernels
    if mode == "decay" and what in ("a", "w1"):
        return
    heads, dk, dv, rank, lens, slots = 2, 32, 32, 8, [70, 40], [1, 0]
    T, n = sum(lens), heads * dk
    g = torch.Generator().manual_seed(3)
    data = {name: torch.randn(T, w, generator=g) for name, w in (("r", n), ("k", n), ("v", heads * dv), ("a", n), ("w1", rank))}
    a_bias, w0 = torch.randn(n, generator=g).to(DEV), torch.randn(n, generator=g).to(DEV)
    w2t = torch.randn(rank, n, generator=g).to(DEV)
    decay = torch.tensor([0.9, 1.0], device=DEV)

    def run(chunked):
        d = {name: t.to(DEV) for name, t in data.items()}
        state, out = torch.zeros(2, heads, dv, dk, device=DEV), torch.empty(T, heads * dv, device=DEV)
        args = (mode, out, d["r"], d["k"], d["v"], state)
        if chunked:
            more = (dict(a=d["a"], low=d["w1"], a_bias=a_bias, w0=w0, w2t=w2t, decay_scale=0.5, key_eps=1e-6) if mode == "delta"
                    else dict(decay=decay))
            kernels.state_chunks(*args, prompt_batch(lens, slots), heads, dk, dv, **more)
        elif mode == "decay":
            kernels.state_scan(*args, batch_of(lens, slots), heads, dk, dv, decay=decay)
        else:
            proj = torch.cat([d["k"], d["a"], d["w1"]], 1)
            pre = torch.empty(T, 3, n, device=DEV)
            kernels.delta_prep(pre, proj, 0, n, 2 * n, a_bias, w0, w2t, heads, dk, 0.5, 1e-6)
            kernels.state_scan(*args, batch_of(lens, slots), heads, dk, dv, w=pre[:, 0], u=pre[:, 1], au=pre[:, 2])
        return out

    clean = run(True)
    assert bool(clean.isfinite().all())
    for t in (0, 2, 3, 17, 30, 35, 69):
        for bad in (math.inf, -math.inf, math.nan):
            if what in ("a", "w1") and bad == bad:
                continue                               # (a sigmoid or tanh of an infinity is finite)
            kept = data[what][t, 5].item()
            data[what][t, 5] = bad
            got, twin = run(True), run(False)
            data[what][t, 5] = kept
            assert torch.equal(got[:t], clean[:t]) and torch.equal(got[lens[0]:], clean[lens[0]:]), (t, bad)
            assert torch.equal(got.isfinite(), twin.isfinite()), (t, bad)
            assert not bool(got[t].isfinite().all())


@pytest.mark.parametrize("mode", ["delta", "decay"])
def test_chunks_of_padding_rows(mode):
    """A sequence without a slot leaves zeros and no state, as token by token."""
    from airframe_b200 import kernels
    heads, dk, dv, rank, lens, slots = 2, 32, 48, 8, [40, 33, 5], [1, -1, 0]
    T, n = sum(lens), heads * dk
    g = torch.Generator().manual_seed(5)
    r, k, v, a, low = (torch.randn(T, w, generator=g).to(DEV) for w in (n, n, heads * dv, n, rank))
    more = (dict(a=a, low=low, a_bias=r[0], w0=k[0], w2t=torch.randn(rank, n, generator=g).to(DEV), decay_scale=0.5, key_eps=1e-6)
            if mode == "delta" else dict(decay=torch.tensor([0.9, 1.0], device=DEV)))
    outs, states = [], []
    for where in (slots, [1, 2, 0]):
        state, out = torch.zeros(3, heads, dv, dk, device=DEV), torch.full((T, heads * dv), float("nan"), device=DEV)
        kernels.state_chunks(mode, out, r, k, v, state, prompt_batch(lens, where), heads, dk, dv, **more)
        outs.append(out), states.append(state)
    assert bool((outs[0][40:73] == 0).all()) and float(states[0][2].abs().sum()) == 0
    for rows in (slice(0, 40), slice(73, T)):
        assert torch.equal(outs[0][rows], outs[1][rows])
    assert torch.equal(states[0][:2], states[1][:2])


def test_chunk_tables_of_other_sizes_in_a_step():
    """A step's tables of chunks go by their size: what another kernel cut into chunks of 64 tokens is not taken for its own."""
    from airframe_b200 import kernels
    heads, dk, dv, lens = 2, 16, 16, [70, 33]
    T, n = sum(lens), heads * dk
    g = torch.Generator().manual_seed(6)
    r, k, v = (torch.randn(T, w, generator=g).to(DEV) for w in (n, n, heads * dv))
    decay, outs = torch.tensor([0.9, 1.0], device=DEV), []
    for other in (None, 64, 16):
        batch = prompt_batch(lens, [1, 0])
        if other is not None:
            starts, first, count = kernels._chunk_table(batch, other)
            assert count == sum(-(-x // other) for x in lens)
            assert starts.tolist() == [*range(0, 70, other), *range(70, 103, other), 103] and first.tolist() == [0, -(-70 // other), count]
        state, out = torch.zeros(2, heads, dv, dk, device=DEV), torch.empty(T, heads * dv, device=DEV)
        kernels.state_chunks("decay", out, r, k, v, state, batch, heads, dk, dv, decay=decay)
        outs.append((out, state))
    assert all(torch.equal(o, outs[0][0]) and torch.equal(s, outs[0][1]) for o, s in outs)


@pytest.mark.parametrize("mode", ["delta", "decay"])
def test_long_sequences_in_several_launches(mode, monkeypatch):
    """Sequences of more chunks than are held at a time are cut and go on from the state in memory: the same bits as in one launch,
    for outputs and states, and no more scratch than allowed."""
    from airframe_b200 import kernels
    heads, dk, dv, rank, lens, slots = 3, 64, 32, 16, [40, 32 * 9 + 5, 1, 7 * 32, 64], [3, 0, 4, 1, 2]
    T, n = sum(lens), heads * dk
    g = torch.Generator().manual_seed(8)
    r, k, v, a, low = (torch.randn(T, w, generator=g).to(DEV) for w in (n, n, heads * dv, n, rank))
    more = (dict(a=a, low=low, a_bias=r[0], w0=k[0], w2t=torch.randn(rank, n, generator=g).to(DEV), decay_scale=0.05, key_eps=1e-6)
            if mode == "delta" else dict(decay=torch.tensor([0.9, 0.99, 1.0], device=DEV)))
    start, got = torch.randn(5, heads, dv, dk, generator=g).to(DEV), []

    def run():
        state, out = start.clone(), torch.full((T, heads * dv), float("nan"), device=DEV)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        kernels.state_chunks(mode, out, r, k, v, state, prompt_batch(lens, slots), heads, dk, dv, **more)
        return out, state, torch.cuda.max_memory_allocated() - before

    whole = run()
    chunk = whole[2] // sum(-(-x // 32) for x in lens)
    for most in (1, 2, 3, 5, 8):
        with monkeypatch.context() as m:
            m.setattr(kernels, "STATE_CHUNKS_AT_ONCE", most)
            got = run()
        assert torch.equal(got[0], whole[0]) and torch.equal(got[1], whole[1]), most
        with monkeypatch.context() as m:
            m.setattr(kernels, "STATE_CHUNKS_BYTES", most * chunk)
            got = run()
        assert torch.equal(got[0], whole[0]) and torch.equal(got[1], whole[1]), most
        assert got[2] <= most * chunk + 8192


@pytest.mark.parametrize("width", [5, 40, 300])
def test_gated_scan_alone_and_in_a_batch(width):
    """A sequence's rows and state are the same bits alone and beside others, shorter and longer: its own length decides how its
    tokens are composed (up to 192 one way, from 193 on another), not the step's."""
    from airframe_b200 import kernels
    lens, slots = [1, 1000, 17, 128, 129, 192, 193, 300], [3, 0, 2, 7, 1, 4, 6, 5]
    T = sum(lens)
    g = torch.Generator().manual_seed(width)
    proj = (torch.randn(T, 3 * width, generator=g) * 2).to(DEV)
    bz, bx, start = (torch.randn(*s, generator=g).to(DEV) for s in ((width,), (width,), (8, width)))

    def run(rows, some, where):
        state, y = start.clone(), torch.full((rows.stop - rows.start, width), float("nan"), device=DEV)
        kernels.gated_scan(y, proj[rows], 0, width, 2 * width, bz, bx, state, prompt_batch(some, where))
        return y, state

    y, state = run(slice(0, T), lens, slots)
    pieces = list(in_order(lens))
    for (rows, n), slot in zip(pieces, slots):
        alone, left = run(rows, [n], [slot])
        assert torch.equal(alone, y[rows]) and torch.equal(left[slot], state[slot]), n
    for some in ([0, 2, 3], [4, 5], [6, 0], [7, 3]):          # (neighbours in another step)
        data = torch.cat([proj[pieces[i][0]] for i in some])
        st, out = start.clone(), torch.empty(len(data), width, device=DEV)
        kernels.gated_scan(out, data, 0, width, 2 * width, bz, bx, st, prompt_batch([lens[i] for i in some], [slots[i] for i in some]))
        assert torch.equal(out, torch.cat([y[pieces[i][0]] for i in some]))
