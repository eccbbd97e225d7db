"""Each kernel of the Kotisun parts alone against the plain functions, on inputs made so that a fault shows: a residual in
streams with a mix that is not symmetric; attention whose one key scores far above all others, placed at the first
position, on both sides of block borders, far back, and just inside and just outside the window; a recurrence fed in
two steps of odd and even lengths from NaN-poisoned neighbours' states."""
import pytest
import torch

import plain_kotisun as plain

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def dev(t, dtype=torch.float32):
    return t.to(device=DEV, dtype=dtype).contiguous()


def close(got, want, tol, what=""):
    got, want = got.double().cpu(), want.double()
    assert torch.isfinite(got).all(), what
    err = float((got - want).abs().max() / want.abs().max().clamp_min(1e-30))
    assert err < tol, (what, err)


@pytest.mark.parametrize("S,d", [(1, 40), (3, 64), (4, 100), (7, 33), (16, 8)])
def test_streams_read_write_embed(S, d):
    from vlrf_b200.csrc import ops
    g = torch.Generator().manual_seed(S)
    T, V = 9, 50
    table = torch.randn(V, d, generator=g)
    toks = torch.randint(0, V, (T,), generator=g)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    x = torch.full((T, S * d), float("nan"), device=DEV)
    ops.embed_streams(dev(table, torch.bfloat16), dev(toks, torch.int32), x, S, 1.75, err)
    want0 = (table.bfloat16().double()[toks] * 1.75)
    close(x.view(T, S, d), want0[:, None, :].expand(T, S, d), 1e-6, "embed")
    xs = torch.randn(T, S, d, generator=g).double()
    a, b, m, w = (torch.randn(n, generator=g).double() for n in (S, S, S * S, d))
    m = m.view(S, S)
    y = torch.randn(T, d, generator=g).double()
    for dtype, tol in ((torch.float32, 1e-5), (torch.bfloat16, 6e-3)):
        out = torch.empty(T, d, dtype=dtype, device=DEV)
        ops.streams_read_norm(dev(xs.view(T, S * d)), S, dev(a), dev(w), 1e-5, out)
        close(out, plain.rms_norm(torch.einsum("s,tsd->td", a, xs), w, 1e-5), tol, "read")
    rows = torch.tensor([5, 0, 5, 8], dtype=torch.int32)
    out = torch.empty(4, d, device=DEV)
    ops.streams_read_norm(dev(xs.view(T, S * d)), S, None, dev(w), 1e-5, out, dev(rows, torch.int32))
    close(out, plain.rms_norm(xs.sum(1)[rows.long()], w, 1e-5), 1e-5, "sum of the streams, gathered rows")
    xd = dev(xs.view(T, S * d))
    ops.streams_write(xd, S, dev(m), dev(b), dev(y), T - 1)
    want = torch.einsum("sj,tsd->tjd", m, xs) + b[None, :, None] * y[:, None, :]
    close(xd.view(T, S, d)[:T - 1], want[:T - 1], 1e-5, "write")
    close(xd.view(T, S, d)[T - 1], xs[T - 1], 1e-7, "rows beyond the step stay")
    a2, w2 = torch.randn(S, generator=g).double(), torch.randn(d, generator=g).double()
    for dtype, tol in ((torch.float32, 1e-5), (torch.bfloat16, 6e-3)):
        xd, h = dev(xs.view(T, S * d)), torch.full((T, d), float("nan"), dtype=dtype, device=DEV)
        ops.streams_write_read(xd, S, dev(m), dev(b), dev(y), dev(a2), dev(w2), 1e-5, h, T - 1)
        close(xd.view(T, S, d)[:T - 1], want[:T - 1], 1e-5, "write of write_read")
        close(h[:T - 1], plain.rms_norm(torch.einsum("j,tjd->td", a2, want), w2, 1e-5)[:T - 1], tol, "read of write_read")
        close(xd.view(T, S, d)[T - 1], xs[T - 1], 1e-7, "rows beyond the step stay")
    lg = torch.randn(5, 37, generator=g) * 40
    ld = dev(lg)
    ops.softcap(ld, 4, 30.0)
    close(ld[:4], 30.0 * torch.tanh(lg[:4].double() / 30.0), 1e-6, "softcap")
    assert torch.equal(ld[4].cpu(), lg[4])


class PagedKV:
    """A paged cache with a permuted block table and NaN in every place that nothing wrote."""

    def __init__(self, n_slots, max_len, G, dk, dv, dtype):
        self.bt = 64
        self.max_blocks = (max_len + 63) // 64
        nb = n_slots * self.max_blocks + 3
        self.k = torch.full((nb, G, 64, dk), float("nan"), dtype=dtype, device=DEV)
        self.v = torch.full((nb, G, 64, dv), float("nan"), dtype=dtype, device=DEV)
        perm = torch.randperm(nb, generator=torch.Generator().manual_seed(1))[:n_slots * self.max_blocks]
        self.table = dev(perm.view(n_slots, self.max_blocks), torch.int32)


def run_attention(q, k, v, positions, slot_of, lens, G, scale, window, rot, dtype, out_scale=1.0, tail=None, splits=None):
    """q [T, H, dk], k [T, G, dk], v [T, G, dv] unrotated, for tokens at (slot_of[t], positions[t]): all appended to the
    cache, then attended.  tail None: every token is a query of one prompt step, by the kernel that takes a warp per token
    and head.  tail = n: the last n tokens of every sequence are the step's new tokens (a later portion of a prompt; n = 1:
    a decode step, its contexts cut into `splits` parts), by the kernel that the step function chooses."""
    import types
    from vlrf_b200.csrc import ops
    from vlrf_b200.parts.context import Workspace
    T, H, dk = q.shape
    dv = v.shape[2]
    cache = PagedKV(max(slot_of) + 1, max(lens), G, dk, dv, dtype)
    proj = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], dim=1)
    wide = torch.full((T, proj.shape[1] + 5), float("nan"))
    wide[:, 3:3 + proj.shape[1]] = proj                       # the rows lie inside wider rows
    wide = dev(wide)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    qo = torch.full((T, H * dk), float("nan"), dtype=dtype, device=DEV)
    freq = None
    if rot:
        base, dims, factor = rot
        freq = dev(torch.tensor([base ** (-2.0 * i / dims) / factor for i in range(dims // 2)], dtype=torch.float64))
    tok_slot, tok_pos = dev(torch.tensor(slot_of), torch.int32), dev(torch.tensor(positions), torch.int32)
    ops.qkv_rope_append(wide[:, 3:3 + proj.shape[1]], 0, H * dk, H * dk + G * dk, freq, rot[1] if rot else 0, qo, cache.k, cache.v,
                        cache.table, tok_slot, tok_pos, T, H, G, dk, dv, True, err)
    pad = 8                                                    # (the tensor-core kernel wants rows on 4-byte boundaries)
    if tail is None:
        out = torch.full((T, H * dv + 2 * pad), float("nan"), dtype=dtype, device=DEV)
        ops.attention_window(qo, cache.k, cache.v, cache.table, tok_slot, tok_pos, out[:, pad:pad + H * dv], T, H, G, dk, dv, scale,
                             window, out_scale, err)
        keep = list(range(T))
    else:
        keep, seq_start, seq_pos0, start = [], [0], [], 0
        for n in lens:
            m = min(tail, n)
            keep += list(range(start + n - m, start + n))
            seq_start.append(seq_start[-1] + m); seq_pos0.append(n - m)
            start += n
        idx = torch.tensor(keep)
        ctx = types.SimpleNamespace(
            n_tokens=len(keep), n_seqs=len(lens), max_new=min(tail, max(lens)), max_context=max(lens), ws=Workspace(DEV), dev_err=err,
            tok_slot=dev(torch.tensor(slot_of)[idx], torch.int32), tok_pos=dev(torch.tensor(positions)[idx], torch.int32),
            seq_slot=dev(torch.tensor(list(range(len(lens)))), torch.int32), seq_start=dev(torch.tensor(seq_start), torch.int32),
            seq_pos0=dev(torch.tensor(seq_pos0), torch.int32))
        out = torch.full((len(keep), H * dv + 2 * pad), float("nan"), dtype=dtype, device=DEV)
        import os
        if splits:
            os.environ["VLRF_B200_DECODE_SPLITS"] = str(splits)
        try:
            ops.attention_window_step(qo[idx.to(DEV)].contiguous(), cache.k, cache.v, cache.table, out[:, pad:pad + H * dv], ctx, H, G, dk, dv,
                                      scale, window, out_scale)
        finally:
            os.environ.pop("VLRF_B200_DECODE_SPLITS", None)
    assert int(err.item()) == 0
    assert torch.isnan(out[:, :pad].float()).all() and torch.isnan(out[:, pad + H * dv:].float()).all()
    return out[:, pad:pad + H * dv].view(len(keep), H, dv), keep


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-5), (torch.bfloat16, 2e-2)])
@pytest.mark.parametrize("H,G,dk,dv,window,rot", [
    (4, 2, 16, 24, 40, (10000.0, 8, 2.0)), (2, 2, 32, 32, 64, (500.0, 32, 1.0)), (6, 1, 8, 16, 0, None), (3, 3, 24, 8, 65, (3e4, 12, 8.0)),
    (3, 1, 12, 20, 1, (3000.0, 6, 1.3)), (5, 5, 80, 48, 130, (250.0, 16, 4.0)), (16, 1, 64, 128, 100, (1e4, 64, 1.0)),
    (8, 2, 128, 104, 0, (1e4, 32, 1.0)), (34, 2, 40, 40, 70, None)])
def test_attention_with_a_key_that_stands_out(H, G, dk, dv, window, rot, dtype, tol):
    """Sequences of 1, 2, 64, 65, 129 and 200 tokens in one step.  For the LAST query of every sequence the oldest key its
    window lets it see is made to score far above the rest, and the key just before that one, which it must not see,
    higher still; without a window the first key of the sequence stands out.  As one prompt step, as a later portion of
    70 and of 3 tokens, and as a decode step whose contexts are whole, cut in 2 and cut in 5."""
    g = torch.Generator().manual_seed(dk + dv)
    lens = [1, 2, 64, 65, 129, 200]
    slot_of, positions = [], []
    for s, n in enumerate(lens):
        slot_of += [s] * n
        positions += list(range(n))
    T = len(slot_of)
    rd = lambda *shape: torch.randn(*shape, generator=g).bfloat16().double()   # noqa: E731
    q, k, v = rd(T, H, dk), rd(T, G, dk), rd(T, G, dv)
    start = 0
    for s, n in enumerate(lens):
        last = start + n - 1
        inside = max(0, n - window) if window else 0               # the oldest key the last query sees
        for hk in range(G):
            # (unrotated entries only, so the rotation cannot undo it) matched to the first query head that reads the key
            h = hk * (H // G)
            lo = rot[1] if rot else 0
            if lo < dk:
                unit = q[last, h, lo:] / max(1e-3, float(q[last, h, lo:].norm()))
                k[start + inside, hk, lo:] = (6.0 * unit).bfloat16().double()
                if inside > 0:
                    k[start + inside - 1, hk, lo:] = (9.0 * unit).bfloat16().double()     # just outside: louder still
        start += n
    pos = torch.tensor(positions)
    rq = plain.rotate_scaled(q, pos, *rot) if rot else q
    rk = plain.rotate_scaled(k, pos, *rot) if rot else k
    want = torch.zeros(T, H, dv, dtype=torch.float64)
    start = 0
    for n in lens:
        want[start:start + n] = plain.window_attention(rq[start:start + n], rk[start:start + n], v[start:start + n], 0.3, window)
        start += n
    for tail, splits in ((None, None), (70, None), (3, None), (1, 1), (1, 2), (1, 5)):
        if tail is None and (H // G > 16 or max(dk, dv) > 256):
            continue
        got, keep = run_attention(q.float(), k.float(), v.float(), positions, slot_of, lens, G, 0.3, window, rot, dtype, 0.6, tail, splits)
        close(got, 0.6 * want[torch.tensor(keep)], tol, f"attention, tail {tail}, {splits} parts")


@pytest.mark.parametrize("Hs,P,N,G,taps,ng", [(4, 8, 16, 2, 4, 2), (2, 24, 8, 1, 2, 1), (3, 16, 24, 3, 3, 3), (5, 6, 10, 5, 5, 3),
                                              (1, 32, 16, 1, 1, 1), (2, 64, 128, 1, 4, 8), (8, 80, 48, 2, 4, 4)])
def test_recurrence_in_steps_of_every_parity(Hs, P, N, G, taps, ng):
    """Three sequences in slots 4, 0 and 2 of six (the others full of NaN, and a padding row in every step): a first step of
    5, 8 and 1 tokens, then single tokens, then a step of 2, 3 and 6 — against the plain functions over the whole."""
    from vlrf_b200.csrc import ops
    g = torch.Generator().manual_seed(Hs * 100 + P)
    inner, channels = Hs * P, Hs * P + 2 * G * N
    width = 2 * inner + 2 * G * N + Hs
    lens = [5 + 3 + 2, 8 + 3 + 3, 1 + 3 + 6]
    slots = [4, 0, 2]
    cuts = [[5, 1, 1, 1, 2], [8, 1, 1, 1, 3], [1, 1, 1, 1, 6]]
    proj = [torch.randn(n, width, generator=g).double() for n in lens]
    conv_w, conv_b = torch.randn(channels, taps, generator=g).double() * 0.5, torch.randn(channels, generator=g).double() * 0.3
    dt_bias, a_log, D = torch.randn(Hs, generator=g).double(), torch.randn(Hs, generator=g).double() - 1.0, torch.randn(Hs, generator=g).double()
    norm_w = torch.randn(inner, generator=g).double()
    want = []
    for pr in proj:
        z, xbc, dt = pr[:, :inner], pr[:, inner:inner + channels], pr[:, inner + channels:]
        xbc = plain.silu(plain.causal_conv(xbc, conv_w, conv_b))
        n = pr.shape[0]
        y = plain.selective_scan(xbc[:, :inner].reshape(n, Hs, P), xbc[:, inner:inner + G * N].reshape(n, G, N),
                                 xbc[:, inner + G * N:].reshape(n, G, N), plain.softplus(dt + dt_bias), a_log, D).reshape(n, inner)
        want.append(0.9 * plain.group_rms_norm(y * plain.silu(z), norm_w, ng, 1e-5))
    state_row = Hs * N * P + (taps - 1) * channels
    state = torch.full((6, 2, state_row), float("nan"), device=DEV)
    for s in slots:
        state[s].zero_()
    got = [[] for _ in lens]
    at = [0, 0, 0]
    for step in range(5):
        rows, seq_slot, seq_start, seq_pos0 = [], [], [0], []
        for i in (1, 0, 2):                                            # the step lists the sequences in another order
            n = cuts[i][step]
            rows.append(proj[i][at[i]:at[i] + n])
            seq_slot.append(slots[i]); seq_pos0.append(at[i]); seq_start.append(seq_start[-1] + n)
            if i == 0:                                                  # a padding row between two sequences
                rows.append(torch.full((1, width), float("nan"), dtype=torch.float64))
                seq_slot.append(-1); seq_pos0.append(0); seq_start.append(seq_start[-1] + 1)
        pr = dev(torch.cat(rows))
        T = pr.shape[0]
        ss, st, sp = (dev(torch.tensor(v), torch.int32) for v in (seq_slot, seq_start, seq_pos0))
        xbc = torch.full((T, channels), float("nan"), device=DEV)
        ops.ssd_conv(pr, inner, dev(conv_w), dev(conv_b), state, Hs * N * P, ss, st, sp, xbc, len(seq_slot), max(c[step] for c in cuts))
        y = torch.full((T, inner), float("nan"), device=DEV)
        ops.ssd_scan(xbc, pr, inner + channels, dev(dt_bias), dev(a_log), dev(D), state, ss, st, sp, y, len(seq_slot), Hs, G, N, P)
        out = torch.full((T, inner + 3), float("nan"), device=DEV)
        ops.ssd_gate_norm(y, pr, 0, dev(norm_w), ng, 1e-5, 0.9, out[:, 2:2 + inner], T)
        r = 0
        for i in (1, 0, 2):
            n = cuts[i][step]
            got[i].append(out[r:r + n, 2:2 + inner].cpu())
            at[i] += n
            r += n + (1 if i == 0 else 0)
    for i in range(3):
        close(torch.cat(got[i]), want[i], 3e-5, f"sequence {i}")
    assert torch.isnan(state[[1, 3, 5]]).all()


@pytest.mark.parametrize("d,groups,rows", [(128, 1, 1), (384, 3, 300), (2048, 4, 9), (4096, 8, 3), (4096, 32, 297), (4608, 9, 2), (640, 1, 5)])
def test_gated_norm_with_rows_in_registers(d, groups, rows):
    """The kernel for whole warps' worth of columns, at the edges of its quads a thread, beside the one for any row (which a column
    that is not on 16 bytes asks for): both within float32 rounding of the plain formula, and of one another."""
    from vlrf_b200.csrc import ops
    g = torch.Generator().manual_seed(d + groups)
    y, z, w = torch.randn(rows, d, generator=g), 2.0 * torch.randn(rows, d, generator=g), torch.randn(d, generator=g)
    want = 0.7 * plain.group_rms_norm(y.double() * plain.silu(z.double()), w.double(), groups, 1e-5)
    for off in (8, 9):                                       # 9: the gate's columns do not begin on 16 bytes
        proj = torch.full((rows, d + 12), float("nan"))
        proj[:, off:off + d] = z
        for dtype, tol in ((torch.float32, 2e-6), (torch.bfloat16, 2.0 ** -8)):
            out = torch.full((rows + 1, d + 4), float("nan"), dtype=dtype, device=DEV)
            ops.ssd_gate_norm(dev(y), dev(proj), off, dev(w), groups, 1e-5, 0.7, out[:, :d], rows)
            close(out[:rows, :d].float().cpu(), want, tol, f"gate at {off}")
            assert torch.isnan(out[rows]).all() and torch.isnan(out[:, d:]).all()


@pytest.mark.parametrize("S,d", [(1, 4), (2, 128), (4, 1024), (4, 1000), (5, 2048), (8, 4096), (8, 4100), (9, 256)])
def test_streams_with_rows_in_registers(S, d):
    """Embedding, write and read of rows that the kernels hold in registers (up to 8 streams of 4,096 numbers) and just beyond."""
    from vlrf_b200.csrc import ops
    g = torch.Generator().manual_seed(S * d)
    T = 5
    x, y, w = torch.randn(T, S, d, generator=g), torch.randn(T, d, generator=g), torch.randn(d, generator=g)
    mix, b, a = torch.randn(S, S, generator=g), torch.randn(S, generator=g), torch.randn(S, generator=g)
    want_x = torch.einsum("sj,tsd->tjd", mix.double(), x.double()) + b.double()[None, :, None] * y.double()[:, None]
    want_h = plain.rms_norm(torch.einsum("s,tsd->td", a.double(), want_x), w.double(), 1e-5)
    for dtype, tol in ((torch.float32, 3e-6), (torch.bfloat16, 2.0 ** -8)):
        xd = dev(x.reshape(T, S * d))
        h = torch.full((T + 1, d), float("nan"), dtype=dtype, device=DEV)
        ops.streams_write_read(xd, S, dev(mix), dev(b), dev(y), dev(a), dev(w), 1e-5, h, T)
        close(xd.cpu().reshape(T, S, d), want_x, 3e-6, "streams")
        close(h[:T].float().cpu(), want_h, tol, "read behind the write")
        assert torch.isnan(h[T].float()).all()
        rows = torch.tensor([3, 0, 3], dtype=torch.int32, device=DEV)
        some = torch.full((3, d), float("nan"), dtype=dtype, device=DEV)
        ops.streams_read_norm(xd, S, None, dev(w), 1e-5, some, rows)
        close(some.float().cpu(), plain.rms_norm(want_x.sum(1)[[3, 0, 3]], w.double(), 1e-5), tol, "sum of the streams")
        table = torch.randn(11, d, generator=g).to(dtype)
        e, err = torch.full((3, S * d), float("nan"), device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
        ops.embed_streams(table.to(DEV), torch.tensor([10, 0, 4], dtype=torch.int32, device=DEV), e, S, 1.5, err)
        close(e.cpu().reshape(3, S, d), (1.5 * table.double()[[10, 0, 4]])[:, None].repeat(1, S, 1), 3e-7, "embedding")
        assert int(err.item()) == 0


@pytest.mark.parametrize("Hs,P,N,G", [(4, 64, 64, 1), (8, 64, 64, 2), (3, 20, 16, 3), (10, 132, 32, 2), (2, 128, 128, 1), (5, 4, 128, 1)])
def test_recurrence_in_chunks(Hs, P, N, G):
    """Runs at the edges of the chunks and of their blocks of 16, from zero and from kept states in both copies, a padding row and
    NaN-poisoned neighbours; heads that forget within a token and heads that keep everything.  The chunked kernels may be as far from
    the plain float64 recurrence as the token-by-token kernel is, or within 2^-21 of the largest result: an operand in three
    bfloat16 parts and the six products of parts are good to 2^-23, and a sum's roundings add.  (Measured: 1.3e-7 to 2.0e-7 of the
    largest result, token by token 4.5e-7 to 1.2e-6.)"""
    import types

    from vlrf_b200.csrc import ops
    from vlrf_b200.parts.context import Workspace
    g = torch.Generator().manual_seed(Hs * 1000 + P * 10 + N)
    inner, channels = Hs * P, Hs * P + 2 * G * N
    lens, pos0, slots = [64, 1, 65, 130, 15, 200, 17], [0, 3, 4, 7, 0, 128, 1], [6, 0, 3, 5, 1, 8, 2]
    rand = lambda *shape: torch.randn(*shape, generator=g)   # noqa: E731
    dt_bias, a_log, D = rand(Hs), torch.linspace(-6.0, 2.5, Hs), rand(Hs)
    state_row = Hs * N * P + 8
    kept = {s: rand(Hs, N, P) if p else torch.zeros(Hs, N, P) for s, p in zip(slots, pos0)}
    state = torch.full((10, 2, state_row), float("nan"))
    for s, p in zip(slots, pos0):
        state[s, p & 1, :Hs * N * P] = kept[s].flatten()
    rows, seq_slot, seq_start, seq_pos0, want, ends = [], [], [0], [], [], {}
    for i, (n, p, s) in enumerate(zip(lens, pos0, slots)):
        xbc, dt = rand(n, channels), rand(n, Hs) * 2.0
        x, B, C = (t.double() for t in (xbc[:, :inner].reshape(n, Hs, P), xbc[:, inner:inner + G * N].reshape(n, G, N), xbc[:, inner + G * N:].reshape(n, G, N)))
        step = plain.softplus(dt.double() + dt_bias.double())
        B, C = (t.repeat_interleave(Hs // G, 1) for t in (B, C))
        S, y = kept[s].double().clone(), torch.empty(n, Hs, P, dtype=torch.float64)
        for t in range(n):
            S = torch.exp(-torch.exp(a_log.double()) * step[t])[:, None, None] * S + (step[t][:, None] * B[t])[:, :, None] * x[t][:, None, :]
            y[t] = (S * C[t][:, :, None]).sum(1) + D.double()[:, None] * x[t]
        want.append(y.reshape(n, inner)); ends[s] = S
        rows.append((xbc, dt)); seq_slot.append(s); seq_pos0.append(p); seq_start.append(seq_start[-1] + n)
        if i == 2:                                                      # a padding row between two sequences
            rows.append((torch.full((1, channels), float("nan")), torch.full((1, Hs), float("nan"))))
            seq_slot.append(-1); seq_pos0.append(0); seq_start.append(seq_start[-1] + 1)
    T = seq_start[-1]
    xbc, proj = dev(torch.cat([r[0] for r in rows])), dev(torch.cat([torch.cat([rand(r[1].shape[0], 3), r[1]], 1) for r in rows]))
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)   # noqa: E731
    ctx = types.SimpleNamespace(n_tokens=T, n_seqs=len(seq_slot), seq_slot=i32(seq_slot), seq_start=i32(seq_start), seq_pos0=i32(seq_pos0),
                                max_new=max(lens), ws=Workspace(torch.device(DEV)), act_dtype=torch.bfloat16)
    ctx.max_new = ops.SSD_CHUNKS_MIN_RUN                              # (the rule asks for longer runs than this test's)
    assert ops.ssd_chunks_takes(torch.bfloat16, ctx, Hs, G, N, P, channels, state_row)
    assert not ops.ssd_chunks_takes(torch.float32, ctx, Hs, G, N, P, channels, state_row)
    ctx.max_new = max(lens)
    keep = torch.ones(T, dtype=torch.bool)
    for s, a in zip(seq_slot, seq_start):
        if s < 0:
            keep[a] = False
    want, off = torch.cat(want), {}
    for chunked in (False, True):
        st, y = state.to(DEV), torch.full((T, inner), float("nan"), device=DEV)
        if chunked:
            ops.ssd_chunks(xbc, proj, 3, dev(dt_bias), dev(a_log), dev(D), st, ctx, y, Hs, G, N, P)
        else:
            ops.ssd_scan(xbc, proj, 3, dev(dt_bias), dev(a_log), dev(D), st, ctx.seq_slot, ctx.seq_start, ctx.seq_pos0, y, ctx.n_seqs, Hs, G, N, P,
                         ctx.max_new)
        y, st = y.cpu(), st.cpu()
        assert torch.isnan(y[~keep]).all() and torch.isfinite(y[keep]).all()
        off[chunked] = [float((y[keep].double() - want).norm() / want.norm()), float((y[keep].double() - want).abs().max() / want.abs().max())]
        for s, p, n in zip(slots, pos0, lens):
            close(st[s, (p + n) & 1, :Hs * N * P].reshape(Hs, N, P), ends[s], 1e-5, f"state of slot {s}")
            if n & 1:
                assert torch.equal(st[s, p & 1, :Hs * N * P], state[s, p & 1, :Hs * N * P])
        assert torch.isnan(st[[4, 7, 9]]).all() and torch.isnan(st[:, :, Hs * N * P:]).all()
    print(f"heads {Hs} of {N} x {P}: token by token {off[False]}, in chunks {off[True]}")
    for a, b in zip(off[True], off[False]):
        assert a <= max(1.5 * b, 2.0 ** -21), off


@pytest.mark.parametrize("Hs,P,N,G", [(4, 64, 64, 2), (3, 132, 16, 1), (2, 128, 128, 2)])
@pytest.mark.parametrize("where", ["x", "B", "C", "dt", "decay", "state", "large"])
def test_recurrence_in_chunks_keeps_to_the_past(where, Hs, P, N, G):
    """A NaN or an infinity at one token (or in the kept state, or a decay of nothing at all, or numbers whose products overflow) changes
    no earlier token and gives what token by token gives, finite where that is finite and the same where it is not; the other sequence
    of the step has nothing of it."""
    import types

    from vlrf_b200.csrc import ops
    from vlrf_b200.parts.context import Workspace
    g = torch.Generator().manual_seed(Hs * 1000 + P * 10 + N)
    inner, channels, lens, pos0, slots = Hs * P, Hs * P + 2 * G * N, [150, 70], [4, 3], [1, 0]
    T, state_row = sum(lens), Hs * N * P
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)   # noqa: E731
    ctx = types.SimpleNamespace(n_tokens=T, n_seqs=2, seq_slot=i32(slots), seq_start=i32([0, 150, 220]), seq_pos0=i32(pos0), max_new=150,
                                ws=Workspace(torch.device(DEV)), act_dtype=torch.bfloat16)
    for token, value in ((77, float("nan")), (77, float("inf")), (149, float("-inf")), (0, float("inf"))):
        xbc, dt = torch.randn(T, channels, generator=g), torch.randn(T, Hs, generator=g)
        dt_bias, a_log, D = torch.randn(Hs, generator=g), torch.linspace(-6.0, 1.0, Hs), torch.randn(Hs, generator=g)
        state = torch.randn(2, 2, state_row, generator=g)
        if where == "x":
            xbc[token, P + 2] = value                                      # head 1, column 2
        elif where in "BC":
            xbc[token, inner + (G * N if where == "C" else 0) + 3] = value
        elif where == "dt":
            dt[token, 1] = value
        elif where == "decay":
            a_log[1] = 95.0                                                # exp overflows: every token forgets all before it
        elif where == "state":
            state[slots[0], pos0[0] & 1, N * P + 5] = value                # head 1, column 5
        else:
            xbc[token, P + 2], xbc[token, inner + 3] = 1e30, 1e30              # one row overflows, none comes near it
        proj = dev(torch.cat([torch.randn(T, 3, generator=g), dt], 1))
        got = []
        for chunked in (False, True):
            st, y = state.to(DEV), torch.full((T, inner), 7.0, device=DEV)
            args = (dev(xbc), proj, 3, dev(dt_bias), dev(a_log), dev(D), st)
            if chunked:
                ops.ssd_chunks(*args, ctx, y, Hs, G, N, P)
            else:
                ops.ssd_scan(*args, ctx.seq_slot, ctx.seq_start, ctx.seq_pos0, y, 2, Hs, G, N, P, 150)
            got.append((y.cpu(), st.cpu()))
        for a, b in zip(*got):                                             # token by token, in chunks
            odd = ~torch.isfinite(a)
            assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(a[odd & ~torch.isnan(a)], b[odd & ~torch.isnan(a)])
            keep = ~odd & (a.abs() < 1e6)
            assert float((a[keep] - b[keep]).abs().max() / a[keep].abs().max()) < 1e-5
            assert torch.allclose(a[~odd], b[~odd], rtol=1e-3, atol=1e-4 * float(a[keep].abs().max()))
        if where in ("x", "B", "C", "dt"):
            assert torch.isfinite(got[1][0][:token]).all() and torch.isfinite(got[1][0][150:]).all()


def chunk_step(lens, pos0, slots, Hs, P, N, G, g, extra=0):
    """The inputs of a step of these runs: (arguments of the recurrence, state, context)."""
    import types

    from vlrf_b200.parts.context import Workspace
    T, channels = sum(lens), Hs * P + 2 * G * N
    start = [0]
    for n in lens:
        start.append(start[-1] + n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)   # noqa: E731
    ctx = types.SimpleNamespace(n_tokens=T, n_seqs=len(lens), seq_slot=i32(slots), seq_start=i32(start), seq_pos0=i32(pos0), max_new=max(lens),
                                min_new=min(lens), ws=Workspace(torch.device(DEV)), act_dtype=torch.bfloat16)
    xbc, proj = torch.randn(T, channels, generator=g), torch.randn(T, 3 + Hs, generator=g)
    a_log = torch.linspace(-6.0, 1.0, Hs)
    weights = [dev(torch.randn(Hs, generator=g)), dev(a_log), dev(torch.randn(Hs, generator=g))]
    state = torch.randn(max(slots) + 1, 2, Hs * N * P + extra, generator=g)
    return (dev(xbc), dev(proj), 3, *weights), state, ctx


def test_chunks_in_passes_and_without_scratch(monkeypatch):
    """Scratch for every head, for three of five groups and for one at a time gives the same bits; with no room for it at all the step goes
    token by token."""
    from vlrf_b200.csrc import ops
    Hs, P, N, G = 10, 68, 32, 5
    args, state, ctx = chunk_step([400, 1, 90], [0, 5, 2], [2, 0, 1], Hs, P, N, G, torch.Generator().manual_seed(1))
    slots, marks = ctx.n_tokens // 64 + 3, Hs * 2

    def run(entry):
        st, y = state.to(DEV), torch.full((ctx.n_tokens, Hs * P), float("nan"), device=DEV)
        entry(*args, st, ctx, y, Hs, G, N, P)
        return y.cpu(), st.cpu()
    want = run(ops.ssd_chunks)
    whole = ctx.ws.get("ssd_chunks", 1, 1, torch.float32).untyped_storage().nbytes()
    assert whole == 4 * slots * (Hs * (N * P + 1) + marks)
    for groups in (3, 1):
        monkeypatch.setattr(ops, "SSD_CHUNKS_MAX_BYTES", 4 * slots * (2 * groups * (N * P + 1) + marks) + 3)
        ctx.ws = type(ctx.ws)(torch.device(DEV))
        for a, b in zip(run(ops.ssd_chunks), want):
            assert torch.equal(a, b)
        assert ctx.ws.get("ssd_chunks", 1, 1, torch.float32).untyped_storage().nbytes() <= ops.SSD_CHUNKS_MAX_BYTES
    monkeypatch.setattr(ops, "SSD_CHUNKS_MAX_BYTES", 4 * slots * (2 * (N * P + 1) + marks) - 4)
    assert not ops.ssd_chunks_takes(torch.bfloat16, ctx, Hs, G, N, P, args[0].shape[1], state.shape[2])
    monkeypatch.undo()
    real = torch.empty

    def full(*a, **k):
        if a and isinstance(a[0], int) and a[0] > 100000:
            raise torch.OutOfMemoryError("no room")
        return real(*a, **k)
    ctx.ws = type(ctx.ws)(torch.device(DEV))
    monkeypatch.setattr(torch, "empty", full)
    got = run(ops.ssd_scan_step)
    monkeypatch.undo()
    for a, b in zip(got, want):
        close(a, b, 1e-5, "token by token")
    assert not torch.equal(got[0], want[0])


def test_a_sequence_does_not_see_what_shares_its_step():
    """Single tokens, runs below and at the chunks' least length, and long ones: each has, bit for bit, the results and the state that it has
    in a step of its own, whatever the longest run of the step is."""
    from vlrf_b200.csrc import ops
    Hs, P, N, G = 4, 64, 64, 2
    least = ops.SSD_CHUNKS_MIN_RUN
    lens, pos0, slots = [1, least - 1, least, 2, 1, 700, 65], [9, 0, 2, 3, 0, 7, 128], [3, 0, 6, 2, 5, 1, 4]
    args, state, ctx = chunk_step(lens, pos0, slots, Hs, P, N, G, torch.Generator().manual_seed(3))
    xbc, proj = args[:2]

    def run(some):
        rows = torch.cat([torch.arange(sum(lens[:i]), sum(lens[:i + 1])) for i in some]).to(DEV)
        _, _, c = chunk_step([lens[i] for i in some], [pos0[i] for i in some], [slots[i] for i in some], Hs, P, N, G, torch.Generator())
        st, y = state.to(DEV), torch.full((len(rows), Hs * P), float("nan"), device=DEV)
        ops.ssd_scan_step(xbc[rows], proj[rows], *args[2:], st, c, y, Hs, G, N, P)
        return y.cpu(), st.cpu()
    own = [run([i]) for i in range(len(lens))]
    for some in (range(7), [0, 1, 3, 4, 6], [5, 4], [0, 4], [3, 0], [6, 5, 2, 1]):
        y, st = run(list(some))
        assert torch.isfinite(y).all()
        at = 0
        for i in some:
            assert torch.equal(y[at:at + lens[i]], own[i][0]), (list(some), i)
            assert torch.equal(st[slots[i]], own[i][1][slots[i]]), (list(some), i)
            at += lens[i]


def test_long_runs_in_chunks():
    """Runs at the length from which the library takes chunks, and at the edges of the eight chunks that a state's thread asks for together,
    beside single tokens, from zero and from kept states, through the rule that chooses the kernels; a kept state shows in the last token
    (decays down to e^-0.002 a token).  As far from the float64 recurrence as token by token is, or within 2^-21 of the largest result."""
    from vlrf_b200.csrc import ops
    Hs, P, N, G = 4, 64, 64, 2
    lens, pos0, slots = [383, 1, 384, 512, 513, 1, 1100], [0, 5, 0, 2, 7, 0, 64], [0, 1, 2, 3, 4, 5, 6]
    args, state, ctx = chunk_step(lens, pos0, slots, Hs, P, N, G, torch.Generator().manual_seed(4))
    for i, p in enumerate(pos0):
        if p == 0:
            state[slots[i], 0] = 0.0
    xbc, proj = args[0].cpu().double(), args[1].cpu().double()
    dt_bias, a_log, D = (t.cpu().double() for t in args[3:])
    a_log = a_log.float()                                              # (as the kernel has it)
    want, ends, at, inner = [], [], 0, Hs * P
    for n, p, s in zip(lens, pos0, slots):
        x, B, C = xbc[at:at + n, :inner].reshape(n, Hs, P), xbc[at:at + n, inner:inner + G * N], xbc[at:at + n, inner + G * N:]
        B, C = (t.reshape(n, G, N).repeat_interleave(Hs // G, 1) for t in (B, C))
        step = plain.softplus(proj[at:at + n, 3:] + dt_bias)
        S, y = state[s, p & 1].double().reshape(Hs, N, P).clone(), torch.empty(n, Hs, P, dtype=torch.float64)
        for t in range(n):
            S = torch.exp(-torch.exp(a_log.double()) * step[t])[:, None, None] * S + (step[t][:, None] * B[t])[:, :, None] * x[t][:, None, :]
            y[t] = (S * C[t][:, :, None]).sum(1) + D[:, None] * x[t]
        want.append(y.reshape(n, inner)); ends.append(S); at += n
    off = {}
    for chunked in (False, True):
        st, y = state.to(DEV), torch.full((at, inner), float("nan"), device=DEV)
        if chunked:
            assert ops.ssd_chunks_takes(torch.bfloat16, ctx, Hs, G, N, P, args[0].shape[1], state.shape[2])
            ops.ssd_scan_step(*args, st, ctx, y, Hs, G, N, P)
        else:
            ops.ssd_scan(*args, st, ctx.seq_slot, ctx.seq_start, ctx.seq_pos0, y, ctx.n_seqs, Hs, G, N, P, ctx.max_new)
        y, st, i, off[chunked] = y.cpu().double(), st.cpu(), 0, []
        for n, p, s, w, e in zip(lens, pos0, slots, want, ends):
            got = y[i:i + n]
            off[chunked].append(float((got - w).norm() / w.norm()))
            assert float((got[-1] - w[-1]).abs().max() / w.abs().max()) < 1e-5, (n, "last token")
            close(st[s, (p + n) & 1].reshape(Hs, N, P), e, 1e-5, f"state of slot {s}")
            i += n
    assert all(a <= max(1.5 * b, 2.0 ** -21) for a, b in zip(off[True], off[False])), off


def test_tokens_one_by_one_with_nothing_between():
    """The one-token kernel launched again and again, each launch reading the state that the one just ahead of it writes (it may begin while
    that one still runs), against the float64 recurrence."""
    from vlrf_b200.csrc import ops
    Hs, P, N, G, T = 4, 64, 64, 2, 40
    inner = Hs * P
    args, state, ctx = chunk_step([1, 1, 1], [0, 3, 4], [2, 0, 1], Hs, P, N, G, torch.Generator().manual_seed(8))
    g = torch.Generator().manual_seed(9)
    xbc, proj = torch.randn(T, 3, inner + 2 * G * N, generator=g), torch.randn(T, 3, 3 + Hs, generator=g)
    xd, pd, y = dev(xbc), dev(proj), torch.empty(T, 3, inner, device=DEV)
    pos = torch.tensor([[0, 3, 4]] * T, dtype=torch.int32) + torch.arange(T, dtype=torch.int32)[:, None]
    pos = pos.to(DEV)
    import types
    steps = [types.SimpleNamespace(**{**vars(ctx), "seq_pos0": pos[t]}) for t in range(T)]
    for _ in range(3):                                                 # (and again: what a run left must not show)
        st = state.to(DEV)
        torch.cuda.synchronize()
        for t in range(T):
            ops.ssd_step(xd[t], pd[t], *args[2:], st, steps[t], y[t], Hs, G, N, P)
        dt_bias, a_log, D = (t.cpu().double() for t in args[3:])
        for i, (slot, p0) in enumerate(((2, 0), (0, 3), (1, 4))):
            S, want = state[slot, p0 & 1].double().reshape(Hs, N, P), []
            for t in range(T):
                x, B, C = xbc[t, i, :inner].double().reshape(Hs, P), xbc[t, i, inner:inner + G * N].double(), xbc[t, i, inner + G * N:].double()
                B, C = (v.reshape(G, N).repeat_interleave(Hs // G, 0) for v in (B, C))
                step = plain.softplus(proj[t, i, 3:].double() + dt_bias)
                S = torch.exp(-torch.exp(a_log) * step)[:, None, None] * S + (step[:, None] * B)[:, :, None] * x[:, None, :]
                want.append(((S * C[:, :, None]).sum(1) + D[:, None] * x).reshape(inner))
            close(y[:, i], torch.stack(want), 1e-5, f"sequence {i}")
            close(st[slot, (p0 + T) & 1].reshape(Hs, N, P), S, 1e-5, f"state {i}")


@pytest.mark.parametrize("which", ["xbc", "state", "y"])
def test_recurrence_of_rows_beside_16_bytes(which):
    """Rows, states or results that do not begin on 16 bytes are taken, as token by token takes them, in decode and in prompt steps."""
    from vlrf_b200.csrc import ops
    Hs, P, N, G = 4, 64, 64, 2
    for lens in ([1, 1], [400, 1, 30]):
        args, state, ctx = chunk_step(lens, [0, 3, 4][:len(lens)], [2, 0, 1][:len(lens)], Hs, P, N, G, torch.Generator().manual_seed(5))

        def beside(t, name):
            if name != which:
                return t.to(DEV)
            flat = torch.empty(t.numel() + 1, device=DEV)[1:]
            return flat.copy_(t.flatten()).view(t.shape)
        results = []
        for shifted in (False, True):
            place = beside if shifted else lambda t, name: t.to(DEV)
            st, y = place(state, "state"), place(torch.zeros(ctx.n_tokens, Hs * P), "y")
            ops.ssd_scan_step(place(args[0], "xbc"), *args[1:], st, ctx, y, Hs, G, N, P)
            results.append((y.cpu(), st.cpu()))
        for a, b in zip(*results):
            close(b, a, 1e-5, which)


@pytest.mark.parametrize("taps", [1, 2, 4, 5])
def test_convolution_over_runs(taps):
    """Runs at the edges of a thread's 16 tokens, from zero and from kept inputs, with the number of taps known when compiling and not; a
    padding row.  Sums of at most five products and x·sigmoid(x) in float32."""
    from vlrf_b200.csrc import ops
    g = torch.Generator().manual_seed(taps)
    channels, ld, off = 130, 200, 7
    lens, pos0, slots = [1, 16, 17, 33, 1, 2], [5, 0, 4, 0, 0, 2], [2, 0, 4, 1, -1, 3]
    w, bias = torch.randn(channels, taps, generator=g), torch.randn(channels, generator=g)
    for some in ((0, 1, 4, 5), (0, 1, 2, 3, 4, 5)):            # all runs at most 16 tokens, or not
        n = [lens[i] for i in some]
        start = torch.tensor([0] + list(torch.tensor(n).cumsum(0)), dtype=torch.int32)
        proj = torch.randn(int(start[-1]), ld, generator=g)
        row = (taps - 1) * channels + 3
        state = torch.randn(5, 2, row, generator=g)
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)   # noqa: E731
        st, out = state.to(DEV), torch.full((int(start[-1]), channels), float("nan"), device=DEV)
        pos = [pos0[i] for i in some]
        ops.ssd_conv(dev(proj), off, dev(w), dev(bias), st, 3, i32([slots[i] for i in some]), start.to(DEV), i32(pos), out, len(some), max(n))
        for j, i in enumerate(some):
            a, b = int(start[j]), int(start[j + 1])
            if slots[i] < 0:
                assert torch.isnan(out[a:b]).all()
                continue
            kept = state[slots[i], pos0[i] & 1, 3:].reshape(taps - 1, channels).double()
            u = torch.cat([kept, proj[a:b, off:off + channels].double()])
            want = torch.stack([(u[t:t + taps] * w.double().T).sum(0) + bias.double() for t in range(b - a)])
            close(out[a:b], want * torch.sigmoid(want), 3e-6, f"run {i}")
            if taps > 1:
                close(st[slots[i], (pos0[i] + b - a) & 1, 3:], u[len(u) - (taps - 1):].reshape(-1), 1e-7, f"kept inputs of run {i}")


@pytest.mark.parametrize("H,G,dk,dv,rot,interleaved,maps,norm", [
    (16, 4, 64, 96, 32, False, 1, None), (3, 1, 12, 4, 8, False, 1, None), (2, 2, 128, 128, 128, False, 2, None), (5, 5, 20, 8, 12, True, 1, None),
    (4, 2, 8, 4, 0, False, 1, None), (3, 3, 16, 12, 4, True, 2, None), (17, 3, 64, 64, 32, False, 1, "head"), (2, 1, 96, 20, 0, True, 1, "head")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rotation_and_append_of_aligned_rows(H, G, dk, dv, rot, interleaved, maps, norm, dtype):
    """Rows on 16-byte boundaries (quads of entries a thread) against the same rows one number further (pairs): queries, keys and
    values, with a padding row, a token whose block is missing, and a layer that keeps no keys.  Both work out an entry from the
    same two products; which of them is fused into the sum may differ, by a rounding of float32, and then of bfloat16."""
    from vlrf_b200.csrc import ops
    g = torch.Generator().manual_seed(H * 100 + dk)
    T, nq, nk = 5, H * maps * dk, G * maps * dk
    rows = torch.randn(T, nq + nk + G * dv, generator=g)
    freq = dev(torch.rand(rot // 2, generator=g)) if rot else None
    slots, pos = dev(torch.tensor([0, 1, -1, 1, 0]), torch.int32), dev(torch.tensor([3, 64, 5, 1000, 127]), torch.int32)
    table = dev(torch.tensor([[2, 0], [3, 1]] if T else []), torch.int32)
    weights = dict(norm=norm, q_norm=dev(torch.randn(dk, generator=g)), k_norm=dev(torch.randn(dk, generator=g)), eps=1e-5) if norm else {}
    got = []
    for shift in (4, 3):
        wide = torch.full((T, rows.shape[1] + 8 + (-rows.shape[1]) % 4), float("nan"))
        wide[:, shift:shift + rows.shape[1]] = rows
        wide = dev(wide)
        for write in (True, False):
            q = torch.full((T, nq), 7.0, dtype=dtype, device=DEV)
            k, v = torch.full((4, G, 64, maps * dk), 7.0, dtype=dtype, device=DEV), torch.full((4, G, 64, dv), 7.0, dtype=dtype, device=DEV)
            err = torch.zeros(1, dtype=torch.int32, device=DEV)
            ops.qkv_rope_append(wide[:, shift:shift + rows.shape[1]], 0, nq, nq + nk, freq, rot, q, k, v, table, slots, pos, T, H, G, dk, dv, write,
                                err, interleaved=interleaved, magnitude=1.25, maps=maps, **weights)
            assert (int(err.item()) != 0) == write                      # position 1,000 has no block
            got.append([t.double().cpu() for t in (q, k, v)])
    for a, b in zip(got[:2], got[2:]):
        for x, y in zip(a, b):
            assert float((x - y).abs().max()) <= (1e-6 if dtype == torch.float32 else 2.0 ** -8) * max(1.0, float(y.abs().max()))
            assert torch.equal(x == 7.0, y == 7.0)
    assert (got[0][0][2] == 7.0).all() and (got[1][1] == 7.0).all() and (got[0][1] != 7.0).any()


@pytest.mark.parametrize("splits", [2, 8, 9, 32, 33, 40])
def test_parts_of_a_context_meet(monkeypatch, splits):
    """A decode step's contexts cut into numbers of parts around the eight that the merge asks for together and the 32 that a warp holds, parts
    without a visible key among them, against the whole softmax in float64 (weights and results are rounded to bfloat16)."""
    from vlrf_b200.csrc import ops
    monkeypatch.setattr(ops, "window_decode_splits", lambda *a, **k: splits)
    g = torch.Generator().manual_seed(splits)
    H, G, dk, dv = 8, 2, 32, 136 - 8
    lens = [700, 65, 1]
    T = sum(lens)
    rd = lambda *shape: torch.randn(*shape, generator=g).bfloat16().double()   # noqa: E731
    q, k, v = rd(T, H, dk), rd(T, G, dk), rd(T, G, dv)
    positions, slot_of = [p for n in lens for p in range(n)], [i for i, n in enumerate(lens) for _ in range(n)]
    want, start = [], 0
    for n in lens:
        want.append(plain.window_attention(q[start:start + n], k[start:start + n], v[start:start + n], 0.3, 0)[-1])
        start += n
    got, _ = run_attention(q.float(), k.float(), v.float(), positions, slot_of, lens, G, 0.3, 0, None, torch.bfloat16, 0.6, 1, None)
    close(got, 0.6 * torch.stack(want), 2e-2, f"{splits} parts")


@pytest.mark.parametrize("Hs,P,N,G", [(4, 64, 64, 2), (3, 4, 16, 3), (2, 132, 34, 1), (32, 128, 128, 8), (2, 20, 512, 1)])
def test_recurrence_of_one_token(Hs, P, N, G):
    """The decode step's kernel from both copies of the state, a padding row, states of rows and columns beside its runs, against the
    float64 step: a state is one product and one sum of float32 away, a result a sum of up to 512 of them over 256 threads."""
    import types

    from vlrf_b200.csrc import ops
    g = torch.Generator().manual_seed(Hs * 1000 + P * 10 + N)
    inner, channels, state_row = Hs * P, Hs * P + 2 * G * N, Hs * N * P + 8 + (-Hs * N * P) % 4
    pos0, slots = [0, 3, 4, 7, 0, 128], [6, 0, 3, 5, -1, 2]
    T = len(slots)
    xbc, dt = torch.randn(T, channels, generator=g), torch.randn(T, Hs, generator=g) * 2.0
    dt_bias, a_log, D = torch.randn(Hs, generator=g), torch.linspace(-6.0, 2.5, Hs), torch.randn(Hs, generator=g)
    state = torch.full((8, 2, state_row), float("nan"))
    for s, p in zip(slots, pos0):
        if s >= 0:
            state[s, p & 1, :Hs * N * P] = torch.randn(Hs * N * P, generator=g)
    proj = dev(torch.cat([torch.randn(T, 3, generator=g), dt], 1))
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)   # noqa: E731
    ctx = types.SimpleNamespace(n_tokens=T, n_seqs=T, seq_slot=i32(slots), seq_start=i32(list(range(T + 1))), seq_pos0=i32(pos0), max_new=1,
                                act_dtype=torch.bfloat16)
    assert ops.ssd_step_takes(torch.bfloat16, ctx, Hs, G, N, P, channels, state_row)
    assert not ops.ssd_step_takes(torch.float32, ctx, Hs, G, N, P, channels, state_row)
    st, y = state.to(DEV), torch.full((T, inner), float("nan"), device=DEV)
    ops.ssd_scan_step(dev(xbc), proj, 3, dev(dt_bias), dev(a_log), dev(D), st, ctx, y, Hs, G, N, P)
    for t, (s, p) in enumerate(zip(slots, pos0)):
        if s < 0:
            assert torch.isnan(y[t]).all()
            continue
        x, B, C = xbc[t, :inner].double().reshape(Hs, P), xbc[t, inner:inner + G * N].double().reshape(G, N), xbc[t, inner + G * N:].double().reshape(G, N)
        B, C = (b.repeat_interleave(Hs // G, 0) for b in (B, C))
        step = plain.softplus(dt[t].double() + dt_bias.double())
        S = state[s, p & 1, :Hs * N * P].double().reshape(Hs, N, P)
        S = torch.exp(-torch.exp(a_log.double()) * step)[:, None, None] * S + (step[:, None] * B)[:, :, None] * x[:, None, :]
        close(st[s, (p + 1) & 1, :Hs * N * P].reshape(Hs, N, P), S, 1e-6, f"state of slot {s}")
        close(y[t].reshape(Hs, P), (S * C[:, :, None]).sum(1) + D.double()[:, None] * x, 3e-6, f"result of slot {s}")
        assert torch.equal(st[s, p & 1].cpu().nan_to_num(7.0), state[s, p & 1].nan_to_num(7.0))
