"""The chunked form of the recurrence scan (b2_channel_scan_ws) against fp64 and against the token-by-token scan it stands in for:
portions around a chunk's edge, several sequences with and without context, padding and stateless sequences, head sizes with
remainders, grouped keys, decays of one, of zero and so strong that a chunk's product underflows.

Tolerance: both forms sum dk + (tokens that still count) products in fp32, so their error is a small multiple of 2^-24 of the sums of
absolute values; the chunked one may be twice the other's (other orders) and both stay below 2e-6 of the result's norm, the delta
correction on unit keys included."""
import math

import pytest
import torch

from b200attn import _lib, ops

pytestmark = pytest.mark.gpu


def _inputs(cuda, lens, H, G, dk, dv, per_channel, delta, decay, seed):
    g = torch.Generator(device=cuda).manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda)           # noqa: E731
    uni = lambda *s: torch.rand(*s, generator=g, device=cuda)            # noqa: E731
    T = sum(lens)
    q, k, v = rnd(T, G, dk), rnd(T, G, dk), rnd(T, H, dv)
    if delta:
        q, k = (x / (x.square().sum(-1, keepdim=True) + 1e-6).sqrt() for x in (q, k))
    wide = H * dk if per_channel else H
    dec = {"mild": 1.0 - 0.1 * uni(T, wide), "one": torch.ones(T, wide, device=cuda), "strong": torch.exp(-20.0 * uni(T, wide)),
           "zero": (uni(T, wide) > 0.1).float() * 0.97}[decay].contiguous()
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], 1).contiguous()
    beta = torch.sigmoid(rnd(T, H)) if delta else None
    state = rnd(len(lens) + 1, H, dk, dv)
    return qkv, beta, dec, state


def _reference(qkv, beta, dec, state, lens, ctx, slots, H, G, dk, dv):
    T = qkv.shape[0]
    x = qkv.double()
    q = x[:, :G * dk].view(T, G, dk).repeat_interleave(H // G, 1)
    k = x[:, G * dk:2 * G * dk].view(T, G, dk).repeat_interleave(H // G, 1)
    v = x[:, 2 * G * dk:].view(T, H, dv)
    d = dec.double().view(T, H, -1)
    out, st = torch.zeros(T, H, dv, dtype=torch.float64, device=qkv.device), state.double().clone()
    at = 0
    for n, c, s in zip(lens, ctx, slots):
        if c >= 0:
            S = st[s].clone() if s >= 0 and c > 0 else torch.zeros(H, dk, dv, dtype=torch.float64, device=qkv.device)
            for t in range(at, at + n):
                S = S * d[t][..., None]
                u = v[t] if beta is None else beta[t].double()[:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
                S = S + k[t][..., None] * u[:, None, :]
                out[t] = torch.einsum("hkv,hk->hv", S, q[t])
            if s >= 0:
                st[s] = S
        at += n
    return out, st


@pytest.mark.parametrize("delta,per_channel", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("lens,ctx,slots,H,G,dk,dv,decay", [
    ([200], [0], [0], 2, 2, 128, 128, "mild"),
    ([31, 32, 33], [0, 7, 3], [0, 1, 2], 3, 3, 64, 20, "mild"),
    ([63, 64, 65, 129], [5, 0, 9, 2], [3, 0, 1, 2], 4, 2, 128, 48, "mild"),
    ([1, 300, 2], [40, 0, 6], [1, 0, 2], 2, 1, 96, 16, "mild"),
    ([100, 50], [-1, 4], [0, 1], 2, 2, 32, 32, "mild"),                  # a padding sequence
    ([90, 70], [3, 0], [-1, 1], 2, 2, 20, 36, "one"),                    # a sequence without state; sizes with remainders
    ([257], [8], [1], 2, 2, 128, 64, "strong"),                          # products of a chunk far below the smallest float
    ([140], [8], [0], 3, 3, 4, 4, "zero"),
    # chains of eight to thirty-three chunks of 64 or 128 tokens, and a short one beside a long one: eight or sixteen loads of a state in flight
    ([576], [3], [0], 2, 2, 32, 32, "mild"),
    ([1151], [0], [0], 2, 1, 20, 36, "mild"),
    ([2100], [5], [0], 2, 2, 32, 32, "mild"),
    ([1500, 40], [0, 7], [1, 0], 2, 2, 64, 16, "mild"),
])
def test_chunked_scan(cuda, lens, ctx, slots, H, G, dk, dv, decay, delta, per_channel):
    qkv, beta, dec, state = _inputs(cuda, lens, H, G, dk, dv, per_channel, delta, decay, seed=len(lens) * 100 + dk + dv)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    T, cu = qkv.shape[0], [0]
    for n in lens:
        cu.append(cu[-1] + n)
    batch = ops.SeqBatch(i32(cu), i32(ctx), None, i32(slots), len(lens), T)
    lib = _lib.load()
    st_new, st_old = state.clone(), state.clone()
    new, old = torch.zeros(T, H, dv, device=cuda), torch.zeros(T, H, dv, device=cuda)
    ws = torch.empty(1 << 25, device=cuda)               # enough for every case: the chunked form, though most are too short to gain by it
    args = lambda st, o: (qkv.data_ptr(), beta.data_ptr() if delta else None, dec.data_ptr(), T, H, G, dk, dv, int(per_channel),  # noqa: E731
                          int(delta), batch.cu_q.data_ptr(), batch.ctx_start.data_ptr(), batch.state_slots.data_ptr(), len(lens),
                          st.data_ptr(), o.data_ptr())
    stream = torch.cuda.current_stream().cuda_stream
    _lib.check(lib.b2_channel_scan_ws(*args(st_new, new), ws.data_ptr(), ws.numel(), stream))
    _lib.check(lib.b2_channel_scan(*args(st_old, old), stream))
    ref, st_ref = _reference(qkv, beta, dec, state, lens, ctx, slots, H, G, dk, dv)
    rows = torch.cat([torch.arange(cu[i], cu[i + 1], device=cuda) for i in range(len(lens)) if ctx[i] >= 0])
    for a, b, r in ((new[rows], old[rows], ref[rows]), (st_new, st_old, st_ref)):
        e_new, e_old = (float((x.double() - r).norm() / r.norm()) for x in (a, b))
        assert e_new < 2e-6 and e_new <= 2.0 * e_old + 1e-7, (e_new, e_old)


@pytest.mark.parametrize("delta,per_channel", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("lens,H,G,dk,dv", [
    ([127, 128, 129, 256, 1], 16, 16, 128, 128),                         # edges of a chunk of 128 tokens
    ([2100], 16, 4, 64, 136),                                            # more items than SMs; two blocks of columns, the second of eight
    ([9] * 40 + [300] + [2] * 30, 2, 2, 68, 12),                         # more sequences than lanes; one feature past a slice
    ([520, 33], 8, 8, 124, 260),
])
def test_chunked_scan_sizes(cuda, lens, H, G, dk, dv, delta, per_channel):
    """Sizes at which the kernels on the tensor cores go on to another item, block or slice; the bound is test_chunked_scan's."""
    n, T = len(lens), sum(lens)
    qkv, beta, dec, state = _inputs(cuda, lens, H, G, dk, dv, per_channel, delta, "mild", seed=T + dk)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    cu, ctx, slots = [0], [(5 * i) % 3 for i in range(n)], list(range(n))
    for m in lens:
        cu.append(cu[-1] + m)
    st, o, ws = state.clone(), torch.zeros(T, H, dv, device=cuda), torch.empty(1 << 27, device=cuda)
    keep = i32(cu), i32(ctx), i32(slots)
    _lib.check(_lib.load().b2_channel_scan_ws(qkv.data_ptr(), beta.data_ptr() if delta else None, dec.data_ptr(), T, H, G, dk, dv, int(per_channel),
                                              int(delta), *(x.data_ptr() for x in keep), n, st.data_ptr(), o.data_ptr(), ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream))
    ref, st_ref = _reference(qkv, beta, dec, state, lens, ctx, slots, H, G, dk, dv)
    assert float((o.double() - ref).norm() / ref.norm()) < 2e-6 and float((st.double() - st_ref).norm() / st_ref.norm()) < 2e-6


@pytest.mark.parametrize("delta,per_channel", [(False, False), (True, False), (False, True), (True, True)])
def test_error_of_chunks_against_tokens(cuda, delta, per_channel):
    """Both forms' errors of the outputs against 64 bits, over sizes and seeds.  Both round a sum of dk products, then a sum over the tokens that count:
    with a result's rounding of 2^-24 each, and no chain of more than 16 additions, the chunks' sums of sums are no worse than the tokens'
    trees, which they beat by measurement (0.81 to 0.94 on average); chains over all of dk are 1.1 to 1.2."""
    ratios = []
    for dk, dv, T in ((128, 128, 600), (96, 80, 500), (64, 128, 700)):
        for seed in (1, 2):
            H = 8
            qkv, beta, dec, state = _inputs(cuda, [T], H, H, dk, dv, per_channel, delta, "mild", seed=seed)
            i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
            keep, lib, ws = (i32([0, T]), i32([7]), i32([0])), _lib.load(), torch.empty(1 << 25, device=cuda)
            ref, _ = _reference(qkv, beta, dec, state, [T], [7], [0], H, H, dk, dv)
            args = lambda st, o: (qkv.data_ptr(), beta.data_ptr() if delta else None, dec.data_ptr(), T, H, H, dk, dv, int(per_channel), int(delta),  # noqa: E731
                                  *(x.data_ptr() for x in keep), 1, st.data_ptr(), o.data_ptr())
            outs = [torch.zeros(T, H, dv, device=cuda) for _ in range(2)]
            stream = torch.cuda.current_stream().cuda_stream
            _lib.check(lib.b2_channel_scan_ws(*args(state.clone(), outs[0]), ws.data_ptr(), ws.numel(), stream))
            _lib.check(lib.b2_channel_scan(*args(state.clone(), outs[1]), stream))
            e = [float((o.double() - ref).norm()) for o in outs]
            ratios.append(e[0] / e[1])
    mean = math.exp(sum(map(math.log, ratios)) / len(ratios))
    assert mean < 1.0 and max(ratios) < 1.05, ratios


@pytest.mark.parametrize("delta,per_channel", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("lens", [[700, 3500, 3, 900], [5103], [40] * 60 + [2800]])
def test_long_batches_go_through_the_scratch_in_pieces(cuda, lens, delta, per_channel):
    """Scratch has a limit, past which a batch is taken piece by piece: sequences that a border cuts, one that goes over several pieces, without
    context, with it, without a slot.  Heads are independent, so 64 of them in pieces give the bits of four at a time, which fit at once."""
    H, dk, dv, n, T = 64, 128, 128, len(lens), sum(lens)
    qkv, beta, dec, state = _inputs(cuda, lens, H, H, dk, dv, per_channel, delta, "mild", seed=n)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    cu, ctx, slots = [0], [(7 * i) % 3 for i in range(n)], [-1 if i % 5 == 2 else n - i for i in range(n)]
    for m in lens:
        cu.append(cu[-1] + m)
    keep, lib = (i32(cu), i32(ctx), i32(slots)), _lib.load()
    ws = torch.empty(1 << 27, device=cuda)               # the limit

    def scan(h0, h1):
        cols = [slice((p * H + h0) * dk, (p * H + h1) * dk) for p in range(3)]
        x = torch.cat([qkv[:, c] for c in cols], 1).contiguous()
        b = beta[:, h0:h1].contiguous() if delta else None
        d = dec.view(T, H, -1)[:, h0:h1].reshape(T, -1).contiguous()
        st, o = state[:, h0:h1].clone(), torch.zeros(T, h1 - h0, dv, device=cuda)
        _lib.check(lib.b2_channel_scan_ws(x.data_ptr(), b.data_ptr() if delta else None, d.data_ptr(), T, h1 - h0, h1 - h0, dk, dv, int(per_channel),
                                          int(delta), *(t.data_ptr() for t in keep), n, st.data_ptr(), o.data_ptr(), ws.data_ptr(), ws.numel(),
                                          torch.cuda.current_stream().cuda_stream))
        return o, st

    out, st = scan(0, H)
    for h in range(0, H, 4):
        o, s = scan(h, h + 4)
        assert torch.equal(out[:, h:h + 4], o) and torch.equal(st[:, h:h + 4], s), h


def test_chunked_scan_leaves_short_portions_to_the_token_scan():
    lib = _lib.load()
    for per_channel in (0, 1):
        for delta in (0, 1):
            assert lib.b2_channel_scan_workspace(4096, 1, 16, 128, 128, per_channel, delta) > 0
            assert lib.b2_channel_scan_workspace(1536, 64, 16, 128, 128, per_channel, delta) == 0
    assert lib.b2_channel_scan_workspace(64, 64, 16, 128, 128, 0, 1) == 0
    assert lib.b2_channel_scan_workspace(4096, 1, 16, 256, 128, 0, 1) == 0
    assert lib.b2_channel_scan_workspace(4096, 1, 16, 126, 128, 0, 1) == 0
    assert lib.b2_channel_scan_workspace(0, 1, 16, 128, 128, 0, 1) == 0


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("delta,per_channel", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("at", [1, 5, 31, 34, 63, 64, 100])
def test_nothing_runs_backwards(cuda, at, delta, per_channel, bad):
    """An infinity or NaN in one token's query, key, value, decay or beta: the tokens before it are bit-equal to the same call without it,
    and so are all tokens but its own where only its query is bad, and the other heads'."""
    H, G, dk, dv, T = 2, 2, 64, 32, 130
    qkv, beta, dec, state = _inputs(cuda, [T], H, G, dk, dv, per_channel, delta, "mild", seed=at)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    cu, ctx, slot = i32([0, T]), i32([5]), i32([0])
    lib = _lib.load()
    ws = torch.empty(1 << 22, device=cuda)

    def scan(x, b, d):
        st, o = state.clone(), torch.zeros(T, H, dv, device=cuda)
        _lib.check(lib.b2_channel_scan_ws(x.data_ptr(), b.data_ptr() if delta else None, d.data_ptr(), T, H, G, dk, dv, int(per_channel),
                                          int(delta), cu.data_ptr(), ctx.data_ptr(), slot.data_ptr(), 1, st.data_ptr(), o.data_ptr(),
                                          ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream))
        return o

    good = scan(qkv, beta, dec)
    for what in ("q", "k", "v", "decay") + (("beta",) if delta else ()):
        x, b, d = qkv.clone(), beta.clone() if delta else None, dec.clone()
        if what == "decay":
            d[at, 0] = bad
        elif what == "beta":
            b[at, 0] = bad
        else:
            x[at, {"q": 3, "k": G * dk + 3, "v": 2 * G * dk + 3}[what]] = bad
        out = scan(x, b, d)
        assert torch.equal(out[:at], good[:at]) and torch.equal(out[:, 1], good[:, 1]), what
        assert what in ("decay", "beta") or not bool(torch.isfinite(out[at, 0]).all()), what
        if what == "q":
            assert torch.equal(out[at + 1:], good[at + 1:])


def _scan(x, b, d, state, lens, ctx, slots, H, dk, dv, per_channel, delta):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=x.device)      # noqa: E731
    cu = [0]
    for m in lens:
        cu.append(cu[-1] + m)
    keep, st, o = (i32(cu), i32(ctx), i32(slots)), state.clone(), torch.zeros(cu[-1], H, dv, device=x.device)
    ws = torch.empty(1 << 27, device=x.device)
    _lib.check(_lib.load().b2_channel_scan_ws(x.data_ptr(), b.data_ptr() if delta else None, d.data_ptr(), cu[-1], H, H, dk, dv, int(per_channel), int(delta),
                                              *(t.data_ptr() for t in keep), len(lens), st.data_ptr(), o.data_ptr(), ws.data_ptr(), ws.numel(),
                                              torch.cuda.current_stream().cuda_stream))
    return o, st


@pytest.mark.parametrize("bad", [float("nan"), float("inf"), 3.4e38])
@pytest.mark.parametrize("delta,per_channel", [(False, False), (True, False), (False, True), (True, True)])
def test_nothing_runs_backwards_across_items(cuda, delta, per_channel, bad):
    """The same where a CTA goes on to other items after one with a bad value, with a second block of columns, two slices of features, a sequence
    that starts fresh behind, and bad values in several chunks, the last column among them: no earlier token, no other head, no other sequence and
    (a bad value) no other column gets another bit.  3.4e38 is finite, but rounds to an infinity in bf16."""
    H, dk, dv, lens, ctx, slots = 16, 128, 136, [2100, 700], [9, 0], [0, 1]
    qkv, beta, dec, state = _inputs(cuda, lens, H, H, dk, dv, per_channel, delta, "mild", seed=3)
    if not delta:
        qkv[:, :2 * H * dk] *= 0.05                      # 3.4e38 stays finite in the results
    run = lambda x, b, d: _scan(x, b, d, state, lens, ctx, slots, H, dk, dv, per_channel, delta)     # noqa: E731
    good, st_good = run(qkv, beta, dec)
    plants = ((200, 3, 135), (1029, 3, 7), (1029, 11, 130), (1090, 11, 135))             # token, head, column
    for what in ("v",) if bad == 3.4e38 else ("q", "k", "v", "decay") + (("beta",) if delta else ()):
        x, b, d = qkv.clone(), beta.clone() if delta else None, dec.clone()
        for t, h, c in plants:
            if what == "decay":
                d[t, (h * dk + c % dk) if per_channel else h] = bad
            elif what == "beta":
                b[t, h] = bad
            else:
                x[t, {"q": h * dk + c % dk, "k": (H + h) * dk + c % dk, "v": 2 * H * dk + h * dv + c}[what]] = bad
        out, st = run(x, b, d)
        clean = [h for h in range(H) if h not in (3, 11)]
        assert torch.equal(out[:, clean], good[:, clean]) and torch.equal(out[2100:], good[2100:]) and torch.equal(st[1], st_good[1]), what
        assert torch.equal(st[0][clean], st_good[0][clean]), what
        assert torch.equal(out[:200, 3], good[:200, 3]) and torch.equal(out[:1029, 11], good[:1029, 11]), what
        if what == "q":
            rest = [t for t in range(2100) if t not in (200, 1029, 1090)]
            assert torch.equal(out[rest], good[rest]) and torch.equal(st, st_good)
        if what == "v":
            for h, cols in ((3, (7, 135)), (11, (130, 135))):
                rest = [c for c in range(dv) if c not in cols]
                assert torch.equal(out[:, h][:, rest], good[:, h][:, rest]) and torch.equal(st[0, h][:, rest], st_good[0, h][:, rest])
            assert torch.equal(out[:1029, 3, 7], good[:1029, 3, 7]) and torch.equal(out[:1090, 11, 135], good[:1090, 11, 135])
            if bad == 3.4e38:
                ref, st_ref = _reference(x, b, d, state, lens, ctx, slots, H, H, dk, dv)
                for a, r in ((out[200:, 3, 135], ref[200:, 3, 135]), (out[1029:, 11, 130], ref[1029:, 11, 130]), (st[0, 3, :, 7], st_ref[0, 3, :, 7])):
                    assert bool(torch.isfinite(a).all()) and float((a.double() - r).norm() / r.norm()) < 4e-6


@pytest.mark.parametrize("delta,per_channel", [(False, False), (True, False), (False, True), (True, True)])
def test_infinities_stay_infinities(cuda, delta, per_channel):
    """A value that is an infinity gives infinities of P's sign in its column's outputs of the same chunk (with the delta rule at its own token; behind
    it different signs meet) and of the key's sign in the state; an infinity in the state those of the query's sign."""
    H, dk, dv, T = 2, 64, 32, 64
    qkv, beta, dec, state = _inputs(cuda, [T], H, H, dk, dv, per_channel, delta, "mild", seed=8)
    run = lambda x, s: _scan(x, beta, dec, s, [T], [4], [0], H, dk, dv, per_channel, delta)      # noqa: E731
    inf = float("inf")
    at = T - 1 if delta else 40
    x = qkv.clone()
    x[at, 2 * H * dk + 5] = inf
    out, st = run(x, state)
    q, k, d = (t.double() for t in (qkv[:, :dk], qkv[:, H * dk:(H + 1) * dk], dec.view(T, H, -1)[:, 0]))
    ratio = torch.cat([torch.ones_like(d[:1]), torch.cumprod(d[at + 1:], 0)])
    p = (q[at:] * ratio * k[at]).sum(-1)
    assert bool((p.abs() > 1e-3).sum() > (T - at) // 2)
    for t in range(at, T):
        if abs(float(p[t - at])) > 1e-3:
            assert float(out[t, 0, 5]) == math.copysign(inf, float(p[t - at])), t
    assert torch.equal(st[0, 0, :, 5], torch.copysign(torch.full((dk,), inf, device=cuda), k[at].float()))
    assert bool(torch.isfinite(out[:at]).all()) and bool(torch.isfinite(out[:, 1]).all())
    if not delta:
        s = state.clone()
        s[0, 0, 3, 5] = inf
        out, st = run(qkv, s)
        assert torch.equal(out[:, 0, 5], torch.copysign(torch.full((T,), inf, device=cuda), qkv[:, 3])) and float(st[0, 0, 3, 5]) == inf
        s[0, 0, 3, 5] = 3.4e38
        out, st = run(qkv * 0.1, s)
        ref, st_ref = _reference(qkv * 0.1, beta, dec, s, [T], [4], [0], H, H, dk, dv)
        assert float((out.double() - ref)[:, 0, 5].norm() / ref[:, 0, 5].norm()) < 2e-6 and float((st.double() - st_ref).norm() / st_ref.norm()) < 2e-6


@pytest.mark.parametrize("delta", [False, True])
def test_decode_rows_do_not_ask_for_scratch(cuda, monkeypatch, delta):
    """A decode step's scan is one call into the library, as many of them are launched one by one."""
    n, H, dk, dv = 3, 2, 32, 32
    qkv, beta, dec, state = _inputs(cuda, [1] * n, H, H, dk, dv, False, delta, "mild", seed=5)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    batch = ops.SeqBatch(i32(list(range(n + 1))), i32([4] * n), None, i32(list(range(n))), n, n)

    def asked(*_):
        raise AssertionError("a scan of decode rows asked for scratch")

    monkeypatch.setattr(_lib.load(), "b2_channel_scan_workspace", asked)
    st, ref = state.clone(), state.clone()
    out = ops.channel_scan(qkv, beta, dec, H, H, dk, dv, batch, st, delta=delta)
    want, ref = _reference(qkv, beta, dec, ref, [1] * n, [4] * n, list(range(n)), H, H, dk, dv)
    assert float((out.double() - want).norm() / want.norm()) < 2e-6 and float((st.double() - ref).norm() / ref.norm()) < 2e-6
