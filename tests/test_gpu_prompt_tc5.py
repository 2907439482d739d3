"""The tcgen05 prompt kernel behind b2_masked_attention and b2_window_attention at the sizes where it can go wrong: tiles of 128
keys and rows with remainders, windows around a tile, page sizes of any kind, padded head sizes, one and two slots a CTA (few and
many CTAs, odd and even heads per kv head), capped scores on both sides of the polynomial, negative scales; against plain fp64.

Tolerance: the queries, keys and values are bf16 in both; the kernel rounds the weights (2^-9 each, relative) and the result
(2^-9): |error| <= 2^-8 (sum_j p_j |v_j| + |out|) for softmax weights.  Sigmoid weights are not normalised: the same bound on
their sum.  Two maps end in a norm, which scales both by 1 / rms: their bound is taken after it."""
import math

import pytest
import torch

from b200attn import ops

pytestmark = pytest.mark.gpu


def _visible(i, n, chunk, window, keep):
    j = torch.arange(n, device=i.device)[None]
    ok = j <= i[:, None]
    if chunk:
        ok &= j // chunk == i[:, None] // chunk
    if window:
        ok &= (i[:, None] - j < window) | (j < keep)
    return ok


def _weights(s, ok, sink, sigmoid, bias):
    if sigmoid:
        return torch.sigmoid(s + bias[:, None, None]) * ok
    s = s.masked_fill(~ok, -math.inf)
    m = s.amax(-1, keepdim=True)
    if sink is not None:
        m = torch.maximum(m, sink[:, None, None])
    e = torch.exp(s - m)
    return e / (e.sum(-1, keepdim=True) + (torch.exp(sink[:, None, None] - m) if sink is not None else 0))


CASES = [
    # lens, ctx, heads, kv heads, dk, dv, page, chunk, window, keep, cap, sink, maps, sigmoid, gate, scale factor
    ([16], [0], 2, 1, 128, 128, 16, 0, 0, 0, 0.0, False, 1, False, False, 1.0),
    ([129, 15, 300], [0, 40, 77], 4, 2, 128, 128, 16, 0, 128, 3, 0.0, True, 1, False, True, 1.0),
    ([257], [1000], 8, 8, 128, 128, 16, 0, 129, 0, 0.0, True, 1, False, False, 1.0),
    ([700, 513], [0, 128], 40, 8, 128, 128, 16, 0, 127, 0, 0.0, False, 1, False, True, 1.0),             # odd heads per kv head
    ([640, 1021], [5, 0], 32, 8, 128, 128, 16, 0, 250, 7, 50.0, True, 1, False, False, 1.0),             # two heads a CTA
    ([640], [5], 32, 8, 128, 128, 16, 0, 0, 0, 1.5, False, 1, False, False, 1.0),                        # scores far above the cap
    ([640], [5], 32, 8, 128, 128, 16, 0, 0, 0, 500.0, False, 1, False, False, 40.0),                     # ... and far apart below it
    ([333], [0], 4, 4, 64, 96, 8, 100, 0, 0, 0.0, True, 1, False, False, 1.0),
    ([500, 20], [31, 129], 4, 2, 96, 32, 24, 256, 0, 0, 30.0, True, 1, False, True, 1.0),                # pages that are no power of two
    ([260], [0], 6, 2, 32, 64, 32, 0, 1, 0, 0.0, False, 1, False, False, 1.0),                           # a window of one key
    ([300, 200], [0, 300], 4, 2, 64, 128, 16, 0, 200, 20, 0.0, False, 2, False, False, 1.0),
    ([150], [130], 8, 2, 32, 64, 16, 64, 0, 0, 4.0, True, 2, False, True, 1.0),
    ([400, 64], [0, 9], 4, 2, 128, 64, 16, 0, 150, 0, 0.0, False, 1, True, True, 1.0),
    ([1300], [0], 16, 16, 96, 96, 16, 0, 0, 0, 0.0, False, 1, True, False, 1.0),                         # two row tiles a CTA
    ([130], [64], 2, 1, 128, 128, 16, 0, 0, 0, 0.0, True, 1, False, False, -1.0),
    ([1] * 40 + [200] + [15] * 20 + [16] + [3] * 9 + [130, 2], [30] * 73, 8, 4, 64, 64, 16, 0, 64, 2, 0.0, True, 1, False, False, 1.0),
    ([0, 0, 40] + [0] * 60 + [16, 0, 17] + [0] * 20, [3] * 86, 2, 2, 32, 32, 16, 0, 0, 0, 0.0, False, 1, False, False, 1.0),      # most are empty
]


@pytest.mark.parametrize("c", CASES)
def test_masked_prompt_rows(cuda, c):
    lens, ctx, H, G, dk, dv, bs, chunk, window, keep, cap, sink, maps, sigmoid, gate, sign = c
    g = torch.Generator(device=cuda).manual_seed(len(lens) * 1000 + H + window)
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda)           # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    n, T = len(lens), sum(lens)
    nb = max(-(-(a + b) // bs) for a, b in zip(lens, ctx))
    tables = torch.randperm(n * nb, generator=g, device=cuda).to(torch.int32).view(n, nb)
    q = (2.0 * rnd(T, H * maps, dk)).bfloat16()
    kc, vc = rnd(n * nb, G * maps, bs, dk).bfloat16(), rnd(n * nb, G, bs, dv).bfloat16()
    for i in range(n):                                                   # what lies behind a sequence's end must not matter
        end = lens[i] + ctx[i]
        for p in range(end, nb * bs):
            kc[tables[i, p // bs].long(), :, p % bs] = float("nan")
            vc[tables[i, p // bs].long(), :, p % bs] = float("nan")
    cu = [0]
    for m in lens:
        cu.append(cu[-1] + m)
    batch = ops.SeqBatch(i32(cu), i32(ctx), tables, None, n, T)
    scale = sign * dk ** -0.5
    sinks = rnd(H) if sink else None
    bias = rnd(H) - 3.0 if sigmoid else None
    gt = rnd(T, H).bfloat16() if gate else None
    wide = torch.full((T, H * dv + 8), 7.0, dtype=torch.bfloat16, device=cuda)
    ops.chunk_attention(q, kc, vc, batch, scale, out=wide[:, :H * dv], chunk=chunk, window=window, keep_first=keep,
                        sink=1.0 if sink else 0.0, sink_logits=sinks, gate=gt, softcap=cap, maps=maps,
                        map_lambda=0.4 if maps == 2 else 0.0, map_eps=1e-5, map_scale=0.6, head_bias=bias,
                        weight_kind=ops.WEIGHT_SIGMOID if sigmoid else ops.WEIGHT_SOFTMAX)
    out = wide[:, :H * dv].reshape(T, H, dv).double()
    assert bool((wide[:, H * dv:] == 7.0).all()), "columns behind the heads were written"
    for i in range(n):
        end = lens[i] + ctx[i]
        rows = lambda c: c[tables[i].long()].transpose(0, 1).reshape(c.shape[1], nb * bs, -1)[:, :end].double()      # noqa: E731
        K, V = rows(kc), rows(vc)
        pos = torch.arange(ctx[i], end, device=cuda)
        ok = _visible(pos, end, chunk, window, keep)
        res, spread = [], []
        for mp in range(maps):
            qs = q[cu[i]:cu[i + 1]].view(-1, H, maps, dk)[:, :, mp].transpose(0, 1).double()
            Kh = K.view(G, maps, end, dk)[:, mp].repeat_interleave(H // G, 0)
            Vh = V.repeat_interleave(H // G, 0)
            s = torch.bmm(qs, Kh.transpose(1, 2)) * scale
            if cap:
                s = cap * torch.tanh(s / cap)
            w = _weights(s, ok, sinks.double() if sink else None, sigmoid, bias.double() if sigmoid else None)
            res.append(torch.bmm(w, Vh).transpose(0, 1))
            spread.append(torch.bmm(w, Vh.abs()).transpose(0, 1))
        ref, spr = res[0], spread[0]
        if maps == 2:
            d = res[0] - 0.4 * res[1]
            r = 0.6 / (d.square().mean(-1, keepdim=True) + 1e-5).sqrt()
            ref, spr = d * r, (spread[0] + 0.4 * spread[1]) * r * 2.0    # the norm of the error moves the root too
        if gate:
            z = torch.sigmoid(gt[cu[i]:cu[i + 1]].double())[:, :, None]
            ref, spr = ref * z, spr * z
        err = (out[cu[i]:cu[i + 1]] - ref).abs()
        # fp32 rounding of a score of size |s| moves its weight by |s| 2^-23 or so: only the case of scores in the hundreds shows it
        bound = (2.0 ** -8 + (2.0 ** -10 if abs(sign) > 1 else 0.0)) * (spr + ref.abs()) + 1e-6
        assert bool((err <= bound).all()), (i, float((err / bound).max()))


@pytest.mark.parametrize("lens,ctx,H,dn,dr,dv,window,sink,gate", [
    ([300, 70], [0, 33], 3, 128, 64, 128, 0, False, 1),                  # three sub-tiles of the key, one stage of V
    ([1400], [0], 16, 128, 64, 128, 300, True, 2),                       # two row tiles a CTA
    ([129, 1, 257], [500, 128, 0], 4, 64, 64, 64, 128, True, 0),
    ([200], [10], 5, 40, 24, 48, 77, False, 1),                          # a sub-tile across both parts of the key: no TMA boxes
    ([200, 30], [0, 10], 2, 24, 8, 112, 0, True, 2),
    ([30, 1, 64, 40] * 12, [0, 20, 0, 9] * 12, 8, 128, 64, 128, 0, True, 1),     # many short portions: the mma.sync kernel
    ([70, 57] * 12, [0, 0] * 12, 12, 64, 64, 96, 50, False, 2),                  # ... 64 keys a portion, and more
    ([70, 57] * 12, [0, 9] * 12, 12, 64, 64, 96, 50, False, 2),
    ([3, 8, 1] * 20, [100, 9, 260] * 20, 6, 128, 64, 128, 0, False, 1),          # ... a few rows each, up to 160 keys, and more
    ([3, 8, 1] * 20, [100, 99, 360] * 20, 6, 128, 64, 128, 0, False, 1),
])
def test_gathered_prompt_rows(cuda, lens, ctx, H, dn, dr, dv, window, sink, gate):
    g = torch.Generator(device=cuda).manual_seed(sum(lens) + H)
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda)           # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    n, T = len(lens), sum(lens)
    N, cu_k, k_lo = ops.latent_prompt_plan(lens, [a + b for a, b in zip(lens, ctx)], window, 1 << 30, cuda)
    qh, kr = rnd(T, H, dn + dr).bfloat16(), rnd(N, 8 + dr).bfloat16()
    kn, v = rnd(N, H, dn).bfloat16(), rnd(N, H, dv).bfloat16()
    sinks = rnd(H) if sink else None
    gt = {0: None, 1: rnd(T, H).bfloat16(), 2: rnd(T, H * dv).bfloat16()}[gate]
    cu = [0]
    for m in lens:
        cu.append(cu[-1] + m)
    scale = (dn + dr) ** -0.5
    out = ops.window_attention(qh[:, :, :dn], qh[:, :, dn:], kn, kr[:, 8:], v, i32(cu), i32(ctx), cu_k, k_lo, n, scale, window, gate=gt,
                               sink_logits=sinks).double()
    ck, lo = cu_k.tolist(), k_lo.tolist()
    for i in range(n):
        K = torch.cat([kn[ck[i]:ck[i + 1]].double(), kr[ck[i]:ck[i + 1], None, 8:].double().expand(-1, H, -1)], 2).transpose(0, 1)
        V = v[ck[i]:ck[i + 1]].double().transpose(0, 1)
        pos = torch.arange(ctx[i], ctx[i] + lens[i], device=cuda)
        ok = _visible(pos, ctx[i] + lens[i], 0, window, 0)[:, lo[i]:]
        w = _weights(torch.bmm(qh[cu[i]:cu[i + 1]].double().transpose(0, 1), K.transpose(1, 2)) * scale, ok,
                     sinks.double() if sink else None, False, None)
        ref, spr = torch.bmm(w, V).transpose(0, 1), torch.bmm(w, V.abs()).transpose(0, 1)
        if gate:
            z = torch.sigmoid(gt[cu[i]:cu[i + 1]].double()).view(lens[i], H, -1)
            ref, spr = ref * z, spr * z
        err = (out[cu[i]:cu[i + 1]] - ref).abs()
        bound = 2.0 ** -8 * (spr + ref.abs()) + 1e-6
        assert bool((err <= bound).all()), (i, float((err / bound).max()))


def test_gathered_padding_rows_are_zero(cuda):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    q, kn, kt, v = (torch.randn(*s, device=cuda).bfloat16() for s in ((40, 2, 64), (20, 2, 48), (20, 16), (20, 2, 64)))
    out = ops.window_attention(q[:, :, :48], q[:, :, 48:], kn, kt, v, i32([0, 20, 40]), i32([0, -1]), i32([0, 20, 20]), i32([0, 0]), 2, 0.1)
    assert bool((out[20:] == 0).all()) and bool(out[:20].isfinite().all()) and bool((out[:20] != 0).any())


def test_more_row_tiles_than_a_grid_dimension_holds(cuda):
    """70000 portions of 16 rows: above the 65535 blocks of a grid's second dimension."""
    g = torch.Generator(device=cuda).manual_seed(3)
    n, m, d = 70000, 16, 32
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda).bfloat16()        # noqa: E731
    q, kc, vc = rnd(n * m, 1, d), rnd(n, 1, m, d), rnd(n, 1, m, d)
    tables = torch.randperm(n, generator=g, device=cuda).to(torch.int32).view(n, 1)
    cu = torch.arange(n + 1, dtype=torch.int32, device=cuda) * m
    batch = ops.SeqBatch(cu, torch.zeros(n, dtype=torch.int32, device=cuda), tables, None, n, n * m)
    out = ops.chunk_attention(q, kc, vc, batch, d ** -0.5).view(n, m, d).double()
    K, V = kc[tables[:, 0].long(), 0].double(), vc[tables[:, 0].long(), 0].double()
    s = torch.bmm(q.view(n, m, d).double(), K.transpose(1, 2)) * d ** -0.5
    w = torch.softmax(s.masked_fill(~torch.ones(m, m, dtype=torch.bool, device=cuda).tril(), -math.inf), -1)
    ref, spr = torch.bmm(w, V), torch.bmm(w, V.abs())
    assert bool(((out - ref).abs() <= 2.0 ** -8 * (spr + ref.abs()) + 1e-6).all())


@pytest.mark.parametrize("cap,low", [(0.0, -30.0), (400.0, -30.0), (8.0, -100.0)])
def test_the_largest_weight_is_exactly_one(cuda, cap, low):
    """A key of the second tile outweighs one of the first by 2^2 to 2^7.9, all others weigh nothing: relative to the row's maximum its
    weight is one and only the small one is rounded (2^-9 of it, at most 2^-11 of the result), so the error is the result's own
    rounding and little more.  Against another reference both are rounded."""
    g = torch.Generator(device=cuda).manual_seed(21)
    n, T, G, H, d, bs, scale = 24, 300, 2, 4, 64, 16, 0.125
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    nb = -(-T // bs)
    q, K = torch.zeros(n, T, H, d, device=cuda), torch.zeros(n, G, nb * bs, d, device=cuda)
    V = torch.randn(n, G, nb * bs, d, generator=g, device=cuda).bfloat16()
    q[..., 0] = 1.0 / scale
    K[..., 0] = low
    K[:, :, 5, 0] = 0.5
    K[:, :, 200, 0] = 0.5 + (2.0 + 5.9 * torch.rand(n, G, generator=g, device=cuda)) * math.log(2.0)
    q, K = q.bfloat16(), K.bfloat16()
    pages = lambda x: x.view(n, G, nb, bs, d).transpose(1, 2).reshape(n * nb, G, bs, d).contiguous()        # noqa: E731
    batch = ops.SeqBatch(i32([T * i for i in range(n + 1)]), i32([0] * n), torch.arange(n * nb, dtype=torch.int32, device=cuda).view(n, nb), None, n, n * T)
    out = ops.chunk_attention(q.view(n * T, H, d), pages(K), pages(V), batch, scale, softcap=cap).view(n, T, H, d)[:, 200:].double()
    s = K[:, :, :201, 0].double()                                        # every row's score of key j
    s = (cap * torch.tanh(s / cap) if cap else s)[:, :, None].expand(-1, -1, T - 200, -1)
    own = torch.full((n, G, T - 200, nb * bs), float(low), device=cuda, dtype=torch.float64)
    own = cap * torch.tanh(own / cap) if cap else own
    own[..., :201] = s
    own = own.masked_fill(torch.arange(nb * bs, device=cuda)[None] > torch.arange(200, T, device=cuda)[:, None], -math.inf)
    ref = (torch.softmax(own, -1) @ V.double()).repeat_interleave(H // G, 1).transpose(1, 2)
    err, rounding = float((out - ref).norm()), float((ref.bfloat16().double() - ref).norm())
    assert err <= 1.1 * rounding, err / rounding
