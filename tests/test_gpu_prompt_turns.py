"""The tcgen05 prompt kernel of many tiles, whose CTAs take several and whose keys come in boxes: tiles in order of their length and, for more prompts
than a warp has lanes, of the batch; kept keys, windows and mask blocks that begin inside a page; pages larger than a key tile; slots
that some tiles leave empty; gathered rows whose number is not given.  Oracle and tolerance are those of test_gpu_prompt_tc5."""
import math

import pytest
import torch

from b200attn import _lib, ops
from test_gpu_prompt_tc5 import _visible, _weights, test_gathered_prompt_rows as gathered_rows, test_masked_prompt_rows as masked_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [
    # lens, ctx, heads, kv heads, dk, dv, page, chunk, window, keep, cap, sink, maps, sigmoid, gate, scale factor
    ([700, 130, 1290], [0, 900, 33], 32, 4, 128, 128, 16, 0, 300, 37, 0.0, True, 1, False, False, 1.0),      # several tiles a CTA, two heads each
    ([700, 130, 1290], [0, 900, 33], 28, 4, 64, 64, 8, 0, 0, 0, 0.0, False, 1, False, True, 1.0),            # ... two row tiles, odd heads
    ([260, 40, 513], [777, 3, 0], 64, 16, 128, 128, 64, 0, 200, 70, 8.0, True, 1, False, False, 1.0),          # the kept keys end in a page's middle
    ([260, 513], [777, 0], 32, 4, 96, 96, 128, 200, 90, 10, 0.0, True, 1, False, False, 1.0),                 # pages of a key tile, blocks inside them
    ([260, 513], [777, 0], 32, 32, 128, 64, 256, 0, 130, 200, 0.0, False, 1, True, False, 1.0),               # ... of two; the parts meet
    ([17 + 13 * (i % 11) for i in range(45)], [i % 5 * 40 for i in range(45)], 16, 4, 64, 128, 16, 0, 64, 5, 0.0, True, 1, False, False, 1.0),
    ([400, 300], [60, 0], 32, 8, 64, 128, 16, 0, 100, 20, 0.0, False, 2, False, False, 1.0),
    ([640, 500], [5, 31], 32, 8, 128, 128, 16, 0, 0, 0, 1.5, False, 1, False, False, 1.0),                    # scores far above the cap
    ([640, 500], [5, 31], 32, 8, 32, 64, 24, 256, 0, 0, 30.0, True, 1, False, True, -1.0),                    # pages that are no box, a negative scale
    ([640, 500], [5, 31], 32, 8, 128, 64, 16, 0, 150, 0, 0.0, False, 1, True, True, 1.0),
    # mask blocks, whose tiles are listed by their length: behind contexts, with an empty prompt between, rows in pairs, blocks beyond every prompt, blocks
    # with a window; more row tiles than the list holds
    ([700, 0, 1290, 16], [777, 5, 33, 299], 32, 8, 64, 64, 16, 300, 0, 0, 0.0, True, 1, False, False, 1.0),
    ([1100, 900], [50, 2000], 28, 4, 64, 64, 16, 589, 0, 0, 0.0, False, 1, False, True, 1.0),
    ([1200, 333], [700, 0], 32, 8, 64, 64, 24, 100000, 0, 0, 0.0, False, 1, True, False, 1.0),
    ([1500, 600], [130, 0], 32, 8, 64, 64, 16, 700, 260, 9, 0.0, True, 1, False, False, 1.0),
    ([1100] * 32, [37 * i for i in range(32)], 2, 1, 32, 32, 16, 400, 0, 0, 0.0, False, 1, False, False, 1.0),
])
def test_tiles_in_turns(cuda, c):
    masked_rows(cuda, c)


@pytest.mark.parametrize("lens,ctx,H,dn,dr,dv,window,sink,gate", [
    ([1400], [0], 32, 128, 64, 128, 300, True, 2),                       # two row tiles a CTA, gates per column
    ([300, 470], [0, 33], 40, 128, 64, 128, 0, False, 1),
    ([129, 1, 257], [500, 128, 0], 64, 64, 64, 64, 128, True, 0),
    ([200, 300], [10, 0], 64, 40, 24, 48, 77, False, 1),                 # a sub-tile across both parts of the key: no boxes
    ([200, 330], [0, 10], 64, 24, 8, 112, 0, True, 2),
])
def test_gathered_tiles_in_turns(cuda, lens, ctx, H, dn, dr, dv, window, sink, gate):
    gathered_rows(cuda, lens, ctx, H, dn, dr, dv, window, sink, gate)


def test_gathered_padding_in_turns(cuda):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    H = 64
    q, kn, kt, v = (torch.randn(*s, device=cuda).bfloat16() for s in ((600, H, 64), (300, H, 48), (300, 16), (300, H, 64)))
    out = ops.window_attention(q[:, :, :48], q[:, :, 48:], kn, kt, v, i32([0, 300, 600]), i32([0, -1]), i32([0, 300, 300]), i32([0, 0]), 2, 0.1)
    assert bool((out[300:] == 0).all()) and bool(out[:300].isfinite().all()) and bool((out[:300] != 0).any())


@pytest.mark.parametrize("bs,cap,sigmoid", [(16, 0.0, False), (64, 30.0, False), (16, 0.0, True)])
def test_keys_beside_the_visible_ones(cuda, bs, cap, sigmoid):
    """NaN and infinity in every key and value between the kept ones and the first window: whole pages are copied, not all of them counts."""
    n, T, ctx, H, G, d, window, keep = 8, 40, 1000, 32, 16, 64, 100, 5
    g = torch.Generator(device=cuda).manual_seed(bs)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    end = T + ctx
    nb = -(-end // bs)
    q = torch.randn(n, T, H, d, generator=g, device=cuda).bfloat16()
    K, V = (torch.randn(n, G, nb * bs, d, generator=g, device=cuda).bfloat16() for _ in range(2))
    for t, bad in ((K, math.nan), (V, math.inf)):
        t[:, :, keep:ctx - window + 1] = bad
        t[:, :, end:] = bad
    pages = lambda x: x.view(n, G, nb, bs, d).transpose(1, 2).reshape(n * nb, G, bs, d).contiguous()        # noqa: E731
    tables = torch.arange(n * nb, dtype=torch.int32, device=cuda).view(n, nb)
    batch = ops.SeqBatch(i32([T * i for i in range(n + 1)]), i32([ctx] * n), tables, None, n, n * T)
    bias = torch.full((H,), -2.0, device=cuda) if sigmoid else None
    out = ops.chunk_attention(q.view(n * T, H, d), pages(K), pages(V), batch, d ** -0.5, window=window, keep_first=keep, softcap=cap, head_bias=bias,
                              weight_kind=ops.WEIGHT_SIGMOID if sigmoid else ops.WEIGHT_SOFTMAX).view(n, T, H, d).double()
    ok = _visible(torch.arange(ctx, end, device=cuda), end, 0, window, keep)
    for i in range(n):
        Kh, Vh = (t[i, :, :end].double().nan_to_num(0.0, 0.0, 0.0).repeat_interleave(H // G, 0) for t in (K, V))
        s = torch.bmm(q[i].double().transpose(0, 1), Kh.transpose(1, 2)) * d ** -0.5
        w = _weights(cap * torch.tanh(s / cap) if cap else s, ok, None, sigmoid, bias.double() if sigmoid else None)
        ref, spr = torch.bmm(w, Vh).transpose(0, 1), torch.bmm(w, Vh.abs()).transpose(0, 1)
        assert bool(((out[i] - ref).abs() <= 2.0 ** -8 * (spr + ref.abs()) + 1e-6).all()), i


@pytest.mark.parametrize("lens,ctx,H,window", [([300, 129, 257], [0, 60, 5], 32, 0), ([1300, 700], [0, 33], 16, 200)])
def test_gathered_rows_of_any_number(cuda, lens, ctx, H, window):
    """The number of gathered rows is a hint: the true one, none, one that is too small or larger than the rows give the same bits (the last keys come in
    boxes or row by row), and those are right.  One portion's keys and values, and the rows behind the last one, are NaN and infinity: boxes reach into
    them, the other portions must not."""
    dn, dr, dv, scale, bad = 128, 64, 128, 0.1, 1
    g = torch.Generator(device=cuda).manual_seed(9)
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda).bfloat16()        # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    T, cu = sum(lens), [0]
    for m in lens:
        cu.append(cu[-1] + m)
    rows, cu_k, k_lo = ops.latent_prompt_plan(lens, [a + b for a, b in zip(lens, ctx)], window, 1 << 30, cuda)
    ck, lo = cu_k.tolist(), k_lo.tolist()
    spare = 300                                                          # rows of the buffers behind the last one
    q, kn, kt, v = rnd(T, H, dn + dr), rnd(rows + spare, H, dn), rnd(rows + spare, dr), rnd(rows + spare, H, dv)
    for t, x in ((kn, math.nan), (kt, math.nan), (v, math.inf)):
        t[ck[bad]:ck[bad + 1]] = x
        t[rows:] = x
    cu_q, start = i32(cu), i32(ctx)
    p = lambda t: t.data_ptr()                                           # noqa: E731

    def run(n_keys):
        out = torch.empty(T, H, dv, dtype=torch.bfloat16, device=cuda)
        _lib.check(_lib.load().b2_window_attention_rows(p(out), p(q), H * (dn + dr), dn + dr, p(q) + 2 * dn, H * (dn + dr), dn + dr, p(kn), p(kt), dr,
                                                        p(v), p(cu_q), p(start), p(cu_k), p(k_lo), len(lens), T, H, dn, dr, dv, scale, window, None, None, 0,
                                                        0, H * dv, n_keys, torch.cuda.current_stream().cuda_stream))
        return out

    want = run(rows)
    for n_keys in (0, 1, rows - 150, rows + 200, 1 << 40):
        assert torch.equal(run(n_keys).view(torch.int16), want.view(torch.int16)), n_keys
    for i in range(len(lens)):
        if i == bad:
            continue
        K = torch.cat([kn[ck[i]:ck[i + 1]].double(), kt[ck[i]:ck[i + 1], None].double().expand(-1, H, -1)], 2).transpose(0, 1)
        V = v[ck[i]:ck[i + 1]].double().transpose(0, 1)
        ok = _visible(torch.arange(ctx[i], ctx[i] + lens[i], device=cuda), ctx[i] + lens[i], 0, window, 0)[:, lo[i]:]
        w = _weights(torch.bmm(q[cu[i]:cu[i + 1]].double().transpose(0, 1), K.transpose(1, 2)) * scale, ok, None, False, None)
        ref, spr = torch.bmm(w, V).transpose(0, 1), torch.bmm(w, V.abs()).transpose(0, 1)
        assert bool(((want[cu[i]:cu[i + 1]].double() - ref).abs() <= 2.0 ** -8 * (spr + ref.abs()) + 1e-6).all()), i


def test_gathered_rows_that_repeat(cuda):
    """Queries and shared key parts with a row stride of zero (one row for all): no box has such a stride."""
    T, H, dn, dr, dv = 1500, 16, 128, 64, 128
    g = torch.Generator(device=cuda).manual_seed(4)
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda).bfloat16()        # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    rows, cu_k, k_lo = ops.latent_prompt_plan([T - 500, 500], [T - 500, 700], 300, 1 << 30, cuda)
    kn, v = rnd(rows, H, dn), rnd(rows, H, dv)
    args = (i32([0, T - 500, T]), i32([0, 200]), cu_k, k_lo, 2, 0.1, 300)
    for qn, qr, kt in ((rnd(1, H, dn).expand(T, -1, -1), rnd(T, H, dr), rnd(rows, dr)), (rnd(T, H, dn), rnd(T, 1, dr).expand(-1, H, -1), rnd(rows, dr)),
                       (rnd(T, H, dn), rnd(T, H, dr), rnd(1, dr).expand(rows, -1))):
        want = ops.window_attention(qn.contiguous(), qr.contiguous(), kn, kt.contiguous(), v, *args)
        assert torch.equal(ops.window_attention(qn, qr, kn, kt, v, *args), want)
