"""Decode rows of b2_latent_attention (one row a sequence) against fp64, by both kernels that take them (block tables as wide as the rows,
and so wide that they promise enough work for the tcgen05 kernel): latents of 128, 256 and 512 numbers with rotated parts that do
and do not fill their 64 columns, more and fewer heads than a CTA takes, key counts around tiles of 64 and boxes of 16, pages TMA boxes
fit and do not fit, windows that begin inside a page, keys split over CTAs, and scores that outgrow the first tile's by 2^60 and more.

Tolerance: queries and rows are bf16 in both; the kernel rounds the weights and the result, 2^-9 each of its own:
|error| <= 2^-8 (sum_j p_j |c_j| + |out|), with 2^-10 more where fp32 scores in the hundreds move the weights."""
import math

import pytest
import torch

from b200attn import ops

pytestmark = pytest.mark.gpu


def _widen(tables, bs, wide):
    """Columns up to 100000 tokens, behind every row's end: the rule between the kernels goes by the table's width."""
    return torch.nn.functional.pad(tables, (0, 100000 // bs - tables.shape[1])).contiguous() if wide else tables


CASES = [
    ([0, 1, 15, 16, 17, 62, 63, 64, 65, 127, 128, 129], 16, 512, 64, 16, 0, False, False, 0.0),
    ([700, -1, 3], 32, 512, 64, 16, 0, True, True, 0.0),                 # split over CTAs, padding between
    ([2000], 33, 512, 64, 32, 0, True, False, 0.0),                      # one head more than a CTA takes, up to 16 shares
    ([300, 1000, 77, 16], 5, 512, 64, 16, 70, False, True, 0.0),         # windows that begin inside a page
    ([300, 1000, 77, 64], 40, 256, 32, 24, 100, True, True, 0.0),        # pages of 24: no boxes
    ([90, 333], 8, 128, 16, 8, 0, False, False, 0.0),
    ([500] * 80, 32, 128, 64, 64, 0, False, True, 0.0),                  # more CTAs than SMs
    ([200, 65, 640], 32, 512, 128, 16, 0, False, False, 0.0),
    ([1500, 130], 16, 512, 64, 16, 0, True, False, 400.0),               # computed a second time
    ([1500] * 150, 4, 256, 64, 16, 0, False, False, 400.0),              # ... without a split, an odd number of tiles
    ([1500, 130], 16, 512, 64, 16, 0, True, False, -400.0),              # falling scores: late weights vanish
    ([3000 - i for i in range(32)], 32, 512, 64, 16, 700, True, False, 0.0),     # windows in the tcgen05 kernel
    ([1500 - 7 * i for i in range(16)], 64, 256, 32, 24, 1100, False, True, 0.0),        # ... pages of 24
    ([700, 40, 3], 18, 512, 256, 16, 0, True, True, 0.0),                # keys of more than 640 numbers
    ([300, 9], 20, 128, 768, 16, 0, False, False, 0.0),                  # ... of more than either kernel takes
]


@pytest.mark.parametrize("ctx,H,R,dr,bs,window,sink,gate,rise", CASES)
def test_latent_decode(cuda, ctx, H, R, dr, bs, window, sink, gate, rise):
    _check(cuda, ctx, H, R, dr, bs, window, sink, gate, rise, False)


@pytest.mark.parametrize("ctx,H,R,dr,bs,window,sink,gate,rise", CASES)
def test_latent_decode_wide_tables(cuda, ctx, H, R, dr, bs, window, sink, gate, rise):
    _check(cuda, ctx, H, R, dr, bs, window, sink, gate, rise, True)


def _check(cuda, ctx, H, R, dr, bs, window, sink, gate, rise, wide_table):
    g = torch.Generator(device=cuda).manual_seed(len(ctx) * 100 + H + window)
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda)           # noqa: E731
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    n, Dc = len(ctx), R + dr
    nb = max(ctx) // bs + 1
    scale = Dc ** -0.5
    cache = rnd(n * nb, bs, Dc).bfloat16()
    tables = torch.randperm(n * nb, generator=g, device=cuda).to(torch.int32).view(n, nb)
    qa = rnd(n, H, Dc).bfloat16()
    if rise:                                                             # one column makes the scores climb from the first key to the last
        qa[:, :, 0] = 8.0
    for i, c in enumerate(ctx):
        rows = torch.arange(nb * bs, device=cuda)
        page, off = tables[i].long()[rows // bs], rows % bs
        if rise:
            cache[page, off, 0] = (rows.float() / (c + 1) * rise / 8.0 / scale * math.log(2.0)).bfloat16()
        lo = max(0, c - window + 1) if window else 0
        dead = (rows > c) | (rows // bs < lo // bs)                      # behind the end, and pages before the window's first
        cache[page[dead], off[dead]] = float("nan")
    sinks = rnd(H) if sink else None
    wide = rnd(n, H + 3).bfloat16()
    batch = ops.SeqBatch(i32(list(range(n + 1))), i32(ctx), _widen(tables, bs, wide_table), None, n, n)
    out = ops.latent_attention(qa, cache, batch, R, scale, window, gate=wide[:, :H] if gate else None, sink_logits=sinks).double()
    for i, c in enumerate(ctx):
        if c < 0:
            assert bool((out[i] == 0).all())
            continue
        lo = max(0, c - window + 1) if window else 0
        rows = torch.arange(lo, c + 1, device=cuda)
        K = cache[tables[i].long()[rows // bs], rows % bs].double()
        s = qa[i].double() @ K.T * scale
        m = s.amax(-1, keepdim=True)
        if sink:
            m = torch.maximum(m, sinks.double()[:, None])
        e = torch.exp(s - m)
        w = e / (e.sum(-1, keepdim=True) + (torch.exp(sinks.double()[:, None] - m) if sink else 0.0))
        ref, spr = w @ K[:, :R], w @ K[:, :R].abs()
        if gate:
            z = torch.sigmoid(wide[i, :H].double())[:, None]
            ref, spr = ref * z, spr * z
        bound = (2.0 ** -8 + (2.0 ** -10 if rise else 0.0)) * (spr + ref.abs()) + 1e-6
        err = (out[i] - ref).abs()
        assert bool((err <= bound).all()), (i, c, float((err / bound).max()))


def test_long_rows_repeat_to_the_bit(cuda):
    """Some forty tiles a share, many times: the issuing warp's choice between the next scores and this output is timing, and neither
    order changes what is summed, so every call returns the same bits."""
    g = torch.Generator(device=cuda).manual_seed(7)
    n, H, R, dr, bs, c = 64, 32, 512, 64, 16, 2559
    nb = c // bs + 1
    cache = torch.randn(n * nb, bs, R + dr, generator=g, device=cuda).bfloat16()
    tables = torch.randperm(n * nb, generator=g, device=cuda).to(torch.int32).view(n, nb)
    qa = torch.randn(n, H, R + dr, generator=g, device=cuda).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    batch = ops.SeqBatch(i32(list(range(n + 1))), i32([c] * n), tables, None, n, n)
    first = ops.latent_attention(qa, cache, batch, R, (R + dr) ** -0.5, 0)
    assert bool(torch.isfinite(first).all())
    for _ in range(40):
        assert torch.equal(first, ops.latent_attention(qa, cache, batch, R, (R + dr) ** -0.5, 0))


@pytest.mark.parametrize("wide", [False, True])
def test_as_many_rows_as_sequences_but_not_one_each(cuda, wide):
    """Rows [2, 0, 1, 3, 0, 0]: every row is its own sequence's, at its own position; the same rows asked one by one give the same bits."""
    g = torch.Generator(device=cuda).manual_seed(9)
    lens, ctx, H, R, dr, bs = [2, 0, 1, 3, 0, 0], [40, 5, 0, 130, 7, 9], 20, 256, 64, 16
    n, nb = len(lens), 10
    cache = torch.randn(n * nb, bs, R + dr, generator=g, device=cuda).bfloat16()
    tables = _widen(torch.randperm(n * nb, generator=g, device=cuda).to(torch.int32).view(n, nb), bs, wide)
    qa = torch.randn(n, H, R + dr, generator=g, device=cuda).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    cu = [sum(lens[:i]) for i in range(n + 1)]
    owner = [i for i, k in enumerate(lens) for _ in range(k)]
    pos = [ctx[i] + r for i, k in enumerate(lens) for r in range(k)]
    scale = (R + dr) ** -0.5
    out = ops.latent_attention(qa, cache, ops.SeqBatch(i32(cu), i32(ctx), tables, None, n, n), R, scale, 0)
    single = ops.SeqBatch(i32(list(range(n + 1))), i32(pos), tables[owner].contiguous(), None, n, n)
    assert torch.equal(out, ops.latent_attention(qa, cache, single, R, scale, 0))


@pytest.mark.parametrize("n", [3, 160])                                  # keys split over CTAs, and not
@pytest.mark.parametrize("where", [0, 1, 700])
@pytest.mark.parametrize("wide", [False, True])
def test_a_nan_in_a_cached_row_stays_one(cuda, wide, n, where):
    """A NaN in the rotated part of a cached row reaches every output of its sequence and no other's, however the keys are shared."""
    g = torch.Generator(device=cuda).manual_seed(11)
    H, R, dr, bs, c = 8, 512, 64, 16, 900
    nb = c // bs + 1
    cache = torch.randn(n * nb, bs, R + dr, generator=g, device=cuda).bfloat16()
    tables = torch.arange(n * nb, dtype=torch.int32, device=cuda).view(n, nb)
    cache[nb + where // bs, where % bs, R + 5] = float("nan")
    qa = torch.randn(n, H, R + dr, generator=g, device=cuda).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    out = ops.latent_attention(qa, cache, ops.SeqBatch(i32(list(range(n + 1))), i32([c] * n), _widen(tables, bs, wide), None, n, n), R, 0.04, 0)
    nan = torch.isnan(out).flatten(1)
    assert bool(nan[1].all()) and not bool(nan[0].any()) and not bool(nan[2:].any())


@pytest.mark.parametrize("n", [2, 150])                                  # keys split over CTAs, and not
@pytest.mark.parametrize("wide", [False, True])
def test_a_sink_far_above_the_first_share(cuda, wide, n):
    """Scores that climb by 400 (in powers of two) over the row and a sink between: above the first share's scores by more than fp32
    holds, far below the last's, so that it weighs nothing; and a sink above all of them, which leaves nothing to the keys."""
    g = torch.Generator(device=cuda).manual_seed(13)
    H, R, dr, bs, c = 4, 256, 64, 16, 1535
    nb = c // bs + 1
    scale = 1.0 / 16
    cache = torch.randn(n * nb, bs, R + dr, generator=g, device=cuda).bfloat16()
    tables = torch.arange(n * nb, dtype=torch.int32, device=cuda).view(n, nb)
    qa = torch.randn(n, H, R + dr, generator=g, device=cuda).bfloat16()
    qa[:, :, R] = 8.0
    row = torch.arange(nb * bs, device=cuda).float()
    cache[..., R] = ((row / c - 0.5) * 400.0 / 8.0 / scale * math.log(2.0)).bfloat16().view(nb, bs).repeat(n, 1)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    batch = ops.SeqBatch(i32(list(range(n + 1))), i32([c] * n), _widen(tables, bs, wide), None, n, n)
    plain = ops.latent_attention(qa, cache, batch, R, scale, 0)
    between = ops.latent_attention(qa, cache, batch, R, scale, 0, sink_logits=torch.full((H,), 0.0, device=cuda))
    above = ops.latent_attention(qa, cache, batch, R, scale, 0, sink_logits=torch.full((H,), 300.0, device=cuda))
    assert bool(torch.isfinite(plain).all())
    assert bool(((between.float() - plain.float()).abs() <= 2.0 ** -6 * plain.float().abs() + 1e-3).all())
    assert bool((above.float().abs() <= 1e-6).all())


@pytest.mark.parametrize("n,H,c", [(8, 64, 3000), (150, 16, 1000)])     # keys split over CTAs, and not
def test_the_error_is_the_rounding_of_the_result(cuda, n, H, c):
    """The tcgen05 kernel: weights are kept to 16 bits, so what is left against fp64 is the result's own rounding to bf16: 5 % above it are allowed for the
    fp32 sums.  (Weights of eight bits against another reference than the row's maximum: 24 % above.)"""
    g = torch.Generator(device=cuda).manual_seed(17)
    R, dr, bs = 512, 64, 16
    nb = c // bs + 1
    cache = torch.randn(n * nb, bs, R + dr, generator=g, device=cuda).bfloat16()
    tables = torch.arange(n * nb, dtype=torch.int32, device=cuda).view(n, nb)
    qa = torch.randn(n, H, R + dr, generator=g, device=cuda).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    out = ops.latent_attention(qa, cache, ops.SeqBatch(i32(list(range(n + 1))), i32([c] * n), tables, None, n, n), R, 0.1, 0).double()
    K = cache.view(n, nb * bs, R + dr)[:, :c + 1].double()
    ref = torch.softmax(torch.bmm(qa.double(), K.transpose(1, 2)) * 0.1, -1) @ K[:, :, :R]
    err, rounding = float((out - ref).norm()), float((ref.bfloat16().double() - ref).norm())
    assert err <= 1.05 * rounding, err / rounding
