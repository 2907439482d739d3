"""Rotation, norm and pool write in bf16 at the sizes that qk_rope_cache_rows_kernel takes (more than 96 threads of sixteen entries a row):
long batches stream their rows through a ring of copies, short ones load them; a row's results depend on the row alone, so a long batch gives
those of its slices bit for bit.  Both are compared with the rotation and the norm in 64 bits."""
import pytest
import torch

import gapidra_ref as R
from b200attn import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,Gv,dk,dv,rot,interleaved,norm,v_from_k,bs", [
    (32, 8, 8, 128, 128, 128, False, True, True, 16),
    (16, 4, 4, 96, 96, 48, False, True, False, 12),              # one warp that is half idle; pages of no power of two
    (8, 8, 4, 128, 72, 64, True, False, False, 16),              # fewer value heads than key heads
    (20, 5, 5, 64, 64, 32, False, False, True, 8),
    (24, 24, 24, 128, 128, 0, False, True, False, 16),           # nothing turns
    (64, 8, 8, 128, 128, 128, True, True, True, 16),
])
def test_a_long_batch_is_its_slices(cuda, H, G, Gv, dk, dv, rot, interleaved, norm, v_from_k, bs):
    T = 2600
    g = torch.Generator(device=cuda).manual_seed(H + dk)
    qkv = torch.randn(T, (H + G) * dk + (0 if v_from_k else Gv * dv), generator=g, device=cuda).bfloat16()
    pos = torch.randint(-3, 900, (T,), generator=g, device=cuda).to(torch.int32)                 # some outside the table of 800
    slots = torch.randperm(T, generator=g, device=cuda)
    slots[::7] = -1
    cs = ops.rotary_table(800, rot, 1e4, None, cuda) if rot else None
    qw, kw = (torch.rand(n * dk, generator=g, device=cuda) + 0.5 for n in (H, G)) if norm else (None, None)
    nb = -(-T // bs)

    def call(cuts):
        kc, vc = torch.zeros(nb, G, bs, dk, device=cuda).bfloat16(), torch.zeros(nb, Gv, bs, dv, device=cuda).bfloat16()
        q = [ops.qk_rope_cache(qkv[a:b], H, G, dk, dv, pos[a:b].contiguous(), cs, rot, slots[a:b].contiguous(), kc, vc, interleaved, v_from_k, qw, kw)
             for a, b in cuts]
        return torch.cat(q), kc, vc

    for x, y in zip(call([(0, T)]), call([(a, min(T, a + 100)) for a in range(0, T, 100)])):
        assert torch.equal(x, y)


@pytest.mark.parametrize("T", [37, 2600])                            # rows loaded by their CTA; rows through the ring
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("H,G,Gv,dk,dv,rot,v_from_k,bs", [
    (32, 8, 8, 128, 128, 128, False, 16),
    (32, 8, 8, 128, 128, 32, True, 16),
    (16, 4, 4, 96, 96, 48, False, 12),
    (20, 5, 5, 64, 64, 32, True, 8),
    (8, 8, 4, 128, 72, 64, False, 16),
    (24, 24, 24, 128, 128, 0, False, 16),
])
def test_rows_against_64_bits(cuda, H, G, Gv, dk, dv, rot, v_from_k, bs, interleaved, norm, T):
    """One head of q and one of k are far larger than the others, so a norm per head or weights in another place would show; positions in any
    order; every third slot is negative: rotated, but not written.  A result is rounded to bf16 (eight bits: half a unit of the last is at most 2^-8
    of it) from fp32 (a few 2^-24 of the row's largest entry after the norm)."""
    if not rot and interleaved:
        pytest.skip("nothing turns")
    assert (H + G) * dk // 16 > 96
    g = torch.Generator(device=cuda).manual_seed(H * dk + rot)
    x = torch.randn(T, (H + G) * dk + (0 if v_from_k else Gv * dv) + 16, generator=g, device=cuda)
    x[:, :dk] *= 9.0
    x[:, H * dk:(H + 1) * dk] *= 5.0
    x[5] *= 1e-3                                                     # eps matters here
    x = x.bfloat16()
    pos = torch.randint(0, 3000, (T,), generator=g, device=cuda).to(torch.int32)
    slots = torch.randperm(T + 50, generator=g, device=cuda)[:T]
    slots[::3] = -1
    base, eps, nb = 1e4, 1e-5, -(-(T + 50) // bs)
    cs = ops.rotary_table(3000, rot, base, None, cuda) if rot else None
    qw, kw = (torch.rand(n * dk, generator=g, device=cuda) + 0.5 for n in (H, G)) if norm else (None, None)
    kc, vc = (torch.full((nb, n, bs, d), float("nan"), device=cuda).bfloat16() for n, d in ((G, dk), (Gv, dv)))
    q = ops.qk_rope_cache(x, H, G, dk, dv, pos, cs, rot, slots, kc, vc, interleaved, v_from_k, qw, kw, eps)

    def turned(rows, n, w):
        y = rows.double()
        if w is not None:
            y = y / (y.square().mean(-1, keepdim=True) + eps).sqrt() * w.double()
        y = y.view(T, n, dk)
        out = y.clone()
        if rot:
            angle = pos.double()[:, None, None] * torch.tensor(R.rotary_frequencies(rot, base), dtype=torch.float64, device=cuda)
            a, b = (slice(0, rot, 2), slice(1, rot, 2)) if interleaved else (slice(0, rot // 2), slice(rot // 2, rot))
            out[..., a] = y[..., a] * angle.cos() - y[..., b] * angle.sin()
            out[..., b] = y[..., b] * angle.cos() + y[..., a] * angle.sin()
        return out

    def close(got, want, what):
        err = (got.double() - want).abs()
        assert bool((err <= want.abs() * 2.0 ** -8 + want.abs().amax((1, 2), keepdim=True) * 2e-6).all()), (what, float((err / want.abs().amax((1, 2), keepdim=True)).max()))

    close(q, turned(x[:, :H * dk], H, qw), "q")
    on = slots >= 0
    at = slots[on]
    close(kc[at // bs, :, at % bs], turned(x[:, H * dk:(H + G) * dk], G, kw)[on], "k")
    v = x[:, H * dk:(H + G) * dk].view(T, G, dk) if v_from_k else x[:, (H + G) * dk:(H + G) * dk + Gv * dv].view(T, Gv, dv)
    assert torch.equal(vc[at // bs, :, at % bs], v[on])
    rest = torch.ones(nb * bs, dtype=torch.bool, device=cuda)
    rest[at] = False
    rest = rest.nonzero().flatten()
    assert bool(kc[rest // bs, :, rest % bs].isnan().all()) and bool(vc[rest // bs, :, rest % bs].isnan().all())
