"""Rotation, norm and pool write in bf16: long batches stream their rows through a ring of copies, short ones load them; a row's results
depend on the row alone, so a long batch gives those of its slices bit for bit.  The values of short batches are the oracle's elsewhere."""
import pytest
import torch

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
