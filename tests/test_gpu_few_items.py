"""Decode of a few long rows: the dynamic schedule cuts them into many runs, which blocks per head merge; against the single-pass grid
(its weights and sums are the same, in another order: both round fp32 results of relative error 2^-20 or so to bf16, so they differ by
at most one place of bf16, 2^-8 of the value, where the sum stands at a rounding boundary, plus 2^-20 of the largest value)."""
import pytest
import torch

from b200attn import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,Hq,Hkv,lens", [
    (1, 8, 2, [8192]),
    (4, 8, 8, [4096, 1, 700, 64]),                       # one head a kv head; rows of one run beside rows of many
    (3, 28, 4, [5000, 0, 4097]),                         # seven heads, an empty row
    (2, 48, 2, [2000, 3333]),                            # 24 heads a kv head: two groups
    (18, 64, 8, [1500] * 18),                            # 144 items: the last size that takes a block per head
    (19, 64, 8, [1500] * 19),
])
def test_few_long_rows(cuda, B, Hq, Hkv, lens):
    g = torch.Generator(device=cuda).manual_seed(B * 100 + Hq)
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda).bfloat16()        # noqa: E731
    nb = -(-max(lens) // 16)
    q, kc, vc = rnd(B, Hq, 128), rnd(B * nb, Hkv, 16, 128), rnd(B * nb, Hkv, 16, 128)
    bt = torch.randperm(B * nb, generator=g, device=cuda).to(torch.int32).view(B, nb)
    sl = torch.tensor(lens, dtype=torch.int32, device=cuda)
    a, b = (ops.paged_decode(q, kc, vc, bt, sl, num_splits=n).double() for n in (0, 1))
    assert bool(((a - b).abs() <= 2.0 ** -7 * b.abs() + 2.0 ** -18 * b.abs().max()).all())
