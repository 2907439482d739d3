"""Short portions of b2_masked_attention (fewer rows than the prompt kernel takes): the forms with the keys or the query heads as the
16 rows of the operand, 4, 8 and 16 warps a CTA, key counts around their tiles of 16 and 32, several rows a sequence, and batches in which
they stand beside prompts and padding; against fp64 by the same check and bound as the prompt rows."""
import pytest
import torch

from b200attn import ops
from test_gpu_prompt_tc5 import test_masked_prompt_rows as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [
    # lens, ctx, heads, kv heads, dk, dv, page, chunk, window, keep, cap, sink, maps, sigmoid, gate, scale factor
    ([1], [0], 8, 1, 128, 128, 16, 0, 0, 0, 0.0, False, 1, False, False, 1.0),
    ([1, 1, 1], [15, 16, 17], 7, 1, 64, 96, 16, 0, 0, 0, 0.0, True, 1, False, True, 1.0),
    ([1, 2, 14], [1000, 255, 256], 8, 2, 128, 128, 16, 0, 0, 0, 0.0, True, 1, False, False, 1.0),        # 16 warps a CTA
    ([1] * 30, list(range(300, 600, 10)), 32, 8, 128, 128, 16, 0, 0, 0, 30.0, True, 1, False, True, 1.0),        # 8
    ([1] * 70, list(range(70)), 32, 8, 96, 64, 8, 0, 33, 5, 0.0, True, 1, False, False, 1.0),            # 4, most with no tile
    ([3] * 40, list(range(40)), 6, 6, 32, 32, 24, 64, 0, 0, 0.0, False, 1, False, False, 1.0),           # one head a kv head
    ([1, 5], [700, 90], 8, 4, 128, 128, 16, 0, 0, 0, 0.0, False, 1, True, True, 1.0),                    # sigmoid
    ([1, 5], [700, 90], 9, 1, 128, 128, 16, 0, 0, 0, 0.0, True, 1, False, False, 1.0),                   # nine heads: the heads are the rows
    ([1, 9], [700, 90], 40, 2, 64, 128, 16, 0, 100, 0, 20.0, True, 1, False, True, 1.0),                 # two passes over the heads
    ([1, 5], [700, 90], 8, 2, 256, 256, 16, 0, 0, 0, 0.0, False, 1, False, False, 1.0),
    ([1, 5], [700, 90], 8, 2, 64, 256, 16, 0, 0, 0, 0.0, False, 1, False, False, 1.0),
    ([1, 7], [300, 20], 12, 1, 128, 64, 16, 0, 0, 0, 0.0, False, 2, False, False, 1.0),                  # two maps
    ([200, 1, 3, 90, 2], [0, 300, 40, 7, 0], 8, 2, 128, 128, 16, 0, 0, 0, 0.0, True, 1, False, False, 1.0),      # beside prompts
    ([1] * 12, [0, 15, 16, 30, 31, 32, 33, 62, 63, 64, 127, 128], 16, 2, 64, 64, 16, 0, 0, 0, 0.0, True, 1, False, False, 1.0),  # keys of 64: 32 a tile
    ([1, 2, 14], [1000, 255, 256], 8, 4, 64, 128, 16, 0, 0, 0, 25.0, True, 1, False, True, 1.0),         # ... 16 warps a CTA
    ([1] * 30, list(range(300, 600, 10)), 32, 8, 32, 256, 16, 0, 200, 3, 0.0, False, 1, False, False, 1.0),      # ... 8
    ([1, 5], [700, 90], 8, 2, 64, 192, 16, 0, 0, 0, 0.0, False, 1, True, True, 1.0),                     # ... sigmoid
])
def test_short_portions(cuda, c):
    _check(cuda, c)


def test_padding_beside_a_prompt_is_zero(cuda):
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    ctx = [0, -1, -1, 5]
    cu = [0, 300, 303, 343, 345]
    q = torch.randn(345, 8, 64, device=cuda).bfloat16()
    kc, vc = (torch.randn(80, 2, 16, 64, device=cuda).bfloat16() for _ in range(2))
    tables = torch.arange(80, dtype=torch.int32, device=cuda).view(4, 20)
    out = torch.full((345, 512), 7.0, dtype=torch.bfloat16, device=cuda)
    ops.chunk_attention(q, kc, vc, ops.SeqBatch(i32(cu), i32(ctx), tables, None, 4, 345), 0.125, out=out)
    assert bool((out[300:343] == 0).all()) and bool((out[:300] != 7.0).any(1).all()) and bool((out[343:] != 7.0).any(1).all())
