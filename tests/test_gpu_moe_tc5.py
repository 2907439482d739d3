"""The experts' grouped products on tcgen05 against fp64: widths with remainders of the 64-column and 64- / 128-row boxes, experts
with no row, one, a whole tile and one more, stacked and separate weights, gathered rows with a stride, every activation.

Tolerance: the products add up in fp32; what is left are two roundings to bf16 of at most 2^-9 of an entry, the activation's (whose
errors add up with random signs in the second product, so their share of its norm stays) and the result's: 2^-8 of the norm."""
import pytest
import torch

from b200attn import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("glu", [ops.GLU_SILU, ops.GLU_CLAMPED, ops.FF_RELU_SQ])
@pytest.mark.parametrize("rows,D,F,E,top,stacked,on_input", [
    (1, 64, 64, 4, 2, True, False),
    (33, 72, 88, 3, 1, False, True),
    (64, 200, 136, 8, 3, True, True),
    (97, 128, 64, 2, 2, False, False),                   # every expert has 97 rows: three tiles and one more row
    (5, 1096, 264, 64, 8, True, False),                  # most experts without a row; a pipeline that goes round
])
def test_experts(cuda, rows, D, F, E, top, stacked, on_input, glu):
    g = torch.Generator(device=cuda).manual_seed(rows * 7 + D)
    rnd = lambda *s: torch.randn(*s, generator=g, device=cuda)           # noqa: E731
    h = rnd(rows, D + 8).bfloat16()[:, :D]
    gate, up = (rnd(E, F, D).mul_(D ** -0.5).bfloat16() for _ in range(2))
    down = rnd(E, D, F).mul_(F ** -0.5).bfloat16()
    gated = glu != ops.FF_RELU_SQ
    if stacked and gated:
        both = torch.cat([gate, up], 1)
        gate, up = both[:, :F], both[:, F:]
    # few tokens leave experts empty, and the first token's choices all differ from the others' first
    ids = torch.stack([torch.randperm(E, generator=g, device=cuda)[:top] for _ in range(rows)]).int().contiguous()
    wts = torch.rand(rows, top, generator=g, device=cuda)
    add = rnd(rows, D).bfloat16()
    y = ops.moe_experts(h, ids, wts, gate if gated else None, up, down, glu=glu, glu_alpha=1.702, glu_limit=7.0, weight_on_input=on_input,
                        add=add)
    ref = add.double()
    for t in range(rows):
        for j in range(top):
            e, w = int(ids[t, j]), wts[t, j].double()
            x = h[t].double() * (w if on_input else 1.0)
            u = up[e].double() @ x
            if not gated:
                a = u.clamp(min=0).square()
            else:
                p = gate[e].double() @ x
                if glu == ops.GLU_CLAMPED:
                    p, u = p.clamp(max=7.0), u.clamp(-7.0, 7.0)
                    a = p * torch.sigmoid(1.702 * p) * (u + 1.0)
                else:
                    a = p * torch.sigmoid(p) * u
            ref[t] += (down[e].double() @ a) * (1.0 if on_input else w)
    assert float((y.double() - ref).norm() / ref.norm()) < 2 ** -8
