"""Squared ReLU and gated norms in 16-byte parts held in registers, at the sizes where they can go wrong: a thread's last vector, one and two
vectors a thread, row strides, both gates, with and without weights; against fp64.  Tolerance: fp32 results rounded to the type
(2^-9 for bf16), the norm's sum of up to 4096 terms in another order and the gate's exponential a few 2^-22."""
import pytest
import torch

from b200attn import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,I,pad", [(1, 8, 0), (3, 2048, 8), (5, 2056, 0), (7, 4096, 16), (2, 20000, 0), (1, 300000, 0), (3, 36, 4)])
def test_relu_sq(cuda, T, I, pad):
    x = torch.randn(T, I + pad, generator=torch.Generator(device=cuda).manual_seed(I), device=cuda).bfloat16()
    x[0, 0], x[0, 1] = float("inf"), float("-inf")
    ref = x[:, :I].double().clamp(min=0).square()
    out = ops.relu_sq(x[:, :I])
    fin = ref.isfinite()
    assert torch.equal(out[~fin].double(), ref[~fin])
    assert bool(((out.double() - ref)[fin].abs() <= 2.0 ** -8 * ref[fin]).all())


@pytest.mark.parametrize("T,H,dv,gate_pad,kind,weights,dtype", [
    (5, 1, 2048, 0, ops.GATE_SILU, True, torch.bfloat16),
    (9, 3, 520, 8, ops.GATE_SIGMOID, False, torch.bfloat16),             # most threads without a vector
    (4, 2, 2056, 0, ops.GATE_SILU, True, torch.bfloat16),                # the first of the second vectors
    (3, 1, 4096, 16, ops.GATE_SIGMOID, True, torch.float32),
    (3, 1, 4104, 0, ops.GATE_SILU, True, torch.bfloat16),                # read twice
    (300, 4, 128, 24, ops.GATE_SILU, True, torch.bfloat16),              # a head in 16 lanes
    (257, 3, 8, 0, ops.GATE_SIGMOID, False, torch.float32),              # ... in one, and lanes behind the last
])
def test_gated_norm(cuda, T, H, dv, gate_pad, kind, weights, dtype):
    g = torch.Generator(device=cuda).manual_seed(T * dv)
    o = torch.randn(T, H, dv, generator=g, device=cuda)
    gate = torch.randn(T, H * dv + gate_pad, generator=g, device=cuda).to(dtype)[:, :H * dv]
    w = torch.rand(dv, generator=g, device=cuda) + 0.5 if weights else None
    got = ops.gated_head_norm(o, gate, w, 1e-5, kind).double().view(T, H, dv)
    z = gate.double().view(T, H, dv)
    act = torch.sigmoid(z) if kind == ops.GATE_SIGMOID else z * torch.sigmoid(z)
    ref = o.double() / (o.double().square().mean(-1, keepdim=True) + 1e-5).sqrt() * (w.double() if weights else 1.0) * act
    # the gate in the type's precision: bf16 rounds it once more
    bound = (2.0 ** -8 + 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -19) * ref.abs() + 1e-7
    assert bool(((got - ref).abs() <= bound).all()), float(((got - ref).abs() / bound).max())
