"""Preparation of a recurrence without a convolution: prompts go by the heads of a row, smaller batches by rows.  Nothing in a row
depends on its neighbours, and both take the same sums in the same order, so a prompt's rows are those of its halves, bit for bit."""
import pytest
import torch

from b200attn import ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,dk,dv", [(3, 3, 128, 20), (2, 1, 32, 64), (5, 5, 4, 12), (16, 4, 64, 132)])
@pytest.mark.parametrize("unit,silu,rot,interleaved,weights", [(False, False, 0, False, False), (True, True, 0, False, True), (True, False, 1, False, False),
                                                               (False, True, 2, False, True), (False, False, 1, True, False), (True, True, 2, True, False)])
@pytest.mark.parametrize("mode", ["const", "channel", "sigmoid"])
def test_prompt_rows_equal_those_of_smaller_batches(cuda, dt, H, G, dk, dv, unit, silu, rot, interleaved, weights, mode):
    if rot and dk // rot % 8:
        pytest.skip("rotated entries in eights")
    T, C = 263, 2 * G * dk + H * dv
    g = torch.Generator(device=cuda).manual_seed(dk + dv)
    proj = torch.randn(T, C + H, generator=g, device=cuda).to(dt)
    proj = torch.nn.functional.pad(proj, (0, -(C + H) % 8))              # every row starts on 16 bytes
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    kw = dict(unit=unit, conv_silu=silu, unit_eps=1e-6, q_scale=0.5, k_scale=2.0)
    if weights:
        kw["conv_w"] = torch.rand(C, 1, generator=g, device=cuda) + 0.5
    if rot:
        kw.update(cos_sin=ops.rotary_table(400, dk // rot, 100.0, None, cuda), interleaved=interleaved)
    a = torch.randn(T, H * dk, generator=g, device=cuda)
    if mode == "const":
        kw.update(decay_mode=ops.DECAY_HEAD_CONST, decay_bias=torch.rand(H, generator=g, device=cuda))
    elif mode == "channel":
        kw.update(decay_mode=ops.DECAY_CHANNEL_SOFTPLUS, A_log=torch.randn(H, generator=g, device=cuda),
                  decay_bias=torch.randn(H * dk, generator=g, device=cuda), off_beta=C)
    else:
        kw.update(decay_mode=ops.DECAY_CHANNEL_SIGMOID_POW, decay_bias=torch.randn(H * dk, generator=g, device=cuda), tau=8.0)

    def call(lo, hi, cu, ctx):
        extra = {} if mode == "const" else {"a": a[lo:hi].contiguous()}
        return ops.recur_prep(proj[lo:hi], H, G, dk, dv, ops.SeqBatch(i32(cu), i32(ctx), None, i32(list(range(len(ctx)))), len(ctx), hi - lo), **extra, **kw)

    whole = call(0, T, [0, 100, 103, T], [5, -1, 0])                     # the second is padding
    parts = [call(0, 100, [0, 100], [5]), call(103, 203, [0, 100], [0]), call(203, T, [0, T - 203], [100])]
    for x, *y in zip(whole, *parts):
        if x is not None:
            assert torch.equal(torch.cat([x[:100], x[103:]]), torch.cat(y))


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,dk,dv,taps", [(4, 64, 64, 4), (2, 32, 20, 3), (16, 128, 128, 2), (1, 8, 4, 4), (16, 128, 128, 4), (16, 128, 128, 3)])
@pytest.mark.parametrize("lengths", [[300, 1, 2, 7, 301], [1, 509, 4, 3, 500, 90, 511, 505], [1] * 513, [400, 300] * 3])
def test_runs_over_several_sequences_equal_each_alone(cuda, dt, H, dk, dv, taps, lengths):
    """From 512 rows on a CTA goes through a run of rows: a sequence that begins or ends within one keeps its own history.  Alone each is
    below that, a row a CTA; the sums are the same, so are the bits."""
    C, T, n = 2 * H * dk + H * dv, sum(lengths), len(lengths)
    g = torch.Generator(device=cuda).manual_seed(taps + n)
    proj = torch.randn(T, C + H * dv + 2 * H, generator=g, device=cuda).to(dt)
    proj = torch.nn.functional.pad(proj, (0, -proj.shape[1] % 8))
    conv_w = torch.randn(C, taps, generator=g, device=cuda)
    state = torch.randn(n, taps - 1, C, generator=g, device=cuda).to(dt)
    bias = torch.rand(H, generator=g, device=cuda)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=cuda)      # noqa: E731
    cu = [0]
    for x in lengths:
        cu.append(cu[-1] + x)
    ctx = [-1 if s == 3 else s % 2 * 5 for s in range(n)]                # one is padding, every second begins

    def call(rows, cu, ctx, slots, m):
        kept = state.clone()
        b = ops.SeqBatch(i32(cu), i32(ctx), None, i32(slots), len(ctx), m)
        return ops.delta_prep(rows, C + H * dv, C + H * dv + H, H, H, dk, dv, taps, conv_w, bias, bias, b, kept), kept

    whole, states = call(proj, cu, ctx, list(range(n)), T)
    for s in range(0, n, max(1, n // 8)):
        if ctx[s] < 0:
            continue
        lo, hi = cu[s], cu[s + 1]
        part, kept = call(proj[lo:hi], [0, hi - lo], [ctx[s]], [s], hi - lo)
        for x, y in zip(whole, part):
            assert torch.equal(x[lo:hi], y)
        assert torch.equal(states[s], kept[s])
