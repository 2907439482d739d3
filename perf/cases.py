"""The work a user of this framework has it do, as cases that can be timed and compared: the attention, recurrence and expert
blocks of the decoders at prompt and decode sizes, and one whole model call, each through the public entry points.

A case is a dict of plain values; "kind" names the block:

  paged    one decode step of one Llama layer: KV write + paged-attention decode (bf16 or fp8 pool)
  prompt   prompt-chunk attention of one Llama layer over the paged pool
  masked   what lies between the projections of a masked grouped-query attention layer: rotation + pool write, then attention
           (sliding window with kept first tokens, mask blocks, sinks, capped scores, two maps, sigmoid weights)
  latent   the same of a latent attention layer; long prompt portions rebuild keys and values per head, as the models do
  mixer    the same of a recurrent mixer: preparation, scan over the per-sequence state, gated norm
  experts  router + routed experts of a feed-forward layer
  model    one forward of a whole decoder over ragged prompts, with the logits of every prompt's last rows

Head counts, widths, windows and vocabularies are those of bench.py / bench_families.py and the model registry; lengths are the
serving range they declare (contexts of 512 to 8192 tokens, 1 to 256 sequences, prompts of up to 8192 rows a step).
"""
import math
import sys
from pathlib import Path

import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "vllm-backend-public_b200"))

BS = 16                                              # tokens per page, the serving default
F64 = torch.float64


def listed():
    return [
        # the smallest call: a handful of short conversations, eight query heads on two KV heads; latency and launches
        dict(name="decode_small", kind="paged", seqs=4, heads=8, kv_heads=2, ctx=512, ragged=False, fp8=False),
        # the serving benchmark's decode step: Llama-3-8B heads, 64 sequences, 4k context, bf16 pool
        dict(name="decode_llama", kind="paged", seqs=64, heads=32, kv_heads=8, ctx=4096, ragged=False, fp8=False),
        # long ragged conversations over the fp8 pool
        dict(name="decode_fp8_ragged", kind="paged", seqs=96, heads=32, kv_heads=8, ctx=8192, ragged=True, fp8=True),
        # a chunked prefill step: two portions behind cached prefixes, 4k rows and an odd rest
        dict(name="prompt_llama", kind="prompt", seqs=2, rows=5003, heads=32, kv_heads=8, ctx=4096),
        # one long prompt through a windowed layer with capped scores and a sink per head, values taken from the keys
        dict(name="masked_prompt", kind="masked", seqs=1, rows=4096, ctx=0, heads=32, kv_heads=8, dim=128, vdim=128, rot=128, window=1024,
             keep=0, chunk=0, cap=50.0, sink=True, maps=1, sigmoid=False, v_from_k=True, norm=True, dtype="bf16"),
        # a decode step of a windowed layer that keeps the first tokens, with a sink per head
        dict(name="masked_decode", kind="masked", seqs=64, rows=64, ctx=2560, heads=32, kv_heads=8, dim=128, vdim=128, rot=64, window=1024,
             keep=4, chunk=0, cap=0.0, sink=True, maps=1, sigmoid=False, v_from_k=True, norm=False, dtype="bf16"),
        # ragged prompts through a causal latent layer (512 + 64 numbers cached per token)
        dict(name="latent_prompt", kind="latent", seqs=3, rows=4096, ctx=0, heads=16, dim=128, rot=64, vdim=128, rank=512, window=0,
             sink=False),
        # a decode step of a causal latent layer
        dict(name="latent_decode", kind="latent", seqs=64, rows=64, ctx=2560, heads=32, dim=128, rot=64, vdim=128, rank=512, window=0,
             sink=False),
        # one long prompt through linear attention with a fixed decay per head
        dict(name="linear_prompt", kind="mixer", mode="const", seqs=1, rows=4096, ctx=0, heads=16, groups=16, dim=128, vdim=128, taps=1,
             dtype="bf16"),
        # ragged prompts, some continuing, through a gated delta rule with a short convolution
        dict(name="delta_prompt", kind="mixer", mode="delta_head", seqs=3, rows=3001, ctx=700, heads=16, groups=16, dim=128, vdim=128, taps=4,
             dtype="bf16"),
        # a decode step of the routed experts: the weights of the chosen experts stream through once
        dict(name="experts_decode", kind="experts", rows=64, width=4096, ff=1792, experts=64, top=8, gated=True, on_input=True),
        # four ragged prompts through a three-layer decoder (windowed, latent and linear attention, dense feed-forwards)
        dict(name="model_prompt", kind="model", seqs=4, rows=4096, width=2048, heads=16, kv_heads=4, ff=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["paged", "paged", "prompt", "masked", "masked", "masked", "latent", "latent", "mixer", "mixer", "mixer", "experts",
                       "experts", "model"])
    if kind == "paged":
        heads, kv = rng.choice([(8, 2), (16, 4), (32, 8), (64, 8), (28, 4)])
        ctx = _log(rng, 128, 8192)
        most = max(1, min(192, (64 * 4096 * 8) // (ctx * kv)))
        return dict(kind=kind, seqs=_log(rng, 1, most), heads=heads, kv_heads=kv, ctx=ctx, ragged=rng.random() < 0.6, fp8=rng.random() < 0.4)
    if kind == "prompt":
        heads, kv = rng.choice([(8, 2), (16, 4), (32, 8)])
        rows = _log(rng, 64, 5000)
        return dict(kind=kind, seqs=min(rng.randint(1, 4), rows // 32), rows=rows, heads=heads, kv_heads=kv, ctx=rng.choice([0, 1000, 4096]))
    if kind == "masked":
        decode = rng.random() < 0.45
        heads, kv = rng.choice([(16, 4), (32, 8), (16, 2), (8, 8)])
        style = rng.choice(["window", "window", "keep", "chunk", "maps", "sigmoid"])
        dim, vdim = (64, 128) if style == "maps" else rng.choice([(128, 128), (128, 128), (64, 64), (96, 96), (128, 64)])
        seqs = _log(rng, 1, 128) if decode else rng.randint(1, 4)
        rows = seqs if decode else _log(rng, 256, 4096)
        f32 = rng.random() < 0.1
        if f32:
            seqs, rows = (min(seqs, 16), min(seqs, 16)) if decode else (1, min(rows, 384))
        return dict(kind=kind, seqs=seqs, rows=rows, ctx=_log(rng, 100, 4096) if decode else rng.choice([0, 0, 777]), heads=heads, kv_heads=kv,
                    dim=dim, vdim=vdim, rot=dim if rng.random() < 0.5 else dim // 2,
                    window=0 if style == "chunk" else _log(rng, 128, 2048), keep=rng.randint(1, 16) if style in ("keep", "maps") else 0,
                    chunk=_log(rng, 256, 2048) if style == "chunk" else 0, cap=30.0 if style == "window" and rng.random() < 0.5 else 0.0,
                    sink=style in ("window", "keep", "chunk") and rng.random() < 0.7, maps=2 if style == "maps" else 1,
                    sigmoid=style == "sigmoid", v_from_k=style in ("window", "keep") and dim == vdim,
                    norm=style in ("window", "sigmoid"), dtype="f32" if f32 else "bf16")
    if kind == "latent":
        decode = rng.random() < 0.5
        seqs = _log(rng, 1, 96) if decode else rng.randint(1, 4)
        heads = rng.choice([8, 16, 16, 32])
        return dict(kind=kind, seqs=seqs, rows=seqs if decode else _log(rng, 300, 4096 if heads <= 16 else 2500),
                    ctx=_log(rng, 100, 4096) if decode else rng.choice([0, 0, 555]), heads=heads, dim=128, rot=64, vdim=128,
                    rank=rng.choice([512, 512, 256]), window=rng.choice([0, 1024, 300]), sink=rng.random() < 0.4)
    if kind == "mixer":
        decode = rng.random() < 0.35
        seqs = _log(rng, 1, 96) if decode else rng.randint(1, 5)
        mode = rng.choice(["const", "delta_head", "delta_channel", "gated_channel"])
        heads = rng.choice([4, 8, 16, 16])
        dim, vdim = rng.choice([(128, 128), (128, 128), (64, 64), (64, 128), (96, 80)])
        return dict(kind=kind, mode=mode, seqs=seqs, rows=seqs if decode else _log(rng, 50 * seqs, 4096), ctx=rng.choice([0, 0, 900]) if not decode
                    else 1000, heads=heads, groups=heads // 2 if mode.startswith("delta") and rng.random() < 0.3 else heads, dim=dim, vdim=vdim,
                    taps=rng.choice([1, 4]) if mode.startswith("delta") else 1, dtype="f32" if rng.random() < 0.15 else "bf16")
    if kind == "experts":
        width, ff, experts = rng.choice([(2048, 1024, 32), (2048, 1024, 32), (4096, 1792, 64), (1024, 768, 16)])
        return dict(kind=kind, rows=_log(rng, 1, 128) if width > 2048 or rng.random() < 0.6 else _log(rng, 200, 2000), width=width, ff=ff, experts=experts,
                    top=rng.randint(1, 8), gated=rng.random() < 0.75, on_input=rng.random() < 0.4)
    return dict(kind=kind, seqs=rng.randint(1, 6), rows=_log(rng, 300, 4000), width=rng.choice([1024, 2048]), heads=rng.choice([8, 16]), kv_heads=4,
                ff=rng.choice([2048, 4096]))


# ---------------------------------------------------------------------------------------------------------------- sizes
def _lens(total, n, seed):
    """n ragged lengths that sum to total."""
    if n == total:
        return [1] * n
    g = torch.Generator().manual_seed(seed + 77)
    w = torch.rand(n, generator=g) + 0.25
    cut = [max(1, int(x)) for x in (w / w.sum() * total).tolist()]
    cut[0] += total - sum(cut)
    return cut


def _shape(case):
    """Rows and cached tokens of every sequence: the sizes are the case's, whatever the seed."""
    n = case["seqs"]
    if case["kind"] == "paged":
        if not case["ragged"]:
            return [1] * n, [case["ctx"] - 1] * n
        g = torch.Generator().manual_seed(5)
        lo, hi = math.log(max(16, case["ctx"] // 32)), math.log(case["ctx"])
        return [1] * n, [int(math.exp(lo + (hi - lo) * x)) - 1 for x in torch.rand(n, generator=g).tolist()]
    q = _lens(case["rows"], n, 1)
    ctx = case.get("ctx", 0)
    if q == [1] * n:                                 # decode rows: contexts around the nominal one
        return q, [max(1, ctx - 13 * (i % 8)) for i in range(n)]
    return q, [ctx if i % 2 == 0 else ctx // 2 for i in range(n)]


def _seen(case, pos):
    """Number of keys the query at a position sees."""
    lo = pos // case["chunk"] * case["chunk"] if case.get("chunk") else 0
    w = case.get("window", 0)
    wlo = max(lo, pos - w + 1) if w else lo
    return pos - wlo + 1 + (max(0, min(case.get("keep", 0), wlo) - lo) if w else 0)


def _pairs(case):
    return sum(_seen(case, c + i) for q, c in zip(*_shape(case)) for i in range(q))


def _read(case):
    """Cached tokens that have to be read: what the union of a sequence's rows sees."""
    n = 0
    for q, c in zip(*_shape(case)):
        first = _seen(case, c)
        n += first + q - 1 if not case.get("chunk") else max(first, _seen(case, c + q - 1)) + (q - 1 if q > case["chunk"] else 0)
    return n


def work(case):
    k = case["kind"]
    if k == "model":
        T, D, F, H, G = case["rows"], case["width"], case["ff"], case["heads"], case["kv_heads"]
        d, R, dr, Q = 128, 512, 64, 1536
        win = dict(seqs=case["seqs"], rows=T, kind="m", window=1024, keep=4)
        full = dict(seqs=case["seqs"], rows=T, kind="m")
        # windowed layer, latent layer (query latent, rebuilt keys and values), linear layer; two squared-ReLU feed-forwards; head
        params = D * (H * d + G * d + H) + H * d * D + D * (Q + H + R + dr) + Q * H * (d + dr) + 2 * H * R * d + H * d * D + \
            D * 4 * H * d + H * d * D + 2 * 2 * D * F
        flops = 2 * T * params + 4 * _pairs(win) * H * d + 2 * _pairs(full) * H * (2 * d + dr) + 6 * T * H * d * d + 2 * case["seqs"] * ROWS * 32000 * D
        return {"bytes": params * 2 + 32000 * D * 2 + T * D * (2 + 4 * 6), "flops": flops}
    if k == "experts":
        T, D, F, E, top = case["rows"], case["width"], case["ff"], case["experts"], case["top"]
        used = E * (1 - (1 - top / E) ** T)          # experts that some row chooses, for evenly spread choices
        mats = 3 if case["gated"] else 2
        return {"bytes": used * mats * F * D * 2 + E * D * 2 + 2 * T * D * 2, "flops": 2 * mats * T * top * F * D + 2 * T * E * D}
    q, ctx = _shape(case)
    T = sum(q)
    if k == "paged":
        H, G, e = case["heads"], case["kv_heads"], 1 if case["fp8"] else 2
        n = sum(c + 1 for c in ctx)
        return {"bytes": n * G * 2 * 128 * e + T * H * 128 * 4 + T * G * 2 * 128 * (2 + e) + sum(-(-(c + 1) // BS) for c in ctx) * 4,
                "flops": 4 * n * H * 128}
    if k == "prompt":
        H, G = case["heads"], case["kv_heads"]
        pairs = sum(m * c + m * (m + 1) // 2 for m, c in zip(q, ctx))
        return {"bytes": sum(m + c for m, c in zip(q, ctx)) * G * 512 + T * H * 512, "flops": 4 * pairs * H * 128}
    es = 4 if case.get("dtype") == "f32" else 2
    if k == "masked":
        H, G, m, dk, dv = case["heads"], case["kv_heads"], case["maps"], case["dim"], case["vdim"]
        wide = H * m * dk + G * m * dk + (0 if case["v_from_k"] else G * dv)
        return {"bytes": (T * (wide + G * m * dk + G * dv + H * dv) + _read(case) * G * (m * dk + dv)) * es,
                "flops": 2 * _pairs(case) * H * m * (dk + dv)}
    if k == "latent":
        H, dn, dr, dv, R = case["heads"], case["dim"], case["rot"], case["vdim"], case["rank"]
        if _per_head(case):
            N = _latent_plan_rows(case)
            return {"bytes": (T * H * (dn + dr + dv) + T * (R + dr) * 2 + N * (R + dr) + H * R * (dn + dv)) * 2,
                    "flops": 2 * _pairs(case) * H * (dn + dr + dv) + 2 * N * R * H * (dn + dv)}
        return {"bytes": (T * H * (R + dr + dr + R) + T * (R + dr) * 2 + _read(case) * (R + dr)) * 2, "flops": 2 * _pairs(case) * H * (2 * R + dr)}
    H, G, dk, dv = case["heads"], case["groups"], case["dim"], case["vdim"]
    C = 2 * G * dk + H * dv
    a = H * dk * 4 if "channel" in case["mode"] else 0
    state = case["seqs"] * H * dk * dv * 4 * 2
    return {"bytes": T * ((C + 2 * H * dv) * es + a) + state, "flops": 2 * T * H * dk * dv * (3 if case["mode"].startswith("delta") else 2)}


def tolerance(case):
    """Two correct bf16 implementations differ by the rounding of q, of the weights before the value product and of the result: each
    up to 2^-9 of a value, 1.7e-3 to 3.6e-3 of the result against 64 bits.  The three-layer model, its prompts cut in two portions:
    8e-4, at most 2.2e-2 of the root mean square.  fp32: sums in another order."""
    if case.get("dtype") == "f32":
        return {"rel": 2e-5, "max": 2e-3}
    return {"rel": 1e-2, "max": 0.1, "differ": 2e-3}


# ---------------------------------------------------------------------------------------------------------------- inputs
class _Made:
    """Random tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        return (torch.randn(*shape, generator=self.g, device="cuda") * std).to(dtype)

    def uniform(self, lo, hi, *shape):
        return torch.rand(*shape, generator=self.g, device="cuda") * (hi - lo) + lo

    def shuffled(self, n):
        return torch.randperm(n, generator=self.g, device="cuda")


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _step(case, made):
    """One engine step's indices: rows, positions, pages in shuffled order, cache slots."""
    from b200attn import ops
    q, ctx = _shape(case)
    n, nb = len(q), max(-(-(a + b) // BS) for a, b in zip(q, ctx))
    tables = made.shuffled(n * nb).to(torch.int32).view(n, nb).contiguous()
    cu = [0]
    for m in q:
        cu.append(cu[-1] + m)
    seq = torch.repeat_interleave(torch.arange(n, device="cuda"), torch.tensor(q, device="cuda"))
    pos = torch.cat([torch.arange(c, c + m, device="cuda") for m, c in zip(q, ctx)])
    slots = tables[seq, pos // BS].long() * BS + pos % BS
    batch = ops.SeqBatch(_i32(cu), _i32(ctx), tables, _i32(list(range(n))), n, cu[-1])
    return dict(batch=batch, tables=tables, slots=slots.contiguous(), pos=pos.to(torch.int32), q_lens=q, kv_lens=[a + b for a, b in zip(q, ctx)],
                blocks=n * nb, T=cu[-1], cu=cu, ctx=ctx)


ROWS = 8                                             # logits rows per prompt of the model case


def _dtype(case):
    return torch.float32 if case.get("dtype") == "f32" else torch.bfloat16


def _per_head(case):
    """Whether the models take the per-head path of a latent layer for these rows."""
    return case["rows"] >= 256 and case["rows"] > case["seqs"]


def _latent_plan_rows(case):
    return sum(c + m - (max(0, c - (case["window"] - 1)) if case["window"] else 0) for m, c in zip(*_shape(case)))


def prepare(case, seed):
    from b200attn import ops
    made, k = _Made(seed), case["kind"]
    if k == "model":
        return _prepare_model(case, made, seed)
    if k == "experts":
        T, D, F, E = case["rows"], case["width"], case["ff"], case["experts"]
        up = made.normal(E, (2 if case["gated"] else 1) * F, D, std=D ** -0.5)
        return dict(case=case, h=made.normal(T, D), router=made.normal(E, D, std=D ** -0.5), up=up, down=made.normal(E, D, F, std=F ** -0.5),
                    shared=made.normal(T, D))
    s = _step(case, made)
    s["case"] = case
    T, nb = s["T"], s["blocks"]
    if k in ("paged", "prompt"):
        H, G, d = case["heads"], case["kv_heads"], 128
        s["q"] = made.normal(T, H, d)
        if case.get("fp8"):
            for n in ("kc", "vc"):
                s[n] = made.normal(nb, G, BS, d, std=40.0, dtype=torch.float8_e4m3fn).view(torch.uint8)
            s["ks"], s["vs"] = torch.full((1,), 0.025, device="cuda"), torch.full((1,), 0.02, device="cuda")
        else:
            s["kc"], s["vc"] = made.normal(nb, G, BS, d), made.normal(nb, G, BS, d)
            s["ks"] = s["vs"] = None
        if k == "paged":
            s["kn"], s["vn"] = made.normal(T, G, d), made.normal(T, G, d)
            s["sl"] = _i32(s["kv_lens"])
            # what the engine keeps: the schedule from the host's lengths, a workspace
            s["splits"] = ops.plan_num_splits(torch.tensor(s["kv_lens"], dtype=torch.int32), H, G, d, BS, 1 if case["fp8"] else 0)
            s["ws"] = torch.zeros(max(ops.decode_workspace_bytes(T, H, G, d, BS, s["tables"].shape[1], 0), 256), dtype=torch.uint8, device="cuda")
        return s
    if k == "masked":
        H, G, m, dk, dv, dt = case["heads"], case["kv_heads"], case["maps"], case["dim"], case["vdim"], _dtype(case)
        s["qkv"] = made.normal(T, (H + G) * m * dk + (0 if case["v_from_k"] else G * dv), dtype=dt)
        s["kc"], s["vc"] = made.normal(nb, G * m, BS, dk, dtype=dt), made.normal(nb, G, BS, dv, dtype=dt)
        s["rot"] = ops.rotary_table(max(s["kv_lens"]), case["rot"], 1e6, None, "cuda")
        if case["norm"]:
            s["qw"], s["kw"] = made.uniform(0.8, 1.2, H * m * dk), made.uniform(0.8, 1.2, G * m * dk)
        s["sinks"] = made.normal(H, dtype=torch.float32) if case["sink"] else None
        s["bias"] = made.normal(H, std=0.5, dtype=torch.float32) - math.log(256.0) if case["sigmoid"] else None
        return s
    if k == "latent":
        H, dn, dr, dv, R = case["heads"], case["dim"], case["rot"], case["vdim"], case["rank"]
        s["qh"] = made.normal(T, H, dn + dr)
        s["kv"] = made.normal(T, R + dr)
        s["nw"] = made.uniform(0.8, 1.2, R)
        s["cache"] = made.normal(nb, BS, R + dr)
        s["rot"] = ops.rotary_table(max(s["kv_lens"]), dr, 1e4, None, "cuda")
        s["uk"], s["uv"] = made.normal(H, dn, R, std=R ** -0.5), made.normal(H, R, dv, std=R ** -0.5)
        s["gate"] = made.normal(T, H)
        s["sinks"] = made.normal(H, dtype=torch.float32) if case["sink"] else None
        if _per_head(case):
            s["plan"] = ops.latent_prompt_plan(s["q_lens"], s["kv_lens"], case["window"], 1 << 30, "cuda")
        else:                                        # decode rows and short portions: the absorbed queries of the product before
            s["qa"] = torch.empty(T, H, R + dr, dtype=torch.bfloat16, device="cuda")
            torch.bmm(s["qh"][:, :, :dn].transpose(0, 1), s["uk"], out=s["qa"][:, :, :R].transpose(0, 1))
        return s
    H, G, dk, dv, dt, n = case["heads"], case["groups"], case["dim"], case["vdim"], _dtype(case), case["seqs"]
    C = 2 * G * dk + H * dv
    s["proj"] = made.normal(T, C + H * dv + 2 * H, dtype=dt)          # q | k | v | gate | beta | a
    s["state"] = made.normal(n, H, dk, dv, std=0.3, dtype=torch.float32)
    s["nw"] = made.uniform(0.8, 1.2, dv)
    if case["taps"] > 1:
        s["conv_w"] = made.normal(C, case["taps"], std=case["taps"] ** -0.5, dtype=torch.float32)
        s["conv"] = made.normal(n, case["taps"] - 1, C, dtype=dt)
    if case["mode"] == "const":
        s["decay"] = torch.tensor([1.0 - 2.0 ** (-5.0 - 3.0 * h / max(H - 1, 1)) for h in range(H)], device="cuda")
        s["rot"] = ops.rotary_table(max(s["kv_lens"]), dk, 1e4, None, "cuda")
    else:
        s["A_log"] = made.uniform(0.0, math.log(8.0), H).contiguous()
        wide = H * dk if "channel" in case["mode"] else H
        s["dt_bias"] = made.uniform(-5.0, -1.0, wide)
        s["a"] = made.normal(T, H * dk, dtype=torch.float32) if wide > H else None
    return s


def _prepare_model(case, made, seed):
    from b200attn import sanarax
    from b200attn.model import PrefillBatch
    s = _step(dict(case, ctx=0), made)
    cfg = sanarax.bench_config(case["width"], 3, case["heads"], case["kv_heads"], 128, case["ff"], 32000)
    s["case"] = case
    s["model"] = sanarax.SanaraxModel(cfg, torch.device("cuda", 0), s["blocks"], BS, seed=int(seed) % (1 << 30), max_position=8192,
                                      max_num_seqs=case["seqs"])
    s["tokens"] = torch.randint(0, cfg.vocab, (s["T"],), generator=made.g, device="cuda")
    b = s["batch"]
    s["prefill"] = PrefillBatch(b.cu_q, b.ctx_start, s["tables"], s["T"], s["kv_lens"], b.state_slots, s["q_lens"])
    s["rows"] = torch.tensor([r for i in range(case["seqs"]) for r in range(max(s["cu"][i], s["cu"][i + 1] - ROWS), s["cu"][i + 1])], device="cuda")
    return s


# ---------------------------------------------------------------------------------------------------------------- a pass
def run(s):
    from b200attn import ops
    case = s["case"]
    k = case["kind"]
    if k == "model":
        return s["model"].forward(s["tokens"], s["pos"], s["slots"], 0, None, None, s["prefill"], s["rows"])
    if k == "experts":
        F, up = case["ff"], s["up"]
        ids, wts = ops.moe_route(s["h"], s["router"], None, case["top"], scoring=ops.ROUTE_SIGMOID_PLAIN)
        if not case["gated"]:
            y = ops.moe_experts(s["h"], ids, wts, None, up, s["down"], glu=ops.FF_RELU_SQ)
        else:
            y = ops.moe_experts(s["h"], ids, wts, up[:, :F], up[:, F:], s["down"], w_gate_up=up, weight_on_input=case["on_input"],
                                add=s["shared"])
        return {"y": y, "ids": ids, "weights": wts}
    if k == "paged":
        out = ops.paged_decode_append(s["q"], s["kn"], s["vn"], s["slots"], s["kc"], s["vc"], s["tables"], s["sl"], k_scale=s["ks"],
                                      v_scale=s["vs"], workspace=s["ws"], num_splits=s["splits"])
        return {"out": out, "k_cache": s["kc"], "v_cache": s["vc"]}
    b = s["batch"]
    if k == "prompt":
        return ops.prefill_attention(s["q"], s["kc"], s["vc"], s["tables"], b.cu_q, b.ctx_start, total_tokens=s["T"])
    if k == "masked":
        H, G, m, dk = case["heads"], case["kv_heads"], case["maps"], case["dim"]
        q = ops.qk_rope_cache(s["qkv"], H * m, G * m, dk, case["vdim"], s["pos"], s["rot"], case["rot"], s["slots"], s["kc"], s["vc"],
                              v_from_k=case["v_from_k"], q_norm=s.get("qw"), k_norm=s.get("kw"))
        o = ops.chunk_attention(q, s["kc"], s["vc"], b, dk ** -0.5, case["chunk"], sink=1.0 if case["sink"] else 0.0, window=case["window"],
                                keep_first=case["keep"], sink_logits=s["sinks"], softcap=case["cap"], maps=m, map_lambda=0.4 if m > 1 else 0.0,
                                map_scale=0.6 if m > 1 else 1.0, weight_kind=ops.WEIGHT_SIGMOID if case["sigmoid"] else ops.WEIGHT_SOFTMAX,
                                head_bias=s["bias"])
        return {"out": o, "k_cache": s["kc"], "v_cache": s["vc"]}
    if k == "latent":
        H, dn, dr, R, T = case["heads"], case["dim"], case["rot"], case["rank"], s["T"]
        scale = (dn + dr) ** -0.5
        qa = ops.latent_prep(s["qh"].view(T, H * (dn + dr)), H, dn, dr, dr, R, 0, 0, s["nw"], 1e-6, s["pos"], s["rot"], s["slots"], s["cache"],
                             qa=s.get("qa"), kv=s["kv"])
        if "plan" not in s:
            o = ops.latent_attention(qa, s["cache"], b, R, scale, case["window"], gate=s["gate"], sink_logits=s["sinks"])
            return {"out": o, "cache": s["cache"]}
        N, cu_k, k_lo = s["plan"]
        lat = ops.latent_gather(s["cache"], s["tables"], cu_k, k_lo, b.n_seq, N)
        kn = torch.nn.functional.linear(lat[:, :R], s["uk"].view(H * dn, R)).view(N, H, dn)
        v = torch.empty(N, H, case["vdim"], dtype=kn.dtype, device=kn.device)
        torch.bmm(lat[:, :R].unsqueeze(0).expand(H, N, R), s["uv"], out=v.transpose(0, 1))
        o = ops.window_attention(s["qh"][:, :, :dn], qa[:, :, R:], kn, lat[:, R:], v, b.cu_q, b.ctx_start, cu_k, k_lo, b.n_seq, scale,
                                 case["window"], gate=s["gate"], sink_logits=s["sinks"])
        return {"out": o, "cache": s["cache"]}
    H, G, dk, dv, mode = case["heads"], case["groups"], case["dim"], case["vdim"], case["mode"]
    C, proj = 2 * G * dk + H * dv, s["proj"]
    gate, off_b, off_a = proj[:, C:C + H * dv], C + H * dv, C + H * dv + H
    if mode == "delta_head":
        w = s.get("conv_w")
        w = w if w is not None else torch.ones(C, 1, device=proj.device)
        qkv, beta, decay = ops.delta_prep(proj, off_b, off_a, H, G, dk, dv, case["taps"], w, s["A_log"], s["dt_bias"], b, s.get("conv"))
        o = ops.delta_scan(qkv, beta, decay, H, G, dk, dv, b, s["state"])
        y = ops.delta_out(o, proj, C, s["nw"], 1e-6)
    elif mode == "const":
        qkv, _, decay = ops.recur_prep(proj, H, G, dk, dv, b, k_scale=dk ** -0.5, decay_mode=ops.DECAY_HEAD_CONST, decay_bias=s["decay"],
                                       cos_sin=s["rot"])
        o = ops.channel_scan(qkv, None, decay, H, G, dk, dv, b, s["state"], delta=False)
        y = ops.gated_head_norm(o, gate, None, 1e-6)
    elif mode == "delta_channel":
        qkv, beta, decay = ops.recur_prep(proj, H, G, dk, dv, b, taps=case["taps"], conv_w=s.get("conv_w"), conv_state=s.get("conv"),
                                          conv_silu=True, unit=True, q_scale=dk ** -0.5, off_beta=off_b, decay_mode=ops.DECAY_CHANNEL_SOFTPLUS,
                                          a=s["a"], A_log=s["A_log"], decay_bias=s["dt_bias"])
        o = ops.channel_scan(qkv, beta, decay, H, G, dk, dv, b, s["state"], delta=True)
        y = ops.gated_head_norm(o, gate, s["nw"], 1e-6, ops.GATE_SIGMOID)
    else:
        qkv, _, decay = ops.recur_prep(proj, H, G, dk, dv, b, q_scale=dk ** -0.5, decay_mode=ops.DECAY_CHANNEL_SIGMOID_POW, a=s["a"],
                                       decay_bias=s["dt_bias"].add(6.0), tau=16.0)
        o = ops.channel_scan(qkv, None, decay, H, G, dk, dv, b, s["state"], delta=False)
        y = ops.gated_head_norm(o, gate, s["nw"], 1e-6, ops.GATE_SILU)
    return {"out": y, "heads": o, "state": s["state"]}


# ---------------------------------------------------------------------------------------------------------------- 64 bits
def _pool_rows(cache, table, n):
    """[heads, n, d] of one sequence from a pool [blocks, heads, BS, d]."""
    nb = -(-n // BS)
    return cache[table[:nb].long()].transpose(0, 1).reshape(cache.shape[1], nb * BS, cache.shape[3])[:, :n]


def _visible(case, pos, n):
    """bool [rows, n]: which positions the rows see."""
    i, j = pos[:, None], torch.arange(n, device=pos.device)[None]
    ok = j <= i
    if case.get("chunk"):
        ok = ok & (j // case["chunk"] == i // case["chunk"])
    if case.get("window"):
        ok = ok & ((i - j < case["window"]) | (j < case.get("keep", 0)))
    return ok


def _soft(s, ok, sink):
    """Softmax weights of scores [h, m, n] with an optional sink logit per head in the denominator."""
    s = s.masked_fill(~ok, -math.inf)
    m = s.amax(-1, keepdim=True)
    if sink is not None:
        m = torch.maximum(m, sink[:, None, None])
    e = torch.exp(s - m)
    den = e.sum(-1, keepdim=True)
    return e / (den + torch.exp(sink[:, None, None] - m) if sink is not None else den)


def _turn(x, rot, pos, interleaved=False):
    """Rotates the first rot.shape[1] entries of x [rows, heads, d]."""
    n = rot.shape[1]
    c, s = rot[pos, : n // 2].to(F64)[:, None], rot[pos, n // 2:].to(F64)[:, None]
    y = x.clone()
    a, b = (x[..., 0:n:2], x[..., 1:n:2]) if interleaved else (x[..., : n // 2], x[..., n // 2:n])
    u, w = a * c - b * s, b * c + a * s
    if interleaved:
        y[..., 0:n:2], y[..., 1:n:2] = u, w
    else:
        y[..., : n // 2], y[..., n // 2:n] = u, w
    return y


def _blocks(n, m):
    return [(a, min(n, a + m)) for a in range(0, n, m)]


def exact(case, seed):
    k = case["kind"]
    if k == "model":
        return None
    s = prepare(case, seed)
    if k == "experts":
        return _exact_experts(case, s)
    if k == "mixer":
        return _exact_mixer(case, s)
    T, pos = s["T"], s["pos"].long()
    if k == "latent":
        return _exact_latent(case, s, pos)
    if k == "masked":
        H, G, m, dk, dv = case["heads"], case["kv_heads"], case["maps"], case["dim"], case["vdim"]
        x = s["qkv"].to(F64)
        nq, nk = H * m * dk, G * m * dk
        q, kk = x[:, :nq], x[:, nq:nq + nk]
        v = kk if case["v_from_k"] else x[:, nq + nk:]
        if case["norm"]:
            q = q / (q.square().mean(-1, keepdim=True) + 1e-6).sqrt() * s["qw"]
            kr = kk / (kk.square().mean(-1, keepdim=True) + 1e-6).sqrt() * s["kw"]
        else:
            kr = kk
        q = _turn(q.view(T, H * m, dk), s["rot"], pos)
        kn, vn = _turn(kr.view(T, G * m, dk), s["rot"], pos), v.view(T, G, dv)
    else:
        H, G, m, dk, dv = case["heads"], case["kv_heads"], 1, 128, 128
        q = s["q"].to(F64)
        if k == "paged":
            kn, vn = s["kn"].to(F64), s["vn"].to(F64)
            if case["fp8"]:
                kn, vn = ((t.float() / sc).to(torch.float8_e4m3fn).to(F64) * sc for t, sc in ((s["kn"], s["ks"]), (s["vn"], s["vs"])))
    out = torch.empty(T, H, dv, dtype=F64, device="cuda")
    for i, (n, ctx) in enumerate(zip(s["q_lens"], s["ctx"])):
        r0, end = s["cu"][i], n + ctx
        pools = []
        for c, sc in ((s["kc"], s.get("ks")), (s["vc"], s.get("vs"))):
            rows = _pool_rows(c, s["tables"][i], end)
            pools.append((rows.view(torch.float8_e4m3fn) if case.get("fp8") else rows).to(F64) * (sc if case.get("fp8") else 1.0))
        K, V = pools
        if k != "prompt":
            K[:, ctx:], V[:, ctx:] = kn[r0:r0 + n].transpose(0, 1), vn[r0:r0 + n].transpose(0, 1)
        for a, b in _blocks(n, max(1, (1 << 27) // (end * H * m))):
            qs, ok = q[r0 + a:r0 + b].transpose(0, 1), _visible(case, torch.arange(ctx + a, ctx + b, device="cuda"), end)
            res = []
            for mp in range(m):
                # query head (h, map) reads key head (h // (H / G), map) and value head h // (H / G)
                qm = qs.reshape(H, m, b - a, dk)[:, mp].reshape(G, H // G * (b - a), dk)
                sc = torch.bmm(qm, K.view(G, m, end, dk)[:, mp].transpose(1, 2)).view(H, b - a, end) * dk ** -0.5
                if case.get("cap"):
                    sc = case["cap"] * torch.tanh(sc / case["cap"])
                if case.get("sigmoid"):
                    w = torch.sigmoid(sc + s["bias"].to(F64)[:, None, None]) * ok
                else:
                    w = _soft(sc, ok, s["sinks"].to(F64) if case.get("sink") else None)
                res.append(torch.bmm(w.view(G, H // G * (b - a), end), V).view(H, b - a, dv))
            o = res[0]
            if m > 1:
                o = o - 0.4 * res[1]
                o = o / (o.square().mean(-1, keepdim=True) + 1e-6).sqrt() * 0.6
            out[r0 + a:r0 + b] = o.transpose(0, 1)
    return out if k == "prompt" else {"out": out, "k_cache": None, "v_cache": None}


def _exact_latent(case, s, pos):
    H, dn, dr, dv, R, T = case["heads"], case["dim"], case["rot"], case["vdim"], case["rank"], s["T"]
    per_head = "plan" in s
    qh, kv = s["qh"].to(F64), s["kv"].to(F64)
    qr = _turn(qh[:, :, dn:], s["rot"], pos, True)
    c = kv[:, :R]
    row = torch.cat([c / (c.square().mean(-1, keepdim=True) + 1e-6).sqrt() * s["nw"], _turn(kv[:, None, R:], s["rot"], pos, True)[:, 0]], 1)
    gate, out = torch.sigmoid(s["gate"].to(F64)), torch.empty(T, H, dv if per_head else R, dtype=F64, device="cuda")
    for i, (n, ctx) in enumerate(zip(s["q_lens"], s["ctx"])):
        r0, end = s["cu"][i], n + ctx
        nb = -(-end // BS)
        L = s["cache"][s["tables"][i, :nb].long()].reshape(nb * BS, R + dr)[:end].to(F64)
        L[ctx:] = row[r0:r0 + n]
        lat, kr = L[:, :R], L[:, R:]
        if per_head:
            K = torch.cat([torch.einsum("nr,hdr->hnd", lat, s["uk"].to(F64)), kr[None].expand(H, end, dr)], 2)
            V = torch.einsum("nr,hrd->hnd", lat, s["uv"].to(F64))
            Q = torch.cat([qh[:, :, :dn], qr], 2)
        else:                                        # the absorbed part of the queries is an input
            K, V = L[None].expand(H, end, R + dr), lat[None].expand(H, end, R)
            Q = torch.cat([s["qa"][:, :, :R].to(F64), qr], 2)
        for a, b in _blocks(n, max(1, (1 << 27) // (end * H))):
            sc = torch.bmm(Q[r0 + a:r0 + b].transpose(0, 1), K.transpose(1, 2)) * (dn + dr) ** -0.5
            w = _soft(sc, _visible(case, torch.arange(ctx + a, ctx + b, device="cuda"), end), s["sinks"].to(F64) if case["sink"] else None)
            out[r0 + a:r0 + b] = torch.bmm(w, V).transpose(0, 1) * gate[r0 + a:r0 + b, :, None]
    return {"out": out, "cache": None}


def _exact_mixer(case, s):
    H, G, dk, dv, mode, T = case["heads"], case["groups"], case["dim"], case["vdim"], case["mode"], s["T"]
    C, taps, delta = 2 * G * dk + H * dv, case["taps"], mode.startswith("delta")
    p = s["proj"].to(F64)
    x = p[:, :C]
    if taps > 1:
        full = []
        for i, (n, ctx) in enumerate(zip(s["q_lens"], s["ctx"])):
            old = s["conv"][i].to(F64) if ctx else torch.zeros(taps - 1, C, dtype=F64, device="cuda")
            z = torch.cat([old[max(0, 0):], x[s["cu"][i]:s["cu"][i + 1]]])
            full.append(sum(z[j:j + n] * s["conv_w"][:, j].to(F64) for j in range(taps)))
        x = torch.cat(full)
    if delta:
        x = torch.nn.functional.silu(x)
    q, k, v = x[:, :G * dk].view(T, G, dk), x[:, G * dk:2 * G * dk].view(T, G, dk), x[:, 2 * G * dk:].view(T, H, dv)
    beta = torch.sigmoid(p[:, C + H * dv:C + H * dv + H]) if delta else None
    sp = torch.nn.functional.softplus
    if mode == "const":
        pos = s["pos"].long()
        q, k = _turn(q, s["rot"], pos), _turn(k, s["rot"], pos) * dk ** -0.5
        g = s["decay"].to(F64)[None, :, None].expand(T, H, 1)
    elif mode == "delta_head":
        g = torch.exp(-torch.exp(s["A_log"].to(F64)) * sp(p[:, C + H * dv + H:] + s["dt_bias"].to(F64)))[:, :, None]
    elif mode == "delta_channel":
        g = torch.exp(-torch.exp(s["A_log"].to(F64))[None, :, None] * sp((s["a"].to(F64) + s["dt_bias"].to(F64)).view(T, H, dk)))
    else:
        q = q * dk ** -0.5
        g = torch.sigmoid((s["a"].to(F64) + s["dt_bias"].add(6.0).to(F64)).view(T, H, dk)) ** (1 / 16.0)
    if delta:
        q = q / (q.square().sum(-1, keepdim=True) + 1e-6).sqrt() * dk ** -0.5
        k = k / (k.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    heads, state = torch.empty(T, H, dv, dtype=F64, device="cuda"), s["state"].to(F64)
    longest = max(s["q_lens"])
    # all sequences advance together: row t of every sequence that has one
    n = case["seqs"]
    S = torch.stack([state[i] if c else torch.zeros_like(state[i]) for i, c in enumerate(s["ctx"])])
    start, lens = torch.tensor(s["cu"][:-1], device="cuda"), s["q_lens"]
    for t in range(longest):
        live = [i for i in range(n) if t < lens[i]]
        r = start[live] + t
        A = S if len(live) == n else S[live]
        A = A * g[r][..., None]
        u = v[r]
        if delta:
            u = beta[r][..., None] * (u - torch.einsum("nhkv,nhk->nhv", A, k[r]))
        A = A + k[r][..., None] * u[..., None, :]
        heads[r] = torch.einsum("nhkv,nhk->nhv", A, q[r])
        if len(live) == n:
            S = A
        else:
            S[live] = A
    z = p[:, C:C + H * dv].view(T, H, dv)
    act = torch.sigmoid(z) if mode == "delta_channel" else torch.nn.functional.silu(z)
    w = 1.0 if mode == "const" else s["nw"].to(F64)
    out = heads / (heads.square().mean(-1, keepdim=True) + 1e-6).sqrt() * w * act
    return {"out": out.reshape(T, H * dv), "heads": heads, "state": S}


def _exact_experts(case, s):
    F, top = case["ff"], case["top"]
    h = s["h"].to(F64)
    sc = torch.sigmoid(h @ s["router"].to(F64).t())
    wts, ids = torch.sort(sc, dim=1, descending=True, stable=True)
    wts, ids = wts[:, :top].contiguous(), ids[:, :top].contiguous()
    y = s["shared"].to(F64).clone() if case["gated"] else torch.zeros_like(h)
    for e in range(case["experts"]):
        r, j = torch.nonzero(ids == e, as_tuple=True)
        if not len(r):
            continue
        on_input = case["gated"] and case["on_input"]
        x = h[r] * wts[r, j, None] if on_input else h[r]
        z = x @ s["up"][e].to(F64).t()
        a = torch.nn.functional.silu(z[:, :F]) * z[:, F:] if case["gated"] else z.clamp(min=0).square()
        o = a @ s["down"][e].to(F64).t()
        y.index_add_(0, r, o if on_input else o * wts[r, j, None])
    return {"y": y, "ids": None, "weights": wts}
