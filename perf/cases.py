"""What a program that uses this library has it do, as cases that can be timed and compared.

A case is a dict of plain values with a "kind":

  product   one Q8_0 product y = x . w^T                      (Q8Context.matmul)
  layer     the four products of a transformer layer: fused QKV, O, fused gate+up, down, as four
            products, or (fused) with the residual add and the gated unit in their stores and the
            live batch in a device word                       (matmul, matmul_fused)
  experts   router, then the routed feed-forward step, gate and up as two tensors or interleaved
            (moe_route, moe_ffn, moe_ffn_fused)
  blocks    one product with a tensor of another block type of the model file   (matmul)
  dequant   rows of a Q8_0 tensor as binary16                 (dequant)

Weights have the benchmark's distribution (bytes uniform, scales half(|N(0, 0.02)| / 127)),
activations are N(0, 1).  A pass is the calls that a program makes in a step, on PyTorch's current
stream, into buffers that it keeps; nothing is captured.
"""
import torch

import aotx_b200

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
SIZE_OF = {"f32": 4, "f16": 2, "bf16": 2}
# the other block types that model files are mostly made of: id -> (weights per block, bytes per
# block, offsets of the binary16 fields of a block)
BLOCKS = {2: (32, 18, (0,)), 12: (256, 144, (0, 2)), 14: (256, 210, (208,))}

_contexts = {}


def _context():
    """The library's handle: one for the device, kept for the life of the program."""
    if "ctx" not in _contexts:
        _contexts["ctx"] = aotx_b200.Q8Context(0)
    return _contexts["ctx"]


def listed():
    return [
        # one token of one sequence against a square projection: the smallest call
        {"name": "gemv_4096_m1", "kind": "product", "n": 4096, "k": 4096, "m": 1, "x": "f16", "y": "f16"},
        # a decode step of 32 sequences through one 8B-shaped layer, bfloat16 throughout
        {"name": "decode_layer_m32", "kind": "layer", "hidden": 4096, "qkv": 6144, "ffn": 14336, "m": 32,
         "x": "bf16", "y": "bf16", "fused": False},
        # the same layer as the decode graph runs it for 8 sequences: half activations, float
        # residual stream, live batch read on the device
        {"name": "decode_layer_fused_m8", "kind": "layer", "hidden": 4096, "qkv": 6144, "ffn": 14336, "m": 8,
         "x": "f16", "y": "f32", "fused": True},
        # the vocabulary projection of a decode step: the largest tensor of a model
        {"name": "lm_head_m8", "kind": "product", "n": 151936, "k": 8192, "m": 8, "x": "bf16", "y": "bf16"},
        # many sequences in one step, a batch that fills no tile
        {"name": "decode_layer_m100", "kind": "layer", "hidden": 4096, "qkv": 6144, "ffn": 14336, "m": 100,
         "x": "bf16", "y": "bf16", "fused": False},
        # a short prompt through a 4B-shaped layer, ragged, with the fused stores
        {"name": "prefill_layer_fused_m300", "kind": "layer", "hidden": 2560, "qkv": 2560, "ffn": 9728, "m": 300,
         "x": "f16", "y": "f32", "fused": True},
        # a full prompt chunk through the 8B-shaped layer: the largest amount of arithmetic
        {"name": "prefill_layer_m2048", "kind": "layer", "hidden": 4096, "qkv": 6144, "ffn": 14336, "m": 2048,
         "x": "bf16", "y": "bf16", "fused": False},
        # routed experts for a batch of 512 tokens, tensors as the model file holds them
        {"name": "experts_t512", "kind": "experts", "tokens": 512, "experts": 128, "used": 8, "hidden": 2048,
         "ffn": 768, "interleaved": False},
        # the same layer in a decode step of 8 sequences, gate and up interleaved at load
        {"name": "experts_t8", "kind": "experts", "tokens": 8, "experts": 128, "used": 8, "hidden": 2048,
         "ffn": 768, "interleaved": True},
        # a width that is no multiple of the tensor-core kernels' depth step, odd rows and batch
        {"name": "ragged_5003x2912_m7", "kind": "product", "n": 5003, "k": 2912, "m": 7, "x": "bf16", "y": "bf16"},
        # a Q4_K projection of a mixed-type model file in a decode step of 4 sequences
        {"name": "q4_k_14336x4096_m4", "kind": "blocks", "type": 12, "n": 14336, "k": 4096, "m": 4, "x": "f16",
         "y": "f32"},
        # a whole projection turned into binary16
        {"name": "dequant_14336x4096", "kind": "dequant", "rows": 14336, "k": 4096},
    ]


def _log(rng, low, high):
    return int(round(low * (high / low) ** rng.random()))


def _step(value, step):
    return max(step, value // step * step)


def draw(rng):
    kind = rng.choice(["product", "product", "product", "layer", "layer", "experts", "blocks", "dequant"])
    if kind == "product":
        x = rng.choice(["f16", "bf16"])
        n = _log(rng, 300, 40000)
        # most widths are multiples of 256, some only of the block of 32
        k = _step(_log(rng, 512, 16384), 256 if rng.random() < 0.75 else 32)
        m = _log(rng, 1, 64) if rng.random() < 0.6 or k % 256 else _log(rng, 65, 2048)
        while n * k > 160e6:
            n //= 2
        return {"kind": kind, "n": n, "k": k, "m": m, "x": x, "y": rng.choice([x, x, "f32"])}
    if kind == "layer":
        fused = rng.random() < 0.5
        hidden = _step(_log(rng, 1024, 4096), 256)
        ffn = _step(int(hidden * rng.uniform(2.5, 3.5)), 256)
        m = _log(rng, 1, 64) if rng.random() < 0.6 else _log(rng, 65, 2048)
        x = "f16" if fused else rng.choice(["f16", "bf16"])
        return {"kind": kind, "hidden": hidden, "qkv": _step(int(hidden * rng.uniform(1.0, 1.5)), 64), "ffn": ffn, "m": m,
                "x": x, "y": "f32" if fused else x, "fused": fused}
    if kind == "experts":
        experts = rng.choice([16, 32, 64, 128])
        return {"kind": kind, "tokens": _log(rng, 1, 700), "experts": experts, "used": rng.choice([2, 4, 6, 8]),
                "hidden": _step(_log(rng, 1024, 2048), 256), "ffn": rng.choice([256, 512, 768]),
                "interleaved": rng.random() < 0.5}
    if kind == "blocks":
        x = rng.choice(["f16", "bf16"])
        return {"kind": kind, "type": rng.choice(sorted(BLOCKS)), "n": _log(rng, 1000, 16000),
                "k": _step(_log(rng, 1024, 8192), 256), "m": _log(rng, 1, 32), "x": x, "y": "f32"}
    return {"kind": "dequant", "rows": _log(rng, 64, 20000), "k": _step(_log(rng, 1024, 8192), 32)}


def _rows(m, k, dtype, gen):
    return torch.randn(m, k, device="cuda", generator=gen).to(DTYPES[dtype])


def _blocks(kind, n, k, gen):
    """n rows of k weights of another block type: random codes, half scales of |N(0, 0.02)| / 16."""
    weights, size, halves = BLOCKS[kind]
    raw = torch.randint(0, 256, (n * (k // weights), size), dtype=torch.uint8, device="cuda", generator=gen)
    for at in halves:
        d = (torch.randn(raw.shape[0], device="cuda", generator=gen).abs() * (0.02 / 16.0)).half()
        raw[:, at:at + 2] = d.view(torch.uint8).view(-1, 2)
    return raw.view(-1)


def _projections(case):
    h, f = case["hidden"], case["ffn"]
    return [("qkv", case["qkv"], h), ("o", h, h), ("gate_up", 2 * f, h), ("down", h, f)]


def prepare(case, seed):
    ctx = _context()
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = dict(case, ctx=ctx)
    kind = case["kind"]
    if kind == "product":
        n, k, m = case["n"], case["k"], case["m"]
        s["w"] = aotx_b200.synth_q8_0_device(n, k, seed)
        s["x"] = _rows(m, k, case["x"], gen)
        s["y"] = torch.empty(m, n, dtype=DTYPES[case["y"]], device="cuda")
    elif kind == "layer":
        m, hidden = case["m"], case["hidden"]
        s["w"] = {name: aotx_b200.synth_q8_0_device(n, k, seed * 4 + i) for i, (name, n, k) in enumerate(_projections(case))}
        s["x"] = {name: _rows(m, k, case["x"], gen) for name, _, k in _projections(case)}
        if case["fused"]:
            s["live"] = torch.tensor([m], dtype=torch.int32, device="cuda")
            s["qkv_out"] = torch.empty(m, case["qkv"], dtype=torch.float32, device="cuda")
            s["stream"] = torch.randn(m, hidden, device="cuda", generator=gen)
            s["act"] = torch.empty(m, case["ffn"], dtype=torch.float16, device="cuda")
        else:
            s["y"] = {name: torch.empty(m, n, dtype=DTYPES[case["y"]], device="cuda") for name, n, _ in _projections(case)}
    elif kind == "experts":
        tokens, experts, hidden, ffn = case["tokens"], case["experts"], case["hidden"], case["ffn"]
        s["x"] = _rows(tokens, hidden, "f16", gen)
        s["router"] = torch.randn(experts, hidden, device="cuda", generator=gen) / hidden ** 0.5
        if case["interleaved"]:
            s["w_gate_up"] = aotx_b200.synth_q8_0_device(experts * 2 * ffn, hidden, seed * 3)
        else:
            s["w_gate"] = aotx_b200.synth_q8_0_device(experts * ffn, hidden, seed * 3)
            s["w_up"] = aotx_b200.synth_q8_0_device(experts * ffn, hidden, seed * 3 + 1)
        s["w_down"] = aotx_b200.synth_q8_0_device(experts * hidden, ffn, seed * 3 + 2)
        s["prob"] = torch.empty(tokens, experts, dtype=torch.float32, device="cuda")
        s["ids"] = torch.empty(tokens, case["used"], dtype=torch.int32, device="cuda")
        s["out"] = torch.empty(tokens, hidden, dtype=torch.float32, device="cuda")
        s["workspace"] = ctx.moe_workspace(tokens, case["used"], hidden, ffn)
    elif kind == "blocks":
        n, k, m = case["n"], case["k"], case["m"]
        s["w"] = _blocks(case["type"], n, k, gen)
        s["x"] = _rows(m, k, case["x"], gen)
        s["y"] = torch.empty(m, n, dtype=DTYPES[case["y"]], device="cuda")
    else:
        s["w"] = aotx_b200.synth_q8_0_device(case["rows"], case["k"], seed)
        s["y"] = torch.empty(case["rows"], case["k"], dtype=torch.float16, device="cuda")
    return s


def run(s):
    ctx, kind = s["ctx"], s["kind"]
    if kind == "product":
        return ctx.matmul(s["w"], s["n"], s["k"], s["x"], y=s["y"])
    if kind == "layer":
        w, x = s["w"], s["x"]
        h, f, m = s["hidden"], s["ffn"], s["m"]
        if s["fused"]:
            live = s["live"]
            ctx.matmul(w["qkv"], s["qkv"], h, x["qkv"], m=m, m_dev=live, y=s["qkv_out"])
            ctx.matmul_fused(w["o"], h, h, x["o"], aotx_b200.EPILOGUE_ADD, m=m, m_dev=live, y=s["stream"])
            ctx.matmul_fused(w["gate_up"], 2 * f, h, x["gate_up"], aotx_b200.EPILOGUE_SWIGLU, m=m, m_dev=live, y=s["act"])
            ctx.matmul_fused(w["down"], h, f, s["act"], aotx_b200.EPILOGUE_ADD, m=m, m_dev=live, y=s["stream"])
            return {"qkv": s["qkv_out"], "act": s["act"], "stream": s["stream"]}
        y = s["y"]
        ctx.matmul(w["qkv"], s["qkv"], h, x["qkv"], y=y["qkv"])
        ctx.matmul(w["o"], h, h, x["o"], y=y["o"])
        ctx.matmul(w["gate_up"], 2 * f, h, x["gate_up"], y=y["gate_up"])
        ctx.matmul(w["down"], h, f, x["down"], y=y["down"])
        return y
    if kind == "experts":
        prob, ids = ctx.moe_route(s["x"], s["router"], s["used"], prob=s["prob"], ids=s["ids"])
        if s["interleaved"]:
            out = ctx.moe_ffn_fused(s["w_gate_up"], s["w_down"], s["experts"], s["hidden"], s["ffn"], s["x"], prob, ids,
                                    out=s["out"], workspace=s["workspace"])
        else:
            out = ctx.moe_ffn(s["w_gate"], s["w_up"], s["w_down"], s["experts"], s["hidden"], s["ffn"], s["x"], prob, ids,
                              out=s["out"], workspace=s["workspace"])
        return {"prob": prob, "ids": ids, "out": out}
    if kind == "blocks":
        return ctx.matmul(s["w"], s["n"], s["k"], s["x"], y=s["y"], type=s["type"])
    return ctx.dequant(s["w"], s["k"], 0, s["rows"], out=s["y"])


def work(case):
    kind = case["kind"]
    if kind == "product":
        n, k, m = case["n"], case["k"], case["m"]
        moved = n * (k // 32) * 34 + m * k * 2 + m * n * SIZE_OF[case["y"]]
        return {"bytes": moved, "flops": 2 * m * n * k}
    if kind == "layer":
        m = case["m"]
        moved, flops = 0, 0
        for name, n, k in _projections(case):
            moved += n * (k // 32) * 34 + m * k * 2
            if not case["fused"]:
                moved += m * n * SIZE_OF[case["y"]]
            elif name == "qkv":
                moved += m * n * 4
            elif name == "gate_up":
                moved += m * (n // 2) * 2
            else:
                moved += 2 * m * n * 4
            flops += 2 * m * n * k
        return {"bytes": moved, "flops": flops}
    if kind == "experts":
        tokens, experts, used, hidden, ffn = (case[c] for c in ("tokens", "experts", "used", "hidden", "ffn"))
        hit = experts * (1.0 - (1.0 - used / experts) ** tokens)
        one = 3 * ffn * hidden // 32 * 34
        moved = hit * one + experts * hidden * 4 + tokens * (hidden * 6 + experts * 4 + used * 4)
        return {"bytes": moved, "flops": 2 * tokens * hidden * (experts + 3 * used * ffn)}
    if kind == "blocks":
        n, k, m = case["n"], case["k"], case["m"]
        weights, size, _ = BLOCKS[case["type"]]
        return {"bytes": n * (k // weights) * size + m * k * 2 + m * n * SIZE_OF[case["y"]], "flops": 2 * m * n * k}
    return {"bytes": case["rows"] * case["k"] * (34 / 32 + 2), "flops": case["rows"] * case["k"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "dequant":
        return "exact"
    if kind == "experts" or (kind == "layer" and case["fused"]):
        return {"rel": 1e-3}      # the activations between the products are binary16
    if case["x"] == "bf16" and kind != "blocks":
        return {"rel": 1e-2}      # above 128 rows the weights are rounded to bfloat16 as well
    return {"rel": {"f32": 3e-5, "f16": 1e-3, "bf16": 1e-2}[case["y"]]}   # float sums in another order
