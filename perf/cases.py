"""The work that programs give to this library, as cases that can be timed and compared.

A case is a dict of plain values; its "kind" names the piece of a program it stands for:

  decode        one projection of a decoder, one token per running sequence (1 to 16 of them), called layer by layer
  decode_block  the frozen-linear calls of one decoder layer for such a step: norm, q/k/v, o, norm, gate/up, down
  batch         one projection for a larger running batch or a short prompt (17 to 1024 tokens)
  fp32          a projection used with fp32 activations, forward and dX (the layers' default element type)
  prefill       one projection over a long prompt or a frozen training batch, forward and dX
  lora          one projection with a trainable adapter, forward and dX/dA/dB
  qkv_train     norm and q/k/v of a fine-tuned layer over shared input, forward and backward
  moe_infer     a frozen mixture-of-experts layer in inference: router, top-k, dispatch, experts, combine
  moe_train     the same layer in training: forward, backward to the input and to the router's logits
  quantize      a float weight turned into codes and scales while a model is loaded

Shapes are those of the repository's benchmark and tests (1024 x 1024; the 4096 / 1024 / 14336 projections; 2048 x 1408
experts, 64 of them, top-6) and generic ones between and around them.  Weights are N(0, 0.02) as the library's own
quantizers store them, activations and gradients N(0, 1), adapters as they look early in a fine-tune.
"""
import math

import torch

from caif_b200 import native as nv

STORAGE = {"int4": nv.I4, "int8": nv.I8}
DTYPE = {"f32": torch.float32, "bf16": torch.bfloat16}
COMPUTE = {"f32": nv.F32, "bf16": nv.BF16}


def listed():
    return [
        # the smallest call there is: one token through one small projection
        {"name": "decode_1024_m1", "kind": "decode", "storage": "int4", "in": 1024, "out": 1024, "m": 1, "layers": 1,
         "group": 128, "compute": "bf16", "y": "f32"},
        # a few sequences through the wide FFN projection of successive layers (242 MB of codes: nothing stays in L2)
        {"name": "decode_ffn_m4", "kind": "decode", "storage": "int4", "in": 4096, "out": 14336, "m": 4, "layers": 8,
         "group": 128, "compute": "bf16", "y": "f32"},
        # a whole decoder layer, five sequences
        {"name": "decode_block_m5", "kind": "decode_block", "storage": "int4", "hidden": 4096, "kv": 1024, "ffn": 14336,
         "m": 5, "group": 128},
        # continuous batching: 96 sequences
        {"name": "batch_m96", "kind": "batch", "storage": "int4", "in": 4096, "out": 14336, "m": 96, "group": 128,
         "compute": "bf16", "y": "bf16"},
        # the fp32 layer, small
        {"name": "fp32_1024_m64", "kind": "fp32", "storage": "int8", "in": 1024, "out": 1024, "m": 64, "group": 128},
        # a long prompt of odd length / a frozen layer inside a training graph
        {"name": "prefill_m2047", "kind": "prefill", "storage": "int4", "in": 4096, "out": 14336, "m": 2047,
         "group": 128, "compute": "bf16"},
        # the training shape with an int8 base: batch 4 x seq 2048, fp32 compute
        {"name": "lora_int8_m8192", "kind": "lora", "storage": "int8", "in": 4096, "out": 4096, "m": 8192, "rank": 16,
         "group": 128, "compute": "f32"},
        # a short ragged batch through the down projection, int4 base
        {"name": "lora_int4_m1000", "kind": "lora", "storage": "int4", "in": 14336, "out": 4096, "m": 1000, "rank": 16,
         "group": 128, "compute": "bf16"},
        # the attention inputs of a fine-tuned layer
        {"name": "qkv_train_m4096", "kind": "qkv_train", "storage": "int4", "hidden": 4096, "kv": 1024, "m": 4096,
         "group": 128},
        # an expert layer while decoding: every expert sees a row or two
        {"name": "moe_infer_t16", "kind": "moe_infer", "storage": "int4", "hidden": 2048, "ffn": 1408, "experts": 64,
         "topk": 6, "tokens": 16, "group": 128},
        # the expert layer of a training step
        {"name": "moe_train_t16384", "kind": "moe_train", "storage": "int4", "hidden": 2048, "ffn": 1408,
         "experts": 64, "topk": 6, "tokens": 16384, "group": 128},
        # loading: the widest projection
        {"name": "quantize_int4_ffn", "kind": "quantize", "storage": "int4", "rows": 14336, "cols": 4096, "group": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dim(rng, lo, hi, step=128):
    return max(lo, min(hi, step * int(round(_log(rng, lo, hi) / step))))


def draw(rng):
    kind = rng.choice(["decode", "decode_block", "batch", "fp32", "prefill", "lora", "qkv_train", "moe_infer",
                       "moe_train", "quantize"])
    storage = rng.choice(["int4", "int8"])
    case = {"kind": kind, "storage": storage, "group": 128}
    if kind == "decode":
        # (feature counts need not be multiples of a tile while decoding: heads, vocabularies, shards)
        case.update({"in": _dim(rng, 512, 14336), "out": _dim(rng, 512, 16384, 8), "m": _log(rng, 1, 16),
                     "layers": rng.choice([1, 2, 8]), "compute": rng.choice(["bf16", "f32"]),
                     "y": rng.choice(["f32", "bf16"])})
    elif kind == "decode_block":
        hidden = _dim(rng, 1024, 6144, 256)
        case.update({"hidden": hidden, "kv": 128 * max(1, hidden // rng.choice([128, 512, 1024])),
                     "ffn": 128 * int(round(hidden * rng.uniform(2.5, 4.0) / 128)), "m": _log(rng, 1, 16)})
    elif kind == "batch":
        case.update({"in": _dim(rng, 512, 14336), "out": _dim(rng, 512, 14336), "m": _log(rng, 17, 1024),
                     "compute": rng.choice(["bf16", "f32"]), "y": rng.choice(["f32", "bf16"])})
    elif kind == "fp32":
        case.update({"in": _dim(rng, 512, 4096), "out": _dim(rng, 512, 4096), "m": _log(rng, 1, 1024)})
    elif kind == "prefill":
        case.update({"in": _dim(rng, 1024, 14336), "out": _dim(rng, 1024, 14336), "m": _log(rng, 1025, 8192),
                     "compute": rng.choice(["bf16", "f32"])})
    elif kind == "lora":
        case.update({"in": _dim(rng, 1024, 14336), "out": _dim(rng, 1024, 14336), "m": _log(rng, 64, 8192),
                     "rank": rng.choice([8, 16, 16, 32, 64]), "compute": "f32" if storage == "int8" else "bf16"})
    elif kind == "qkv_train":
        hidden = _dim(rng, 1024, 6144, 256)
        case.update({"hidden": hidden, "kv": 128 * max(1, hidden // rng.choice([128, 512, 1024])),
                     "m": _log(rng, 64, 8192)})
    elif kind in ("moe_infer", "moe_train"):
        case.update({"hidden": _dim(rng, 1024, 4096), "ffn": _dim(rng, 512, 2048),
                     "experts": rng.choice([8, 16, 32, 64]), "topk": rng.choice([2, 4, 6]),
                     "tokens": _log(rng, 1, 1024) if kind == "moe_infer" else _log(rng, 512, 8192)})
    else:
        case.update({"storage": rng.choice(["int4", "int8", "int8_channel"]), "rows": _log(rng, 256, 14336),
                     "cols": _dim(rng, 512, 4096), "group": rng.choice([64, 128])})
    # no drawn case is more work than the largest listed one
    if kind in ("prefill", "lora"):
        case["m"] = min(case["m"], int(8e11) // (case["in"] * case["out"]))
    elif kind == "moe_train":
        case["tokens"] = min(case["tokens"], int(2.8e11) // (case["topk"] * case["hidden"] * case["ffn"]))
    return case


# ---------------------------------------------------------------- what a program has in hand

class _Source:
    def __init__(self, seed):
        self.dev = torch.device("cuda")
        self.gen = torch.Generator(device=self.dev).manual_seed(seed)

    def normal(self, *shape, dtype=torch.bfloat16, std=1.0):
        t = torch.randn(*shape, generator=self.gen, device=self.dev)
        return (t.mul_(std) if std != 1.0 else t).to(dtype)

    def weight(self, out_dim, in_dim, storage, group):
        return self.weights(1, out_dim, in_dim, storage, group)[0]

    def weights(self, count, out_dim, in_dim, storage, group):
        """`count` frozen weights of one shape; int4 ones are slices of one quantized stack, as a loader leaves them."""
        if storage == "int4":
            codes, scales = nv.quantize_int4(self.normal(count * out_dim * in_dim, dtype=torch.float32, std=0.02), group)
            n, g = out_dim * in_dim // 2, out_dim * in_dim // group
            return [nv.Weight(codes[i * n:(i + 1) * n], nv.I4, in_dim, out_dim, scales[i * g:(i + 1) * g],
                              group_size=group) for i in range(count)]
        out = []
        for _ in range(count):
            q, s = nv.quantize_int8_per_tensor(self.normal(out_dim, in_dim, dtype=torch.float32, std=0.02))
            out.append(nv.Weight(q, nv.I8, in_dim, out_dim, s))
        return out


def prepare(case, seed):
    kind, g, st = case["kind"], case["group"], case["storage"]
    src = _Source(seed)
    s = dict(case)
    if kind == "decode":
        s["w"] = src.weights(case["layers"], case["out"], case["in"], st, g)
        s["x"] = [src.normal(case["m"], case["in"]) for _ in s["w"]]
    elif kind in ("batch", "prefill"):
        s["w"] = src.weight(case["out"], case["in"], st, g)
        s["x"] = src.normal(case["m"], case["in"])
        if kind == "prefill":
            s["dy"] = src.normal(case["m"], case["out"])
    elif kind == "fp32":
        s["w"] = src.weight(case["out"], case["in"], st, g)
        s["x"] = src.normal(case["m"], case["in"], dtype=torch.float32)
        s["dy"] = src.normal(case["m"], case["out"], dtype=torch.float32)
    elif kind == "decode_block":
        h, kv, f = case["hidden"], case["kv"], case["ffn"]
        s["qkv"] = [src.weight(o, h, st, g) for o in (h, kv, kv)]
        s["o"] = src.weight(h, h, st, g)
        s["gate_up"] = [src.weight(f, h, st, g) for _ in range(2)]
        s["down"] = src.weight(h, f, st, g)
        s["gamma"] = [1.0 + src.normal(h, dtype=torch.float32, std=0.1) for _ in range(2)]
        s["stream"] = src.normal(case["m"], h)      # the residual stream, updated in place by o and down
        s["attn"] = src.normal(case["m"], h)        # attention and the activation lie between the library's calls
        s["act"] = src.normal(case["m"], f)
    elif kind == "lora":
        s["w"] = src.weight(case["out"], case["in"], st, g)
        a = src.normal(case["rank"], case["in"], std=1.0 / math.sqrt(case["in"]))
        b = src.normal(case["out"], case["rank"], std=1e-2)
        s["lora"] = nv.Lora(a, b, 2.0 * case["rank"])
        s["x"] = src.normal(case["m"], case["in"])
        s["dy"] = src.normal(case["m"], case["out"])
        # the scratch that a layer keeps
        c = COMPUTE[case["compute"]]
        s["ws"] = [torch.empty(max(1, f(s["w"], s["lora"], case["m"], c, True)), dtype=torch.uint8, device=src.dev)
                   for f in (nv.lora_fwd_workspace_bytes, nv.lora_bwd_workspace_bytes)]
    elif kind == "qkv_train":
        h, kv = case["hidden"], case["kv"]
        s["w"] = [src.weight(o, h, st, g) for o in (h, kv, kv)]
        s["gamma"] = 1.0 + src.normal(h, dtype=torch.float32, std=0.1)
        s["x"] = src.normal(case["m"], h)
        s["dy"] = src.normal(case["m"], h + 2 * kv)
        s["ws"] = torch.empty((h + 2 * kv) * h * 2 + 256, dtype=torch.uint8, device=src.dev)
    elif kind in ("moe_infer", "moe_train"):
        h, f, e = case["hidden"], case["ffn"], case["experts"]
        s["gate"], s["up"] = (src.weights(e, f, h, st, g) for _ in range(2))
        s["down"] = src.weights(e, h, f, st, g)
        router = src.normal(e, h, std=1.0 / math.sqrt(h))
        s["router"] = nv.Weight(router, nv.BF16, h, e)
        s["x"] = src.normal(case["tokens"], h)
        if kind == "moe_train":
            s["dy"] = src.normal(case["tokens"], h)
            # scratch for the experts' bf16 copies, filled once per step
            n = nv.grouped_expert_expanded_bytes(s["gate"], s["up"], s["down"], nv.BF16, nv.BF16)
            s["expanded"] = torch.empty(n, dtype=torch.uint8, device=src.dev) if n else None
    else:
        s["wf"] = src.normal(case["rows"], case["cols"], dtype=torch.float32, std=0.02)
    return s


# ---------------------------------------------------------------- one pass

def _moe_forward(s, expanded):
    """The layer's forward as its owner writes it: the expert offsets are read back to size the packed rows."""
    tokens = s["tokens"]
    logits = nv.linear_fwd(s["router"], s["x"], torch.float32)
    probs = nv.moe_softmax(logits)
    idx, val = nv.moe_topk(probs, s["topk"])
    wts = nv.cast(nv.moe_normalize_rows(val), torch.bfloat16)
    dmap, offs = nv.moe_build_dispatch(idx, s["experts"])
    host = offs.tolist()
    buf = nv.moe_dispatch(s["x"], idx, dmap, offs, host[-1])
    out, g_out, u_out = nv.grouped_expert_fwd(s["gate"], s["up"], s["down"], host, buf, nv.BF16, expanded)
    y = nv.moe_combine(out, idx, wts, dmap, offs, tokens)
    return y, (probs, idx, wts, dmap, offs, host, out, g_out, u_out)


def run(s):
    kind = s["kind"]
    if kind == "decode":
        return [nv.linear_fwd(w, x, DTYPE[s["y"]], COMPUTE[s["compute"]]) for w, x in zip(s["w"], s["x"])]
    if kind == "batch":
        return nv.linear_fwd(s["w"], s["x"], DTYPE[s["y"]], COMPUTE[s["compute"]])
    if kind == "fp32":
        return nv.linear_fwd(s["w"], s["x"]), nv.linear_dx(s["w"], s["dy"])
    if kind == "prefill":
        c = COMPUTE[s["compute"]]
        return nv.linear_fwd(s["w"], s["x"], torch.bfloat16, c), nv.linear_dx(s["w"], s["dy"], torch.bfloat16, c)
    if kind == "decode_block":
        n1, _ = nv.rmsnorm_fwd(s["stream"], s["gamma"][0])
        qkv = nv.linear_fwd_multi(s["qkv"], n1, torch.bfloat16, nv.BF16)
        nv.linear_fwd_residual(s["o"], s["attn"], s["stream"], nv.BF16)
        n2, _ = nv.rmsnorm_fwd(s["stream"], s["gamma"][1])
        gate_up = nv.linear_fwd_multi(s["gate_up"], n2, torch.bfloat16, nv.BF16)
        return qkv, gate_up, nv.linear_fwd_residual(s["down"], s["act"], s["stream"], nv.BF16)
    if kind == "lora":
        c = COMPUTE[s["compute"]]
        y, hidden = nv.lora_linear_fwd(s["w"], s["lora"], s["x"], c, workspace=s["ws"][0], expanded=True)
        dx, d_a, d_b = nv.lora_linear_bwd(s["w"], s["lora"], s["dy"], s["x"], hidden, c, workspace=s["ws"][1],
                                          expanded=True)
        return y, hidden, dx, d_a, d_b
    if kind == "qkv_train":
        n, rms = nv.rmsnorm_fwd(s["x"], s["gamma"])
        y = nv.linear_concat(s["w"], n, workspace=s["ws"])
        dn = nv.linear_concat(s["w"], s["dy"], backward=True, workspace=s["ws"])
        dx, d_gamma = nv.rmsnorm_bwd(dn, s["x"], s["gamma"], rms)
        return y, dx, d_gamma
    if kind == "moe_infer":
        return _moe_forward(s, None)[0]
    if kind == "moe_train":
        if s["expanded"] is not None:
            nv.grouped_expert_expand(s["gate"], s["up"], s["down"], s["expanded"], nv.BF16, nv.BF16)
        y, (probs, idx, wts, dmap, offs, host, out, g_out, u_out) = _moe_forward(s, s["expanded"])
        d_buf = nv.moe_combine_bwd_grad_expert(s["dy"], idx, wts, dmap, offs, host[-1])
        d_wts = nv.moe_combine_bwd_grad_weights(s["dy"], out, idx, dmap, offs)
        d_in = nv.grouped_expert_bwd(s["gate"], s["up"], s["down"], host, d_buf, g_out, u_out, nv.BF16, s["expanded"])
        dx = nv.moe_dispatch_bwd(d_in, idx, dmap, offs, s["tokens"])
        d_logits, _ = nv.moe_router_bwd(nv.cast(d_wts, torch.float32), probs, idx)
        return y, dx, d_logits
    if s["storage"] == "int4":
        return nv.quantize_int4(s["wf"], s["group"])
    if s["storage"] == "int8":
        return nv.quantize_int8_per_tensor(s["wf"])
    return nv.quantize_int8_per_channel(s["wf"])


# ---------------------------------------------------------------- what a pass cannot do without

def _weight_bytes(storage, n, group):
    return n / 2 + 2 * n / group if storage == "int4" else n


def work(case):
    kind, st, g = case["kind"], case["storage"], case["group"]
    if kind == "quantize":
        n = case["rows"] * case["cols"]
        return {"bytes": 4 * n + _weight_bytes(st, n, g), "flops": 0}
    if kind in ("decode", "batch", "fp32", "prefill", "lora"):
        m, i, o = case["m"], case["in"], case["out"]
        wb = _weight_bytes(st, i * o, g)
        if kind in ("decode", "batch"):
            layers = case.get("layers", 1)
            return {"bytes": layers * (wb + 2 * m * i + (4 if case["y"] == "f32" else 2) * m * o),
                    "flops": layers * 2 * m * i * o}
        if kind == "lora":
            # in: x, dy, hidden as saved, factors; out: y, hidden, dx, dA, dB
            r = case["rank"]
            return {"bytes": wb + 4 * m * (i + o) + 2 * m * r + 4 * r * (i + o), "flops": 4 * m * i * o + 6 * m * r * (i + o)}
        e = 4 if kind == "fp32" else 2
        return {"bytes": wb + 2 * e * m * (i + o), "flops": 4 * m * i * o}
    if kind == "decode_block":
        m, h, kv, f = case["m"], case["hidden"], case["kv"], case["ffn"]
        n = h * (h + 2 * kv) + h * h + 3 * h * f
        return {"bytes": _weight_bytes(st, n, g) + 8 * h + 2 * m * (2 * h + f) + 2 * m * (h + 2 * kv + 2 * f + h),
                "flops": 2 * m * n}
    if kind == "qkv_train":
        m, h, o = case["m"], case["hidden"], case["hidden"] + 2 * case["kv"]
        return {"bytes": _weight_bytes(st, h * o, g) + 2 * m * (2 * h + 2 * o) + 8 * h, "flops": 4 * m * h * o}
    t, h, f, e, k = case["tokens"], case["hidden"], case["ffn"], case["experts"], case["topk"]
    hit = e * (1.0 - (1.0 - k / e) ** t)     # experts that at least one token picks
    wb = hit * _weight_bytes(st, 3 * h * f, g) + 2 * e * h
    flops = 6 * t * k * h * f + 2 * t * h * e
    if kind == "moe_infer":
        return {"bytes": wb + 4 * t * h, "flops": flops}
    return {"bytes": wb + 8 * t * h + 4 * t * e, "flops": 12 * t * k * h * f + 2 * t * h * e}


def tolerance(case):
    kind = case["kind"]
    if kind == "quantize":
        return "exact"      # codes and scales are whole values of a storage format
    if kind == "fp32":
        return {"rel": 1e-5}
    if kind in ("decode", "batch", "prefill") and case["compute"] == "f32":
        # the int4 weight may enter as two bf16 terms (2^-17 relative); a bf16 result is rounded once
        return {"rel": 2e-5} if case.get("y") == "f32" else {"rel": 4e-3}
    if kind == "moe_train":
        return {"rel": 2e-2}    # two chains of three bf16 products, and differences of nearly equal terms
    return {"rel": 1e-2}
