"""The work this library is timed on: the MoE block of one model shape, from a single decode row to
a 32768-row prefill, through the public entry points of `ane_fieldfare_b200.hotpath`.

A case is a dict:
  path    how a program calls the block, once for each of its resident layers:
            "layer"      HotpathContext.moeLayer, one call after the other
            "graph"      the same calls captured in a CUDA graph that the program replays
            "host"       HotpathContext.moeLayerHost on page-locked host rows
            "stack"      HotpathContext.moeStack, the block behind its RMSNorm
            "operators"  the separate operators of a model's forward: the fused setup behind attention,
                         router, shared FFN and routed experts on their three inputs, combine, layer tail
  tokens  rows of a call: 1 decode, 2..16 a verify block, more prefill
  layers  resident layers, each with a router, a shared FFN, input and output rows of its own (the rows
          are not chained: in a model, attention stands between two blocks)
  form    "int4": bf16 router and INT4 shared FFN (the benchmark configurations); "int8": INT8 affine
          router with effective scale and per-expert gain, and INT8 shared FFN (the shipped checkpoints)
  skew    how uneven the routing is: "none", "normal" (N(0,1) per expert) or "zipf" (log of a Zipf(1.1)
          prior), an additive bias of the router's logits as in the benchmark configurations
"""
import math

import numpy as np
import torch

from ane_fieldfare_b200 import gturbo, hotpath, synth

# the benchmark configurations' model shape
D, F, FS, E, K = 2816, 704, 2112, 128, 8
EPS = 1e-6


def listed():
    def case(name, path, tokens, layers, form, skew):
        return {"name": name, "path": path, "tokens": tokens, "layers": layers, "form": form, "skew": skew}

    return [
        # the smallest call a program makes: one row through one layer, where launches and latency count
        case("decode call", "layer", 1, 1, "int4", "none"),
        # a decode loop: one token through a model's layers (more of them than L2 holds), replayed as a graph
        case("decode graph", "graph", 1, 8, "int4", "none"),
        # decode for a caller with host rows: row in, row out, complete on return
        case("decode host", "host", 1, 4, "int4", "none"),
        # a decode step of a model's forward on the shipped checkpoint's forms
        case("decode forward int8", "operators", 1, 4, "int8", "none"),
        # a short speculative block
        case("verify 5", "layer", 5, 4, "int4", "normal"),
        # the largest speculative block (benchmark configuration 2)
        case("verify 16", "layer", 16, 4, "int4", "normal"),
        # a short prompt: nearly every expert is used by a few rows
        case("prefill 77", "layer", 77, 2, "int4", "zipf"),
        # a chunk of a prompt in a model's forward, shipped forms
        case("prefill forward int8 613", "operators", 613, 2, "int8", "zipf"),
        # an ordinary prompt
        case("prefill 1500", "layer", 1500, 1, "int4", "normal"),
        # an ordinary prompt on the shipped forms
        case("prefill int8 2000", "layer", 2000, 1, "int8", "zipf"),
        # benchmark configuration 3
        case("prefill 4096", "layer", 4096, 1, "int4", "zipf"),
        # benchmark configuration 4's rows through some of its layers, RMSNorm included
        case("stack 32768", "stack", 32768, 3, "int4", "zipf"),
    ]


def draw(rng):
    regime = rng.choice(["decode", "verify", "prefill", "prefill"])
    if regime == "decode":
        tokens, layers = 1, rng.randint(1, 8)
        path = rng.choice(["layer", "graph", "host", "stack", "operators"])
    elif regime == "verify":
        tokens, layers = rng.randint(2, 16), rng.randint(1, 6)
        path = rng.choice(["layer", "graph", "host", "stack", "operators"])
    else:
        tokens, layers = int(math.exp(rng.uniform(math.log(17), math.log(6000)))), rng.randint(1, 2)
        path = rng.choice(["layer", "layer", "host", "stack", "operators"])
    return {"path": path, "tokens": tokens, "layers": layers, "form": rng.choice(["int4", "int4", "int8"]),
            "skew": rng.choice(["none", "normal", "zipf"])}


# ---- inputs ----------------------------------------------------------------------------------


def _bits(t):
    """bf16 tensor -> its bit patterns on the host."""
    return hotpath.bf16_numpy(t)


def _int4_blobs(gen, dev, count, f):
    """`count` blobs of gate, up and down as the layer files hold them: codes uniform in 0..15, scale
    0.002 + U(0, 0.01), bias -scale * U(6, 10)."""
    lay = gturbo.expert_layout(D, f)
    blobs = torch.zeros((count, lay.stride), dtype=torch.uint8, device=dev)
    off = lay.offsets.as_tuple()
    codes, groups = D * f // 2, D * f // 64
    for m in range(3):
        w, s, b = off[3 * m:3 * m + 3]
        blobs[:, w:w + codes] = torch.randint(0, 256, (count, codes), dtype=torch.uint8, device=dev, generator=gen)
        scale = (0.002 + 0.01 * torch.rand((count, groups), device=dev, generator=gen)).bfloat16()
        bias = (-scale.float() * (6 + 4 * torch.rand((count, groups), device=dev, generator=gen))).bfloat16()
        blobs[:, s:s + 2 * groups] = scale.view(torch.uint8)
        blobs[:, b:b + 2 * groups] = bias.view(torch.uint8)
    return lay, blobs.cpu().numpy()


def _int8_matrix(gen, dev, rows, cols):
    """(codes, scale bits, bias bits) of weights about as large as the INT4 ones."""
    codes = torch.randint(0, 256, (rows, cols), dtype=torch.uint8, device=dev, generator=gen)
    scale = ((0.002 + 0.01 * torch.rand((rows, cols // 64), device=dev, generator=gen)) / 16).bfloat16()
    bias = (-scale.float() * (96 + 64 * torch.rand(scale.shape, device=dev, generator=gen))).bfloat16()
    return codes.cpu().numpy(), _bits(scale), _bits(bias)


def _int8_router(gen, dev):
    amp = 3.0 / math.sqrt(D)
    codes = torch.randint(0, 256, (E, D), dtype=torch.uint8, device=dev, generator=gen)
    scale = ((0.5 + torch.rand((E, D // 64), device=dev, generator=gen)) * (2 * amp / 255)).bfloat16()
    bias = (-scale.float() * (120 + 15 * torch.rand(scale.shape, device=dev, generator=gen))).bfloat16()
    return codes.cpu().numpy(), _bits(scale), _bits(bias)


def _logit_bias(skew, seed, layer):
    if skew == "none":
        return None
    if skew == "normal":
        return synth.normal(synth.seedtree_key(seed, f"bias.{layer}"), E).astype(np.float32)
    return synth.zipf_log_prior(E, 1.1, seed, f"zipf.{layer}")


def _rows(gen, dev, layers, tokens):
    x = torch.randn((layers, tokens, D), device=dev, generator=gen, dtype=torch.float32).bfloat16()
    return [x[i] for i in range(layers)]


def prepare(case, seed):
    tokens, layers, path = case["tokens"], case["layers"], case["path"]
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    ctx = hotpath.HotpathContext(layers=layers, experts=E, d=D, f=F, sharedF=FS, topK=K, maxTokens=max(16, tokens),
                                 device=dev.index)
    lay, blobs = _int4_blobs(gen, dev, E, F)
    for i in range(layers):
        # (every layer slot has memory of its own; the routed bytes repeat so that preparing stays quick)
        ctx.loadLayer(i, blobs, lay.stride, lay.offsets)
        bias = _logit_bias(case["skew"], seed, i)
        if case["form"] == "int8":
            ctx.loadSharedInt8(i, _int8_matrix(gen, dev, FS, D), _int8_matrix(gen, dev, FS, D), _int8_matrix(gen, dev, D, FS))
            eff = (0.5 + torch.rand(D, device=dev, generator=gen)).bfloat16()
            gain = (0.5 + torch.rand(E, device=dev, generator=gen)).bfloat16()
            ctx.loadRouterInt8(i, *_int8_router(gen, dev), effectiveScale=_bits(eff), perExpertScale=_bits(gain), logitBias=bias)
        else:
            sharedLay, shared = _int4_blobs(gen, dev, 1, FS)
            ctx.loadShared(i, *[gturbo.sub_tensor(shared[0], sharedLay, role) for role in gturbo.ROLES])
            router = 0.02 * torch.randn((E, D), device=dev, generator=gen)
            ctx.loadRouter(i, _bits(router.bfloat16()), logitBias=bias)
    x = _rows(gen, dev, layers, tokens)
    s = {"case": case, "ctx": ctx, "x": x, "layers": layers, "tokens": tokens}
    if path == "host":
        s["x"] = [t.cpu().pin_memory() for t in x]
        s["y"] = [torch.empty((tokens, D), dtype=torch.bfloat16).pin_memory() for _ in range(layers)]
    elif path == "operators":
        # the residual stream and the attention output of each layer, and a model's buffers
        s["attn"] = _rows(gen, dev, layers, tokens)
        s["norms"] = [[(1 + 0.1 * torch.randn(D, device=dev, generator=gen)).bfloat16() for _ in range(5)] for _ in range(layers)]
        s["hidden"] = [torch.empty_like(t) for t in x]
        s["ids"] = [torch.empty((tokens, K), dtype=torch.int32, device=dev) for _ in range(layers)]
        row = lambda n=tokens: torch.empty((n, D), dtype=torch.bfloat16, device=dev)  # noqa: E731
        s["denseX"], s["routedX"], s["routerX"], s["h1"], s["h2"] = row(), row(), row(), row(), row()
        s["weights"] = torch.empty((tokens, K), dtype=torch.bfloat16, device=dev)
        s["partials"] = row(tokens * K)
        s["ops"] = (hotpath.MoE(ctx), hotpath.PrefillRouter(ctx), hotpath.PrefillSharedExpert(ctx),
                    hotpath.PrefillGroupedRoutedMoE(ctx), hotpath.PrefillMoE(ctx), hotpath.PrefillLayerGlue(ctx))
    else:
        s["y"] = [torch.empty_like(t) for t in x]
        if path == "graph":
            _layers(s)  # once, so that every kernel is set up before the capture
            torch.cuda.synchronize()
            s["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["graph"]):
                _layers(s)
    return s


# ---- one pass ----------------------------------------------------------------------------------


def _layers(s):
    for i in range(s["layers"]):
        s["ctx"].moeLayer(i, s["x"][i], s["y"][i])


def _forward_layer(s, i):
    """One layer of a model's forward behind attention, operator by operator."""
    moe, router, shared, routed, combine, glue = s["ops"]
    tokens, hidden, ids, weights = s["tokens"], s["hidden"][i], s["ids"][i], s["weights"]
    wPostAttn, wPreFfn, wPreFfn2, wPostFfn2, wPostFfn = s["norms"][i]
    hidden.copy_(s["x"][i])  # the residual stream arrives (the operators below update it in place)
    glue.encodePostAttnSetupBlock(None, hidden, s["attn"][i], wPostAttn, wPreFfn, wPreFfn2, EPS, s["denseX"], s["routedX"],
                                  s["routerX"])
    if tokens == 1:
        moe.encodeRouterGemma4(None, i, s["routerX"], ids, weights)
        shared.encode(None, i, s["denseX"], s["h1"])
        moe.encodeRoutedPersistentGPUSlots(None, i, ids, s["routedX"], weights, None, s["h2"])
    else:
        router.encodeGemma4Block(None, i, s["routerX"], ids, weights, tokens)
        shared.encodeBlock(None, i, s["denseX"], s["h1"], tokens)
        if tokens <= routed.verifyMaxRows:
            routed.encodeVerifyBound(None, i, s["routedX"], ids, s["partials"], tokens)
        else:
            routed.encodeStreamedBatched(None, i, s["routedX"], ids, s["partials"], tokens)
        combine.encodeReduceTokenMajor(None, s["partials"], weights, s["h2"], tokens)
    glue.encodeLayerTailBlock(None, s["h2"], s["h1"], hidden, wPostFfn2, wPostFfn, EPS, 0.75)


def run(s):
    path = s["case"]["path"]
    if path == "operators":
        for i in range(s["layers"]):
            _forward_layer(s, i)
        return {"hidden": s["hidden"], "ids": s["ids"]}
    if path == "graph":
        s["graph"].replay()
    elif path == "layer":
        _layers(s)
    elif path == "host":
        for i in range(s["layers"]):
            s["ctx"].moeLayerHost(i, s["x"][i], s["y"][i])
    else:
        for i in range(s["layers"]):
            s["ctx"].moeStack(i, 1, s["x"][i], EPS, s["y"][i])
    return s["y"]


# ---- what a pass cannot do without ---------------------------------------------------------------


def _active_experts(tokens, skew):
    """Experts that `tokens` rows use, on average: from every expert's chance of being in a row's top K."""
    rng = np.random.RandomState(1)
    bias = np.zeros(E)
    if skew == "normal":
        bias = rng.randn(E)
    elif skew == "zipf":
        bias = -1.1 * np.log(np.arange(1, E + 1))
    logits = 0.02 * math.sqrt(D) * rng.randn(2048, E) + bias
    top = np.argpartition(-logits, K - 1, axis=1)[:, :K]
    p = np.bincount(top.ravel(), minlength=E) / 2048.0
    return float(np.sum(1 - (1 - p) ** tokens))


def work(case):
    tokens, layers = case["tokens"], case["layers"]

    def ffn(f, bits):
        return 3 * (f * D * bits // 8 + 2 * (f * D // 64) * 2)

    wide = case["form"] == "int8"
    weights = _active_experts(tokens, case["skew"]) * ffn(F, 4) + ffn(FS, 8 if wide else 4)
    weights += E * D + 4 * E * (D // 64) + 2 * D if wide else 2 * E * D
    rows = 3 if case["path"] == "operators" else 2  # residual stream and attention in, residual stream out
    flops = 2 * tokens * (3 * K * F * D + 3 * FS * D + E * D)
    return {"bytes": layers * (weights + rows * tokens * D * 2), "flops": layers * flops}


def tolerance(case):
    # bf16 rows out of bf16-rounded activations; the expert ids (whole values) are equal
    return {"rel": 1e-2}
