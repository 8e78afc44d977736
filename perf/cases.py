"""The expert-FFN work that a program gives this library, as a list of cases to time and to compare.

Three ways into the library, each on layers of the model's own shape (hidden 2048, intermediate 512, 256 routed experts and
a shared one, top-8):
  stack   residual blocks chained by moe_b200.Stack and replayed once per decode step (`host`: through pinned host buffers)
  layers  one moe_b200.Layer.forward per layer, as an engine calls it between its attention blocks; every layer gets a batch
          of its own (`block`: with the norm before and the residual after; `ids`: the selected experts are wanted too)
  engine  the pointer-level calls in the order the reference engine makes them for a chunk, on reference-layout blobs:
          router rows, top-k, grouping by expert, experts, combine, shared expert
Formats: "sym_f16" (int4, fp16 scale per 64), "sym_f32" (int4, f32 scale per 64: the reference container), "zp" (GGUF Q4_K as
zero-point blobs). Weights, router and tokens are made on the GPU from the seed.
"""
import math

import torch

import moe_b200 as m

E, K, EH = 256, 8, 2048
DEV = "cuda:0"
FMT = {"sym_f32": m.FMT_SYM_F32, "sym_f16": m.FMT_SYM_F16, "zp": m.FMT_ZP}
BLOB = {"sym_f32": 1769472, "sym_f16": 1671168, "zp": 1818624}


def case(way, tokens, layers, fmt="sym_f16", x="f32", router="f32", **options):
    c = {"way": way, "tokens": tokens, "layers": layers, "fmt": fmt, "x": x, "router": router, "host": False, "block": False, "ids": False}
    c.update(options)
    return c


def listed():
    def named(name, *a, **k):
        return dict(case(*a, **k), name=name)

    return [
        # the smallest call: one token through one layer, as an engine makes it between two attention blocks
        named("layer-1", "layers", 1, 1),
        # one decode step of one user over the whole 40-layer model, activations on the device
        named("stack-1", "stack", 1, 40),
        # the same for a Q4_K model whose engine keeps the activations on the host
        named("stack-1-q4k-host", "stack", 1, 40, "zp", host=True),
        # speculative verification: four tokens through the model
        named("stack-4", "stack", 4, 40),
        # a serving step: 64 users at once, bf16 tokens
        named("stack-64-bf16", "stack", 64, 40, x="bf16"),
        # a ragged serving step layer by layer, experts as the reference container holds them, F16 router, ids wanted
        named("layers-23-f32s", "layers", 23, 8, "sym_f32", router="f16", block=True, ids=True),
        # many users, or a short prompt: between the decode batch and the prefill chunk
        named("layers-160-bf16", "layers", 160, 4, x="bf16"),
        # a full prefill chunk
        named("prefill-2048-bf16", "layers", 2048, 1, x="bf16"),
        # the rest of a prompt: not a multiple of anything, f32 tokens, container scales, as a residual block
        named("prefill-777-f32s", "layers", 777, 1, "sym_f32", router="f16", block=True),
        # a prompt on a Q4_K model
        named("prefill-512-q4k", "layers", 512, 2, "zp"),
        # the reference engine's own calls: a chunk of 16 tokens, then one token, on blobs in the reference layout
        named("engine-16", "engine", 16, 2, "sym_f32", router="f16"),
        named("engine-1", "engine", 1, 2, "sym_f32", router="f16"),
    ]


def draw(rng):
    """One more case: tokens over their whole range by logarithm, every format, input type and option."""
    def tokens(most):
        return min(most, int(math.exp(rng.uniform(0.0, math.log(most + 1)))))

    way = rng.choice(["stack", "layers", "layers", "layers", "engine"])
    common = {"fmt": rng.choice(["sym_f16", "sym_f16", "sym_f32", "zp"]), "router": rng.choice(["f32", "f16"])}
    if way == "stack":
        # up to 36 layers of the largest format hold no more than 40 of the usual one
        return case("stack", tokens(64), rng.randint(6, 36), x=rng.choice(["f32", "bf16"]), host=rng.random() < 0.4, **common)
    if way == "layers":
        t = tokens(2048)
        return case("layers", t, rng.randint(1, max(1, min(8, 1024 // t))), x=rng.choice(["f32", "bf16"]), block=rng.random() < 0.4,
                    ids=rng.random() < 0.3, **common)
    # the reference engine's router is F16
    return case("engine", tokens(64), rng.randint(1, 4), fmt=common["fmt"], router="f16")


class Model:
    """What a program keeps: the context, the resident layers, for a stack its handle; closed in order when it goes."""

    def __init__(self):
        self.stack, self.layers, self.ctx = None, [], None

    def __del__(self):
        try:
            for part in [self.stack] + self.layers + [self.ctx]:
                if part is not None:
                    part.close()
        except (AttributeError, TypeError):   # the interpreter is shutting down
            pass


_engine_ctx = None


def engine_context():
    """The one context that a program names at start-up as the workspace of the pointer-level calls."""
    global _engine_ctx
    if _engine_ctx is None:
        _engine_ctx = m.Context(0, max_tokens=64, max_experts=E, top_k=K)
        _engine_ctx.make_default()
    return _engine_ctx


def prepare(case, seed):
    T, NL, engine = case["tokens"], case["layers"], case["way"] == "engine"
    gen = torch.Generator(device=DEV).manual_seed(seed)
    s = Model()
    s.case, s.T, s.fmt = case, T, FMT[case["fmt"]]
    if engine:
        ctx = engine_context()
    else:
        ctx = s.ctx = m.Context(0, max_tokens=T, max_experts=E, top_k=K)
    router_type = torch.float16 if case["router"] == "f16" else torch.float32
    # router rows and the shared expert's gate vector as the last row, N(0, 0.02)
    W = (torch.randn(NL, E + 1, EH, device=DEV, generator=gen) * 0.02).to(router_type)
    W_host = W.cpu().numpy()
    for l in range(NL):
        L = m.Layer(ctx, s.fmt, E, router_dtype=m.F16 if case["router"] == "f16" else m.F32,
                    layout=m.LAYOUT_REFERENCE if engine else m.LAYOUT_TILED)
        L.fill_synth(seed, l)
        L.set_router(W_host[l])
        s.layers.append(L)
    x_type = torch.bfloat16 if case["x"] == "bf16" else torch.float32
    n_inputs = 1 if case["way"] == "stack" else NL
    s.X = [torch.randn(T, EH, device=DEV, generator=gen).to(x_type) for _ in range(n_inputs)]
    if case["way"] == "stack":
        s.stack = m.Stack(ctx, s.layers, T, K, m.BF16 if case["x"] == "bf16" else m.F32)
        if case["host"]:
            s.X = [x.cpu().pin_memory() for x in s.X]
            s.out = torch.empty(T, EH).pin_memory()
        else:
            s.out = torch.empty(T, EH, device=DEV)
    elif engine:
        s.W = [W[l].contiguous() for l in range(NL)]
        s.slots = [torch.tensor([L.blob_ptr(e) for e in range(E)], dtype=torch.int64, device=DEV) for L in s.layers]
        s.ypair = torch.empty(T * K, EH, device=DEV)
        s.ctx_shared = ctx
    else:
        s.out = [torch.empty(T, EH, device=DEV) for _ in range(NL)]
        s.idx = [torch.empty(T, K, device=DEV, dtype=torch.int32) if case["ids"] else None for _ in range(NL)]
    return s


def engine_layer(s, l):
    """One layer through the pointer-level calls; nothing is read back on the host."""
    L, x, T, fmt = s.layers[l], s.X[l], s.T, s.fmt
    logits = m.gemv_f16(s.W[l], x, rows=T)
    idx, w = m.router_topk(logits, E, K, True, T, E + 1)
    if T == 1:
        out = m.experts_forward(fmt, s.slots[l][idx.view(-1).long()], w, K, x).view(1, EH)
    else:
        items, pairs, _ = m.group_pairs(idx, w, T, K, E, L.slot_table())
        # the items that no token selected hold no pairs
        s.ctx_shared.pairs_forward_tc(fmt, items, E, pairs, x, T, T * K, None, s.ypair)
        out = m.pairs_reduce(s.ypair, None, torch.empty(T, EH, device=DEV), K, EH, T)
    # the shared expert's gate logit is the last column of the router rows
    m.shared_expert_add(fmt, L.blob_ptr(E), logits.data_ptr() + 4 * E, E + 1, x, T, out)
    return {"out": out, "idx": idx, "w": w}


def run(s):
    c = s.case
    if c["way"] == "stack":
        return s.stack.run_host(s.X[0], s.out) if c["host"] else s.stack.run(s.X[0], s.out)
    if c["way"] == "engine":
        return [engine_layer(s, l) for l in range(c["layers"])]
    flags = 2 if c["block"] else 0
    for l, L in enumerate(s.layers):
        L.forward(s.X[l], s.T, K, out=s.out[l], idx=s.idx[l], flags=flags)
    return {"out": s.out, "idx": s.idx}


def distinct_experts(case):
    """Routed experts that a layer's tokens select, on average. Independent tokens: E * (1 - (1 - K/E)^T). The tokens of a
    deep synthetic stack grow alike and share experts: 140 a layer were counted at 64 tokens and 40 layers, which is what
    64^0.774 = 25 independent tokens select."""
    T = case["tokens"]
    t = T ** 0.774 if case["way"] == "stack" else T
    return E * (1.0 - (1.0 - K / E) ** t)


def work(case):
    """One pass: the blobs of the selected experts and the shared one, the router and the tokens read once, the results
    written once; two operations per weight of each of a token's nine experts, and the router's."""
    T, NL = case["tokens"], case["layers"]
    per_layer = (distinct_experts(case) + 1) * BLOB[case["fmt"]] + (E + 1) * EH * (2 if case["router"] == "f16" else 4)
    io = T * EH * ((2 if case["x"] == "bf16" else 4) + 4)
    if case["way"] != "stack":
        io *= NL
    return {"bytes": NL * per_layer + io, "flops": NL * T * (2.0 * (K + 1) * 3 * EH * 512 + 2.0 * (E + 1) * EH)}


def tolerance(case):
    """Activations enter the tensor cores as two 16-bit halves and sums are fp32: 16 to 22 bits, about 1e-5. The selected
    experts are the same. In a stack of several tokens a token whose eighth and ninth expert are within rounding of each
    other may take the other one in some layer, and is another token from there on: then one row of many differs."""
    if case["way"] == "stack" and case["tokens"] > 1:
        return {"rel": 3e-3, "max": 0.5}
    return {"rel": 5e-5, "max": 5e-3}
