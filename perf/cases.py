"""What this framework is used for, as timed cases.

    stack     one training step of a whole stack of narrow counter linears (forward, backward to the input, weight
              gradient, counter update of every linear), recorded once and replayed: `CounterStack.step`
    wide      one training step of a transformer block of wide counter linears, layer by layer: `WideStack.step`
    layer     what autograd does around ONE layer object: `CounterStateLinear.forward` and `.backward` (with its update)
    prefill   forward of one wide layer from its packed counter state, many rows: `Context.counter_forward`
    decode    the matrices of a few transformer blocks at decode time from their 2-bit words, 1 to 16 activation rows,
              recorded once and replayed: `Context.ternary_gemv`
    update    the counter update of one layer or row shard from a given gradient: `Context.counter_update_dense`
    block     the fp32 ops around the counter linears of one transformer block, forward and backward: rmsnorm, rope,
              grouped-query attention, swiglu
    head      the dense classifier at the end of a language model, forward and backward: logits, mean cross-entropy,
              gradients of logits, hidden states and classifier weights
"""
import math

import numpy as np
import torch

from motifcl_b200.counter import CounterStateLinear
from motifcl_b200.runtime import Context
from motifcl_b200.step import CounterLinearState, CounterStack, Hyper, WideStack
from motifcl_b200.synth import LinearShape

HYPER = Hyper()


def listed():
    return [
        # the benchmark's own configuration: six layers of dim 288, ffn 768, a batch of 32 x 256 tokens
        {"name": "stack_8192", "kind": "stack", "layers": 6, "dim": 288, "ffn": 768, "tokens": 8192},
        # the same stack on a short ragged batch: launches and short products count
        {"name": "stack_1000", "kind": "stack", "layers": 6, "dim": 288, "ffn": 768, "tokens": 1000},
        # one block of the 1B-scale configuration at its full token count
        {"name": "wide_1b_16384", "kind": "wide", "dim": 2048, "kv": 2048, "ffn": 5632, "tokens": 16384},
        # one block of the 8B-scale configuration (grouped heads: narrow k / v) on a ragged number of tokens
        {"name": "wide_8b_2050", "kind": "wide", "dim": 4096, "kv": 1024, "ffn": 14336, "tokens": 2050},
        # the single-layer configuration of the repository: the smallest training call
        {"name": "layer_256", "kind": "layer", "in": 288, "out": 288, "batch": 256},
        # the trainer's largest layer (w1 and w3 in one) at its batch of 16 x 256 tokens
        {"name": "layer_4096", "kind": "layer", "in": 288, "out": 1536, "batch": 4096},
        # a prompt of odd length through the largest layer of an 8B-scale model
        {"name": "prefill_777", "kind": "prefill", "in": 4096, "out": 14336, "tokens": 777},
        # one sequence being generated; 16 sequences being generated (8B-scale, 4 blocks: more bytes than L2 holds)
        {"name": "decode_1", "kind": "decode", "rows": 1, "dim": 4096, "ffn": 14336, "blocks": 4},
        {"name": "decode_16", "kind": "decode", "rows": 16, "dim": 4096, "ffn": 14336, "blocks": 4},
        # a data-parallel rank's update of one large layer from the reduced gradient
        {"name": "update_8192x4096", "kind": "update", "rows": 8192, "in": 4096, "offset": 0},
        # the trainer's block at 16 sequences of 256 tokens
        {"name": "block_16x256", "kind": "block", "seqs": 16, "len": 256, "heads": 6, "kv_heads": 6, "head_dim": 48, "ffn": 768},
        # the trainer's classifier over 32000 tokens at the same batch
        {"name": "head_4096", "kind": "head", "tokens": 4096, "dim": 288, "vocab": 32000},
    ]


def _spread(rng, low, high, step=1):
    """A multiple of `step` between low and high, even over the logarithm."""
    v = math.exp(rng.uniform(math.log(low), math.log(high + step)))
    return max(low, min(high, int(v) // step * step))


def draw(rng):
    kind = rng.choice(["stack", "stack", "wide", "wide", "layer", "layer", "prefill", "decode", "decode", "update", "block", "head"])
    if kind == "stack":
        # tokens of any count: whole batches, short tails, odd ones
        return {"kind": kind, "layers": rng.randint(1, 6), "dim": rng.choice([256, 288, 320, 384, 512]),
                "ffn": rng.choice([512, 768, 1024]), "tokens": _spread(rng, 64, 8192, rng.choice([1, 4, 128]))}
    if kind == "wide":
        dim = rng.choice([1024, 1536, 2048, 3072, 4096])
        ffn = _spread(rng, 2 * dim, 7 * dim // 2, 64)
        most = min(16384, int(16384 * (4 * 2048 * 2048 + 3 * 2048 * 5632) / (4 * dim * dim + 3 * dim * ffn)))
        return {"kind": kind, "dim": dim, "kv": rng.choice([dim, dim // 4]), "ffn": ffn, "tokens": _spread(rng, 256, most, rng.choice([1, 2, 256]))}
    if kind == "layer":
        # from the sizes of the reference's own tests up to the trainer's
        return {"kind": kind, "in": _spread(rng, 64, 1024, rng.choice([4, 32])), "out": _spread(rng, 32, 1536, rng.choice([1, 32])),
                "batch": _spread(rng, 32, 8192, rng.choice([1, 4, 128]))}
    if kind == "prefill":
        return {"kind": kind, "in": _spread(rng, 1024, 8192, 64), "out": _spread(rng, 1024, 14336, 64), "tokens": _spread(rng, 17, 4096)}
    if kind == "decode":
        return {"kind": kind, "rows": rng.choice([1, 1, 2, 3, 4, 6, 8, 11, 16]), "dim": _spread(rng, 1024, 5120, 256),
                "ffn": _spread(rng, 4096, 14336, 256), "blocks": rng.randint(1, 6)}
    if kind == "update":
        return {"kind": kind, "rows": _spread(rng, 64, 12000), "in": _spread(rng, 256, 8192, rng.choice([16, 64])), "offset": rng.choice([0, 512])}
    if kind == "block":
        heads = rng.choice([4, 6, 8, 12])
        return {"kind": kind, "seqs": _spread(rng, 1, 16), "len": _spread(rng, 32, 512), "heads": heads, "kv_heads": rng.choice([heads, heads // 2]),
                "head_dim": rng.choice([32, 48, 64]), "ffn": rng.choice([512, 768, 1024])}
    return {"kind": "head", "tokens": _spread(rng, 128, 8192), "dim": rng.choice([256, 288, 512]), "vocab": _spread(rng, 4096, 32000, 4)}


# -- inputs ----------------------------------------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, sigma=1.0):
    t = torch.randn(*shape, device="cuda", generator=g)
    return t if sigma == 1.0 else t.mul_(sigma)


def _counter_state(g, out_features, in_features):
    """Packed 6-bit codes, uniform over all 64 as in the repository's synthetic states."""
    c = torch.randint(0, 64, (out_features, in_features // 4, 4), device="cuda", generator=g, dtype=torch.int32)
    w = c[..., 0] | (c[..., 1] << 6) | (c[..., 2] << 12) | (c[..., 3] << 18)
    return torch.stack([w & 255, (w >> 8) & 255, (w >> 16) & 255], -1).to(torch.uint8).reshape(-1).contiguous()


def _start_scale(in_features):
    return float(np.sqrt(np.float32(3.0) / np.float32(2.0 * in_features)))


def _context():
    """A context on a torch stream of its own, as a recorded step needs it."""
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        return stream, Context.on_torch_stream(torch.cuda.current_device())


def _arena(tensors, dtype):
    """One flat tensor and a view of it, 256-byte aligned, in the shape of each of `tensors`."""
    per = 256 // torch.empty(0, dtype=dtype).element_size()
    starts, n = [], 0
    for t in tensors:
        starts.append(n)
        n += (t.numel() + per - 1) // per * per
    flat = torch.zeros(n, dtype=dtype, device="cuda")
    return flat, [flat[s:s + t.numel()].view(t.shape) for s, t in zip(starts, tensors)]


def _prepare_stack(case, seed):
    g, rng = _gen(seed), np.random.default_rng(seed)
    dim, ffn, tokens = case["dim"], case["ffn"], case["tokens"]
    shapes = []
    for l in range(case["layers"]):
        shapes += [LinearShape("l%d.w%s" % (l, n), dim, dim) for n in "qkvo"]
        shapes += [LinearShape("l%d.w1" % l, ffn, dim), LinearShape("l%d.w3" % l, ffn, dim), LinearShape("l%d.w2" % l, dim, ffn)]
    linears, xs, dys = [], [], []
    for s in shapes:
        O, I = s.out_features, s.in_features
        linears.append(CounterLinearState(s, rng.integers(0, 256, O * (I // 4 * 3), dtype=np.uint8), np.full(O, _start_scale(I), np.float32),
                                          np.zeros(O, np.float32), torch.device("cuda")))
        xs.append(_randn(g, tokens, I))
        dys.append(_randn(g, tokens, O, sigma=0.02))
    stream, ctx = _context()
    stack = CounterStack(ctx, linears, HYPER, tokens, grouped=True)
    # a program that saves or exchanges a stack's tensors keeps each kind of them in one buffer
    outputs = []
    for name in ("y", "dx", "grad_w", "state", "scale", "v", "packed2"):
        old = [getattr(l, name) for l in linears]
        flat, views = _arena(old, old[0].dtype)
        for l, o, view in zip(linears, old, views):
            if name in ("state", "scale", "v"):
                view.copy_(o)
            setattr(l, name, view)
        outputs.append(flat)
    stream.wait_stream(torch.cuda.current_stream())
    return {"stack": stack, "xs": xs, "dys": dys, "stream": stream, "outputs": outputs}


def _prepare_wide(case, seed):
    dim, kv, ffn = case["dim"], case["kv"], case["ffn"]
    shapes = [LinearShape("wq", dim, dim), LinearShape("wk", kv, dim), LinearShape("wv", kv, dim), LinearShape("wo", dim, dim),
              LinearShape("w1", ffn, dim), LinearShape("w3", ffn, dim), LinearShape("w2", dim, ffn)]
    stream, ctx = _context()
    with torch.cuda.stream(stream):
        stack = WideStack(ctx, shapes, case["tokens"], HYPER, "cuda", 0.01, seed=seed)
    # the layers' own tensors, and the buffers that all layers of one shape share
    outputs = [L[n] for L in stack.layers for n in ("state", "scale", "v", "packed2")]
    for b in stack.buf.values():
        outputs += [b["y"], b["dx"], b["gw"][0]]
    return {"stack": stack, "stream": stream, "outputs": outputs}


def _prepare_layer(case, seed):
    g = _gen(seed)
    layer = CounterStateLinear(Context.on_torch_stream(torch.cuda.current_device()), case["in"], case["out"], seed=seed & 0xFFFFFFFF)
    return {"layer": layer, "x": _randn(g, case["batch"], case["in"]), "dy": _randn(g, case["batch"], case["out"], sigma=0.02)}


def _prepare_prefill(case, seed):
    g = _gen(seed)
    return {"ctx": Context.on_torch_stream(torch.cuda.current_device()), "state": _counter_state(g, case["out"], case["in"]),
            "scale": torch.full((case["out"],), _start_scale(case["in"]), device="cuda"), "x": _randn(g, case["tokens"], case["in"])}


def _prepare_decode(case, seed):
    g = _gen(seed)
    dim, ffn, M = case["dim"], case["ffn"], case["rows"]
    mats = []
    for _ in range(case["blocks"]):
        for O, I in ((dim, dim), (dim, dim), (ffn, dim), (ffn, dim), (dim, ffn)):      # q, o, w1, w3, w2
            # two random bits a weight, with the field that no weight has turned into a plain one
            words = torch.randint(-2 ** 31, 2 ** 31, (O, I // 16), dtype=torch.int64, device="cuda", generator=g)
            words = (words ^ ((words & (words >> 1) & 0x55555555) << 1)) & 0xFFFFFFFF
            words = torch.where(words >= 2 ** 31, words - 2 ** 32, words).to(torch.int32)
            mats.append((words, torch.full((O,), _start_scale(I), device="cuda"), O, I))
    xs = {I: _randn(g, M, I) for I in {dim, ffn}}
    flat, ys = _arena([torch.empty(M, O, device="meta") for _, _, O, _ in mats], torch.float32)
    stream, ctx = _context()

    def sweep():
        for (words, scale, O, I), y in zip(mats, ys):
            ctx.ternary_gemv(xs[I], words, scale, y, M, I, O)
    with torch.cuda.stream(stream):
        sweep()                     # sizes the context's workspace
        ctx.finish()
        ctx.batch_begin()
        sweep()
        batch = ctx.batch_end()
    return {"ctx": ctx, "batch": batch, "mats": mats, "xs": xs, "y": flat, "stream": stream}


def _prepare_update(case, seed):
    g = _gen(seed)
    rows, I = case["rows"], case["in"]
    return {"ctx": Context.on_torch_stream(torch.cuda.current_device()), "state": _counter_state(g, rows, I), "scale": torch.full((rows,), _start_scale(I), device="cuda"),
            "v": torch.rand(rows, device="cuda", generator=g).mul_(0.01), "grad_w": _randn(g, rows, I, sigma=0.9),
            "packed2": torch.zeros(rows, I // 16, dtype=torch.int32, device="cuda"), "in": I, "rows": rows, "offset": case["offset"], "seed": 12345}


def _prepare_block(case, seed):
    g = _gen(seed)
    N, dim, kvd, H = case["seqs"] * case["len"], case["heads"] * case["head_dim"], case["kv_heads"] * case["head_dim"], case["ffn"]
    s = {n: _randn(g, N, w) for n, w in (("x", dim), ("q", dim), ("k", kvd), ("v", kvd), ("packed", 2 * H))}
    s.update({"d" + n: _randn(g, N, w, sigma=0.02) for n, w in (("att", dim), ("act", H), ("norm", dim))})
    s["weight"] = 1.0 + _randn(g, dim, sigma=0.1)
    return {"ctx": Context.on_torch_stream(torch.cuda.current_device()), "case": case, **s}


def _prepare_head(case, seed):
    g = _gen(seed)
    N, D, V = case["tokens"], case["dim"], case["vocab"]
    return {"ctx": Context.on_torch_stream(torch.cuda.current_device()), "h": _randn(g, N, D), "w": _randn(g, V, D, sigma=D ** -0.5),
            "targets": torch.randint(0, V, (N,), device="cuda", generator=g, dtype=torch.int32), "one": torch.ones(1, device="cuda")}


def prepare(case, seed):
    return {"kind": case["kind"], **globals()["_prepare_" + case["kind"]](case, seed)}


# -- one pass --------------------------------------------------------------------------------------------------------

def _run_stack(s):
    with torch.cuda.stream(s["stream"]):
        s["stack"].step(s["xs"], s["dys"], recorded=True)
    return s["outputs"]


def _run_wide(s):
    with torch.cuda.stream(s["stream"]):
        s["stack"].step()
    return s["outputs"]


def _run_layer(s):
    layer = s["layer"]
    y = layer.forward(s["x"])
    gx = layer.backward(s["x"], s["dy"], layer.next_seed())
    return [y, gx, layer.state, layer.scale, layer.v]


def _run_prefill(s):
    x, O = s["x"], s["scale"].numel()
    y = torch.empty(x.shape[0], O, device="cuda")
    s["ctx"].counter_forward(x, s["state"], s["scale"], y, x.shape[0], x.shape[1], O, HYPER.C)
    return y


def _run_decode(s):
    s["batch"].launch()
    return s["y"]


def _run_update(s):
    h = HYPER
    s["ctx"].counter_update_dense(s["state"], s["scale"], s["v"], s["grad_w"], s["packed2"], h.C, s["in"], s["rows"], s["offset"], h.lr, h.lr_scale,
                                  h.rms_beta, h.rms_eps, s["seed"])
    s["seed"] += 1
    return [s["state"], s["scale"], s["v"], s["packed2"]]


def _run_block(s):
    ctx, c, eps = s["ctx"], s["case"], 1e-5
    B, T, H, G, hd, ffn = c["seqs"], c["len"], c["heads"], c["kv_heads"], c["head_dim"], c["ffn"]
    x, N, dim, scale = s["x"], c["seqs"] * c["len"], H * hd, hd ** -0.5
    new = torch.empty_like
    norm, q, k, att = new(x), new(s["q"]), new(s["k"]), new(s["q"])
    ctx.rmsnorm(x, s["weight"], norm, N, dim, eps)
    ctx.rope(s["q"], q, B, T, dim, H, hd)
    ctx.rope(s["k"], k, B, T, G * hd, G, hd)
    ctx.gqa_forward(q, k, s["v"], att, B, T, T, T, H, G, hd, hd, True, 0, 0, scale)
    act = torch.empty(N, ffn, device="cuda")
    ctx.swiglu(s["packed"], act, N, ffn)
    dpacked = new(s["packed"])
    ctx.swiglu_backward(s["packed"], s["dact"], dpacked, N, ffn)
    probs, ds = torch.empty(B * H * T * T, device="cuda"), torch.empty(B * H * T * T, device="cuda")
    dq, dk, dv, dq0, dk0 = new(q), new(k), new(k), new(q), new(k)
    ctx.gqa_backward(q, k, s["v"], s["datt"], probs, ds, dq, dk, dv, B, T, T, H, G, hd, True, 0, scale)
    ctx.rope(dq, dq0, B, T, dim, H, hd, inverse=True)
    ctx.rope(dk, dk0, B, T, G * hd, G, hd, inverse=True)
    dx, inv, dw = new(x), torch.empty(N, device="cuda"), new(s["weight"])
    ctx.rmsnorm_backward_x(x, s["weight"], s["dnorm"], dx, N, dim, eps)
    ctx.rmsnorm_backward_weight(x, s["dnorm"], inv, dw, N, dim, eps)
    return [norm, q, k, att, act, dpacked, dq0, dk0, dv, dx, dw]


def _run_head(s):
    ctx, h, w = s["ctx"], s["h"], s["w"]
    (N, D), V = h.shape, w.shape[0]
    logits, partial, loss = torch.empty(N, V, device="cuda"), torch.empty(N, device="cuda"), torch.empty(1, device="cuda")
    ctx.matmul_f32(h, w, logits, N, D, V, trans_b=True)
    ctx.softmax_cross_entropy(logits, s["targets"], partial, loss, N, V)
    grad, dh, dw = torch.empty_like(logits), torch.empty_like(h), torch.empty_like(w)
    ctx.softmax_cross_entropy_backward(logits, s["targets"], s["one"], grad, N, V)
    ctx.matmul_f32(grad, w, dh, N, V, D)
    ctx.matmul_f32(grad, h, dw, V, N, D, trans_a=True)
    return [logits, partial, loss, grad, dh, dw]


def run(state):
    return globals()["_run_" + state["kind"]](state)


# -- what a pass cannot do without -----------------------------------------------------------------------------------

def _linear_step(N, I, O):
    """x and dy read, y, dx and dw written; state read and written, 2-bit words written; the three products."""
    return 8.0 * N * (I + O) + (4 + 1.5 + 0.25) * I * O + 16.0 * O, 6.0 * N * I * O


def work(case):
    kind = case["kind"]
    if kind in ("stack", "wide"):
        dim, ffn, kv = case["dim"], case["ffn"], case.get("kv", case["dim"])
        each = [_linear_step(case["tokens"], I, O) for O, I in ((dim, dim), (kv, dim), (kv, dim), (dim, dim), (ffn, dim), (ffn, dim), (dim, ffn))]
        n = case.get("layers", 1)
        return {"bytes": n * sum(b for b, _ in each), "flops": n * sum(f for _, f in each)}
    if kind == "layer":
        N, I, O = case["batch"], case["in"], case["out"]
        return {"bytes": 8.0 * N * (I + O) + 1.5 * I * O + 16.0 * O, "flops": 6.0 * N * I * O}      # dw is never stored
    if kind == "prefill":
        N, I, O = case["tokens"], case["in"], case["out"]
        return {"bytes": 4.0 * N * (I + O) + 0.75 * I * O + 4.0 * O, "flops": 2.0 * N * I * O}
    if kind == "decode":
        M, d, f, n = case["rows"], case["dim"], case["ffn"], case["blocks"]
        w = n * (2 * d * d + 3 * d * f)
        return {"bytes": w / 4 + n * (4.0 * (3 * d + 2 * f) + 4.0 * M * (3 * d + 2 * f)) + 4.0 * M * (d + f), "flops": 2.0 * M * w}
    if kind == "update":
        return {"bytes": 5.75 * case["rows"] * case["in"] + 16.0 * case["rows"], "flops": 0.0}
    if kind == "block":
        N, T, H, hd = case["seqs"] * case["len"], case["len"], case["heads"], case["head_dim"]
        dim, kvd, ffn = H * hd, case["kv_heads"] * hd, case["ffn"]
        # x, q, k, v, packed and five gradients in; eleven results out; two causal products forward, five backward
        return {"bytes": 4.0 * N * (9 * dim + 5 * kvd + 6 * ffn) + 8.0 * dim, "flops": 7.0 * 2 * case["seqs"] * H * hd * (T * (T + 1) / 2)}
    N, D, V = case["tokens"], case["dim"], case["vocab"]
    return {"bytes": 8.0 * N * V + 8.0 * (N * D + V * D) + 8.0 * N, "flops": 6.0 * N * D * V}


def tolerance(case):
    kind = case["kind"]
    if kind == "update":
        return "exact"              # the gradient is an input: every rounding of the update is fixed
    if kind in ("stack", "wide", "layer"):
        # Products of fp32 tensors agree to 1e-5.  The update rounds a tick of about half a counter step up or down by
        # a hash; gradients that differ by 1e-5 of themselves round the other way for a few of 100000 counters, and
        # the few of those that carry into a ternary digit change an output of the NEXT pass by one weight times one
        # activation (measured between two correct settings: 1e-3 of a result, 0.15 at one element, 6e-5 of bytes).
        n = case["in"] * case["out"] if kind == "layer" else 1 << 30
        return {"rel": max(2e-3, (1.5 / n) ** 0.5), "max": 0.5, "differ": max(1e-4, 4.0 / n)}
    return {"rel": 1e-5}            # 32-bit sums of 32-bit values
