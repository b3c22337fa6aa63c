"""The calls whose speed counts: the operators of the tensor path as a program calls them, from one-launch products to the
largest contractions, over the sizes, layouts and element types each of them is used with.

A case is a dict with a "kind" (one of the keys of KINDS) and that kind's sizes and options. `listed` names twelve of them,
`draw` makes another one of the same ranges, `prepare` puts the operands on the device, `run` is one call of the public
operators, `work` counts what the call cannot do without, and `tolerance` says how far two correct implementations differ.
"""
import math

import torch
import torch.nn.functional as F

from mimir_b200 import tensor as T

BF16, F32 = torch.bfloat16, torch.float32


def listed():
    return [
        # the smallest product: a lowered program's f32 matmul of 256 x 256 matrices, where launch and latency are everything
        dict(name="product_f32_256", kind="product", dtype="f32", batch=1, m=256, n=256, k=256, b_nk=False, post="id"),
        # one training step of the tanh MLP 128 / 784 / 1024 / 10 in f32: about twenty small and middling calls, forward and backward
        dict(name="train_step_f32", kind="train", batch=128, inputs=784, hidden=1024, classes=10),
        # the large bf16 contraction, B stored column-major
        dict(name="product_bf16_8192", kind="product", dtype="bf16", batch=1, m=8192, n=8192, k=8192, b_nk=True, post="id"),
        # a few rows against a large weight matrix: one step of generation for 16 sequences, bound by the weights' bytes
        dict(name="product_bf16_16_rows", kind="product", dtype="bf16", batch=1, m=16, n=14336, k=4096, b_nk=True, post="id"),
        # a layer whose width is no multiple of anything (an output layer over an odd number of classes), with its epilogue
        dict(name="product_bf16_odd_width", kind="product", dtype="bf16", batch=1, m=2000, n=5003, k=2048, b_nk=True, post="bias_relu"),
        # causal attention over whole sequences (prefill, training forward)
        dict(name="attention_causal_4096", kind="attention", dtype="bf16", bh=128, sq=4096, sk=4096, d=128, causal=True),
        # one new query per sequence against 4096 cached keys and values (generation)
        dict(name="attention_one_query", kind="attention", dtype="bf16", bh=128, sq=1, sk=4096, d=128, causal=False),
        # attention of an f32 program (the element type every program of the compiler has today), a ragged length
        dict(name="attention_f32_1000", kind="attention", dtype="f32", bh=32, sq=1000, sk=1000, d=64, causal=False),
        # row softmax and row RMSNorm of one f32 matrix into bf16
        dict(name="rows_16384x8192", kind="rows", dtype="f32", rows=16384, cols=8192),
        # the gated MLP block
        dict(name="mlp_gated_8192", kind="mlp", m=8192, k=4096, f=14336, n=4096, b_nk=False),
        # per-channel statistics of a [batch, positions, channels] activation (two folds along the middle axis, one with an
        # inlined producer) and the broadcast scaling with its activation
        dict(name="channel_stats", kind="stats", dtype="f32", outer=32, length=2048, inner=512),
        # a convolution layer: 3 x 3 with padding, activation, 2 x 2 maximum pooling
        dict(name="conv_layer_f32", kind="conv", dtype="f32", n=16, cin=128, h=56, w=56, cout=128, k=3, stride=1),
    ]


# ---------------------------------------------------------------------------------------------------------------- products
def _draw_product(rng):
    dtype = rng.choice(["f32", "bf16", "bf16"])
    batch = rng.choice([1, 1, 1, _log(rng, 2, 64)])
    top = 4096 if dtype == "f32" else 16384
    m, n, k = _log(rng, 1 if dtype == "bf16" else 32, 8192 if dtype == "bf16" else top), _log(rng, 64, top), _log(rng, 64, top)
    if rng.random() < 0.5:     # widths that are whole tiles; the other half stay as drawn, odd ones among them
        n, k = _up(n, 64), _up(k, 64)
    return dict(kind="product", dtype=dtype, batch=batch, m=m, n=n, k=k, b_nk=rng.random() < 0.5,
                post=rng.choice(["id", "bias_relu"]) if batch == 1 else "id")


def _prepare_product(c, g):
    dt = _dtype(c)
    lead = () if c["batch"] == 1 else (c["batch"],)
    a = _normal(g, lead + (c["m"], c["k"]), dt, 0.02 if dt == BF16 else None)
    b = _normal(g, lead + ((c["n"], c["k"]) if c["b_nk"] else (c["k"], c["n"])), dt, 0.02 if dt == BF16 else None)
    bias = _normal(g, (c["n"],), F32, 0.01) if c["post"] != "id" else None
    return dict(a=a, b=b.transpose(-1, -2) if c["b_nk"] else b, bias=bias)


def _run_product(c, s):
    if c["batch"] > 1:
        return T.bmm(s["a"], s["b"])
    return T.product_2d(s["a"], s["b"], post=c["post"], bias=s["bias"])


def _exact_product(c, s):
    y = s["a"].double() @ s["b"].double()
    return y if c["post"] == "id" else (y + s["bias"].double()).clamp_(min=0)


def _work_product(c):
    m, n, k = c["m"], c["n"], c["k"]
    return c["batch"] * _size(c) * (m * k + k * n + m * n) + (4 * n if c["post"] != "id" else 0), 2 * c["batch"] * m * n * k


# --------------------------------------------------------------------------------------------------------------- attention
def _draw_attention(rng):
    dtype = rng.choice(["f32", "bf16", "bf16", "bf16"])
    d = rng.choice([64, 128]) if dtype == "bf16" else rng.choice([32, 64, 80, 128])
    sk = _log(rng, 128, 8192 if dtype == "bf16" else 2048)
    if dtype == "bf16" and rng.random() < 0.4:      # generation: a few queries against the keys seen so far
        return dict(kind="attention", dtype=dtype, bh=_log(rng, 8, 256), sq=_log(rng, 1, 16), sk=sk, d=d, causal=rng.random() < 0.5)
    return dict(kind="attention", dtype=dtype, bh=_log(rng, 8, 128), sq=sk, sk=sk, d=d, causal=rng.random() < 0.5)


def _prepare_attention(c, g):
    dt = _dtype(c)
    return dict(q=_normal(g, (c["bh"], c["sq"], c["d"]), dt, 1.0), k=_normal(g, (c["bh"], c["sk"], c["d"]), dt, 1.0),
                v=_normal(g, (c["bh"], c["sk"], c["d"]), dt, 1.0))


def _run_attention(c, s):
    return T.attention(s["q"], s["k"], s["v"], scale=1.0 / math.sqrt(c["d"]), causal=c["causal"])


def _exact_attention(c, s):
    out = torch.empty(s["q"].shape, dtype=torch.float64, device=s["q"].device)
    hidden = torch.ones((c["sq"], c["sk"]), dtype=torch.bool, device=out.device).triu_(c["sk"] - c["sq"] + 1) if c["causal"] else None
    for i in range(c["bh"]):
        scores = (s["q"][i].double() @ s["k"][i].double().t()).mul_(1.0 / math.sqrt(c["d"]))
        if hidden is not None:
            scores.masked_fill_(hidden, -math.inf)
        out[i] = torch.softmax(scores, -1) @ s["v"][i].double()
    return out


def _work_attention(c):
    bh, sq, sk, d = c["bh"], c["sq"], c["sk"], c["d"]
    scores = sq * sk - (sq * (sq - 1) // 2 if c["causal"] else 0)
    return _size(c) * bh * d * (2 * sq + 2 * sk), 4 * bh * d * scores


# -------------------------------------------------------------------------------------------------------- rows and channels
def _draw_rows(rng):
    cols = _log(rng, 100, 16384)
    if rng.random() < 0.5:
        cols = _up(cols, 64)
    return dict(kind="rows", dtype=rng.choice(["f32", "bf16"]), rows=_log(rng, 64, min(32768, (1 << 27) // cols)), cols=cols)


def _prepare_rows(c, g):
    return dict(x=_normal(g, (c["rows"], c["cols"]), _dtype(c), 1.0),
                gamma=torch.rand((c["cols"],), generator=g, device="cuda") + 0.5)


def _run_rows(c, s):
    return T.softmax(1, s["x"], out_dtype=BF16), T.rmsnorm(s["x"], s["gamma"], 1e-6, out_dtype=BF16)


def _exact_rows(c, s):
    x = s["x"].double()
    return torch.softmax(x, 1), x * torch.rsqrt(x.square().mean(1, keepdim=True) + 1e-6) * s["gamma"].double()


def _work_rows(c):
    cells = c["rows"] * c["cols"]
    return cells * (_size(c) + 2 + 2) + 4 * c["cols"], 9 * cells


def _draw_stats(rng):
    inner = _log(rng, 32, 2048)
    length = _log(rng, 64, 8192)
    if rng.random() < 0.5:
        inner = _up(inner, 32)
    return dict(kind="stats", dtype=rng.choice(["f32", "f32", "bf16"]), outer=_log(rng, 1, max(1, min(64, (1 << 27) // (inner * length)))),
                length=length, inner=inner)


def _prepare_stats(c, g):
    dt = _dtype(c)
    return dict(x=_normal(g, (c["outer"], c["length"], c["inner"]), dt, 1.0), scale=_normal(g, (c["outer"], c["inner"]), dt, 1.0))


def _run_stats(c, s):
    x = s["x"]
    return T.reduce("sum", 1, x), T.reduce_fused("sum", 1, x, "square"), T.binary_ax("mul", 1, x, s["scale"], then="relu")


def _exact_stats(c, s):
    x = s["x"].double()
    return x.sum(1), x.square().sum(1), (x * s["scale"].double().unsqueeze(1)).clamp_(min=0)


def _work_stats(c):
    cells = c["outer"] * c["length"] * c["inner"]
    return _size(c) * (2 * cells + 3 * c["outer"] * c["inner"]), 5 * cells


# --------------------------------------------------------------------------------------------------------------------- MLPs
def _draw_mlp(rng):
    k, n = 64 * _log(rng, 8, 64), 64 * _log(rng, 8, 64)
    return dict(kind="mlp", m=_log(rng, 1, 8192), k=k, f=64 * _log(rng, 16, 224), n=n, b_nk=rng.random() < 0.5)


def _prepare_mlp(c, g):
    def weight(i, o):
        return _normal(g, (o, i), BF16, 0.02).t() if c["b_nk"] else _normal(g, (i, o), BF16, 0.02)
    return dict(x=_normal(g, (c["m"], c["k"]), BF16, 1.0), w1=weight(c["k"], c["f"]), w3=weight(c["k"], c["f"]), w2=weight(c["f"], c["n"]))


def _run_mlp(c, s):
    return T.mlp_gated(s["x"], s["w1"], s["w3"], s["w2"])


def _exact_mlp(c, s):
    x = s["x"].double()
    return (F.silu(x @ s["w1"].double()) * (x @ s["w3"].double())) @ s["w2"].double()


def _work_mlp(c):
    m, k, f, n = c["m"], c["k"], c["f"], c["n"]
    return 2 * (m * k + 2 * k * f + f * n + m * n), 2 * m * f * (2 * k + n)


def _draw_train(rng):
    return dict(kind="train", batch=_log(rng, 16, 512), inputs=_log(rng, 64, 2048), hidden=_log(rng, 128, 2048), classes=_log(rng, 10, 1000))


def _prepare_train(c, g):
    b, i, h, o = c["batch"], c["inputs"], c["hidden"], c["classes"]
    y = torch.zeros((b, o), device="cuda")
    y[torch.arange(b, device="cuda"), torch.randint(0, o, (b,), generator=g, device="cuda")] = 1.0
    return dict(x=torch.rand((b, i), generator=g, device="cuda"), y=y,
                w1=_normal(g, (i, h), F32, i ** -0.5), w2=_normal(g, (h, h), F32, h ** -0.5), w3=_normal(g, (h, o), F32, h ** -0.5),
                b1=_normal(g, (h,), F32, 0.01), b2=_normal(g, (h,), F32, 0.01), b3=_normal(g, (o,), F32, 0.01))


def _run_train(c, s):
    """Logits and gradients of the softmax cross-entropy of x -> tanh -> tanh -> classes."""
    x, w2, w3 = s["x"], s["w2"], s["w3"]

    def through_tanh(d, h):      # d (1 - h^2)
        return T.binary("sub", d, T.binary("mul", d, T.unary("square", h)))

    h1 = T.product_2d(x, s["w1"], post="bias_tanh", bias=s["b1"])
    h2 = T.product_2d(h1, w2, post="bias_tanh", bias=s["b2"])
    logits = T.product_2d(h2, w3, post="bias", bias=s["b3"])
    d3 = T.binary("sub", T.softmax(1, logits), s["y"])
    d2 = through_tanh(T.product_2d(d3, T.transpose_2d(w3)), h2)
    d1 = through_tanh(T.product_2d(d2, T.transpose_2d(w2)), h1)
    return {"logits": logits,
            "w3": T.product_2d(T.transpose(h2, (1, 0)), d3), "b3": T.reduce("sum", 0, d3),
            "w2": T.product_2d(T.transpose(h1, (1, 0)), d2), "b2": T.reduce("sum", 0, d2),
            "w1": T.product_2d(T.transpose(x, (1, 0)), d1), "b1": T.reduce("sum", 0, d1)}


def _exact_train(c, s):
    x, y, w1, w2, w3, b1, b2, b3 = (s[k].double() for k in ("x", "y", "w1", "w2", "w3", "b1", "b2", "b3"))
    h1 = torch.tanh(x @ w1 + b1)
    h2 = torch.tanh(h1 @ w2 + b2)
    logits = h2 @ w3 + b3
    d3 = torch.softmax(logits, 1) - y
    d2 = d3 @ w3.t() * (1 - h2 * h2)
    d1 = d2 @ w2.t() * (1 - h1 * h1)
    return {"logits": logits, "w3": h2.t() @ d3, "b3": d3.sum(0), "w2": h1.t() @ d2, "b2": d2.sum(0), "w1": x.t() @ d1, "b1": d1.sum(0)}


def _work_train(c):
    b, i, h, o = c["batch"], c["inputs"], c["hidden"], c["classes"]
    weights = i * h + h * h + h * o
    return 4 * (b * i + 2 * b * o + 2 * (weights + 2 * h + o)), 2 * b * (2 * i * h + 3 * h * h + 3 * h * o)


# ------------------------------------------------------------------------------------------------------------- convolutions
def _draw_conv(rng):
    side = _log(rng, 14, 112)
    return dict(kind="conv", dtype=rng.choice(["f32", "f32", "bf16"]), n=_log(rng, 1, 32), cin=rng.choice([3, 16, 32, 64, 128, 256]),
                h=side, w=side + rng.choice([0, 0, 1, 5]), cout=rng.choice([32, 64, 96, 128, 256]), k=rng.choice([1, 3, 3, 5]),
                stride=rng.choice([1, 1, 2]))


def _prepare_conv(c, g):
    fan = c["cin"] * c["k"] ** 2
    return dict(x=_normal(g, (c["n"], c["cin"], c["h"], c["w"]), _dtype(c), 1.0),
                w=_normal(g, (c["cout"], c["cin"], c["k"], c["k"]), _dtype(c), fan ** -0.5))


def _run_conv(c, s):
    y = T.conv(s["x"], s["w"], stride=(c["stride"],) * 2, padding=(c["k"] // 2,) * 2)
    return T.pool("max", T.unary("relu", y), (2, 2))


def _exact_conv(c, s):
    w = s["w"].double().flatten(1)
    y = []
    for x in s["x"].double().split(1):
        oh, ow = (c["h"] - 1) // c["stride"] + 1, (c["w"] - 1) // c["stride"] + 1
        y.append((w @ F.unfold(x, c["k"], padding=c["k"] // 2, stride=c["stride"])).view(1, c["cout"], oh, ow))
    return F.max_pool2d(torch.cat(y).clamp_(min=0), 2)


def _work_conv(c):
    oh, ow = (c["h"] - 1) // c["stride"] + 1, (c["w"] - 1) // c["stride"] + 1
    taps = c["cin"] * c["k"] ** 2
    return (_size(c) * (c["n"] * c["cin"] * c["h"] * c["w"] + c["cout"] * taps + c["n"] * c["cout"] * (oh // 2) * (ow // 2)),
            2 * c["n"] * c["cout"] * oh * ow * taps)


# ------------------------------------------------------------------------------------------------------------------- common
KINDS = {
    "product": (_draw_product, _prepare_product, _run_product, _work_product, _exact_product),
    "attention": (_draw_attention, _prepare_attention, _run_attention, _work_attention, _exact_attention),
    "rows": (_draw_rows, _prepare_rows, _run_rows, _work_rows, _exact_rows),
    "stats": (_draw_stats, _prepare_stats, _run_stats, _work_stats, _exact_stats),
    "mlp": (_draw_mlp, _prepare_mlp, _run_mlp, _work_mlp, _exact_mlp),
    "train": (_draw_train, _prepare_train, _run_train, _work_train, _exact_train),
    "conv": (_draw_conv, _prepare_conv, _run_conv, _work_conv, _exact_conv),
}
# how often each kind is drawn: contractions and attention are most of what programs do
WEIGHTS = {"product": 4, "attention": 4, "rows": 2, "stats": 1, "mlp": 2, "train": 1, "conv": 2}


def _log(rng, lo, hi):
    """A whole number from lo to hi, uniform in its logarithm."""
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _up(v, to):
    return (v + to - 1) // to * to


def _dtype(c):
    return BF16 if c.get("dtype") == "bf16" else F32


def _size(c):
    return 2 if c.get("dtype", "bf16") == "bf16" else 4


def _normal(g, shape, dtype, std):
    """Normal(0, std) values, or uniform in [-1, 1] where std is None."""
    if std is None:
        return torch.rand(shape, generator=g, device="cuda").mul_(2).sub_(1).to(dtype)
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype).mul_(std)


def draw(rng):
    kinds = list(KINDS)
    while True:
        c = KINDS[rng.choices(kinds, [WEIGHTS[k] for k in kinds])[0]][0](rng)
        w = work(c)
        # f32 work and odd widths cost more time for the same count, and no drawn case is to cost more than the largest listed one
        slow = c.get("dtype") == "f32" or c["kind"] == "conv" or (c["kind"] == "product" and (c["k"] % 8 or c["n"] % 8))
        if w["flops"] <= (3e10 if slow else 1e12) and w["bytes"] <= 1e9:
            return c


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    state = KINDS[case["kind"]][1](case, g)
    state["case"] = case
    return state


def run(state):
    c = state["case"]
    return KINDS[c["kind"]][2](c, state)


def work(case):
    nbytes, flops = KINDS[case["kind"]][3](case)
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    """What `run` returns for these inputs, as plain torch gives it in 64 bits."""
    return KINDS[case["kind"]][4](case, prepare(case, seed))


def tolerance(case):
    # About four times what one pass differs by from the same path in 64 bits (relative 2-norm; largest difference over the
    # value, or over the root mean square where that is larger). bf16 results: 1.7e-3 and 3.9e-3, the rounding of the result
    # alone; with a rounded intermediate, which the MLP's hidden layer and attention's probabilities are, 2.4e-3 and
    # 1.1e-2 / 4.2e-2. f32 results: 2.2e-6 and 9.2e-6.
    if case["kind"] == "attention" and case["dtype"] == "bf16":
        return {"rel": 1e-2, "max": 0.16}
    if case["kind"] == "mlp":
        return {"rel": 1e-2, "max": 0.045}
    if case["kind"] == "rows" or case.get("dtype") == "bf16":
        return {"rel": 7e-3, "max": 0.016}
    return {"rel": 1e-5, "max": 4e-5}
