"""The work this library is used for, as cases that can be timed and checked.

One case is one call, or one short chain of calls, through the public Python entry points
(``Flint``, ``Generator``, ``Trainer``) over buffers that a program would already hold. The
kinds, with the range of sizes each stands for:

    mlp          a transformer block's MLP, forward and backward, FP16 operands with FP32
                 residual and gradients: 64 to 8,192 token rows, widths 256 to 1,600
    attention    fused causal attention, forward and backward: 4 to 96 heads of up to
                 1,024 positions
    scores       attention with materialised scores (the layout of ``flint_gpt2_create``):
                 heads split and merged, batched GEMMs, causal softmax and their gradients
    norm         LayerNorm forward and backward: 64 to 16,384 rows
    loss         softmax cross-entropy with its gradient over GPT-2's vocabulary
    embedding    token and position embedding, forward and backward, on tokens distributed
                 like text (a few words make up most of it)
    decode       a prompt, then one token at a time through the KV cache, FP16 or int8
                 weights, 1 to 16 sequences; returns the logits after the prompt and after
                 the last token
    prefill      a prompt alone: the latency of the first token
    train        whole optimizer steps of a GPT-2 model

Sizes are those of GPT-2 124M (the benchmark's and the tests' model) and other sizes of the
ranges that the entry points state, odd and ragged ones among them.
"""

import math
import weakref

import torch

from flint_b200.binding import Flint, Gpt2, Gpt2Config
from flint_b200.generate import Generator
from flint_b200.trainer import Trainer, TrainerConfig

VOCAB, PADDED = 50257, 50304
HEAD = 64

_library = []


def flint():
    if not _library:
        _library.append(Flint())
    return _library[0]


def listed():
    return [
        # The MLP at a ragged batch far below the tuned size: fine-tuning on one short batch.
        {"name": "mlp_1000x768", "kind": "mlp", "rows": 1000, "width": 768},
        # The MLP of one block of a GPT-2 124M step on 8 x 1,024 tokens.
        {"name": "mlp_8192x768", "kind": "mlp", "rows": 8192, "width": 768},
        # Attention of one block of the same step: 8 sequences x 12 heads.
        {"name": "attention_96x1024", "kind": "attention", "batches": 96, "length": 1024},
        # One sequence whose length does not fill the 128-row tiles.
        {"name": "attention_12x1000", "kind": "attention", "batches": 12, "length": 1000},
        # The drop-in model's attention (scores in memory) on 2 sequences.
        {"name": "scores_2x1024", "kind": "scores", "sequences": 2, "heads": 12, "length": 1024},
        # One of the 25 LayerNorms of a step.
        {"name": "norm_8192x768", "kind": "norm", "rows": 8192, "width": 768},
        # The loss of 4 x 1,024 tokens.
        {"name": "loss_4096", "kind": "loss", "rows": 4096},
        # Both embedding tables, forward and backward, for 8 x 1,024 tokens.
        {"name": "embedding_8x1024", "kind": "embedding", "sequences": 8, "length": 1024, "width": 768},
        # Interactive use: one sequence, FP16 weights; latency is all that counts.
        {"name": "decode_1_fp16", "kind": "decode", "layers": 12, "width": 768, "sequences": 1,
         "prompt": 256, "steps": 32, "int8": False},
        # A small server: eight sequences on int8 weights.
        {"name": "decode_8_int8", "kind": "decode", "layers": 12, "width": 768, "sequences": 8,
         "prompt": 512, "steps": 32, "int8": True},
        # The first token of four short prompts.
        {"name": "prefill_4x256", "kind": "prefill", "layers": 12, "width": 768, "sequences": 4,
         "prompt": 256, "int8": False},
        # The training step of GPT-2 124M on 8 x 1,024 tokens with AdamW.
        {"name": "train_8x1024", "kind": "train", "layers": 12, "width": 768, "sequences": 8, "length": 1024},
    ]


def draw(rng):
    def spread(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["mlp", "mlp", "attention", "attention", "scores", "norm", "loss", "embedding",
                       "decode", "decode", "prefill", "train"])
    if kind == "mlp":
        width = rng.choice([256, 512, 768, 1024, 1280, 1600])
        most = min(8192, 8192 * 768 * 768 // (width * width))
        return {"kind": kind, "rows": spread(64, most), "width": width}
    if kind == "attention":
        length = 8 * rng.randint(8, 128)
        return {"kind": kind, "batches": spread(4, 96), "length": length}
    if kind == "scores":
        return {"kind": kind, "sequences": rng.randint(1, 4), "heads": rng.choice([4, 8, 12, 16]),
                "length": 8 * rng.randint(8, 128)}
    if kind == "norm":
        return {"kind": kind, "rows": spread(64, 16384), "width": rng.choice([256, 512, 768, 1024, 1280, 1600])}
    if kind == "loss":
        return {"kind": kind, "rows": spread(64, 8192)}
    if kind == "embedding":
        return {"kind": kind, "sequences": rng.randint(1, 16), "length": 8 * rng.randint(8, 128),
                "width": rng.choice([256, 512, 768])}
    if kind == "train":
        return {"kind": kind, "layers": rng.randint(2, 6), "width": rng.choice([256, 512, 768]),
                "sequences": rng.randint(1, 4), "length": 8 * rng.randint(16, 128)}
    case = {"kind": kind, "layers": rng.randint(2, 12), "width": rng.choice([256, 512, 768]),
            "sequences": spread(1, 16), "prompt": 8 * rng.randint(1, 96), "int8": rng.random() < 0.5}
    if kind == "decode":
        case["steps"] = rng.randint(8, 32)
    return case


# ---- inputs ---------------------------------------------------------------------------------


class _Inputs:
    """Seeded values on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator("cuda").manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=torch.float16):
        return (torch.randn(*shape, generator=self.gen, device="cuda") * std).to(dtype)

    def tokens(self, *shape):
        """uint16 tokens in int16 tensors, rank r drawn about as often as 1 / r (as in text),
        the ranks spread over the vocabulary."""
        u = torch.rand(*shape, generator=self.gen, device="cuda", dtype=torch.float64)
        rank = (VOCAB ** u).long().clamp_(max=VOCAB) - 1
        return (rank * 7919 % VOCAB).to(torch.int16)


def _model_weights(case, seed, half):
    """GPT-2's initialisation with biases and LayerNorm parameters that are not trivially 0
    and 1. half: matrices hold values that FP16 represents (weights to decode with)."""
    source = _Inputs(seed)
    w, layers = case["width"], case["layers"]
    residual = 0.02 / math.sqrt(2 * layers)
    state = {}

    def matrix(name, shape, std=0.02):
        value = source.normal(*shape, std=std, dtype=torch.float32)
        state[name] = value.half().float() if half else value

    def vector(name, n, mean=0.0):
        state[name] = mean + source.normal(n, std=0.02, dtype=torch.float32)

    matrix("wte.weight", (PADDED, w))
    state["wte.weight"][VOCAB:] = 0
    matrix("wpe.weight", (1024, w))
    for i in range(layers):
        p = f"blocks.{i}."
        vector(p + "ln_1.weight", w, 1.0)
        vector(p + "ln_1.bias", w)
        matrix(p + "attn.c_attn.weight", (3 * w, w))
        vector(p + "attn.c_attn.bias", 3 * w)
        matrix(p + "attn.c_proj.weight", (w, w), residual)
        vector(p + "attn.c_proj.bias", w)
        vector(p + "ln_2.weight", w, 1.0)
        vector(p + "ln_2.bias", w)
        matrix(p + "mlp.c_fc.weight", (4 * w, w))
        vector(p + "mlp.c_fc.bias", 4 * w)
        matrix(p + "mlp.c_proj.weight", (w, 4 * w), residual)
        vector(p + "mlp.c_proj.bias", w)
    vector("ln_f.weight", w, 1.0)
    vector("ln_f.bias", w)
    return state


class _View:
    """Device memory of `owner`, which lives as long as a tensor on it does."""

    def __init__(self, owner, address, count):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f4", "data": (address, False),
                                         "version": 2}


def _empty(*shape, dtype=torch.float16):
    return torch.empty(*shape, device="cuda", dtype=dtype)


def _workspace(nbytes):
    return torch.empty(max(nbytes, 16), device="cuda", dtype=torch.uint8)


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state["kind"]](state)


def exact(case, seed):
    with torch.no_grad():
        return globals()["_exact_" + case["kind"]](case, seed)


def _double(values, *names):
    return [values[name].double() for name in names]


# ---- the MLP of a block ---------------------------------------------------------------------


def _mlp_inputs(case, seed):
    s, m, w = _Inputs(seed), case["rows"], case["width"]
    return {"x": s.normal(m, w), "residual": s.normal(m, w, dtype=torch.float32),
            "w1": s.normal(4 * w, w, std=0.02), "b1": s.normal(4 * w, std=0.02, dtype=torch.float32),
            "w2": s.normal(w, 4 * w, std=0.02), "b2": s.normal(w, std=0.02, dtype=torch.float32),
            "dy": s.normal(m, w, std=0.1)}


def _prepare_mlp(case, seed):
    m, w = case["rows"], case["width"]
    f32 = torch.float32
    st = _mlp_inputs(case, seed)
    st.update(kind="mlp", m=m, w=w, act=_empty(m, 4 * w), pre=_empty(m, 4 * w), y=_empty(m, w, dtype=f32),
              dpre=_empty(m, 4 * w), dx=_empty(m, w), dw1=_empty(4 * w, w, dtype=f32),
              dw2=_empty(w, 4 * w, dtype=f32), db1=_empty(4 * w, dtype=f32), db2=_empty(w, dtype=f32))
    lib = flint()
    st["workspace"] = _workspace(max(lib.gemm_tn_workspace(w, 4 * w, m), lib.gemm_tn_workspace(4 * w, w, m),
                                     lib.bias_gradient_workspace(m, 4 * w)))
    return st


def _run_mlp(s):
    lib, m, w, space = flint(), s["m"], s["w"], s["workspace"]
    lib.gemm_nt_bias_gelu(s["act"], s["pre"], s["x"], s["w1"], s["b1"], m, 4 * w, w)
    lib.gemm_nt_bias_residual(s["y"], s["act"], s["w2"], s["b2"], s["residual"], m, w, 4 * w)
    lib.gemm_nn_dgelu(s["dpre"], s["dy"], s["w2"], s["pre"], m, 4 * w, w)
    lib.gemm_tn(s["dw2"], s["dy"], s["act"], w, 4 * w, m, workspace=space)
    lib.bias_gradient(s["db2"], s["dy"], m, w, workspace=space)
    lib.gemm_nn(s["dx"], s["dpre"], s["w1"], m, w, 4 * w)
    lib.gemm_tn(s["dw1"], s["dpre"], s["x"], 4 * w, w, m, workspace=space)
    lib.bias_gradient(s["db1"], s["dpre"], m, 4 * w, workspace=space)
    return [s[name] for name in ("act", "y", "dx", "dw1", "db1", "dw2", "db2")]


def _exact_mlp(case, seed):
    x, residual, w1, b1, w2, b2, dy = _double(_mlp_inputs(case, seed), "x", "residual", "w1", "b1", "w2",
                                              "b2", "dy")
    pre = x @ w1.T + b1
    inner = math.sqrt(2 / math.pi) * (pre + 0.044715 * pre ** 3)
    t = torch.tanh(inner)
    act = 0.5 * pre * (1 + t)
    slope = 0.5 * (1 + t) + 0.5 * pre * (1 - t * t) * math.sqrt(2 / math.pi) * (1 + 3 * 0.044715 * pre ** 2)
    dpre = (dy @ w2) * slope
    return [act, residual + (act @ w2.T + b2), dpre @ w1, dpre.T @ x, dpre.sum(0), dy.T @ act, dy.sum(0)]


# ---- fused attention ------------------------------------------------------------------------


def _attention_inputs(case, seed):
    s, shape = _Inputs(seed), (case["batches"], case["length"], HEAD)
    return {name: s.normal(*shape) for name in ("q", "k", "v", "d_o")}


def _prepare_attention(case, seed):
    st = _attention_inputs(case, seed)
    b, t = case["batches"], case["length"]
    st.update(kind="attention", b=b, t=t, lse=_empty(b, t, dtype=torch.float32),
              delta=_empty(b, t, dtype=torch.float32),
              **{name: _empty(b, t, HEAD) for name in ("o", "dq", "dk", "dv")})
    return st


def _run_attention(s):
    lib, b, t = flint(), s["b"], s["t"]
    lib.attention_forward(s["o"], s["lse"], s["q"], s["k"], s["v"], b, t, HEAD, 0.125)
    lib.attention_backward(s["dq"], s["dk"], s["dv"], s["d_o"], s["o"], s["lse"], s["delta"], s["q"], s["k"],
                           s["v"], b, t, HEAD, 0.125)
    return [s[name] for name in ("o", "lse", "dq", "dk", "dv")]


def _attention_64(q, k, v, d_o):
    scores = 0.125 * (q @ k.transpose(1, 2))
    scores.masked_fill_(torch.ones_like(scores[0], dtype=torch.bool).triu(1), -math.inf)
    lse = scores.logsumexp(2)
    p = scores.sub_(lse.unsqueeze(2)).exp_()
    o = p @ v
    ds = 0.125 * p * (d_o @ v.transpose(1, 2) - (d_o * o).sum(2, keepdim=True))
    return o, lse, ds @ k, ds.transpose(1, 2) @ q, p.transpose(1, 2) @ d_o


def _exact_attention(case, seed):
    return list(_attention_64(*_double(_attention_inputs(case, seed), "q", "k", "v", "d_o")))


# ---- attention with its scores in memory -------------------------------------------------------


def _scores_inputs(case, seed):
    s, rows, w = _Inputs(seed), case["sequences"] * case["length"], case["heads"] * HEAD
    return {"qkv": s.normal(rows, 3 * w), "dy": s.normal(rows, w)}


def _prepare_scores(case, seed):
    n, h, t = case["sequences"], case["heads"], case["length"]
    st = _scores_inputs(case, seed)
    st.update(kind="scores", n=n, h=h, t=t, y=_empty(n * t, h * HEAD), dqkv=_empty(n * t, 3 * h * HEAD),
              **{name: _empty(n * h, t, HEAD) for name in ("q", "k", "v", "o", "d_o", "dq", "dk", "dv")},
              **{name: _empty(n * h, t, t) for name in ("s", "p", "dp")})
    return st


def _run_scores(s):
    lib, n, h, t = flint(), s["n"], s["h"], s["t"]
    b, w = n * h, h * HEAD
    for i, name in enumerate("qkv"):
        lib.heads_split(s[name], s["qkv"], n, t, h, HEAD, 3 * w, i * w)
    lib.gemm_nt_batched(s["s"], s["q"], s["k"], b, t, t, HEAD, 0.125)
    lib.causal_softmax_forward(s["p"], s["s"], b, t)
    lib.gemm_nn_batched(s["o"], s["p"], s["v"], b, t, HEAD, t)
    lib.heads_merge(s["y"], s["o"], n, t, h, HEAD, w)
    lib.heads_split(s["d_o"], s["dy"], n, t, h, HEAD, w)
    lib.gemm_nt_batched(s["dp"], s["d_o"], s["v"], b, t, t, HEAD)
    lib.gemm_tn_batched(s["dv"], s["p"], s["d_o"], b, t, HEAD, t)
    lib.causal_softmax_backward(s["dp"], s["p"], s["dp"], b, t, 0.125)
    lib.gemm_nn_batched(s["dq"], s["dp"], s["k"], b, t, HEAD, t)
    lib.gemm_tn_batched(s["dk"], s["dp"], s["q"], b, t, HEAD, t)
    for i, name in enumerate(("dq", "dk", "dv")):
        lib.heads_merge(s["dqkv"], s[name], n, t, h, HEAD, 3 * w, i * w)
    return [s["p"], s["y"], s["dqkv"]]


def _exact_scores(case, seed):
    n, h, t = case["sequences"], case["heads"], case["length"]
    qkv, dy = _double(_scores_inputs(case, seed), "qkv", "dy")

    def split(x):
        return x.view(n, t, h, HEAD).transpose(1, 2).reshape(n * h, t, HEAD)

    def merge(x):
        return x.view(n, h, t, HEAD).transpose(1, 2).reshape(n * t, h * HEAD)

    q, k, v = (split(x) for x in qkv.split(h * HEAD, 1))
    o, lse, dq, dk, dv = _attention_64(q, k, v, split(dy))
    p = (0.125 * (q @ k.transpose(1, 2)) - lse.unsqueeze(2)).exp().tril()
    return [p, merge(o), torch.cat([merge(x) for x in (dq, dk, dv)], 1)]


# ---- LayerNorm ------------------------------------------------------------------------------


def _norm_inputs(case, seed):
    s, m, w = _Inputs(seed), case["rows"], case["width"]
    return {"x": s.normal(m, w, dtype=torch.float32), "gamma": 1 + s.normal(w, std=0.1, dtype=torch.float32),
            "beta": s.normal(w, std=0.1, dtype=torch.float32), "dy": s.normal(m, w)}


def _prepare_norm(case, seed):
    m, w, f32 = case["rows"], case["width"], torch.float32
    st = _norm_inputs(case, seed)
    st.update(kind="norm", m=m, w=w, y=_empty(m, w), mean=_empty(m, dtype=f32), rstd=_empty(m, dtype=f32),
              dx=_empty(m, w, dtype=f32), dgamma=_empty(w, dtype=f32), dbeta=_empty(w, dtype=f32),
              workspace=_workspace(flint().layernorm_backward_workspace(m, w)))
    return st


def _run_norm(s):
    lib, m, w = flint(), s["m"], s["w"]
    lib.layernorm_forward(s["y"], s["mean"], s["rstd"], s["x"], s["gamma"], s["beta"], m, w)
    lib.layernorm_backward(s["dx"], s["dgamma"], s["dbeta"], s["dy"], s["x"], s["mean"], s["rstd"], s["gamma"],
                           m, w, workspace=s["workspace"])
    return [s[name] for name in ("y", "mean", "rstd", "dx", "dgamma", "dbeta")]


def _exact_norm(case, seed):
    x, gamma, beta, dy = _double(_norm_inputs(case, seed), "x", "gamma", "beta", "dy")
    mean = x.mean(1)
    rstd = (x.var(1, unbiased=False) + 1e-5).rsqrt()
    hat = (x - mean[:, None]) * rstd[:, None]
    g = dy * gamma
    dx = rstd[:, None] * (g - g.mean(1, keepdim=True) - hat * (g * hat).mean(1, keepdim=True))
    return [hat * gamma + beta, mean, rstd, dx, (dy * hat).sum(0), dy.sum(0)]


# ---- cross-entropy --------------------------------------------------------------------------


def _loss_inputs(case, seed):
    s, m = _Inputs(seed), case["rows"]
    logits = _empty(m, PADDED)
    logits.normal_(0.0, 2.0, generator=s.gen)
    return {"logits": logits, "targets": s.tokens(m)}


def _prepare_loss(case, seed):
    st, m = _loss_inputs(case, seed), case["rows"]
    st.update(kind="loss", m=m, dlogits=_empty(m, PADDED), row_loss=_empty(m, dtype=torch.float32))
    return st


def _run_loss(s):
    flint().softmax_cross_entropy(s["dlogits"], s["row_loss"], s["logits"], s["targets"], 65536.0 / s["m"],
                                  s["m"], VOCAB, PADDED)
    return [s["dlogits"], s["row_loss"]]


def _exact_loss(case, seed):
    values, m = _loss_inputs(case, seed), case["rows"]
    logits, dlogits = values["logits"], torch.zeros(m, PADDED, dtype=torch.float64, device="cuda")
    targets = values["targets"].long() & 0xFFFF
    losses = []
    for first in range(0, m, 1024):
        part = logits[first:first + 1024, :VOCAB].double()
        hot = targets[first:first + 1024, None]
        lse = part.logsumexp(1)
        losses.append(lse - part.gather(1, hot)[:, 0])
        grad = (part - lse[:, None]).exp()
        grad.scatter_add_(1, hot, -torch.ones_like(hot, dtype=torch.float64))
        dlogits[first:first + 1024, :VOCAB] = grad * (65536.0 / m)
    return [dlogits, torch.cat(losses)]


# ---- embedding ------------------------------------------------------------------------------


def _embedding_inputs(case, seed):
    s, n, t, w = _Inputs(seed), case["sequences"], case["length"], case["width"]
    return {"tokens": s.tokens(n * t), "wte": s.normal(PADDED, w, std=0.02, dtype=torch.float32),
            "wpe": s.normal(t, w, std=0.02, dtype=torch.float32), "dx": s.normal(n * t, w, dtype=torch.float32)}


def _prepare_embedding(case, seed):
    n, t, w, f32 = case["sequences"], case["length"], case["width"], torch.float32
    st = _embedding_inputs(case, seed)
    st.update(kind="embedding", n=n, t=t, w=w, x=_empty(n * t, w, dtype=f32), dwte=_empty(PADDED, w, dtype=f32),
              dwpe=_empty(t, w, dtype=f32),
              workspace=_workspace(flint().embedding_backward_workspace(n, t, PADDED, w)))
    return st


def _run_embedding(s):
    lib, n, t, w = flint(), s["n"], s["t"], s["w"]
    lib.embedding_forward(s["x"], s["tokens"], s["wte"], s["wpe"], n, t, PADDED, w)
    lib.embedding_backward(s["dwte"], s["dwpe"], s["dx"], s["tokens"], n, t, PADDED, w, workspace=s["workspace"])
    return [s["x"], s["dwte"], s["dwpe"]]


def _exact_embedding(case, seed):
    n, t, w = case["sequences"], case["length"], case["width"]
    values = _embedding_inputs(case, seed)
    wte, wpe, dx = _double(values, "wte", "wpe", "dx")
    tokens = values["tokens"].long() & 0xFFFF
    dwte = torch.zeros_like(wte).index_add_(0, tokens, dx)
    return [wte[tokens] + wpe.repeat(n, 1), dwte, dx.view(n, t, w).sum(0)]


# ---- a whole model in 64 bits ---------------------------------------------------------------


def _blocks_64(case, p, tokens, last_only):
    """Logits [sequences * positions, VOCAB] (of each sequence's last position with last_only)."""
    w, heads = case["width"], case["width"] // HEAD
    n, t = tokens.shape
    norm, linear = torch.nn.functional.layer_norm, torch.nn.functional.linear
    mask = torch.ones(t, t, dtype=torch.bool, device="cuda").triu(1)
    x = p["wte.weight"][tokens] + p["wpe.weight"][:t]
    for i in range(case["layers"]):
        b = f"blocks.{i}."
        h = norm(x, (w,), p[b + "ln_1.weight"], p[b + "ln_1.bias"], 1e-5)
        qkv = linear(h, p[b + "attn.c_attn.weight"], p[b + "attn.c_attn.bias"])
        q, k, v = (a.view(n, t, heads, HEAD).transpose(1, 2) for a in qkv.split(w, 2))
        s = (0.125 * (q @ k.transpose(2, 3))).masked_fill(mask, -math.inf).softmax(3)
        o = (s @ v).transpose(1, 2).reshape(n, t, w)
        x = x + linear(o, p[b + "attn.c_proj.weight"], p[b + "attn.c_proj.bias"])
        h = norm(x, (w,), p[b + "ln_2.weight"], p[b + "ln_2.bias"], 1e-5)
        a = torch.nn.functional.gelu(linear(h, p[b + "mlp.c_fc.weight"], p[b + "mlp.c_fc.bias"]),
                                     approximate="tanh")
        x = x + linear(a, p[b + "mlp.c_proj.weight"], p[b + "mlp.c_proj.bias"])
    if last_only:
        x = x[:, -1:]
    x = norm(x, (w,), p["ln_f.weight"], p["ln_f.bias"], 1e-5)
    return linear(x.reshape(-1, w), p["head"][:VOCAB])


def _int8_weights(w):
    """What int8 weights stand for: q * scale per row, scale = max|w| / 127."""
    scale = w.abs().amax(1, keepdim=True) / 127
    scale = torch.where(scale > 0, scale, torch.ones_like(scale))
    return (w * (1 / scale)).round().clamp(-127, 127).double() * scale.double()


# ---- decoding -------------------------------------------------------------------------------


def _close_all(*owners):
    for owner in owners:
        owner.close()


def _decode_tokens(case, seed):
    return _Inputs(seed + 1).tokens(case["sequences"], case["prompt"] + case.get("steps", 0))


def _prepare_decode(case, seed):
    w = case["width"]
    lib = flint()
    model = Gpt2(lib, Gpt2Config(case["layers"], w // HEAD, w, 1024, VOCAB, PADDED, 1, 8, 0, 0), True)
    model.load(_model_weights(case, seed, True))
    tokens = _decode_tokens(case, seed)
    generator = Generator(lib, model, case["sequences"], 1024, case["int8"])
    state = {"kind": "decode", "generator": generator, "prompt": tokens[:, :case["prompt"]].contiguous(),
             "rest": tokens[:, case["prompt"]:].t().contiguous()}
    weakref.finalize(generator, _close_all, _Handle(generator), model)
    torch.cuda.synchronize()
    return state


class _Handle:
    """Frees what a Generator or a Trainer holds once the object itself is gone."""

    def __init__(self, owner):
        self.handle = owner.handle
        lib = owner.flint
        self.destroy = (lib.lib.flint_b200_generator_destroy if isinstance(owner, Generator)
                        else lib.train.flint_trainer_destroy)

    def close(self):
        torch.cuda.synchronize()
        self.destroy(self.handle)


def _run_decode(s):
    generator = s["generator"]
    generator.prefill(s["prompt"])
    out = [generator.logits()]
    for i in range(s["rest"].shape[0]):
        generator.step(s["rest"][i], graph=i > 0)
    if s["rest"].shape[0]:
        out.append(generator.logits())
    return out


def _exact_decode(case, seed):
    p = _model_weights(case, seed, True)
    head = p["wte.weight"]
    if case["int8"]:
        p = {k: _int8_weights(v) if k.endswith("weight") and v.dim() == 2 and k.startswith("blocks.") else v
             for k, v in p.items()}
        head = _int8_weights(head)
    p = {k: v.double() for k, v in p.items()}
    p["head"] = head.double()
    tokens = _decode_tokens(case, seed).long() & 0xFFFF
    ends = [case["prompt"]] + ([tokens.shape[1]] if case.get("steps") else [])
    return [_blocks_64(case, p, tokens[:, :end], True) for end in ends]


_prepare_prefill, _run_prefill, _exact_prefill = _prepare_decode, _run_decode, _exact_decode


# ---- a training step ------------------------------------------------------------------------


def _train_tokens(case, seed):
    ids = _Inputs(seed + 1).tokens(case["sequences"], case["length"] + 1)
    return ids[:, :-1].contiguous(), ids[:, 1:].contiguous()


def _prepare_train(case, seed):
    w = case["width"]
    config = TrainerConfig(layers=case["layers"], heads=w // HEAD, width=w, sequences=case["sequences"],
                           length=case["length"])
    trainer = Trainer(flint(), config, state=_model_weights(case, seed, False))
    weakref.finalize(trainer, _Handle(trainer).close)
    tokens, targets = _train_tokens(case, seed)
    base = trainer.layout[0][1]
    if any(address - base != 4 * first for _, address, _, _, first in trainer.layout):
        raise RuntimeError("the weights are not laid out like their gradients")
    count = trainer.gradient_count
    arrays = [torch.as_tensor(_View(trainer, address, count), device="cuda")
              for address in (base, trainer.gradient_address, trainer.m.data_ptr(), trainer.v.data_ptr())]
    return {"kind": "train", "trainer": trainer, "tokens": tokens, "targets": targets, "arrays": arrays}


def _run_train(s):
    s["trainer"].step(s["tokens"], s["targets"])
    return [s["trainer"].finish_step()] + s["arrays"]


def _exact_train(case, seed):
    config = TrainerConfig()
    with torch.enable_grad():
        p = {k: v.double().requires_grad_() for k, v in _model_weights(case, seed, False).items()}
        tokens, targets = (t.long() & 0xFFFF for t in _train_tokens(case, seed))
        logits = _blocks_64(case, {**p, "head": p["wte.weight"]}, tokens, False)
        loss = torch.nn.functional.cross_entropy(logits, targets.reshape(-1))
        loss.backward()
    weights, grads, ms, vs = [], [], [], []
    for value in p.values():
        g = value.grad
        m, v = (1 - config.beta1) * g, (1 - config.beta2) * g * g
        decay = config.weight_decay if value.dim() > 1 else 0.0
        step = (m / (1 - config.beta1)) / ((v / (1 - config.beta2)).sqrt() + config.eps)
        weights.append((value.detach() - config.lr * (decay * value.detach() + step)).flatten())
        grads.append(g.flatten() * config.loss_scale)
        ms.append(m.flatten())
        vs.append(v.flatten())
    return [float(loss)] + [torch.cat(part) for part in (weights, grads, ms, vs)]


# ---- what a pass cannot do without ---------------------------------------------------------


def _parameters(case):
    w = case["width"]
    return PADDED * w + 1024 * w + case["layers"] * (12 * w * w + 13 * w) + 2 * w


def work(case):
    kind = case["kind"]
    if kind == "mlp":
        m, w = case["rows"], case["width"]
        # Read: x, dy, both weights (FP16), the residual; write: act, y, dx, the gradients.
        return {"bytes": m * w * (2 + 2 + 4 + 4 + 2 + 8) + 8 * w * w * (2 + 4), "flops": 48 * m * w * w}
    if kind == "attention":
        b, t = case["batches"], case["length"]
        return {"bytes": b * t * (8 * HEAD * 2 + 4), "flops": 3.5 * 2 * b * t * (t + 1) * HEAD}
    if kind == "scores":
        b, t = case["sequences"] * case["heads"], case["length"]
        return {"bytes": b * t * (8 * HEAD * 2 + 2 * t), "flops": 3.5 * 2 * b * t * (t + 1) * HEAD}
    if kind == "norm":
        m, w = case["rows"], case["width"]
        return {"bytes": m * w * (4 + 2 + 2 + 4) + 8 * m + 16 * w, "flops": 16 * m * w}
    if kind == "loss":
        m = case["rows"]
        return {"bytes": m * (4 * PADDED + 6), "flops": 6 * m * VOCAB}
    if kind == "embedding":
        m, t, w = case["sequences"] * case["length"], case["length"], case["width"]
        return {"bytes": m * (2 + 4 * w + 4 * w) + 8 * t * w + 4 * PADDED * w + 4 * min(m, VOCAB) * w // 2,
                "flops": 3 * m * w}
    if kind == "train":
        m, n = case["sequences"] * case["length"], _parameters(case)
        triangle = case["layers"] * 3.5 * 2 * case["width"] * m * (case["length"] + 1)
        # Weights, both moments read and written, gradients written; a block's activations
        # (16 w values of 2 bytes) written and read once.
        return {"bytes": 28 * n + 64 * m * case["width"] * case["layers"] + 8 * m * PADDED,
                "flops": 6 * n * m + triangle}
    w, n, layers, prompt = case["width"], case["sequences"], case["layers"], case["prompt"]
    weights = PADDED * w + layers * 12 * w * w
    size = 1 if case["int8"] else 2
    each = 2 * layers * n * w * 2
    flops = 2 * n * (prompt * layers * 12 * w * w + PADDED * w) + layers * 2 * n * w * prompt * (prompt + 1)
    total = weights * size + each * prompt + 4 * n * PADDED
    for i in range(case.get("steps", 0)):
        total += weights * size + each * (prompt + i + 1)
        flops += 2 * n * weights + layers * 4 * n * w * (prompt + i + 1)
    return {"bytes": total, "flops": flops}


def tolerance(case):
    # About four times the largest relative error against 64 bits that any output of the kind
    # showed (one rounding to FP16 leaves 2e-4, chains of them more). A first AdamW step moves a
    # weight by its gradient's sign: the few gradients near zero explain train's "max".
    return {
        "mlp": {"rel": 1.2e-3},
        "attention": {"rel": 1.3e-3},
        "scores": {"rel": 2e-3},
        "norm": {"rel": 8e-4},
        "loss": {"rel": 2e-4},
        "embedding": {"rel": 1e-6},
        "decode": {"rel": 2e-3},
        "prefill": {"rel": 2e-3},
        "train": {"rel": 2.5e-3, "max": 0.9},
    }[case["kind"]]
