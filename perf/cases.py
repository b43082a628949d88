"""Performance cases of the library: what its users run, through the public entry points, on one GPU.

kind "lm"     one step of ``FusedLMTrainer`` on the rotated ``TransformerLM`` (the headline benchmark's path)
kind "gpt"    rotated modules + autograd + ``ShardedAdamW`` on the GPT model: a training step, or the logits alone
kind "llama"  the same for the Llama-shaped model
kind "attn"   ``flash_attention`` forward and backward on caller-made q, k, v
kind "moe"    one mixture-of-experts layer (gate, dispatch, experts, combine) forward and backward
kind "conv"   one rotated convolution forward and backward

Everything is bf16 with fp32 accumulation, which is what the kernels are for.  Weights start as the models initialise
them; token ids are uniform, as in the benchmark.
"""
import math

import torch
import torch.nn.functional as F

DEV = "cuda"
BF = torch.bfloat16


def listed():
    return [
        # The smallest model of the benchmark: a step of short kernels, bound by launches and their latency.
        dict(name="lm-tiny", kind="lm", vocab=1024, d=256, heads=4, ff=1024, layers=2, seq=32, batch=8, dropout=0.1,
             keep_grads=True),
        # The headline workload: the README model of the benchmark, dropout on, optimizer inside backward.
        dict(name="lm-readme", kind="lm", vocab=10240, d=2048, heads=32, ff=2048, layers=10, seq=32, batch=32, dropout=0.1,
             keep_grads=False),
        # A model whose sizes fit no tile: 650 tokens of sequences that are not a multiple of 32, no dropout.
        dict(name="lm-ragged", kind="lm", vocab=4000, d=768, heads=12, ff=3080, layers=3, seq=50, batch=13, dropout=0.0,
             keep_grads=True),
        # The benchmark's small GPT: a whole module-path step replayed from a CUDA graph.
        dict(name="gpt-small", kind="gpt", vocab=8192, d=512, heads=8, ff=2048, layers=4, seq=256, batch=4, train=True,
             graph=True),
        # Four layers of the 1.3 B GPT at its sequence length with a full vocabulary, launched eagerly by a torch loop.
        dict(name="gpt-2k", kind="gpt", vocab=50304, d=2048, heads=16, ff=8192, layers=4, seq=2048, batch=4, train=True,
             graph=False),
        # Scoring: logits of ragged sequences, no gradients (two layers of the same model).
        dict(name="gpt-score", kind="gpt", vocab=50304, d=2048, heads=16, ff=8192, layers=2, seq=999, batch=3, train=False,
             graph=False),
        # The benchmark's small Llama on ragged sequences.
        dict(name="llama-ragged", kind="llama", vocab=8192, d=512, heads=8, ff=1536, layers=4, seq=250, batch=3, train=True,
             graph=True),
        # One layer of the Llama-shaped 13 B model: the widest matrices, RMSNorm, rotary embedding, SwiGLU.
        dict(name="llama-wide", kind="llama", vocab=32000, d=5120, heads=40, ff=13824, layers=1, seq=2048, batch=2, train=True,
             graph=False),
        # Long-context causal attention.
        dict(name="attn-long", kind="attn", batch=1, heads=16, sq=8192, sk=8192, hd=128, causal=True, pad=False, dropout=0.0),
        # Encoder attention over padded batches: ragged length, key-padding mask, narrow heads.
        dict(name="attn-padded", kind="attn", batch=6, heads=12, sq=700, sk=700, hd=64, causal=False, pad=True, dropout=0.0),
        # The feed-forward layer of the benchmark's MoE model.
        dict(name="moe", kind="moe", batch=8, seq=1024, d=2048, ff=8192, experts=8, capacity=1.25),
        # The larger convolution of the MNIST example at its batch size: a single small layer, called eagerly.
        dict(name="conv-mnist", kind="conv", batch=64, cin=32, cout=64, size=26, kernel=3, stride=1, padding=0),
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of ``step`` spread evenly over the logarithm of [lo, hi]."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["lm", "lm", "gpt", "gpt", "llama", "attn", "attn", "moe", "conv"])
    while True:
        if kind == "lm":
            heads = rng.choice([4, 6, 8, 10, 12, 16, 20, 24, 32])
            layers = rng.randint(1, 5)
            c = dict(kind=kind, vocab=_log(rng, 512, 16384, 8), d=64 * heads, heads=heads, ff=_log(rng, 512, 8192, 8),
                     layers=layers, seq=rng.choice([32, 64, rng.randint(8, 96)]), batch=_log(rng, 2, 64),
                     dropout=rng.choice([0.0, 0.1]), keep_grads=rng.random() < 0.5)
            if c["dropout"] and c["seq"] * c["batch"] % 4:
                c["batch"] = c["batch"] // 4 * 4 + 4
        elif kind in ("gpt", "llama"):
            hd = rng.choice([64, 128])
            heads = rng.choice([4, 6, 8, 12, 16])
            train = rng.random() < 0.7
            c = dict(kind=kind, vocab=_log(rng, 1024, 50304, 8), d=hd * heads, heads=heads, ff=_log(rng, 512, 8192, 8),
                     layers=rng.randint(1, 4), seq=_log(rng, 100, 2048), batch=_log(rng, 1, 8), train=train,
                     graph=rng.random() < 0.5)
        elif kind == "attn":
            causal = rng.random() < 0.5
            sq = _log(rng, 100, 8192)
            c = dict(kind=kind, batch=_log(rng, 1, 16), heads=rng.randint(2, 24), sq=sq,
                     sk=sq if causal or rng.random() < 0.6 else _log(rng, 100, 8192), hd=rng.choice([64, 128]), causal=causal,
                     pad=rng.random() < 0.4, dropout=rng.choice([0.0, 0.0, 0.1]))
        elif kind == "moe":
            experts = rng.choice([2, 4, 8])
            c = dict(kind=kind, batch=_log(rng, 1, 8), seq=_log(rng, 128, 1024, 16), d=_log(rng, 256, 2048, 8),
                     ff=_log(rng, 512, 8192, 8), experts=experts, capacity=rng.choice([1.0, 1.25]))
            # capacities are whole k-blocks of the expert kernels, as in the benchmark's configurations
            if int(c["capacity"] * 2 * c["batch"] * c["seq"] // experts) % 64:
                continue
        else:
            kernel = rng.choice([3, 3, 5])
            c = dict(kind=kind, batch=_log(rng, 8, 256), cin=rng.choice([1, 3, 16, 32, 64]), cout=rng.choice([16, 32, 64, 128]),
                     size=rng.randint(12, 56), kernel=kernel, stride=rng.choice([1, 1, 2]), padding=rng.choice([0, 1]))
        w = work(c)
        if w["flops"] <= 2.4e13 and w["bytes"] <= 2.2e10:
            return c


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _shapes(c):
    """(name, shape, fill) of every parameter of a case's model; fill: a bound of a uniform draw (negative: the standard
    deviation of a normal one), 0 for zeros, 1 for ones."""
    D, V, L, H = c["d"], c["vocab"], c["layers"], c["ff"]
    out = []
    if c["kind"] == "lm":
        out.append(("0.embedding.embedding.weight", (V, D), 0.1))
        b = 1 / math.sqrt(D)
        for i in range(2, 2 + L):
            a = f"{i}.self_attn.MultiheadAttention."
            f = f"{i}.ff_block."
            out += [(a + "in_proj_weight", (3 * D, D), math.sqrt(6 / (4 * D))), (a + "in_proj_bias", (3 * D,), 0),
                    (a + "out_proj.weight", (D, D), b), (a + "out_proj.bias", (D,), 0),
                    (f + "linear1.linear.weight", (H, D), b), (f + "linear1.linear.bias", (H,), b),
                    (f + "linear2.linear.weight", (D, H), 1 / math.sqrt(H)),
                    (f + "linear2.linear.bias", (D,), 1 / math.sqrt(H))]
            for n in ("norm1", "norm2"):
                out += [(f"{i}.{n}.weight", (D,), 1), (f"{i}.{n}.bias", (D,), 0)]
        out += [(f"{2 + L}.linear.linear.weight", (V, D), 0.1), (f"{2 + L}.linear.linear.bias", (V,), 0)]
        return out
    s = -0.02
    out.append(("tok.embedding.weight", (V, D), s))
    if c["kind"] == "gpt":
        out.append(("pos", (c["seq"], D), s))
        for i in range(L):
            p = f"blocks.{i}."
            a = p + "attn.MultiheadAttention."
            out += [(p + "ln1.weight", (D,), 1), (p + "ln1.bias", (D,), 0), (a + "in_proj_weight", (3 * D, D), s),
                    (a + "in_proj_bias", (3 * D,), 0), (a + "out_proj.weight", (D, D), s), (a + "out_proj.bias", (D,), 0),
                    (p + "ln2.weight", (D,), 1), (p + "ln2.bias", (D,), 0), (p + "fc1.linear.weight", (H, D), s),
                    (p + "fc1.linear.bias", (H,), 0), (p + "fc2.linear.weight", (D, H), s), (p + "fc2.linear.bias", (D,), 0)]
        out += [("ln_f.weight", (D,), 1), ("ln_f.bias", (D,), 0)]
    else:
        for i in range(L):
            p = f"blocks.{i}."
            out += [(p + "norm1.weight", (D,), 1), (p + "qkv.linear.weight", (3 * D, D), s),
                    (p + "proj.linear.weight", (D, D), s), (p + "norm2.weight", (D,), 1),
                    (p + "gate_up.linear.weight", (2 * H, D), s), (p + "down.linear.weight", (D, H), s)]
        out.append(("norm.weight", (D,), 1))
    out.append(("head.linear.weight", (V, D), s))
    return out


def _weights(c, g):
    """The bf16 weights of a case's model by name."""
    w = {}
    for name, shape, fill in _shapes(c):
        t = torch.empty(shape, dtype=torch.float32, device=DEV)
        if fill in (0, 1):
            t.fill_(fill)
        elif fill < 0:
            t.normal_(0.0, -fill, generator=g)
        else:
            t.uniform_(-fill, fill, generator=g)
        w[name] = t.to(BF)
    return w


def _tokens(c, g):
    """ids and next-token targets: [seq, batch] for the reference-layout model, [batch, seq] for the others."""
    S, B = c["seq"], c["batch"]
    stream = torch.randint(0, c["vocab"], (S + 1, B), generator=g, device=DEV)
    ids, tgt = stream[:-1], stream[1:]
    if c["kind"] != "lm":
        ids, tgt = ids.t(), tgt.t()
    return ids.contiguous(), tgt.contiguous()


def _load(model, w):
    own = dict(model.named_parameters())
    assert set(own) == set(w)
    with torch.no_grad():
        for n, t in w.items():
            own[n].copy_(t)
    return [own[n] for n in w]


def _tensors(c, seed):
    """Inputs of the kinds without a model."""
    g = _gen(seed)

    def rnd(*shape, scale=1.0):
        return (torch.randn(shape, generator=g, device=DEV) * scale).to(BF)
    if c["kind"] == "attn":
        B, H, hd, sq, sk = c["batch"], c["heads"], c["hd"], c["sq"], c["sk"]
        q, k, v, do = rnd(B, sq, H, hd), rnd(B, sk, H, hd), rnd(B, sk, H, hd), rnd(B, sq, H, hd)
        kpm = None
        if c["pad"]:     # every sequence keeps between half and all of its keys
            n = torch.randint((sk + 1) // 2, sk + 1, (B, 1), generator=g, device=DEV)
            kpm = torch.arange(sk, device=DEV)[None] >= n
        return q, k, v, do, kpm
    if c["kind"] == "moe":
        D, H, E = c["d"], c["ff"], c["experts"]
        ws = [rnd(E, D, scale=0.02)]
        for _ in range(E):
            ws += [rnd(H, D, scale=0.02), rnd(H, scale=0.02), rnd(D, H, scale=0.02), rnd(D, scale=0.02)]
        return rnd(c["batch"], c["seq"], D), rnd(c["batch"], c["seq"], D), ws
    B, ci, co, n, k = c["batch"], c["cin"], c["cout"], c["size"], c["kernel"]
    o = (n + 2 * c["padding"] - k) // c["stride"] + 1
    s = 1 / math.sqrt(ci * k * k)
    return rnd(B, ci, n, n), rnd(B, co, o, o), rnd(co, ci, k, k, scale=s), rnd(co, scale=s)


def prepare(case, seed):
    c = case
    g = _gen(seed)
    if c["kind"] == "lm":
        from rtp_b200.models.fused_lm import FusedLMTrainer
        from rtp_b200.models.transformer_lm_rtp import TransformerLM
        model = TransformerLM(c["vocab"], c["d"], c["heads"], c["ff"], c["dropout"], 0.1, c["layers"], 1, 0, device=DEV)
        model = model.to(dtype=BF)
        params = _load(model, _weights(c, g))
        trainer = FusedLMTrainer(model, lr=1e-3, clip_value=0.05, state_dtype="mixed", keep_grads=c["keep_grads"])
        if not c["keep_grads"]:
            params = [p for (n, _, _), p in zip(_shapes(c), params) if n.endswith("weight")]
        return dict(c=c, trainer=trainer, params=params, batch=_tokens(c, g))
    if c["kind"] in ("gpt", "llama"):
        from rtp_b200.optim import ShardedAdamW
        if c["kind"] == "gpt":
            from rtp_b200.models.gpt import GPT as Model, GPTConfig as Config
        else:
            from rtp_b200.models.llama import Llama as Model, LlamaConfig as Config
        model = Model(Config(c["vocab"], c["d"], c["layers"], c["heads"], c["ff"], c["seq"]), device=DEV, dtype=BF)
        w = _weights(c, g)
        params = _load(model, w)
        ids, tgt = _tokens(c, g)
        st = dict(c=c, model=model, params=params, batch=(ids, tgt))
        if c["train"]:
            opt = ShardedAdamW(model.parameters(), lr=1e-4, weight_decay=0.01, state_dtype="mixed")

            def step(i, t):
                opt.zero_grad(set_to_none=not c["graph"])
                loss = model(i, t)
                loss.backward()
                opt.step()
                return loss.detach()
        else:
            model.eval()

            def step(i, t):
                with torch.no_grad():
                    return model(i)
        if c["graph"]:
            from rtp_b200.utils.graphed import GraphedStep
            step = GraphedStep(step, (ids, tgt))
            _load(model, w)          # the warm-up steps have trained it
        st["step"] = step
        return st
    if c["kind"] == "attn":
        q, k, v, do, kpm = _tensors(c, seed)
        return dict(c=c, q=q.requires_grad_(), k=k.requires_grad_(), v=v.requires_grad_(), do=do, kpm=kpm)
    if c["kind"] == "moe":
        from rtp_b200.models.moe_lm import Expert
        from rtp_b200.module.moe import WeightMOELayer
        from rtp_b200.module.top2gate import WeightTop2Gate
        x, dy, ws = _tensors(c, seed)
        gate = WeightTop2Gate(c["d"], c["experts"], device=DEV, dtype=BF, capacity_factor=c["capacity"])
        with torch.device(DEV):
            experts = torch.nn.ModuleList([Expert(c["d"], c["ff"]) for _ in range(c["experts"])])
        layer = WeightMOELayer(gate, experts, device=DEV, dtype=BF)
        params = [gate.wg.weight]
        for e in layer.experts:
            params += [e.linear1.weight, e.linear1.bias, e.linear2.weight, e.linear2.bias]
        with torch.no_grad():
            for p, t in zip(params, ws):
                p.copy_(t)
        torch.manual_seed(int(seed))     # the noise of the second choice
        return dict(c=c, layer=layer, params=params, x=x.requires_grad_(), dy=dy)
    from rtp_b200.module.conv import ColumnParallelConv2d
    x, dy, w, b = _tensors(c, seed)
    conv = ColumnParallelConv2d(c["cin"], c["cout"], c["kernel"], c["stride"], c["padding"], device=DEV, dtype=BF)
    with torch.no_grad():
        conv.conv.weight.copy_(w)
        conv.conv.bias.copy_(b)
    return dict(c=c, conv=conv, params=[conv.conv.weight, conv.conv.bias], x=x.requires_grad_(), dy=dy)


def run(state):
    c = state["c"]
    if c["kind"] == "lm":
        loss = state["trainer"].step(*state["batch"])
        return [loss, [p.grad if c["keep_grads"] else p.detach() for p in state["params"]]]
    if c["kind"] in ("gpt", "llama"):
        out = state["step"](*state["batch"])
        return [out, [p.grad for p in state["params"]]] if c["train"] else out
    if c["kind"] == "attn":
        from rtp_b200.ops.flash import flash_attention
        q, k, v = state["q"], state["k"], state["v"]
        o = flash_attention(q, k, v, causal=c["causal"], key_padding_mask=state["kpm"], dropout_p=c["dropout"], seed=7, offset=3)
        return [o.detach(), *torch.autograd.grad(o, (q, k, v), state["do"])]
    if c["kind"] == "moe":
        y = state["layer"](state["x"])
        aux = state["layer"].l_aux
        grads = torch.autograd.grad((y, aux), [state["x"], *state["params"]], (state["dy"], torch.ones_like(aux)))
        return [y.detach(), aux.detach(), *grads]
    y = state["conv"](state["x"])
    return [y.detach(), *torch.autograd.grad(y, [state["x"], *state["params"]], state["dy"])]


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def work(case):
    c = case
    if c["kind"] in ("lm", "gpt", "llama"):
        T, D, L, V, H = c["seq"] * c["batch"], c["d"], c["layers"], c["vocab"], c["ff"]
        mats = L * (4 * D * D + (3 if c["kind"] == "llama" else 2) * D * H) + V * D
        params = sum(math.prod(s) for _, s, _ in _shapes(c))
        attn = 2 * T * c["seq"] * D * L                       # causal: half of 4 S^2 d per head
        train = c["kind"] == "lm" or c["train"]
        if not train:
            return {"bytes": 2 * params + 2 * T * V, "flops": 2 * T * mats + attn}
        # bf16 weight, bf16 first and fp32 second moment, each read and written once; gradients where they are results
        per = 16 + (2 if c["kind"] != "lm" or c["keep_grads"] else 0)
        return {"bytes": per * params, "flops": 6 * T * mats + 3.5 * attn}
    if c["kind"] == "attn":
        rows = c["batch"] * c["heads"] * c["hd"] * 2
        f = 14 * c["batch"] * c["heads"] * c["hd"] * c["sq"] * c["sk"] * (0.5 if c["causal"] else 1.0)
        return {"bytes": rows * (4 * c["sq"] + 4 * c["sk"]), "flops": f}
    if c["kind"] == "moe":
        S, D, H, E = c["seq"] * c["batch"], c["d"], c["ff"], c["experts"]
        return {"bytes": 4 * E * (2 * D * H + H + D) + 8 * S * D, "flops": 6 * 2 * S * 2 * D * H}
    o = (c["size"] + 2 * c["padding"] - c["kernel"]) // c["stride"] + 1
    k = c["cin"] * c["kernel"] ** 2
    n_in, n_out = c["batch"] * c["cin"] * c["size"] ** 2, c["batch"] * c["cout"] * o * o
    return {"bytes": 2 * (2 * n_in + 2 * n_out + 2 * c["cout"] * k), "flops": 6 * n_out * k}


def tolerance(case):
    """About four times the distance from 64 bits that was measured (rel / max): models 0.008-0.014 / 0.3 (gradients behind
    a ReLU up to 0.06 / 0.8, because rounding moves units across zero), attention 0.0024 / 0.19, experts 0.0043 / 0.034,
    convolution 0.0024 / 0.011."""
    if case["kind"] in ("lm", "gpt", "llama"):
        return {"rel": 0.03, "max": 0.9}
    if case["kind"] == "attn":
        return {"rel": 0.01, "max": 0.8}
    return {"rel": 0.017, "max": 0.2}


# ---------------------------------------------------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------------------------------------------------
def _attention(q, k, v, causal, kpm=None):
    """q, k, v [B, H, S, hd]; one sequence at a time, so that the scores of the large cases fit."""
    outs = []
    for b in range(q.shape[0]):
        s = q[b] @ k[b].transpose(-1, -2) * q.shape[-1] ** -0.5
        if causal:
            s = s.masked_fill(torch.ones(s.shape[-2:], dtype=torch.bool, device=DEV).triu(1), float("-inf"))
        if kpm is not None:
            s = s.masked_fill(kpm[b][None, None], float("-inf"))
        outs.append(torch.softmax(s, -1) @ v[b])
    return torch.stack(outs)


def _self_attention(x, w, b, heads, causal=True, rope=None):
    """x [B, S, D] -> [B, S, D] before the output projection."""
    B, S, D = x.shape
    q, k, v = (t.view(B, S, heads, D // heads).transpose(1, 2) for t in F.linear(x, w, b).split(D, -1))
    if rope is not None:
        q, k = rope(q), rope(k)
    return _attention(q, k, v, causal).transpose(1, 2).reshape(B, S, D)


def _rope(S, hd):
    inv = 1.0 / (10000.0 ** (torch.arange(0, hd, 2, device=DEV, dtype=torch.float64) / hd))
    fr = torch.outer(torch.arange(S, device=DEV, dtype=torch.float64), inv)
    c, s = fr.cos(), fr.sin()

    def turn(x):
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, a * s + b * c], -1).flatten(-2)
    return turn


def _logits(c, w, ids):
    """Logits of the models in the weights' precision, [B, S, V]."""
    D, L, heads = c["d"], c["layers"], c["heads"]
    if c["kind"] == "lm":
        S = c["seq"]
        div = torch.exp(torch.arange(0, D, 2).float() * (-math.log(10000.0) / D))
        pos = torch.arange(0, S, dtype=torch.float).unsqueeze(1) * div
        pe = torch.zeros(S, D)
        pe[:, 0::2], pe[:, 1::2] = torch.sin(pos), torch.cos(pos)
        x = w["0.embedding.embedding.weight"][ids.t()] * math.sqrt(D) + pe.to(DEV, BF).double()
        for i in range(2, 2 + L):
            a, f = f"{i}.self_attn.MultiheadAttention.", f"{i}.ff_block."
            y = _self_attention(x, w[a + "in_proj_weight"], w[a + "in_proj_bias"], heads)
            x = x + F.linear(y, w[a + "out_proj.weight"], w[a + "out_proj.bias"])
            x = F.layer_norm(x, (D,), w[f"{i}.norm1.weight"], w[f"{i}.norm1.bias"])
            y = torch.relu(F.linear(x, w[f + "linear1.linear.weight"], w[f + "linear1.linear.bias"]))
            x = x + F.linear(y, w[f + "linear2.linear.weight"], w[f + "linear2.linear.bias"])
            x = F.layer_norm(x, (D,), w[f"{i}.norm2.weight"], w[f"{i}.norm2.bias"])
        return F.linear(x, w[f"{2 + L}.linear.linear.weight"], w[f"{2 + L}.linear.linear.bias"])
    x = w["tok.embedding.weight"][ids]
    if c["kind"] == "gpt":
        x = x + w["pos"][:ids.shape[1]]
        for i in range(L):
            p = f"blocks.{i}."
            a = p + "attn.MultiheadAttention."
            y = F.layer_norm(x, (D,), w[p + "ln1.weight"], w[p + "ln1.bias"])
            y = _self_attention(y, w[a + "in_proj_weight"], w[a + "in_proj_bias"], heads)
            x = x + F.linear(y, w[a + "out_proj.weight"], w[a + "out_proj.bias"])
            y = F.layer_norm(x, (D,), w[p + "ln2.weight"], w[p + "ln2.bias"])
            y = F.gelu(F.linear(y, w[p + "fc1.linear.weight"], w[p + "fc1.linear.bias"]))
            x = x + F.linear(y, w[p + "fc2.linear.weight"], w[p + "fc2.linear.bias"])
        x = F.layer_norm(x, (D,), w["ln_f.weight"], w["ln_f.bias"])
    else:
        def rms(t, g):
            return t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + 1e-5) * g
        rope = _rope(ids.shape[1], D // heads)
        for i in range(L):
            p = f"blocks.{i}."
            y = _self_attention(rms(x, w[p + "norm1.weight"]), w[p + "qkv.linear.weight"], None, heads, rope=rope)
            x = x + F.linear(y, w[p + "proj.linear.weight"])
            u, v = F.linear(rms(x, w[p + "norm2.weight"]), w[p + "gate_up.linear.weight"]).chunk(2, -1)
            x = x + F.linear(F.silu(u) * v, w[p + "down.linear.weight"])
        x = rms(x, w["norm.weight"])
    return F.linear(x, w["head.linear.weight"])


def exact(case, seed):
    c = case
    if c.get("dropout"):
        return None                    # the masks come from the library's own generator
    if c["kind"] in ("lm", "gpt", "llama"):
        g = _gen(seed)
        w = {n: t.double() for n, t in _weights(c, g).items()}
        ids, tgt = _tokens(c, g)
        if c["kind"] != "lm" and not c["train"]:
            with torch.no_grad():
                return _logits(c, w, ids)
        if c["kind"] == "lm" and not c["keep_grads"]:
            return None                # updated weights: an update's direction hangs on the sign of gradients near zero
        for t in w.values():
            t.requires_grad_()
        target = tgt.t() if c["kind"] == "lm" else tgt
        loss = F.cross_entropy(_logits(c, w, ids).flatten(0, 1), target.reshape(-1))
        grads = torch.autograd.grad(loss, list(w.values()))
        return [loss.detach().reshape(1) if c["kind"] == "lm" else loss.detach(), list(grads)]
    if c["kind"] == "attn":
        if c["batch"] * c["heads"] * c["sq"] * c["sk"] > 3e9:
            return None
        q, k, v, do, kpm = _tensors(c, seed)
        q, k, v = (t.double().requires_grad_() for t in (q, k, v))
        o = _attention(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), c["causal"], kpm).transpose(1, 2)
        return [o.detach(), *torch.autograd.grad(o, (q, k, v), do.double())]
    if c["kind"] == "moe":
        return _exact_moe(c, seed)
    x, dy, w, b = (t.double() for t in _tensors(c, seed))
    for t in (x, w, b):
        t.requires_grad_()
    cols = F.unfold(x, c["kernel"], 1, c["padding"], c["stride"])
    y = (w.flatten(1) @ cols + b[:, None]).view(dy.shape)
    return [y.detach(), *torch.autograd.grad(y, (x, w, b), dy)]


def _exact_moe(c, seed):
    x, dy, ws = _tensors(c, seed)
    E, D = c["experts"], c["d"]
    S = x.shape[0] * x.shape[1]
    cap = int(c["capacity"] * 2 * S // E)
    # which experts a token goes to is decided on bf16 logits and the seeded noise; everything behind it is in 64 bits
    lg = F.linear(x.view(S, D), ws[0])
    torch.manual_seed(int(seed))
    one = torch.tensor(1.0, device=DEV)
    noise = torch.distributions.gumbel.Gumbel(torch.zeros_like(one), one).rsample((S, E))
    i1 = torch.softmax(lg.float(), 1).argmax(1)
    m1 = F.one_hot(i1, E)
    i2 = (lg.float() + noise).masked_fill(m1.bool(), float("-inf")).argmax(1)
    m2 = F.one_hot(i2, E)
    l1 = ((m1.cumsum(0) - 1) * m1).sum(1)
    l2 = ((m2.cumsum(0) - 1 + m1.sum(0)) * m2).sum(1)
    keep1, keep2 = (l1 < cap).double(), (l2 < cap).double()
    x = x.double().requires_grad_()
    ws = [t.double().requires_grad_() for t in ws]
    xs = x.view(S, D)
    gates = torch.softmax(F.linear(xs, ws[0]), 1)
    aux = (gates.mean(0) * m1.double().mean(0)).mean()
    g1, g2 = gates.gather(1, i1[:, None])[:, 0] * keep1, gates.gather(1, i2[:, None])[:, 0] * keep2
    den = (g1 + g2).clamp(min=torch.finfo(torch.float32).eps)
    out = torch.zeros(S, D, dtype=torch.float64, device=DEV)
    for e in range(E):
        w1, b1, w2, b2 = ws[1 + 4 * e: 5 + 4 * e]
        for i, g, keep in ((i1, g1, keep1), (i2, g2, keep2)):
            rows = ((i == e) & (keep > 0)).nonzero()[:, 0]
            h = F.linear(F.gelu(F.linear(xs[rows], w1, b1)), w2, b2) * (g / den)[rows, None]
            out = out.index_add(0, rows, h)
    out = out.view(dy.shape)
    grads = torch.autograd.grad((out, aux), [x, *ws], (dy.double(), torch.ones_like(aux)))
    return [out.detach(), aux.detach(), *grads]
