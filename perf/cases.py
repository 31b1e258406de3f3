"""The work this framework is timed on.

Each case is one call that a training or serving program makes, through the package's own operators and models, on the
shapes of the configurations in ``linear_moe_b200/config/presets.py`` and of the benchmarks:

* ``scan``       linear attention with a scalar decay per head (lightning, retention, simple GLA / SSD)
* ``gated``      linear attention with a decay per key channel (GLA, HGRN2)
* ``delta``      the delta rule, plain and gated (DeltaNet, Gated DeltaNet)
* ``attention``  causal grouped-query softmax attention (the ``N`` layers of a hybrid)
* ``moe``        the experts of a mixture-of-experts layer: dispatch, expert MLPs, weighted combine
* ``decode``     one-token steps of a linear model, replayed from a CUDA graph
* ``train``      loss and gradients of a whole (small) linear transformer

``train: True`` is a forward and a backward pass with every input's gradient, ``False`` a forward pass as in evaluation
and prefill.  All of it runs in bf16 with fp32 decays, states and routing weights, as the presets do.
"""
import math

import torch
import torch.nn.functional as F

from linear_moe_b200 import ops
from linear_moe_b200.config.presets import get_preset
from linear_moe_b200.infer.generation import GraphedDecodeStep
from linear_moe_b200.models.transformer import CausalLM
from linear_moe_b200.ops.moe_fused import fused_moe
from linear_moe_b200.parallel import fused_comm

EPS_NORM, EPS_HEAD = 1e-5, 1e-5          # norm constants of the llama3 presets: block norms, per-head output norm


def listed():
    return [
        # lightning attention of the 1B dense model, its 16384 tokens per GPU: one layer's scan in a training step
        dict(name="scan_train_16k", kind="scan", B=1, T=16384, H=16, D=128, decay="head", train=True),
        # a short ragged prompt through a per-token-decay model with 64-wide heads, going on from a cached state
        dict(name="scan_prefill_777", kind="scan", B=1, T=777, H=8, D=64, decay="token", train=False),
        # GLA of the A0.3B-2B model: 8 sequences of 2048 tokens, 8 heads of 128
        dict(name="gated_train_8x2k", kind="gated", B=8, T=2048, H=8, D=128, train=True),
        # Gated DeltaNet of the A1B-7B hybrid: 2 sequences of 4096 tokens, 16 heads of 128
        dict(name="delta_train_2x4k", kind="delta", B=2, T=4096, H=16, D=128, gate=True, train=True),
        # ragged prompts through plain DeltaNet layers
        dict(name="delta_prefill_3x1111", kind="delta", B=3, T=1111, H=8, D=128, gate=False, train=False),
        # softmax layer of the same hybrid: 16 query heads on 4 kv heads
        dict(name="attention_train_2x4k", kind="attention", B=2, T=4096, ctx=0, H=16, HKV=4, D=128, window=0, train=True),
        # the second half of a prompt against a cached context, 64-wide heads as in the 1B llama3 preset
        dict(name="attention_prefill_1531", kind="attention", B=1, T=1531, ctx=1021, H=32, HKV=8, D=64, window=0, train=False),
        # experts of the A0.3B-2B model: 64 experts of 896, top 8, 8192 tokens
        dict(name="moe_train_8k", kind="moe", T=8192, E=64, K=8, hidden=1024, ffn=896, train=True),
        # four layers of the 1B dense model generating for 8 requests
        dict(name="decode_b8", kind="decode", B=8, layers=4, hidden=2048, ffn=8192, vocab=128256),
        # two layers of the 1B dense model with a 32000-token vocabulary: forward, loss and every weight's gradient
        dict(name="train_2_layers_4k", kind="train", B=1, T=4096, layers=2, hidden=2048, ffn=8192, vocab=32000),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan", "scan", "gated", "gated", "delta", "delta", "attention", "attention", "moe", "decode", "train"])
    D = rng.choice([64, 128, 128])
    train = rng.random() < 0.6
    if kind in ("scan", "gated", "delta"):
        H = rng.choice([4, 8, 12, 16, 32])
        B = rng.choice([1, 1, 2, 4, 8])
        T = _log(rng, 100, max(200, (262144 if kind == "scan" else 131072) // (H * B)))
        T -= T % rng.choice([1, 64])
        more = {"scan": {"decay": rng.choice(["none", "head", "token"])}, "gated": {}, "delta": {"gate": rng.random() < 0.5}}[kind]
        return dict(kind=kind, B=B, T=T, H=H, D=D, train=train, **more)
    if kind == "attention":
        rep = rng.choice([1, 2, 4, 7])
        H = rep * rng.choice([2, 4, 8])
        B = rng.choice([1, 1, 2, 4])
        T = _log(rng, 100, min(6000, int(math.sqrt(2 * 16 * 4096 * 4096 / (B * H)))))
        return dict(kind=kind, B=B, T=T, ctx=0 if train else rng.choice([0, T // 3]), H=H, HKV=H // rep, D=D,
                    window=rng.choice([0, 0, max(64, T // 3)]), train=train)
    if kind == "moe":
        E = rng.choice([8, 16, 64])
        hidden, ffn = rng.choice([(1024, 896), (1024, 512), (512, 896)])
        return dict(kind=kind, T=_log(rng, 200, 8192), E=E, K=rng.choice([2, 4, 8]), hidden=hidden, ffn=ffn, train=train)
    hidden = rng.choice([512, 1024, 2048])
    if kind == "decode":
        return dict(kind=kind, B=rng.randint(1, 16), layers=rng.randint(1, 4), hidden=hidden, ffn=4 * hidden,
                    vocab=rng.choice([32000, 128256]))
    return dict(kind=kind, B=rng.choice([1, 2]), T=_log(rng, 200, 2048), layers=rng.randint(1, 2), hidden=hidden,
                ffn=4 * hidden, vocab=rng.choice([8000, 32000]))


# ---- inputs ----------------------------------------------------------------------------------------
def _inputs(case, seed):
    """Tensors of a case on the GPU, from the seed alone."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed) * 1000003 + 17)

    def normal(*shape, std=1.0):
        return torch.randn(*shape, device=dev, generator=gen).mul_(std)

    kind, x = case["kind"], {}
    if kind in ("scan", "gated", "delta"):
        B, T, H, D = case["B"], case["T"], case["H"], case["D"]
        # one projection holds q | k | v of every head, as the layers lay it out
        x["qkv"] = normal(B, T, H, 3 * D, std=0.5).bfloat16()
        if kind == "scan":
            if case["decay"] == "head":          # slopes 2^(-8 i / H)
                x["g"] = -torch.exp2(-8.0 * torch.arange(1, H + 1, device=dev, dtype=torch.float32) / H)
            elif case["decay"] == "token":       # simple GLA / SSD: log decays around -0.05
                x["g"] = F.logsigmoid(normal(B, T, H)) / 16
        elif kind == "gated":
            x["g"] = F.logsigmoid(normal(B, T, H, D)) / 16
        else:
            q, k, v = x["qkv"].float().split(D, dim=-1)          # unit keys and queries, as after ops.l2_norm
            x = {"q": F.normalize(q, dim=-1).bfloat16(), "k": F.normalize(k, dim=-1).bfloat16(), "v": v.bfloat16(),
                 "beta": torch.sigmoid(normal(B, T, H))}
            if case["gate"]:
                x["g"] = F.logsigmoid(normal(B, T, H)) / 16
        if case["train"]:
            x["d_o"] = normal(B, T, H, D).bfloat16()
        else:
            x["init"] = normal(B, H, D, D, std=0.3)              # the state a cache holds
    elif kind == "attention":
        B, T, H, HKV, D, n = case["B"], case["T"], case["H"], case["HKV"], case["D"], case["T"] + case["ctx"]
        x["q"], x["k"], x["v"] = normal(B, T, H, D).bfloat16(), normal(B, n, HKV, D).bfloat16(), normal(B, n, HKV, D).bfloat16()
        if case["train"]:
            x["d_o"] = normal(B, T, H, D).bfloat16()
    elif kind == "moe":
        T, E, K, hid, f = case["T"], case["E"], case["K"], case["hidden"], case["ffn"]
        x["h"] = normal(T, hid).bfloat16()
        probs, x["idx"] = torch.topk(torch.softmax(normal(T, E), -1), K, dim=-1)
        x["probs"] = probs.contiguous()
        x["w1"], x["w2"] = normal(E, hid, 2 * f, std=0.03).bfloat16(), normal(E, f, hid, std=0.03).bfloat16()
        if case["train"]:
            x["d_o"] = normal(T, hid).bfloat16()
    else:
        n = 64 if kind == "decode" else case["T"]
        x["ids"] = torch.randint(0, case["vocab"], (case["B"], n + 1), device=dev, generator=gen)
    return x


def _model(case, seed):
    h, n = case["hidden"], case["layers"]
    cfg = get_preset("bench-lasp2-llama3-1b", num_layers=n, layer_type_list="L" * n, hidden_size=h, num_attention_heads=h // 128,
                     ffn_hidden_size=case["ffn"], vocab_size=case["vocab"])
    model = CausalLM(cfg, device=torch.device("cuda"))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 7919 + 5)
    with torch.no_grad():
        for p in model.parameters():             # trained weights are no longer exactly what the initialiser gave
            p.mul_(torch.empty_like(p, dtype=torch.float32).uniform_(0.5, 1.5, generator=gen).to(p.dtype))
    return model


def _params(model):
    return [p for _, p in model.named_parameters()]


def prepare(case, seed):
    x = _inputs(case, seed)
    s = {"case": case, "x": x}
    if case["kind"] == "train":
        s["model"] = _model(case, seed).train()
    elif case["kind"] == "decode":
        model = _model(case, seed).eval()
        with torch.no_grad():
            caches = model.new_cache()
            model(x["ids"][:, :-1], caches=caches)                       # the prompt
            tok = x["ids"][:, -1:].contiguous()
            keep = [{k: v.clone() for k, v in c.items()} for c in caches]
            for _ in range(2):
                model(tok, caches=caches, position_offset=0)
            step = GraphedDecodeStep(model, caches, case["B"], tok.device)
            step(tok)                                                    # captures; the state goes back to the prompt's end
            for c, kept in zip(caches, keep):
                for name, v in kept.items():
                    c[name].copy_(v)
        s.update(step=step, caches=caches, tok=tok)
    else:
        for name, t in x.items():
            if case["train"] and t.is_floating_point() and name not in ("d_o", "init"):
                t.requires_grad_(not (name == "g" and t.dim() == 1))     # slopes are constants of the model
        if case["kind"] == "moe":
            rows = case["T"] * case["K"] + 256 * case["E"]
            s["ws"] = fused_comm.local_moe_workspace(case["E"], case["hidden"], rows, x["h"].device)
    return s


def _forward(case, x, ws=None):
    kind = case["kind"]
    if kind in ("scan", "gated"):
        D = case["D"]
        q, k, v = x["qkv"].split(D, dim=-1)
        if kind == "scan":
            return ops.lsm_scalar(q, k, v, x.get("g"), 1.0 if case["decay"] == "head" else None, x.get("init"))
        return ops.lsm_vector(q, k, v, x["g"], None, x.get("init"))
    if kind == "delta":
        return ops.lsm_delta(x["q"], x["k"], x["v"], x["beta"], x.get("g"), None, x.get("init"))
    if kind == "attention":
        return (ops.softmax_attention(x["q"], x["k"], x["v"], None, True, case["ctx"], case["window"] or None),)
    return (fused_moe(x["h"], x["probs"], x["idx"], x["w1"], x["w2"], ws),)


def run(state):
    case, x = state["case"], state["x"]
    if case["kind"] == "decode":
        with torch.no_grad():
            logits = state["step"](state["tok"])
        return {"logits": logits, "states": [c["state"] for c in state["caches"]]}
    if case["kind"] == "train":
        model, ids = state["model"], x["ids"]
        loss = model(ids[:, :-1], ids[:, 1:].contiguous())
        return {"loss": loss, "grads": list(torch.autograd.grad(loss.mean(), _params(model)))}
    if not case["train"]:
        with torch.no_grad():
            return {"out": list(_forward(case, x, state.get("ws")))}
    out = _forward(case, x, state.get("ws"))
    wrt = [t for t in x.values() if t.requires_grad]
    grads = torch.autograd.grad(out[0], wrt, x["d_o"])
    return {"out": [o.detach() for o in out], "grads": list(grads)}


# ---- what a pass cannot do without -------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("scan", "gated", "delta"):
        B, T, H, D = case["B"], case["T"], case["H"], case["D"]
        n, s = B * T * H, B * H * D * D
        gates = {"scan": 4 * n if case.get("decay") == "token" else 0, "gated": 4 * n * D,
                 "delta": 4 * n * (2 if case.get("gate") else 1)}[kind]
        fwd = n * D * 2 * 4 + gates + s * 4                      # q, k, v in, o out, decays, final state
        per = 6 if kind == "delta" else 4                        # multiply-adds with the D x D state: 2 D^2 flops each
        if not case["train"]:
            return {"bytes": fwd + s * 4, "flops": per * n * D * D}
        # backward: q, k, v, d_o and the decays in, their gradients out
        return {"bytes": fwd + n * D * 2 * 7 + 2 * gates, "flops": 3.5 * per * n * D * D}
    if kind == "attention":
        B, T, H, HKV, D, ctx, w = (case[k] for k in ("B", "T", "H", "HKV", "D", "ctx", "window"))
        pairs = sum(min(i + 1 + ctx, w or i + 1 + ctx) for i in range(T)) * B * H
        q, kv = B * T * H * D * 2, B * (T + ctx) * HKV * D * 2
        if not case["train"]:
            return {"bytes": 2 * q + 2 * kv, "flops": 4 * pairs * D}
        return {"bytes": 2 * q + 2 * kv + 4 * q + 4 * kv, "flops": 14 * pairs * D}
    if kind == "moe":
        T, E, K, hid, f = (case[k] for k in ("T", "E", "K", "hidden", "ffn"))
        weights, acts, flops = E * hid * 3 * f * 2, 2 * T * hid * 2 + T * K * 8, 6 * T * K * hid * f
        if not case["train"]:
            return {"bytes": weights + acts, "flops": flops}
        return {"bytes": 3 * weights + 2 * acts + T * hid * 2, "flops": 3 * flops}
    h, f, n, V, B = (case[k] for k in ("hidden", "ffn", "layers", "vocab", "B"))
    per_layer = h * 5 * h + 3 * h * f                            # q|k|v, output gate, output; gate|up, down
    if kind == "decode":
        state = n * B * (h // 128) * 128 * 128 * 4
        return {"bytes": 2 * (n * per_layer + V * h) + 2 * state + 2 * B * V, "flops": 2 * B * (n * per_layer + V * h)}
    T = case["T"]
    weights = n * per_layer + V * h
    mix = n * B * T * h * 128 * 14
    return {"bytes": 2 * 2 * (weights + V * h), "flops": 6 * B * T * weights + mix}


def tolerance(case):
    """About four times the distance from 64-bit results that these paths show: bf16 operands and results leave 0.002 - 0.0045.
    A gradient of per-token decays is a running sum over bf16 products (0.024 - 0.043), and in whole models the roundings of
    every layer add up (logits and states 0.03, weight gradients 0.04)."""
    if case["kind"] in ("decode", "train"):
        return {"rel": 0.1}
    if case["train"] and (case["kind"] == "gated" or (case["kind"] == "scan" and case["decay"] == "token")):
        return {"rel": 0.12}
    return {"rel": 0.016}


# ---- the same in 64 bits --------------------------------------------------------------------------------
def _recurrence(kind, q, k, v, g, beta, scale, init):
    """Chunked form of the three recurrences for ``[B, H, T, D]``; the decays ``g [B, H, T, D or 1]`` may be None."""
    B, H, T, D = q.shape
    S = q.new_zeros(B, H, D, v.shape[-1]) if init is None else init
    out = []
    C = 32
    lower = torch.ones(C, C, dtype=torch.bool, device=q.device).tril()
    for t in range(0, T, C):
        Q, K, V = q[:, :, t:t + C], k[:, :, t:t + C], v[:, :, t:t + C]
        n = Q.shape[2]
        m = lower[:n, :n]
        b = torch.zeros_like(Q[..., :1]) if g is None else g[:, :, t:t + n].cumsum(2)
        end = b[:, :, -1:]
        up, down = Q * b.exp(), K * (-b).exp()
        if kind == "delta":
            bt = beta[:, :, t:t + n, None]
            A = ((K * b.exp()) @ down.transpose(-1, -2)).masked_fill(~m.tril(-1), 0.0) * bt
            eye = torch.eye(n, dtype=q.dtype, device=q.device)
            rhs = bt * (V - (K * b.exp()) @ S)
            V = torch.linalg.solve_triangular(eye + A, rhs, upper=False, unitriangular=True)
        P = (up @ down.transpose(-1, -2)).masked_fill(~m, 0.0)
        out.append(scale * (P @ V + up @ S))
        S = end.exp().transpose(-1, -2) * S + (K * (end - b).exp()).transpose(-1, -2) @ V
    return torch.cat(out, 2), S


def _exact_mixer(case, x):
    kind, D = case["kind"], case["D"]
    d = {n: t.detach().double().requires_grad_(case["train"] and n not in ("d_o", "init") and not (n == "g" and t.dim() == 1))
         for n, t in x.items()}
    heads = lambda t: t.transpose(1, 2)                          # noqa: E731
    q, k, v = d["qkv"].split(D, dim=-1) if "qkv" in d else (d["q"], d["k"], d["v"])
    g = d.get("g")
    if g is not None:
        if g.dim() == 1:
            g = g[None, None, :].expand(case["B"], case["T"], -1)
        g = heads(g[..., None] if g.dim() == 3 else g)
    scale = 1.0 if case.get("decay") == "head" else D ** -0.5
    beta = heads(d["beta"]) if "beta" in d else None
    o, S = _recurrence(kind, heads(q), heads(k), heads(v), g, beta, scale, d.get("init"))
    o = heads(o)
    if not case["train"]:
        return {"out": [o, S]}
    wrt = [t for t in d.values() if t.requires_grad]
    return {"out": [o.detach(), S.detach()], "grads": list(torch.autograd.grad(o, wrt, d["d_o"]))}


def _exact_attention(case, x):
    B, T, H, HKV, D, ctx, w = (case[k] for k in ("B", "T", "H", "HKV", "D", "ctx", "window"))
    q, k, v = (x[n].detach().double() for n in ("q", "k", "v"))
    i = torch.arange(T, device=q.device)[:, None] + ctx
    j = torch.arange(T + ctx, device=q.device)[None, :]
    hidden = (j > i) | (j <= i - w) if w else j > i
    out, dq, dk, dv = torch.empty_like(q), torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
    for b in range(B):
        for h in range(H):
            e = h * HKV // H
            Q, K, V = q[b, :, h], k[b, :, e], v[b, :, e]
            P = torch.softmax((Q @ K.t() * D ** -0.5).masked_fill(hidden, -math.inf), -1)
            out[b, :, h] = P @ V
            if case["train"]:
                dO = x["d_o"][b, :, h].double()
                dP = dO @ V.t()
                dS = P * (dP - (P * dP).sum(-1, keepdim=True)) * D ** -0.5
                dq[b, :, h] = dS @ K
                dk[b, :, e] += dS.t() @ Q
                dv[b, :, e] += P.t() @ dO
    return {"out": [out], "grads": [dq, dk, dv]} if case["train"] else {"out": [out]}


def _exact_moe(case, x):
    f = case["ffn"]
    names = ("h", "probs", "w1", "w2")
    h, probs, w1, w2 = (x[n].detach().double() for n in names)
    dO = x["d_o"].double() if case["train"] else None
    out, grads = torch.zeros_like(h), [torch.zeros_like(t) for t in (h, probs, w1, w2)]
    for e in range(case["E"]):
        t, slot = (x["idx"] == e).nonzero(as_tuple=True)
        X, p = h[t], probs[t, slot][:, None]
        y = X @ w1[e]
        gate, up = y[:, :f], y[:, f:]
        s = torch.sigmoid(gate)
        act = gate * s * up
        z = act @ w2[e]
        out.index_add_(0, t, p * z)
        if case["train"]:
            grads[1][t, slot] = (z * dO[t]).sum(-1)
            dz = p * dO[t]
            da = dz @ w2[e].t()
            dy = torch.cat([da * up * s * (1 + gate * (1 - s)), da * gate * s], 1)
            grads[0].index_add_(0, t, dy @ w1[e].t())
            grads[2][e], grads[3][e] = X.t() @ dy, act.t() @ dz
    return {"out": [out], "grads": grads} if case["train"] else {"out": [out]}


def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _exact_model(case, p, ids):
    """The dense transformer with lightning attention; ``p``: its weights by name.  Returns hidden rows and the states."""
    H, D = case["hidden"] // 128, 128
    slopes = -torch.exp2(-8.0 * torch.arange(1, H + 1, device=ids.device, dtype=torch.float64) / H)
    if H & (H - 1):
        raise ValueError("the slopes of this model are those of a power of two")
    r = p["embedding.word_embeddings.weight"][ids]
    B, T, _ = r.shape
    states = []
    for i in range(case["layers"]):
        at = lambda n, i=i: p["decoder.layers.%d.%s" % (i, n)]   # noqa: E731
        x = _rms(r, at("input_layernorm.weight"), EPS_NORM)
        q, k, v = (x @ at("self_attention.qkv_proj.weight").t()).view(B, T, H, 3 * D).transpose(1, 2).split(D, dim=-1)
        gate = x @ at("self_attention.o_gate_proj.weight").t()
        o, S = _recurrence("scan", q, k, v, slopes[None, :, None, None].expand(B, H, T, 1), None, 1.0, None)
        states.append(S)
        o = _rms(o.transpose(1, 2), at("self_attention.core_linear_attention.la_output_norm.weight"), EPS_HEAD)
        r = r + (o.reshape(B, T, H * D) * F.silu(gate)) @ at("self_attention.o_proj.weight").t()
        x = _rms(r, at("pre_mlp_layernorm.weight"), EPS_NORM)
        a, b = (x @ at("mlp.linear_fc1.weight").t()).chunk(2, -1)
        r = r + (F.silu(a) * b) @ at("mlp.linear_fc2.weight").t()
    return _rms(r, p["decoder.final_layernorm.weight"], EPS_NORM), states


def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode", "train"):
        x = _inputs(case, seed)
        named = [(n, t.detach()) for n, t in _model(case, seed).named_parameters()]
        p = {n: t.double().requires_grad_(kind == "train") for n, t in named}
        ids = x["ids"]
        if kind == "decode":
            h, states = _exact_model(case, p, ids)
            return {"logits": h[:, -1:] @ p["output_layer.weight"].t(), "states": states}
        h, _ = _exact_model(case, p, ids[:, :-1])
        lp = F.log_softmax(h @ p["output_layer.weight"].t(), -1)
        loss = -lp.gather(-1, ids[:, 1:, None]).squeeze(-1)
        return {"loss": loss.detach(), "grads": list(torch.autograd.grad(loss.mean(), list(p.values())))}
    x = _inputs(case, seed)
    if kind == "attention":
        return _exact_attention(case, x)
    if kind == "moe":
        return _exact_moe(case, x)
    return _exact_mixer(case, x)
