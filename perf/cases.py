"""Measured cases: the dense decoder at the work that its users have it do - training steps (``TrainEngine.step``), scoring of given
tokens (``DenseModel.forward``) and serving (``InferenceEngine.feed``: prompts, then one token at a time over the paged cache).

The shapes are the framework's own presets: "50m" (llama-50m: heads of 64), "gpt2" (gpt2-small: layer norms, biases, learned positions, gelu;
its vocabulary padded to a multiple of 128) and "8b" (the widths of llama-3-8b: heads of 128, 32 over 8 key heads; 2 layers to train, 8 to
score and serve, and a vocabulary of 32000 so that head and layers keep the proportion of the full depth).  Weights are random, token ids uniform; as in
a trained model the residual stream is more than what one sublayer adds to it (rounding is not amplified from layer to layer).

``exact`` states the same decoder in float64.  Where weights or cache are quantised it is the decoder without quantisation: the rounding of the
format is then part of the error, the same on both sides."""
from __future__ import annotations

import math
import random

import torch

from transformers_fusion_b200.inference.engine import EngineConfig, InferenceEngine, Request
from transformers_fusion_b200.models.config import TransformerConfig
from transformers_fusion_b200.models.dense import DenseModel
from transformers_fusion_b200.trainer.engine import TrainEngine

SHAPES = {
    "50m": dict(V=32000, H=512, L=8, heads=8, kv=8, ff=1408, theta=10000.0, gpt2=False),
    "gpt2": dict(V=50304, H=768, L=12, heads=12, kv=12, ff=3072, theta=0.0, gpt2=True),
    "8b": dict(V=32000, H=4096, L=8, heads=32, kv=8, ff=14336, theta=500000.0, gpt2=False),
}
MAX_POS = 4096
EPS = {"50m": 1e-5, "gpt2": 1e-5, "8b": 1e-5}
LR, BETA1, BETA2, ADAM_EPS, DECAY, CLIP = 3e-4, 0.9, 0.95, 1e-8, 0.1, 1.0


def listed():
    train = lambda name, model, B, S, layers=0: dict(name=name, kind="train", model=model, batch=B, seq=S, layers=layers)
    serve = lambda name, model, n, lo, hi, steps, kv="bf16", weights="": dict(
        name=name, kind="serve", model=model, sequences=n, shortest=lo, longest=hi, steps=steps, kv=kv, weights=weights)
    return [
        train("train_50m_64x1024", "50m", 64, 1024),       # the headline configuration: one GPU takes the whole batch
        train("train_50m_8x1024", "50m", 8, 1024),         # the same as one of eight ranks sees it
        train("train_50m_1x131", "50m", 1, 131),           # smallest: a debugging or fine-tuning step on one short text, launches count
        train("train_gpt2_6x777", "gpt2", 6, 777),         # layer norms, biases, learned positions, gelu; a sequence length that fits no tile
        train("train_8b_1x4096", "8b", 1, 4096, 2),        # one sequence per GPU of the large configuration: grouped heads of 128
        dict(name="score_8b_2x2500", kind="score", model="8b", batch=2, seq=2500),       # perplexity, log-probabilities of given texts
        serve("prompts_8b_4", "8b", 4, 1000, 4000, 8),     # long prompts, short answers
        serve("decode_8b_1", "8b", 1, 200, 200, 64),       # one user: latency of a token
        serve("decode_8b_64", "8b", 64, 64, 256, 48),      # a full batch of chats
        serve("decode_8b_64_mxfp8_q4", "8b", 64, 64, 256, 48, "q4", "mxfp8"),    # the same in the formats of the serving load
        serve("decode_8b_8_int8_fp8", "8b", 8, 1500, 3000, 32, "fp8", "int8"),   # longer contexts, 8-bit weights and cache
        serve("decode_50m_16", "50m", 16, 32, 512, 64),    # a small model: steps of many short kernels
    ]


def _log_between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "score", "serve", "serve", "serve"])
    model = rng.choice(["50m", "50m", "gpt2", "8b"]) if kind != "serve" else rng.choice(["50m", "8b", "8b"])
    if kind == "serve":
        n = _log_between(rng, 1, 64)
        hi = _log_between(rng, 24, min(3000, 10000 // n) if model == "8b" else min(900, 20000 // n))
        lo = _log_between(rng, 16, hi)
        kv, weights = rng.choice([("bf16", ""), ("bf16", ""), ("fp8", ""), ("fp8", "int8"), ("q4", "mxfp8")]) if model == "8b" else rng.choice([("bf16", ""), ("fp8", "")])
        return dict(kind="serve", model=model, sequences=n, shortest=lo, longest=hi, steps=_log_between(rng, 8, 48), kv=kv, weights=weights)
    most = {"50m": 65536, "gpt2": 8192, "8b": 4096 if kind == "train" else 5000}[model]
    S = _log_between(rng, 64, {"50m": 1024, "gpt2": 1024, "8b": 4000}[model])
    B = max(1, min(_log_between(rng, 128, most), most) // S)
    return dict(kind=kind, model=model, batch=B, seq=S, layers=2 if model == "8b" and kind == "train" else 0)


# ------------------------------------------------------------------------------------------------- weights and inputs
def _shape(case):
    s = dict(SHAPES[case["model"]])
    s["L"] = case.get("layers") or s["L"]
    s["D"] = s["H"] // s["heads"]
    s["eps"] = EPS[case["model"]]
    return s


def _flat(s):
    """(name, shape) of every parameter in the order of the flat buffers; fused projections are named by their first part."""
    H, nq, nkv, F = s["H"], s["heads"] * s["D"], s["kv"] * s["D"], s["ff"]
    out = [("emb", (s["V"], H))]
    if s["gpt2"]:
        out += [("pos", (1024, H)), ("norm", (H,)), ("norm_b", (H,))]
    else:
        out += [("norm", (H,))] + ([("head", (s["V"], H))] if not _tied(s) else [])
    for i in range(s["L"]):
        if s["gpt2"]:
            out += [(f"{i}.n1", (H,)), (f"{i}.n1_b", (H,)), (f"{i}.qkv", (nq + 2 * nkv, H)), (f"{i}.qkv_b", (nq + 2 * nkv,)), (f"{i}.o", (H, nq)), (f"{i}.o_b", (H,)),
                    (f"{i}.n2", (H,)), (f"{i}.n2_b", (H,)), (f"{i}.up", (F, H)), (f"{i}.up_b", (F,)), (f"{i}.down", (H, F)), (f"{i}.down_b", (H,))]
        else:
            out += [(f"{i}.n1", (H,)), (f"{i}.qkv", (nq + 2 * nkv, H)), (f"{i}.o", (H, nq)), (f"{i}.n2", (H,)), (f"{i}.up", (2 * F, H)), (f"{i}.down", (H, F))]
    return out


def _tied(s):
    return s["H"] < 4096


def _weights(s, seed, dev):
    """name -> bf16 tensor: matrices N(0, 0.02), those that write to the residual divided by sqrt(2 layers), an embedding that is not the head
    as well N(0, 1), norms near one, biases near zero."""
    g = torch.Generator(device=dev).manual_seed(seed)
    W = {}
    for name, shape in _flat(s):
        r = torch.randn(shape, generator=g, device=dev, dtype=torch.float32)
        std = 1.0 if name == "emb" and not _tied(s) else 0.02 / math.sqrt(2 * s["L"]) if name.endswith((".o", ".down")) else 0.02
        W[name] = (r * std if len(shape) > 1 or name.endswith("_b") else 1 + 0.1 * r).bfloat16()
    return W


def _parts(s, W):
    """The weights under the names of the model's files (``named_tensors``)."""
    nq, nkv, F = s["heads"] * s["D"], s["kv"] * s["D"], s["ff"]
    out = {"tok_embeddings.weight": W["emb"], "norm.weight": W["norm"]}
    for ours, theirs in (("pos", "pos_embeddings.weight"), ("norm_b", "norm.bias"), ("head", "lm_head.weight")):
        if ours in W:
            out[theirs] = W[ours]
    for i in range(s["L"]):
        p = f"layers.{i}."
        w = lambda n: W[f"{i}.{n}"]
        for kind, sfx in (("weight", ""), ("bias", "_b")) if s["gpt2"] else (("weight", ""),):
            out[p + f"attention_norm.{kind}"], out[p + f"ffn_norm.{kind}"] = w("n1" + sfx), w("n2" + sfx)
            qkv = w("qkv" + sfx)
            out[p + f"attention.q_proj.{kind}"], out[p + f"attention.k_proj.{kind}"], out[p + f"attention.v_proj.{kind}"] = qkv[:nq], qkv[nq:nq + nkv], qkv[nq + nkv:]
            out[p + f"attention.o_proj.{kind}"], out[p + f"ffn.down_proj.{kind}"] = w("o" + sfx), w("down" + sfx)
            if s["gpt2"]:
                out[p + f"ffn.up_proj.{kind}"] = w("up" + sfx)
            else:
                out[p + f"ffn.gate_proj.{kind}"], out[p + f"ffn.up_proj.{kind}"] = w("up")[:F], w("up")[F:]
    return out


def _model(s, seed):
    dev = torch.device("cuda", 0)
    kw = dict(max_seq_len=1024, activation="gelu", norm_type="layernorm", position_type="learned", attention_bias=True, tie_embeddings=True) if s["gpt2"] else \
        dict(num_kv_heads=s["kv"], rope_theta=s["theta"], max_seq_len=MAX_POS, activation="swiglu", tie_embeddings=_tied(s))
    cfg = TransformerConfig(vocab_size=s["V"], hidden_size=s["H"], num_layers=s["L"], num_heads=s["heads"], ffn_hidden_size=s["ff"], norm_eps=s["eps"], **kw)
    model = DenseModel(cfg, device=dev, dtype=torch.bfloat16, seed=None)
    parts = _parts(s, _weights(s, seed, dev))
    with torch.no_grad():
        for name, t in model.named_tensors():
            t.copy_(parts.pop(name))
    assert not parts, sorted(parts)
    return model


def _ids(s, shape, seed, dev):
    return torch.randint(0, s["V"], shape, generator=torch.Generator(device=dev).manual_seed(seed + 7919), device=dev)


def _lengths(case):
    """Prompt lengths: a property of the case, the same for every seed."""
    n, lo, hi = case["sequences"], case["shortest"], case["longest"]
    rng = random.Random(n * 1000003 + lo * 1009 + hi)
    return [rng.randint(lo, hi) for _ in range(n)]


def prepare(case, seed):
    dev, s = torch.device("cuda", 0), _shape(case)
    model = _model(s, seed)
    if case["kind"] == "serve":
        lens, steps = _lengths(case), case["steps"]
        cfg = EngineConfig(max_batch=len(lens), num_pages=sum((n + steps) // 16 + 2 for n in lens), kv_mode=case["kv"], max_seq_len=max(lens) + steps + 16,
                           enable_prefix_cache=False, weight_format=case["weights"])
        ids = _ids(s, (sum(lens) + steps * len(lens),), seed, dev).tolist()      # what a tokenizer returns: lists
        prompts, at = [], 0
        for n in lens:
            prompts.append(ids[at:at + n])
            at += n
        return dict(kind="serve", engine=InferenceEngine(model, None, cfg), prompts=prompts, answers=[ids[at + t * len(lens):at + (t + 1) * len(lens)] for t in range(steps)])
    ids = _ids(s, (case["batch"], case["seq"] + 1), seed, dev)
    if case["kind"] == "score":
        return dict(kind="score", model=model, ids=ids[:, :-1].contiguous())
    engine = TrainEngine(model, lr=LR, betas=(BETA1, BETA2), eps=ADAM_EPS, weight_decay=DECAY, max_grad_norm=CLIP, cuda_graph=True)
    return dict(kind="train", engine=engine, ids=ids[:, :-1].contiguous(), labels=ids[:, 1:].contiguous())


def run(state):
    if state["kind"] == "train":                  # the first moments are the clipped gradients' running mean: after one step a tenth of them
        e = state["engine"]
        loss = e.step(state["ids"], state["labels"])
        return {"loss": loss, "master": e.opt.master, "m": e.opt.m, "v": e.opt.v}
    with torch.no_grad():
        if state["kind"] == "score":
            return {"logits": state["model"](state["ids"])}
        eng = state["engine"]
        reqs = [Request([]) for _ in state["prompts"]]
        first = eng.feed([(r, p, [len(p) - 1]) for r, p in zip(reqs, state["prompts"])])
        last = None
        for t, answer in enumerate(state["answers"]):
            want = [0] if t == len(state["answers"]) - 1 else []       # the last step's logits depend on all that was cached before
            last = eng.feed([(r, [tok], want) for r, tok in zip(reqs, answer)])
        for r in reqs:
            eng.end(r)
        return {"first": torch.cat(first), "last": torch.cat(last)}


# ------------------------------------------------------------------------------------------------- what a pass cannot do without
def _matrix_params(s):
    nq, nkv = s["heads"] * s["D"], s["kv"] * s["D"]
    return s["L"] * s["H"] * (nq + 2 * nkv + nq + (2 if s["gpt2"] else 3) * s["ff"])


def work(case):
    s = _shape(case)
    per_layer, head = _matrix_params(s), s["V"] * s["H"]
    nq, kv_row = s["heads"] * s["D"], 2 * s["kv"] * s["D"] * s["L"]
    if case["kind"] == "serve":
        lens, steps = _lengths(case), case["steps"]
        n, tokens, pairs = len(lens), sum(lens), sum(x * (x + 1) // 2 for x in lens)
        later = sum(steps * x + steps * (steps + 1) // 2 for x in lens)
        width = {"": 2.0, "int8": 1.0 + 2 / 32, "mxfp8": 1.0 + 2 / 32}[case["weights"]]
        cached = {"bf16": 2.0, "fp8": 1.0 + 4 / s["D"], "q4": 0.5 + 2 / 32}[case["kv"]]
        flops = 2.0 * per_layer * (tokens + n * steps) + 2.0 * head * 2 * n + 4.0 * nq * s["L"] * (pairs + later)
        return {"flops": flops, "bytes": (per_layer * width) * (steps + 1) + 2.0 * head * 2 + kv_row * cached * (tokens + n * steps + later) + 4.0 * n * s["V"]}
    B, S = case["batch"], case["seq"]
    T, pairs = B * S, B * (S * (S + 1) // 2)
    if case["kind"] == "score":
        return {"flops": 2.0 * (per_layer + head) * T + 4.0 * nq * s["L"] * pairs, "bytes": 2.0 * (per_layer + 2 * head) + 2.0 * T * s["V"]}
    n = sum(math.prod(shape) for _, shape in _flat(s))
    return {"flops": 6.0 * (per_layer + head) * T + 14.0 * nq * s["L"] * pairs, "bytes": n * (2 + 2 + 24.0) + T * 16.0}


def tolerance(case):
    # bf16 activations: 0.8 - 1.2 % from the float64 statement, two correct orders of the sums up to sqrt(2) times that apart (measured: up to
    # 1.4 % between two runs whose split sums meet in another order; 2.6 % where rounding to 8-bit weights or cache entries flips as well)
    if case["kind"] == "train":
        return {"rel": 0.03, "max": 0.95}
    return {"rel": 0.03, "max": 0.9 if case.get("weights") or case.get("kv", "bf16") != "bf16" else 0.3}


# ------------------------------------------------------------------------------------------------- the same in 64 bits
def _norm64(s, x, w, b):
    if s["gpt2"]:
        x = x - x.mean(-1, keepdim=True)
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + s["eps"]) * w + b
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + s["eps"]) * w


def _turn64(s, x, pos):
    half = s["D"] // 2
    ang = pos[:, None] * s["theta"] ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / s["D"])
    c, sn = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * sn, b * c + a * sn], -1)


def _attend64(s, q, k, v):
    """q [n, heads, D], k, v [n, kv, D] of one sequence, causal; a few heads at a time."""
    n, out = q.shape[0], []
    G = s["heads"] // s["kv"]
    hidden = torch.ones((n, n), dtype=torch.bool, device=q.device).triu(1)
    step = max(1, 2 ** 27 // (n * n))
    for h in range(0, s["heads"], step):
        hs = list(range(h, min(h + step, s["heads"])))
        kh = [i // G for i in hs]
        a = (q[:, hs].transpose(0, 1) @ k[:, kh].permute(1, 2, 0)) / math.sqrt(s["D"])
        out.append(torch.softmax(a.masked_fill(hidden, float("-inf")), -1) @ v[:, kh].transpose(0, 1))
    return torch.cat(out).transpose(0, 1).reshape(n, -1)


def _decoder64(s, get, ids, lens):
    """Final-normed hidden states of the sequences of ``lens`` tokens that stand one after the other in ids; get(name): a float64 weight."""
    pos = torch.cat([torch.arange(n, device=ids.device) for n in lens])
    h = get("emb", ids)
    if s["gpt2"]:
        h = h + get("pos", pos)
    nq, nkv, F = s["heads"] * s["D"], s["kv"] * s["D"], s["ff"]
    opt = lambda n: get(n) if s["gpt2"] else None
    for i in range(s["L"]):
        a = _norm64(s, h, get(f"{i}.n1"), opt(f"{i}.n1_b"))
        qkv = torch.nn.functional.linear(a, get(f"{i}.qkv"), opt(f"{i}.qkv_b"))
        q, k, v = (x.reshape(x.shape[0], -1, s["D"]) for x in qkv.split([nq, nkv, nkv], -1))
        if not s["gpt2"]:
            q, k = _turn64(s, q, pos.double()), _turn64(s, k, pos.double())
        o = torch.cat([_attend64(s, *t) for t in zip(q.split(lens), k.split(lens), v.split(lens))])
        h = h + torch.nn.functional.linear(o, get(f"{i}.o"), opt(f"{i}.o_b"))
        f = _norm64(s, h, get(f"{i}.n2"), opt(f"{i}.n2_b"))
        u = torch.nn.functional.linear(f, get(f"{i}.up"), opt(f"{i}.up_b"))
        u = torch.nn.functional.gelu(u, approximate="tanh") if s["gpt2"] else torch.nn.functional.silu(u[:, :F]) * u[:, F:]
        h = h + torch.nn.functional.linear(u, get(f"{i}.down"), opt(f"{i}.down_b"))
    return _norm64(s, h, get("norm"), opt("norm_b"))


def _exact_step(case, s, W, ids):
    """Gradients over a few sequences at a time, then one AdamW step; outputs in the layout of the flat buffers."""
    P = {n: w.double().requires_grad_(True) for n, w in W.items()}
    B, S = case["batch"], case["seq"]
    get = lambda n, rows=None: P[n] if rows is None else torch.nn.functional.embedding(rows, P[n])
    head = P["emb"] if "head" not in P else P["head"]
    loss, k = 0.0, max(1, 4096 // S)
    for b in range(0, B, k):
        part = ids[b:b + k]
        f = _decoder64(s, get, part[:, :-1].reshape(-1), [S] * part.shape[0])
        one = torch.nn.functional.cross_entropy(f @ head.t(), part[:, 1:].reshape(-1), reduction="sum") / (B * S)
        one.backward()
        loss += float(one)
        del f, one
    norm = math.sqrt(sum(float(p.grad.square().sum()) for p in P.values()))
    clip = CLIP / (norm + 1e-6) if norm > CLIP else 1.0
    total = -(-sum(-(-p.numel() // 128) * 128 for p in P.values()) // 1024) * 1024
    out = {n: torch.zeros(total, dtype=torch.float64, device=ids.device) for n in ("master", "m", "v")}
    at = 0
    for name, _ in _flat(s):
        p = P[name]
        w, g = p.detach().reshape(-1), p.grad.reshape(-1) * clip
        m, v = (1 - BETA1) * g, (1 - BETA2) * g * g
        z = slice(at, at + w.numel())
        out["m"][z], out["v"][z] = m, v
        out["master"][z] = w - LR * ((m / (1 - BETA1)) / ((v / (1 - BETA2)).sqrt() + ADAM_EPS) + DECAY * w)
        at += -(-w.numel() // 128) * 128
        p.grad = None
    return {"loss": torch.tensor(loss, dtype=torch.float64, device=ids.device), **out}


def exact(case, seed):
    dev, s = torch.device("cuda", 0), _shape(case)
    W = _weights(s, seed, dev)
    if case["kind"] == "train":
        return _exact_step(case, s, W, _ids(s, (case["batch"], case["seq"] + 1), seed, dev))
    get = lambda n, rows=None: W[n].double() if rows is None else W[n][rows].double()
    head = (W["emb"] if "head" not in W else W["head"]).double().t()
    with torch.no_grad():
        if case["kind"] == "score":
            B, S = case["batch"], case["seq"]
            ids = _ids(s, (B, S + 1), seed, dev)[:, :-1].reshape(-1)
            return {"logits": (_decoder64(s, get, ids, [S] * B) @ head).reshape(B, S, -1)}
        lens, steps = _lengths(case), case["steps"]
        n, ids = len(lens), _ids(s, (sum(lens) + steps * len(lens),), seed, dev)
        answers = ids[sum(lens):].view(steps, n)
        whole, at, firsts, lasts = [], 0, [], []
        for i, m in enumerate(lens):
            firsts.append(sum(lens[:i + 1]) + steps * i - 1)
            whole += [ids[at:at + m], answers[:, i]]
            at += m
            lasts.append(firsts[-1] + steps)
        f = _decoder64(s, get, torch.cat(whole), [m + steps for m in lens])
        return {"first": f[firsts] @ head, "last": f[lasts] @ head}
