"""The work that users of the framework wait for, as cases that can be timed and compared.

Training: one micro-batch, forward and backward, of a Llama-style decoder whose gradients go into the optimizer's fp32
buffer.  Serving: prompts that start, prompts that go on from a cached context, and the decode step that generation
replays, for the three families that serve through one cache / state manager (Llama, Pafodra, Megozen).  Widths, heads,
feed-forward and expert sizes are those of the serving benchmark and of the 7B preset; a few layers stand for the model,
so that embedding and head keep about the share that they have in use.

A case is ``{"work": train | prompt | continue | decode, "model", "width", "kv", ...}``; sequence lengths are spread
unevenly around their mean by ``lengths``.
"""
import math
import random

import torch
import torch.nn.functional as F

HEAD = 128                                        # head size of every attention layer
FF = {1024: 2816, 2048: 5632, 4096: 11008}        # feed-forward width of a dense layer
EXPERT_FF = {1024: 704, 2048: 1408, 4096: 2752}   # of one expert; 16 experts, 2 per token, a shared one
EXPERTS, TOP = 16, 2
VOCAB = {1024: 8192, 2048: 32000, 4096: 32000}
LATENT = {"dim": 128, "rot": 64, "vdim": 128, "rank": 512, "window": 1024}
REPLY = 256                                       # tokens of a reply before the decode cases start the next one
BF = torch.bfloat16


def listed():
    return [
        # the first steps of a fine-tuning run on a small model and one short document: launches and host time
        {"name": "train_small", "work": "train", "model": "llama", "width": 1024, "kv": 8, "alibi": False, "tokens": 200,
         "sequences": 1},
        # instruction tuning: documents of unequal length packed in one row, grouped key heads, nothing a multiple of a tile
        {"name": "train_docs", "work": "train", "model": "llama", "width": 2048, "kv": 4, "alibi": False, "tokens": 3001,
         "sequences": 7},
        # pre-training at the 7B sizes: one document of 4096 tokens
        {"name": "train_7b", "work": "train", "model": "llama", "width": 4096, "kv": 32, "alibi": False, "tokens": 4096,
         "sequences": 1},
        # a short question: the time to the first token
        {"name": "prompt_short", "work": "prompt", "model": "llama", "width": 2048, "kv": 8, "tokens": 77, "sequences": 1},
        # a batch of prompts at 4k width
        {"name": "prompt_batch", "work": "prompt", "model": "llama", "width": 4096, "kv": 8, "tokens": 4096, "sequences": 8},
        # one long prompt through the recurrent layers
        {"name": "prompt_pafodra", "work": "prompt", "model": "pafodra", "width": 2048, "kv": 8, "experts": False,
         "tokens": 4096, "sequences": 1},
        # a ragged batch of prompts with latent attention, a window and experts
        {"name": "prompt_megozen", "work": "prompt", "model": "megozen", "width": 2048, "tokens": 3777, "sequences": 5},
        # the second turn of two conversations
        {"name": "continue_llama", "work": "continue", "model": "llama", "width": 2048, "kv": 8, "tokens": 301,
         "sequences": 2, "context": 3000},
        # one user's reply, token by token
        {"name": "decode_single", "work": "decode", "model": "llama", "width": 4096, "kv": 8, "sequences": 1,
         "context": 1000},
        # a full serving batch
        {"name": "decode_batch", "work": "decode", "model": "llama", "width": 4096, "kv": 8, "sequences": 64,
         "context": 2048},
        # a small batch of long conversations on recurrent states, caches and experts
        {"name": "decode_pafodra", "work": "decode", "model": "pafodra", "width": 2048, "kv": 8, "experts": True,
         "sequences": 8, "context": 4096},
        # a full batch on latent rows
        {"name": "decode_megozen", "work": "decode", "model": "megozen", "width": 2048, "sequences": 64, "context": 4096},
    ]


def draw(rng):
    def spread(lo, hi):
        return round(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    work = rng.choice(("train", "train", "prompt", "prompt", "continue", "decode", "decode"))
    model = "llama" if work == "train" else rng.choice(("llama", "llama", "pafodra", "megozen"))
    width = rng.choice((1024, 2048, 4096) if model == "llama" else (2048, 4096))
    c = {"work": work, "model": model, "width": width}
    if model != "megozen":
        c["kv"] = width // HEAD // rng.choice((1, 2, 4) if width < 4096 or work != "train" else (1, 4))
    if model == "pafodra":
        c["experts"] = rng.random() < 0.5
    if work == "train":
        c.update(alibi=rng.random() < 0.25, tokens=spread(128, 4096), sequences=spread(1, 8))
    elif work == "prompt":
        c.update(tokens=spread(32, 4096), sequences=spread(1, 8))
    elif work == "continue":
        c.update(tokens=spread(16, 512), sequences=spread(1, 4), context=spread(64, 4096))
    else:
        c.update(sequences=spread(1, 64), context=spread(64, 4096))
    return c


def lengths(case):
    """Tokens per sequence: uneven around the mean, at least one each."""
    n, total = case["sequences"], case["tokens"]
    rng = random.Random(total * 64 + n)
    w = [rng.uniform(0.4, 1.6) for _ in range(n)]
    out = [max(1, int(total * x / sum(w))) for x in w]
    out[0] += total - sum(out)
    return out


def layer_count(case):
    return {"llama": 2 if case["work"] == "train" else 4, "pafodra": 5, "megozen": 4}[case["model"]]


def config(case):
    """``config.json`` of the model."""
    W = case["width"]
    H, n = W // HEAD, layer_count(case)
    if case["model"] == "llama":
        return {"model_type": "baichuan2-13b" if case.get("alibi") else "llama", "vocab_size": VOCAB[W], "hidden_size": W,
                "intermediate_size": FF[W], "num_hidden_layers": n, "num_attention_heads": H,
                "num_key_value_heads": case["kv"], "rms_norm_eps": 1e-6, "max_position_embeddings": 4096}
    moe = {"kind": "moe", "router": {"experts": EXPERTS, "top": TOP}, "expert": {"ff": EXPERT_FF[W]},
           "shared": {"ff": EXPERT_FF[W]}}
    if case["model"] == "megozen":
        m = LATENT
        rot = {"dims": m["rot"], "base": 10000.0, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}
        layer = {"type": "latent_attention", "mlp": moe,
                 "mixer": {"heads": H, "dim": m["dim"], "rot_dim": m["rot"], "vdim": m["vdim"], "kv_rank": m["rank"],
                           "scale": (m["dim"] + m["rot"]) ** -0.5, "rot": rot, "mask": {"size": m["window"]}}}
        return {"architecture": "Megozen", "vocab": VOCAB[W], "width": W, "norm": {"eps": 1e-6},
                "embedding": {"bigram": {"buckets": VOCAB[W] - 1, "mul_prev": 7919, "mul_cur": 104729}}, "layers": [layer] * n}
    dense = {"kind": "dense", "ff": FF[W]}
    moe = moe if case["experts"] else dense
    att = {"type": "attention", "mlp": dense, "mixer": {"heads": H, "kv_heads": case["kv"], "dim": HEAD, "vdim": HEAD,
                                                       "scale": HEAD ** -0.5}}
    wkv = {"type": "wkv", "mixer": {"heads": W // 64, "dim": 64}}
    delta = {"type": "channel_delta", "mlp": moe,
             "mixer": {"heads": H, "kv_heads": H, "dim": HEAD, "vdim": HEAD, "conv": 4}}
    return {"architecture": "Pafodra", "vocab": VOCAB[W], "width": W, "norm": {"eps": 1e-5}, "embedding": {"scale": 4.0},
            "layers": [dict(wkv, mlp=moe), att, delta, att, dict(wkv, mlp=dense)][:n]}


def build(case, seed):
    """The model with random weights: 0.02 as at the start of training; in the families with a fixed residual stream the
    embedding and the decays are spread as in a trained model, where the stream is several times what a layer adds to it."""
    from easyllm_b200.models.hf_models import CausalLM, arch_from_hf_config
    torch.manual_seed(seed)
    with torch.device("cuda"):
        model = CausalLM(arch_from_hf_config(config(case)), dtype=BF)
    with torch.no_grad():
        for name, p in model.named_parameters():
            if name.endswith((".w0", ".A_log")):
                p.uniform_(-6.0, -1.0)
            elif name.endswith(".sink"):
                p.normal_()
            elif "embed" in name and case["model"] != "llama":
                p.mul_(30 if case["model"] == "pafodra" else 100)
    return model


def ids_of(case, count, gen):
    return torch.randint(0, VOCAB[case["width"]], (count,), generator=gen)


def prepare(case, seed):
    gen = torch.Generator().manual_seed(seed)
    model = build(case, seed)
    if case["work"] == "train":
        return prepare_train(case, model, gen)
    model.eval()
    n, dev = case["sequences"], "cuda"
    s = {"work": case["work"], "model": model, "context": case.get("context", 0)}
    room = s["context"] + (REPLY + 1 if case["work"] == "decode" else max(lengths(case)))
    s["state"] = state = model.new_state(n, room)
    if case["work"] == "prompt":
        s["prompts"] = [ids_of(case, m, gen).to(dev) for m in lengths(case)]
        return s
    s["slots"] = [state.open() for _ in range(n)]
    if case["work"] == "decode":
        s["ids"] = ids_of(case, n, gen).to(dev)
        model.logits(model.step(state, s["slots"], s["ids"])[0])     # the step runs once before it is captured
    else:
        s["prompts"] = [ids_of(case, m, gen).to(dev) for m in lengths(case)]
    rewind(s)
    fill(state, s["context"])
    if case["work"] == "decode":
        from easyllm_b200.models.hf_models.state import DecodeGraph
        s["graph"] = g = DecodeGraph(model, state, s["slots"])
        s["start"] = {k: g.meta[k].clone() for k in ("seq_pos0", "position_ids", "kv_len")}
    return s


def prepare_train(case, model, gen):
    """What the HF runner holds: the model, its optimizer (whose fp32 buffer takes the gradients) and a packed row of
    documents as the loader delivers it, on the host."""
    from easyllm_b200.optim.zero import ZeroOptimizer
    opt = ZeroOptimizer(model.named_parameters(), lr=1e-4, stage=0)
    n = lengths(case)
    cu = [0]
    for m in n:
        cu.append(cu[-1] + m)
    return {"work": "train", "model": model.train(), "opt": opt,
            "batch": {"input_ids": ids_of(case, cu[-1], gen).unsqueeze(0), "labels": ids_of(case, cu[-1], gen).unsqueeze(0),
                      "position_ids": torch.cat([torch.arange(m) for m in n]).unsqueeze(0),
                      "cu_seqlens": torch.tensor(cu, dtype=torch.int32)}}


def fill(state, context):
    """What ``context`` tokens would have left behind: unit keys and values, recurrent states and last inputs."""
    for c in state.layers + ([state.tokens] if state.tokens is not None else []):
        for name in c.names:
            t = getattr(c, name)
            if not t.is_floating_point():
                t.random_(0, 1000)
            elif name == "s":                     # rows past the keys' own stay zero
                t.normal_(0, 0.1)
            else:
                t.normal_()


def rewind(s):
    for slot in s["slots"]:
        s["state"].lengths[slot] = s["context"]
    for name, t in s.get("start", {}).items():
        s["graph"].meta[name].copy_(t)


def kept(state):
    """The caches and states themselves."""
    return [getattr(c, name) for c in state.layers for name in c.names]


def run(s):
    model, state = s["model"], s.get("state")
    if s["work"] == "train":
        s["opt"].zero_grad()
        loss = model(**s["batch"])["loss"]
        loss.backward()
        s["opt"].accumulate_grads()
        return [loss.detach()] + [p.main_grad for p in s["opt"].params]
    if s["work"] == "decode":
        if state.lengths[s["slots"][0]] >= s["context"] + REPLY:
            rewind(s)                             # the next reply
        return [s["graph"].step(s["ids"])] + kept(state)
    if s["work"] == "continue":
        rewind(s)
        h, meta = model.step(state, s["slots"], s["prompts"])
        return [model.logits(h[meta["last_rows"].to(h.device, non_blocking=True)])] + kept(state)
    slots = [state.open() for _ in s["prompts"]]
    h, meta = model.step(state, slots, s["prompts"])
    logits = model.logits(h[meta["last_rows"].to(h.device, non_blocking=True)])
    for slot in reversed(slots):
        state.close(slot)
    return [logits] + kept(state)


def work(case):
    """Weights once, every cached row that is read or written once, tokens in and logits out; products of weights and
    attention over the pairs of query and key.  The backward pass takes twice the products, and writes fp32 gradients."""
    W, V, n = case["width"], VOCAB[case["width"]], case["sequences"]
    T = n if case["work"] == "decode" else case["tokens"]
    ctx = case.get("context", 0)
    each = [1] * n if case["work"] == "decode" else lengths(case)
    rows_out = T if case["work"] == "train" else n
    cfg = config(case)
    H = W // HEAD
    hit = min(EXPERTS, TOP * T)
    weights, flops, moved, pairs = V * W, 2.0 * rows_out * V * W, 0.0, float(sum(m * ctx + m * (m + 1) / 2 for m in each))

    def dense(params, tokens=None):
        nonlocal weights, flops
        weights += params
        flops += 2.0 * params * (T if tokens is None else tokens)

    def experts(matrices):
        nonlocal weights, flops
        one = matrices * W * EXPERT_FF[W]
        weights += one * (hit + 1)
        flops += 2.0 * one * T * (TOP + 1)

    def attention(kv):
        nonlocal flops, moved
        flops += 4.0 * pairs * H * HEAD
        moved += 4.0 * (sum(each) + (ctx * n)) * kv * HEAD

    if case["model"] == "llama":
        for _ in range(layer_count(case)):
            dense(2 * W * W + 2 * W * case["kv"] * HEAD + 3 * W * FF[W])
            attention(case["kv"])
    elif case["model"] == "megozen":
        m, win = LATENT, LATENT["window"]
        seen = float(sum(min(ctx + i + 1, win) for x in each for i in range(x)))
        keys = float(sum(min(ctx, win) + x for x in each))
        for _ in range(layer_count(case)):
            dense(W * (H * (m["dim"] + m["rot"]) + m["rank"] + m["rot"] + H) + m["rank"] * H * 2 * 128 + W * W)
            experts(3)
            flops += seen * H * 2 * ((m["dim"] + m["rot"] + m["vdim"]) if not ctx else (2 * m["rank"] + m["rot"]))
            moved += 2.0 * keys * (m["rank"] + m["rot"])
    else:
        for layer in cfg["layers"]:
            if layer["type"] == "attention":
                dense(2 * W * W + 2 * W * case["kv"] * HEAD)
                attention(case["kv"])
            else:
                wkv = layer["type"] == "wkv"
                d = 64 if wkv else HEAD
                dense((5 if wkv else 4) * W * W)
                flops += T * W * d * (5.0 if wkv else 7.0)
                moved += n * W * d * (8 if ctx else 4)
            experts(2) if layer["mlp"]["kind"] == "moe" else dense(3 * W * FF[W])
    if case["work"] == "train":
        return {"bytes": 2.0 * weights + 4.0 * (weights + V * W) + 16.0 * T, "flops": 3 * flops - 2 * pairs * H * HEAD}
    return {"bytes": 2.0 * (weights + T * W) + moved + 4.0 * rows_out * V, "flops": flops}


def tolerance(case):
    """Every layer rounds its activations to bf16 (relative 2^-9) a dozen times: logits and gradients are 1 to 3 % off a 64-bit
    evaluation, and two orders of the atomic sums in the backward pass 0.2 % off each other.  A token between two experts may
    go to either, which moves single values by a good part of their size."""
    return {"rel": 0.03, "max": 0.9}


# ---- the same numbers in 64 bits, plain torch ------------------------------------------------------
def rms(x, w, eps):
    return x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def rotate_halves(x, pos):
    """x [T, heads, d] at positions ``pos``; the angles are those of the fp32 tables."""
    d = x.shape[-1]
    inv = 1.0 / (10000.0 ** (torch.arange(0, d, 2, dtype=torch.float32, device=x.device) / d))
    a = torch.outer(pos.float(), inv).unsqueeze(1)
    c, s = a.cos().double(), a.sin().double()
    u, v = x[..., :d // 2], x[..., d // 2:]
    return torch.cat((u * c - v * s, v * c + u * s), -1)


def slopes(heads):
    def geometric(n):
        return [2.0 ** (-8.0 * (i + 1) / n) for i in range(n)]
    p = 1 << (heads.bit_length() - 1)
    out = geometric(p) + geometric(2 * p)[0::2][:heads - p]
    return torch.tensor(out, dtype=torch.float32, device="cuda").double()


def attend(q, k, v, scale, alibi=None, sink=None):
    """q [n, H, d] at the last rows of k, v [m, G, d]; causal."""
    n, H, _ = q.shape
    m, G = k.shape[0], k.shape[1]
    place = torch.arange(m, device=q.device) - torch.arange(m - n, m, device=q.device).unsqueeze(1)
    out = []
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].t() * scale
        if alibi is not None:
            s = s + alibi[h] * place
        s = s.masked_fill(place > 0, -math.inf)
        if sink is not None:
            s = torch.cat((s, sink[h].expand(n, 1)), 1)
        out.append(torch.softmax(s, -1)[:, :m] @ v[:, h * G // H])
    return torch.stack(out, 1)


def llama64(case, w, ids, each, past=None):
    """Final hidden rows [T, W] in 64 bits; ``past``: keys and values per layer, [sequences, context, heads, d] each."""
    W, kv, alibi = case["width"], case["kv"], case.get("alibi")
    H, ctx = W // HEAD, case.get("context", 0)
    pos = torch.cat([torch.arange(m) + ctx for m in each]).cuda()
    x = F.embedding(ids, w["model.embed_tokens.weight"])
    for i in range(layer_count(case)):
        p = "model.layers.%d." % i
        h = rms(x, w[p + "input_layernorm.weight"], 1e-6)
        q, k, v = ((h @ w[p + "self_attn.%s_proj.weight" % n].t()).view(len(pos), -1, HEAD) for n in "qkv")
        if not alibi:
            q, k = rotate_halves(q, pos), rotate_halves(k, pos)
        out, at = [], 0
        for j, m in enumerate(each):
            kj, vj = k[at:at + m], v[at:at + m]
            if past is not None:
                kj, vj = (torch.cat((c[j, :ctx].double(), y)) for c, y in ((past[i][0], kj), (past[i][1], vj)))
            out.append(attend(q[at:at + m], kj, vj, HEAD ** -0.5, slopes(H) if alibi else None))
            at += m
        x = x + torch.cat(out).reshape(len(pos), W) @ w[p + "self_attn.o_proj.weight"].t()
        h = rms(x, w[p + "post_attention_layernorm.weight"], 1e-6)
        g, u = (h @ w[p + "mlp.%s_proj.weight" % n].t() for n in ("gate", "up"))
        x = x + (F.silu(g) * u) @ w[p + "mlp.down_proj.weight"].t()
    return rms(x, w["model.norm.weight"], 1e-6)


def head_norm(o, w, gate, act):
    o = o / torch.sqrt(o.pow(2).mean(-1, keepdim=True) + 1e-5)
    T, H, d = o.shape
    o = o * (w.view(H, d) if w.numel() == H * d else w)
    return (o * act(gate).view(T, H, d)).reshape(T, H * d)


def wkv64(h, w, heads, each, past):
    prev = torch.cat([torch.cat((h.new_zeros(1, h.shape[1]) if past is None else past["last"][j:j + 1], x[:-1]))
                      for j, x in enumerate(h.split(each))])
    mix = [h + (prev - h) * m for m in w["mu"]]
    r, k, v, g = (mix[i] @ w[n + "_proj.weight"].t() for i, n in enumerate("rkvg"))
    decay = torch.exp(-torch.exp(torch.tanh(mix[4] @ w["w1_proj.weight"].t()) @ w["w2_proj.weight"].t() + w["w0"]))
    r, k, v, decay = (t.view(h.shape[0], heads, -1) for t in (r, k, v, decay))
    o, t = [], 0
    for j, m in enumerate(each):
        S = torch.zeros(heads, 64, 64, dtype=h.dtype, device=h.device) if past is None else past["s"][j, ..., :64]
        for t in range(t, t + m):
            kv = v[t].unsqueeze(-1) * k[t].unsqueeze(-2)
            o.append(((S + kv * w["u"].unsqueeze(-2)) * r[t].unsqueeze(-2)).sum(-1))
            S = S * decay[t].unsqueeze(-2) + kv
        t += 1
    return head_norm(torch.stack(o), w["norm"], g, F.silu) @ w["o_proj.weight"].t()


def delta64(h, w, H, each, past):
    T, n = h.shape[0], w["q_conv"].shape[1]
    x = torch.cat([h @ w[c + "_proj.weight"].t() for c in "qkv"], 1)
    taps = torch.cat([w[c + "_conv"] for c in "qkv"])
    y = []
    for j, part in enumerate(x.split(each)):
        before = x.new_zeros(n - 1, x.shape[1]) if past is None else past["tail"][j].t()
        full = torch.cat((before, part))
        y.append(F.silu(sum(full[i:i + part.shape[0]] * taps[:, i] for i in range(n))))
    q, k, v = (t.view(T, H, HEAD) for t in torch.cat(y).chunk(3, -1))
    q, k = (t / torch.sqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q = q * HEAD ** -0.5
    a = (h @ w["a1_proj.weight"].t()) @ w["a2_proj.weight"].t() + w["dt_bias"]
    g = torch.exp(-torch.exp(w["A_log"]).view(H, 1) * F.softplus(a).view(T, H, HEAD))
    beta = torch.sigmoid(h @ w["b_proj.weight"].t())
    o, t = [], 0
    for j, m in enumerate(each):
        S = torch.zeros(H, HEAD, HEAD, dtype=h.dtype, device=h.device) if past is None else past["s"][j, ..., :HEAD]
        for t in range(t, t + m):
            S = S * g[t].unsqueeze(-2)
            e = beta[t].unsqueeze(-1) * (v[t] - (S * k[t].unsqueeze(-2)).sum(-1))
            S = S + e.unsqueeze(-1) * k[t].unsqueeze(-2)
            o.append((S * q[t].unsqueeze(-2)).sum(-1))
        t += 1
    gate = (h @ w["g1_proj.weight"].t()) @ w["g2_proj.weight"].t()
    return head_norm(torch.stack(o), w["norm"], gate, torch.sigmoid) @ w["o_proj.weight"].t()


def pafodra64(case, w, ids, each, past=None):
    W, ctx = case["width"], case.get("context", 0)
    H = W // HEAD
    x = F.embedding(ids, w["model.embed_tokens.weight"]) * 4.0

    def dyt(x, p):
        return torch.tanh(w[p + "alpha"] * x) * w[p + "weight"] + w[p + "bias"]

    for i, layer in enumerate(config(case)["layers"]):
        p = "model.layers.%d." % i
        m = {k[len(p) + 6:]: t for k, t in w.items() if k.startswith(p + "mixer.")}
        h = dyt(x, p + "input_layernorm.")
        old = None if past is None else {k: t.double() for k, t in past[i].items()}
        if layer["type"] == "attention":
            q, k, v = ((h @ m[n + "_proj.weight"].t()).view(len(h), -1, HEAD) for n in "qkv")
            out, at = [], 0
            for j, n in enumerate(each):
                kj, vj = k[at:at + n], v[at:at + n]
                if old is not None:
                    kj, vj = torch.cat((old["k"][j, :ctx], kj)), torch.cat((old["v"][j, :ctx], vj))
                out.append(attend(q[at:at + n], kj, vj, HEAD ** -0.5, sink=m["sink"]))
                at += n
            y = torch.cat(out).reshape(len(h), W) @ m["o_proj.weight"].t()
        else:
            y = wkv64(h, m, W // 64, each, old) if layer["type"] == "wkv" else delta64(h, m, H, each, old)
        f = {k[len(p) + 4:]: t for k, t in w.items() if k.startswith(p + "mlp.")}
        g, u = (h @ f[n + "_proj.weight"].t() + f[n + "_proj.bias"] for n in ("gate", "up"))
        act = 0.5 * g * (1 + torch.tanh(math.sqrt(2 / math.pi) * (g + 0.044715 * g ** 3)))
        x = x + y + (act * u) @ f["down_proj.weight"].t() + f["down_proj.bias"]
    return dyt(x, "model.norm.")


def exact(case, seed):
    """None where experts are chosen: a token between two of them may go either way.  Otherwise loss and gradients, or the
    logits (the caches are inputs with a few rows written, they come without a value)."""
    if case["model"] == "megozen" or case.get("experts"):
        return None
    s = prepare(case, seed)
    w = {k: p.detach().double() for k, p in s["model"].named_parameters()}
    if case["work"] == "train":
        names = s["opt"].names
        b = s["batch"]
        del s
        for p in w.values():
            p.requires_grad_()
        ids, each = b["input_ids"].reshape(-1).cuda(), lengths(case)
        h = llama64(case, w, ids, each)
        head = w["lm_head.weight"]
        head = F.normalize(head, dim=-1) if case["alibi"] else head
        # the row is shifted as a whole: the last token alone has no target
        loss = F.cross_entropy((h @ head.t())[:-1], b["labels"].reshape(-1)[1:].cuda())
        loss.backward()
        return [loss.detach()] + [w[n].grad for n in names]
    with torch.no_grad():
        ids = s["ids"] if case["work"] == "decode" else torch.cat(s["prompts"])
        each = [1] * case["sequences"] if case["work"] == "decode" else lengths(case)
        past = None
        if case["work"] != "prompt":
            at = torch.tensor(s["slots"], device="cuda")
            past = [{n: getattr(c, n)[at] for n in c.names} for c in s["state"].layers]
        if case["model"] == "llama":
            h = llama64(case, w, ids, each, past and [(c["k"], c["v"]) for c in past])
        else:
            h = pafodra64(case, w, ids, each, past)
        last = torch.tensor(each).cumsum(0).cuda() - 1
        return [h[last] @ w["lm_head.weight"].t()] + [None] * len(kept(s["state"]))
