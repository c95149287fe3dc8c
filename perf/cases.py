"""The work that is timed when this framework's speed is looked at: requests to models of the families it serves, through the
public binding (nano_b200.engine.Engine) as a program calls it.

Every case is one or more whole requests to a resident model: a prompt goes in at once, then tokens one by one, and the logits of the
prompt's last position and of every later token come back to the host (what a program that samples or scores needs).  A model
file (the "nano" and "qwen3" architectures, 32-bit or Q80 weights) takes its prompt through decode_greedy and each token through
forward; a model folder (the layered designs) takes both through step on a sequence that is opened and closed with the request.
Q4K files are left out: their 4-bit activations are re-rounded in every layer, and the logits of two engine modes that are both right
differ by 5 to 20 % from two layers on, so no tolerance could hold them.  The tokens after the prompt are given, not chosen from the logits, so that two correct engines do the same work.

Shapes are those of bench.py (nano-168m, qwen3-0.6b and 4b layers; width 1024 and 2048 of the layered designs) with as many layers as
the case says; prompts of 5 to 2000 tokens, most of them no round number.  Weights are random: a file's or folder's contents depend on
the case alone and are written once; a request's tokens come from the seed."""
import dataclasses
import hashlib
import json
import math
import os
import struct
import tempfile
from collections import OrderedDict

import numpy as np
import torch

from nano_b200 import engine as E
from nano_b200 import modeldir as md
from nano_b200 import modelfile as mf

FILE_DESIGNS = ("nano", "qwen3")
QUANT = {"f32": mf.QUANT_F32, "q80": mf.QUANT_Q80}
GROUP = 128          # Q80 group size of bench.py's files
HEADS, KV_HEADS = 16, 4          # of the layered designs' attention


def listed():
    return [
        # chat on the flagship file: a short question, a short answer, every layer and the real vocabulary
        dict(name="nano-168m q80 chat", design="nano", width=768, layers=24, vocab=16384, type="q80", prompt=16, tokens=24, requests=1),
        # a document of nearly the whole context of that model, then a few tokens (four of its layers)
        dict(name="nano q80 document", design="nano", width=768, layers=4, vocab=16384, type="q80", prompt=487, tokens=8, requests=1),
        # the 32-bit file that results are checked against
        dict(name="nano f32 chat", design="nano", width=768, layers=4, vocab=16384, type="f32", prompt=12, tokens=64, requests=1),
        # the whole Qwen3-0.6B: a page of text and an answer's beginning
        dict(name="qwen3-0.6b q80 page", design="qwen3", width=1024, layers=28, vocab=151936, type="q80", prompt=250, tokens=16, requests=1),
        # the same layers in 32 bits
        dict(name="qwen3-0.6b f32 page", design="qwen3", width=1024, layers=2, vocab=16384, type="f32", prompt=333, tokens=32, requests=1),
        # decoding at the far end of a long context in layers of Qwen3-4B's width
        dict(name="qwen3-4b q80 long context", design="qwen3", width=2560, layers=2, vocab=4096, type="q80", prompt=1500, tokens=48, requests=1),
        # layered designs.  Chat on eight layers: a few tokens in, an answer out
        dict(name="famudra w1024 chat", design="famudra", width=1024, layers=8, vocab=32000, type="bf16", prompt=11, tokens=48, requests=1),
        # a long prompt through the recurrent block and the latent attention (routed and shared experts in both layers)
        dict(name="famudra w2048 long prompt", design="famudra", width=2048, layers=2, vocab=4096, type="bf16", prompt=2000, tokens=4, requests=1),
        # the true-32-bit mode
        dict(name="famudra w1024 float32", design="famudra", width=1024, layers=2, vocab=4096, type="f32", prompt=203, tokens=8, requests=1),
        # a prompt through grouped-query attention and both forms of the gated delta rule, dense gated feed-forwards
        dict(name="kadesun w2048 prompt", design="kadesun", width=2048, layers=2, vocab=4096, type="bf16", prompt=1024, tokens=4, requests=1),
        # a ragged long prompt through attention in blocks of positions and the matrix memory, dense and grouped-expert feed-forwards
        dict(name="fidatar w2048 long prompt", design="fidatar", width=2048, layers=2, vocab=32000, type="bf16", prompt=1777, tokens=4, requests=1),
        # the smallest: three one-line requests with a few tokens each
        dict(name="fidatar w1024 short requests", design="fidatar", width=1024, layers=2, vocab=4096, type="bf16", prompt=5, tokens=6, requests=3),
    ]


def draw(rng):
    def spread(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))
    design = rng.choice(["nano", "qwen3", "famudra", "famudra", "kadesun", "kadesun", "fidatar", "fidatar"])
    c = dict(design=design, layers=rng.randint(1, 4), vocab=rng.choice([2048, 4096, 16384, 32000]), prompt=spread(2, 2000), tokens=spread(1, 48), requests=1)
    if design in FILE_DESIGNS:
        c["type"] = rng.choice(["q80", "q80", "f32"])
        c["width"] = 768 if design == "nano" else rng.choice([1024, 2048])
    else:
        c["type"] = rng.choice(["bf16", "bf16", "bf16", "f32"])
        c["width"] = 64 * rng.randint(8, 32)
        c["layers"] = min(c["layers"], 2)
        if c["type"] == "f32":
            c["prompt"] = min(c["prompt"], 700)
    if c["prompt"] < 40:
        c["requests"] = rng.randint(1, 3)
    return c


# ---- models ----
def file_spec(c):
    base = mf.PRESETS["nano-168m"] if c["design"] == "nano" else mf.PRESETS[{1024: "qwen3-0.6b", 2048: "qwen3-1.7b", 2560: "qwen3-4b"}[c["width"]]]
    block = base.block_size if c["design"] == "qwen3" or c["prompt"] + c["tokens"] < base.block_size else 4096
    return dataclasses.replace(base, name="perf", n_layer=c["layers"], vocab=c["vocab"], block_size=block), base.n_layer


def folder_config(c):
    w, n = c["width"], c["layers"]
    dim = w // HEADS
    if c["design"] == "famudra":
        mlp = {"experts": 16, "top": 2, "ff": w // 2, "shared_ff": w}
        rec = ("rglru", {"width": w, "blocks": 8 if w < 2048 else 16, "conv": 4}, mlp)
        att = ("latent_attention", {"heads": HEADS, "dim": dim, "vdim": dim, "kv_rank": w // 4, "q_rank": 512 if w < 2048 else 768, "scale": dim ** -0.5}, mlp)
        return md.famudra_config(c["vocab"], w, [(att, rec)[(i + n) % 2] for i in range(n)])          # the last layer is recurrent, an odd number begins with one
    if c["design"] == "kadesun":
        heads = w // 128
        par = {"left": {"heads": HEADS, "kv_heads": KV_HEADS, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "softcap": 50.0, "rot": {"dims": dim, "base": 500000.0}},
               "right": {"heads": heads, "kv_heads": heads, "dim": 128, "vdim": 128, "conv": 4}}
        dl = {"heads": heads, "kv_heads": heads // 2 if heads % 2 == 0 else heads, "dim": 128, "vdim": 128, "conv": 4}
        return md.kadesun_config(c["vocab"], w, [("parallel", par, 3 * w) if i % 2 == 0 else ("delta", dl, 3 * w) for i in range(n)])
    att = {"heads": HEADS, "kv_heads": KV_HEADS, "dim": dim, "vdim": dim, "scale": dim ** -0.5, "mask": {"size": 4096},
           "rot": {"dims": dim // 4 * 2, "base": 10000.0, "scaling": {"factor": 4.0, "original": 2048, "fast": 32.0, "slow": 1.0}}}
    mem = {"heads": w // 128, "dim": 128, "vdim": 128, "gate_cap": 15.0}
    moe = {"kind": "moe", "router": {"experts": 16, "top": 2, "groups": {"count": 4, "keep": 2}, "scale": 1.5}, "expert": {"ff": w}}
    return md.fidatar_config(c["vocab"], w, [("attention", att, {"kind": "dense", "ff": 4 * w}) if i % 2 == 0 else ("mlstm", mem, moe) for i in range(n)],
                             alpha=2.5, scale=w ** 0.5, softcap=30.0)


def model_key(c):
    return hashlib.sha1(json.dumps([c[k] for k in ("design", "width", "layers", "vocab", "type")] + [c["design"] == "nano" and c["prompt"] + c["tokens"] >= 512]).encode()).hexdigest()[:16]


def file_weights(c):
    """The file's weights before they are quantised: the same every time, on the GPU (the wide tensors) and in 32 bits."""
    spec, depth = file_spec(c)
    g = torch.Generator(device="cuda").manual_seed(int(model_key(c), 16) % (1 << 31))
    L, W, F, Q, K = spec.n_layer, spec.n_embd, spec.n_hidden, spec.q_dim, spec.kv_dim
    std, std_o = 0.02, 0.02 / math.sqrt(2 * depth)
    shapes = [("attn_norm", (L, W), 0), ("ffn_norm", (L, W), 0), ("final_norm", (W,), 0), ("emb", (spec.vocab, W), std), ("wq", (L, Q, W), std), ("wk", (L, K, W), std),
              ("wv", (L, K, W), std), ("wo", (L, W, Q), std_o), ("w1", (L, F, W), std), ("w2", (L, W, F), std), ("w3", (L, F, W), std_o)]
    if spec.arch == mf.ARCH_QWEN3:
        shapes += [("q_norm", (L, spec.hd), 0), ("k_norm", (L, spec.hd), 0)]
    out = {}
    for name, shape, s in shapes:
        w = torch.randn(shape, generator=g, device="cuda")
        out[name] = w * s if s else 1.0 + 0.02 * w
    return out


def model_path(c):
    """Where the case's model file or folder is; written if it is not there."""
    root = os.path.join(tempfile.gettempdir(), "nb200_models")
    os.makedirs(root, exist_ok=True)
    path = os.path.join(root, "perf-" + model_key(c))
    if os.path.exists(path):
        return path
    part = "%s.%d" % (path, os.getpid())
    if c["design"] in FILE_DESIGNS:
        w = {k: v.cpu().numpy() for k, v in file_weights(c).items()}
        mf.write_model_from_weights(part, file_spec(c)[0], QUANT[c["type"]], GROUP, w)
    else:
        cfg = folder_config(c)
        seed = int(model_key(c), 16) % (1 << 31)
        if c["design"] == "kadesun":
            t = md.kadesun_random(cfg, seed, decay_rank=64 if c["width"] < 2048 else 128, gate_rank=64 if c["width"] < 2048 else 128)
        else:
            t = {"famudra": md.famudra_random, "fidatar": md.fidatar_random}[c["design"]](cfg, seed)
            for k in t:          # what a sublayer adds is small beside the stream, as in a deep trained model
                if k.endswith((".o", ".down")):
                    t[k] = t[k] * np.float32(0.2)
        md.write_model_dir(part, cfg, t)
    os.replace(part, path)
    return path


_engines = OrderedDict()          # the models a program keeps resident: at most two


def engine(c):
    key = json.dumps({k: v for k, v in c.items() if k != "name"}, sort_keys=True)
    if key not in _engines:
        while len(_engines) >= 2:
            _engines.popitem(last=False)
        room = 512
        while room < c["prompt"] + c["tokens"] + 1:
            room *= 2
        _engines[key] = E.Engine(model_path(c), room, flags=E.FLAG_F32 if c["design"] not in FILE_DESIGNS and c["type"] == "f32" else 0)
    _engines.move_to_end(key)
    return _engines[key]


def tokens_of(c, seed):
    rng = np.random.default_rng([seed, c["prompt"], c["tokens"]])
    return rng.integers(0, c["vocab"], size=(c["requests"], c["prompt"] + c["tokens"])).astype(np.uint32)


# ---- the passes ----
def prepare(case, seed):
    return {"case": case, "engine": engine(case), "ids": tokens_of(case, seed)}


def run(state):
    c, eng = state["case"], state["engine"]
    n = c["prompt"]
    out = []
    for ids in state["ids"]:
        if c["design"] in FILE_DESIGNS:
            buf = np.zeros(n + 2, np.uint32)
            buf[:n] = ids[:n]
            eng.decode_greedy(buf, n, n + 1)
            rows = [eng.logits()]
            for pos in range(n, ids.size):
                rows.append(eng.forward(int(ids[pos]), pos))
        else:
            seq = eng.seq_open()
            rows = [eng.step(seq, ids[:n], [n - 1])[0]]
            for pos in range(n, ids.size):
                rows.append(eng.step(seq, ids[pos:pos + 1], [0])[0])
            eng.seq_close(seq)
        out.append(np.stack(rows))
    return out


# ---- what a pass cannot do without ----
def layer_sizes(c):
    """(weights a layer's token reads, weights of all its matrices, floats its cache holds for a token, floats of its state, multiply-adds of its attention for a token and key) of every layer"""
    if c["design"] in FILE_DESIGNS:
        s, _ = file_spec(c)
        n = s.q_dim * s.n_embd * 2 + 2 * s.kv_dim * s.n_embd + 3 * s.n_hidden * s.n_embd
        return [(n, n, 2 * s.kv_dim, 0, 2 * s.q_dim)] * s.n_layer
    out, w = [], c["width"]
    for L in folder_config(c)["layers"]:
        m, f = L["mixer"], L.get("mlp")
        cache = state = att = 0
        if L["type"] == "rglru":
            mix, state = 3 * w * w + 2 * w * (w // m["blocks"]), 4 * w
        elif L["type"] == "latent_attention":
            d, r, q = m["heads"] * m["dim"], m["kv_rank"], m["q_rank"]
            mix, cache, att = (q + r) * w + d * q + 2 * d * r + w * d, r, 2 * d
        elif L["type"] in ("attention", "parallel"):
            a = m["left"] if "left" in m else m
            d, k = a["heads"] * a["dim"], a["kv_heads"] * a["dim"]
            mix, cache, att = 2 * d * w + 2 * k * w, 2 * k, 2 * d
        else:
            mix = 0
        if L["type"] in ("delta", "parallel"):
            a = m.get("right", m)
            d, k = a["heads"] * a["vdim"], a["kv_heads"] * a["dim"]
            mix, state = mix + (2 * k + 2 * d) * w + d * w, state + a["heads"] * a["dim"] * a["vdim"]
        if L["type"] == "mlstm":
            mix, state = 5 * m["heads"] * 128 * w, m["heads"] * 128 * 129
        if f["kind"] == "moe":
            one = 2 * w * f["expert"]["ff"]
            sh = 2 * w * f["shared"]["ff"] if f.get("shared") else 0
            used, held = f["router"]["top"] * one + sh, f["router"]["experts"] * one + sh
        else:
            used = held = (2 if c["design"] == "fidatar" else 3) * w * f["ff"]
        out.append((mix + used, mix + held, cache, state, att))
    return out


def work(case):
    c = case
    per = {"f32": 4.0, "q80": 1.0 + 4.0 / GROUP, "bf16": 2.0}[c["type"]]
    n, m, head = c["prompt"], c["tokens"], c["vocab"] * c["width"]
    mean = sum(range(n, n + m)) / m
    b = f = 0.0
    for used, held, cache, state, att in layer_sizes(c):
        b += per * (min(held, used * n) + m * used) + 4.0 * cache * (n + m * (mean + 1)) + 8.0 * state * (m + 1)
        f += 2.0 * used * (n + m) + 2.0 * att * (n * (n + 1) / 2 + m * mean) + 6.0 * state * (n + m)
    b += per * head * (m + 1) + 4.0 * c["vocab"] * (m + 1)
    f += 2.0 * head * (m + 1)
    return {"bytes": c["requests"] * b, "flops": c["requests"] * f}


def tolerance(case):
    # Measured between two engine modes that are both right, or against exact(): 32-bit weights 5e-7 to 2e-6 (files) and 2e-7 (folders).
    # Q80: a change in the last place turns an int8 activation code here and there, which settles at 0.01 to 0.02 after two to four
    # layers however small the change was.  bfloat16 operands: 2e-3 to 3e-3; with routed experts a close call of the router can
    # also send a token to another expert.
    if case["type"] == "f32":
        return {"rel": 1e-5}
    if case["type"] == "q80":
        return {"rel": 0.03, "max": 0.2}
    return {"rel": 0.01 if case["design"] == "kadesun" else 0.03, "max": 0.2}


# ---- the same requests in 64 bits ----
def exact(case, seed):
    ids = torch.from_numpy(tokens_of(case, seed).astype(np.int64)).cuda()
    with torch.no_grad():
        if case["design"] in FILE_DESIGNS:
            w = file_weights(case)
            return [file_forward(case, w, row)[case["prompt"] - 1:].cpu().numpy() for row in ids]
        w = read_folder(model_path(case))
        return [folder_forward(case, w, row)[case["prompt"] - 1:].cpu().numpy() for row in ids]


def groups_q80(x, dt, half_even):
    """Every group of GROUP values over its largest magnitude / 127 as a whole number, times that again."""
    g = x.to(dt).reshape(-1, GROUP)
    s = g.abs().amax(1, keepdim=True) / 127.0
    r = torch.where(s > 0, g / s, torch.zeros_like(g))
    q = torch.round(r) if half_even else torch.sign(r) * torch.floor(r.abs() + 0.5)
    return (q.double() * s.double()).reshape(x.shape)


def file_forward(c, w, ids):
    spec, _ = file_spec(c)
    H, G, D, T = spec.n_head, spec.n_kv_head, spec.hd, ids.numel()

    def weight(x):
        return x.double() if c["type"] == "f32" else groups_q80(x, torch.float32, True)

    def mul(x, m):
        x = x if c["type"] == "f32" else groups_q80(x, torch.float64, False)
        return x @ weight(m).T

    def norm(x, gain):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-5) * gain.double()

    i = np.arange(0, D, 2, dtype=np.float32) / np.float32(D)
    freq = (np.float32(1.0) / np.power(np.float32(10000.0 if c["design"] == "nano" else 1e6), i)).astype(np.float32)
    ang = torch.from_numpy((np.arange(T, dtype=np.float32)[:, None] * freq[None]).astype(np.float64)).cuda()[:, None]
    cos, sin = torch.cos(ang), torch.sin(ang)

    def rotate(v):
        if c["design"] == "nano":
            a, b = v[..., 0::2], v[..., 1::2]
            return torch.stack([a * cos - b * sin, a * sin + b * cos], -1).reshape(v.shape)
        a, b = v[..., : D // 2], v[..., D // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    x = weight(w["emb"])[ids]
    for l in range(spec.n_layer):
        h = norm(x, w["attn_norm"][l])
        q, k, v = mul(h, w["wq"][l]).reshape(T, H, D), mul(h, w["wk"][l]).reshape(T, G, D), mul(h, w["wv"][l]).reshape(T, G, D)
        if c["design"] == "qwen3":
            q, k = norm(q, w["q_norm"][l]), norm(k, w["k_norm"][l])
        o = softmax_heads(rotate(q), rotate(k), v, D ** -0.5)
        x = x + mul(o, w["wo"][l])
        h = norm(x, w["ffn_norm"][l])
        a = mul(h, w["w1"][l])
        x = x + mul(a * torch.sigmoid(a) * mul(h, w["w3"][l]), w["w2"][l])
    return mul(norm(x, w["final_norm"]), w["emb"])


def softmax_heads(q, k, v, scale, cap=None, sink=None, gate=None):
    """Causal attention: q [T, H, D], k [T, G, D], v [T, G, VD] -> [T, H VD]; sink: a number per head that joins the denominator."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    seen = torch.ones(T, T, dtype=torch.bool, device=q.device).tril()
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h // (H // G)].T) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~seen, -math.inf)
        top = s.amax(1, keepdim=True)
        if sink is not None:
            top = top.clamp_min(float(sink[h]))
        e = torch.exp(s - top)
        den = e.sum(1, keepdim=True) + (torch.exp(sink[h] - top) if sink is not None else 0.0)
        o = (e / den) @ v[:, h // (H // G)]
        out.append(o * gate[:, h:h + 1] if gate is not None else o)
    return torch.cat(out, 1)


def read_folder(path):
    """name -> 64-bit tensor on the GPU, of a model.safetensors that holds bfloat16."""
    with open(os.path.join(path, "model.safetensors"), "rb") as f:
        size = struct.unpack("<Q", f.read(8))[0]
        head, data = json.loads(f.read(size)), np.frombuffer(f.read(), np.uint8)
    out = {}
    for name, t in head.items():
        a, b = t["data_offsets"]
        out[name] = torch.from_numpy(data[a:b].view(np.int16).copy()).cuda().view(torch.bfloat16).reshape(t["shape"])
    return Weights(out)


class Weights(dict):
    """Widened when they are read, so that a large model fits."""

    def __getitem__(self, k):
        return dict.__getitem__(self, k).double()


def unit_rms(u, eps):
    return u / torch.sqrt((u * u).mean(-1, keepdim=True) + eps)


def before(u, back):
    """u a number of tokens earlier, zeros before the start"""
    return torch.cat([torch.zeros_like(u[:back]), u[: u.shape[0] - back]]) if back else u


def conv(u, taps):
    n = taps.shape[1]
    return sum(taps[:, j] * before(u, n - 1 - j) for j in range(n) if n - 1 - j < u.shape[0])


def turn_halves(u, dims, angles, amp=1.0):
    half = dims // 2
    c, s = amp * torch.cos(angles)[:, None], amp * torch.sin(angles)[:, None]
    a, b = u[..., :half], u[..., half:dims]
    return torch.cat([a * c - b * s, b * c + a * s, u[..., dims:]], -1)


def angles_of(rot, T):
    dims, base = rot["dims"], rot["base"]
    f = np.array([base ** (-2.0 * i / dims) for i in range(dims // 2)])
    amp, sc = 1.0, rot.get("scaling")
    if sc:
        place = [dims * math.log(sc["original"] / (2.0 * math.pi * sc[k])) / (2.0 * math.log(base)) for k in ("fast", "slow")]
        lo, hi = max(math.floor(place[0]), 0), min(math.ceil(place[1]), dims - 1)
        ramp = np.clip((np.arange(dims // 2) - lo) / max(hi - lo, 0.001), 0.0, 1.0)
        f, amp = f / sc["factor"] * ramp + f * (1.0 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
    return torch.arange(T, dtype=torch.float64, device="cuda")[:, None] * torch.from_numpy(f).cuda(), amp


def squared_relu_ff(w, p, h):
    return torch.relu(h @ w[p + "up"].T).square() @ w[p + "down"].T


def experts(f, w, p, h, idx, wt):
    out = torch.zeros_like(h)
    for e in range(f["router"]["experts"]):
        t, j = torch.nonzero(idx == e, as_tuple=True)
        if t.numel():
            out[t] += wt[t, j, None] * squared_relu_ff(w, p + "e%d." % e, h[t])
    return out


def famudra_mix(kind, m, w, p, h, eps):
    T = h.shape[0]
    if kind == "latent_attention":
        H, D = m["heads"], m["dim"]
        q = ((unit_rms(h @ w[p + "dq"].T, eps) * w[p + "dq.norm"]) @ w[p + "uq"].T).reshape(T, H, D)
        z = unit_rms(h @ w[p + "dkv"].T, eps) * w[p + "dkv.norm"]
        return softmax_heads(q, (z @ w[p + "uk"].T).reshape(T, H, D), (z @ w[p + "uv"].T).reshape(T, H, m["vdim"]), m["scale"]) @ w[p + "o"].T
    y = torch.nn.functional.gelu(h @ w[p + "y"].T + w[p + "y.b"], approximate="tanh")
    u = conv(h @ w[p + "x"].T + w[p + "x.b"], w[p + "conv"]) + w[p + "conv.b"]
    ub = u.reshape(T, m["blocks"], -1)
    r = torch.sigmoid(torch.einsum("tbi,boi->tbo", ub, w[p + "ra"]) + w[p + "ra.b"]).reshape(T, -1)
    i = torch.sigmoid(torch.einsum("tbi,boi->tbo", ub, w[p + "ri"]) + w[p + "ri.b"]).reshape(T, -1)
    a = torch.exp(-8.0 * r * torch.nn.functional.softplus(w[p + "lam"]))
    drive, S, out = torch.sqrt(1.0 - a * a) * i * u, torch.zeros_like(u[0]), []
    for t in range(T):
        S = a[t] * S + drive[t]
        out.append(S)
    return (torch.stack(out) * y) @ w[p + "o"].T


def famudra_forward(cfg, w, ids):
    eps, x = cfg["norm"]["eps"], w["embed"][ids]
    for n, L in enumerate(cfg["layers"]):
        p, f = "l%d." % n, L["mlp"]
        h = unit_rms(x, eps) * w[p + "norm1"]
        d = famudra_mix(L["type"], L["mixer"], w, p + "mix.", h + (before(h, 1) - h) * w[p + "shift"], eps)
        h = unit_rms(x, eps) * w[p + "norm2"]
        z, idx = torch.topk(h @ w[p + "mlp.router"].T, f["router"]["top"], dim=1)
        x = x + d + experts(f, w, p + "mlp.", h, idx, torch.softmax(z, 1)) + squared_relu_ff(w, p + "mlp.shared.", h)
    return unit_rms(x, eps) * w["final.norm"] @ w["head"].T


def delta_rule(m, w, p, h, eps):
    T, H, G, D, VD = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    silu = torch.nn.functional.silu

    def unit(u):
        return (u / torch.sqrt((u * u).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 1)
    q = unit(silu(conv(h @ w[p + "q"].T, w[p + "q.conv"])).reshape(T, G, D)) / math.sqrt(D)
    k = unit(silu(conv(h @ w[p + "k"].T, w[p + "k.conv"])).reshape(T, G, D))
    v = silu(conv(h @ w[p + "v"].T, w[p + "v.conv"])).reshape(T, H, VD)
    if p + "a1" in w:
        z = (h @ w[p + "a1"].T @ w[p + "a2"].T + w[p + "dt_bias"]).reshape(T, H, D)
        gate = torch.sigmoid(h @ w[p + "g1"].T @ w[p + "g2"].T)
    else:
        z = (h @ w[p + "a"].T + w[p + "dt_bias"])[..., None].expand(T, H, D)
        gate = silu(h @ w[p + "g"].T)
    g = torch.exp(-torch.exp(w[p + "A_log"])[:, None] * torch.nn.functional.softplus(z))
    beta, S, out = torch.sigmoid(h @ w[p + "b"].T), torch.zeros(H, D, VD, dtype=torch.float64, device=h.device), []
    for t in range(T):
        S = S * g[t][..., None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t][..., None] * u[:, None]
        out.append(torch.einsum("hdv,hd->hv", S, q[t]))
    return ((unit_rms(torch.stack(out), eps) * w[p + "norm"]).reshape(T, -1) * gate) @ w[p + "o"].T


def kadesun_forward(cfg, w, ids):
    eps, x = cfg["norm"]["eps"], w["embed"][ids]
    T = ids.numel()
    for n, L in enumerate(cfg["layers"]):
        p, m = "l%d." % n, L["mixer"]
        if L["type"] == "delta":
            d = delta_rule(m, w, p + "mix.", x, eps)
        else:
            a, q = m["left"], p + "mix.left."
            ang, amp = angles_of(a["rot"], T)
            Q = turn_halves((unit_rms(x @ w[q + "q"].T, eps) * w[q + "q.norm"]).reshape(T, a["heads"], -1), a["rot"]["dims"], ang, amp)
            K = turn_halves((unit_rms(x @ w[q + "k"].T, eps) * w[q + "k.norm"]).reshape(T, a["kv_heads"], -1), a["rot"]["dims"], ang, amp)
            o = softmax_heads(Q, K, (x @ w[q + "v"].T).reshape(T, a["kv_heads"], -1), a["scale"], a["softcap"], w[q + "sink"], torch.sigmoid(x @ w[q + "g"].T)) @ w[q + "o"].T
            r = delta_rule(m["right"], w, p + "mix.right.", x, eps)
            d = 0.5 * (unit_rms(o, eps) * w[p + "mix.left.out"] + unit_rms(r, eps) * w[p + "mix.right.out"])
        x = x + unit_rms(d, eps) * w[p + "norm1"]
        y = (torch.nn.functional.silu(x @ w[p + "mlp.gate"].T) * (x @ w[p + "mlp.up"].T)) @ w[p + "mlp.down"].T
        x = x + unit_rms(y, eps) * w[p + "norm2"]
    return unit_rms(x, eps) * w["final.norm"] @ w["head"].T


def matrix_memory(m, w, p, h, eps):
    T, H, D, VD, cap = h.shape[0], m["heads"], m["dim"], m["vdim"], m["gate_cap"]
    q, k, v = [(h @ w[p + n].T).reshape(T, H, -1) for n in "qkv"]
    q = q / math.sqrt(D)
    li = cap * torch.tanh((h @ w[p + "i"].T + w[p + "i.b"]) / cap)
    lf = torch.nn.functional.logsigmoid(cap * torch.tanh((h @ w[p + "f"].T + w[p + "f.b"]) / cap))
    new = lambda *s: torch.zeros(*s, dtype=torch.float64, device=h.device)          # noqa: E731
    S, n, mx, out = new(H, D, VD), new(H, D), new(H), []
    for t in range(T):
        top = torch.maximum(lf[t] + mx, li[t])
        keep, put = torch.exp(lf[t] + mx - top)[:, None], torch.exp(li[t] - top)[:, None]
        S = keep[..., None] * S + (put * k[t])[..., None] * v[t][:, None]
        n = keep * n + put * k[t]
        mx = top
        den = torch.maximum((n * q[t]).sum(1).abs(), torch.exp(-mx)) + 1e-6
        out.append(torch.einsum("hdv,hd->hv", S, q[t]) / den[:, None])
    o = unit_rms(torch.stack(out), eps).reshape(T, -1)
    return (o * w[p + "norm"] * torch.sigmoid(h @ w[p + "g"].T)) @ w[p + "o"].T


def fidatar_forward(cfg, w, ids):
    eps, alpha, T = cfg["norm"]["eps"], cfg["postln_alpha"], ids.numel()
    x = w["embed"][ids] * cfg["embedding"]["scale"]
    for n, L in enumerate(cfg["layers"]):
        p, m, f = "l%d." % n, L["mixer"], L["mlp"]
        q = p + "mix."
        if L["type"] == "mlstm":
            d = matrix_memory(m, w, q, x, eps)
        else:          # (a request is shorter than a block of positions)
            ang, amp = angles_of(m["rot"], T)
            Q, K, V = [(x @ w[q + s].T + w[q + s + ".b"]).reshape(T, g, -1) for s, g in (("q", m["heads"]), ("k", m["kv_heads"]), ("v", m["kv_heads"]))]
            Q, K = unit_rms(Q, eps) * w[q + "q.norm"], unit_rms(K, eps) * w[q + "k.norm"]
            one = torch.zeros(m["heads"], dtype=torch.float64, device=x.device)
            d = softmax_heads(turn_halves(Q, m["rot"]["dims"], ang, amp), turn_halves(K, m["rot"]["dims"], ang, amp), V, m["scale"], sink=one) @ w[q + "o"].T
        x = unit_rms(alpha * x + d, eps) * w[p + "norm1"]
        if f["kind"] == "moe":
            r, gc = f["router"], f["router"]["groups"]["count"]
            s = torch.sigmoid(x @ w[p + "mlp.router"].T)
            best = s.reshape(T, gc, -1).topk(2, dim=2)[0].sum(2).topk(r["groups"]["keep"], dim=1)[1]
            closed = torch.ones(T, gc, dtype=torch.bool, device=x.device).scatter_(1, best, False).repeat_interleave(r["experts"] // gc, 1)
            wt, idx = s.masked_fill(closed, -1.0).topk(r["top"], dim=1)
            y = experts(f, w, p + "mlp.", x, idx, wt * r["scale"])
        else:
            y = squared_relu_ff(w, p + "mlp.", x)
        x = unit_rms(alpha * x + y, eps) * w[p + "norm2"]
    z = unit_rms(x, eps) * w["final.norm"] @ w["head"].T
    return cfg["logit_softcap"] * torch.tanh(z / cfg["logit_softcap"])


def folder_forward(c, w, ids):
    return {"famudra": famudra_forward, "kadesun": kadesun_forward, "fidatar": fidatar_forward}[c["design"]](folder_config(c), w, ids)
