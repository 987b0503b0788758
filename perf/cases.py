"""What a user of this library has it do, as cases that can be timed.

A case is one model, one kind of call and its sizes:

  rounds   speculative decoding the way the command line runs it: the last prompt token, then R rounds of draft, chained drafts
           and a verify block of M tokens through the blocking calls.  The drafts of a random head are worthless, so a table
           replaces them that agrees with the model's own greedy stream with probability 0.8, as in the benchmark.
  plain    n tokens of a given text, one forward each, logits on the host (sampling or scoring on the host side)
  prompt   n tokens of a prompt at position pos0, logits of the last one

A session is opened once per model and kept, as a server keeps it; what comes before the call -- `depth` or `pos0` tokens of one
fixed text -- is in the cache already, the tokens of the call itself come from the seed.  The models are written to a folder for
temporary files at their first use.  Block-quantised models are the conditioned twins of the benchmark's (query norms of
hd^-0.5, as real checkpoints have bounded scores) with weights large enough that the token's own embedding stays visible in
the residual: a random model of 48 layers otherwise picks between near ties, and any rounding would change its stream.
"""
from __future__ import annotations

import dataclasses
import importlib
import json
import math
import os
import struct
import tempfile

import numpy as np
import torch

lg = importlib.import_module("little-gemma_b200")
synth = importlib.import_module("little-gemma_b200.synth")

CACHE = os.path.join(tempfile.gettempdir(), f"lg_cases_{os.getuid()}")
ACCEPT = 0.8            # how often a replayed draft is the model's own next token


# ------------------------------------------------------------------------------------------------------------------------
# models
# ------------------------------------------------------------------------------------------------------------------------

def _latent_8b():
    lay = [synth.LatentLayer(heads=32, dim=128, rot_dim=64, vdim=128, q_rank=1536, kv_rank=512, ff=14336) for _ in range(6)]
    return synth.LatentShape(width=4096, vocab=32768, layers=lay)


def _hybrid_2b():
    ssm = synth.SsmLayer(heads=64, vdim=64, state=128, groups=8, norm_groups=8, conv=4, ff=8192)
    att = synth.DiffLayer(heads=16, kv_heads=4, dim=64, vdim=128, window=1024, conv=4, ff=8192)
    return synth.HybridShape(width=2048, vocab=32768, layers=[ssm, ssm, ssm, att] * 2)


def _quant(shape, sigma, **kw):
    return dataclasses.replace(shape, q_norm_scale=shape.head_dim ** -0.5, sigma=sigma, **kw)


# name -> (shape, draft head's shape, rows of the cache)
MODELS = {
    "tiny": (_quant(synth.TINY, 0.2), synth.TINY_HEAD, 1024),
    "b12": (_quant(synth.B12, 0.05), synth.B12_HEAD, 4096),
    "e4b": (_quant(synth.E4B, 0.1), synth.E4B_HEAD, 16384),
    "b12k": (_quant(synth.B12, 0.05, n_layer=8, n_vocab=32768, wtype=synth.Q4_K), synth.B12_HEAD, 4096),
    "latent": (_latent_8b(), None, 8192),
    "hybrid": (_hybrid_2b(), None, 4096),
}


def listed():
    return [
        # a chat turn on the smallest model: launches and waits are all there is
        {"name": "tiny_rounds", "model": "tiny", "kind": "rounds", "depth": 100, "width": 4, "n": 16},
        # the headline: 12B-class q4_0, verify blocks of 4, 1024 tokens of context
        {"name": "b12_rounds", "model": "b12", "kind": "rounds", "depth": 1024, "width": 4, "n": 16},
        # the same model without a draft head, host-side sampling, an odd position past the sliding window
        {"name": "b12_plain", "model": "b12", "kind": "plain", "depth": 2999, "width": 1, "n": 8},
        # the reference's prompt length
        {"name": "b12_prompt", "model": "b12", "kind": "prompt", "depth": 0, "width": 1, "n": 929},
        # a long document on the model with per-layer embeddings
        {"name": "e4b_rounds_deep", "model": "e4b", "kind": "rounds", "depth": 8192, "width": 4, "n": 16},
        # the user's next message in a running chat: a short, ragged prompt
        {"name": "e4b_turn", "model": "e4b", "kind": "prompt", "depth": 701, "width": 1, "n": 45},
        # the other block format; wide verify blocks (two activation panels)
        {"name": "b12k_rounds_wide", "model": "b12k", "kind": "rounds", "depth": 500, "width": 8, "n": 16},
        {"name": "b12k_prompt", "model": "b12k", "kind": "prompt", "depth": 0, "width": 1, "n": 2048},
        # layer-plan models in bf16: latent attention ...
        {"name": "latent_plain", "model": "latent", "kind": "plain", "depth": 2048, "width": 1, "n": 16},
        {"name": "latent_prompt", "model": "latent", "kind": "prompt", "depth": 0, "width": 1, "n": 2048},
        # ... and state-space layers with windowed attention between them
        {"name": "hybrid_plain", "model": "hybrid", "kind": "plain", "depth": 1300, "width": 1, "n": 24},
        {"name": "hybrid_prompt", "model": "hybrid", "kind": "prompt", "depth": 0, "width": 1, "n": 1999},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    model = rng.choice(["tiny", "b12", "e4b", "b12k", "latent", "hybrid"])
    kind = rng.choice(["rounds", "plain", "prompt"] if MODELS[model][1] is not None else ["plain", "prompt"])
    rows = MODELS[model][2]
    if kind == "rounds":
        return {"model": model, "kind": kind, "depth": _log(rng, 8, min(8192, rows - 200)), "width": rng.randint(2, 8), "n": rng.randint(4, 16)}
    if kind == "plain":
        return {"model": model, "kind": kind, "depth": _log(rng, 8, min(8192, rows - 200)), "width": 1, "n": rng.randint(4, 8 if model == "b12" else 24)}
    n = _log(rng, 9, min(2048, rows // 2) if model != "b12" else 929)
    return {"model": model, "kind": kind, "depth": rng.choice([0, _log(rng, 8, rows // 2 - 100)]), "width": 1, "n": n}


def _checkpoint(path, shape, seed):
    """A seeded checkpoint folder with matrices N(0, 1/k), drawn on the GPU."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator("cuda").manual_seed(seed)
    w = {}
    for name, dims in shape.tensors().items():
        own = shape.special(name, dims, rng) if hasattr(shape, "special") else None
        if own is not None:
            w[name] = synth.to_bf16(own)
        elif len(dims) == 1:
            mean, std = (1.0, 0.5) if name.endswith("sink") else (1.0, 0.2)
            w[name] = synth.to_bf16(mean + std * rng.standard_normal(dims))
        else:
            v = torch.randn(dims, generator=gen, device="cuda") * (1.0 if name == "embed" else dims[1] ** -0.5)
            w[name] = v.to(torch.bfloat16).view(torch.int16).cpu().numpy().view(np.uint16)
    synth.write_checkpoint(path, shape, weights=w)


def _files(model):
    """(target, draft head or None) of a model, written at its first use."""
    shape, head, _ = MODELS[model]
    os.makedirs(CACHE, exist_ok=True)
    if not isinstance(shape, synth.TargetShape):
        path = os.path.join(CACHE, model)
        if not os.path.exists(os.path.join(path, "config.json")):
            tmp = f"{path}.{os.getpid()}"
            _checkpoint(tmp, shape, 11)
            os.replace(tmp, path)
        return path, None
    dev = "cuda" if shape.weight_bytes() > (1 << 28) else "cpu"
    return (synth.cached(CACHE, f"{model}.gguf", synth.write_target, shape, 11, dev),
            synth.cached(CACHE, f"{model}_head.gguf", synth.write_head, head, shape, 12, dev))


_open = {"key": None, "session": None, "saved": None}     # the library runs one model per process


def _session(model, width):
    key = (model, width)
    if _open["key"] != key:
        if _open["session"] is not None:
            _open["session"].close()
        _open.update(key=None, session=None, saved=None)
        target, head = _files(model)
        _open["session"] = lg.Session(target, head, MODELS[model][2], mtp_n=width)
        _open["key"] = key
    return _open["session"]


def _text(model, n, seed):
    return synth.prompt_ids(n, _vocab(model), seed=seed)


def _vocab(model):
    s = MODELS[model][0]
    return s.n_vocab if isinstance(s, synth.TargetShape) else s.vocab


def _tokens(case, seed):
    """the call's own tokens"""
    return _text(case["model"], 1 if case["kind"] == "rounds" else case["n"], 1000 + seed)


def prepare(case, seed):
    model, kind, depth = case["model"], case["kind"], case["depth"]
    s = _session(model, case["width"])
    state = {"case": case, "session": s, "tokens": _tokens(case, seed)}
    if model == "hybrid":
        # recurrent states cannot be rewound: the context is a saved prefix that every call starts from
        if depth and _open["saved"] != depth:
            s.prefill(_text(model, depth, 5), 0)
            s.save_prefix(depth)
            _open["saved"] = depth
    elif depth:
        s.prefill(_text(model, depth, 5), 0)
    if kind == "rounds":
        n = case["n"] * case["width"] + 2
        first = s.next(int(state["tokens"][0]), depth)
        stream, _ = s.rounds_host(first, depth + 1, 1, n, 0, 0)
        state["replay"] = synth.replay_drafts(np.concatenate([[first], stream]), _vocab(model), ACCEPT, seed=seed)
    return state


def run(state):
    case, s, toks = state["case"], state["session"], state["tokens"]
    if s is not _open["session"]:
        raise RuntimeError("another model was opened since this state was prepared")
    depth, n = case["depth"], case["n"]
    if case["model"] == "hybrid" and depth:
        s.restore_prefix(depth)
    if case["kind"] == "prompt":
        return s.prefill_logits(toks, depth, [n - 1])
    if case["kind"] == "plain":
        return np.stack([s.forward(int(t), depth + i) for i, t in enumerate(toks)])
    first = s.next(int(toks[0]), depth)
    stream, stats = s.rounds_host(first, depth + 1, 1, n * case["width"] + 2, n, 3, state["replay"])
    return {"first": first, "stream": _padded(stream, case), "position": stats["pos"], "accepted": stats["n_accept"], "hidden": s.last_hidden()}


def _padded(stream, case):
    """the emitted tokens, -1 behind the last one: how many there are depends on what was accepted"""
    out = np.full(case["n"] * case["width"] + 1, -1, dtype=np.int32)
    out[:len(stream)] = stream
    return out


# ------------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------------------------------

def _layers(case):
    """per layer run: (weights, cached values per position and the most positions a query sees, operations per query and seen
    position, state bytes), and the head's weights"""
    s = MODELS[case["model"]][0]
    out = []
    if isinstance(s, synth.TargetShape):
        for l in range(s.n_layer):
            q, kv = s.n_head * s.hd(l), s.n_head_kv * s.hd(l)
            out.append((s.n_embd * (2 * q + 2 * kv + 3 * s.n_ff + 2 * s.ple) + s.n_embd * s.ple, 2 * kv, s.window if s.is_local(l) else None, 4 * q, 0))
        return out, s.n_vocab * s.n_embd
    W = s.width
    for i, l in enumerate(s.layers):
        w = sum(int(np.prod(d)) for k, d in s.tensors().items() if k.startswith(f"l{i}."))
        if isinstance(l, synth.LatentLayer):
            out.append((w, l.kv_rank + l.rot_dim, None, 2 * l.heads * (l.dim + l.rot_dim + l.vdim), 0))
        elif isinstance(l, synth.SsmLayer):
            out.append((w, 0, 0, 0, 4 * l.heads * l.vdim * l.state))
        else:
            out.append((w, l.kv_heads * (2 * l.dim + l.vdim), l.window, 2 * l.heads * (2 * l.dim + 2 * l.vdim), 0))
    return out, s.vocab * W


def work(case):
    """Weights once per forward, cached rows once per forward and layer, states in and out; 2 operations per weight and token and
    the scores and weighted sums of attention (of a state: decay, update and output)."""
    layers, head = _layers(case)
    per = 0.5625 if isinstance(MODELS[case["model"]][0], synth.TargetShape) else 2.0
    weights = sum(l[0] for l in layers)

    def forward(pos, n, heads, wide=True):
        by, fl = per * (weights + (head if heads else 0)), 2.0 * (weights * n + head * heads)
        for _, row, window, ops, state in layers:
            seen = lambda p: p + 1 if window is None else min(p + 1, window)
            first = 0 if window is None else max(0, pos + 1 - window)
            by += 2.0 * row * (pos + n - first) + 2 * state
            fl += ops * sum(seen(p) for p in range(pos, pos + n)) + 1.5 * state * n
        return by, fl

    depth, n = case["depth"], case["n"]
    vocab = 4.0 * _vocab(case["model"])
    if case["kind"] == "prompt":
        by, fl = forward(depth, n, 1)
        return {"bytes": by + vocab, "flops": fl}
    if case["kind"] == "plain":
        steps = [forward(depth + i, 1, 1) for i in range(n)]
        return {"bytes": sum(b for b, _ in steps) + vocab * n, "flops": sum(f for _, f in steps)}
    M, (t, h, _) = case["width"], MODELS[case["model"]]
    block = h.n_inner * (2 * h.n_head * t.head_dim + 3 * h.n_ff)
    draft = 2 * t.n_embd * h.n_inner + t.n_vocab * h.n_inner + h.n_layer * block
    chain = h.n_inner * t.n_embd
    b1, f1 = forward(depth, 1, 1)
    b2, f2 = forward(depth + n * 2, M, M)
    drafts = (M - 1) * draft + (M - 2) * chain
    return {"bytes": b1 + n * (b2 + per * drafts), "flops": f1 + n * (f2 + 2.0 * drafts)}


def tolerance(case):
    """About four times what two orders of the sums make of 16-bit operands: f16 and 16-bit groups in the block-quantised models
    (0.0007 off the 64-bit result), bf16 in the others (0.006 off)."""
    if isinstance(MODELS[case["model"]][0], synth.TargetShape):
        return {"rel": 0.003, "max": 0.03, "differ": 0.01}
    return {"rel": 0.02, "max": 0.2, "differ": 0.01}


# ------------------------------------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------------------------------------

class _Gguf:
    """Tensors of a GGUF file as float64 on the GPU."""

    def __init__(self, path):
        self.raw = np.memmap(path, dtype=np.uint8, mode="r")
        self.at, self.t = 4, {}
        _, n_t, n_kv = self._take("<IQQ")
        for _ in range(n_kv):
            self._text()
            self._value(self._take("<I")[0])
        for _ in range(n_t):
            name = self._text()
            dims = self._take("<%dQ" % self._take("<I")[0])
            self.t[name] = (dims,) + self._take("<IQ")
        self.base = (self.at + 31) // 32 * 32

    def _take(self, fmt):
        v = struct.unpack_from(fmt, self.raw, self.at)
        self.at += struct.calcsize(fmt)
        return v

    def _text(self):
        n = self._take("<Q")[0]
        self.at += n
        return bytes(self.raw[self.at - n:self.at]).decode()

    def _value(self, kind):
        size = {0: 1, 1: 1, 2: 2, 3: 2, 4: 4, 5: 4, 6: 4, 7: 1, 10: 8, 11: 8, 12: 8}
        if kind == 8:
            self._text()
        elif kind == 9:
            of, n = self._take("<IQ")
            if of == 8:
                for _ in range(n):
                    self.at += 8 + struct.unpack_from("<Q", self.raw, self.at)[0]
            else:
                self.at += size[of] * n
        else:
            self.at += size[kind]

    def rows(self, name, at=None, stop=None):
        """rows [at, stop) (at: also a list of rows) as float64 [rows, k]"""
        dims, kind, off = self.t[name]
        k, m = dims[0], dims[1] if len(dims) > 1 else 1
        per, blk = {0: (4, 1), 2: (18, 32), 12: (144, 256)}[kind]
        table = self.raw[self.base + off:self.base + off + m * k // blk * per].reshape(m, k // blk * per)
        some = table[0 if at is None else at:m if stop is None else stop] if at is None or np.isscalar(at) else table[np.asarray(at)]
        b = torch.from_numpy(np.ascontiguousarray(some)).cuda()
        n = b.shape[0]
        if kind == 0:
            return b.view(torch.float32).double().reshape(n, k)
        b = b.reshape(n, k // blk, per)
        half = lambda x: x.contiguous().view(torch.float16).double()
        if kind == 2:
            q = torch.cat([b[..., 2:] & 15, b[..., 2:] >> 4], -1).double() - 8
            return (q * half(b[..., :2])).reshape(n, k)
        d, dmin, s, q = half(b[..., :2]), half(b[..., 2:4]), b[..., 4:16], b[..., 16:]
        sc = torch.cat([s[..., :4] & 63, (s[..., 8:] & 15) | ((s[..., :4] >> 6) << 4)], -1).double()
        mn = torch.cat([s[..., 4:8] & 63, (s[..., 8:] >> 4) | ((s[..., 4:8] >> 6) << 4)], -1).double()
        q = q.reshape(*q.shape[:-1], 4, 32)
        q = torch.stack([q & 15, q >> 4], -2).reshape(*q.shape[:-2], 8, 32).double()
        return (d[..., None] * sc[..., None] * q - dmin[..., None] * mn[..., None]).reshape(n, k)

    def vec(self, name):
        return self.rows(name).reshape(-1)

    def mul(self, name, x):
        """x [n, k] times the matrix: [n, m]"""
        m = self.t[name][0][1]
        step = max(1, (1 << 28) // x.shape[1])
        return torch.cat([x @ self.rows(name, i, min(m, i + step)).T for i in range(0, m, step)], 1)


def _unit(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, window, sink=None):
    """Causal attention of a whole sequence: q [n, H, d], k [n, G, d], v [n, G, vd] -> [n, H, vd]"""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    k, v = k.permute(1, 2, 0), v.permute(1, 0, 2)                # [G, d, n], [G, n, vd]
    out = []
    step = max(16, (1 << 28) // (n * H))
    for i in range(0, n, step):
        j = min(n, i + step)
        lo = 0 if window is None else max(0, i - window + 1)
        s = torch.matmul(q[i:j].reshape(j - i, G, H // G, -1).permute(1, 2, 0, 3), k[:, None, :, lo:j]) * scale
        back = torch.arange(i, j, device="cuda")[:, None] - torch.arange(lo, j, device="cuda")[None, :]
        seen = (back >= 0) if window is None else (back >= 0) & (back < window)
        s = s.masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.reshape(G, H // G, 1, 1).expand(-1, -1, j - i, 1)], -1)
        p = torch.softmax(s, -1)[..., :j - lo]
        out.append(torch.matmul(p, v[:, None, lo:j]).permute(2, 0, 1, 3).reshape(j - i, H, -1))
    return torch.cat(out)


def _neox(x, base):
    """x [n, heads, hd]: pairs (i, i + hd / 2) turn by position * base^(-2i / hd)"""
    n, hd = x.shape[0], x.shape[-1]
    a = torch.outer(torch.arange(n, device="cuda").double(), base ** (-torch.arange(0, hd, 2, device="cuda").double() / hd))[:, None]
    u, w = x[..., :hd // 2], x[..., hd // 2:]
    return torch.cat([u * a.cos() - w * a.sin(), u * a.sin() + w * a.cos()], -1)


def _exact_quant(shape, path, tokens, places):
    """(normed hidden rows, logits) of the block-quantised model at `places`"""
    f = _Gguf(path)
    ne, eps, n = shape.n_embd, shape.eps, len(tokens)
    gelu = lambda z: 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))
    x = f.rows("token_embd.weight", tokens) * math.sqrt(ne)
    if shape.ple:
        P = shape.ple
        row = f.rows("per_layer_token_embd.weight", tokens) * math.sqrt(P)
        proj = (f.mul("per_layer_model_proj.weight", x) / math.sqrt(ne)).reshape(n, -1, P)
        proj = _unit(proj, eps) * f.vec("per_layer_proj_norm.weight")
        ipl = (proj + row.reshape(n, -1, P)) / math.sqrt(2)
    for l in range(shape.n_layer):
        p, hd, local = f"blk.{l}.", shape.hd(l), shape.is_local(l)
        base = shape.rope_base_swa if local else shape.rope_base
        h = _unit(x, eps) * f.vec(p + "attn_norm.weight")
        q, k, v = (f.mul(p + f"attn_{t}.weight", h).reshape(n, -1, hd) for t in "qkv")
        q = _neox(_unit(q, eps) * f.vec(p + "attn_q_norm.weight"), base)
        k = _neox(_unit(k, eps) * f.vec(p + "attn_k_norm.weight"), base)
        o = _attend(q, k, _unit(v, eps), 1.0, shape.window if local else None).reshape(n, -1)
        x = x + _unit(f.mul(p + "attn_output.weight", o), eps) * f.vec(p + "post_attention_norm.weight")
        h = _unit(x, eps) * f.vec(p + "ffn_norm.weight")
        g = gelu(f.mul(p + "ffn_gate.weight", h)) * f.mul(p + "ffn_up.weight", h)
        x = x + _unit(f.mul(p + "ffn_down.weight", g), eps) * f.vec(p + "post_ffw_norm.weight")
        if shape.ple:
            g = gelu(f.mul(p + "inp_gate.weight", x)) * ipl[:, l]
            x = x + _unit(f.mul(p + "proj.weight", g), eps) * f.vec(p + "post_norm.weight")
    h = _unit(x[places], eps) * f.vec("output_norm.weight")
    return h, f.mul("token_embd.weight", h)


class _Tensors:
    """A checkpoint folder's tensors as float64 on the GPU."""

    def __init__(self, path):
        with open(os.path.join(path, "model.safetensors"), "rb") as f:
            n = struct.unpack("<Q", f.read(8))[0]
            self.head = json.loads(f.read(n))
        self.raw = np.memmap(os.path.join(path, "model.safetensors"), dtype=np.uint8, mode="r", offset=8 + n)

    def __call__(self, name):
        t = self.head[name]
        a, b = t["data_offsets"]
        return torch.from_numpy(np.array(self.raw[a:b])).view(torch.bfloat16).cuda().double().reshape(t["shape"])


def _exact_latent(shape, path, tokens, places):
    w, eps, n = _Tensors(path), shape.eps, len(tokens)
    embed = w("embed")
    x = embed[torch.from_numpy(np.asarray(tokens)).long().cuda()]

    def norm(z, name):
        z = z - z.mean(-1, keepdim=True)
        return _unit(z, eps) * w(name)

    def turn(z, base):
        a = torch.outer(torch.arange(n, device="cuda").double(), base ** (-torch.arange(0, z.shape[-1], 2, device="cuda").double() / z.shape[-1]))[:, None]
        u, v = z[..., ::2], z[..., 1::2]
        return torch.stack([u * a.cos() - v * a.sin(), u * a.sin() + v * a.cos()], -1).flatten(-2)

    for i, l in enumerate(shape.layers):
        p, H = f"l{i}.mix.", l.heads
        h = norm(x, f"l{i}.norm1")
        q = ((_unit(h @ w(p + "dq").T, eps) * w(p + "dq.norm")) @ w(p + "uq").T).reshape(n, H, -1)
        r = h @ w(p + "dkv").T
        c = _unit(r[:, :l.kv_rank], eps) * w(p + "dkv.norm")
        k_rot = turn(r[:, None, l.kv_rank:], l.base).expand(-1, H, -1)
        k = torch.cat([(c @ w(p + "uk").T).reshape(n, H, -1), k_rot], -1)
        q = torch.cat([q[..., :l.dim], turn(q[..., l.dim:], l.base)], -1)
        o = _attend(q, k, (c @ w(p + "uv").T).reshape(n, H, -1), l.score_scale(), None, w(p + "sink")).reshape(n, -1)
        x = x + shape.residual_mult * norm((o * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T, f"l{i}.norm1b")
        h = norm(x, f"l{i}.norm2")
        g = torch.relu(h @ w(f"l{i}.mlp.gate").T) * (h @ w(f"l{i}.mlp.up").T)
        x = x + shape.residual_mult * norm(g @ w(f"l{i}.mlp.down").T, f"l{i}.norm2b")
    return norm(x[places], "final.norm") @ embed.T


def _exact_hybrid(shape, path, tokens, places):
    w, eps, n = _Tensors(path), shape.eps, len(tokens)
    embed = w("embed")
    x = embed[torch.from_numpy(np.asarray(tokens)).long().cuda()]
    norm = lambda z, name: _unit(z, eps) * (1 + w(name))

    def conv(u, name, bias=None):
        f = w(name)
        out = torch.zeros_like(u)
        for back in range(f.shape[1]):
            out[back:] += u[:n - back] * f[:, f.shape[1] - 1 - back]
        return out if bias is None else out + w(bias)

    for i, l in enumerate(shape.layers):
        p, H = f"l{i}.mix.", l.heads
        h = norm(x, f"l{i}.norm1")
        if isinstance(l, synth.SsmLayer):
            inner, gn = H * l.vdim, l.groups * l.state
            z, xbc, dt = torch.split(h @ w(p + "in").T, [inner, inner + 2 * gn, H], 1)
            xs, B, C = torch.split(torch.nn.functional.silu(conv(xbc, p + "conv", p + "conv.b")), [inner, gn, gn], 1)
            xs = xs.reshape(n, H, l.vdim)
            B, C = (t.reshape(n, l.groups, l.state).repeat_interleave(H // l.groups, 1) for t in (B, C))
            dt = torch.nn.functional.softplus(dt + w(p + "dt_bias"))
            decay, dx, S, ys = torch.exp(-torch.exp(w(p + "A_log")) * dt), dt[..., None] * xs, torch.zeros(H, l.vdim, l.state, dtype=torch.float64, device="cuda"), []
            for t in range(n):
                S = S * decay[t][:, None, None] + dx[t][:, :, None] * B[t][:, None, :]
                ys.append(torch.matmul(S, C[t][:, :, None])[..., 0])
            y = (torch.stack(ys) + w(p + "D")[:, None] * xs).reshape(n, inner) * torch.nn.functional.silu(z)
            o = _unit(y.reshape(n, l.norm_groups, -1), eps).reshape(n, inner) * w(p + "norm")
        else:
            q, k, v = (conv(h @ w(p + t).T, p + t + ".conv") for t in "qkv")
            q, k, v = q.reshape(n, H, 2, l.dim), k.reshape(n, l.kv_heads, 2, l.dim), v.reshape(n, l.kv_heads, l.vdim)
            lam = torch.exp(w(p + "lq1") @ w(p + "lk1")) - torch.exp(w(p + "lq2") @ w(p + "lk2")) + l.diff
            a, b = (_attend(q[:, :, m], k[:, :, m], v, l.dim ** -0.5, l.window) for m in (0, 1))
            o = (_unit(a - lam * b, eps) * (1 - l.diff)).reshape(n, -1)
        x = x + o @ w(p + "o").T + torch.relu(norm(x, f"l{i}.norm2") @ w(f"l{i}.mlp.up").T) ** 2 @ w(f"l{i}.mlp.down").T
    return norm(x[places], "final.norm") @ embed.T * shape.logit_scale


def exact(case, seed):
    model, depth, n = case["model"], case["depth"], case["n"]
    shape = MODELS[model][0]
    context = np.concatenate([_text(model, depth, 5), _tokens(case, seed)]) if depth else _tokens(case, seed)
    path = _files(model)[0]
    if isinstance(shape, synth.TargetShape):
        if case["kind"] == "prompt":
            return _exact_quant(shape, path, context, [len(context) - 1])[1].cpu().numpy()
        if case["kind"] == "plain":
            return _exact_quant(shape, path, context, list(range(depth, depth + n)))[1].cpu().numpy()
        # greedy stream: a guess (the last token again and again) that is corrected until it is its own continuation
        M, stream = case["width"], [int(context[-1])] * (n * case["width"] + 2)
        for _ in range(3):
            places = list(range(depth, depth + len(stream) + 1))
            hidden, logits = _exact_quant(shape, path, np.concatenate([context, stream]).astype(np.int64), places)
            greedy = logits.argmax(1).tolist()[:len(stream)]
            if greedy == stream:
                break
            stream = greedy
        else:
            return None
        replay = synth.replay_drafts(np.array(stream), shape.n_vocab, ACCEPT, seed=seed)
        g, pos, accepted = 1, depth + 1, 0
        for _ in range(n):
            adv = 1
            while adv < M and replay[g + adv - 1] == stream[g + adv - 1]:
                adv += 1
            g, pos, accepted = g + adv, pos + adv, accepted + adv - 1
        return {"first": stream[0], "stream": _padded(stream[1:g], case), "position": pos, "accepted": accepted,
                "hidden": hidden[pos - 1 - depth].cpu().numpy()}
    places = [len(context) - 1] if case["kind"] == "prompt" else list(range(depth, depth + n))
    return (_exact_latent if model == "latent" else _exact_hybrid)(shape, path, context, places).cpu().numpy()
