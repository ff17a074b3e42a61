"""Workloads of the framework, through its public entry points: what a program that serves models with it calls, from the
smallest decode call to whole prompts and whole requests.

    layer       one decode layer for a batch of sequences: the two fused C entry points a host calls per layer
    tokens      greedy tokens of a whole Llama-type model (begin + generate, replayed as a graph)
    compressed  last-token attention over the FP16-K / q4-V cache, one call per sequence
    prefill     packed variable-length causal prompt attention
    prompt      new prompts through step() of a whole model
    requests    whole requests: prompts in one step(), then greedy tokens by generate()

Models: Llama-type stacks (DecodeModel), Lamutar and Sidalorn (models.read_config + build), at the sizes of bench.py.
All data is made on the GPU from the seed.
"""
from __future__ import annotations

import importlib.util
import math
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_DEV = "cuda"
F64 = torch.float64
EPS = 1e-5
VOCAB = 32000

# hidden, q heads, kv heads, head size, feed-forward size, Q8_0 feed-forward (else f16), RoPE layout, RoPE base, q/k/v biases
LAYERS = {
    "llama3-8b": (4096, 32, 8, 128, 14336, True, 0, 5e5, False),
    "qwen2.5-3b": (2048, 16, 2, 128, 11008, False, 1, 1e6, True),
    "tinyllama": (2048, 32, 4, 64, 5632, False, 0, 1e4, False),
}
# width, feed-forward size, q heads, kv heads, head size, delta heads, delta size, low rank, layers
STACKS = {
    "tinyllama-sized": (2048, 5632, 32, 4, 64, 32, 64, 64, 8),
    "llama3-8b-sized": (4096, 14336, 32, 8, 128, 64, 64, 128, 4),
}
# heads, head size, latent size, recurrence blocks, experts, identity outputs, groups, kept groups, chosen, expert ff, shared ff
SIDALORN = {
    "tinyllama-sized": (16, 128, 512, 16, 60, 4, 8, 4, 6, 704, 1408),
    "llama3-8b-sized": (32, 128, 512, 16, 60, 4, 8, 4, 6, 1792, 3584),
}
COMPRESSED = (16, 2, 128, 512, 64, 64)  # q heads, kv heads, head size, recent ring, block, selected blocks


def listed():
    return [
        # one user, one layer of the headline model at a long context: latency of the smallest decode call
        {"name": "layer-1", "kind": "layer", "shape": "llama3-8b", "rows": 1, "low": 7969, "high": 7969, "mix": 1},
        # a lightly loaded server
        {"name": "layer-6", "kind": "layer", "shape": "llama3-8b", "rows": 6, "low": 512, "high": 8192, "mix": 2},
        # the headline batch: 32 sequences, contexts 512 to 8192
        {"name": "layer-32", "kind": "layer", "shape": "llama3-8b", "rows": 32, "low": 512, "high": 8192, "mix": 3},
        # a full server
        {"name": "layer-128", "kind": "layer", "shape": "llama3-8b", "rows": 128, "low": 128, "high": 8192, "mix": 4},
        # one chat on a small model, a burst of eight tokens
        {"name": "tokens-tinyllama", "kind": "tokens", "sequences": 1, "layers": 22, "context": 2048, "new": 8},
        # one long document in the compressed cache
        {"name": "compressed-32k", "kind": "compressed", "sequences": 1, "context": 32768},
        # four ragged prompts in one packed attention call
        {"name": "prefill-packed", "kind": "prefill", "heads": 32, "kv_heads": 8, "dim": 128, "sequences": 4, "low": 509, "high": 2048,
         "past": 0, "mix": 5},
        # a long prompt of each model family
        {"name": "prompt-llama", "kind": "prompt", "model": "llama", "size": "llama3-8b-sized", "sequences": 1, "tokens": 2000},
        {"name": "prompt-lamutar", "kind": "prompt", "model": "lamutar", "size": "tinyllama-sized", "sequences": 1, "tokens": 2048},
        {"name": "prompt-sidalorn", "kind": "prompt", "model": "sidalorn", "size": "llama3-8b-sized", "sequences": 3, "tokens": 2048},
        # a batch of chat requests: ragged prompts, then a burst of tokens for all of them
        {"name": "requests-lamutar", "kind": "requests", "model": "lamutar", "size": "llama3-8b-sized", "sequences": 16, "tokens": 1500,
         "new": 24},
        {"name": "requests-sidalorn", "kind": "requests", "model": "sidalorn", "size": "tinyllama-sized", "sequences": 32, "tokens": 1800,
         "new": 16},
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("layer", "layer", "tokens", "compressed", "prefill", "prompt", "prompt", "requests"))
    if kind == "layer":
        high = _log(rng, 300, 8192)
        return {"kind": kind, "shape": rng.choice(sorted(LAYERS)), "rows": _log(rng, 1, 128), "low": max(1, high // _log(rng, 1, 16)),
                "high": high, "mix": rng.randrange(1 << 20)}
    if kind == "tokens":
        return {"kind": kind, "sequences": _log(rng, 1, 6), "layers": rng.randint(4, 22), "context": _log(rng, 40, 4000),
                "new": rng.randint(1, 8)}
    if kind == "compressed":
        return {"kind": kind, "sequences": _log(rng, 1, 4), "context": _log(rng, 1000, 32768)}
    if kind == "prefill":
        heads, kv_heads, dim = rng.choice(((32, 8, 128), (32, 4, 64), (16, 2, 128)))
        high = _log(rng, 40, 2048)
        return {"kind": kind, "heads": heads, "kv_heads": kv_heads, "dim": dim, "sequences": rng.randint(1, 4),
                "low": max(1, high // _log(rng, 1, 8)), "high": high, "past": rng.choice((0, 0, rng.randint(1, 1000))),
                "mix": rng.randrange(1 << 20)}
    model = rng.choice(("llama", "lamutar", "sidalorn")) if kind == "prompt" else rng.choice(("lamutar", "sidalorn"))
    size = rng.choice(sorted(STACKS))
    if kind == "prompt":
        sequences = _log(rng, 1, 6)
        return {"kind": kind, "model": model, "size": size, "sequences": sequences, "tokens": max(sequences, _log(rng, 16, 2048))}
    sequences = _log(rng, 1, 32)
    return {"kind": kind, "model": model, "size": size, "sequences": sequences, "tokens": sequences * _log(rng, 4, 56),
            "new": rng.randint(4, 16)}


# --------------------------------------------------------------------------------------------------------- the program
def _package():
    """The package's folder carries a hyphen, so it is loaded by path."""
    if "m40_llm_b200" not in sys.modules:
        folder = os.path.join(_ROOT, "m40-llm_b200")
        spec = importlib.util.spec_from_file_location("m40_llm_b200", os.path.join(folder, "__init__.py"),
                                                      submodule_search_locations=[folder])
        module = importlib.util.module_from_spec(spec)
        sys.modules["m40_llm_b200"] = module
        spec.loader.exec_module(module)
    return sys.modules["m40_llm_b200"]


_native = None
_stage = None


def _nat():
    """One context per program."""
    global _native
    if _native is None:
        pkg = _package()
        torch.zeros(1, device=_DEV)
        _native = pkg.native.Native(pkg.native.lib(), 0)
    return _native


def _check(rc):
    if rc != 0:
        raise RuntimeError(f"call failed: {rc}")


class State:
    """What a program holds: tensors, a cache, a model. Gives the library's objects back when it goes."""

    def __init__(self, case):
        self.case, self.kv, self.model, self.t = case, None, None, {}

    def __del__(self):
        torch.cuda.synchronize()
        if self.model is not None:
            self.model.close()
        if self.kv is not None:
            _native.lib.m40llm_kvcache_destroy(self.kv)


def _gen(seed, *tags):
    g = torch.Generator(device=_DEV)
    g.manual_seed(hash((int(seed),) + tags) & 0x7FFFFFFFFFFF)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=_DEV)


def _matrix(g, n, k, dtype, gain=1.0):
    out = torch.empty(n, k, dtype=dtype, device=_DEV)
    for i in range(0, n, 16384):
        out[i:i + 16384] = _randn(g, min(16384, n - i), k) * (gain / k ** 0.5)
    return out


def _lengths(case):
    """The sequences' lengths: part of the case, not of the seed."""
    r = random.Random(case["mix"])
    n = case["rows"] if case["kind"] == "layer" else case["sequences"]
    return [r.randint(case["low"], case["high"]) for _ in range(n)]


def _portions(case):
    """Lengths of the prompts of a step, `tokens` in all."""
    n, total = case["sequences"], case["tokens"]
    r = random.Random(1000 * n + total)
    parts = [r.uniform(0.4, 1.6) for _ in range(n)]
    lens = [max(1, int(total * p / sum(parts))) for p in parts]
    lens[-1] = max(1, total - sum(lens[:-1]))
    return lens


def _prompts(case, seed):
    r = np.random.default_rng(seed)
    return [r.integers(0, VOCAB, n).astype(np.uint32) for n in _portions(case)]


def _cached(seed, slot, tokens, heads, dim):
    """Keys and values of a sequence that is already in the cache."""
    g = _gen(seed, 7, slot)
    return _randn(g, tokens, heads, dim).half(), _randn(g, tokens, heads, dim).half()


def _fill(kv, slot, k, v, final_len):
    """Loads a sequence's keys and values from (pinned) host memory."""
    global _stage
    if _stage is None or _stage.numel() < 2 * k.numel():
        _stage = torch.empty(max(2 * k.numel(), 1 << 24), dtype=torch.float16, pin_memory=True)
    hk, hv = _stage[:k.numel()], _stage[k.numel():2 * k.numel()]
    hk.copy_(k.reshape(-1))
    hv.copy_(v.reshape(-1))
    nat = _nat()
    _check(nat.lib.m40llm_kvcache_debug_write_range(nat.ctx, kv, slot, 0, k.shape[0], hk.data_ptr(), hv.data_ptr(), final_len))


def _q80(w):
    """Rows of Q8_0 blocks: an f16 scale, then 32 signed bytes."""
    b = w.reshape(w.shape[0], -1, 32)
    d = (b.abs().amax(-1, keepdim=True) / 127.0)
    q = torch.where(d > 0, torch.round(b / d), torch.zeros_like(b)).to(torch.int8)
    return torch.cat([d.half().view(torch.uint8), q.view(torch.uint8)], -1).reshape(w.shape[0], -1).contiguous()


def _q80_f64(q):
    b = q.reshape(q.shape[0], -1, 34)
    d = b[:, :, :2].contiguous().view(torch.float16).to(F64)
    return (d * b[:, :, 2:].contiguous().view(torch.int8).to(F64)).reshape(q.shape[0], -1)


def _llama_layer(g, shape):
    H, qh, kvh, hd, F, q80, _, _, bias = shape
    w = {"wq": _matrix(g, qh * hd, H, torch.float16), "wk": _matrix(g, kvh * hd, H, torch.float16),
         "wv": _matrix(g, kvh * hd, H, torch.float16), "wo": _matrix(g, H, qh * hd, torch.float16)}
    for n, a, b in (("wg", F, H), ("wu", F, H), ("wd", H, F)):
        w[n] = _q80(_matrix(g, a, b, torch.float32)) if q80 else _matrix(g, a, b, torch.float16)
    for n in ("attn_norm", "ffn_norm"):
        w[n] = 1.0 + 0.05 * _randn(g, H)
    if bias:
        for n, a in (("bq", qh * hd), ("bk", kvh * hd), ("bv", kvh * hd)):
            w[n] = 0.1 * _randn(g, a)
    return w


def _tables(g, width, dtype):
    """Embeddings, and an output matrix that is sure of its tokens as a trained one is: each token's row of it is near the
    embedding of one other token, its usual predecessor."""
    e = _randn(g, VOCAB, width).to(dtype)
    order = torch.randperm(VOCAB, generator=g, device=_DEV)
    head = ((e[order].float() + 0.1 * _randn(g, VOCAB, width)) / width ** 0.5).to(dtype)
    return e, head


def _llama_shape(case):
    if case["kind"] == "tokens":
        return LAYERS["tinyllama"], case["layers"]
    W, F, qh, kvh, hd, _, _, _, n = STACKS[case["size"]]
    return (W, qh, kvh, hd, F, False, 0, 1e4, False), n


def _llama_weights(case, seed):
    shape, n = _llama_shape(case)
    g = _gen(seed, 1)
    layers = [_llama_layer(g, shape) for _ in range(n)]
    e, head = _tables(g, shape[0], torch.float16)
    return shape, layers, e, head, 1.0 + 0.05 * _randn(g, shape[0])


def _decode_model(s, seed, sequences, max_len, max_rows):
    host, nat = _package().host, _nat()
    shape, layers, e, head, norm = _llama_weights(s.case, seed)
    H, qh, kvh, hd, F, _, layout, base, _ = shape
    s.t["weights"] = (layers, e, head, norm)
    packed = []
    for w in layers:
        p = host.Weights()
        for n, t in w.items():
            setattr(p, n, t.data_ptr())
        packed.append(p)
    s.kv = nat.kv_dense(max_len, sequences * len(layers), kvh, hd)
    s.model = host.DecodeModel(nat.ctx, host.LayerCfg(H, qh, kvh, hd, F, layout, EPS, base, 1.0), packed,
                               host.ModelHead(e.data_ptr(), norm.data_ptr(), head.data_ptr(), VOCAB), s.kv, sequences, max_rows=max_rows)


# -------------------------------------------------------------------------------------------------------- layer stacks
def _config(case):
    W, F, qh, kvh, hd, dh, dd, _, n = STACKS[case["size"]]
    dense = {"kind": "dense", "ff": F}
    if case["model"] == "lamutar":
        att = {"type": "attention", "mlp": dense,
               "mixer": {"heads": qh, "kv_heads": kvh, "dim": hd, "vdim": hd, "scale": hd ** -0.5,
                         "rot": {"base": 1e6, "dims": hd // 2, "scaling": {"factor": 8.0, "fast": 32.0, "original": 4096, "slow": 1.0}}}}
        delta = {"type": "general_delta", "mlp": dense, "mixer": {"heads": dh, "dim": dd}}
        return {"architecture": "Lamutar", "width": W, "vocab": VOCAB, "norm": {"eps": EPS}, "logit_softcap": 30.0,
                "layers": [att if i % 4 == 0 else delta for i in range(n)]}
    H, D, R, B, E, I, G, keep, top, FE, FS = SIDALORN[case["size"]]
    moe = {"kind": "moe", "expert": {"ff": FE}, "shared": {"ff": FS},
           "router": {"experts": E, "identity": I, "top": top, "scale": 2.5, "groups": {"count": G, "keep": keep}}}
    lat = {"type": "latent_attention", "mixer": {"heads": H, "dim": D, "vdim": D, "kv_rank": R, "scale": D ** -0.5}}
    rec = {"type": "rglru", "mixer": {"width": W, "blocks": B, "conv": 4}}
    cycle = [{**lat, "mlp": dense}, {**rec, "mlp": moe}, {**rec, "mlp": dense}, {**lat, "mlp": moe}]
    return {"architecture": "Sidalorn", "width": W, "vocab": VOCAB, "norm": {"eps": EPS, "groups": 8}, "canon": {"taps": 4},
            "layers": [cycle[i % 4] for i in range(n)]}


def _tensors(case, seed):
    """The model's named tensors, as a file of it would hold them (bf16), on the GPU."""
    cfg, g, out = _config(case), _gen(seed, 2), {}
    W = cfg["width"]

    def mat(name, n, k, gain=1.0):
        out[name] = _matrix(g, n, k, torch.bfloat16, gain)

    def vec(name, value):
        out[name] = value.bfloat16()

    def uniform(low, high, n):
        return low + (high - low) * torch.rand(n, generator=g, device=_DEV)

    def norm(name):
        vec(name, 1.0 + 0.1 * _randn(g, W))
        if cfg["architecture"] == "Lamutar":
            vec(name + ".b", 0.1 * _randn(g, W))
            vec(name + ".alpha", torch.full((1,), 0.75, device=_DEV))

    out["embed"], out["head"] = _tables(g, W, torch.bfloat16)
    norm("final.norm")
    for i, ly in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", ly["mixer"], ly["mlp"]
        x = p + "mix."
        norm(p + "norm1")
        norm(p + "norm2")
        if ly["type"] == "attention":
            norm(p + "norm1b")
            H, G, D, V = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            for n, rows in (("q", H * D), ("k", G * D), ("v", G * V), ("g", H)):
                mat(x + n, rows, W)
            vec(x + "q.norm", 1.0 + 0.1 * _randn(g, H * D))
            vec(x + "k.norm", 1.0 + 0.1 * _randn(g, G * D))
            mat(x + "o", W, H * V)
        elif ly["type"] == "general_delta":
            norm(p + "norm1b")
            HD, R = m["heads"] * m["dim"], STACKS[case["size"]][7]
            for n in ("r", "k", "v", "g", "a"):
                mat(x + n, HD, W)
            mat(x + "w1", R, W)
            mat(x + "w2", HD, R)
            vec(x + "w0", uniform(-4.0, 2.0, HD))
            vec(x + "a.b", 0.3 * _randn(g, HD))
            vec(x + "norm", 1.0 + 0.1 * _randn(g, HD))
            mat(x + "o", W, HD)
        elif ly["type"] == "latent_attention":
            H, D, V, R = m["heads"], m["dim"], m["vdim"], m["kv_rank"]
            vec(p + "canon1", 0.3 * _randn(g, W, cfg["canon"]["taps"]))
            mat(x + "q", H * D, W)
            mat(x + "dkv", R, W)
            vec(x + "dkv.norm", 1.0 + 0.1 * _randn(g, R))
            mat(x + "uk", H * D, R)
            mat(x + "uv", H * V, R)
            vec(x + "sink", uniform(-1.0, 3.0, H))
            mat(x + "o", W, H * V)
        else:
            D, B = m["width"], m["blocks"]
            vec(p + "canon1", 0.3 * _randn(g, W, cfg["canon"]["taps"]))
            for n in "yx":
                mat(x + n, D, W)
                vec(x + n + ".b", 0.1 * _randn(g, D))
            vec(x + "conv", 0.5 * _randn(g, D, m["conv"]))
            vec(x + "conv.b", 0.1 * _randn(g, D))
            for n in ("ra", "ri"):
                out[x + n] = _matrix(g, D, D // B, torch.bfloat16).reshape(B, D // B, D // B)
                vec(x + n + ".b", 0.3 * _randn(g, B, D // B))
            vec(x + "lam", uniform(-9.0, 0.5, D))
            mat(x + "o", W, D)
        f = p + "mlp."
        if cfg["architecture"] == "Lamutar":
            norm(p + "norm2b")
            for n, a, b in (("gate", mlp["ff"], W), ("up", mlp["ff"], W), ("down", W, mlp["ff"])):
                mat(f + n, a, b)
        elif mlp["kind"] == "dense":
            mat(f + "up", mlp["ff"], W)
            mat(f + "down", W, mlp["ff"])
            vec(f + "act", torch.tensor([0.6, 0.3, 0.2, 0.05], device=_DEV))
        else:
            r, F, S = mlp["router"], mlp["expert"]["ff"], mlp["shared"]["ff"]
            for e in range(r["experts"]):
                mat(f"{f}e{e}.up", F, W)
                mat(f"{f}e{e}.down", W, F)
            mat(f + "router", r["experts"] + r["identity"], W)
            vec(f + "correction", 0.002 * _randn(g, r["experts"] + r["identity"]))
            mat(f + "shared.up", S, W)
            mat(f + "shared.down", W, S)
    return out


def _stack_model(s, seed, sequences, max_len, max_rows):
    pkg, nat, case = _package(), _nat(), s.case
    from m40_llm_b200 import models
    from m40_llm_b200.models.stack import StackWeights

    class OnGpu(StackWeights):
        """The builder's view of tensors that are on the GPU already (a loader's view reads a file and uploads it)."""

        def __init__(self, tensors):
            super().__init__(nat, None)
            self.tensors, self.keep = tensors, []

        def _own(self, key, make):
            if key not in self._mat:
                self.keep.append(make())
                self._mat[key] = self.keep[-1].data_ptr()
            return self._mat[key]

        def shape(self, name):
            return tuple(self.tensors[name].shape)

        def matrix(self, *names, shapes=None, rows=0):
            def make():
                parts = [self.tensors.pop(n) for n in names]
                missing = rows - sum(len(t) for t in parts)
                if missing > 0:
                    parts.append(parts[0].new_zeros(missing, *parts[0].shape[1:]))
                return torch.cat(parts) if len(parts) > 1 else parts[0]
            return self._own(names, make)

        def blocks_transposed(self, name, shape, blocks):
            return self._own((name, "transposed"), lambda: self.first[name].reshape(blocks, -1, shape[1]).transpose(1, 2).contiguous())

        def vectors(self, names, sizes, total):
            def make():
                out = torch.zeros(total, device=_DEV)
                v = torch.cat([self.tensors[n].float().reshape(-1) for n in names])
                out[:len(v)] = v
                return out
            return self._own(("vectors", *names), make)

        def vector(self, name, size, row=None):
            return self._own(("vector", name), lambda: self.tensors[name].float().reshape(-1).contiguous())

        def table(self, values):
            return self._own(("table", values.tobytes()), lambda: torch.from_numpy(np.ascontiguousarray(values, np.float64)).to(_DEV))

        def dynamic_tanh(self, name, size):
            alpha = float(self.tensors[name + ".alpha"][0])
            return pkg.native.Norm(pkg.native.NORM_DYT, 0.0, alpha, self.vector(name, size), self.vector(name + ".b", size))

    w = OnGpu(_tensors(case, seed))
    w.first = {n: t for n, t in w.tensors.items() if n.endswith(".uk")}
    s.model = models.read_config(_config(case)).build(nat, w, sequences=sequences, max_len=max_len, max_rows=max_rows)
    s.t["weights"] = w.keep


# ----------------------------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    nat, s = _nat(), State(case)
    kind = case["kind"]
    if kind == "layer":
        H, qh, kvh, hd, F, _, _, _, _ = LAYERS[case["shape"]]
        lens, rows = _lengths(case), case["rows"]
        s.kv = nat.kv_dense(max(lens) + 1, rows, kvh, hd)
        for r, n in enumerate(lens):
            if n > 1:
                _fill(s.kv, r, *_cached(seed, r, n - 1, kvh, hd), n - 1)
        t = s.t = {**_llama_layer(_gen(seed, 1), LAYERS[case["shape"]]), "x": _randn(_gen(seed, 3), rows, H)}
        for n, width in (("q", qh * hd), ("att", qh * hd), ("x1", H), ("hid", F), ("out", H)):
            t[n] = torch.empty(rows, width, device=_DEV)
        t["ids"] = torch.arange(rows, dtype=torch.int32, device=_DEV)
        t["lens"] = torch.tensor(lens, dtype=torch.int32, device=_DEV)
        t["pos"] = t["lens"] - 1
    elif kind == "tokens":
        n, layers, ctx = case["sequences"], case["layers"], case["context"]
        _decode_model(s, seed, n, ctx + case["new"] + 1, 0)
        for slot in range(n * layers):
            _fill(s.kv, slot, *_cached(seed, slot, ctx - slot // layers, 4, 64), ctx - slot // layers)
        s.t["first"] = np.random.default_rng(seed).integers(0, VOCAB, n).astype(np.uint32)
        s.t["positions"] = np.array([ctx - i for i in range(n)], np.uint32)
    elif kind == "compressed":
        qh, kvh, hd, recent, block, top = COMPRESSED
        n, ctx = case["sequences"], case["context"]
        s.kv = nat.kv_compressed(ctx, n, kvh, hd, recent, block, top)
        for i in range(n):
            k, v = _cached(seed, i, ctx - 97 * i, kvh, hd)
            _fill(s.kv, i, k, v, len(k))
        s.t = {"q": _randn(_gen(seed, 3), n, qh * hd), "out": torch.empty(n, qh * hd, device=_DEV)}
    elif kind == "prefill":
        lens = np.array(_lengths(case), np.int64)
        kv_lens = lens + case["past"]
        g, H, G, D = _gen(seed, 3), case["heads"], case["kv_heads"], case["dim"]
        s.t = {"q": _randn(g, int(lens.sum()), H, D), "k": _randn(g, int(kv_lens.sum()), G, D), "v": _randn(g, int(kv_lens.sum()), G, D)}
        s.t["out"] = torch.empty_like(s.t["q"])
        for n, a in (("q_off", np.cumsum(lens) - lens), ("kv_off", np.cumsum(kv_lens) - kv_lens), ("q_len", lens), ("kv_len", kv_lens)):
            s.t[n] = torch.tensor(a, dtype=torch.int32, device=_DEV)
    else:
        n, new = case["sequences"], case.get("new", 0)
        longest = max(_portions(case)) + new + 1
        if case["model"] == "llama":  # its projections take 256 rows a call
            _decode_model(s, seed, n, longest, 256)
        else:
            _stack_model(s, seed, n, longest, 2048)
        s.t["prompts"] = _prompts(case, seed)
        s.t["want"] = np.cumsum([len(p) for p in s.t["prompts"]]) - 1
    torch.cuda.synchronize()
    return s


def run(s):
    case, t, nat = s.case, s.t, _native
    kind, L, ctx = case["kind"], nat.lib, nat.ctx
    if kind == "layer":
        H, qh, kvh, hd, F, q80, layout, base, _ = LAYERS[case["shape"]]
        p = lambda n: t[n].data_ptr() if n in t else None  # noqa: E731
        _check(L.m40llm_qkv_rope_append_attention_async(
            ctx, s.kv, p("x"), p("attn_norm"), 1, EPS, p("wq"), p("wk"), p("wv"), p("bq"), p("bk"), p("bv"), p("ids"), p("pos"),
            p("lens"), case["rows"], H, qh, base, 1.0, layout, p("q"), p("att")))
        _check(L.m40llm_attn_out_ffn_async(ctx, p("att"), p("wo"), p("x"), p("ffn_norm"), 1, EPS, p("wg"), p("wu"), p("wd"),
                                           1 if q80 else 0, p("x1"), p("hid"), p("out"), case["rows"], H, qh * hd, F))
        return {"q": t["q"], "attention": t["att"], "out": t["out"]}
    if kind == "tokens":
        s.model.begin(t["first"], t["positions"])
        ids, logits = s.model.generate(case["new"], want_logits=True)
        return {"ids": ids, "logits": logits}
    if kind == "compressed":
        qh, kvh, hd, recent, block, top = COMPRESSED
        for i in range(case["sequences"]):
            _check(L.m40llm_attention_last_token_f32_gqa_block_select_exact_fp16_k_q4_v_old_direct_async(
                ctx, s.kv, i, t["q"][i].data_ptr(), qh, case["context"] - 97 * i, recent, block, top, t["out"][i].data_ptr()))
        return t["out"]
    if kind == "prefill":
        _check(L.m40llm_attention_prefill_f32_gqa_varlen_async(
            ctx, t["q"].data_ptr(), t["k"].data_ptr(), t["v"].data_ptr(), t["q_off"].data_ptr(), t["kv_off"].data_ptr(),
            t["q_len"].data_ptr(), t["kv_len"].data_ptr(), case["sequences"], case["heads"], case["kv_heads"], case["dim"],
            t["out"].data_ptr()))
        return t["out"]
    m = s.model
    slots = [m.acquire() for _ in t["prompts"]]
    entries = list(zip(slots, t["prompts"]))
    if kind == "prompt":
        got = m.step(entries, t["want"], want_next=True)
        out = {"next": got["next"], "logits": got["logits"]}
    else:
        first = m.step(entries, t["want"], want_logits=False, want_next=True)["next"]
        m.begin_sequences(slots, first)
        ids, logits = m.generate(case["new"], want_logits=True)
        out = {"first": first, "ids": ids, "logits": logits}
    for slot in slots:
        m.release(slot)
    return out


# ---------------------------------------------------------------------------------------------------------------- work
def _pairs(lens, past=0):
    return sum(n * (n + 1) // 2 + n * past for n in lens)


def _stack_work(case):
    """(bytes of the weights of the layers that every pass reads, of one expert, expert layers, multiply-adds per token, cache bytes per
    token of context and attention multiply-adds per pair, recurrent state bytes per sequence)."""
    if case["kind"] == "tokens" or case.get("model") == "llama":
        (H, qh, kvh, hd, F, _, _, _, _), n = _llama_shape(case)
        per = (2 * qh + 2 * kvh) * hd * H + 3 * H * F
        return 2.0 * per * n, 0.0, 0, float(per * n), 4.0 * kvh * hd * n, 2.0 * hd * qh * n, 0.0
    W, F, qh, kvh, hd, dh, dd, rank, n = STACKS[case["size"]]
    fixed = experts = moe_layers = macs = cache = att = state = 0.0
    for ly in _config(case)["layers"]:
        m, mlp = ly["mixer"], ly["mlp"]
        if ly["type"] == "attention":
            p = (2 * qh + 2 * kvh) * hd * W
            cache, att = cache + 4.0 * kvh * hd, att + 2.0 * hd * qh
        elif ly["type"] == "general_delta":
            p = 6 * dh * dd * W + rank * (W + dh * dd)
            state, macs = state + 8.0 * dh * dd * dd, macs + 4.0 * dh * dd * dd
        elif ly["type"] == "latent_attention":
            H, D, R = m["heads"], m["dim"], m["kv_rank"]
            p = 2 * H * D * W + R * W + 2 * H * D * R
            cache, att = cache + 2.0 * R, att + 2.0 * H * D
        else:
            p = 3 * W * W + 2 * W * W // m["blocks"]
            state = state + 8.0 * W * 5
        if mlp["kind"] == "moe":
            r, FE = mlp["router"], mlp["expert"]["ff"]
            p += (r["experts"] + r["identity"]) * W + 2 * mlp["shared"]["ff"] * W
            macs += r["top"] * 2.0 * FE * W
            experts, moe_layers = 4.0 * FE * W, moe_layers + 1
        else:
            p += (3 if case["model"] == "lamutar" else 2) * F * W
        fixed, macs = fixed + 2.0 * p, macs + p
    return fixed, experts, moe_layers, macs, cache, att, state


def work(case):
    kind = case["kind"]
    if kind == "layer":
        H, qh, kvh, hd, F, q80, _, _, _ = LAYERS[case["shape"]]
        ctx, rows = sum(_lengths(case)), case["rows"]
        att, ffn = (2 * qh + 2 * kvh) * hd * H, 3 * H * F
        return {"bytes": 2.0 * att + ffn * (34 / 32 if q80 else 2) + 4.0 * ctx * kvh * hd + 4.0 * rows * (2 * H + 2 * qh * hd),
                "flops": 2.0 * rows * (att + ffn) + 4.0 * hd * qh * ctx}
    if kind == "compressed":
        qh, kvh, hd, recent, block, top = COMPRESSED
        out = {"bytes": 0.0, "flops": 0.0}
        for i in range(case["sequences"]):
            n = case["context"] - 97 * i
            old = max(0, n - recent)
            picked = min(old, top * block)
            out["bytes"] += 2.0 * old * kvh * hd + qh * picked * (hd // 2 + 4) + 4.0 * min(n, recent) * kvh * hd + 8.0 * qh * hd
            out["flops"] += 2.0 * qh * hd * old / block + 4.0 * qh * hd * (picked + min(n, recent))
        return out
    if kind == "prefill":
        lens = _lengths(case)
        q, kv = sum(lens), sum(lens) + case["past"] * len(lens)
        return {"bytes": 8.0 * case["dim"] * (q * case["heads"] + kv * case["kv_heads"]),
                "flops": 4.0 * case["dim"] * case["heads"] * _pairs(lens, case["past"])}
    fixed, expert, moe_layers, macs, cache, att, state = _stack_work(case)
    n = case["sequences"]
    W = LAYERS["tinyllama"][0] if kind == "tokens" else STACKS[case["size"]][0]
    head = 2.0 * VOCAB * W

    def one(rows, pairs, context, wanted):  # a pass over the whole model
        touched = 60 * (1.0 - (1.0 - 6 / 64) ** rows) if expert else 0.0
        return (fixed + expert * moe_layers * touched + head + cache * context + state * n + 4.0 * wanted * VOCAB + 2.0 * rows * W,
                2.0 * rows * macs + 2.0 * att * pairs + 2.0 * VOCAB * W * wanted)

    passes = []
    lens = [case["context"]] * n if kind == "tokens" else _portions(case)
    if kind != "tokens":
        passes.append(one(sum(lens), _pairs(lens), sum(lens), n))
    for t in range(case.get("new", 0)):
        context = sum(lens) + n * (t + 1)
        passes.append(one(n, context, context, n))
    return {"bytes": sum(p[0] for p in passes), "flops": sum(p[1] for p in passes)}


def tolerance(case):
    """About four times the distance to exact(), which f16 caches and probabilities make (1.7e-4 for decode attention, 3.2e-4 for prompts).
    Sidalorn: now and then two experts are as good as equal and the other one is chosen (up to 7.5e-3). A token may differ where
    two logits are as good as equal."""
    if case.get("model") == "sidalorn":
        return {"rel": 0.025, "max": 0.99, "differ": 0.005}
    return {"rel": 1.3e-3, "max": 0.05, "differ": 0.005}


# ------------------------------------------------------------------------------------------------- the same in 64 bits
def _rms(x, w, groups=1):
    p = x.reshape(*x.shape[:-1], groups, -1)
    return (p * torch.rsqrt(p.square().mean(-1, keepdim=True) + EPS)).reshape(x.shape) * w.to(F64)


def _lin(x, w):
    return x @ w.to(F64).T


def _turn(x, pos, freqs, layout, amp=1.0, sign=1.0):
    """x [T, heads, d]: pairs turn by sign * pos * freqs; layout 0: neighbours, 1: the halves of the first 2 len(freqs)."""
    a = sign * pos.to(F64)[:, None, None] * freqs
    c, s, n = torch.cos(a) * amp, torch.sin(a) * amp, len(freqs)
    if layout == 0:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, u * s + v * c], -1).reshape(x.shape)
    u, v = x[..., :n], x[..., n:2 * n]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * n:]], -1)


def _attend(q, K, V, scale, first, sink=None):
    """q [T, heads, d] at positions first, first + 1, ... over K, V [n, kv heads, d]; causal."""
    T, H, _ = q.shape
    G = K.shape[1]
    out = torch.empty(T, H, V.shape[2], dtype=F64, device=q.device)
    mask = torch.arange(K.shape[0], device=q.device)[None, :] > (first + torch.arange(T, device=q.device))[:, None]
    for h in range(H):
        z = (q[:, h] @ K[:, h * G // H].to(F64).T * scale).masked_fill(mask, -math.inf)
        if sink is not None:
            z = torch.cat([z, sink[h].to(F64).expand(T, 1)], 1)
        p = torch.softmax(z, -1)[:, :K.shape[0]]
        out[:, h] = p @ V[:, h * G // H].to(F64)
    return out


def _freqs(base, dims):
    return float(base) ** (-torch.arange(0, dims, 2, dtype=F64, device=_DEV) / dims)


def _ffn(x, w, q80):
    up = _q80_f64 if q80 else (lambda a: a.to(F64))
    z = x @ up(w["wg"]).T
    return (z * torch.sigmoid(z) * (x @ up(w["wu"]).T)) @ up(w["wd"]).T


def _llama_step(w, shape, x, K, V, first):
    """One layer for consecutive tokens of one sequence; K, V hold the earlier ones. Returns (q, attention, out, K, V)."""
    H, qh, kvh, hd, F, q80, layout, base, bias = shape
    h = _rms(x, w["attn_norm"])
    pos = torch.arange(first, first + len(x), device=x.device)
    q, k, v = (_lin(h, w["w" + n]) + (w["b" + n].to(F64) if bias else 0.0) for n in "qkv")
    f = _freqs(base, hd)
    q = _turn(q.reshape(-1, qh, hd), pos, f, layout)
    K = torch.cat([K.to(F64), _turn(k.reshape(-1, kvh, hd), pos, f, layout)])
    V = torch.cat([V.to(F64), v.reshape(-1, kvh, hd)])
    att = _attend(q, K, V, hd ** -0.5, first).reshape(len(x), -1)
    x1 = x + _lin(att, w["wo"])
    return q.reshape(len(x), -1), att, x1 + _ffn(_rms(x1, w["ffn_norm"]), w, q80), K, V


class _Llama:
    def __init__(self, case, seed):
        self.shape, self.layers, self.e, self.head, self.norm = _llama_weights(case, seed)

    def fresh(self):
        none = torch.empty(0, self.shape[2], self.shape[3], dtype=F64, device=_DEV)
        return [[none, none] for _ in self.layers]

    def step(self, tokens, state, first):
        x = self.e[torch.as_tensor(tokens.astype(np.int64), device=_DEV)].to(F64)
        for w, st in zip(self.layers, state):
            _, _, x, st[0], st[1] = _llama_step(w, self.shape, x, st[0], st[1], first)
        return _lin(_rms(x[-1:], self.norm), self.head)[0]


def _gelu_tanh(z):
    return torch.nn.functional.gelu(z, approximate="tanh")


def _conv(x, past, w):
    seq = torch.cat([past, x])
    taps = w.shape[1]
    return sum(w[:, j].to(F64) * seq[j:j + len(x)] for j in range(taps)), seq[len(seq) - taps + 1:]


class _Stack:
    """Lamutar and Sidalorn, one sequence at a time."""

    def __init__(self, case, seed):
        self.cfg, self.w = _config(case), _tensors(case, seed)
        self.lamutar = case["model"] == "lamutar"

    def fresh(self):
        z = lambda *shape: torch.zeros(*shape, dtype=F64, device=_DEV)  # noqa: E731
        state = []
        for ly in self.cfg["layers"]:
            m = ly["mixer"]
            st = {"canon": None if self.lamutar else z(self.cfg["canon"]["taps"] - 1, self.cfg["width"])}
            if ly["type"] == "attention":
                st["K"], st["V"] = z(0, m["kv_heads"], m["dim"]), z(0, m["kv_heads"], m["vdim"])
            elif ly["type"] == "general_delta":
                st["S"] = z(m["heads"], m["dim"], m["dim"])
            elif ly["type"] == "latent_attention":
                st["C"] = z(0, m["kv_rank"])
            else:
                st["S"], st["past"] = z(m["width"]), z(m["conv"] - 1, m["width"])
            state.append(st)
        return state

    def norm(self, name, x):
        w = self.w
        if self.lamutar:
            return torch.tanh(w[name + ".alpha"].to(F64) * x) * w[name].to(F64) + w[name + ".b"].to(F64)
        return _rms(x, w[name], self.cfg["norm"]["groups"])

    def step(self, tokens, state, first):
        x = self.w["embed"][torch.as_tensor(tokens.astype(np.int64), device=_DEV)].to(F64)
        pos = torch.arange(first, first + len(x), device=_DEV)
        for i, (ly, st) in enumerate(zip(self.cfg["layers"], state)):
            p, m = f"l{i}.", ly["mixer"]
            mix = lambda n: self.w[f"l{i}.mix.{n}"]  # noqa: B023,E731
            if self.lamutar:
                y = getattr(self, "_" + ly["type"])(self.norm(p + "norm1", x), mix, m, st, pos, first)
                x = x + self.norm(p + "norm1b", _lin(y, mix("o")))
                h, f = self.norm(p + "norm2", x), p + "mlp."
                y = _lin(_gelu_tanh(_lin(h, self.w[f + "gate"])) * _lin(h, self.w[f + "up"]), self.w[f + "down"])
                x = x + self.norm(p + "norm2b", y)
            else:
                c, st["canon"] = _conv(x, st["canon"], self.w[p + "canon1"])
                y = getattr(self, "_" + ly["type"])(x + c, mix, m, st, pos, first)
                x = x + self.norm(p + "norm1", _lin(y, mix("o")))
                x = x + self.norm(p + "norm2", self._dense(x, p + "mlp.") if ly["mlp"]["kind"] == "dense" else
                                  self._moe(x, p + "mlp.", ly["mlp"]["router"]))
        z = _lin(self.norm("final.norm", x[-1:]), self.w["head"])[0]
        return 30.0 * torch.tanh(z / 30.0) if self.lamutar else z

    def _attention(self, h, w, m, st, pos, first):
        H, G, D, V, rot = m["heads"], m["kv_heads"], m["dim"], m["vdim"], m["rot"]
        n, sc = rot["dims"], rot["scaling"]
        f = _freqs(rot["base"], n)
        at = lambda turns: n * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))  # noqa: E731
        lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), n - 1)
        ramp = ((torch.arange(n // 2, dtype=F64, device=_DEV) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f, amp = f / sc["factor"] * ramp + f * (1 - ramp), 0.1 * math.log(sc["factor"]) + 1.0
        fv = _freqs(rot["base"], V)
        q = _rms(_lin(h, w("q")), w("q.norm")).reshape(-1, H, D)
        k = _rms(_lin(h, w("k")), w("k.norm")).reshape(-1, G, D)
        st["K"] = torch.cat([st["K"], _turn(k, pos, f, 1, amp)])
        st["V"] = torch.cat([st["V"], _turn(_lin(h, w("v")).reshape(-1, G, V), pos, fv, 1)])
        y = _turn(_attend(_turn(q, pos, f, 1, amp), st["K"], st["V"], m["scale"], first), pos, fv, 1, sign=-1.0)
        return (y * torch.sigmoid(_lin(h, w("g")))[:, :, None]).reshape(len(h), -1)

    def _general_delta(self, h, w, m, st, pos, first):
        shape = (len(h), m["heads"], m["dim"])
        r, k, v = (_lin(h, w(n)).reshape(shape) for n in "rkv")
        decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(_lin(torch.tanh(_lin(h, w("w1"))), w("w2")) + w("w0").to(F64))).reshape(shape)
        a = torch.sigmoid(_lin(h, w("a")) + w("a.b").to(F64)).reshape(shape)
        u = k / torch.sqrt(k.square().sum(-1, keepdim=True) + 1e-6)
        S, out, au = st["S"], [], a * u
        for t in range(len(h)):
            S = decay[t, :, :, None] * S + torch.baddbmm(k[t, :, :, None] * v[t, :, None, :], au[t, :, :, None],
                                                         torch.bmm(u[t, :, None, :], S), alpha=-1.0)
            out.append(torch.bmm(r[t, :, None, :], S)[:, 0])
        st["S"], o = S, torch.stack(out)
        o = o * torch.rsqrt(o.square().mean(-1, keepdim=True) + EPS)
        return o.reshape(len(h), -1) * w("norm").to(F64) * torch.sigmoid(_lin(h, w("g")))

    def _latent_attention(self, h, w, m, st, pos, first):
        H, D, V = m["heads"], m["dim"], m["vdim"]
        st["C"] = torch.cat([st["C"], _rms(_lin(h, w("dkv")), w("dkv.norm"))])
        K, Vs = _lin(st["C"], w("uk")).reshape(-1, H, D), _lin(st["C"], w("uv")).reshape(-1, H, V)
        return _attend(_lin(h, w("q")).reshape(-1, H, D), K, Vs, m["scale"], first, w("sink")).reshape(len(h), -1)

    def _rglru(self, h, w, m, st, pos, first):
        y = _gelu_tanh(_lin(h, w("y")) + w("y.b").to(F64))
        u, st["past"] = _conv(_lin(h, w("x")) + w("x.b").to(F64), st["past"], w("conv"))
        u = u + w("conv.b").to(F64)
        parts = u.reshape(len(u), m["blocks"], -1)
        gate = lambda n: torch.sigmoid(torch.einsum("tbi,boi->tbo", parts, w(n).to(F64)) + w(n + ".b").to(F64)).reshape(u.shape)  # noqa: E731
        log_a = -8.0 * gate("ra") * torch.nn.functional.softplus(w("lam").to(F64))
        a, inp = torch.exp(log_a), torch.sqrt(-torch.expm1(2 * log_a)) * gate("ri") * u
        S, out = st["S"], []
        for t in range(len(u)):
            S = a[t] * S + inp[t]
            out.append(S)
        st["S"] = S
        return torch.stack(out) * y

    def _dense(self, x, f):
        z = _lin(x, self.w[f + "up"])
        n = lambda v: v * torch.rsqrt(v.square().mean(-1, keepdim=True) + EPS)  # noqa: E731
        a, b, c, e = self.w[f + "act"].to(F64)
        return _lin(a * n(z) + b * n(z * z) + c * n(z ** 3) + e, self.w[f + "down"])

    def _moe(self, x, f, r):
        gelu = torch.nn.functional.gelu
        s = torch.softmax(_lin(x, self.w[f + "router"]), -1)
        choice = s + self.w[f + "correction"].to(F64)
        parts = choice.reshape(len(x), r["groups"]["count"], -1)
        best = parts.amax(-1).topk(r["groups"]["keep"], -1).indices
        keep = torch.zeros_like(parts[:, :, 0], dtype=torch.bool).scatter_(1, best, True)
        ids = parts.masked_fill(~keep[:, :, None], -math.inf).reshape(choice.shape).topk(r["top"], -1).indices
        g = s.gather(1, ids)
        g = g / (g.sum(-1, keepdim=True) + 1e-20) * r["scale"]
        out = _lin(gelu(_lin(x, self.w[f + "shared.up"])), self.w[f + "shared.down"])
        out = out + x * (g * (ids >= r["experts"])).sum(-1, keepdim=True)
        for e in range(r["experts"]):
            rows, at = torch.nonzero(ids == e, as_tuple=True)
            if len(rows):
                out[rows] += g[rows, at, None] * _lin(gelu(_lin(x[rows], self.w[f"{f}e{e}.up"])), self.w[f"{f}e{e}.down"])
        return out


def _q4_values(v):
    """What the cache's 4-bit values stand for: a scale per token and head, steps -7 .. 7, rounded through f16."""
    v = v.float()
    top = v.abs().amax(-1, keepdim=True)
    scale = top / torch.full_like(top, 7.0)  # a true division: steps half way between two values depend on it
    return ((v / scale).round().clamp(-7, 7) * scale).half()


def exact(case, seed):
    kind = case["kind"]
    if kind == "layer":
        shape = LAYERS[case["shape"]]
        w, x = _llama_layer(_gen(seed, 1), shape), _randn(_gen(seed, 3), case["rows"], shape[0]).to(F64)
        lens, out = _lengths(case), {"q": [], "attention": [], "out": []}
        plain = {n: (_q80_f64(t) if t.dtype == torch.uint8 else t.to(F64)) for n, t in w.items()}
        shape = shape[:5] + (False,) + shape[6:]
        for r, n in enumerate(lens):
            k, v = _cached(seed, r, n - 1, shape[2], shape[3]) if n > 1 else (torch.empty(0, shape[2], shape[3], device=_DEV),) * 2
            q, att, y, _, _ = _llama_step(plain, shape, x[r:r + 1], k, v, n - 1)
            for name, value in zip(out, (q, att, y)):
                out[name].append(value)
        return {name: torch.cat(rows) for name, rows in out.items()}
    if kind == "compressed":
        qh, kvh, hd, recent, block, top = COMPRESSED
        q, rows = _randn(_gen(seed, 3), case["sequences"], qh, hd).to(F64), []
        for i in range(case["sequences"]):
            n = case["context"] - 97 * i
            k, v = _cached(seed, i, n, kvh, hd)
            old = max(0, n - recent)
            v = torch.cat([_q4_values(v[:old]), v[old:]]).to(F64)
            for h in range(qh):
                kh, vh = k[:, h * kvh // qh].to(F64), v[:, h * kvh // qh]
                z = kh @ q[i, h] * hd ** -0.5
                seen = torch.arange(n, device=_DEV) >= old
                if old:
                    blocks = -(-old // block)
                    of = torch.arange(old, device=_DEV) // block
                    mean = torch.zeros(blocks, dtype=F64, device=_DEV).index_add_(0, of, z[:old]) / torch.bincount(of)
                    picked = torch.zeros(blocks, dtype=torch.bool, device=_DEV)
                    picked[mean.topk(min(top, blocks)).indices] = True
                    seen[:old] = picked[of]
                rows.append(torch.softmax(z.masked_fill(~seen, -math.inf), 0) @ vh)
        return torch.cat(rows).reshape(case["sequences"], qh * hd)
    if kind == "prefill":
        s, at, kat, out = prepare(case, seed), 0, 0, []
        for n in _lengths(case):
            k = slice(kat, kat + n + case["past"])
            out.append(_attend(s.t["q"][at:at + n].to(F64), s.t["k"][k], s.t["v"][k], case["dim"] ** -0.5, case["past"]))
            at, kat = at + n, k.stop
        return torch.cat(out)
    if kind == "tokens":
        m, n, layers, ctx = _Llama(case, seed), case["sequences"], case["layers"], case["context"]
        first = np.random.default_rng(seed).integers(0, VOCAB, n).astype(np.uint32)
        states = [[list(_cached(seed, i * layers + l, ctx - i, 4, 64)) for l in range(layers)] for i in range(n)]
        last, done, ids = list(first), [ctx - i for i in range(n)], []
    else:
        m = _Llama(case, seed) if case["model"] == "llama" else _Stack(case, seed)
        prompts = _prompts(case, seed)
        states = [m.fresh() for _ in prompts]
        logits = torch.stack([m.step(p, st, 0) for p, st in zip(prompts, states)])
        if kind == "prompt":
            return {"next": None, "logits": logits}
        last, done, ids = list(logits.argmax(-1).cpu().numpy()), [len(p) for p in prompts], []
    for _ in range(case["new"]):
        logits = torch.stack([m.step(np.array([t]), st, d) for t, st, d in zip(last, states, done)])
        last, done = list(logits.argmax(-1).cpu().numpy()), [d + 1 for d in done]
    out = {"ids": None, "logits": logits}
    return out if kind == "tokens" else {"first": None, **out}
