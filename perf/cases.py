"""What a user has this framework do: linears with int8 weights, linears on GGUF blocks, and steps of the three models.

    listed()            the cases that are measured
    draw(rng)           another case of the same ranges
    prepare(case, seed) what a program holds before the call: inputs, weights, recorded graphs, models with their sequences
    run(state)          one pass through the public entry points -> its outputs
    exact(case, seed)   what `run` returns, computed in 64 bits with plain torch
    work(case)          bytes and operations that a pass cannot do without
    tolerance(case)     how far another correct implementation may be off

Linears come as a stack of `layers` matrices of one shape, as the layers of a model bring them: few rows as one recorded graph
(a decode step), many rows call by call (a prompt).  Model cases take one period of each design: four layers, two of the Llama.
"""
import ctypes as C
import math
import zlib

import numpy as np
import torch

from peregrine_b200 import _lib
from peregrine_b200.gguf import GgufWeight
from peregrine_b200.runtime import GpuContext

DEV = "cuda"
GRAPH_ROWS = 128      # up to here a stack of linears is replayed as a graph


def listed():
    return [
        # the query projection of one token: the smallest call, where launches count
        {"name": "w8a8 1 row 4096x4096", "kind": "w8a8", "m": 1, "k": 4096, "n": 4096, "layers": 12},
        # sixteen sequences decoding through the wide feed-forward matrix
        {"name": "w8a8 16 rows 4096x14336", "kind": "w8a8", "m": 16, "k": 4096, "n": 14336, "layers": 4},
        # a short portion of a prompt together with decoding sequences: a ragged number of rows, the long K of `down`
        {"name": "w8a8 100 rows 14336x4096", "kind": "w8a8", "m": 100, "k": 14336, "n": 4096, "layers": 4},
        # a prompt
        {"name": "w8a8 2048 rows 4096x14336", "kind": "w8a8", "m": 2048, "k": 4096, "n": 14336, "layers": 2},
        # one token through a 4-bit model
        {"name": "q4_0 1 row 4096x14336", "kind": "gguf", "type": "q4_0", "m": 1, "k": 4096, "n": 14336, "layers": 6},
        # eight sequences through an 8-bit model
        {"name": "q8_0 8 rows 4096x14336", "kind": "gguf", "type": "q8_0", "m": 8, "k": 4096, "n": 14336, "layers": 4},
        # a ragged prompt through a 4-bit model
        {"name": "q4_0 300 rows 4096x14336", "kind": "gguf", "type": "q4_0", "m": 300, "k": 4096, "n": 14336, "layers": 1},
        # the int8 Llama step: sixteen sequences behind 2048 positions
        {"name": "llama step 16 at 2048", "kind": "llama", "batch": 16, "context": 2048},
        # a long prompt of the dense Sonalorn
        {"name": "sonalorn prompt 4096", "kind": "lm", "model": "dense", "dtype": "bfloat16", "running": 0, "context": 0, "prompt": 4096},
        # fifteen sequences decoding while a ragged portion of a prompt comes in, with experts
        {"name": "experts mixed 15 and 777", "kind": "lm", "model": "moe", "dtype": "bfloat16", "running": 15, "context": 1000, "prompt": 777},
        # sixteen Bubotar sequences decoding
        {"name": "bubotar step 16 at 2048", "kind": "lm", "model": "bubotar", "dtype": "bfloat16", "running": 16, "context": 2048, "prompt": 0},
        # a ragged prompt in f32
        {"name": "sonalorn f32 prompt 333", "kind": "lm", "model": "dense", "dtype": "float32", "running": 0, "context": 0, "prompt": 333},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what = rng.random()
    shapes = [(4096, 4096), (4096, 6144), (4096, 14336), (4096, 28672), (14336, 4096)]
    if what < 0.35:
        k, n = rng.choice(shapes) if rng.random() < 0.6 else (rng.randrange(8, 225) * 64, rng.randrange(500, 16000))
        m = _log_int(rng, 1, 4096)
        return {"kind": "w8a8", "m": m, "k": k, "n": n, "layers": max(1, min(12, int(2.4e8 / (k * n)))) if m <= GRAPH_ROWS else 2}
    if what < 0.6:
        k, n = rng.choice(shapes) if rng.random() < 0.6 else (rng.randrange(4, 57) * 256, rng.randrange(500, 16000))
        m = _log_int(rng, 1, 512)
        return {"kind": "gguf", "type": rng.choice(["q4_0", "q8_0"]), "m": m, "k": k, "n": n,
                "layers": max(1, min(6, int(2.4e8 / (k * n)))) if m <= GRAPH_ROWS else 1}
    if what < 0.68:
        return {"kind": "llama", "batch": rng.randrange(1, 33), "context": _log_int(rng, 30, 4000)}
    model, f32 = rng.choice(["dense", "moe", "bubotar"]), rng.random() < 0.25
    case = {"kind": "lm", "model": model, "dtype": "float32" if f32 else "bfloat16", "running": 0, "context": 0, "prompt": 0}
    mode = rng.choice(["prompt", "decode", "mixed"])
    if mode != "prompt":
        case["running"], case["context"] = rng.randrange(1, 17), _log_int(rng, 20, 400 if f32 else 2000)
    if mode != "decode":
        case["prompt"] = _log_int(rng, 5, 330 if f32 else 4000 if mode == "prompt" else 1200)
    return case


# ---- contexts: one per component and process, on a stream that torch shares ---------------------------------------
_contexts = {}


def _context(component):
    if component not in _contexts:
        stream = torch.cuda.Stream()
        _contexts[component] = (GpuContext(0, stream.cuda_stream, component), stream)
    return _contexts[component]


def _gen(seed, name=""):
    return torch.Generator(device=DEV).manual_seed((seed * 1000003 + zlib.crc32(name.encode())) % (1 << 62))


class Stack:
    """Matrices of one shape, their input and outputs, and the graph of a pass over them."""

    def __init__(self, gpu, weights, x, ys, free, call):
        self.gpu, self.weights, self.x, self.ys, self.free, self.call, self.graph = gpu, weights, x, ys, free, call, None
        if x.shape[0] <= GRAPH_ROWS:
            self.enqueue()
            gpu.sync()
            with gpu.record() as g:
                self.enqueue()
            self.graph = g

    def enqueue(self):
        for w, y in zip(self.weights, self.ys):
            self.call(w, y)

    def run(self):
        if self.graph is not None:
            self.graph.launch()
        else:
            self.enqueue()
        return self.ys

    def __del__(self):
        torch.cuda.synchronize()
        if self.graph is not None:
            self.graph.free()
        for w in self.weights:
            self.free(w)


# ---- int8 linears -------------------------------------------------------------------------------------------------
def _activations(case, seed):
    """N(0, 1); decoding meets channels that stand out."""
    x = torch.randn(case["m"], case["k"], generator=_gen(seed, "x"), device=DEV)
    if case["m"] <= GRAPH_ROWS:
        x[:, torch.rand(case["k"], generator=_gen(seed, "channels"), device=DEV) < 0.01] *= 20.0
    return x


def _linear_weight(case, seed, i):
    return torch.randn(case["k"], case["n"], generator=_gen(seed, "w%d" % i), device=DEV) * 0.02


def _prepare_w8a8(case, seed):
    gpu, _stream = _context("int8")
    m, k, n = case["m"], case["k"], case["n"]
    x, weights = _activations(case, seed), []
    for i in range(case["layers"]):
        w = _linear_weight(case, seed, i)
        torch.cuda.synchronize()
        h = C.c_void_p()
        _lib.check(gpu.lib.pg_qtensor_from_f32(gpu.handle, w.data_ptr(), k, n, 0, C.byref(h)))
        gpu.sync()
        weights.append(h)
    ys = [torch.zeros(m, n, device=DEV) for _ in weights]
    torch.cuda.synchronize()
    return Stack(gpu, weights, x, ys, lambda w: gpu.lib.pg_qtensor_free(gpu.handle, w),
                 lambda w, y: _lib.check(gpu.lib.pg_matmul_quantized(gpu.handle, x.data_ptr(), m, k, w, y.data_ptr())))


def _away(v):
    """Rounding of whole f32 values, halves away from zero."""
    v = v.double()
    return torch.sign(v) * torch.floor(v.abs() + 0.5)


def _quantised_columns(w):
    """f32 [k, n] -> whole values in 64 bits, scales per column."""
    s = w.abs().amax(0) / torch.tensor(127.0, device=DEV)      # (by a Python number torch multiplies with the reciprocal)
    s = torch.where(s == 0, torch.ones_like(s), s)
    return _away(w / s).clamp(-127, 127), s.double()


def _quantised_rows(x):
    """Rows as the int8 path takes them: f32 scales and reciprocals."""
    x = x.float()
    s = x.abs().amax(1, keepdim=True) / torch.tensor(127.0, device=DEV)
    s = torch.where(s == 0, torch.ones_like(s), s)
    return _away(x * (1.0 / s)).clamp(-127, 127), s.double()


def _int8_product(x, w):
    (q, s), (wq, ws) = _quantised_rows(x), _quantised_columns(w)
    return (q @ wq) * s * ws


def _exact_w8a8(case, seed):
    x = _activations(case, seed)
    return [_int8_product(x, _linear_weight(case, seed, i)) for i in range(case["layers"])]


# ---- linears on GGUF blocks ---------------------------------------------------------------------------------------
def _blocks(case, seed, i):
    """Quants and f16 scales of an N(0, 0.02) matrix [n, k] in blocks of 32, as the formats' own quantisers choose them."""
    w = (torch.randn(case["n"], case["k"], generator=_gen(seed, "w%d" % i), device=DEV) * 0.02).view(case["n"], -1, 32)
    if case["type"] == "q8_0":
        d = w.abs().amax(2) / 127.0
        q = _away(w / d[..., None]).clamp(-127, 127)
    else:
        top = w.gather(2, w.abs().argmax(2, keepdim=True))[..., 0]
        d = top / -8.0
        q = torch.floor(w / d[..., None] + 8.5).clamp(0, 15)
    return q.to(torch.int16), d.half()


def _raw_blocks(case, q, d):
    scale = d.view(torch.uint8).view(*d.shape, 2)
    if case["type"] == "q8_0":
        body = q.to(torch.int8).view(torch.uint8)
    else:
        body = (q[..., 0::2] + 16 * q[..., 1::2]).to(torch.uint8)
    return torch.cat([scale, body], 2).contiguous().cpu().numpy()


def _prepare_gguf(case, seed):
    gpu, _stream = _context("int8")
    m, k, n = case["m"], case["k"], case["n"]
    x = _activations(case, seed)
    weights = [GgufWeight(case["type"], _raw_blocks(case, *_blocks(case, seed, i)), n, k, gpu) for i in range(case["layers"])]
    ys = [torch.zeros(m, n, device=DEV) for _ in weights]
    torch.cuda.synchronize()
    return Stack(gpu, weights, x, ys, lambda w: w.free(), lambda w, y: w.matmul_device(x, m, y))


def _exact_gguf(case, seed):
    x, out = _activations(case, seed).double(), []
    for i in range(case["layers"]):
        q, d = _blocks(case, seed, i)
        w = (q.double() - (8.0 if case["type"] == "q4_0" else 0.0)) * d.double()[..., None]
        out.append(x @ w.view(case["n"], case["k"]).t())
    return out


# ---- the int8 Llama step ------------------------------------------------------------------------------------------
# (rounding to int8 turns the last bit of a sum into a step of 1 / 127 somewhere, layer upon layer: two layers keep that below
# the tolerance)
LLAMA_LAYERS, LLAMA_VOCAB = 2, 32768


def _llama_config(case):
    from peregrine_b200.llama import LlamaConfig

    return LlamaConfig(layers=LLAMA_LAYERS, vocab=LLAMA_VOCAB, batch=case["batch"], capacity=case["context"] + 128)


class LlamaWeights:
    def __init__(self, c, seed):
        self.c, self.seed = c, seed

    def __getitem__(self, name):
        c, last = self.c, name.split(".")[-1]
        shape = {"embedding": (c.vocab, c.hidden), "lm_head": (c.hidden, c.vocab), "qkv": (c.hidden, c.qkv_dim), "o": (c.hidden, c.hidden),
                 "gate_up": (c.hidden, 2 * c.ffn), "down": (c.ffn, c.hidden)}.get(last)
        w = torch.ones(c.hidden, device=DEV) if shape is None else torch.randn(*shape, generator=_gen(self.seed, name), device=DEV) * 0.02
        torch.cuda.synchronize()
        return w


def _llama_cache(c, context, seed, i, name):
    shape = (c.batch, c.n_kv_heads, context, c.head_dim)
    return torch.randn(*shape, generator=_gen(seed, "%s%d" % (name, i)), device=DEV)


class LlamaState:
    def __init__(self, case, seed):
        from peregrine_b200.llama import LlamaInt8Decoder

        gpu, self.stream = _context("int8")
        c = self.cfg = _llama_config(case)
        self.context = case["context"]
        with torch.cuda.stream(self.stream):
            m = self.model = LlamaInt8Decoder(c, gpu, LlamaWeights(c, seed))
            for i in range(c.layers):
                m.kcache[i, :, :, :self.context] = _llama_cache(c, self.context, seed, i, "k")
                m.vcache[i, :, :, :self.context] = _llama_cache(c, self.context, seed, i, "v")
            self.tokens = torch.randint(0, c.vocab, (c.batch,), generator=_gen(seed, "tokens"), device=DEV, dtype=torch.int32)
            self.place()
            torch.cuda.synchronize()
            m.record()
        torch.cuda.synchronize()

    def place(self):
        """The tokens and the position that the next step starts from."""
        self.model.pos.fill_(self.context)
        self.model.tokens.copy_(self.tokens)
        self.model.embed()

    def run(self):
        m = self.model
        with torch.cuda.stream(self.stream):
            self.place()
            m.graph.launch()
        # logits and what the step added to the caches
        return {"logits": m.logits, "k": m.kcache[:, :, :, self.context], "v": m.vcache[:, :, :, self.context]}

    def __del__(self):
        torch.cuda.synchronize()
        if hasattr(self, "model"):
            if self.model.graph is not None:
                self.model.graph.free()
            self.model.free()


def _exact_llama(case, seed):
    from math import sqrt

    c, W = _llama_config(case), None
    W = LlamaWeights(c, seed)
    B, Hq, G, D, T = c.batch, c.n_q_heads, c.n_kv_heads, c.head_dim, case["context"]
    tokens = torch.randint(0, c.vocab, (B,), generator=_gen(seed, "tokens"), device=DEV, dtype=torch.int32)
    x = W["embedding"][tokens.long()].double()
    # (the reference's table of angles is made in 32 bits)
    inv = np.power(np.float32(c.rope_base), np.float32(2.0) * np.arange(D // 2, dtype=np.float32) / np.float32(D)).astype(np.float32)
    a = torch.from_numpy((np.float32(T) / inv).astype(np.float64)).to(DEV)
    cos, sin = torch.cos(a), torch.sin(a)

    def turn(v):
        u, w = v[..., :D // 2], v[..., D // 2:]
        return torch.cat([u * cos - w * sin, u * sin + w * cos], -1)

    def norm(v):
        return v / torch.sqrt((v * v).mean(-1, keepdim=True) + c.eps)

    ks, vs = [], []
    for i in range(c.layers):
        qkv = _int8_product(norm(x), W["l%d.qkv" % i]).view(B, Hq + 2 * G, D)
        q, k, v = turn(qkv[:, :Hq]), turn(qkv[:, Hq:Hq + G]), qkv[:, Hq + G:]
        ks.append(k), vs.append(v)
        K = torch.cat([_llama_cache(c, T, seed, i, "k").double(), k[:, :, None]], 2)
        V = torch.cat([_llama_cache(c, T, seed, i, "v").double(), v[:, :, None]], 2)
        p = torch.softmax(torch.einsum("bgrd,bgtd->bgrt", q.view(B, G, Hq // G, D), K) / sqrt(D), -1)
        o = torch.einsum("bgrt,bgtd->bgrd", p, V).reshape(B, Hq * D)
        x = x + _int8_product(o, W["l%d.o" % i])
        g = _int8_product(norm(x), W["l%d.gate_up" % i])
        x = x + _int8_product(torch.nn.functional.silu(g[:, :c.ffn]) * g[:, c.ffn:], W["l%d.down" % i])
    return {"logits": _int8_product(norm(x), W["lm_head"]), "k": torch.stack(ks), "v": torch.stack(vs)}


# ---- the bf16 / f32 models ----------------------------------------------------------------------------------------
LM_VOCAB, LM_EPS = 32768, 1e-5


def _lm_config(case):
    """Four layers at the sizes of the framework's own benchmark models."""
    if case["model"] == "bubotar":
        latent = {"heads": 32, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5, "rot": {"base": 10000.0, "dims": 64}}
        attn = {"heads": 32, "kv_heads": 8, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 4096}}
        scan = {"inner": 8192, "state": 16, "dt_rank": 256, "conv": 4}
        mlp = {"kind": "dense", "ff": 14336, "limit": 7.0}
        layers = [{"type": t, "mixer": p, "mlp": m} for t, p, m in
                  (("mamba1", scan, None), ("latent_attention", latent, mlp), ("mamba1", scan, None), ("attention", attn, mlp))]
        return {"architecture": "Bubotar", "vocab": LM_VOCAB, "width": 4096, "norm": {"eps": LM_EPS}, "logit_scale": 1.0, "layers": layers}
    dense = case["model"] == "dense"
    width, H, G = (4096, 32, 16) if dense else (2048, 16, 8)
    delta = {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "conv": 4}
    attn = {"heads": H, "kv_heads": G // 2, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "q_temp": {"coef": 0.1, "every": 4096}}
    mlp = {"kind": "dense", "ff": 14336} if dense else {
        "kind": "moe", "expert": {"ff": 1024, "limit": 7.0}, "router": {"experts": 64, "identity": 16, "top": 8, "groups": {"count": 8, "keep": 4}}}
    return {"architecture": "Sonalorn", "vocab": LM_VOCAB, "width": width, "max_positions": 8192, "norm": {"eps": LM_EPS},
            "layers": [{"type": "attention" if i == 3 else "delta", "mixer": attn if i == 3 else delta, "mlp": mlp} for i in range(4)]}


def _mixer_shapes(kind, p, N):
    H, D, V, G, taps = p.get("heads"), p.get("dim"), p.get("vdim"), p.get("kv_heads"), p.get("conv")
    if kind == "delta":
        return {"q": (G * D, N), "k": (G * D, N), "v": (H * V, N), "g": (H * V, N), "b": (H, N), "a": (H, N), "o": (N, H * V), "q.conv": (G * D, taps),
                "k.conv": (G * D, taps), "v.conv": (H * V, taps), "A_log": (H,), "dt_bias": (H,), "norm": (V,)}
    if kind == "attention":
        return {"q": (H * D, N), "k": (G * D, N), "v": (G * V, N), "o": (N, H * V), "q.norm": (D,), "k.norm": (D,)}
    if kind == "latent_attention":
        K, R = p["kv_rank"], p["rot_dim"]
        return {"q": (H * (D + R), N), "dkv": (K + R, N), "dkv.norm": (K,), "uk": (H * D, K), "uv": (H * V, K), "g": (H * V, N), "o": (N, H * V)}
    I, S, R = p["inner"], p["state"], p["dt_rank"]
    return {"in": (2 * I, N), "conv": (I, taps), "conv.b": (I,), "x": (R + 2 * S, I), "dt": (I, R), "dt.b": (I,), "A_log": (I, S), "D": (I,), "o": (N, I)}


class LmWeights:
    """Tensors by name, each drawn from the seed and its name: bf16 matrices, f32 vectors."""

    def __init__(self, cfg, seed):
        self.cfg, self.seed, self.kept = cfg, seed, {}

    def shape(self, name):
        c = self.cfg
        N = c["width"]
        if name in ("embed", "head"):
            return (c["vocab"], N)
        if name == "pos":
            return (c["max_positions"], N)
        if not name.startswith("l"):
            return (N,)
        i, rest = name[1:].split(".", 1)
        L = c["layers"][int(i)]
        if rest.startswith("mix."):
            return _mixer_shapes(L["type"], L["mixer"], N)[rest[4:]]
        if rest.startswith("mlp."):
            m, last = L["mlp"], rest.split(".")[-1]
            if last in ("router", "correction"):
                n = m["router"]["experts"] + m["router"]["identity"]
                return (n, N) if last == "router" else (n,)
            F = m["ff"] if m["kind"] == "dense" else m["expert"]["ff"]
            return (N, F) if last == "down" else (F, N)
        return (N,)

    def __getitem__(self, name):
        if name in self.kept:
            return self.kept[name]
        s, g = self.shape(name), _gen(self.seed, name)
        if name.endswith("A_log"):
            # decay rates between 1 and 16; a scan's states each have their own
            w = torch.log(1.0 + 15.0 * torch.rand(*s, generator=g, device=DEV)) if len(s) == 1 else torch.log(torch.arange(1.0, s[1] + 1, device=DEV)).expand(s).contiguous()
        elif name.endswith(("dt_bias", "dt.b")):
            # steps between 0.001 and 0.1
            w = torch.log(torch.expm1(torch.exp(torch.empty(*s, device=DEV).uniform_(math.log(1e-3), math.log(0.1), generator=g))))
        elif name.endswith(("correction", "conv.b")):
            w = torch.randn(*s, generator=g, device=DEV) * 0.01
        elif len(s) == 1:
            w = 1.0 + 0.1 * torch.randn(*s, generator=g, device=DEV)
        else:
            w = torch.randn(*s, generator=g, device=DEV, dtype=torch.bfloat16)
            # (a trained router is decided: what falls either way near a tie has little weight)
            w = w if name in ("embed", "pos") else (w * (s[1] ** -0.5 * (3.0 if name.endswith("router") else 1.0))).to(torch.bfloat16)
        self.kept[name] = w
        return w


def _lm_tokens(case, seed, which, n):
    g = _gen(seed, "tokens" + which)
    return torch.randint(0, LM_VOCAB, (n,), generator=g, device=DEV).tolist()


class LmState:
    def __init__(self, case, seed):
        from peregrine_b200.bubotar import BubotarModel
        from peregrine_b200.engine import Engine
        from peregrine_b200.sonalorn import SonalornModel

        gpu, _stream = _context("lm")
        cfg = _lm_config(case)
        Model = BubotarModel if case["model"] == "bubotar" else SonalornModel
        self.n, self.context = case["running"], case["context"]
        longest = max(self.context + 1, case["prompt"])
        weights = LmWeights(cfg, seed)
        self.model = Model(Model.Config.from_dict(cfg), weights, gpu, dtype=case["dtype"], slots=self.n + (1 if case["prompt"] else 0),
                           capacity=longest + 64, step_rows=4096)
        weights.kept.clear()
        torch.cuda.synchronize()
        self.engine = Engine(self.model)
        self.prompt = _lm_tokens(case, seed, "prompt", case["prompt"])
        said = [_lm_tokens(case, seed, str(i), self.context + 1) for i in range(self.n)]
        self.next = [s[-1] for s in said]
        if self.n:
            # the running sequences have been read
            self.engine.step([(i, s[:-1], []) for i, s in enumerate(said)])
        self.decoder = None
        if self.n and not self.prompt:
            d = self.decoder = self.model.decoder(self.n)
            # as an engine does: the first step records the graph
            saved = [{k: v.clone() for k, v in L["state"].items()} for L in self.model.layers]
            self.decode()
            for L, old in zip(self.model.layers, saved):
                for k, v in old.items():
                    L["state"][k].copy_(v)
            del saved, d
        torch.cuda.synchronize()

    def decode(self):
        """One step of the engine's decoding: where the sequences stand, the recorded step, the tokens it chose."""
        d, live = self.decoder, self.engine.live
        d.load([(live[i].slot, self.context, t) for i, t in enumerate(self.next)])
        d.run()
        d.tokens()
        return self.model.logits[:self.n]

    def run(self):
        if self.decoder is not None:
            logits = self.decode()
        else:
            e = self.engine
            entries = [(i, [t], [0]) for i, t in enumerate(self.next)] + [("prompt", self.prompt, [len(self.prompt) - 1])]
            logits = e.step(entries)
            e.end("prompt")
            for i in range(self.n):
                e.live[i].length = self.context
        # logits, and the caches and recurrent states that the step has advanced
        return {"logits": logits, "state": [L["state"] for L in self.model.layers]}

    def __del__(self):
        torch.cuda.synchronize()
        if getattr(self, "decoder", None) is not None:
            self.decoder.free()
        if hasattr(self, "model"):
            self.model.free()


# the models in 64 bits; x [B, T, width], every sequence of a call equally long
def _rms(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + LM_EPS) * w


def _conv(x, w, b=0.0):
    taps = w.shape[1]
    full = torch.nn.functional.pad(x, (0, 0, taps - 1, 0))
    return torch.nn.functional.silu(sum(full[:, j:j + x.shape[1]] * w[:, j] for j in range(taps)) + b)


def _softmax_rows(s, sink):
    m = s.amax(-1, keepdim=True)
    m = m.clamp(min=0.0) if sink else m
    e = torch.exp(s - m)
    return e / (e.sum(-1, keepdim=True) + (torch.exp(-m) if sink else 0.0))


def _attend(q, k, v, scale, sink, slopes=None, more=None):
    """q [T, H, D], k [T, G, D], v [T, G, V] of one sequence; more: scores to add, by head."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    i = torch.arange(T, device=DEV)
    hidden = i[None, :] > i[:, None]
    out = []
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].t()
        s = (s if more is None else s + more(h)) * scale
        if slopes is not None:
            s = s - slopes[h] * (i[:, None] - i[None, :])
        out.append(_softmax_rows(s.masked_fill(hidden, -math.inf), sink) @ v[:, h * G // H])
    return torch.stack(out, 1).flatten(1)


def _rotate(x, pos, base):
    dims = x.shape[-1]
    a = pos[:, None].double() * base ** (-2.0 * torch.arange(dims // 2, device=DEV, dtype=torch.float64) / dims)
    a = a.view(len(pos), *([1] * (x.dim() - 2)), dims // 2)
    u, w = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * a.cos() - w * a.sin(), w * a.cos() + u * a.sin()], -1).flatten(-2)


def _delta64(h, W, p):
    B, T = h.shape[:2]
    H, G, D, V = p["heads"], p["kv_heads"], p["dim"], p["vdim"]
    q, k, v = (_conv(h @ W(n).t(), W(n + ".conv")) for n in ("q", "k", "v"))
    unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)
    q = unit(q.view(B, T, G, D)).repeat_interleave(H // G, 2) * D ** -0.5
    k = unit(k.view(B, T, G, D)).repeat_interleave(H // G, 2)
    v = v.view(B, T, H, V)
    beta = torch.sigmoid(h @ W("b").t())
    g = torch.exp(-torch.exp(W("A_log")) * torch.nn.functional.softplus(h @ W("a").t() + W("dt_bias")))
    S, o = torch.zeros(B, H, D, V, dtype=h.dtype, device=DEV), torch.empty_like(v)
    for t in range(T):
        S.mul_(g[:, t, :, None, None])
        u = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None, :] @ S)[:, :, 0])
        S.addcmul_(k[:, t, :, :, None], u[:, :, None, :])
        o[:, t] = (q[:, t, :, None, :] @ S)[:, :, 0]
    o = _rms(o, W("norm")) * torch.nn.functional.silu(h @ W("g").t()).view(B, T, H, V)
    return o.flatten(2) @ W("o").t(), S


def _attention64(h, W, p, bubotar):
    B, T = h.shape[:2]
    H, G, D, V = p["heads"], p["kv_heads"], p["dim"], p["vdim"]
    q, k, v = (h @ W("q").t()).view(B, T, H, D), (h @ W("k").t()).view(B, T, G, D), (h @ W("v").t()).view(B, T, G, V)
    slopes = None
    if bubotar:
        slopes = [2.0 ** (-8.0 * (i + 1) / H) for i in range(H)]
    else:
        q, k = _rms(q, W("q.norm")), _rms(k, W("k.norm"))
        t = torch.floor((torch.arange(T, device=DEV) + 1) / p["q_temp"]["every"]).double() + 1.0
        q = q * (1.0 + p["q_temp"]["coef"] * torch.log(t))[:, None, None]
    o = torch.stack([_attend(q[b], k[b], v[b], p["scale"], not bubotar, slopes) for b in range(B)])
    return o @ W("o").t(), None


def _latent64(h, W, p):
    B, T = h.shape[:2]
    H, D, R, V, K = (p[n] for n in ("heads", "dim", "rot_dim", "vdim", "kv_rank"))
    pos, base = torch.arange(T, device=DEV), p["rot"]["base"]
    out = []
    for b in range(B):
        both = h[b] @ W("dkv").t()
        c, kr = _rms(both[:, :K], W("dkv.norm")), _rotate(both[:, K:], pos, base)
        q = (h[b] @ W("q").t()).view(T, H, D + R)
        qr = _rotate(q[..., D:], pos, base)
        k, v = (c @ W("uk").t()).view(T, H, D), (c @ W("uv").t()).view(T, H, V)
        out.append(_attend(q[..., :D], k, v, p["scale"], False, None, lambda i: qr[:, i] @ kr.t()))
    return (torch.stack(out) * torch.sigmoid(h @ W("g").t())) @ W("o").t(), None


def _scan64(h, W, p):
    I, N, R, T = p["inner"], p["state"], p["dt_rank"], h.shape[1]
    xz = h @ W("in").t()
    x = _conv(xz[..., :I], W("conv"), W("conv.b"))
    low = x @ W("x").t()
    dt = torch.nn.functional.softplus(low[..., :R] @ W("dt").t() + W("dt.b"))
    A, S, y = -torch.exp(W("A_log")), torch.zeros(h.shape[0], I, N, dtype=h.dtype, device=DEV), torch.empty_like(x)
    for t in range(T):
        S = torch.exp(dt[:, t, :, None] * A) * S + (dt[:, t] * x[:, t])[..., None] * low[:, t, None, R:R + N]
        y[:, t] = (S @ low[:, t, R + N:, None])[..., 0]
    y = y + W("D") * x
    return (y * torch.nn.functional.silu(xz[..., I:])) @ W("o").t(), S


def _ff64(h, W, m):
    if m["kind"] == "moe":
        return _experts64(h.flatten(0, 1), W, m).view(h.shape)
    g, u = h @ W("gate").t(), h @ W("up").t()
    return (_clamped(g, u, m["limit"]) if "limit" in m else torch.nn.functional.gelu(g, approximate="tanh") * u) @ W("down").t()


def _clamped(g, u, limit):
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


def _experts64(h, W, m):
    r = m["router"]
    s = torch.softmax(h @ W("router").t(), -1)
    c, (count, keep) = s + W("correction"), (r["groups"]["count"], r["groups"]["keep"])
    best = c.view(len(h), count, -1).amax(-1)
    ok = torch.zeros_like(best, dtype=torch.bool).scatter_(1, best.topk(keep, -1).indices, True)
    idx = c.masked_fill(~ok.repeat_interleave(c.shape[1] // count, 1), -math.inf).topk(r["top"], -1).indices
    w = torch.zeros_like(s).scatter_(1, idx, s.gather(1, idx))
    y = h * w[:, r["experts"]:].sum(1, keepdim=True)
    for e in range(r["experts"]):
        t = w[:, e].nonzero()[:, 0]
        if len(t):
            x = h[t]
            y[t] += w[t, e, None] * (_clamped(x @ W("e%d.gate" % e).t(), x @ W("e%d.up" % e).t(), m["expert"]["limit"]) @ W("e%d.down" % e).t())
    return y


def _lm64(cfg, weights, ids):
    """Logits behind the last token of each of the equally long sequences, and the recurrent states."""
    get = lambda prefix: (lambda n: weights[prefix + n].double())
    W, bubotar = get(""), cfg["architecture"] == "Bubotar"
    ids = torch.tensor(ids, device=DEV)
    x = weights["embed"][ids].double()
    if not bubotar:
        x = _rms(x + weights["pos"][:ids.shape[1]].double(), W("embed.norm"))
    states = []
    for i, L in enumerate(cfg["layers"]):
        w, mix, mlp = get("l%d." % i), get("l%d.mix." % i), get("l%d.mlp." % i)
        h = _rms(x, w("norm1")) if bubotar else x
        p = L["mixer"]
        y, S = {"delta": _delta64, "mamba1": _scan64, "latent_attention": _latent64}[L["type"]](h, mix, p) if L["type"] != "attention" else _attention64(h, mix, p, bubotar)
        states.append(S)
        x = x + _rms(y, w("norm1b")) if bubotar else x + _rms(y, w("norm1")) * w("ls1")
        if L["mlp"]:
            y = _ff64(_rms(x, w("norm2")) if bubotar else x, mlp, L["mlp"])
            x = x + _rms(y, w("norm2b")) if bubotar else x + _rms(y, w("norm2")) * w("ls2")
    return _rms(x[:, -1], W("final.norm")) @ W("head").t(), states


def _exact_lm(case, seed):
    cfg = _lm_config(case)
    weights = LmWeights(cfg, seed)
    logits, states = [], [[] for _ in cfg["layers"]]
    groups = [[_lm_tokens(case, seed, str(i), case["context"] + 1)] for i in range(case["running"])]
    groups = [sum(groups, [])] if groups else []
    if case["prompt"]:
        groups.append([_lm_tokens(case, seed, "prompt", case["prompt"])])
    for ids in groups:
        l, s = _lm64(cfg, weights, ids)
        logits.append(l)
        for into, S in zip(states, s):
            into.append(S)
    out = []
    for L, S in zip(cfg["layers"], states):
        # caches and convolution inputs are stored roundings of what the logits depend on
        out.append({"ring": None, "state": torch.cat(S)} if L["type"] in ("delta", "mamba1") else None)
    return {"logits": torch.cat(logits), "state": out}


# ---- the interface ------------------------------------------------------------------------------------------------
def prepare(case, seed):
    return {"w8a8": _prepare_w8a8, "gguf": _prepare_gguf, "llama": LlamaState, "lm": LmState}[case["kind"]](case, seed)


def run(state):
    return state.run()


def exact(case, seed):
    return {"w8a8": _exact_w8a8, "gguf": _exact_gguf, "llama": _exact_llama, "lm": _exact_lm}[case["kind"]](case, seed)


def work(case):
    if case["kind"] in ("w8a8", "gguf"):
        m, k, n, layers = (case[x] for x in ("m", "k", "n", "layers"))
        weight = k * n + 4 * n if case["kind"] == "w8a8" else k * n // 32 * (18 if case["type"] == "q4_0" else 34)
        return {"bytes": 4 * m * k + layers * (weight + 4 * m * n), "flops": 2 * m * k * n * layers}
    if case["kind"] == "llama":
        c = _llama_config(case)
        B, T = c.batch, case["context"]
        weights = c.layers * c.hidden * (c.qkv_dim + c.n_q_heads * c.head_dim + 3 * c.ffn) + c.hidden * c.vocab
        kv = c.layers * B * c.n_kv_heads * (T + 1) * c.head_dim
        return {"bytes": weights + 8 * kv + 4 * B * c.vocab, "flops": 2 * B * weights + 4 * kv * (c.n_q_heads // c.n_kv_heads)}
    cfg = _lm_config(case)
    rows, N, n, ctx, T = case["running"] + case["prompt"], cfg["width"], case["running"], case["context"], case["prompt"]
    act = 2 if case["dtype"] == "bfloat16" else 4
    seqs = n + (1 if T else 0)
    nbytes, flops = 2.0 * cfg["vocab"] * N + 4.0 * seqs * cfg["vocab"], 2.0 * seqs * cfg["vocab"] * N
    pairs = n * (ctx + 1) + T * (T + 1) / 2          # query positions times the keys they see
    held = n * (ctx + 1) + T                         # cached positions read or written
    for L in cfg["layers"]:
        p = L["mixer"]
        size = sum(s[0] * s[1] for s in _mixer_shapes(L["type"], p, N).values() if len(s) == 2)
        nbytes, flops = nbytes + 2.0 * size, flops + 2.0 * rows * size
        if L["type"] == "attention":
            nbytes += held * p["kv_heads"] * (p["dim"] + p["vdim"]) * act
            flops += 2.0 * pairs * p["heads"] * (p["dim"] + p["vdim"])
        elif L["type"] == "latent_attention":
            nbytes += held * (p["kv_rank"] + p["rot_dim"]) * act
            flops += 2.0 * pairs * p["heads"] * (p["dim"] + p["rot_dim"] + p["vdim"])
        else:
            one = p["heads"] * p["dim"] * p["vdim"] if L["type"] == "delta" else p["inner"] * p["state"]
            nbytes += 4.0 * one * (2 * n + (1 if T else 0))
            flops += 6.0 * rows * one
        m = L["mlp"]
        if m and m["kind"] == "dense":
            nbytes, flops = nbytes + 6.0 * N * m["ff"], flops + 6.0 * rows * N * m["ff"]
        elif m:
            r, F = m["router"], m["expert"]["ff"]
            every = r["experts"] + r["identity"]
            used = r["experts"] * (1.0 - (1.0 - r["top"] / every) ** rows)
            nbytes += 2.0 * every * N + 6.0 * N * F * used
            flops += 2.0 * rows * every * N + 6.0 * N * F * rows * r["top"] * r["experts"] / every
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "w8a8":
        return "exact"                               # whole sums, two rounded products
    if case["kind"] == "gguf":
        return {"rel": 2e-6, "max": 2e-5}            # 32-bit sums in any order
    if case["kind"] == "llama":
        return {"rel": 3e-2, "max": 0.5}             # another order of a sum moves int8 activations by one step
    if case["dtype"] == "float32":
        # a near tie of the router falls either way
        return {"rel": 2e-2, "max": 0.9} if case["model"] == "moe" else {"rel": 1e-4, "max": 1e-2}
    return {"rel": 3e-2, "max": 0.9}                 # bf16 operands through four layers
