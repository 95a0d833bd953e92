"""What the framework is used for, as cases that can be timed and compared.

Three kinds of case:

``product``  one quantized matrix times activations: the reference's ``Backend`` operators, either over host arrays
             (``CudaBackend.matmul`` / ``matmul_decode``, as a server that keeps its activations on the host calls them) or over device
             memory (``ob_matmul_device``).
``prefill``  a prompt into an empty cache through ``forward``: the logits of its last token.
``decode``   a number of sequences that hold `context` tokens each go on by `steps` tokens: one step whose logits the caller
             sees (``forward_batch_decode``), then the rest greedily without the host in between (``decode_loop``).  The bfloat16
             designs go on by given tokens instead, a call per step, as a server does that samples on the host.

Models are the shapes of ``synth.CONFIGS`` and of bench.py's comparisons with fewer layers and a vocabulary of 32,768: every kernel
runs at its real widths, weights exceed the 126 MB of L2, and a model is made in seconds.  Weights are fixed, as a program keeps
its model; prompts, tokens and activations come from the seed.
"""
from __future__ import annotations

import ctypes as C
import gc
import math
import zlib

import numpy as np
import torch

import orangu_b200
from orangu_b200 import capi, synth
from orangu_b200.backend import QuantMatrix, tensor_byte_size
from orangu_b200.model import LlamaModel

TYPES = {"Q8_0": 8, "Q4_K": 12, "Q6_K": 14}
VOCAB = 32768
LAYERS = {"llama 1b": 8, "llama 8b": 4, "qwen 8b": 4, "fenipel 8b": 4, "nenodra 8b": 4}
MAX_LEN = 4352


def listed():
    return [
        # a single projection for a single token: latency of a launch, and the smallest call there is
        dict(name="q8_0 square, one token", kind="product", type="Q8_0", rows=4096, columns=4096, tokens=1, order="decode", memory="device"),
        # the down projection of eight users' tokens as a host-side server calls it
        dict(name="q6_k down, 8 users, host arrays", kind="product", type="Q6_K", rows=4096, columns=14336, tokens=8, order="decode", memory="host"),
        # the gate projection of a prompt's portion, with a ragged number of tokens
        dict(name="q4_k gate, 509 token portion", kind="product", type="Q4_K", rows=14336, columns=4096, tokens=509, order="prefill", memory="device"),
        # a chat turn on a small model: prompt, then one user's answer
        dict(name="llama 1b, prompt of 512", kind="prefill", model="llama 1b", tokens=512),
        dict(name="llama 1b, decode 1 at 512", kind="decode", model="llama 1b", batch=1, context=512, steps=16),
        # a long prompt on the 8B shape: whole portions of 512 and a ragged last one
        dict(name="llama 8b, prompt of 1900", kind="prefill", model="llama 8b", tokens=1900),
        # one user with a long context, the headline of the framework's own benchmark, and its 64 users
        dict(name="llama 8b, decode 1 at 4096", kind="decode", model="llama 8b", batch=1, context=4096, steps=16),
        dict(name="llama 8b, decode 64 at 4096", kind="decode", model="llama 8b", batch=64, context=4096, steps=8),
        # a few users of a model with biases, head norms and the other rotation layout
        dict(name="qwen 8b, decode 8 at 700", kind="decode", model="qwen 8b", batch=8, context=700, steps=16),
        # the bfloat16 designs: latent attention and retention; softmax attention and experts
        dict(name="fenipel 8b, prompt of 4096", kind="prefill", model="fenipel 8b", tokens=4096),
        dict(name="fenipel 8b, decode 8 at 1024", kind="decode", model="fenipel 8b", batch=8, context=1024, steps=16),
        dict(name="nenodra 8b, decode 64 at 4096", kind="decode", model="nenodra 8b", batch=64, context=4096, steps=8),
    ]


def _log_uniform(rng, low, high):
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high + 0.49))))))


def draw(rng):
    kind = rng.choice(["product", "prefill", "decode"])
    if kind == "product":
        rows, columns = rng.choice([(4096, 4096), (14336, 4096), (4096, 14336), (1024, 4096), (2048, 2048), (8192, 2048), (2048, 8192)])
        tokens = 1 if rng.random() < 0.25 else _log_uniform(rng, 2, 512)
        return dict(kind=kind, type=rng.choice(sorted(TYPES)), rows=rows, columns=columns, tokens=tokens, order=rng.choice(["decode", "prefill"]),
                    memory="host" if tokens <= 64 and rng.random() < 0.25 else "device")
    model = rng.choice(["llama 1b", "llama 8b", "llama 8b", "qwen 8b", "fenipel 8b", "nenodra 8b"])
    if kind == "prefill":
        return dict(kind=kind, model=model, tokens=_log_uniform(rng, 16, 4096 if model in _LAYERED else 2048))
    return dict(kind=kind, model=model, batch=_log_uniform(rng, 1, 64), context=_log_uniform(rng, 64, 4096), steps=rng.randint(4, 16))


# ---------------------------------------------------------------------------------------------- models
_FENIPEL = {"width": 4096, "ff": 14336, "side": 256, "latent": {"heads": 32, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512},
            "retention": {"heads": 16, "dim": 128, "vdim": 256}, "window": 1024}
_NENODRA = {"width": 4096, "ff": 14336, "experts": 16, "top": 2, "expert_ff": 2048, "window": 1024,
            "attention": {"heads": 32, "kv_heads": 8, "dim": 64, "vdim": 128, "diff": 0.5}, "attention_2": {"heads": 32, "kv_heads": 8, "dim": 128, "vdim": 128}}
_LAYERED = {"fenipel 8b", "nenodra 8b"}


def _llama_tensors(name):
    cfg = dict(synth.CONFIGS[name.split()[1]], n_layer=LAYERS[name], n_vocab=VOCAB)
    tensors = synth.model_tensors(cfg, seed=20240)
    if name.startswith("qwen"):
        cfg["rope_neox"] = True
        synth.add_qwen_extras(cfg, tensors, seed=20240)
    return cfg, tensors


def _normal(name, rows, columns, std=None):
    """bfloat16 [rows, columns] on the GPU, normal with `std` (by default 1 / sqrt(columns)), the same for a name every time."""
    g = torch.Generator("cuda")
    g.manual_seed(zlib.crc32(name.encode()))
    return (torch.randn(rows, columns, generator=g, device="cuda") * (columns ** -0.5 if std is None else std)).bfloat16()


def _full(value, n):
    return torch.full((n,), float(value), device="cuda").bfloat16()


def _fenipel():
    """Configuration and bfloat16 tensors, as bench.py's comparison has them."""
    z, n_layer = _FENIPEL, LAYERS["fenipel 8b"]
    E, side, ff = z["width"], z["side"], z["ff"]
    one = torch.ones((), device="cuda").bfloat16()
    t, layers = {"final.norm": one}, []

    def lin(name, rows, columns, std=None):
        t[name] = _normal("fenipel " + name, rows, columns, std)

    lin("embed", VOCAB, E)
    lin("head", VOCAB, E)
    lin("side.embed", VOCAB, n_layer * side)
    for n in range(n_layer):
        at, m = f"l{n}.mix.", dict(z["latent" if n % 2 == 0 else "retention"])
        H, d, v = m["heads"], m["dim"], m["vdim"]
        if n % 2 == 0:
            R, K = m["rot_dim"], m["kv_rank"]
            m.update(mask={"size": z["window"]}, rot={"base": 10000.0, "dims": R}, scale=(d + R) ** -0.5)
            for key, rows, columns in (("q", H * (d + R), E), ("dkv", K + R, E), ("uk", H * d, K), ("uv", H * v, K), ("g", H, E)):
                lin(at + key, rows, columns)
            t[at + "dkv.norm"] = _full(1, K)
        else:
            m.update(rot={"base": 10000.0, "dims": d}, decay=[1 - 2.0 ** (-5 - 0.5 * h) for h in range(H)])
            for key, rows in (("q", H * d), ("k", H * d), ("v", H * v), ("g", H * v)):
                lin(at + key, rows, E)
        lin(at + "o", E, H * v)
        for key, rows, columns in (("mlp.gate", ff, E), ("mlp.up", ff, E), ("mlp.down", E, ff), ("side.gate", side, E), ("side.proj", E, side)):
            lin(f"l{n}.{key}", rows, columns)
        t[f"l{n}.norm1"], t[f"l{n}.side.norm"] = one, _full(1, E)
        layers.append({"type": "latent_attention" if n % 2 == 0 else "retention", "mixer": m, "mlp": {"kind": "dense", "ff": ff, "limit": 7.0}})
    return {"architecture": "Fenipel", "vocab": VOCAB, "width": E, "norm": {"eps": 1e-6}, "token_side": {"dim": side}, "layers": layers}, t


def _nenodra():
    """Configuration and bfloat16 tensors, as bench.py's comparison has them."""
    z, E, t, layers = _NENODRA, _NENODRA["width"], {}, []

    def lin(name, rows, columns, std=None):
        t[name] = _normal("nenodra " + name, rows, columns, std)

    lin("embed", VOCAB, E, 4.0)  # tokens differ enough to choose different experts
    lin("head", VOCAB, E)
    t["final.norm"] = _full(0, E)
    for n in range(LAYERS["nenodra 8b"]):
        kind, maps = ("attention", 2) if n % 2 == 0 else ("attention_2", 1)
        at, m = f"l{n}.mix.", dict(z[kind], mask={"size": z["window"]})
        H, G, d, v = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        m.update(rot={"base": 10000.0, "dims": d}, scale=d ** -0.5)
        lin(at + "q", H * maps * d, E)
        lin(at + "k", G * maps * d, E)
        lin(at + "o", E, H * v)
        t.update({at + "q.norm": _full(1, d), at + "k.norm": _full(1, d), f"l{n}.norm1": _full(0, E), f"l{n}.norm2": _full(0, E)})
        if maps == 2:
            lin(at + "v", G * v, E)
            for key, size in (("q", H * 2 * d), ("k", G * 2 * d), ("v", G * v), ("o", E)):
                t[f"{at}{key}.b"] = _full(0.1, size)
            for key in ("lq1", "lk1", "lq2", "lk2"):
                t[at + key] = _full(0.05, d)
            lin(f"l{n}.mlp.up", z["ff"], E)
            lin(f"l{n}.mlp.down", E, z["ff"])
            mlp = {"kind": "dense", "ff": z["ff"]}
        else:
            lin(at + "g", H * v, E)
            lin(f"l{n}.mlp.router", z["experts"], E)
            for e in range(z["experts"]):
                for key, rows, columns in (("gate", z["expert_ff"], E), ("up", z["expert_ff"], E), ("down", E, z["expert_ff"])):
                    lin(f"l{n}.mlp.e{e}.{key}", rows, columns)
            mlp = {"kind": "moe", "router": {"experts": z["experts"], "top": z["top"]}, "expert": {"ff": z["expert_ff"]}}
        layers.append({"type": kind, "mixer": m, "mlp": mlp})
    return {"architecture": "Nenodra", "vocab": VOCAB, "width": E, "norm": {"eps": 1e-6}, "residual_mult": 1.0, "logit_scale": 1.0, "layers": layers}, t


_DESIGNS = {"fenipel 8b": (_fenipel, orangu_b200.FenipelModel), "nenodra 8b": (_nenodra, orangu_b200.NenodraModel)}
_backend = None
_model = (None, None)  # the model in use: one at a time


def _get_backend():
    global _backend
    if _backend is None:
        _backend = orangu_b200.CudaBackend.init(0)
    return _backend


def _get_model(name):
    global _model
    if _model[0] == name:
        return _model[1]
    if _model[1] is not None:
        _model[1].close()
    _model = (None, None)
    gc.collect()
    be, pool = _get_backend(), 4 * 64 * MAX_LEN  # the caches of several callers
    if name in _LAYERED:
        make, cls = _DESIGNS[name]
        cfg, t = make()
        bits = {k: v.view(torch.uint16).cpu().numpy() for k, v in t.items()}
        t.clear()
        torch.cuda.empty_cache()
        kwargs = {"state_slots": 272} if name.startswith("fenipel") else {}
        model = cls(be, cfg, bits, max_seq_len=MAX_LEN, max_batch_tokens=4096, kv_pool_tokens=pool, **kwargs)
    else:
        cfg, tensors = _llama_tensors(name)
        model = LlamaModel(be, cfg, tensors, max_seq_len=MAX_LEN, max_batch_tokens=512, kv_pool_tokens=pool)
    _model = (name, model)
    return model


# ---------------------------------------------------------------------------------------------- cases
class _DeviceProduct:
    """A registered matrix and activations in device memory."""

    def __init__(self, case, be, data, x):
        self.be, self.lib, self.tokens, self.decode = be, capi.load(), case["tokens"], int(case["order"] == "decode")
        self.handle = C.c_void_p()
        kind = TYPES[case["type"]]
        capi.check(be._h, self.lib.ob_weight_register(be._h, data.ctypes.data, tensor_byte_size(kind, case["columns"]), kind, case["columns"], case["rows"], C.byref(self.handle)))
        self.x = torch.from_numpy(x).cuda()
        self.y = torch.zeros(case["tokens"], case["rows"], device="cuda")

    def run(self):
        capi.check(self.be._h, self.lib.ob_matmul_device(self.be._h, self.x.data_ptr(), self.tokens, self.handle, self.y.data_ptr(), self.decode, None))
        return self.y

    def __del__(self):
        torch.cuda.synchronize()
        self.lib.ob_weight_release(self.be._h, self.handle)


def _activations(case, seed):
    return np.random.default_rng(seed).standard_normal((case["tokens"], case["columns"]), dtype=np.float32)


def _matrix(case, seed):
    return synth.matrix(TYPES[case["type"]], case["rows"], case["columns"], synth.seed_of(seed, case["type"]))["data"]


def _prompt(case, seed):
    n = case["tokens"] if case["kind"] == "prefill" else case["context"]
    return np.random.default_rng([seed, 1]).integers(0, VOCAB, n)


def _continuation(case, seed):
    """What the sequences go on with: [steps, batch], of which greedy decoding uses the first row."""
    return np.random.default_rng([seed, 2]).integers(0, VOCAB, (case["steps"], case["batch"]))


def prepare(case, seed):
    if case["kind"] == "product":
        be, data, x = _get_backend(), _matrix(case, seed), _activations(case, seed)
        if case["memory"] == "device":
            return case, _DeviceProduct(case, be, data, x)
        w = QuantMatrix(data, TYPES[case["type"]], case["columns"], case["rows"])
        return case, (be, w, x)
    model, prompt = _get_model(case["model"]), _prompt(case, seed)
    if case["kind"] == "prefill":
        return case, (model, model.new_kv_cache(case["tokens"]), prompt)
    room = case["context"] + case["steps"]
    first = model.new_kv_cache(room)
    model.forward_maybe_sampling(first, prompt, 0)
    caches = [first]
    if model_is_recurrent := case["model"].startswith("fenipel"):
        caches = []  # a recurrent state cannot be rolled back: every pass starts from copies of the held prefix
    while len(caches) < case["batch"]:
        caches.append(model.new_kv_cache(room))
        if not model_is_recurrent:
            caches[-1].copy_prefix_from(first, case["context"])
    return case, (model, first, caches, _continuation(case, seed))


def run(state):
    case, s = state
    if case["kind"] == "product":
        if case["memory"] == "device":
            return s.run()
        be, w, x = s
        return be.matmul_decode(x, case["tokens"], w) if case["order"] == "decode" else be.matmul(x, case["tokens"], w)
    if case["kind"] == "prefill":
        model, cache, prompt = s
        cache.truncate(0)
        return model.forward(cache, prompt, 0)
    model, first, caches, tokens = s
    for cache in caches:
        if case["model"].startswith("fenipel"):
            cache.truncate(0)
            cache.copy_prefix_from(first, case["context"])
        else:
            cache.truncate(case["context"])
    if case["model"] in _LAYERED:
        for step in tokens[:-1]:
            model.forward_batch_decode(caches, step)
        return model.forward_batch_decode(caches, tokens[-1], want_logits=True)[1]
    chosen, logits = model.forward_batch_decode(caches, tokens[0], want_logits=True)
    return {"logits": logits, "tokens": model.decode_loop(caches, chosen, case["steps"] - 1)}


def _sizes(name):
    """(weight bytes per step by batch, weights that a token meets, cache bytes per token of context, flops per token and token of context,
    longest window) without the embedding; logits apart."""
    if name == "fenipel 8b":
        z, la, re = _FENIPEL, _FENIPEL["latent"], _FENIPEL["retention"]
        E, half = z["width"], LAYERS[name] // 2
        latent = la["heads"] * (la["dim"] + la["rot_dim"]) * E + (la["kv_rank"] + la["rot_dim"]) * E + la["heads"] * (la["dim"] + la["vdim"]) * la["kv_rank"] + la["heads"] * E + la["heads"] * la["vdim"] * E
        retention = re["heads"] * (2 * re["dim"] + 3 * re["vdim"]) * E
        n = half * (latent + retention) + 2 * half * (3 * E * z["ff"] + 2 * z["side"] * E)
        return (lambda batch: 2 * n), n, half * (la["kv_rank"] + la["rot_dim"]) * 2, half * 2 * la["heads"] * (la["dim"] + la["rot_dim"] + la["vdim"]), z["window"]
    if name == "nenodra 8b":
        z, half = _NENODRA, LAYERS[name] // 2
        E, expert = z["width"], 3 * z["width"] * z["expert_ff"]
        n, cache, flops = 0, 0, 0
        for kind, maps in (("attention", 2), ("attention_2", 1)):
            m = z[kind]
            n += half * E * (m["heads"] * maps * m["dim"] + m["kv_heads"] * maps * m["dim"] + m["heads"] * m["vdim"] + (m["kv_heads"] if maps == 2 else m["heads"]) * m["vdim"])
            cache += half * 2 * m["kv_heads"] * (maps * m["dim"] + m["vdim"])
            flops += half * 2 * m["heads"] * maps * (m["dim"] + m["vdim"])
        n += half * (2 * E * z["ff"] + z["experts"] * E)
        read = lambda batch: 2 * (n + half * expert * z["experts"] * (1 - (1 - z["top"] / z["experts"]) ** batch))  # noqa: E731
        return read, n + half * z["top"] * expert, cache, flops, z["window"]
    c = synth.CONFIGS[name.split()[1]]
    e, qd, kvd, ff = c["n_embd"], c["n_head"] * c["head_dim"], c["n_head_kv"] * c["head_dim"], c["n_ff"]
    per = lambda kind, o, i: o * tensor_byte_size(kind, i)  # noqa: E731
    layer = per(12, 2 * qd, e) + per(12, kvd, e) + per(14, kvd, e) + per(12, 3 * ff, e)
    n = LAYERS[name] * (2 * qd * e + 2 * kvd * e + 3 * ff * e)
    return (lambda batch: LAYERS[name] * layer), n, LAYERS[name] * 2 * kvd * 2, LAYERS[name] * 4 * qd, 1 << 30


def work(case):
    if case["kind"] == "product":
        n = case["rows"] * case["columns"]
        return {"bytes": case["rows"] * tensor_byte_size(TYPES[case["type"]], case["columns"]) + 4 * case["tokens"] * (case["rows"] + case["columns"]), "flops": 2 * n * case["tokens"]}
    read, n, cache, pairs, window = _sizes(case["model"])
    E = synth.CONFIGS[case["model"].split()[1]]["n_embd"]
    head = VOCAB * E * (2 if case["model"] in _LAYERED else 210 / 256)
    if case["kind"] == "prefill":
        t = case["tokens"]
        seen = sum(min(i + 1, window) for i in range(t))
        return {"bytes": read(t) + head + t * cache + 4 * VOCAB, "flops": 2 * t * n + seen * pairs + 2 * VOCAB * E}
    b, s = case["batch"], case["steps"]
    seen = sum(min(case["context"] + i + 1, window) for i in range(s)) * b
    state = 0
    if case["model"] == "fenipel 8b":
        re = _FENIPEL["retention"]
        state = b * s * (LAYERS["fenipel 8b"] // 2) * re["heads"] * re["dim"] * re["vdim"] * 8
    return {"bytes": s * (read(b) + head) + seen * cache + state + 4 * b * VOCAB, "flops": s * b * 2 * (n + VOCAB * E) + seen * pairs}


def tolerance(case):
    """Products: sums of up to 14336 terms in fp32 in another order.  Quantized models: an activation that differs in its last bit
    now and then gets another 8-bit code, and a few layers spread that to the noise of the codes themselves.  bfloat16 designs: the
    rounding of activations, and with experts, now and then, which of two nearly equal ones a token takes."""
    if case["kind"] == "product":
        return {"rel": 2e-6, "max": 5e-5}
    if case["model"] == "fenipel 8b":
        return {"rel": 0.02, "max": 0.2}
    if case["model"] == "nenodra 8b":
        return {"rel": 0.03, "max": 1 - 2.0 ** -10}
    return {"rel": 0.03, "max": 0.4, "differ": 0.01}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
def _dequantized(kind, data, rows, columns):
    """GGUF blocks as float64 [rows, columns] on the GPU."""
    raw = torch.from_numpy(data).cuda()

    def halves(b):
        return b.contiguous().view(torch.float16).double()

    if kind == TYPES["Q8_0"]:
        b = raw.view(-1, 34)
        return (halves(b[:, :2]) * b[:, 2:].contiguous().view(torch.int8).double()).view(rows, columns)
    if kind == TYPES["Q4_K"]:
        b = raw.view(-1, 144)
        d, dmin, s = halves(b[:, 0:2]), halves(b[:, 2:4]), b[:, 4:16].int()
        sc = torch.cat([s[:, 0:4] & 63, (s[:, 8:12] & 15) | ((s[:, 0:4] >> 6) << 4)], 1)
        mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:12] >> 4) | ((s[:, 4:8] >> 6) << 4)], 1)
        q = b[:, 16:].view(-1, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 2).view(-1, 8, 32).double()
        return ((d * sc)[:, :, None] * q - (dmin * mn)[:, :, None]).view(rows, columns)
    b = raw.view(-1, 210)
    ql, qh, s, d = b[:, 0:128].view(-1, 2, 2, 32), b[:, 128:192].view(-1, 2, 1, 32), b[:, 192:208].contiguous().view(torch.int8), halves(b[:, 208:210])
    low = torch.stack([ql[:, :, 0] & 15, ql[:, :, 1] & 15, ql[:, :, 0] >> 4, ql[:, :, 1] >> 4], 2)
    high = torch.cat([qh & 3, (qh >> 2) & 3, (qh >> 4) & 3, qh >> 6], 2)
    q = (low.int() | (high.int() << 4)).double() - 32
    return ((d * s.double())[:, :, None] * q.view(-1, 16, 16)).view(rows, columns)


def _coded(x, kind):
    """float64 activations as the 8-bit codes and scales in which a product of this type reads them."""
    group = 32 if kind == TYPES["Q8_0"] else 256
    v = x.float().view(-1, group)
    most = v.abs().amax(1, keepdim=True)
    scale = most / torch.full_like(most, 127.0)  # (a division by a number may be done as a multiplication)
    r = torch.where(scale > 0, v * (torch.ones_like(scale) / scale), torch.zeros_like(v)).double()
    code = (r.sign() * torch.floor(r.abs() + 0.5)).clamp(-127, 127)
    return (code * scale.double()).view(x.shape)


def _over_rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _rotated(x, positions, base, dims, pairs):
    """x [n, heads, width]; its first `dims` entries turn by position: neighbours, or entries half of `dims` apart."""
    a = positions.double()[:, None, None] * (float(base) ** (-2.0 * torch.arange(dims // 2, device="cuda").double() / dims))
    cos, sin = torch.cos(a), torch.sin(a)
    y = x.clone()
    u, v = (x[..., 0:dims:2], x[..., 1:dims:2]) if pairs else (x[..., : dims // 2], x[..., dims // 2: dims])
    if pairs:
        y[..., 0:dims:2], y[..., 1:dims:2] = u * cos - v * sin, v * cos + u * sin
    else:
        y[..., : dims // 2], y[..., dims // 2: dims] = u * cos - v * sin, v * cos + u * sin
    return y


class _Sequences:
    """A prompt and rows that go on from it.  Layers see the prompt's rows first and then, step by step, a row of every sequence."""

    def __init__(self, prompt, steps):
        self.n, self.batch = len(prompt), steps.shape[1] if steps is not None else 0
        self.tokens = torch.from_numpy(np.concatenate([prompt, steps.reshape(-1)]) if self.batch else np.asarray(prompt)).cuda()
        tail = torch.arange(self.tokens.numel() - self.n, device="cuda")
        self.positions = torch.cat([torch.arange(self.n, device="cuda"), self.n + tail // max(1, self.batch)])
        self.sequence = torch.cat([torch.full((self.n,), -1, device="cuda"), tail % max(1, self.batch)])
        self.wanted = slice(self.tokens.numel() - max(1, self.batch), self.tokens.numel())

    def attend(self, q, k, v, scale, window=1 << 30):
        """Softmax average of one head over what a row sees: the prompt and its own sequence, up to itself, within the window."""
        out = torch.empty(q.shape[0], v.shape[1], dtype=torch.float64, device="cuda")
        for r0 in range(0, q.shape[0], 1024):
            r = slice(r0, r0 + 1024)
            ahead = self.positions[r, None] - self.positions[None]
            sees = (ahead >= 0) & (ahead < window) & ((self.sequence[None] < 0) | (self.sequence[None] == self.sequence[r, None]))
            s = torch.where(sees, q[r] @ k.T * scale, torch.full((), -math.inf, dtype=torch.float64, device="cuda"))
            out[r] = torch.softmax(s, 1) @ v
        return out


def _exact_llama(name, rows):
    cfg, t = _llama_tensors(name)
    hd, H, G, eps = cfg["head_dim"], cfg["n_head"], cfg["n_head_kv"], cfg["rms_eps"]

    def vector(key):
        return torch.from_numpy(t[key]["data"]).cuda().double()

    def product(x, key):
        m = t[key]
        return _coded(x, m["type"]) @ _dequantized(m["type"], m["data"], m["out_dim"], m["in_dim"]).T

    m = t["token_embd.weight"]
    x = _dequantized(m["type"], m["data"], m["out_dim"], m["in_dim"])[rows.tokens]
    qwen = name.startswith("qwen")
    for i in range(cfg["n_layer"]):
        p = f"blk.{i}."
        h = _over_rms(x, eps) * vector(p + "attn_norm.weight")
        q, k, v = (product(h, f"{p}attn_{c}.weight") for c in "qkv")
        if qwen:
            q, k, v = q + vector(p + "attn_q.bias"), k + vector(p + "attn_k.bias"), v + vector(p + "attn_v.bias")
        q, k, v = q.view(-1, H, hd), k.view(-1, G, hd), v.view(-1, G, hd)
        if qwen:
            q, k = _over_rms(q, eps) * vector(p + "attn_q_norm.weight"), _over_rms(k, eps) * vector(p + "attn_k_norm.weight")
        q, k = (_rotated(a, rows.positions, cfg["rope_freq_base"], hd, not qwen) for a in (q, k))
        k, v = k.half().double(), v.half().double()  # the cache holds 16 bits
        o = torch.cat([rows.attend(q[:, a], k[:, a * G // H], v[:, a * G // H], hd ** -0.5) for a in range(H)], 1)
        x = x + product(o, p + "attn_output.weight")
        h = _over_rms(x, eps) * vector(p + "ffn_norm.weight")
        gate, up = product(h, p + "ffn_gate.weight"), product(h, p + "ffn_up.weight")
        x = x + product(gate * torch.sigmoid(gate) * up, p + "ffn_down.weight")
    return product(_over_rms(x[rows.wanted], eps) * vector("output_norm.weight"), "output.weight")


def _retention(rows, q, k, v, decay):
    """Decayed sums over the rows before: q, k [n, dim], v [n, vdim] of one head, its state handed from the prompt to every sequence."""
    n, out = rows.n, torch.empty(q.shape[0], v.shape[1], dtype=torch.float64, device="cuda")
    state, block, log = torch.zeros(q.shape[1], v.shape[1], dtype=torch.float64, device="cuda"), 256, math.log(decay)
    for b0 in range(0, n, block):
        b = slice(b0, min(n, b0 + block))
        i = torch.arange(b.stop - b0, device="cuda").double()
        ago = i[:, None] - i[None]
        out[b] = torch.where(ago >= 0, torch.exp(ago * log), torch.zeros_like(ago)) * (q[b] @ k[b].T) @ v[b] + torch.exp((i + 1) * log)[:, None] * (q[b] @ state)
        state = decay ** (b.stop - b0) * state + (torch.exp((i[-1] - i) * log)[:, None] * k[b]).T @ v[b]
    states = state.expand(rows.batch, -1, -1)
    for b0 in range(n, q.shape[0], max(1, rows.batch)):
        b = slice(b0, b0 + rows.batch)
        states = decay * states + k[b, :, None] * v[b, None, :]
        out[b] = (q[b, None, :] @ states)[:, 0]
    return out


def _exact_fenipel(rows):
    cfg, t = _fenipel()
    E, eps, side = cfg["width"], cfg["norm"]["eps"], cfg["token_side"]["dim"]
    x = t["embed"][rows.tokens].double()
    for n, layer in enumerate(cfg["layers"]):
        at, m = f"l{n}.", layer["mixer"]
        w = {k[len(at):]: v.double() for k, v in t.items() if k.startswith(at)}
        H, D, V, base = m["heads"], m["dim"], m["vdim"], m["rot"]["base"]
        h = _over_rms(x, eps) * w["norm1"]
        q = (h @ w["mix.q"].T).view(len(h), H, -1)
        if layer["type"] == "retention":
            k, v = (h @ w["mix.k"].T).view(len(h), H, D), (h @ w["mix.v"].T).view(len(h), H, V)
            q, k = (_rotated(a, rows.positions, base, m["rot"]["dims"], False) for a in (q, k))
            o = torch.stack([_retention(rows, q[:, a], k[:, a] * D ** -0.5, v[:, a], m["decay"][a]) for a in range(H)], 1)
            g = h @ w["mix.g"].T
            o = _over_rms(o, eps).reshape(len(h), -1) * (g * torch.sigmoid(g))
        else:
            K = m["kv_rank"]
            dkv = h @ w["mix.dkv"].T
            c = _over_rms(dkv[:, :K], eps) * w["mix.dkv.norm"]
            kn, v = (c @ w["mix.uk"].T).view(len(h), H, D), (c @ w["mix.uv"].T).view(len(h), H, V)
            kr = _rotated(dkv[:, None, K:], rows.positions, base, m["rot_dim"], True)[:, 0]
            qr = _rotated(q[:, :, D:], rows.positions, base, m["rot_dim"], True)
            gate = torch.sigmoid(h @ w["mix.g"].T)
            o = torch.cat([rows.attend(torch.cat([q[:, a, :D], qr[:, a]], 1), torch.cat([kn[:, a], kr], 1), v[:, a], m["scale"], m["mask"]["size"]) * gate[:, a, None] for a in range(H)], 1)
        lim = layer["mlp"]["limit"]
        g, u = (h @ w["mlp.gate"].T).clamp(max=lim), (h @ w["mlp.up"].T).clamp(-lim, lim)
        x = x + o @ w["mix.o"].T + (g * torch.sigmoid(1.702 * g) * (u + 1)) @ w["mlp.down"].T
        e = t["side.embed"][rows.tokens, n * side:(n + 1) * side].double()
        y = (torch.nn.functional.gelu(x @ w["side.gate"].T, approximate="tanh") * e) @ w["side.proj"].T
        x = x + _over_rms(y, eps) * w["side.norm"]
    return (_over_rms(x[rows.wanted], eps) * t["final.norm"].double()) @ t["head"].double().T


def _exact_nenodra(rows):
    cfg, t = _nenodra()
    eps = cfg["norm"]["eps"]
    x = t["embed"][rows.tokens].double()
    for n, layer in enumerate(cfg["layers"]):
        at, m, mlp = f"l{n}.", layer["mixer"], layer["mlp"]
        w = {k[len(at):]: v.double() for k, v in t.items() if k.startswith(at)}
        H, G, D, V = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        q, k = x @ w["mix.q"].T, x @ w["mix.k"].T
        turn = lambda a, heads, norm: _rotated(_over_rms(a.view(len(x), heads, D), eps) * norm, rows.positions, m["rot"]["base"], D, False)  # noqa: E731
        if layer["type"] == "attention":
            q, k = turn(q + w["mix.q.b"], 2 * H, w["mix.q.norm"]), turn(k + w["mix.k.b"], 2 * G, w["mix.k.norm"])
            v = (x @ w["mix.v"].T + w["mix.v.b"]).view(len(x), G, V)
            weight = float(torch.exp((w["mix.lq1"] * w["mix.lk1"]).sum()) - torch.exp((w["mix.lq2"] * w["mix.lk2"]).sum())) + m["diff"]
            heads = []
            for a in range(H):
                g = a * G // H
                one, two = (rows.attend(q[:, 2 * a + i], k[:, 2 * g + i], v[:, g], m["scale"], m["mask"]["size"]) for i in (0, 1))
                heads.append(_over_rms(one - weight * two, eps) * (1 - m["diff"]))
            y = torch.cat(heads, 1) @ w["mix.o"].T + w["mix.o.b"]
        else:
            v = k.view(len(x), G, V)
            q, k = turn(q, H, w["mix.q.norm"]), turn(k, G, w["mix.k.norm"])
            o = torch.cat([rows.attend(q[:, a], k[:, a * G // H], v[:, a * G // H], m["scale"], m["mask"]["size"]) for a in range(H)], 1)
            y = (o * torch.sigmoid(x @ w["mix.g"].T)) @ w["mix.o"].T
        x = x + cfg["residual_mult"] * _over_rms(y, eps) * (1 + w["norm1"])
        if mlp["kind"] == "dense":
            y = (x @ w["mlp.up"].T).clamp(min=0) ** 2 @ w["mlp.down"].T
        else:
            score, best = torch.sigmoid(x @ w["mlp.router"].T).topk(mlp["router"]["top"], dim=1)
            y = torch.zeros_like(x)
            for e in range(mlp["router"]["experts"]):
                row, place = torch.nonzero(best == e, as_tuple=True)
                z = score[row, place, None] * x[row]
                g = z @ w[f"mlp.e{e}.gate"].T
                y.index_add_(0, row, (g * torch.sigmoid(g) * (z @ w[f"mlp.e{e}.up"].T)) @ w[f"mlp.e{e}.down"].T)
        x = x + cfg["residual_mult"] * _over_rms(y, eps) * (1 + w["norm2"])
    return (_over_rms(x[rows.wanted], eps) * (1 + t["final.norm"].double())) @ t["head"].double().T * cfg["logit_scale"]


def exact(case, seed):
    if case["kind"] == "product":
        kind = TYPES[case["type"]]
        w = _dequantized(kind, _matrix(case, seed), case["rows"], case["columns"])
        return _coded(torch.from_numpy(_activations(case, seed)).cuda(), kind) @ w.T
    layered = case["model"] in _LAYERED
    steps = None if case["kind"] == "prefill" else _continuation(case, seed)[: None if layered else 1]
    rows = _Sequences(_prompt(case, seed), steps)
    if case["model"] == "fenipel 8b":
        logits = _exact_fenipel(rows)
    elif case["model"] == "nenodra 8b":
        logits = _exact_nenodra(rows)
    else:
        logits = _exact_llama(case["model"], rows)
    if case["kind"] == "prefill":
        return logits[0]
    return logits if layered else {"logits": logits, "tokens": None}  # (which tokens follow is decided by differences below the rounding)
