"""The work that users of this package have it do, as cases to be timed and compared: GPT-2 steps and prompts over the
weight formats and precisions it takes, prompts and whole requests of the layer-list decoders, `relu(matmul)`, and
schedule items run one by one.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` builds the model and the inputs,
``run`` is one pass through the public entry points, ``exact`` the same in 64 bits in plain torch, ``work`` the bytes and
operations a pass cannot do without.  Models have the repository's own sizes and random weights (one set per
configuration, as a user keeps one model); prompts, tokens and plain inputs come from the seed."""
import ctypes
import functools
import math

import numpy as np
import torch

from caten_b200 import _lib as L
from caten_b200 import binusun, expr, goselix, synthetic
from caten_b200.gpt2 import GPT2
from caten_b200.runtime import B200Buffer, B200Runtime

DEV = "cuda"
VOCAB = 32000   # of the layer-list decoders; GPT-2 has its own 50257
PRECISIONS = {"fp32": L.PREC_FP32, "bf16": L.PREC_BF16, "bf16x3": L.PREC_BF16X3}

# the layers that `bench.py --compare` times, at its two widths
BINUSUN = {1024: dict(order="wAAwAAAAAAAA", ff=2816, heads=8, kv_heads=4, dim=128, vdim=128, window=1024, wkv_heads=16, wkv_dim=64, rot_dims=64),
           2048: dict(order="wAAwAAAA", ff=5632, heads=16, kv_heads=4, dim=128, vdim=128, window=1024, wkv_heads=32, wkv_dim=64, rot_dims=64)}
GOSELIX = {1024: dict(order="ldlmrdlmrmldlmrd", ff=2816, heads=16, dim=48, rot_dim=16, vdim=64, q_rank=384, kv_rank=128, ret_heads=8, ret_dim=64,
                      ret_vdim=128, ret_rot=64, experts=8, top=2, expert_ff=704),
           2048: dict(order="ldlmrdlmrmld", ff=5632, heads=16, dim=96, rot_dim=32, vdim=128, q_rank=768, kv_rank=256, ret_heads=8, ret_dim=128,
                      ret_vdim=256, ret_rot=128, experts=8, top=2, expert_ff=1408)}
LOW_RANK = 64


def listed():
    return [
        # one interactive user of the small model: a token at a time, latency is all
        {"name": "small-f32-step-1", "kind": "gpt2", "model": "gpt2", "wtype": "f32", "precision": "fp32", "batch": 1, "context": 66, "tokens": 1},
        # one interactive user of the largest model, quantised
        {"name": "xl-q4_0-step-1", "kind": "gpt2", "model": "gpt2-xl", "wtype": "q4_0", "precision": "bf16x3", "batch": 1, "context": 640, "tokens": 1},
        # a server's ordinary batch
        {"name": "medium-q4_0-step-64", "kind": "gpt2", "model": "gpt2-medium", "wtype": "q4_0", "precision": "bf16x3", "batch": 64, "context": 199, "tokens": 1},
        # the largest batch, at a context whose cache leaves room for more than one of them
        {"name": "xl-q4_0-step-256", "kind": "gpt2", "model": "gpt2-xl", "wtype": "q4_0", "precision": "bf16x3", "batch": 256, "context": 203, "tokens": 1},
        # reading prompts before such a batch is decoded
        {"name": "xl-q4_0-prompt-16x512", "kind": "gpt2", "model": "gpt2-xl", "wtype": "q4_0", "precision": "bf16x3", "batch": 16, "context": 0, "tokens": 512},
        # a few prompts of no particular length, weights as they were trained
        {"name": "medium-bf16-prompt-5x333", "kind": "gpt2", "model": "gpt2-medium", "wtype": "bf16", "precision": "bf16", "batch": 5, "context": 0, "tokens": 333},
        # the fused pair of the reference's introduction, at a feed-forward's size
        {"name": "relu-matmul-4096x768x3072", "kind": "relu_matmul", "m": 4096, "k": 768, "n": 3072, "precision": "bf16x3"},
        # prompts through windowed attention and time mixing
        {"name": "binusun-2048-prompt-8x1024", "kind": "binusun", "width": 2048, "batch": 8, "prompt": 1024, "decode": 0, "precision": "bf16"},
        # whole requests: prompts, then token by token
        {"name": "binusun-1024-request-16", "kind": "binusun", "width": 1024, "batch": 16, "prompt": 1023, "decode": 64, "precision": "bf16"},
        # ragged prompts through latent attention, retention and experts
        {"name": "goselix-2048-prompt-3x777", "kind": "goselix", "width": 2048, "batch": 3, "prompt": 777, "decode": 0, "precision": "bf16"},
        {"name": "goselix-1024-request-64", "kind": "goselix", "width": 1024, "batch": 64, "prompt": 200, "decode": 48, "precision": "bf16"},
        # a graph without kernels of its own: softmax as the reference composes it, item by item
        {"name": "items-softmax-12800x511", "kind": "items", "what": "softmax", "rows": 12800, "cols": 511},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "prompt", "prompt", "relu_matmul", "binusun", "binusun", "goselix", "goselix", "items"])
    if kind in ("step", "prompt"):
        model = rng.choice(["gpt2", "gpt2-medium", "gpt2-large", "gpt2-xl"])
        wtype = rng.choice(["f32", "f16", "bf16", "q8_0", "q8_0", "q4_0", "q4_0", "q4_0", "q4_1", "q5_0", "q5_1"])
        precision = rng.choice(["fp32", "bf16", "bf16x3", "bf16x3"])
        p = synthetic.GPT2_SIZES[model]
        case = {"kind": "gpt2", "model": model, "wtype": wtype, "precision": precision}
        if kind == "step":
            batch, context = _log(rng, 1, 256), _log(rng, 8, 900)
            kv = 8 * p.n_layers * p.dim
            case.update(batch=batch, context=max(8, min(context, int(35e9 / (kv * batch)))), tokens=1)
            if precision == "fp32":   # the exact kernels are for checking and for a few sequences
                case["batch"] = min(batch, 8)
        else:
            most = 8192 * (1 if model == "gpt2-xl" else 2) // (16 if precision == "fp32" else 1)
            tokens = _log(rng, 5, 1000)
            case.update(batch=_log(rng, 1, max(1, min(64, most // tokens))), context=0, tokens=min(tokens, most))
        return case
    if kind == "relu_matmul":
        return {"kind": kind, "m": _log(rng, 64, 8192), "k": 64 * _log(rng, 2, 48), "n": 64 * _log(rng, 2, 64), "precision": rng.choice(["bf16", "bf16x3"])}
    if kind == "items":
        return {"kind": kind, "what": rng.choice(["softmax", "gelu"]), "rows": _log(rng, 16, 16384), "cols": _log(rng, 16, 2048)}
    width = rng.choice([1024, 2048])
    case = {"kind": kind, "width": width, "precision": "bf16"}
    if rng.random() < 0.5:
        tokens = _log(rng, 32, 2048)
        case.update(batch=_log(rng, 1, max(1, min(256, 8192 // tokens))), prompt=tokens, decode=0)
    else:
        tokens = _log(rng, 32, 1024)
        case.update(batch=_log(rng, 1, max(1, min(256, 16384 // tokens))), prompt=tokens, decode=_log(rng, 8, 96 if width == 1024 else 48))
    return case


# ---- inputs ---------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) % (1 << 40))


def _tokens(seed, batch, count, vocab):
    return torch.randint(0, vocab, (batch, count), generator=_generator(seed), device=DEV, dtype=torch.int64)


@functools.cache
def _runtime():
    return B200Runtime(0)


class _DeviceArray:
    """Device memory of a model, for torch.as_tensor, which keeps this object and with it the model."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": "<f4", "version": 2, "strides": None}


def _view(owner, ptr, shape):
    return torch.as_tensor(_DeviceArray(owner, ptr, shape), device=DEV)


# ---- GPT-2 ----------------------------------------------------------------------------------------
BLOCKS = {"q4_0": (L.Q4_0, 18), "q4_1": (L.Q4_1, 20), "q5_0": (L.Q5_0, 22), "q5_1": (L.Q5_1, 24), "q8_0": (L.Q8_0, 34)}
DENSE = {"f32": (L.F32, torch.float32), "f16": (L.F16, torch.float16), "bf16": (L.BF16, torch.bfloat16)}


class _Matrix:
    """A weight as its file holds it, on the GPU: what GPT2 wants to know of it, and its values in 64 bits."""

    def __init__(self, gen, rows, cols, wtype):
        self.rows, self.cols, self.wtype, std = rows, cols, wtype, 0.02
        if wtype in DENSE:
            self.ggml_type, kind = DENSE[wtype]
            self.data = (torch.randn(rows, cols, generator=gen, device=DEV) * std).to(kind)
            return
        self.ggml_type, size = BLOCKS[wtype]
        n = rows * cols // 32
        self.data = torch.randint(0, 256, (n, size), generator=gen, device=DEV, dtype=torch.uint8)
        half = {"q8_0": 127, "q4_0": 8, "q4_1": 8, "q5_0": 16, "q5_1": 16}[wtype]
        d = (torch.randn(n, generator=gen, device=DEV).abs() * (std / half)).half()
        self.data[:, 0:2] = d.view(torch.uint8).view(n, 2)
        if wtype.endswith("_1"):   # a minimum that centres the codes
            m = (d.float() * -half + torch.randn(n, generator=gen, device=DEV) * (std / 16)).half()
            self.data[:, 2:4] = m.view(torch.uint8).view(n, 2)

    def double(self):
        if self.wtype in DENSE:
            return self.data.double()
        b, n = self.data, self.data.shape[0]
        d = b[:, 0:2].contiguous().view(torch.float16).double()
        if self.wtype == "q8_0":
            return (b[:, 2:].contiguous().view(torch.int8).double() * d).view(self.rows, self.cols)
        at = 4 if self.wtype.endswith("_1") else 2
        code = torch.cat([b[:, -16:] & 15, b[:, -16:] >> 4], 1)
        if self.wtype.startswith("q5"):
            shift = torch.arange(8, device=DEV, dtype=torch.uint8)
            code = code + (((b[:, at:at + 4, None] >> shift) & 1).view(n, 32) << 4)
        code = code.double()
        if self.wtype.endswith("_1"):
            return (code * d + b[:, 2:4].contiguous().view(torch.float16).double()).view(self.rows, self.cols)
        return ((code - (16 if self.wtype == "q5_0" else 8)) * d).view(self.rows, self.cols)


def _gpt2_tensors(case):
    """State-dict key -> _Matrix or fp32 tensor, the same at every call."""
    p, gen = synthetic.GPT2_SIZES[case["model"]], _generator(7)
    d, T = p.dim, case["context"] + case["tokens"] + 7
    vec = lambda n, mean: mean + 0.1 * torch.randn(n, generator=gen, device=DEV)
    mat = lambda rows, cols: _Matrix(gen, rows, cols, case["wtype"])
    sd = {"wte.weight": 0.02 * torch.randn(p.vocab_size, d, generator=gen, device=DEV), "wpe.weight": 0.02 * torch.randn(T, d, generator=gen, device=DEV)}
    for i in range(p.n_layers):
        for n, rows, cols in (("attn.c_attn", 3 * d, d), ("attn.c_proj", d, d), ("mlp.c_fc", 4 * d, d), ("mlp.c_proj", d, 4 * d)):
            sd[f"h.{i}.{n}.weight"], sd[f"h.{i}.{n}.bias"] = mat(rows, cols), vec(rows, 0.0)
        for n in ("ln_1", "ln_2"):
            sd[f"h.{i}.{n}.affine"], sd[f"h.{i}.{n}.bias"] = vec(d, 1.0), vec(d, 0.0)
    sd["ln_f.affine"], sd["ln_f.bias"], sd["lm_head.weight"] = vec(d, 1.0), vec(d, 0.0), mat(p.vocab_size, d)
    return sd, T


class _Gpt2:
    def __init__(self, case, seed):
        p = synthetic.GPT2_SIZES[case["model"]]
        sd, T = _gpt2_tensors(case)
        torch.cuda.synchronize()
        blobs = {k: (v.data if isinstance(v, _Matrix) else v).data_ptr() for k, v in sd.items()}
        rt = _runtime()
        self.model = m = GPT2(rt, p, sd, max_seq_len=T, batch=case["batch"], precision=case["precision"], device_blobs=blobs)
        rt.sync()
        del sd
        torch.cuda.empty_cache()
        B, self.n, self.s = case["batch"], case["context"], case["tokens"]
        ids = _tokens(seed, B, self.n + self.s, p.vocab_size).cpu().numpy()
        if self.n:
            m.forward(ids[:, :self.n], self.n, 0)
        self.ids = np.ascontiguousarray(ids[:, self.n:])
        self.out = {"logits": _view(m, m._logits_ptr(), (B, p.vocab_size))}
        k, v = ctypes.c_void_p(), ctypes.c_void_p()
        L.check(rt.ctx, rt.lib.caten_b200_gpt2_kv(m._h, p.n_layers - 1, ctypes.byref(k), ctypes.byref(v)))
        for name, ptr in (("k", k), ("v", v)):   # the rows that this step appends to the last layer's caches
            self.out[name] = _view(m, ptr.value, (B, p.n_heads, T, 64))[:, :, self.n:self.n + self.s]
        self.keep_ids = case["precision"] != "bf16"   # at that precision near ties go either way

    def run(self):
        ids = self.model.forward(self.ids, self.s, self.n)
        return {**self.out, "ids": ids} if self.keep_ids else dict(self.out)


def _layer_norm(x, g, b):
    return torch.nn.functional.layer_norm(x, x.shape[-1:], g.double(), b.double(), 1e-5)


def _exact_gpt2(case, seed):
    p = synthetic.GPT2_SIZES[case["model"]]
    B, n, s, H = case["batch"], case["context"], case["tokens"], p.n_heads
    S, weights = n + s, 1.3e-8 * p.n_layers * p.dim ** 2   # seconds per 500 tokens, about
    if weights * B * S / 500 > 15:
        return None
    ids, (sd, _) = _tokens(seed, B, S, p.vocab_size), _gpt2_tensors(case)
    mask = torch.ones(S, S, device=DEV, dtype=torch.bool).tril()
    lin = lambda x, w, b: x @ w.T + b.double()
    x = sd["wte.weight"][ids].double() + sd["wpe.weight"][:S].double()
    step = max(1, 8192 // S)   # sequences at once
    for i in range(p.n_layers):
        t = {k[len(f"h.{i}."):]: v for k, v in sd.items() if k.startswith(f"h.{i}.")}
        w = {k: v.double() for k, v in t.items() if isinstance(v, _Matrix)}
        kept = []
        for b in range(0, B, step):
            y = x[b:b + step]
            q, k, v = lin(_layer_norm(y, t["ln_1.affine"], t["ln_1.bias"]), w["attn.c_attn.weight"], t["attn.c_attn.bias"]).view(
                y.shape[0], S, 3, H, 64).permute(2, 0, 3, 1, 4)
            a = torch.softmax((q @ k.transpose(-1, -2) * 0.125).masked_fill(~mask, -math.inf), -1) @ v
            y = y + lin(a.transpose(1, 2).reshape(y.shape), w["attn.c_proj.weight"], t["attn.c_proj.bias"])
            h = torch.nn.functional.gelu(lin(_layer_norm(y, t["ln_2.affine"], t["ln_2.bias"]), w["mlp.c_fc.weight"], t["mlp.c_fc.bias"]), approximate="tanh")
            x[b:b + step] = y + lin(h, w["mlp.c_proj.weight"], t["mlp.c_proj.bias"])
            if i == p.n_layers - 1:
                kept.append((k[:, :, n:], v[:, :, n:]))
    logits = _layer_norm(x[:, -1], sd["ln_f.affine"], sd["ln_f.bias"]) @ sd["lm_head.weight"].double().T
    out = {"logits": logits, "k": torch.cat([a for a, _ in kept]), "v": torch.cat([a for _, a in kept])}
    return {**out, "ids": None} if case["precision"] != "bf16" else out


def _work_gpt2(case):
    p = synthetic.GPT2_SIZES[case["model"]]
    B, n, s, d = case["batch"], case["context"], case["tokens"], p.dim
    per = BLOCKS[case["wtype"]][1] / 32 if case["wtype"] in BLOCKS else DENSE[case["wtype"]][1].itemsize
    mats, head, rows = 12 * p.n_layers * d * d, p.vocab_size * d, B * s
    pairs = B * sum(n + i + 1 for i in range(s))   # (query, key)
    return {"bytes": (mats + head) * per + 8 * p.n_layers * d * B * (n + s) + 8 * rows * d + 4 * B * p.vocab_size,
            "flops": 2 * rows * mats + 2 * B * head + 4 * p.n_layers * d * pairs}


# ---- layer-list decoders --------------------------------------------------------------------------
def _rms(x, eps=1e-5):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


class _Draw:
    """Random bf16 tensors by name, on the GPU."""

    def __init__(self):
        self.gen, self.t = _generator(11), {}

    def mat(self, name, rows, cols, gain=1.0):
        self.t[name] = (torch.randn(rows, cols, generator=self.gen, device=DEV) * (gain * cols ** -0.5)).bfloat16()

    def vec(self, name, shape, mean, std):
        self.t[name] = (mean + std * torch.randn(shape, generator=self.gen, device=DEV)).bfloat16()


def _binusun_tensors(width):
    z, r = BINUSUN[width], _Draw()
    H, G, D, E = z["heads"], z["kv_heads"], z["dim"], z["vdim"]
    hd = z["wkv_heads"] * z["wkv_dim"]
    r.mat("embed", VOCAB, width, width ** 0.5)
    for i, c in enumerate(z["order"]):
        pre = f"l{i}."
        for n in ("norm1", "norm1b") + (("norm2", "norm2b") if c.isupper() else ()):
            r.vec(pre + n, (), 1.0, 0.1)
        if c in "aA":
            for n, rows in (("q", H * D), ("k", G * D), ("v", G * E), ("g", H)):
                r.mat(pre + "mix." + n, rows, width)
            r.mat(pre + "mix.o", width, H * E)
        else:
            for n in "rkvgw":
                r.vec(pre + "mix.mu." + n, (width,), 0.5, 0.25)
            for n in "rkvg":
                r.mat(pre + "mix." + n, hd, width)
            r.mat(pre + "mix.w1", LOW_RANK, width)
            r.mat(pre + "mix.w2", hd, LOW_RANK)
            r.vec(pre + "mix.w0", (hd,), -2.0, 1.5)
            r.vec(pre + "mix.u", (z["wkv_heads"], z["wkv_dim"]), 0.0, 0.5)
            r.vec(pre + "mix.norm", (hd,), 1.0, 0.1)
            r.mat(pre + "mix.o", width, hd)
        if c.isupper():
            for n, rows, cols in (("gate", z["ff"], width), ("up", z["ff"], width), ("down", width, z["ff"])):
                r.mat(pre + "mlp." + n, rows, cols)
    r.vec("final.norm", (), 1.0, 0.1)
    r.mat("head", VOCAB, width)
    return r.t


def _goselix_tensors(width):
    z, r = GOSELIX[width], _Draw()

    def glu(pre, ff):
        for n, rows, cols in (("gate", ff, width), ("up", ff, width), ("down", width, ff)):
            r.mat(pre + n, rows, cols)

    # tokens of as many kinds as there are experts, and routers that know them, as trained ones do: with unrelated rows many
    # of a batch's choices are near ties, which rounding decides
    kinds = torch.nn.functional.normalize(torch.randn(z["experts"], width, generator=r.gen, device=DEV), dim=1)
    of = torch.arange(VOCAB, device=DEV) % z["experts"]
    r.t["embed"] = (torch.randn(VOCAB, width, generator=r.gen, device=DEV) + 3.0 * width ** 0.5 * kinds[of]).bfloat16()
    for i, (a, b) in enumerate(zip(z["order"][0::2], z["order"][1::2])):
        pre, mix = f"l{i}.", f"l{i}.mix."
        r.vec(pre + "norm1", (width,), 1.0, 0.1)
        r.vec(pre + "norm2", (width,), 1.0, 0.1)
        if a == "l":
            H, E, K, Q = z["heads"], z["vdim"], z["kv_rank"], z["q_rank"]
            r.mat(mix + "dq", Q, width)
            r.vec(mix + "dq.norm", (Q,), 1.0, 0.1)
            r.mat(mix + "uq", H * (z["dim"] + z["rot_dim"]), Q)
            r.mat(mix + "dkv", K + z["rot_dim"], width)
            r.vec(mix + "dkv.norm", (K,), 1.0, 0.1)
            r.mat(mix + "uk", H * z["dim"], K)
            r.mat(mix + "uv", H * E, K)
        else:
            H, E = z["ret_heads"], z["ret_vdim"]
            for n, size in (("q", z["ret_dim"]), ("k", z["ret_dim"]), ("v", E), ("g", E)):
                r.mat(mix + n, H * size, width)
        r.mat(mix + "o", width, H * E)
        if b == "d":
            glu(pre + "mlp.", z["ff"])
        else:
            rows = kinds + 0.8 * kinds.roll(-1, 0) + 0.07 * torch.randn(z["experts"], width, generator=r.gen, device=DEV) * width ** -0.5
            r.t[pre + "mlp.router"] = (rows * (4.0 * width ** -0.5)).bfloat16()
            for e in range(z["experts"]):
                glu(f"{pre}mlp.e{e}.", z["expert_ff"])
    r.vec("final.norm", (width,), 1.0, 0.1)
    r.mat("head", VOCAB, width)
    return r.t


def _decoder_config(case):
    if case["kind"] == "binusun":
        return synthetic.binusun_config(case["width"], VOCAB, **BINUSUN[case["width"]])
    return synthetic.goselix_config(case["width"], VOCAB, **GOSELIX[case["width"]])


def _decoder_tensors(case):
    return (_binusun_tensors if case["kind"] == "binusun" else _goselix_tensors)(case["width"])


@functools.lru_cache(2)
def _host_tensors(kind, width):
    """What a safetensors file holds: name -> bf16 bit patterns."""
    return {k: v.view(torch.int16).cpu().numpy().view(np.uint16) for k, v in _decoder_tensors({"kind": kind, "width": width}).items()}


class _Decoder:
    def __init__(self, case, seed):
        module, make = (binusun, binusun.Binusun) if case["kind"] == "binusun" else (goselix, goselix.Goselix)
        B, self.s, self.more = case["batch"], case["prompt"], case["decode"]
        self.model = make(_runtime(), module.parse_config(_decoder_config(case)), _host_tensors(case["kind"], case["width"]),
                          max_seq_len=self.s + self.more, batch=B, precision=case["precision"])
        ids = _tokens(seed, B, self.s + self.more, VOCAB).cpu().numpy()
        self.prompt = np.ascontiguousarray(ids[:, :self.s])
        self.next = [np.ascontiguousarray(ids[:, self.s + i:self.s + i + 1]) for i in range(self.more)]
        self.logits = None

    def run(self):
        m = self.model
        m.forward(self.prompt, self.s, 0)
        for i, tok in enumerate(self.next):   # a given continuation, so that a near tie cannot change what follows
            m.forward(tok, 1, self.s + i)
        if self.logits is None:
            self.logits = _view(m, m._logits_ptr(), (m.batch, VOCAB))
        return self.logits


def _rotate(x, base, dims, interleaved):
    """x [.., tokens, dim]: pairs turn by position * base^(-2 i / dims)."""
    if not dims:
        return x
    pos = torch.arange(x.shape[-2], device=DEV, dtype=torch.float64)
    a = pos[:, None] * base ** (-2.0 * torch.arange(dims // 2, device=DEV, dtype=torch.float64) / dims)
    c, s, r = a.cos(), a.sin(), x[..., :dims]
    u, v = (r[..., 0::2], r[..., 1::2]) if interleaved else (r[..., :dims // 2], r[..., dims // 2:])
    y = torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2) if interleaved else torch.cat([u * c - v * s, v * c + u * s], -1)
    return torch.cat([y, x[..., dims:]], -1)


def _heads(x, H):
    """[B, tokens, H * D] -> [B, H, tokens, D]"""
    return x.view(*x.shape[:2], H, -1).transpose(1, 2)


def _attend(q, k, v, scale, window):
    S = q.shape[-2]
    i = torch.arange(S, device=DEV)
    seen = i[:, None] >= i
    if window:
        seen &= i[:, None] - i < window
    out = torch.empty(*q.shape[:-1], v.shape[-1], device=DEV, dtype=q.dtype)
    for b in range(q.shape[0]):
        out[b] = torch.softmax((q[b] @ k[b].transpose(-1, -2) * scale).masked_fill(~seen, -math.inf), -1) @ v[b]
    return out


def _binusun_mixer(h, W, pre, z, attention):
    lin = lambda x, n: x @ W(pre + n).T
    if attention:
        H, G = z["heads"], z["kv_heads"]
        q, k = (_rms(_rotate(_heads(lin(h, n), c), 10000.0, z["rot_dims"], True)) for n, c in (("q", H), ("k", G)))
        v = _heads(lin(h, "v"), G)
        o = _attend(q, k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1), z["dim"] ** -0.5, z["window"])
        o = o * torch.sigmoid(_heads(lin(h, "g"), H))
        return lin(o.transpose(1, 2).flatten(2), "o")
    H = z["wkv_heads"]
    before = torch.cat([torch.zeros_like(h[:, :1]), h[:, :-1]], 1)
    mix = {c: h + (before - h) * W(pre + "mu." + c) for c in "rkvgw"}
    r, k, v = (_heads(lin(mix[c], c), H) for c in "rkv")
    w = _heads(torch.exp(-torch.exp(torch.tanh(lin(mix["w"], "w1")) @ W(pre + "w2").T + W(pre + "w0"))), H)
    u = W(pre + "u")[:, :, None]
    state = torch.zeros(h.shape[0], H, k.shape[-1], v.shape[-1], device=DEV, dtype=h.dtype)
    o = torch.empty_like(v)
    for t in range(h.shape[1]):
        kv = k[:, :, t, :, None] * v[:, :, t, None, :]
        o[:, :, t] = ((state + u * kv) * r[:, :, t, :, None]).sum(2)
        state = state * w[:, :, t, :, None] + kv
    o = _rms(o).transpose(1, 2).flatten(2) * W(pre + "norm") * torch.nn.functional.silu(lin(mix["g"], "g"))
    return lin(o, "o")


def _goselix_mixer(h, W, pre, z, latent):
    lin = lambda x, n: x @ W(pre + n).T
    if latent:
        H, D, P, K = z["heads"], z["dim"], z["rot_dim"], z["kv_rank"]
        q = _heads(lin(_rms(lin(h, "dq")) * W(pre + "dq.norm"), "uq"), H)
        q = torch.cat([q[..., :D], _rotate(q[..., D:], 10000.0, P, False)], -1)
        down = lin(h, "dkv")
        c = _rms(down[..., :K]) * W(pre + "dkv.norm")
        common = _rotate(down[:, None, :, K:], 10000.0, P, False).expand(-1, H, -1, -1)
        k = torch.cat([_heads(lin(c, "uk"), H), common], -1)
        o = _attend(q, k, _heads(lin(c, "uv"), H), (D + P) ** -0.5, 0)
        return lin(o.transpose(1, 2).flatten(2), "o")
    H, D = z["ret_heads"], z["ret_dim"]
    q, k = (_rotate(_heads(lin(h, n), H), 10000.0, z["ret_rot"], False) for n in "qk")
    v = _heads(lin(h, "v"), H)
    decay = torch.tensor([1.0 - 2.0 ** (-3 - a % 8) for a in range(H)], device=DEV, dtype=torch.float64)
    state = torch.zeros(h.shape[0], H, D, v.shape[-1], device=DEV, dtype=h.dtype)
    o = torch.empty_like(v)
    i = torch.arange(64, device=DEV, dtype=torch.float64)
    for t in range(0, h.shape[1], 64):   # S = decay S + k v^T, o = S^T q, 64 tokens at a time
        qt, kt, vt = (x[:, :, t:t + 64] for x in (q, k * D ** -0.5, v))
        n = qt.shape[2]
        far = (i[:n, None] - i[:n]).clamp(min=0)
        within = torch.where(i[:n, None] >= i[:n], decay[:, None, None] ** far, 0.0)
        o[:, :, t:t + n] = (qt @ kt.transpose(-1, -2) * within) @ vt + decay[:, None, None] ** (i[:n, None] + 1) * (qt @ state)
        state = decay[:, None, None] ** n * state + (kt * decay[:, None, None] ** (n - 1 - i[:n, None])).transpose(-1, -2) @ vt
    return lin(_rms(o).transpose(1, 2).flatten(2) * torch.nn.functional.silu(lin(h, "g")), "o")


def _experts(h, W, pre, z):
    flat = h.reshape(-1, h.shape[-1])
    score, chosen = torch.sigmoid(flat @ W(pre + "router").T).topk(z["top"], -1)
    out = torch.zeros_like(flat)
    for e in range(z["experts"]):
        row, place = (chosen == e).nonzero(as_tuple=True)
        x = flat[row] * score[row, place, None]
        out.index_add_(0, row, (torch.nn.functional.silu(x @ W(f"{pre}e{e}.gate").T) * (x @ W(f"{pre}e{e}.up").T)) @ W(f"{pre}e{e}.down").T)
    return out.view(h.shape)


def _exact_decoder(case, seed):
    B, S, width = case["batch"], case["prompt"] + case["decode"], case["width"]
    if B * S * (width / 2048) ** 2 > 16384:
        return None
    t = _decoder_tensors(case)
    W = lambda name: t[name].double()
    ids = _tokens(seed, B, S, VOCAB)
    x = t["embed"][ids].double()
    if case["kind"] == "binusun":
        z = BINUSUN[width]
        for i, c in enumerate(z["order"]):
            pre = f"l{i}."
            x = x + _rms(_binusun_mixer(_rms(x) * W(pre + "norm1"), W, pre + "mix.", z, c in "aA")) * W(pre + "norm1b")
            if c.isupper():
                h = _rms(x) * W(pre + "norm2")
                h = (torch.relu(h @ W(pre + "mlp.gate").T) * (h @ W(pre + "mlp.up").T)) @ W(pre + "mlp.down").T
                x = x + _rms(h) * W(pre + "norm2b")
    else:
        z = GOSELIX[width]
        for i, (a, b) in enumerate(zip(z["order"][0::2], z["order"][1::2])):
            pre, u = f"l{i}.", _rms(x)
            h = u * W(pre + "norm2")
            if b == "d":
                f = (torch.nn.functional.silu(h @ W(pre + "mlp.gate").T) * (h @ W(pre + "mlp.up").T)) @ W(pre + "mlp.down").T
            else:
                f = _experts(h, W, pre + "mlp.", z)
            x = x + _goselix_mixer(u * W(pre + "norm1"), W, pre + "mix.", z, a == "l") + f
    return _rms(x[:, -1]) * W("final.norm") @ W("head").T


def _work_decoder(case):
    """Weights once per call of the model (of an expert those that some row uses), caches and states once per token decoded,
    the products that the tokens need."""
    width, B, s, more = case["width"], case["batch"], case["prompt"], case["decode"]
    w = float(VOCAB * width)   # the head
    mix = pairs = cache = state = experts = used = 0.0
    if case["kind"] == "binusun":
        z = BINUSUN[width]
        for c in z["order"]:
            if c in "aA":
                w += width * (2 * z["heads"] * z["dim"] + 2 * z["kv_heads"] * z["dim"])
                pairs += 4 * z["heads"] * z["dim"]
                cache += 8 * z["kv_heads"] * z["dim"]
            else:
                hd = z["wkv_heads"] * z["wkv_dim"]
                w += 5 * width * hd + LOW_RANK * (width + hd)
                mix += 5 * hd * z["wkv_dim"]
                state += 8 * hd * z["wkv_dim"]
            w += 3 * width * z["ff"] if c.isupper() else 0
        window = z["window"]
    else:
        z = GOSELIX[width]
        H, D, P, E, K, Q = z["heads"], z["dim"], z["rot_dim"], z["vdim"], z["kv_rank"], z["q_rank"]
        for a, b in zip(z["order"][0::2], z["order"][1::2]):
            if a == "l":
                w += width * (Q + K + P + H * E) + Q * H * (D + P) + K * H * (D + E)
                pairs += 2 * H * (D + P + E)
                cache += 2 * (K + P)
            else:
                h, e = z["ret_heads"], z["ret_vdim"]
                w += width * h * (2 * z["ret_dim"] + 3 * e)
                mix += 5 * h * z["ret_dim"] * e
                state += 8 * h * z["ret_dim"] * e
            if b == "d":
                w += 3 * width * z["ff"]
            else:
                w += width * z["experts"]
                experts += 3 * width * z["expert_ff"] * z["experts"]
                used += 3 * width * z["expert_ff"] * z["top"]
        window = 0
    read = lambda rows: 2 * (w + experts * (1 - (1 - z.get("top", 0) / z.get("experts", 1)) ** rows))
    seen = lambda i: min(i + 1, window) if window else i + 1
    return {"bytes": read(B * s) + cache * B * s + sum(read(B) + B * (cache * seen(s + i) + state) for i in range(more)) + 4 * B * VOCAB * (1 + more),
            "flops": 2 * B * (s + more) * (w - VOCAB * width + used) + 2 * B * (1 + more) * VOCAB * width + B * (s + more) * mix +
            B * pairs * sum(seen(i) for i in range(s + more))}


# ---- relu(matmul) ---------------------------------------------------------------------------------
def _matmul_inputs(case, seed):
    gen, std = _generator(seed), case["k"] ** -0.5
    return (torch.randn(case["m"], case["k"], generator=gen, device=DEV) * std, torch.randn(case["k"], case["n"], generator=gen, device=DEV) * std)


class _ReluMatmul:
    def __init__(self, case, seed):
        self.case, (self.a, self.b) = case, _matmul_inputs(case, seed)
        self.c = torch.empty(case["m"], case["n"], device=DEV)

    def run(self):
        rt, z = _runtime(), self.case
        L.check(rt.ctx, rt.lib.caten_b200_relu_matmul(rt.ctx, self.a.data_ptr(), self.b.data_ptr(), self.c.data_ptr(), z["m"], z["k"], z["n"],
                                                      PRECISIONS[z["precision"]]))
        return self.c


# ---- schedule items -------------------------------------------------------------------------------
def _item_input(case, seed):
    return torch.randn(case["rows"], case["cols"], generator=_generator(seed), device=DEV) * 3


class _Items:
    """Programs and buffers are what a compiled graph keeps; a pass runs its items."""

    def __init__(self, case, seed):
        rt, R, C = _runtime(), case["rows"], case["cols"]
        self.x = _item_input(case, seed)   # kept: the buffer below only points at it
        self.y = torch.empty_like(self.x)
        buffer = lambda t: B200Buffer(rt, t.data_ptr(), t.shape, np.float32, owned=False)
        wrap = lambda t: expr.View(buffer(t))
        x, y = wrap(self.x), wrap(self.y)
        if case["what"] == "gelu":   # x / 2 (1 + tanh(sqrt(2 / pi) (x + 0.044715 x^3))), tanh through exp2
            v = expr.load(x)
            z = (v + v * v * v * 0.044715) * 0.7978845608028654
            sig = expr.recip(expr.exp2(z * 2.0 * (-1.0 / math.log(2.0))) + 1.0)
            self.items = [(expr.Program(v * 0.5 * (sig * 2.0 + (-1.0) + 1.0)), y, (R, C), 0, None)]
            return
        self.m, self.e, self.t = torch.empty(R, device=DEV), torch.empty_like(self.x), torch.empty(R, device=DEV)
        m, t = (expr.View(buffer(b), strides=(1, 0)) for b in (self.m, self.t))
        e = wrap(self.e)
        self.items = [(expr.Program(expr.load(x)), m, (R, C), 1, "max"),
                      (expr.Program(expr.exp2((expr.load(x) - expr.load(m)) * (1.0 / math.log(2.0)))), e, (R, C), 0, None),
                      (expr.Program(expr.load(e)), t, (R, C), 1, "sum"),
                      (expr.Program(expr.load(e) / expr.load(t)), y, (R, C), 0, None)]

    def run(self):
        for program, out, shape, n_reduce, op in self.items:
            expr.run(_runtime(), program, out, shape, n_reduce, op)
        return self.y


# ---- the interface --------------------------------------------------------------------------------
STATES = {"gpt2": _Gpt2, "binusun": _Decoder, "goselix": _Decoder, "relu_matmul": _ReluMatmul, "items": _Items}


def prepare(case, seed):
    state = STATES[case["kind"]](case, seed)
    torch.cuda.synchronize()   # the library queues its work on a stream of its own
    return state


def run(state):
    return state.run()


def exact(case, seed):
    if case["kind"] == "gpt2":
        return _exact_gpt2(case, seed)
    if case["kind"] in ("binusun", "goselix"):
        return _exact_decoder(case, seed)
    if case["kind"] == "relu_matmul":
        a, b = _matmul_inputs(case, seed)
        return torch.relu(a.double() @ b.double())
    x = _item_input(case, seed).double()
    return torch.softmax(x, -1) if case["what"] == "softmax" else torch.nn.functional.gelu(x, approximate="tanh")


def work(case):
    if case["kind"] == "gpt2":
        return _work_gpt2(case)
    if case["kind"] in ("binusun", "goselix"):
        return _work_decoder(case)
    if case["kind"] == "relu_matmul":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 4 * (m * k + k * n + m * n), "flops": 2 * m * k * n}
    # gelu: read, write.  softmax: max (read), exp2 (read, write), sum (read), product (read, write)
    n = case["rows"] * case["cols"]
    return {"bytes": (8 if case["what"] == "gelu" else 24) * n, "flops": (14 if case["what"] == "gelu" else 6) * n}


def tolerance(case):
    """About four times the largest error against ``exact`` that was seen in the ranges above."""
    if case["kind"] == "items":
        return {"rel": 1.5e-6}
    if case["kind"] in ("binusun", "goselix"):
        return {"rel": 0.03}
    return {"rel": {"fp32": 2e-5, "bf16x3": 1e-4, "bf16": 0.025}[case["precision"]], "differ": 0.01}
