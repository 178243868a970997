"""The work this framework is used for, as cases that can be timed and compared.

A model case is a request as a serving program makes it: prompts in (host ids), greedy tokens and logits out, through Model and
KvCache. `reply` is a whole request, `decode` the continuation of running sequences. An operator case is one call of the C ABI on
device buffers, as a host with its own model code makes it: linear layers with E4M3, int8 and bf16 weights, and attention.

Weights, prompts and operands come from torch generators seeded with the case's seed. The rows of the output head are those of the
embedding (moved by one token where the two are separate tensors), and the embedding is as large as what the layers add to it, so that a
greedy pick is as decided as in a trained model and does not hang on a rounding.
"""
import math

import numpy as np
import torch

from strict_b200 import native as N
from strict_b200.kernel import Context
from strict_b200.model import CONFIGS, STACK, Model, attention_layer, gated_layer, latent_layer, retention_layer, stack_config

DEV = "cuda"


# ------------------------------------------------------------------ what is measured
def listed():
    return [
        # a short chat turn on the smallest model, fp32, one user: latency of a chain of small launches
        dict(name="gpt2 reply", kind="reply", model="gpt2-small", batch=1, prompt=128, new=32, ragged=False),
        # scoring or embedding documents with it: prompts of uneven length near its 1024 positions, no decoding
        dict(name="gpt2 prompts", kind="reply", model="gpt2-small", batch=8, prompt=901, new=0, ragged=True),
        # one user, a question of a few words, a short answer
        dict(name="qwen3-0.6b one short reply", kind="reply", model="qwen3-0.6b", batch=1, prompt=37, new=16, ragged=False),
        # the single-GPU configuration as it is specified (batch 8, prompts of 512), an eighth of its tokens
        dict(name="qwen3-0.6b batch reply", kind="reply", model="qwen3-0.6b", batch=8, prompt=512, new=32, ragged=False),
        # the flagship: running sequences of the large model, 32 continuations of one prompt of 2048 tokens
        dict(name="qwen3-8b decode", kind="decode", model="qwen3-8b", batch=32, prompt=2048, new=16),
        # documents of uneven length into the large model
        dict(name="qwen3-8b prompts", kind="reply", model="qwen3-8b", batch=4, prompt=2048, new=0, ragged=True),
        # the latent-attention design (bf16 weights, sliding window), uneven prompts and an answer
        dict(name="kipatar reply", kind="reply", model="kipatar", batch=8, prompt=1000, new=32, ragged=True),
        # the design with recurrent, retention and attention layers
        dict(name="morarax reply", kind="reply", model="morarax", batch=4, prompt=777, new=32, ragged=True),
        # a linear layer of a batched decode step, E4M3 weights, called by a host with its own model code
        dict(name="linear e4m3 decode", kind="linear", dtype="e4m3", M=32, N=14336, K=4096),
        # a linear layer over a prompt, int8 weights
        dict(name="linear int8 prompt", kind="linear", dtype="int8", M=2048, N=4096, K=4096),
        # attention of a serving batch whose sequences are between 1k and 32k tokens long
        dict(name="attention decode", kind="attn_decode", B=64, low=1024, high=32768, Hq=32, Hkv=8),
        # attention over long prompts
        dict(name="attention prompts", kind="attn_prefill", B=4, S=8192, Hq=32, Hkv=8, ragged=False),
    ]


def _log(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(step, int(round(v / step)) * step)


def draw(rng):
    kind = rng.choice(["reply"] * 8 + ["decode"] + ["linear"] * 3 + ["attn_decode", "attn_prefill"])
    if kind == "reply":
        model = rng.choice(["gpt2-small", "gpt2-small", "qwen3-0.6b", "qwen3-0.6b", "qwen3-8b", "kipatar", "morarax"])
        new = rng.choice([0, 0, _log(rng, 4, 48)])
        longest = 960 if model == "gpt2-small" else 4000
        prompt = _log(rng, 12, longest)
        rows = min(8192, 6000 if model == "qwen3-8b" else 16384)  # tokens of all prompts together
        batch = _log(rng, 1, max(1, min(32, rows // prompt)))
        return dict(kind=kind, model=model, batch=batch, prompt=prompt, new=new, ragged=batch > 1 and rng.random() < 0.6)
    if kind == "decode":
        model = rng.choice(["qwen3-0.6b", "qwen3-8b"])
        return dict(kind=kind, model=model, batch=_log(rng, 1, 32), prompt=_log(rng, 100, 2048), new=_log(rng, 4, 16))
    if kind == "linear":
        dtype = rng.choice(["e4m3", "e4m3", "int8", "bf16"])
        k = {"e4m3": 64, "int8": 128, "bf16": 8}[dtype]
        return dict(kind=kind, dtype=dtype, M=_log(rng, 1, 4096), N=_log(rng, 768, 28672, 16), K=_log(rng, 768, 14336, k))
    heads = rng.choice([(32, 8), (16, 8), (8, 8), (32, 4)])
    if kind == "attn_decode":
        high = _log(rng, 200, 32768)
        return dict(kind=kind, B=_log(rng, 1, 64), low=max(1, high // rng.choice([1, 4, 32])), high=high, Hq=heads[0], Hkv=heads[1])
    S = _log(rng, 33, 8192)
    B = _log(rng, 1, max(1, min(16, 32768 // S)))
    return dict(kind=kind, B=B, S=S, Hq=heads[0], Hkv=heads[1], ragged=B > 1 and rng.random() < 0.5)


# ------------------------------------------------------------------ models
MAX_POS = 4096


def _design(name):
    """The two designs that are described layer by layer, at the sizes bench.py --design uses beside Qwen3-0.6B."""
    q = CONFIGS["qwen3-0.6b"]
    H, D, d, ff = q["n_q_heads"], q["head_dim"], q["d_model"], q["d_ff"]
    if name == "kipatar":
        layers = [latent_layer(heads=H, dim=D, rot_dim=64, vdim=D, kv_rank=256, scale=(D + 64) ** -0.5, rot_base=1e6, window=1024,
                               kv_from=i - 1 if i % 4 == 3 else -1, d_ff=ff) for i in range(q["n_layers"])]
        return stack_config(layers, d_model=d, vocab=q["vocab"], max_pos=MAX_POS, norm_groups=8, eps=1e-6)
    make = [lambda: gated_layer(d, 8, 4, d_ff=ff),
            lambda: retention_layer(H, D, D, [1.0 - 2.0 ** (-5 - 7 * h / (H - 1)) for h in range(H)], rot_dim=D, rot_base=1e4, d_ff=ff),
            lambda: retention_layer(H, D, D, [1.0 - 2.0 ** (-5 - 7 * h / (H - 1)) for h in range(H)], rot_dim=D, rot_base=1e4, d_ff=ff),
            lambda: attention_layer(H, q["n_kv_heads"], D, D, D ** -0.5, rot_dim=D, rot_base=1e6, qk_norm=True, sink=True, gate=True, d_ff=ff,
                                    rot_scaling=dict(factor=4.0, original=4096, fast=32.0, slow=1.0))]
    return stack_config([make[i % 4]() for i in range(q["n_layers"])], d_model=d, vocab=q["vocab"], max_pos=MAX_POS, norm_groups=1, eps=1e-6,
                        shared_norm=True, layer_scale=True, residual_mult=0.5)


def _config(name):
    return dict(CONFIGS[name]) if name in CONFIGS else _design(name)


def _gen(seed, what):
    return torch.Generator(DEV).manual_seed((seed * 1000003 + what) & 0x7FFFFFFFFFFF)


def _randn(g, *shape, std=1.0, dtype=torch.float32):
    return torch.randn(shape, generator=g, device=DEV, dtype=dtype) * std


def _e4m3(g, rows, cols):
    """Random E4M3 values whose rows reach 448, as a quantiser with one scale per row leaves them."""
    q = _randn(g, rows, cols, std=105.0, dtype=torch.bfloat16).clamp_(-448, 448)
    q[torch.arange(rows, device=DEV), torch.randint(0, cols, (rows,), generator=g, device=DEV)] = 448.0
    return q.to(torch.float8_e4m3fn)


def _shapes(cfg):
    """Name -> (shape, centre, spread) of every tensor of a layer of the designs."""
    d, out = cfg["d_model"], {}
    for i, y in enumerate(cfg["layers"]):
        p, t = f"l{i}.", {}
        t["norm1"] = ((d,), 1.0, 0.1)
        if "kv_rank" in y:
            H, r = y["heads"], y["kv_rank"]
            t["mix.q"] = ((H * (y["dim"] + y["rot_dim"]), d), 0, 0.03)
            if y["kv_from"] < 0:
                t["mix.dkv"] = ((r + y["rot_dim"], d), 0, 0.03)
                t["mix.dkv.norm"] = ((r,), 1.0, 0.1)
            t["mix.uk"], t["mix.uv"] = ((H * y["dim"], r), 0, 0.06), ((H * y["vdim"], r), 0, 0.06)
            t["mix.o"] = ((d, H * y["vdim"]), 0, 0.02)
            t["norm2"] = ((d,), 1.0, 0.1)
            t["mlp.act"] = ((2,), 0.2, 0.3)
        else:
            t["ls1"], t["ls2"] = ((d,), 1.0, 0.2), ((d,), 1.0, 0.2)
            t["mlp.gate"] = ((y["d_ff"], d), 0, 0.03)
            if "width" in y:
                w, b = y["width"], y["blocks"]
                for k in ("y", "x"):
                    t["mix." + k], t[f"mix.{k}.b"] = ((w, d), 0, 0.03), ((w,), 0, 0.3)
                t["mix.conv"], t["mix.conv.b"] = ((w, y["conv"]), 0, 0.5), ((w,), 0, 0.2)
                for k in ("ra", "ri"):
                    t["mix." + k], t[f"mix.{k}.b"] = ((b, w // b, w // b), 0, 0.09), ((b, w // b), 0, 0.5)
                t["mix.lam"], t["mix.o"] = ((w,), -2.0, 1.5), ((d, w), 0, 0.03)
            else:
                H, G = y["heads"], y.get("kv_heads", y["heads"])
                t["mix.q"], t["mix.k"] = ((H * y["dim"], d), 0, 0.03), ((G * y["dim"], d), 0, 0.03)
                t["mix.v"], t["mix.o"] = ((G * y["vdim"], d), 0, 0.03), ((d, H * y["vdim"]), 0, 0.02)
                t["mix.g"] = ((H if "kv_heads" in y else H * y["vdim"], d), 0, 0.03)
        t["mlp.up"], t["mlp.down"] = ((y["d_ff"], d), 0, 0.03), ((d, y["d_ff"]), 0, 0.02)
        out.update({p + k: v for k, v in t.items()})
    return out


def _tensors(name, cfg, seed):
    """(tensor name, values) of a whole model, one after the other: its layers, then embedding and head."""
    g, d, V = _gen(seed, 1), cfg["d_model"], cfg["vocab"]
    if name == "gpt2-small":
        for i in range(cfg["n_layers"]):
            for k, n, m in (("wqkv", 3 * d, d), ("wo", d, d), ("wfc", cfg["d_ff"], d), ("wproj", d, cfg["d_ff"])):
                yield f"layers.{i}.{k}.w", _randn(g, n, m, std=0.03)
                yield f"layers.{i}.{k}.b", _randn(g, n, std=0.05)
            for k in ("norm1", "norm2"):
                yield f"layers.{i}.{k}.g", 1 + _randn(g, d, std=0.1)
                yield f"layers.{i}.{k}.b", _randn(g, d, std=0.05)
        yield "normf.g", 1 + _randn(g, d, std=0.1)
        yield "normf.b", _randn(g, d, std=0.05)
        yield "wpe", _randn(g, cfg["max_pos"], d, std=0.2)
        yield "embed", _randn(g, V, d, std=1.5)
    elif name in CONFIGS:
        nq, nkv, ff = cfg["n_q_heads"] * cfg["head_dim"], cfg["n_kv_heads"] * cfg["head_dim"], cfg["d_ff"]
        for i in range(cfg["n_layers"]):
            for k, n, m in (("wqkv", nq + 2 * nkv, d), ("wo", d, nq), ("wgu", 2 * ff, d), ("wdown", d, ff)):
                yield f"layers.{i}.{k}.q", _e4m3(g, n, m)
                yield f"layers.{i}.{k}.s", (1 + _randn(g, n, std=0.1)) * (0.02 / 105)
            for k, n in (("norm1", d), ("norm2", d), ("qnorm", cfg["head_dim"]), ("knorm", cfg["head_dim"])):
                yield f"layers.{i}.{k}.g", 1 + _randn(g, n, std=0.1)
        yield "normf.g", 1 + _randn(g, d, std=0.1)
        q = _e4m3(g, V, d)
        if not cfg["tied"]:
            yield "head.q", q.view(torch.uint8).roll(1, 0).view(torch.float8_e4m3fn)
            yield "head.s", (1 + _randn(g, V, std=0.02)) * (0.02 / 105)
        yield "embed", q.float() * 2.0 ** -5  # exact in bf16, and in E4M3 with one scale per row
    else:
        for k, (shape, centre, spread) in _shapes(cfg).items():
            yield k, (centre + _randn(g, *shape, std=spread)).to(torch.bfloat16)
        yield "final.norm", (1 + _randn(g, d, std=0.1)).to(torch.bfloat16)
        e = _randn(g, V, d, std=3.0).to(torch.bfloat16)
        yield "head", e.roll(1, 0) * 0.125
        yield "embed", e


_kept = {}


def _context():
    """The program's one context."""
    if "ctx" not in _kept:
        _kept["ctx"] = Context(0)
    return _kept["ctx"]


def _to_host(t):
    """Values of a device tensor in a pinned buffer that is used again for the next one."""
    raw = t.contiguous().view(torch.uint8).reshape(-1)
    if _kept.get("pinned") is None or _kept["pinned"].numel() < raw.numel():
        _kept["pinned"] = torch.empty(raw.numel(), dtype=torch.uint8, pin_memory=True)
    host = _kept["pinned"][:raw.numel()]
    host.copy_(raw)
    a = host.numpy()
    if t.dtype == torch.float32:
        return a.view(np.float32)
    return a.view(np.uint16) if t.dtype == torch.bfloat16 else a


class _Serving:
    """A model with its weights, a cache and the prompts of a case."""

    def __init__(self, case, seed):
        self.cfg, self.new = _config(case["model"]), case["new"]
        self.tokens, self.lens, self.first = _prompts(case, seed)
        self.model = self.kv = None
        self.model = Model(_context(), self.cfg)
        for name, t in _tensors(case["model"], self.cfg, seed):
            self.model.set_tensor(name, _to_host(t))
        room = case["prompt"] + (case["new"] + 1 if case["kind"] == "reply" else 1024)
        self.maxlen = min(room, self.cfg["max_pos"])
        self.kv = self.model.new_cache(case["batch"], self.maxlen)
        self.held = 0

    def start(self):
        self.kv.reset()
        self.kv.prefill(self.tokens, self.lens)
        self.held, self.ids = int(self.lens.max()), self.first

    def __del__(self):
        if self.kv is not None:
            self.kv.dispose()
        if self.model is not None:
            self.model.dispose()


def _prompts(case, seed):
    """Ids [batch, prompt], real lengths, and (decode cases) the token every sequence goes on with."""
    rng = np.random.default_rng([seed, 2])
    V, B, S = _config(case["model"])["vocab"], case["batch"], case["prompt"]
    if case["kind"] == "decode":  # continuations of one prompt
        tokens = np.tile(rng.integers(0, V, S, dtype=np.int32), (B, 1))
        return tokens, np.full(B, S, np.int32), rng.integers(0, V - 64, B, dtype=np.int32)
    lens = rng.integers(max(1, S // 3), S + 1, B).astype(np.int32) if case["ragged"] else np.full(B, S, np.int32)
    lens[0] = S
    return rng.integers(0, V - 64, (B, S), dtype=np.int32), lens, None


def prepare(case, seed):
    if case["kind"] == "reply":
        return "reply", _Serving(case, seed)
    if case["kind"] == "decode":
        s = _Serving(case, seed)
        s.start()
        return "decode", s
    t = _operands(case, seed)
    t["ctx"] = _context()
    if case["kind"] == "linear":
        t["y"] = torch.empty(case["M"], case["N"], device=DEV, dtype=torch.bfloat16)
    else:
        t["y"] = torch.zeros_like(t["q"])
    return case["kind"], {**t, **{k: v for k, v in case.items() if k != "kind"}}


def run(state):
    kind, s = state
    if kind == "reply":
        s.kv.reset()
        ids, logits = s.kv.prefill(s.tokens, s.lens, want_logits=True)
        if not s.new:
            return {"logits": logits}
        tokens = s.kv.generate(ids, s.new - 1)
        _, last = s.kv.decode_step(tokens[-1], want_logits=True)
        return {"logits": logits, "tokens": tokens, "last": last}
    if kind == "decode":
        if s.held + s.new > s.maxlen:  # the sequences are full: the next ones
            s.start()
        tokens = s.kv.generate(s.ids, s.new - 1)
        s.ids, logits = s.kv.decode_step(tokens[-1], want_logits=True)
        s.held += s.new
        return {"tokens": tokens, "last": logits}
    L, h, p = N.lib(), s["ctx"].h, lambda k: s[k].data_ptr()  # noqa: E731
    if kind == "linear":
        if s["dtype"] == "e4m3":
            N.check(L.strictb200_gemm_fp8w(h, s["M"], s["N"], s["K"], p("x"), p("w"), p("sw"), p("y"), 0))
        elif s["dtype"] == "int8":
            N.check(L.strictb200_gemm_int8w(h, s["M"], s["N"], s["K"], p("x"), p("w"), p("sw"), p("y")))
        else:
            N.check(L.strictb200_gemm_bf16(h, s["M"], s["N"], s["K"], p("x"), p("w"), p("y"), 0))
    elif kind == "attn_decode":
        N.check(L.strictb200_attn_decode(h, p("q"), p("k"), p("v"), p("lens"), s["B"], s["Hq"], s["Hkv"], 128, s["high"], 128 ** -0.5, p("y")))
    else:
        N.check(L.strictb200_attn_prefill(h, p("q"), p("k"), p("v"), p("lens"), None, s["B"], s["S"], s["Hq"], s["Hkv"], 128, s["S"], 128 ** -0.5, p("y")))
    return s["y"]


def _operands(case, seed):
    g = _gen(seed, 3)
    if case["kind"] == "linear":
        M, n, K = case["M"], case["N"], case["K"]
        t = {"x": _randn(g, M, K, dtype=torch.bfloat16)}
        if case["dtype"] == "e4m3":
            t["w"], t["sw"] = _e4m3(g, n, K), (1 + _randn(g, n, std=0.1)) * (0.02 / 105)
        elif case["dtype"] == "int8":
            t["w"], t["sw"] = (_randn(g, n, K, std=30.0)).round_().clamp_(-127, 127).to(torch.int8), (1 + _randn(g, n, std=0.1)) * (0.02 / 30)
        else:
            t["w"] = _randn(g, n, K, std=0.02, dtype=torch.bfloat16)
        return t
    B, Hq, Hkv = case["B"], case["Hq"], case["Hkv"]
    decode = case["kind"] == "attn_decode"
    maxlen = case["high"] if decode else case["S"]
    t = {k: _randn(g, B, Hkv, maxlen, 128, dtype=torch.bfloat16) for k in ("k", "v")}
    t["q"] = _randn(g, *((B, Hq, 128) if decode else (B, maxlen, Hq, 128)), dtype=torch.bfloat16)
    lens = torch.full((B,), maxlen, dtype=torch.int32, device=DEV)
    if decode and case["low"] < maxlen:
        lens = torch.randint(case["low"], maxlen + 1, (B,), generator=g, device=DEV, dtype=torch.int32)
    elif not decode and case["ragged"]:
        lens = torch.randint(max(1, maxlen // 3), maxlen + 1, (B,), generator=g, device=DEV, dtype=torch.int32)
        lens[0] = maxlen
    t["lens"] = lens
    return t


# ------------------------------------------------------------------ what a pass cannot do without
def _layer_elements(cfg):
    """Weights of all layers (elements) and, per layer, what one position keeps and one position's work on the kept rows costs."""
    if cfg["arch"] == STACK:
        weights = sum(int(np.prod(shape)) for shape, _, _ in _shapes(cfg).values())
        rows = []  # (elements kept per position, flops per visible position, window, floats of state, flops per token on the state)
        for y in cfg["layers"]:
            if "kv_rank" in y:
                rows.append((y["kv_rank"] + y["rot_dim"] if y["kv_from"] < 0 else 0, 2 * y["heads"] * (y["dim"] + y["rot_dim"] + y["vdim"]), y["window"], 0, 0))
            elif "kv_heads" in y:
                rows.append((y["kv_heads"] * (y["dim"] + y["vdim"]), 2 * y["heads"] * (y["dim"] + y["vdim"]), 0, 0, 0))
            elif "width" in y:
                rows.append((0, 0, 0, y["width"] * y["conv"], 8 * y["width"]))
            else:
                rows.append((0, 0, 0, y["heads"] * y["dim"] * y["vdim"], 4 * y["heads"] * y["dim"] * y["vdim"]))
        return weights, rows
    d, D, H, G, ff = cfg["d_model"], cfg["head_dim"], cfg["n_q_heads"], cfg["n_kv_heads"], cfg["d_ff"]
    per = d * (H + 2 * G) * D + d * H * D + (3 if cfg["rope_theta"] else 2) * d * ff
    return cfg["n_layers"] * per, [(2 * G * D, 4 * H * D, 0, 0, 0)] * cfg["n_layers"]


def _seen(first, n, window):
    """Sum over n positions from `first` on of the positions each sees."""
    if not window:
        return n * first + n * (n + 1) // 2
    return sum(min(first + i + 1, window) for i in range(n))


def work(case):
    if case["kind"] == "linear":
        M, n, K = case["M"], case["N"], case["K"]
        w = 2 if case["dtype"] == "bf16" else 1
        return {"bytes": w * n * K + 2 * M * K + 2 * M * n + (0 if w == 2 else 4 * n), "flops": 2 * M * n * K}
    if case["kind"].startswith("attn"):
        B, Hq, Hkv = case["B"], case["Hq"], case["Hkv"]
        if case["kind"] == "attn_decode":
            keys = B * (case["low"] + case["high"]) / 2
            return {"bytes": keys * Hkv * 512 + B * Hq * 512, "flops": 4 * keys * Hq * 128}
        mean = 2 / 3 if case["ragged"] else 1.0
        square = (1 + 1 / 3 + 1 / 9) / 3 if case["ragged"] else 1.0
        return {"bytes": B * case["S"] * mean * (Hkv * 512 + Hq * 512), "flops": 2 * B * Hq * 128 * case["S"] ** 2 * square}
    cfg = _config(case["model"])
    weights, rows = _layer_elements(cfg)
    esz = 4 if case["model"] == "gpt2-small" else 2  # bytes of a cache element
    wsz = {"gpt2-small": 4, "qwen3-0.6b": 1, "qwen3-8b": 1}.get(case["model"], 2)
    V, d, B, S, new = cfg["vocab"], cfg["d_model"], case["batch"], case["prompt"], case["new"]
    pass_bytes = wsz * (weights + V * d)
    lens = [S] * B
    if case.get("ragged"):
        lens = [S] + [2 * S // 3] * (B - 1)
    bytes_ = flops = 0
    if case["kind"] == "reply":
        bytes_ += pass_bytes + sum(lens) * esz * sum(r[0] for r in rows) + 4 * B * V
        flops += 2 * sum(lens) * weights + 2 * B * V * d
        flops += sum(r[1] * sum(_seen(0, n, r[2]) for n in lens) + r[4] * sum(lens) for r in rows)
    for i in range(new):
        bytes_ += pass_bytes
        for n in lens:
            bytes_ += sum(esz * r[0] * min(n + i + 1, r[2] or n + i + 1) + 8 * r[3] for r in rows)
            flops += sum(r[1] * min(n + i + 1, r[2] or n + i + 1) + r[4] for r in rows)
        flops += 2 * B * (weights + V * d)
    return {"bytes": bytes_ + 4 * B * V, "flops": flops}


# Four times the distance to the same in 64 bits, which is what two orders of the sums, or two sets of bf16 roundings that fall
# the other way, can put between two results (0.03 where that is more).
_REL = {"gpt2-small": 2e-6, "qwen3-0.6b": 0.01, "qwen3-8b": 0.03, "kipatar": 0.016, "morarax": 0.012}


def tolerance(case):
    if case["kind"] == "linear":
        return {"rel": 4e-3, "max": 2e-2}  # one rounding to bf16
    if case["kind"].startswith("attn"):
        return {"rel": 5e-3, "max": 5e-2}
    rel = _REL[case["model"]]
    return {"rel": rel, "max": 25 * rel}  # logits: normal errors, the largest of millions


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    if case["kind"] == "linear":
        t = _operands(case, seed)
        y = t["x"].double() @ t["w"].to(torch.float32).double().T
        return y * t["sw"].double() if "sw" in t else y
    if case["kind"].startswith("attn"):
        return _exact_attention(case, _operands(case, seed))
    cfg = _config(case["model"])
    w = dict(_tensors(case["model"], cfg, seed))
    tokens, lens, first = _prompts(case, seed)
    tokens, lens = torch.from_numpy(tokens).to(DEV).long(), torch.from_numpy(lens).to(DEV).long()
    new, B = case["new"], len(lens)
    step = 0 if cfg["arch"] != STACK and cfg["tied"] else 1  # what a pick adds to the token before it
    tail = torch.arange(new + 1, device=DEV) * step
    if case["kind"] == "decode":
        prefix, rows = tokens[0], torch.from_numpy(first).to(DEV).long()[:, None] + tail[None, :new]
        at = torch.zeros(B, dtype=torch.long, device=DEV)
    else:
        prefix, rows = tokens[0, :0], torch.zeros(B, int(lens.max()) + new, dtype=torch.long, device=DEV)
        for b in range(B):
            n = int(lens[b])
            rows[b, :n] = tokens[b, :n]
            rows[b, n:n + new] = tokens[b, n - 1] + tail[1:]
        at = lens - 1
    x = _exact_stack(cfg, w, rows) if cfg["arch"] == STACK else _exact_decoder(cfg, w, prefix, rows)
    steps = at[:, None] + torch.arange(new + (case["kind"] == "reply"), device=DEV)[None, :]
    logits = _exact_head(cfg, w, x[torch.arange(B, device=DEV)[:, None], steps])  # [B, steps, vocab]
    picks = logits.argmax(-1).int()
    if case["kind"] == "reply" and not new:
        return {"logits": logits[:, 0]}
    if not torch.equal(picks[:, :-1].long(), rows.gather(1, steps)[:, 1:]):
        return None  # a pick is not the token that was taken for granted
    if case["kind"] == "decode":
        return {"tokens": picks[:, :-1].T, "last": logits[:, -1]}
    return {"logits": logits[:, 0], "tokens": picks[:, 1:-1].T, "last": logits[:, -1]}


def _exact_attention(case, t):
    B, Hq, G = case["B"], case["Hq"], case["Hq"] // case["Hkv"]
    out = torch.zeros(t["q"].shape, dtype=torch.float64, device=DEV)
    for b in range(B):
        n = int(t["lens"][b])
        for h in range(case["Hkv"]):
            k, v = t["k"][b, h, :n].double(), t["v"][b, h, :n].double()
            if case["kind"] == "attn_decode":
                out[b, h * G:(h + 1) * G] = torch.softmax(t["q"][b, h * G:(h + 1) * G].double() @ k.T * 128 ** -0.5, -1) @ v
                continue
            mask = torch.ones(n, n, dtype=torch.bool, device=DEV).triu(1)
            for a in range(h * G, (h + 1) * G):
                s = (t["q"][b, :n, a].double() @ k.T * 128 ** -0.5).masked_fill_(mask, -math.inf)
                out[b, :n, a] = torch.softmax(s, -1) @ v
    return out


def _weight(w, name):
    """[outputs, inputs] of a linear layer in 64 bits."""
    if name + ".q" in w:
        return w[name + ".q"].float().double() * w[name + ".s"].double()[:, None]
    return w[name + ".w" if name + ".w" in w else name].double()


def _rms(x, eps, groups=1):
    g = x.reshape(*x.shape[:-1], groups, -1)
    return (g * torch.rsqrt(g.square().mean(-1, keepdim=True) + eps)).reshape(x.shape)


def _layer_norm(x, w, name, eps):
    x = x - x.mean(-1, keepdim=True)
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w[name + ".g"].double() + w[name + ".b"].double()


def _exact_head(cfg, w, x):
    if cfg["arch"] == STACK:
        return (_rms(x, cfg["eps"], cfg["norm_groups"]) * w["final.norm"].double()) @ w["head"].double().T * cfg["logit_scale"]
    if not cfg["rope_theta"]:
        return _layer_norm(x, w, "normf", cfg["eps"]) @ w["embed"].double().T
    h = _rms(x, cfg["eps"]) * w["normf.g"].double()
    return h @ (w["embed"].double() if cfg["tied"] else _weight(w, "head")).T


def _rotate_half(x, pos, freq, gain=1.0):
    """x [..., positions, heads, n]: entry i turns with entry i + n/2."""
    a = pos.double()[:, None] * freq[None]
    c, s = (gain * a.cos())[:, None], (gain * a.sin())[:, None]
    u, v = x.chunk(2, -1)
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _softmax_attention(q, k, v, scale, first, window=0, sink=False):
    """One sequence: q [T, H, n] at positions first.. over k, v [K, G, n] of positions 0..; a few heads at a time."""
    T, H, K, G = q.shape[0], q.shape[1], k.shape[0], k.shape[1]
    i, j = first + torch.arange(T, device=DEV)[:, None], torch.arange(K, device=DEV)[None]
    hidden = (j > i) | (i - j >= window) if window else j > i
    out = []
    for a in range(G):
        s = torch.einsum("thd,kd->htk", q[:, a * (H // G):(a + 1) * (H // G)], k[:, a]) * scale
        s.masked_fill_(hidden, -math.inf)
        if sink:
            s = torch.cat([s, torch.zeros_like(s[..., :1])], -1)
            out.append(torch.einsum("htk,kd->thd", torch.softmax(s, -1)[..., :-1], v[:, a]))
        else:
            out.append(torch.einsum("htk,kd->thd", torch.softmax(s, -1), v[:, a]))
    return torch.cat(out, 1)


def _exact_decoder(cfg, w, prefix, rows):
    """GPT-2 and Qwen3: hidden rows [B, n, d] of `rows`, each sequence behind the same prefix."""
    P, (B, n), d, D, H, G = len(prefix), rows.shape, cfg["d_model"], cfg["head_dim"], cfg["n_q_heads"], cfg["n_kv_heads"]
    ids = torch.cat([prefix, rows.reshape(-1)])
    pos = torch.cat([torch.arange(P, device=DEV), (P + torch.arange(n, device=DEV)).repeat(B)])
    x = w["embed"][ids].double()
    rope = cfg["rope_theta"]
    if rope:
        freq = rope ** (-2.0 * torch.arange(D // 2, device=DEV, dtype=torch.float64) / D)
    else:
        x = x + w["wpe"][pos].double()
    for i in range(cfg["n_layers"]):
        p = f"layers.{i}."
        g = lambda k: w[p + k].double()  # noqa: E731, B023
        h = _rms(x, cfg["eps"]) * g("norm1.g") if rope else _layer_norm(x, w, p + "norm1", cfg["eps"])
        y = h @ _weight(w, p + "wqkv").T + (0 if rope else g("wqkv.b"))
        q, k, v = y.split([H * D, G * D, G * D], -1)
        q, k, v = q.reshape(-1, H, D), k.reshape(-1, G, D), v.reshape(-1, G, D)
        if rope:
            q = _rotate_half(_rms(q, cfg["eps"]) * g("qnorm.g"), pos, freq)
            k = _rotate_half(_rms(k, cfg["eps"]) * g("knorm.g"), pos, freq)
        att = []
        if P:
            att.append(_softmax_attention(q[:P], k[:P], v[:P], D ** -0.5, 0))
        for b in range(B):
            r = slice(P + b * n, P + (b + 1) * n)
            att.append(_softmax_attention(q[r], torch.cat([k[:P], k[r]]), torch.cat([v[:P], v[r]]), D ** -0.5, P))
        x = x + torch.cat(att).reshape(-1, H * D) @ _weight(w, p + "wo").T + (0 if rope else g("wo.b"))
        if rope:
            h = _rms(x, cfg["eps"]) * g("norm2.g")
            gate, up = (h @ _weight(w, p + "wgu").T).chunk(2, -1)
            x = x + (torch.nn.functional.silu(gate) * up) @ _weight(w, p + "wdown").T
        else:
            h = torch.nn.functional.gelu(_layer_norm(x, w, p + "norm2", cfg["eps"]) @ _weight(w, p + "wfc").T + g("wfc.b"), approximate="tanh")
            x = x + h @ _weight(w, p + "wproj").T + g("wproj.b")
    return x[P:].reshape(B, n, d)


def _yarn(y):
    """Angular steps of the rotated pairs and the factor on cos and sin."""
    n, base, gain = y["rot_dim"], y["rot_base"], 1.0
    f = base ** (-2.0 * torch.arange(n // 2, device=DEV, dtype=torch.float64) / n)
    if y["rot_factor"] > 0:
        at = lambda t: n * math.log(y["rot_original"] / (2 * math.pi * t)) / (2 * math.log(base))  # noqa: E731
        lo, hi = max(math.floor(at(y["rot_fast"])), 0), min(math.ceil(at(y["rot_slow"])), n - 1)
        ramp = ((torch.arange(n // 2, device=DEV, dtype=torch.float64) - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f, gain = f / y["rot_factor"] * ramp + f * (1 - ramp), 0.1 * math.log(y["rot_factor"]) + 1.0
    return f, gain


def _exact_latent(y, i, g, h, kept, eps):
    B, T, H = h.shape[0], h.shape[1], y["heads"]
    pos = torch.arange(T, device=DEV).double()
    r = y["rot_dim"]
    a = pos[:, None] * y["rot_base"] ** (-2.0 * torch.arange(r // 2, device=DEV, dtype=torch.float64) / r)[None]

    def turn(x):  # [B, T, ..., r]: dimension 2i with 2i + 1
        c, s = (t.reshape(T, *([1] * (x.ndim - 3)), r // 2) for t in (a.cos(), a.sin()))
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).reshape(x.shape)

    if y["kv_from"] < 0:
        t = h @ g("mix.dkv").T
        kept[i] = _rms(t[..., :y["kv_rank"]], eps) * g("mix.dkv.norm"), turn(t[..., y["kv_rank"]:])
    latent, k_rot = kept[i if y["kv_from"] < 0 else y["kv_from"]]
    q = (h @ g("mix.q").T).reshape(B, T, H, -1)
    q = torch.cat([q[..., :y["dim"]], turn(q[..., y["dim"]:])], -1)
    k = torch.cat([(latent @ g("mix.uk").T).reshape(B, T, H, -1), k_rot[:, :, None].expand(-1, -1, H, -1)], -1)
    v = (latent @ g("mix.uv").T).reshape(B, T, H, -1)
    return torch.stack([_softmax_attention(q[b], k[b], v[b], y["scale"], 0, y["window"]) for b in range(B)]).reshape(B, T, -1)


def _exact_gated(y, g, h):
    T, w, b = h.shape[1], y["width"], y["blocks"]
    gate = torch.nn.functional.gelu(h @ g("mix.y").T + g("mix.y.b"), approximate="tanh")
    x, taps = h @ g("mix.x").T + g("mix.x.b"), g("mix.conv")
    padded = torch.nn.functional.pad(x, (0, 0, y["conv"] - 1, 0))
    u = sum(padded[:, k:k + T] * taps[:, k] for k in range(y["conv"])) + g("mix.conv.b")
    blocks = u.reshape(*u.shape[:-1], b, w // b)
    r, i = (torch.sigmoid((torch.einsum("btgi,goi->btgo", blocks, g("mix." + k)) + g(f"mix.{k}.b")).reshape(u.shape)) for k in ("ra", "ri"))
    log_a = -8.0 * r * torch.nn.functional.softplus(g("mix.lam"))
    a, z = log_a.exp(), torch.sqrt(-torch.expm1(2 * log_a)) * i * u
    s, out = torch.zeros_like(u[:, 0]), torch.empty_like(u)
    for t in range(T):
        s = a[:, t] * s + z[:, t]
        out[:, t] = s
    return out * gate


def _exact_retention(y, g, h, eps):
    B, T, H = h.shape[0], h.shape[1], y["heads"]
    pos = torch.arange(T, device=DEV)
    f, gain = _yarn(y)
    q = _rotate_half((h @ g("mix.q").T).reshape(B, T, H, -1), pos, f, gain)
    k = _rotate_half((h @ g("mix.k").T).reshape(B, T, H, -1), pos, f, gain) * y["dim"] ** -0.5
    v = (h @ g("mix.v").T).reshape(B, T, H, -1)
    back = (pos[:, None] - pos[None]).double()
    out = torch.empty_like(v)
    for a in range(H):
        decay = torch.where(back >= 0, y["decay"][a] ** back.clamp(min=0), 0.0)
        out[:, :, a] = (q[:, :, a] @ k[:, :, a].transpose(1, 2) * decay) @ v[:, :, a]
    return _rms(out, eps).reshape(B, T, -1) * torch.nn.functional.silu(h @ g("mix.g").T)


def _exact_heads(y, g, h, eps):
    B, T, H, G = h.shape[0], h.shape[1], y["heads"], y["kv_heads"]
    pos = torch.arange(T, device=DEV)
    f, gain = _yarn(y)
    q = _rms(_rotate_half((h @ g("mix.q").T).reshape(B, T, H, -1), pos, f, gain), eps)
    k = _rms(_rotate_half((h @ g("mix.k").T).reshape(B, T, G, -1), pos, f, gain), eps)
    v = (h @ g("mix.v").T).reshape(B, T, G, -1)
    o = torch.stack([_softmax_attention(q[b], k[b], v[b], y["scale"], 0, sink=True) for b in range(B)])
    return (o * torch.sigmoid(h @ g("mix.g").T)[..., None]).reshape(B, T, -1)


def _exact_stack(cfg, w, rows):
    """The two designs: hidden rows [B, n, d]."""
    x, kept, eps, m = w["embed"][rows].double(), {}, cfg["eps"], cfg["residual_mult"]
    for i, y in enumerate(cfg["layers"]):
        g = lambda k: w[f"l{i}.{k}"].double()  # noqa: E731, B023
        h = _rms(x, eps, cfg["norm_groups"]) * g("norm1")
        if "kv_rank" in y:
            o = _exact_latent(y, i, g, h, kept, eps) @ g("mix.o").T
            z = (_rms(x, eps, cfg["norm_groups"]) * g("norm2")) @ g("mlp.up").T
            p, q = torch.nn.functional.softplus(g("mlp.act"))
            low = z.clamp(max=0)
            ff = torch.where(z > 0, p * z * z, (0.5 + q) * (torch.expm1(low) - low)) + z / 2
            x = x + o + ff @ g("mlp.down").T
            continue
        o = _exact_gated(y, g, h) if "width" in y else _exact_heads(y, g, h, eps) if "kv_heads" in y else _exact_retention(y, g, h, eps)
        ff = (h @ g("mlp.gate").T).relu() * (h @ g("mlp.up").T)
        x = x + m * (g("ls1") * (o @ g("mix.o").T) + g("ls2") * (ff @ g("mlp.down").T))
    return x
