"""Performance cases of the NVFP4 W4A16 linear layer: what a decoding or prefilling engine has it do.

Sizes are those of the repository's own benchmark (a 27B-class dense model: hidden size 5120, MLP width 17408,
attention projections 7168 x 5120 and 5120 x 6144, a BF16 lm_head of 248320 rows), their tensor-parallel shards, and
generic hidden sizes.  K is a multiple of 256 throughout, as in all of these.  Weights are NVFP4 as a checkpoint
holds them: uniform E2M1 codes, one E4M3 scale per 16 elements of a normally distributed weight (sigma 0.02), the
largest block scale of a tensor at 448; activations are BF16 ~ N(0, 1).
"""
import ctypes
import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "qwen3-27b-thor-runner_b200")
for _p in (os.getcwd() + "/qwen3-27b-thor-runner_b200", _PKG):
    if os.path.isdir(_p):
        sys.path.insert(0, _p)
        break

import nvfp4  # noqa: E402

EPS = 1e-6


def listed():
    big = {"hidden": 5120, "inter": 17408, "q": 6144, "kv": 512}
    return [
        # One projection of one decode step, called eagerly: the smallest call, all latency and launches.
        {"name": "linear_m1", "kind": "linear", "m": 1, "n": 5120, "k": 5120, "residual": False},
        # Decode of one sequence: two layers' linears, norms and SwiGLU as the engine replays them from a CUDA graph,
        # norm and SwiGLU inside the linears (rows interleaved at load time).
        {"name": "decode_m1", "kind": "decode", "m": 1, "layers": 2, "form": "fused", **big},
        # The same with three drafted tokens to verify, gate and up kept as two weights (the dual GEMV).
        {"name": "decode_m4", "kind": "decode", "m": 4, "layers": 2, "form": "dual", **big},
        # Decode of a batch of 16 sequences, plain linears over merged gate/up.
        {"name": "decode_m16", "kind": "decode", "m": 16, "layers": 2, "form": "plain", **big},
        # A call on pinned host buffers (activations in, result out), two tokens.
        {"name": "host_m2", "kind": "host", "m": 2, "n": 34816, "k": 5120, "residual": False},
        # The MLP block on a batch of a few dozen sequences, or a short prompt.
        {"name": "mlp_m40", "kind": "mlp", "m": 40, "hidden": 5120, "inter": 17408},
        # A prompt of odd length.
        {"name": "mlp_m149", "kind": "mlp", "m": 149, "hidden": 5120, "inter": 17408},
        # One prefill chunk of the engine (256 tokens) through a whole layer's linears.
        {"name": "layer_m256", "kind": "layer", "m": 256, **big},
        # A prompt of odd length that spans many tiles.
        {"name": "mlp_m1111", "kind": "mlp", "m": 1111, "hidden": 5120, "inter": 17408},
        # A long prefill, the largest work.
        {"name": "mlp_m8192", "kind": "mlp", "m": 8192, "hidden": 5120, "inter": 17408},
        # The output projection of a decode step, kept in BF16.
        {"name": "lm_head_m3", "kind": "dense", "m": 3, "n": 248320, "k": 5120},
        # A BF16 projection in prefill.
        {"name": "dense_m512", "kind": "dense", "m": 512, "n": 5120, "k": 5120},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: 1..8192 tokens, hidden sizes 2048..8192, MLP widths 2.5 to 4 times that, shards of 1/2/4/8."""
    kind = rng.choice(["linear", "linear", "decode", "decode", "host", "mlp", "mlp", "mlp", "layer", "dense"])
    hidden = 256 * rng.randint(8, 32) if rng.random() < 0.6 else 5120
    inter = 17408 if hidden == 5120 else 256 * int(round(hidden * rng.uniform(2.5, 4.0) / 256))
    shard = rng.choice([1, 1, 2, 4, 8])
    q, kv = hidden + 256 * rng.randint(0, 4), 256 * rng.randint(1, 4)
    if kind == "linear":
        n = 8 * _log_int(rng, 128, 4352) if rng.random() < 0.5 else 2 * inter // shard // 16 * 16
        return {"kind": kind, "m": _log_int(rng, 1, 1024), "n": n, "k": hidden, "residual": rng.random() < 0.5}
    if kind == "decode":
        form = rng.choice(["fused", "dual", "plain"])
        return {"kind": kind, "m": _log_int(rng, 1, 16), "layers": 2, "form": form, "hidden": hidden, "inter": inter, "q": q, "kv": kv}
    if kind == "host":
        return {"kind": kind, "m": _log_int(rng, 1, 64), "n": 16 * _log_int(rng, 128, 2176), "k": hidden, "residual": rng.random() < 0.5}
    if kind == "mlp":
        return {"kind": kind, "m": _log_int(rng, 17, 8192 if hidden <= 5120 else 2048), "hidden": hidden, "inter": max(256, inter // shard // 256 * 256)}
    if kind == "layer":
        return {"kind": kind, "m": _log_int(rng, 17, 512), "hidden": hidden, "inter": inter, "q": q, "kv": kv}
    n = 8 * _log_int(rng, 2048, 31040) if rng.random() < 0.5 else hidden
    return {"kind": kind, "m": _log_int(rng, 1, 1024), "n": n, "k": hidden}


# ---------------------------------------------------------------- inputs

class _Weight:
    """An NVFP4 weight [n, k] on the device; its own seed, its own global scale."""

    def __init__(self, gen, n, k):
        self.n, self.k = n, k
        self.packed = torch.randint(0, 256, (n, k // 2), dtype=torch.uint8, device="cuda", generator=gen)
        # the largest of 16 |N(0, 0.02)| by its distribution function, over 6: the scale of a block
        u = torch.rand((n, k // 16), device="cuda", generator=gen).clamp_(1e-6, 1 - 1e-6)
        block = torch.erfinv(u.pow_(1.0 / 16)).mul_(0.02 * math.sqrt(2.0) / 6)
        self.gs = float(torch.tensor(448.0) / block.max().cpu())
        self.scale = block.mul_(self.gs).clamp_(max=448.0).to(torch.float8_e4m3fn).view(torch.uint8)


def _acts(gen, *shape):
    return torch.randn(shape, device="cuda", generator=gen).to(torch.bfloat16)


def _norm_weight(gen, k):
    return (0.1 * torch.randn(k, device="cuda", generator=gen)).to(torch.bfloat16)


def _empty(*shape):
    return torch.empty(shape, dtype=torch.bfloat16, device="cuda")


def _handle(m, n, k):
    size = ctypes.c_size_t(0)
    nvfp4.load().nvfp4_workspace_bytes(m, n, k, ctypes.byref(size))
    return nvfp4.Handle(torch.cuda.current_device(), max(size.value, 64 << 20))


class _Layer:
    """One decoder layer's weights and norms; the attention between qkv and o is the caller's, its output an input here."""

    def __init__(self, gen, c, form="plain"):
        hidden, inter, q, kv, m = c["hidden"], c["inter"], c["q"], c["kv"], c["m"]
        self.qkv = _Weight(gen, q + 2 * kv, hidden)
        self.o = _Weight(gen, hidden, q)
        if form == "dual":
            self.gate, self.up = _Weight(gen, inter, hidden), _Weight(gen, inter, hidden)
            self.gate_out, self.up_out = _empty(m, inter), _empty(m, inter)
        else:
            self.gate_up = _Weight(gen, 2 * inter, hidden)
            self.gate_up_out = _empty(m, 2 * inter)
        self.down = _Weight(gen, hidden, inter)
        self.norm1, self.norm2 = _norm_weight(gen, hidden), _norm_weight(gen, hidden)
        self.attn = _acts(gen, m, q)
        self.qkv_out, self.x, self.act = _empty(m, q + 2 * kv), _empty(m, hidden), _empty(m, inter)


def _linear(h, A, m, w, C, residual=None):
    h.linear(A, m, w.packed, w.scale, w.gs, w.n, w.k, C, residual=residual)


def _run_layer(h, c, layer, x, normed, form):
    """x -> layer.x, through qkv, o + residual, norm, gate/up, SwiGLU, down + residual."""
    m, hidden, inter = c["m"], c["hidden"], c["inter"]
    if form == "fused":
        w = layer.qkv
        h.linear_ex(x, m, w.packed, w.scale, w.gs, w.n, w.k, layer.qkv_out, norm_weight=layer.norm1, norm_eps=EPS)
        _linear(h, layer.attn, m, layer.o, layer.x, residual=x)
        w = layer.gate_up
        h.linear_ex(layer.x, m, w.packed, w.scale, w.gs, w.n, w.k, layer.act, norm_weight=layer.norm2, norm_eps=EPS, swiglu_epilogue=True)
    else:
        h.rmsnorm(x, layer.norm1, EPS, m, hidden, normed)
        _linear(h, normed, m, layer.qkv, layer.qkv_out)
        _linear(h, layer.attn, m, layer.o, layer.x, residual=x)
        h.rmsnorm(layer.x, layer.norm2, EPS, m, hidden, normed)
        if form == "dual":
            g, u = layer.gate, layer.up
            h.linear_dual(normed, m, g.packed, g.scale, g.gs, u.packed, u.scale, u.gs, inter, hidden, layer.gate_out, layer.up_out)
            h.swiglu(layer.gate_out, layer.up_out, m, inter, layer.act)
        else:
            _linear(h, normed, m, layer.gate_up, layer.gate_up_out)
            h.swiglu(layer.gate_up_out, None, m, inter, layer.act)
    _linear(h, layer.act, m, layer.down, layer.x, residual=layer.x)


class _State:
    pass


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    s = _State()
    s.case = c = dict(case)
    kind, m = c["kind"], c["m"]
    if kind in ("linear", "host"):
        s.h = _handle(m, c["n"], c["k"])
        s.w = _Weight(gen, c["n"], c["k"])
        s.A = _acts(gen, m, c["k"])
        s.res = _acts(gen, m, c["n"]) if c["residual"] else None
        s.C = _empty(m, c["n"])
        if kind == "host":
            s.A = s.A.cpu().pin_memory()
            s.res = None if s.res is None else s.res.cpu().pin_memory()
            s.C = s.C.cpu().pin_memory()
    elif kind == "dense":
        s.h = _handle(m, c["n"], c["k"])
        s.W = _acts(gen, c["n"], c["k"]).mul_(0.02)
        s.A = _acts(gen, m, c["k"])
        s.C = _empty(m, c["n"])
    elif kind == "mlp":
        s.h = _handle(m, 2 * c["inter"], max(c["hidden"], c["inter"]))
        s.gate_up, s.down = _Weight(gen, 2 * c["inter"], c["hidden"]), _Weight(gen, c["hidden"], c["inter"])
        s.norm = _norm_weight(gen, c["hidden"])
        s.x = _acts(gen, m, c["hidden"])
        s.normed, s.gate_up_out, s.act, s.out = _empty(m, c["hidden"]), _empty(m, 2 * c["inter"]), _empty(m, c["inter"]), _empty(m, c["hidden"])
    else:
        s.h = _handle(m, 2 * c["inter"], max(c["hidden"], c["inter"], c["q"]))
        s.form = c.get("form", "plain")
        s.layers = [_Layer(gen, c, s.form) for _ in range(c.get("layers", 1))]
        s.x = _acts(gen, m, c["hidden"])
        s.normed = _empty(m, c["hidden"])
        if kind == "decode":     # a decode step is captured once and replayed for every token
            torch.cuda.synchronize()
            s.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s.graph):
                _step(s)
    return s


def _step(s):
    x = s.x
    for layer in s.layers:
        _run_layer(s.h, s.case, layer, x, s.normed, s.form)
        x = layer.x


def run(s):
    c, h = s.case, s.h
    kind, m = c["kind"], c["m"]
    if kind == "linear":
        _linear(h, s.A, m, s.w, s.C, residual=s.res)
        return s.C
    if kind == "host":
        h.linear_host(s.A, m, s.w.packed, s.w.scale, s.w.gs, s.w.n, s.w.k, s.C, residual_host=s.res)
        return s.C
    if kind == "dense":
        h.linear_bf16(s.A, m, s.W, c["n"], c["k"], s.C)
        return s.C
    if kind == "mlp":
        h.rmsnorm(s.x, s.norm, EPS, m, c["hidden"], s.normed)
        _linear(h, s.normed, m, s.gate_up, s.gate_up_out)
        h.swiglu(s.gate_up_out, None, m, c["inter"], s.act)
        _linear(h, s.act, m, s.down, s.out, residual=s.x)
        return {"act": s.act, "out": s.out}
    if kind == "decode":
        s.graph.replay()
    else:
        _step(s)
    return {"qkv": [layer.qkv_out for layer in s.layers], "x": [layer.x for layer in s.layers], "act": [layer.act for layer in s.layers]}


def work(case):
    """Bytes: every weight, activation, residual and norm once in, every output once out (intermediates of a block not counted)."""
    c = case
    m = c["m"]

    def fp4(n, k):
        return n * k // 2 + n * k // 16

    if c["kind"] in ("linear", "host"):
        n, k = c["n"], c["k"]
        return {"bytes": fp4(n, k) + 2 * m * (k + n + (n if c["residual"] else 0)), "flops": 2 * m * n * k}
    if c["kind"] == "dense":
        n, k = c["n"], c["k"]
        return {"bytes": 2 * n * k + 2 * m * (k + n), "flops": 2 * m * n * k}
    hidden, inter = c["hidden"], c["inter"]
    mlp = {"bytes": fp4(2 * inter, hidden) + fp4(hidden, inter) + 2 * hidden, "flops": 6 * m * hidden * inter}
    if c["kind"] == "mlp":
        return {"bytes": mlp["bytes"] + 2 * m * (2 * hidden + inter), "flops": mlp["flops"]}
    q, kv, layers = c["q"], c["kv"], c.get("layers", 1)
    each = mlp["bytes"] + fp4(q + 2 * kv, hidden) + fp4(hidden, q) + 2 * hidden + 2 * m * (q + q + 2 * kv + hidden + inter)
    return {"bytes": layers * each + 2 * m * hidden, "flops": layers * (mlp["flops"] + 2 * m * hidden * (2 * q + 2 * kv))}


def tolerance(case):
    """BF16 results of FP32 sums: another summation order flips some last bits, and a sequence of layers carries the flips on.
    Four times what the tensor-core and the mma.sync kernels, or split and whole tiles, differ by (against FP64 a linear is off
    by its BF16 rounding, 1.65e-3, and 1.3e-4 more)."""
    return {"rel": {"decode": 2e-2, "layer": 5e-3}.get(case["kind"], 1e-3)}
