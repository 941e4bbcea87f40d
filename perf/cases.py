"""Performance cases of the quantized matvec / matmul path: what a program that serves quantized models has it do.

A decoder's linear layers are called with one activation row per generated token, a few rows for a batch of sequences,
some tens to a few hundred for short prompts and ragged batches, and thousands for long prompts; weights come in int4,
16:32 sparse int4, int3 and int2 with groups of 64 or more.  Matrix sizes are those of the benchmark's configurations
(5120 and 13824 wide 13B-class layers, 20480 wide MLPs, 16384 x 16384) and sizes in between that are not powers of two.

Packed words drawn uniformly over 32 bits are fields drawn uniformly over their range, in every dense format.
"""
from __future__ import annotations

import math

import torch

import int4matmul_kernels_b200 as pkg
from int4matmul_kernels_b200 import sharding
from int4matmul_kernels_b200.quantize import QuantLinear

_module = None


def _int4matmul():
    global _module
    if _module is None:
        _module = pkg.load_extension()
    return _module


def _mult(name, bits, n, s, m, g, sparse=False, api="operator"):
    c = dict(kind="mult", bits=bits, n=n, s=s, m=m, g=g, sparse=sparse, api=api)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one token through the smallest matrix of a 13B-class layer: latency
        _mult("int4_m1_5120x5120", 4, 5120, 5120, 1, 128),
        # one token through the largest matrix: the bandwidth half of the headline benchmark
        _mult("int4_m1_16384x16384", 4, 16384, 16384, 1, 128),
        # the same for the 16:32 sparse format
        _mult("sparse_m1_16384x16384", 4, 16384, 16384, 1, 64, sparse=True),
        # one token, 3-bit weights
        _mult("int3_m1_20480x5120", 3, 20480, 5120, 1, 64),
        # a few sequences decoded together, through the module that a model would hold
        _mult("int4_linear_m4_5120x13824", 4, 5120, 13824, 4, 128, api="module"),
        # a batch of sequences decoded together, 2-bit weights
        _mult("int2_m16_20480x5120", 2, 20480, 5120, 16, 64),
        # a larger decoding batch or a short prompt
        _mult("int4_m48_13824x5120", 4, 13824, 5120, 48, 128),
        # a prompt of 128 tokens, 3-bit weights
        _mult("int3_m128_20480x5120", 3, 20480, 5120, 128, 64),
        # a ragged batch: odd row count, sizes that fill no tile, a group of 192
        _mult("int4_m333_5184x6976", 4, 5184, 6976, 333, 192),
        # a long prompt: the matmul half of the headline benchmark
        _mult("int4_m2048_5120x20480", 4, 5120, 20480, 2048, 128),
        # the same for the 16:32 sparse format
        _mult("sparse_m2048_5120x20480", 4, 5120, 20480, 2048, 64, sparse=True),
        # one token through whole layers (four matrices and the row norms between them): launches and the gaps between them
        dict(name="stack_2_layers_m1", kind="stack", layers=2, m=1, hidden=5120, mlp=13824, g=128),
    ]


_MOST_WEIGHTS = 16384 * 16384
_MOST_PRODUCTS = 2048 * 5120 * 20480


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    if rng.random() < 0.06:
        return dict(kind="stack", layers=rng.choice([1, 2]), m=rng.choice([1, 2, 5, 16]), hidden=64 * _log_int(rng, 16, 80),
                    mlp=64 * _log_int(rng, 40, 216), g=64)
    fmt = rng.choice([(4, False), (4, False), (4, True), (3, False), (2, False)])
    while True:
        n, s = 64 * _log_int(rng, 16, 320), 64 * _log_int(rng, 16, 320)
        m = 1 if rng.random() < 0.3 else _log_int(rng, 1, 2048)
        if n * s <= _MOST_WEIGHTS and m * n * s <= _MOST_PRODUCTS:
            break
    g = rng.choice([64, 64, 128, 128, 128, 192, 256, -1])
    return _mult(None, fmt[0], n, s, m, g, fmt[1], rng.choice(["operator", "operator", "module"]))


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed(seed * 1000003 + salt)


def _words(gen, rows, cols):
    return torch.randint(-2 ** 31, 2 ** 31, (rows, cols), dtype=torch.int32, device="cuda", generator=gen)


def _keep_masks(gen, rows, cols):
    """int32 (rows, cols): 16 of the 32 bits set, positions uniform."""
    out = torch.empty((rows, cols), dtype=torch.int32, device="cuda")
    for r in range(0, rows, 64):
        k = min(64, rows - r)
        kept = torch.rand((k, cols, 32), device="cuda", generator=gen).argsort(dim=2)[..., :16]
        bits = (torch.ones((), dtype=torch.int64, device="cuda") << kept).sum(dim=2)
        out[r:r + k] = torch.where(bits >= 2 ** 31, bits - 2 ** 32, bits).to(torch.int32)
    return out


def _weights(gen, bits, n, s, g, sparse):
    groups = 1 if g < 0 else -(-n // g)
    lo, hi = (0.002, 0.02) if bits == 4 else (0.005, 0.05)
    return dict(matrix=_words(gen, n // 16 if sparse else n * bits // 32, s),
                mask=_keep_masks(gen, n // 32, s) if sparse else None,
                scales=(torch.rand((groups, s), device="cuda", generator=gen) * (hi - lo) + lo).to(torch.float16),
                zeros=torch.randint(0, 1 << bits, (groups, s), device="cuda", generator=gen).to(torch.float16))


def _rows(gen, m, n):
    return torch.randn((1, m, n), device="cuda", generator=gen).to(torch.float16)


def _mult_inputs(case, seed):
    gen = _generator(seed, 1)
    return _weights(gen, case["bits"], case["n"], case["s"], case["g"], case["sparse"]), _rows(gen, case["m"], case["n"])


def _stack_config(case):
    return sharding.StackConfig(hidden=case["hidden"], mlp=case["mlp"], layers=case["layers"], bits=4, group_size=case["g"])


def _stack_inputs(case, seed):
    gen = _generator(seed, 2)
    h, m = case["hidden"], case["mlp"]
    layers = [{name: _weights(gen, 4, n, s, case["g"], False)
               for name, n, s in (("qkv", h, 3 * h), ("o", h, h), ("gate_up", h, 2 * m), ("down", m, h))}
              for _ in range(case["layers"])]
    return layers, _rows(gen, case["m"], h)[0]


def prepare(case, seed):
    if case["kind"] == "stack":
        layers, x = _stack_inputs(case, seed)
        stack = sharding.DecoderStack(_stack_config(case), 0, 1, "cuda", layers=0)
        stack.layers = [{name: sharding.QuantWeights(4, w["matrix"].shape[0] * 8, w["matrix"].shape[1], case["g"],
                                                     w["matrix"], w["scales"], w["zeros"]) for name, w in mats.items()}
                        for mats in layers]
        return dict(kind="stack", stack=stack, x=x)
    w, x = _mult_inputs(case, seed)
    if case["api"] == "module":
        layer = QuantLinear(case["bits"], case["n"], case["s"], case["g"], w["matrix"], w["scales"], w["zeros"], w["mask"])
        return dict(kind="module", layer=layer, x=x)
    return dict(kind="operator", bits=case["bits"], g=case["g"], s=case["s"], x=x, call=_int4matmul().quant_matmul, **w)


def run(state):
    if state["kind"] == "stack":
        return state["stack"].forward(state["x"])
    if state["kind"] == "module":
        return state["layer"](state["x"])
    x = state["x"]
    # one row adds into the output buffer, more rows overwrite it
    make = torch.zeros if x.shape[1] == 1 else torch.empty
    out = make((1, x.shape[1], state["s"]), dtype=torch.float16, device="cuda")
    state["call"](state["bits"], out, state["matrix"], x, state["scales"], state["zeros"], state["g"], state["mask"])
    return out


def _mult_work(bits, n, s, m, g, sparse):
    weights = (n // 16 if sparse else n * bits // 32) * s * 4 + ((n // 32) * s * 4 if sparse else 0)
    groups = 1 if g < 0 else -(-n // g)
    return weights + 2 * groups * s * 2 + m * n * 2 + m * s * 2, 2 * m * n * s


def work(case):
    if case["kind"] == "stack":
        h, f, m, g = case["hidden"], case["mlp"], case["m"], case["g"]
        per_layer = [_mult_work(4, a, b, m, g, False) for a, b in ((h, 3 * h), (h, h), (h, 2 * f), (f, h))]
        return {"bytes": case["layers"] * sum(b for b, _ in per_layer), "flops": case["layers"] * sum(f for _, f in per_layer)}
    b, f = _mult_work(case["bits"], case["n"], case["s"], case["m"], case["g"], case["sparse"])
    return {"bytes": b, "flops": f}


def tolerance(case):
    # one product: fp16 results (half an ulp is 2^-12 .. 2^-11 of the value) of fp32 sums; the stack rounds to fp16
    # after every matrix and every norm
    return {"rel": 3e-3} if case["kind"] == "stack" else {"rel": 8e-4}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------
def _fields(bits, matrix, mask, n, lo, hi):
    """integer fields (n, hi - lo) of columns lo .. hi, int64, and the keep flags (None for the dense formats)."""
    w = matrix[:, lo:hi].to(torch.int64) & 0xFFFFFFFF
    cols = hi - lo
    if mask is not None:
        k = (mask[:, lo:hi].to(torch.int64) & 0xFFFFFFFF).view(n // 32, 1, cols) >> torch.arange(32, device="cuda").view(1, 32, 1) & 1
        rank = k.cumsum(dim=1) - k
        pair = w.view(n // 32, 2, cols)
        word = torch.where(rank < 8, pair[:, :1], pair[:, 1:])
        return (word >> (4 * (rank & 7)) & 15).view(n, cols), k.view(n, cols)
    if bits == 3:
        w = w.view(n // 32, 3, cols)
        parts = []
        for i in range(32):
            word, off = divmod(3 * i, 32)
            v = w[:, word] >> off
            if off > 29:
                v = v | w[:, word + 1] << (32 - off)
            parts.append(v & 7)
        return torch.stack(parts, dim=1).view(n, cols), None
    per = 32 // bits
    shifts = (torch.arange(per, device="cuda") * bits).view(1, per, 1)
    return (w.view(n // per, 1, cols) >> shifts & ((1 << bits) - 1)).view(n, cols), None


def _exact_mult(w, bits, n, g, x):
    """x (m, n) float64 times the weights, which are fp16 numbers by definition: fp16((q - zero) * scale), two roundings."""
    s = w["matrix"].shape[1]
    group = torch.arange(n, device="cuda") // (n if g < 0 else g)
    out = torch.empty((x.shape[0], s), dtype=torch.float64, device="cuda")
    step = max(64, 2 ** 25 // n // 64 * 64)
    for lo in range(0, s, step):
        hi = min(s, lo + step)
        q, keep = _fields(bits, w["matrix"], w["mask"], n, lo, hi)
        v = (q.to(torch.float16) - w["zeros"][group, lo:hi]) * w["scales"][group, lo:hi]
        if keep is not None:
            v = torch.where(keep.bool(), v, torch.zeros_like(v))
        out[:, lo:hi] = x @ v.double()
    return out


def _unit_rows(v):
    return v / (v.pow(2).mean(dim=-1, keepdim=True) + 1e-6).sqrt()


def exact(case, seed):
    if case["kind"] == "stack":
        layers, x = _stack_inputs(case, seed)
        hidden, mlp, g = case["hidden"], case["mlp"], case["g"]
        h = x.double()
        y = _unit_rows(h)
        for mats in layers:
            q, k, v = _exact_mult(mats["qkv"], 4, hidden, g, y).chunk(3, dim=1)
            o = _exact_mult(mats["o"], 4, hidden, g, _unit_rows(q + k + v))
            h = _unit_rows(h + _unit_rows(o))
            gate, up = _exact_mult(mats["gate_up"], 4, hidden, g, h).chunk(2, dim=1)
            d = _exact_mult(mats["down"], 4, mlp, g, _unit_rows(gate * up))
            h = _unit_rows(h + _unit_rows(d))
            y = _unit_rows(h)
        return h
    w, x = _mult_inputs(case, seed)
    return _exact_mult(w, case["bits"], case["n"], case["g"], x[0].double()).unsqueeze(0)
