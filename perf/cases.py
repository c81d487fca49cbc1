"""The work that users of this library have it do, as cases that can be timed.

Four things are called, each through the Python surface (``weft_b200.compile`` and ``ProjectionChain``):

* ``mul_mat``     one projection: fp32 activations are quantized and multiplied with a packed weight matrix.  Up to eight
                  token rows go through ``production_mul_mat_<format>_decode`` (a decode step of one sequence or of a
                  small batch), more through the tiled form (prefill of a prompt of any length).
* ``host``        the same for one token row with the activations and results in ordinary host memory and the weights
                  on the device: a program written for the CPU runtime that moved its weights only.
* ``block``       the seven projections of a Llama-style block for one token, as one call.
* ``dequantize``  packed rows back to fp32: from one row (an embedding lookup) to a whole matrix.

Formats are those that quantized models come in: the K family, Q4_0 / Q8_0, the IQ2_XXS codebook and ternary TQ1_0.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import weft_b200 as weft
from weft_b200.formats import TQ1_POWERS, row_bytes
from weft_b200.kernels import dequantize, mul_mat, rows
from weft_b200.layers import Projection, ProjectionChain
from weft_b200.runtime import Buffer
from weft_b200.runtime.driver import Toolchain, load_library

TILED = {"Q4_K": "production_mul_mat_q4_k_staged", "IQ2_XXS": "production_mul_mat_iq2_xxs_staged"}
#: how often a format is drawn: Q4_K and the Q6_K of its mixes are what most models are shipped in
FORMATS = ("Q4_K",) * 4 + ("Q6_K",) * 3 + ("Q5_K",) * 2 + ("Q8_0",) * 2 + ("Q4_0",) * 2 + ("Q3_K", "Q2_K", "IQ2_XXS", "TQ1_0")
DECODE_ROWS = 8                          # token rows up to which a program takes the decode form
MOST_WEIGHTS = 28672 * 8192              # elements of the largest weight matrix
MOST_PRODUCTS = 512 * 14336 * 4096       # of one drawn mul_mat
MOST_DEQUANTIZED = 14336 * 4096          # elements of the largest dequantized matrix


def listed() -> list[dict]:
    return [
        # one row of a quantized token embedding: the smallest call there is
        {"name": "embedding row q4_k", "op": "dequantize", "format": "Q4_K", "n": 1, "k": 4096},
        # a whole projection back to fp32 (conversion, merging of adapters)
        {"name": "dequantize q4_k", "op": "dequantize", "format": "Q4_K", "n": 14336, "k": 4096},
        # decode of one token: a small layer, a feed-forward layer, and the low-bit layer of a 70B-shaped model
        {"name": "decode q4_0", "op": "mul_mat", "format": "Q4_0", "m": 1, "n": 4096, "k": 4096},
        {"name": "decode q4_k", "op": "mul_mat", "format": "Q4_K", "m": 1, "n": 14336, "k": 4096},
        {"name": "decode iq2_xxs 70b", "op": "mul_mat", "format": "IQ2_XXS", "m": 1, "n": 28672, "k": 8192},
        # the same feed-forward layer for a program that keeps its activations in host memory
        {"name": "decode q4_k host", "op": "host", "format": "Q4_K", "m": 1, "n": 14336, "k": 4096},
        # all projections of one block of a Llama-3-8B-shaped model, Q4_K with the Q6_K ffn_down of the common mix
        {"name": "block decode q4_k mix", "op": "block", "format": "Q4_K", "down": "Q6_K", "hidden": 4096, "kv": 1024, "ffn": 14336},
        # one step of eight sequences decoded together
        {"name": "batch of 8 q4_k", "op": "mul_mat", "format": "Q4_K", "m": 8, "n": 14336, "k": 4096},
        # a short prompt of an odd length
        {"name": "prompt of 77 q8_0", "op": "mul_mat", "format": "Q8_0", "m": 77, "n": 4096, "k": 4096},
        # full prompt batches: feed-forward up and down (the latter Q6_K in the common mix), and the ternary 70B-shaped layer
        {"name": "prefill 512 q4_k", "op": "mul_mat", "format": "Q4_K", "m": 512, "n": 14336, "k": 4096},
        {"name": "prefill 512 q6_k", "op": "mul_mat", "format": "Q6_K", "m": 512, "n": 4096, "k": 14336},
        {"name": "prefill 512 tq1_0 70b", "op": "mul_mat", "format": "TQ1_0", "m": 512, "n": 28672, "k": 8192},
    ]


def _log_uniform(rng, low: float, high: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _columns(rng, most: float) -> int:
    """K: whole 256-element records."""
    return 256 * max(2, _log_uniform(rng, 2, min(56, max(2, most // 256))))


def _rows(rng, low: int, most: float) -> int:
    """N: layer widths are multiples of 64, vocabularies and shards need not be."""
    n = _log_uniform(rng, low, max(low, most))
    return max(64, n // 64 * 64) if low >= 64 and rng.random() < 0.6 else n


def draw(rng) -> dict:
    op = rng.choice(("mul_mat",) * 7 + ("host", "block", "dequantize", "dequantize"))
    fmt = rng.choice(FORMATS)
    if op == "block":
        hidden = 256 * rng.randint(4, 20)
        return {"op": op, "format": "Q4_K", "down": rng.choice(("Q4_K", "Q6_K")), "hidden": hidden,
                "kv": max(128, hidden // rng.choice((1, 4, 8)) // 64 * 64), "ffn": 256 * rng.randint(hidden // 128, hidden // 64)}
    if op == "dequantize":
        k = _columns(rng, 14336)
        return {"op": op, "format": fmt, "n": _rows(rng, 1, min(14336, MOST_DEQUANTIZED // k)), "k": k}
    if op == "host":
        k = _columns(rng, 14336)
        return {"op": op, "format": fmt, "m": 1, "n": _rows(rng, 256, min(32768, MOST_WEIGHTS // k)), "k": k}
    kind = rng.random()
    m = 1 if kind < 0.35 else rng.randint(2, DECODE_ROWS) if kind < 0.55 else _log_uniform(rng, DECODE_ROWS + 1, 512)
    k = _columns(rng, 14336)
    most = min(32768, MOST_WEIGHTS // k, MOST_PRODUCTS // (m * k))
    return {"op": op, "format": fmt, "m": m, "n": _rows(rng, 256, most), "k": k}


# ---- inputs: packed records with every field in the range that a quantizer fills, made on the device from the seed

def _bytes(gen, *shape) -> torch.Tensor:
    return torch.randint(0, 256, shape, dtype=torch.uint8, device="cuda", generator=gen)


def _nibbles(gen, *shape) -> torch.Tensor:
    """Two bell-shaped 4-bit codes per byte (quantized normal weights crowd the middle codes)."""
    return (_bytes(gen, *shape) & 0x77) + (_bytes(gen, *shape) & 0x77) + (_bytes(gen, *shape) & 0x11)


def _pairs(gen, *shape) -> torch.Tensor:
    """Four bell-shaped 2-bit codes per byte."""
    return (_bytes(gen, *shape) & 0x55) + (_bytes(gen, *shape) & 0x55) + (_bytes(gen, *shape) & 0x55)


def _scale(gen, records: int, typical: float) -> torch.Tensor:
    """An f16 scale per record as two bytes."""
    d = (0.5 + torch.rand((records, 1), device="cuda", generator=gen)) * typical
    return d.to(torch.float16).view(torch.uint8)


def _trits(gen, records: int, count: int, digits: int) -> torch.Tensor:
    """``digits`` balanced base-3 digits per byte as the top digits of five, in the fixed-point form of TQ1_0."""
    value = torch.randint(0, 3 ** digits, (records, count), device="cuda", generator=gen) * 3 ** (5 - digits)
    return ((value * 256 + 242) // 243).to(torch.uint8)


def _records(fmt: str, gen, records: int) -> torch.Tensor:
    if fmt == "Q4_0":
        fields = [_scale(gen, records, 0.007), _nibbles(gen, records, 16)]
    elif fmt == "Q8_0":
        codes = (torch.randn((records, 32), device="cuda", generator=gen) * 42).round_().clamp_(-127, 127).to(torch.int8)
        fields = [_scale(gen, records, 0.0005), codes.view(torch.uint8)]
    elif fmt == "Q4_K":
        fields = [_scale(gen, records, 0.0002), _scale(gen, records, 0.0012), _bytes(gen, records, 12), _nibbles(gen, records, 128)]
    elif fmt == "Q5_K":
        fields = [_scale(gen, records, 0.0001), _scale(gen, records, 0.0012), _bytes(gen, records, 12), _bytes(gen, records, 32), _nibbles(gen, records, 128)]
    elif fmt == "Q6_K":
        fields = [_nibbles(gen, records, 128), _pairs(gen, records, 64), _bytes(gen, records, 16), _scale(gen, records, 0.00002)]
    elif fmt == "Q3_K":
        fields = [_bytes(gen, records, 32), _pairs(gen, records, 64), _bytes(gen, records, 12), _scale(gen, records, 0.0006)]
    elif fmt == "Q2_K":
        fields = [_bytes(gen, records, 16), _pairs(gen, records, 64), _scale(gen, records, 0.002), _scale(gen, records, 0.003)]
    elif fmt == "IQ2_XXS":
        fields = [_scale(gen, records, 0.0003), _bytes(gen, records, 64)]
    elif fmt == "TQ1_0":
        fields = [_trits(gen, records, 48, 5), _trits(gen, records, 4, 4), _scale(gen, records, 0.02)]
    else:
        raise ValueError(fmt)
    return torch.cat(fields, dim=1).contiguous()


def _weights(fmt: str, gen, n: int, k: int) -> torch.Tensor:
    return _records(fmt, gen, n * k // (32 if fmt in ("Q4_0", "Q8_0") else 256)).view(n, row_bytes(fmt, k))


def _activation(fmt: str) -> str:
    return "Q8_0" if fmt in ("Q4_0", "Q8_0") else "Q8_K"


@functools.lru_cache(maxsize=None)
def _sign_table() -> np.ndarray:
    """IQ2_XXS sign rows: seven stored bits, the eighth makes the parity even; entries +1 / -1."""
    bits = (np.arange(128)[:, None] >> np.arange(7)) & 1
    bits = np.concatenate([bits, bits.sum(1, keepdims=True) & 1], axis=1)
    return (1 - 2 * bits).astype(np.int8)


def _tables(fmt: str, gen) -> dict:
    """The tables a format's kernels take as arguments, by parameter name."""
    if fmt == "TQ1_0":
        return {"powers": torch.tensor(TQ1_POWERS, dtype=torch.int64).to(torch.uint32).cuda()}
    if fmt == "IQ2_XXS":
        grid = torch.tensor([8, 25, 43], dtype=torch.int8, device="cuda")[torch.randint(0, 3, (256, 8), device="cuda", generator=gen)]
        return {"grid": grid.contiguous(), "signs": torch.from_numpy(_sign_table()).cuda()}
    return {}


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    op, fmt = case["op"], case["format"]
    if op == "block":
        return _prepare_block(case, gen)
    n, k = case["n"], case["k"]
    w = Buffer(_weights(fmt, gen, n, k), shape=(n, k), encoding=fmt)
    tables = _tables(fmt, gen)
    if op == "dequantize":
        one = n == 1
        kernel = weft.compile(getattr(dequantize if one else rows, f"row_dequantize_{fmt.lower()}" + ("" if one else "_rows")))
        if one:
            w = Buffer(w._owner, shape=(k,), encoding=fmt)
        y = torch.zeros((k,) if one else (n, k), device="cuda")
        flat = [Buffer(t.reshape(-1)) for t in tables.values()]
        return {"call": kernel, "args": (w, *flat, Buffer(y)), "out": (y,)}
    m = case["m"]
    act = _activation(fmt)
    name = f"production_mul_mat_{fmt.lower()}_decode" if m <= DECODE_ROWS else TILED.get(fmt, f"production_mul_mat_{fmt.lower()}")
    kernel = weft.compile(getattr(mul_mat, name))
    x = torch.randn((m, k), device="cuda", generator=gen)
    xq = torch.zeros((m, row_bytes(act, k)), dtype=torch.uint8, device="cuda")
    y = torch.zeros((m, n), device="cuda")
    if op == "host":
        x, xq, y = x.cpu().numpy(), xq.cpu().numpy(), y.cpu().numpy()
    extra = [Buffer(t) if fmt == "TQ1_0" else Buffer(t, shape=tuple(t.shape), encoding="I8X8") for t in tables.values()]
    return {"call": kernel, "args": (w, Buffer(x), Buffer(xq, shape=(m, k), encoding=act), *extra, Buffer(y)), "out": (y, xq)}


def _block_shapes(case: dict) -> list[tuple[str, str, int, int]]:
    """(name, format, N, K) of the projections of one block."""
    h, kv, f, fmt = case["hidden"], case["kv"], case["ffn"], case["format"]
    return [("attn_q", fmt, h, h), ("attn_k", fmt, kv, h), ("attn_v", fmt, kv, h), ("attn_output", fmt, h, h),
            ("ffn_gate", fmt, f, h), ("ffn_up", fmt, f, h), ("ffn_down", case["down"], h, f)]


_BLOCK_INPUT = {"attn_q": "normed", "attn_k": "normed", "attn_v": "normed", "attn_output": "attention", "ffn_gate": "ffn_normed",
                "ffn_up": "ffn_normed", "ffn_down": "gated"}


def _prepare_block(case: dict, gen) -> dict:
    widths = {_BLOCK_INPUT[name]: k for name, _, _, k in _block_shapes(case)}
    x = {key: torch.randn((1, k), device="cuda", generator=gen) for key, k in widths.items()}
    xq = {key: torch.zeros((1, row_bytes("Q8_K", k)), dtype=torch.uint8, device="cuda") for key, k in widths.items()}
    steps, keep, out, seen = [], [], {}, set()
    for name, fmt, n, k in _block_shapes(case):
        w, key = _weights(fmt, gen, n, k), _BLOCK_INPUT[name]
        out[name] = torch.zeros((1, n), device="cuda")
        keep.append(w)
        steps.append(Projection(fmt, w.data_ptr(), x[key].data_ptr(), xq[key].data_ptr(), out[name].data_ptr(), n, k, reuse_xq=key in seen))
        seen.add(key)
    chain = ProjectionChain(load_library(Toolchain().resolve().compiler), steps)
    return {"call": chain.run, "args": (), "out": (out, xq), "keep": (keep, x)}


def run(state: dict):
    state["call"](*state["args"])
    return state["out"]


# ---- what a pass cannot do without

def _mul_mat_work(fmt: str, m: int, n: int, k: int, have_xq: bool = False) -> tuple[float, float]:
    xq = m * row_bytes(_activation(fmt), k)
    tables = {"IQ2_XXS": 256 * 8 + 128 * 8, "TQ1_0": 20}.get(fmt, 0)
    return n * row_bytes(fmt, k) + (0 if have_xq else 4 * m * k) + xq + tables + 4 * m * n, 2.0 * m * n * k


def work(case: dict) -> dict:
    op, fmt = case["op"], case["format"]
    if op == "dequantize":
        n, k = case["n"], case["k"]
        return {"bytes": n * row_bytes(fmt, k) + 4 * n * k, "flops": 2 * n * k}
    if op != "block":
        size, flops = _mul_mat_work(fmt, case["m"], case["n"], case["k"])
        return {"bytes": size, "flops": flops}
    total, flops, seen = 0, 0, set()
    for name, step_fmt, n, k in _block_shapes(case):
        key = _BLOCK_INPUT[name]
        size, more = _mul_mat_work(step_fmt, 1, n, k)
        if key in seen:                  # the input and its quantized form are shared
            size -= 4 * k + row_bytes("Q8_K", k)
        seen.add(key)
        total, flops = total + size, flops + more
    return {"bytes": total, "flops": flops}


def tolerance(case: dict):
    # dequantized values and activation codes are exact; dot products are exact integer sums per record, added up in fp32
    return "exact" if case["op"] == "dequantize" else {"rel": 1e-5}
