"""Performance cases of the quantized MoE expert path: what a program that serves a Q4_K / Q4_K_M model asks of this
package, as functions that a timing harness calls (listed, draw, prepare, run, work, tolerance).

Four kinds of call:
  stack    FusedMoeStack.step: the layers of the resident stack for one decode step of 1..64 sequences
  decode   MoeFfnLayer.decode: one layer for one decode step, when attention runs between the layers
  prefill  MoeFfnLayer.prefill: one layer over the tokens of one or several prompts
  matmul   ops.q4k_matmul: one dense Q4_K matrix times activation rows

Options that files and callers bring: the down matrices in Q4_K, in Q6_K, or Q6_K in every second layer ("mixed", as
Q4_K_M files hold them); f32 or bf16 rows; uniform or Zipf(1.1) expert popularity; RMSNorm and residual inside the
call or not. Geometry "full" is hidden 2048, ffn 768, 128 experts; "small" is hidden 1024, ffn 512, 32 experts; both
route to 8 experts.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from kanjoos_b200 import ops
from kanjoos_b200.moe import ExpertBank, FusedMoeStack, MoeFfnLayer

GEOMETRY = {"full": (128, 2048, 768), "small": (32, 1024, 512)}  # experts, hidden, ffn
TOP_K = 8
DTYPE = {"f32": torch.float32, "bf16": torch.bfloat16}
ZIPF_S = 1.1


def _stack(name, tokens, layers, dtype, down, geometry="full"):
    return {"name": name, "kind": "stack", "tokens": tokens, "layers": layers, "dtype": dtype, "down": down,
            "geometry": geometry}


def _layer(name, kind, tokens, dtype, out, down, routing, norm=False, geometry="full"):
    return {"name": name, "kind": kind, "tokens": tokens, "dtype": dtype, "out": out, "down": down, "routing": routing,
            "norm": norm, "geometry": geometry}


def listed():
    return [
        # one matrix-vector product, the smallest unit of the path: launch latency
        {"name": "matmul_m1", "kind": "matmul", "m": 1, "n_out": 768, "n_in": 2048, "dtype": "f32"},
        # a dense projection over the rows of a short prompt, an odd number of them
        {"name": "matmul_m301", "kind": "matmul", "m": 301, "n_out": 2048, "n_in": 2048, "dtype": "bf16"},
        # a single user's token through one layer of a program that calls the layers itself
        _layer("decode_b1", "decode", 1, "bf16", "f32", "q4k", "uniform"),
        # a small batch through one layer of a smaller model: launches and host work weigh most
        _layer("decode_b17_small", "decode", 17, "bf16", "bf16", "q4k", "zipf", norm=True, geometry="small"),
        # a single user's token through the whole resident stack, f32 residual stream
        _stack("stack_b1", 1, 48, "f32", "q4k"),
        # a few users, the stack as Q4_K_M files hold it
        _stack("stack_b8_mixed", 8, 48, "f32", "mixed"),
        # a pipeline stage of four layers with a bf16 stream and an odd batch
        _stack("stack_b37_bf16", 37, 4, "bf16", "q4k"),
        # the largest decode batch of the stack launch
        _stack("stack_b64", 64, 12, "f32", "q4k"),
        # a short prompt: less than one token tile per expert
        _layer("prefill_t100", "prefill", 100, "bf16", "bf16", "q4k", "uniform", norm=True),
        # the usual prefill chunk with popular and rare experts
        _layer("prefill_t512_zipf", "prefill", 512, "bf16", "f32", "q4k", "zipf"),
        # a long ragged prompt over a layer with Q6_K down matrices
        _layer("prefill_t4001_q6k", "prefill", 4001, "bf16", "f32", "q6k", "zipf"),
        # many prompts at once: the largest call
        _layer("prefill_t16384", "prefill", 16384, "bf16", "bf16", "q4k", "uniform"),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng: random.Random):
    kind = rng.choice(["stack", "stack", "decode", "prefill", "prefill", "matmul"])
    if kind == "matmul":
        case = {"kind": kind, "m": _log_int(rng, 1, 512), "n_out": 16 * _log_int(rng, 16, 256),
                "n_in": 256 * _log_int(rng, 1, 16), "dtype": rng.choice(["f32", "bf16"])}
        return case
    geometry = rng.choice(["full", "full", "full", "small"])
    if kind == "stack":
        # a bf16 stream is drawn with few layers: every layer rounds it anew, and near-ties of the routing that fall
        # the other way add up with depth (an f32 stream has neither)
        tokens, dtype = _log_int(rng, 1, 64), rng.choice(["f32", "f32", "bf16"])
        layers = rng.randint(2, 4) if dtype == "bf16" else rng.randint(4, 48 if tokens <= 8 else 12)
        return {k: v for k, v in _stack("", tokens, layers, dtype, rng.choice(["q4k", "mixed"]), geometry).items() if k != "name"}
    tokens = _log_int(rng, 1, 64) if kind == "decode" else _log_int(rng, 65, 16384)
    case = _layer("", kind, tokens, rng.choice(["bf16", "bf16", "f32"]), rng.choice(["bf16", "f32"]),
                  rng.choice(["q4k", "q4k", "q6k"]), rng.choice(["uniform", "zipf"]), rng.choice([False, True]), geometry)
    return {k: v for k, v in case.items() if k != "name"}


# ------------------------------------------------------------------------------------------------------- inputs

def _random_bytes(shape, g) -> torch.Tensor:
    n = math.prod(shape)
    words = torch.empty((n + 7) // 8, dtype=torch.int64, device="cuda")
    words.random_(-2**63, None, generator=g)
    return words.view(torch.uint8)[:n].view(shape)


def _q4k(shape, g) -> torch.Tensor:
    """Q4_K superblocks [..., 144] whose weights are centred with a standard deviation of about 0.02, as those of a
    trained model are: uniform codes and sub-block scales, minima at 7.5 times the scale, d around 1.2e-4."""
    blk = _random_bytes(shape + (144,), g)
    d = (1.0 + 0.2 * torch.randn(shape, device="cuda", generator=g)) * 1.2e-4
    head = torch.stack((d, 7.5 * d), dim=-1).to(torch.float16)
    blk[..., 0:4] = head.view(torch.uint8)
    blk[..., 8:12] = blk[..., 4:8]                       # the eight 6-bit minima equal the eight 6-bit scales
    blk[..., 12:16] = (blk[..., 12:16] & 15) * 17
    return blk


def _q6k(shape, g) -> torch.Tensor:
    blk = _random_bytes(shape + (210,), g)
    d = (1.0 + 0.2 * torch.randn(shape, device="cuda", generator=g)) * 1.5e-5
    blk[..., 208:210] = d.to(torch.float16).unsqueeze(-1).view(torch.uint8)
    return blk


def _bank(geometry: str, down: str, routing: str, norm: bool, g) -> ExpertBank:
    E, H, F = GEOMETRY[geometry]
    bias = None
    if routing == "zipf":
        p = _zipf(E)[torch.randperm(E, device="cuda", generator=g).cpu().numpy()]
        bias = torch.from_numpy(np.log(p).astype(np.float32)).cuda()
    return ExpertBank(
        gate=_q4k((E, F, H // 256), g), up=_q4k((E, F, H // 256), g),
        down=_q6k((E, H, F // 256), g) if down == "q6k" else _q4k((E, H, F // 256), g),
        router=(torch.randn((E, H), device="cuda", generator=g) * 0.02).to(torch.bfloat16), router_bias=bias,
        norm_w=(1.0 + 0.02 * torch.randn(H, device="cuda", generator=g)).to(torch.bfloat16) if norm else None)


def _layer_down(case, layer: int) -> str:
    if case["down"] == "mixed":
        return "q6k" if layer % 2 else "q4k"
    return case["down"]


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    dtype = DTYPE[case["dtype"]]
    if case["kind"] == "matmul":
        return {"kind": "matmul", "w": _q4k((case["n_out"], case["n_in"] // 256), g),
                "x": torch.randn((case["m"], case["n_in"]), device="cuda", generator=g).to(dtype)}
    H = GEOMETRY[case["geometry"]][1]
    x = torch.randn((case["tokens"], H), device="cuda", generator=g).to(dtype)
    if case["kind"] == "stack":
        banks = [_bank(case["geometry"], _layer_down(case, l), "uniform", True, g) for l in range(case["layers"])]
        stack = FusedMoeStack(banks, top_k=TOP_K, n_tokens=case["tokens"], dtype=dtype)
        return {"kind": "stack", "stack": stack, "x": x}
    bank = _bank(case["geometry"], case["down"], case["routing"], case["norm"], g)
    layer = MoeFfnLayer(bank, top_k=TOP_K, max_tokens=case["tokens"], residual=case["norm"], use_norm=case["norm"])
    return {"kind": case["kind"], "layer": layer, "x": x, "out_dtype": DTYPE[case["out"]]}


# ---------------------------------------------------------------------------------------------------------- run

def run(state):
    kind = state["kind"]
    if kind == "matmul":
        return ops.q4k_matmul(state["w"], state["x"])
    if kind == "stack":
        return state["stack"].step(state["x"])
    if kind == "decode":
        return state["layer"].decode(state["x"], out_dtype=state["out_dtype"])
    return state["layer"].prefill(state["x"], out_dtype=state["out_dtype"])


# ------------------------------------------------------------------------------------------- what a pass needs

def _zipf(E: int) -> np.ndarray:
    p = np.arange(1, E + 1, dtype=np.float64) ** -ZIPF_S
    return p / p.sum()


def _distinct(E: int, tokens: int, routing: str) -> float:
    """Expected number of experts that at least one of the tokens routes to."""
    p = np.full(E, TOP_K / E) if routing == "uniform" else np.minimum(0.98, TOP_K * _zipf(E))
    return float((1.0 - (1.0 - p) ** tokens).sum())


def work(case):
    size = {"f32": 4, "bf16": 2}
    if case["kind"] == "matmul":
        m, n, k = case["m"], case["n_out"], case["n_in"]
        return {"bytes": n * (k // 256) * 144 + m * k * size[case["dtype"]] + m * n * 4, "flops": 2.0 * m * n * k}
    E, H, F = GEOMETRY[case["geometry"]]
    T = case["tokens"]
    layers = case.get("layers", 1)
    n_bytes = 0.0
    for l in range(layers):
        expert = 2 * F * (H // 256) * 144 + H * (F // 256) * (210 if _layer_down(case, l) == "q6k" else 144)
        n_bytes += _distinct(E, T, case.get("routing", "uniform")) * expert + E * H * 2
    n_bytes += T * H * (size[case["dtype"]] + size[case.get("out", case["dtype"])])
    return {"bytes": n_bytes, "flops": float(layers) * T * (6.0 * TOP_K * H * F + 2.0 * H * E)}


def tolerance(case):
    if case["kind"] == "matmul":
        return {"rel": 1e-5}   # f32 sums
    if case["kind"] == "stack":
        # bf16: every layer rounds the stream, and a rounding that falls the other way is carried on
        return {"rel": 1e-5} if case["dtype"] == "f32" else {"rel": 1e-2}
    if case["out"] == "bf16":
        return {"rel": 4e-3}   # one bf16 rounding of the result
    # decode: f32 sums; prefill: fp16 tensor-core operands, f32 sums
    return {"rel": 1e-5} if case["kind"] == "decode" else {"rel": 1e-3}
