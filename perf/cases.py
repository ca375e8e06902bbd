"""The calls whose speed is followed from version to version: what a serving program asks of this library, through the
entry points it would use - a routed layer at decode and at prompt sizes, with affine 4-bit and with EXL3 experts, and
the dense 4-bit and EXL3 projections beside it.

A case is a dict of plain values; ``kind`` says which entry point it takes:

``layer``   one routed layer on affine 4-bit experts; ``form`` = ``runner`` (``moe.Runner``, the CUDA-graph holder of a
            decode loop), ``run`` (``moe.run``, decode arithmetic) or ``prompt`` (``moe.run(prefill=True)``)
``exl3``    one routed layer on EXL3 experts: ``moe.router`` + ``moe.select_rows`` + ``exl3.experts.routed``; ``bits`` a
            width, or 0 = every tensor its own width from 2 to 8; ``graph`` = replayed from a CUDA graph
``affine``  a dense 4-bit projection: ``qmm.matmul`` (decode) or ``qmm.prefill_matmul`` (prompt)
``linear``  a dense EXL3 projection: ``Exl3Linear`` (up to 128 rows) or ``exl3.prefill.matmul`` (prompt)
"""

from __future__ import annotations

import math

import numpy as np
import torch

from tensorfold_b200 import experts, moe, qmm
from tensorfold_b200.exl3 import experts as exl3
from tensorfold_b200.exl3 import prefill as exl3_prefill
from tensorfold_b200.exl3.linear import Exl3Linear

DEV = "cuda"
SCALES = {"fp16": torch.float16, "bf16": torch.bfloat16}


def _layer(name: str, rows: int, form: str, dims: int = 2048, count: int = 128, width: int = 768, top_k: int = 8,
           shared: bool = False, scales: str = "fp16", skew: float = 0.0) -> dict:
    case = {"kind": "layer", "rows": rows, "form": form, "dims": dims, "experts": count, "width": width,
            "top_k": top_k, "shared": shared, "scales": scales, "skew": skew}
    return {"name": name, **case} if name else case


def _exl3(name: str, rows: int, graph: bool, bits: int, dims: int = 2048, count: int = 128, width: int = 768,
          top_k: int = 8, codebook: str = "3inst") -> dict:
    case = {"kind": "exl3", "rows": rows, "graph": graph, "dims": dims, "experts": count, "width": width,
            "top_k": top_k, "bits": bits, "codebook": codebook}
    return {"name": name, **case} if name else case


def _dense(name: str, kind: str, rows: int, n: int, k: int, prompt: bool, scales: str = "bf16", bits: int = 4,
           codebook: str = "3inst") -> dict:
    case = {"kind": kind, "rows": rows, "n": n, "k": k, "prompt": prompt}
    case.update({"scales": scales} if kind == "affine" else {"bits": bits, "codebook": codebook})
    return {"name": name, **case} if name else case


def listed() -> list[dict]:
    return [
        # one user's decode step: one token through a layer of 128 experts, replayed from the graph of a decode loop
        _layer("decode-1", 1, "runner"),
        # a speculative window of one user (or a dozen users), called eagerly; a layer with a shared expert, bf16 scales
        _layer("decode-13-shared", 13, "run", shared=True, scales="bf16"),
        # a full decode batch
        _layer("decode-64", 64, "runner"),
        # a large layer with a shared expert and skewed routing, 256 tokens a step
        _layer("large-decode-256", 256, "run", dims=6144, count=256, width=2048, shared=True, skew=1.1),
        # a short ragged prompt, bf16 scales and a shared expert
        _layer("prompt-317-shared", 317, "prompt", shared=True, scales="bf16"),
        # a prompt chunk
        _layer("prompt-2048", 2048, "prompt"),
        # EXL3 experts at 4.00 bits: one user's decode step, and a full decode batch
        _exl3("exl3-decode-1", 1, True, 4),
        _exl3("exl3-decode-64", 64, True, 4),
        # a larger EXL3 layer whose tensors differ in width: a decode batch, and a prompt chunk
        _exl3("exl3-mixed-128", 128, True, 0, dims=4096, count=160, width=1536),
        _exl3("exl3-mixed-512", 512, False, 0, dims=4096, count=160, width=1536),
        # the projections beside the experts: a few users' rows through a 4-bit projection, a prompt through an EXL3 one
        _dense("affine-dense-5", "affine", 5, 6144, 2048, False),
        _dense("exl3-dense-prompt-1000", "linear", 1000, 4096, 4096, True),
    ]


def _log(rng, lo: int, hi: int) -> int:
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    """One more case: row counts spread over their logarithm, layer sizes over those of the named configurations and
    between them."""

    kind = rng.choice(["decode", "decode", "prompt", "prompt", "exl3", "exl3", "affine", "linear"])
    if kind in ("decode", "prompt"):
        dims, width = rng.choice([1024, 2048, 3072, 4096]), 64 * rng.randint(6, 24)
        rows = _log(rng, 1, 256) if kind == "decode" else _log(rng, 64, 2048)
        return _layer("", rows, "prompt" if kind == "prompt" else rng.choice(["runner", "run"]), dims,
                      rng.choice([32, 64, 96, 128, 160]), width, rng.choice([4, 6, 8]), rng.random() < 0.5,
                      rng.choice(["fp16", "bf16"]), rng.choice([0.0, 0.0, 1.1]))
    if kind == "exl3":
        rows = _log(rng, 1, 512)
        return _exl3("", rows, rows <= 128, rng.choice([0, 3, 4, 4, 5, 6]), rng.choice([1024, 2048, 4096]),
                     rng.choice([32, 64, 128]), 128 * rng.randint(4, 12), rng.choice([4, 8]),
                     rng.choice(["3inst", "mcg", "mul1"]))
    prompt = rng.random() < 0.5
    n, k = 128 * rng.randint(8, 64), 128 * rng.randint(8, 48)
    rows = _log(rng, 129, 4096) if prompt else _log(rng, 1, 128 if kind == "linear" else 64)
    return _dense("", kind, rows, n, k, prompt, rng.choice(["fp16", "bf16"]), rng.choice([3, 4, 5, 6, 8]),
                  rng.choice(["3inst", "mcg", "mul1"]))


# ---- inputs -------------------------------------------------------------------------------------------------------


def _words(g: torch.Generator, shape, dtype) -> torch.Tensor:
    bits = 8 * torch.empty((), dtype=dtype).element_size()
    return torch.randint(-(2 ** (bits - 1)), 2 ** (bits - 1) - 1, shape, generator=g, device=DEV, dtype=dtype)


def _affine_matrix(g, count: int, n: int, k: int, dtype: torch.dtype) -> tuple:
    """MLX words of uniform nibbles, scales |N(0, 0.01)| and biases near -7.5 scales (weights about zero)."""

    scales = torch.randn((count, n, k // 64), generator=g, device=DEV).mul_(0.01).abs_()
    biases = -7.5 * scales + 0.002 * torch.randn((count, n, k // 64), generator=g, device=DEV)
    return _words(g, (count, n, k // 8), torch.int32), scales.to(dtype), biases.to(dtype)


def _exl3_matrix(g, k: int, n: int, bits: int) -> tuple:
    """A trellis of uniform bits, input scales near +-1 and output scales +-|N(0, 0.02)|."""

    def signs(m: int) -> torch.Tensor:
        return torch.randint(0, 2, (m,), generator=g, device=DEV).float() * 2 - 1

    suh = signs(k) * (1 + 0.1 * torch.randn((k,), generator=g, device=DEV))
    svh = signs(n) * (0.02 * torch.randn((n,), generator=g, device=DEV)).abs()
    return _words(g, (k // 16, n // 16, 16 * bits), torch.int16), suh.half(), svh.half()


def _router(case: dict, g, x: torch.Tensor) -> torch.Tensor:
    """Router rows N(0, 0.02); with ``skew``, x's first input is a constant 4 that adds log(rank^-skew) to the logits."""

    count = case["experts"]
    shared = 1 if case.get("shared") else 0
    rows = torch.randn((count + shared, case["dims"]), generator=g, device=DEV) * 0.02
    if case.get("skew"):
        x[:, 0] = 4.0
        rank = torch.randperm(count, generator=g, device=DEV).float() + 1
        rows[:count, 0] = -case["skew"] * torch.log(rank) / 4.0
    return rows.to(torch.bfloat16)


class _Shape:
    def __init__(self, case: dict) -> None:
        self.num_experts_per_tok, self.num_experts = case["top_k"], case["experts"]
        self.moe_intermediate_size, self.hidden_size = case["width"], case["dims"]


def _layer_tensors(case: dict, g, x: torch.Tensor) -> tuple:
    """(gate, up, down, router rows) of an affine layer; sets x's first input when the case is skewed."""

    count = case["experts"] + (1 if case["shared"] else 0)
    dims, width, dtype = case["dims"], case["width"], SCALES[case["scales"]]
    gate, up = (_affine_matrix(g, count, width, dims, dtype) for _ in range(2))
    down = _affine_matrix(g, count, dims, width, dtype)
    return gate, up, down, _router(case, g, x)


def _prepare_layer(case: dict, g, x: torch.Tensor) -> dict:
    gate, up, down, router = _layer_tensors(case, g, x)
    layer = moe.Routed(router, experts.make([gate, up], down, 64), case["top_k"], case["shared"])
    if case["form"] == "runner":
        return {"case": case, "x": x, "runner": moe.Runner(layer, case["rows"])}
    return {"case": case, "x": x, "layer": layer}


def _exl3_tensors(case: dict, g) -> list:
    """[gate, up, down], each a list over the experts of (trellis, suh, svh)."""

    dims, width = case["dims"], case["width"]
    # a width a tensor, the same for every seed (as a checkpoint's): 2 to 8 bits
    widths = np.random.RandomState(5).randint(2, 9, (case["experts"], 3))

    def bits(e: int, m: int) -> int:
        return case["bits"] or int(widths[e, m])

    return [[_exl3_matrix(g, *kn, bits(e, m)) for e in range(case["experts"])]
            for m, kn in enumerate([(dims, width), (dims, width), (width, dims)])]


def _prepare_exl3(case: dict, g, x: torch.Tensor) -> dict:
    dims, rows = case["dims"], case["rows"]
    gate, up, down = _exl3_tensors(case, g)
    ex = exl3.prepare(gate, up, down, case["codebook"], device=DEV)
    s = {"case": case, "x": x, "router": _router(case, g, x), "experts": ex,
         "buf": moe.MoEBuffers(rows, _Shape(case), DEV, shared=False),
         "scratch": exl3.Scratch(ex, rows, case["top_k"], device=DEV),
         "out": torch.empty((rows, dims), dtype=torch.float32, device=DEV)}
    if case["graph"]:
        s["static"] = torch.zeros_like(x)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            _exl3_step(s, s["static"])
        torch.cuda.current_stream().wait_stream(side)
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"], stream=side):
            _exl3_step(s, s["static"])
    return s


def _exl3_step(s: dict, x: torch.Tensor) -> None:
    case, buf = s["case"], s["buf"]
    moe.router(x, s["router"], buf.logits)
    moe.select_rows(buf.logits, buf, case["top_k"], case["experts"])
    exl3.routed(x, buf.pick, buf.wts, s["experts"], s["scratch"], s["out"], case["rows"])


def _tokens(case: dict, seed: int) -> tuple:
    g = torch.Generator(device=DEV).manual_seed(seed)
    return g, torch.randn((case["rows"], case.get("dims") or case["k"]), generator=g, device=DEV).to(torch.bfloat16)


def prepare(case: dict, seed: int) -> dict:
    g, x = _tokens(case, seed)
    if case["kind"] == "layer":
        return _prepare_layer(case, g, x)
    if case["kind"] == "exl3":
        return _prepare_exl3(case, g, x)
    n, k = case["n"], case["k"]
    if case["kind"] == "affine":
        w = _affine_matrix(g, 1, n, k, SCALES[case["scales"]])
        return {"case": case, "x": x, "weight": qmm.pack(*(t[0] for t in w), 64)}
    layer = Exl3Linear.from_tensors(*_exl3_matrix(g, k, n, case["bits"]), case["codebook"])
    return {"case": case, "x": x, "linear": layer, "ws": exl3_prefill.Workspace(),
            "out": torch.empty((case["rows"], n), dtype=torch.bfloat16, device=DEV)}


def run(state: dict):
    case, x = state["case"], state["x"]
    if case["kind"] == "layer":
        if case["form"] == "runner":
            return state["runner"](x)
        return moe.run(x, state["layer"], prefill=case["form"] == "prompt")
    if case["kind"] == "exl3":
        if case["graph"]:
            state["static"].copy_(x, non_blocking=True)
            state["graph"].replay()
        else:
            _exl3_step(state, x)
        return {"out": state["out"], "pick": state["buf"].pick}
    if case["kind"] == "affine":
        return (qmm.prefill_matmul if case["prompt"] else qmm.matmul)(x, state["weight"])
    if case["prompt"]:
        return exl3_prefill.matmul(state["linear"], x, state["out"], state["ws"])
    return state["linear"](x)


# ---- the same results in 64 bits, by plain torch ---------------------------------------------------------------------


def _affine_weight(words: torch.Tensor, scales: torch.Tensor, biases: torch.Tensor) -> torch.Tensor:
    """[N, K] in 64 bits: nibble i of a word is input i, groups of 64 inputs share a scale and a bias."""

    q = (words.unsqueeze(-1) >> (4 * torch.arange(8, device=DEV))) & 15
    q = q.reshape(words.shape[0], -1, 64).double()
    return (q * scales.double().unsqueeze(-1) + biases.double().unsqueeze(-1)).reshape(words.shape[0], -1)


def _codebook(name: str) -> torch.Tensor:
    """The 16-bit values of the 65536 states, as doubles."""

    s = np.arange(65536, dtype=np.uint64)
    if name == "mul1":
        v = (s * 0x83DCD12D) & 0xFFFFFFFF
        total = 1024.0 + sum(((v >> k) & 255).astype(np.float64) for k in (0, 8, 16, 24))
        scale, bias = np.array([0x1EEE, 0xC931], np.uint16).view(np.float16).astype(np.float64)
        return torch.from_numpy((total * scale + bias).astype(np.float16).astype(np.float64)).to(DEV)
    v = (s * 0xCBAC1FED if name == "mcg" else s * 89226354 + 64248484) & 0xFFFFFFFF
    v = (v & 0x8FFF8FFF) ^ 0x3B603B60
    low, high = ((v >> k).astype(np.uint16).view(np.float16) for k in (0, 16))
    return torch.from_numpy((low + high).astype(np.float64)).to(DEV)


def _trellis_weight(trellis: torch.Tensor, book: torch.Tensor) -> torch.Tensor:
    """[K, N] in 64 bits.  A 16 x 16 tile is a circular stream of its 32-bit words, first bit first; value p's state
    is the 16 bits that end where the widths of the values up to p end."""

    k2 = trellis.shape[-1] // 8
    words = trellis.view(torch.int32).long() & 0xFFFFFFFF
    p = torch.arange(256, device=DEV)
    first = (p >> 1) * k2 + torch.where(p % 2 == 1, k2, k2 >> 1) - 16 + 128 * k2
    at, off = (first // 32) % (4 * k2), first % 32
    # the 16 bits from bit ``off`` of a word and, where it ends, of the next
    state = ((words[..., at] << off) & 0xFFFFFFFF | (words[..., (at + 1) % (4 * k2)] << off >> 32)) >> 16
    lane, j = p // 8, p % 8
    row, col = 2 * (lane % 4) + (j & 1) + 8 * ((j >> 1) & 1), lane // 4 + 8 * (j >> 2)
    tiles = torch.empty((*words.shape[:2], 16, 16), dtype=torch.float64, device=DEV)
    tiles[:, :, row, col] = book[state]
    return tiles.transpose(1, 2).reshape(16 * words.shape[0], 16 * words.shape[1])


def _rotated(x: torch.Tensor) -> torch.Tensor:
    i = torch.arange(128, device=DEV)
    bits = sum(((i[:, None] & i[None, :]) >> k) & 1 for k in range(7))
    return (x.reshape(-1, x.shape[1] // 128, 128) @ ((1 - 2 * (bits % 2)).double() / math.sqrt(128))).reshape(x.shape)


def _exl3_product(x: torch.Tensor, matrix: tuple, book: torch.Tensor) -> torch.Tensor:
    trellis, suh, svh = matrix
    return _rotated(_rotated(x * suh.double()) @ _trellis_weight(trellis, book)) * svh.double()


def _weighted(case: dict, x: torch.Tensor, router: torch.Tensor, expert) -> torch.Tensor:
    """The layer's result [R, D]; ``expert(e, rows)`` gives expert e's rows."""

    count = case["experts"]
    logits = x @ router.double().T
    best, pick = logits[:, :count].topk(case["top_k"], dim=1)
    wts = torch.softmax(best, dim=1)
    out = torch.zeros_like(x)
    for e in range(count):
        r, slot = (pick == e).nonzero(as_tuple=True)
        if r.numel():
            out.index_add_(0, r, wts[r, slot].unsqueeze(1) * expert(e, x[r]))
    if case.get("shared"):
        out += torch.sigmoid(logits[:, count:]) * expert(count, x)
    return out


def exact(case: dict, seed: int):
    """``run``'s results for these inputs in 64 bits (the picks are whole numbers: no such value)."""

    g, x16 = _tokens(case, seed)
    if case["kind"] == "layer":
        gate, up, down, router = _layer_tensors(case, g, x16)

        def affine(e: int, rows: torch.Tensor) -> torch.Tensor:
            a, b, c = (_affine_weight(*(t[e] for t in m)) for m in (gate, up, down))
            return torch.nn.functional.silu(rows @ a.T) * (rows @ b.T) @ c.T

        return _weighted(case, x16.double(), router, affine)
    if case["kind"] == "exl3":
        mats, book = _exl3_tensors(case, g), _codebook(case["codebook"])
        router = _router(case, g, x16)

        def trellis(e: int, rows: torch.Tensor) -> torch.Tensor:
            act = torch.nn.functional.silu(_exl3_product(rows, mats[0][e], book)) * _exl3_product(rows, mats[1][e], book)
            return _exl3_product(act, mats[2][e], book)

        return {"out": _weighted(case, x16.double(), router, trellis), "pick": None}
    n, k = case["n"], case["k"]
    if case["kind"] == "affine":
        w = _affine_matrix(g, 1, n, k, SCALES[case["scales"]])
        return x16.double() @ _affine_weight(*(t[0] for t in w)).T
    return _exl3_product(x16.double(), _exl3_matrix(g, k, n, case["bits"]), _codebook(case["codebook"]))


# ---- what a pass cannot do without --------------------------------------------------------------------------------


def _distinct(case: dict) -> float:
    """Experts that the rows' picks are expected to touch."""

    count, top_k, rows = case["experts"], case["top_k"], case["rows"]
    if not case.get("skew"):
        return count * (1 - (1 - top_k / count) ** rows)
    r = np.random.RandomState(7)
    logits = -case["skew"] * np.log(np.arange(1, count + 1)) + 0.02 * math.sqrt(case["dims"]) * r.randn(rows, count)
    return float(len(np.unique(np.argsort(-logits, axis=1)[:, :top_k])))


def work(case: dict) -> dict:
    """Weights of the experts in use once, router rows once, tokens in and results out once; two operations a
    multiply-add of the (row, expert) pairs."""

    rows = case["rows"]
    if case["kind"] in ("layer", "exl3"):
        dims, width, shared = case["dims"], case["width"], 1 if case.get("shared") else 0
        params = 3 * dims * width
        if case["kind"] == "layer":
            expert, out = params * 4.5 / 8, 2
        else:
            expert, out = params * (case["bits"] or 5) / 8 + 2 * 3 * (dims + width), 4
        router = (case["experts"] + shared) * dims
        return {"bytes": (_distinct(case) + shared) * expert + 2 * router + rows * dims * (2 + out),
                "flops": 2.0 * rows * ((case["top_k"] + shared) * params + router)}
    n, k = case["n"], case["k"]
    weight = n * k * (4.5 if case["kind"] == "affine" else case["bits"]) / 8
    return {"bytes": weight + 2 * rows * (n + k), "flops": 2.0 * rows * n * k}


def tolerance(case: dict):
    """About four times the distance to the same layer in 64 bits (same picks, same dequantised weights), measured:
    0.0042 (largest value 0.034) for a layer whose activations and results are rounded to bf16, 0.0004 (0.005) for
    fp32 results behind fp16 intermediates, 0.0017 (0.005) for a projection rounded once to bf16."""

    if case["kind"] == "layer":
        return {"rel": 1.5e-2, "max": 0.13}
    if case["kind"] == "exl3":
        return {"rel": 1.5e-3, "max": 0.02, "differ": 0.0}
    return {"rel": 7e-3, "max": 0.02}
