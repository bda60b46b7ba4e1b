"""The work that users of this package have it do, as cases that can be timed one by one.

A case is a dict of plain values. `prepare` makes what a program holds before the call (matrices compressed once,
vectors, layers, a captured decode step), `run` is one pass through the public entry points, `work` the bytes and
operations that the pass cannot do without, `tolerance` how far two correct implementations may be apart.

Kinds of case:
  multiply    y = M @ x through `multiply`: one vector, the decode path. fp16 (the reference's type), bfloat16 and
              int8 values; the plain 5-tuple of `compress` or a matrix declared final with `freeze` (serving)
  linear      `MackoLinear` on a [tokens, in] batch: 2..16 tokens are sequences decoded side by side (or drafted
              tokens that are checked together), more are a prompt (prefill)
  decode      one token of a Llama-architecture decoder (`LlamaDecoder`), replayed as a captured CUDA graph, the
              way `llama_decode.generate` runs it
  compress    dense weights -> compressed buffers, once per weight matrix of a checkpoint
  decompress  compressed buffers -> dense weights (export, fine-tuning, checks)

Masks: "magnitude" keeps the same number of largest weights in every row, "bernoulli" is iid, "skewed" has rows
from empty to fully dense with clustered non-zeros. Sizes of the listed cases are the Llama-2-7B layer shapes, the
large and the skewed shapes that the benchmark and the tests of this repository use, or odd ones near them.
"""
from __future__ import annotations

import math

import torch

import macko_spmv_b200 as macko_spmv
from macko_spmv_b200 import workloads
from macko_spmv_b200.linear import MackoLinear
from macko_spmv_b200.llama_decode import LlamaDecoder

DEV = "cuda"
DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "int8": torch.int8}


def listed():
    return [
        # the single product of an attention projection through the reference's two calls, nothing declared
        {"name": "multiply_4096x4096", "kind": "multiply", "rows": 4096, "cols": 4096, "density": 0.5, "dtype": "fp16",
         "frozen": False, "mask": "bernoulli"},
        # a small layer of odd size: what is left is the call itself
        {"name": "multiply_small_odd", "kind": "multiply", "rows": 1003, "cols": 771, "density": 0.3, "dtype": "fp16",
         "frozen": False, "mask": "bernoulli"},
        # LM head of a served model, weights final: the tall matrix of the layer sweep
        {"name": "multiply_lm_head", "kind": "multiply", "rows": 32000, "cols": 4096, "density": 0.5, "dtype": "fp16",
         "frozen": True, "mask": "magnitude"},
        # MLP down projection of a model kept in bfloat16, pruned hard
        {"name": "multiply_down_bf16", "kind": "multiply", "rows": 4096, "cols": 11008, "density": 0.2, "dtype": "bf16",
         "frozen": True, "mask": "magnitude"},
        # MLP up projection with int8 values
        {"name": "multiply_up_int8", "kind": "multiply", "rows": 11008, "cols": 4096, "density": 0.5, "dtype": "int8",
         "frozen": True, "mask": "bernoulli"},
        # the largest matrix of the benchmark on one GPU
        {"name": "multiply_large", "kind": "multiply", "rows": 12288, "cols": 49152, "density": 0.5, "dtype": "fp16",
         "frozen": True, "mask": "bernoulli"},
        # rows from empty to dense: the planned launch
        {"name": "multiply_skewed", "kind": "multiply", "rows": 8192, "cols": 28672, "density": 0.2, "dtype": "fp16",
         "frozen": True, "mask": "skewed"},
        # eight sequences decoded side by side through one layer
        {"name": "linear_8_tokens", "kind": "linear", "rows": 11008, "cols": 4096, "density": 0.5, "tokens": 8, "mask": "magnitude"},
        # a 128-token prompt through one layer
        {"name": "linear_128_tokens", "kind": "linear", "rows": 4096, "cols": 11008, "density": 0.5, "tokens": 128, "mask": "magnitude"},
        # one token through four blocks and the LM head
        {"name": "decode_token", "kind": "decode", "layers": 4, "density": 0.5, "position": 200, "max_len": 384},
        # one weight matrix of a pruned checkpoint
        {"name": "compress_up", "kind": "compress", "rows": 11008, "cols": 4096, "density": 0.5, "dtype": "fp16", "mask": "magnitude"},
        # export of a matrix whose sizes fit no vector width, pruned hard
        {"name": "decompress_odd", "kind": "decompress", "rows": 11003, "cols": 4093, "density": 0.2, "dtype": "fp16", "mask": "bernoulli"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, lo, hi, most):
    """Rows and columns spread over their logarithm; every second one rounded to the multiples that models have."""
    while True:
        rows, cols = _log_int(rng, lo, hi), _log_int(rng, lo, hi)
        if rng.random() < 0.5:
            rows, cols = max(128, rows // 128 * 128), max(128, cols // 128 * 128)
        if rows * cols <= most:
            return rows, cols


def draw(rng):
    kind = rng.choice(["multiply"] * 7 + ["linear"] * 2 + ["decode", "compress", "decompress"])
    density = round(rng.uniform(0.1, 0.9), 3)
    if kind == "multiply":
        mask = rng.choice(["magnitude", "bernoulli", "bernoulli", "skewed"])
        if mask == "skewed":
            rows, cols = _shape(rng, 2048, 32000, 8192 * 28672)
            return {"kind": kind, "rows": rows, "cols": cols, "density": 0.2, "dtype": "fp16", "frozen": True, "mask": mask}
        rows, cols = _shape(rng, 512, 49152, 12288 * 49152 if mask == "bernoulli" else 32000 * 4096)
        if rows * cols > 256 << 20:
            density = min(density, 0.5)
        return {"kind": kind, "rows": rows, "cols": cols, "density": density, "dtype": rng.choice(["fp16", "fp16", "bf16", "int8"]),
                "frozen": rng.random() < 0.6, "mask": mask}
    if kind == "linear":
        rows, cols = _shape(rng, 1024, 16384, 64 << 20)
        return {"kind": kind, "rows": rows, "cols": cols, "density": density, "tokens": rng.choice([_log_int(rng, 2, 16), _log_int(rng, 17, 512)]),
                "mask": "magnitude"}
    if kind == "decode":
        max_len = rng.choice([256, 384, 1024])
        return {"kind": kind, "layers": rng.randint(1, 4), "density": density, "position": rng.randint(0, max_len - 1), "max_len": max_len}
    rows, cols = _shape(rng, 512, 32000, 96 << 20)
    return {"kind": kind, "rows": rows, "cols": cols, "density": density, "dtype": rng.choice(["fp16", "fp16", "bf16", "int8"] if kind == "compress" else ["fp16", "fp16", "bf16"]),
            "mask": rng.choice(["magnitude", "bernoulli"])}


def _matrix(case, seed):
    """The dense pruned matrix on the GPU: weights N(0, 0.02^2), or int8 weights over their whole range."""
    rows, cols, d = case["rows"], case["cols"], case["density"]
    dtype = DTYPES[case.get("dtype", "fp16")]
    if case["mask"] == "skewed":
        return workloads.skewed_matrix(rows, cols, seed, device=DEV, mean_density=d)
    if case["mask"] == "magnitude":
        w = workloads.magnitude_pruned_matrix(rows, cols, d, seed, device=DEV)
    else:
        w = workloads.bernoulli_matrix(rows, cols, d, seed, device=DEV, scale=0.02)
    if dtype is torch.int8:
        return (w.float() * (127.0 / 0.08)).round_().clamp_(-127, 127).to(torch.int8)
    return w.to(dtype)


def _vectors(shape, seed, dtype=torch.float16, scale=1.0):
    g = torch.Generator(device=DEV).manual_seed(seed + 500)
    return (scale * torch.randn(*shape, generator=g, device=DEV)).to(dtype)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "multiply":
        comp = macko_spmv.compress(_matrix(case, seed))
        if case["frozen"]:
            comp = macko_spmv.freeze(comp)
        int8 = case["dtype"] == "int8"
        # int8 weights stand for values around 1/50 of them: the vector is scaled so that y fits fp16
        x = _vectors((case["cols"],), seed, torch.float16 if int8 else DTYPES[case["dtype"]], 0.1 if int8 else 1.0)
        return {"kind": kind, "matrix": comp, "x": x}
    if kind == "linear":
        layer = MackoLinear(macko_spmv.compress(_matrix(case, seed))).freeze()
        return {"kind": kind, "layer": layer, "x": _vectors((case["tokens"], case["cols"]), seed)}
    if kind == "decode":
        model = LlamaDecoder(case["density"], layers=case["layers"], device=DEV, max_len=case["max_len"], seed=4000 + seed)
        for i, blk in enumerate(model.blocks):
            blk.k_cache[:, :, : case["position"]] = _vectors(tuple(blk.k_cache[:, :, : case["position"]].shape), seed + 10 * i)
            blk.v_cache[:, :, : case["position"]] = _vectors(tuple(blk.v_cache[:, :, : case["position"]].shape), seed + 10 * i + 5)
        token = torch.tensor([(7919 * seed + 17) % model.cfg["vocab"]], device=DEV)
        pos = torch.tensor([case["position"]], device=DEV)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.no_grad(), torch.cuda.stream(side):
            for _ in range(2):
                model.logits(token, pos)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.no_grad(), torch.cuda.graph(graph):
            logits = model.logits(token, pos)
        caches = [c for blk in model.blocks for c in (blk.k_cache, blk.v_cache)]
        return {"kind": kind, "model": model, "token": token, "pos": pos, "graph": graph, "logits": logits, "caches": caches}
    m = _matrix(case, seed)
    if kind == "compress":
        return {"kind": kind, "dense": m}
    return {"kind": kind, "matrix": macko_spmv.compress(m)}


def run(state):
    kind = state["kind"]
    if kind == "multiply":
        return macko_spmv.multiply(state["matrix"], state["x"])
    if kind == "linear":
        with torch.no_grad():
            return state["layer"](state["x"])
    if kind == "decode":
        state["graph"].replay()
        return [state["logits"], *state["caches"]]
    if kind == "compress":
        return list(macko_spmv.compress(state["dense"]))
    return macko_spmv.decompress(state["matrix"])


def _stored(rows, cols, density, mask="bernoulli"):
    """Expected stored elements: the non-zeros plus, for gaps of 16 zeros and more, the pads of an iid mask."""
    if mask == "skewed":   # 5 % of the rows dense, 5 % empty, the others Beta-distributed around the mean
        return rows * cols * (0.9 * density + 0.05) * 1.1
    q = (1.0 - density) ** 16
    return rows * cols * density * (1.0 + q / (1.0 - q))


def work(case):
    kind = case["kind"]
    if kind == "decode":
        cfg = {"h": 4096, "f": 11008, "v": 32000}
        block = [(3 * cfg["h"], cfg["h"]), (cfg["h"], cfg["h"]), (2 * cfg["f"], cfg["h"]), (cfg["h"], cfg["f"])]
        mats = block * case["layers"] + [(cfg["v"], cfg["h"])]
        stored = sum(_stored(r, c, case["density"]) for r, c in mats)
        cache = case["layers"] * 2 * cfg["h"] * (case["position"] + 1)
        return {"bytes": 2.5 * stored + 2 * cache + sum(4 * r + 2 * (r + c) for r, c in mats), "flops": 2 * stored + 2 * cache}
    rows, cols = case["rows"], case["cols"]
    stored = _stored(rows, cols, case["density"], case["mask"])
    width = 1 if case.get("dtype") == "int8" else 2
    packed = (width + 0.5) * stored + 4 * (rows + 1)
    if kind == "multiply":
        return {"bytes": packed + 2 * (rows + cols), "flops": 2 * stored}
    if kind == "linear":
        return {"bytes": packed + 2 * case["tokens"] * (rows + cols), "flops": 2 * stored * case["tokens"]}
    return {"bytes": packed + width * rows * cols, "flops": 0}


def tolerance(case):
    """About four times what the rounding of the results alone shows. Against float64 products of the same matrices:
    rel 2.1e-4, max 5e-4 with fp16 results, 1.6e-3 and 3.6e-3 with bfloat16 results; the decode step with its fused
    kernels against the same step through PyTorch operators: rel 2.2e-3 (logits), max 1.2e-2 (cache rows)."""
    kind = case["kind"]
    if kind in ("compress", "decompress"):
        return "exact"
    if kind == "decode":
        return {"rel": 9e-3, "max": 5e-2}
    if case.get("dtype") == "bf16":
        return {"rel": 6.5e-3, "max": 1.5e-2}
    return {"rel": 8.5e-4, "max": 2e-3}
