"""The work this library is timed on: what a program that runs a quantized mixture-of-experts model has it do.

Four kinds of case, all through the package's public classes:

* ``moe``   the feed-forward block of one decoder layer (`MlpOrMoe`), k-quant experts: a few rows per step while
            decoding, about a hundred when many sequences decode together or a prompt arrives in small chunks,
            thousands for a whole prompt.  ``layer`` takes the block with its norm and residual add
            (`MlpOrMoe.forward_layer`, what a decoder calls), otherwise `MlpOrMoe.forward`.
* ``fine``  the fine-grained variant: many small Q8_0 experts and an always-on shared expert.
* ``proj``  a dense quantized projection (`QMatMul`): attention projections and the language-model head.
* ``step``  one decode step of a model around the block (`DecodeStep`): attention over the cache included.

``prepack`` is the one-time repack of the weights that a program makes unless it cannot spare the memory.
"""
import math
import random

import torch

from candle_b200 import GgmlDType, Mlp, MlpOrMoe, QMatMul, QTensor
from candle_b200.llama_decode import DecodeConfig, DecodeStep

DTYPES = {"q4k": GgmlDType.Q4K, "q6k": GgmlDType.Q6K, "q80": GgmlDType.Q8_0}
BYTES_PER_WEIGHT = {"q4k": 144 / 256, "q6k": 210 / 256, "q80": 34 / 32}


def listed():
    mixtral = {"kind": "moe", "d": 4096, "ff": 14336, "experts": 8, "top_k": 2, "w13": "q4k", "w2": "q6k", "prepack": True}
    fine = {"kind": "fine", "d": 2048, "ff": 1408, "experts": 60, "top_k": 4, "ff_shared": 5632, "prepack": True}
    return [
        # one sequence decoding: two of eight experts are read, five launches per layer
        dict(mixtral, name="moe_rows1", rows=1, layer=True),
        # a handful of sequences
        dict(mixtral, name="moe_rows8", rows=8, layer=True),
        # a served batch: every expert is read, a few rows each
        dict(mixtral, name="moe_rows32", rows=32, layer=False),
        # many sequences at once, or a short prompt chunk beside them: a ragged number of rows
        dict(mixtral, name="moe_rows100", rows=100, layer=False),
        # a whole prompt
        dict(mixtral, name="moe_rows2048", rows=2048, layer=True),
        # a small block straight from its GGUF bytes (no repacked copy), an odd number of prompt rows
        {"name": "moe_small_gguf_rows257", "kind": "moe", "d": 1024, "ff": 3584, "experts": 8, "top_k": 2, "w13": "q4k", "w2": "q4k",
         "prepack": False, "rows": 257, "layer": False},
        # fine-grained experts, a served batch
        dict(fine, name="fine_rows16", rows=16),
        # fine-grained experts, a long prompt: many small groups
        dict(fine, name="fine_rows4096", rows=4096),
        # the fused query/key/value projection of one sequence: the smallest call
        {"name": "proj_qkv_rows1", "kind": "proj", "n": 6144, "k": 4096, "dtype": "q4k", "rows": 1, "prepack": True},
        # the language-model head of a served batch
        {"name": "proj_head_rows32", "kind": "proj", "n": 32000, "k": 4096, "dtype": "q6k", "rows": 32, "prepack": True},
        # an attention projection over a prompt
        {"name": "proj_rows777", "kind": "proj", "n": 4096, "k": 4096, "dtype": "q4k", "rows": 777, "prepack": True},
        # a decode step of a one-layer model, 32 sequences with 4095 positions in the cache
        {"name": "step_batch32", "kind": "step", "batch": 32, "context": 4096, "prepack": True},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(("moe", "fine", "proj", "step"), (5, 2, 2, 1))[0]
    if kind == "moe":
        w13, w2 = rng.choices((("q4k", "q6k"), ("q4k", "q4k"), ("q6k", "q6k")), (4, 2, 1))[0]
        return {"kind": kind, "d": 512 * rng.randint(2, 8), "ff": 512 * rng.randint(4, 28), "experts": 8, "top_k": 2, "w13": w13, "w2": w2,
                "prepack": rng.random() < 0.8, "rows": _log_int(rng, 1, 2048), "layer": rng.random() < 0.5}
    if kind == "fine":
        return {"kind": kind, "d": 512 * rng.randint(2, 4), "ff": 128 * rng.randint(8, 11), "experts": rng.randint(16, 60), "top_k": rng.choice((2, 4)),
                "ff_shared": rng.choice((2816, 4096, 5632)), "prepack": rng.random() < 0.8, "rows": _log_int(rng, 1, 4096)}
    if kind == "proj":
        dtype = rng.choices(("q4k", "q6k", "q80"), (3, 2, 1))[0]
        return {"kind": kind, "n": 256 * rng.randint(4, 125), "k": 512 * rng.randint(2, 8), "dtype": dtype, "rows": _log_int(rng, 1, 1024),
                "prepack": rng.random() < 0.8}
    return {"kind": kind, "batch": _log_int(rng, 1, 32), "context": _log_int(rng, 128, 4096), "prepack": True}


def _step_config(case):
    return DecodeConfig(n_layer=1, max_seq=case["context"])


def _prepare_step(case, seed):
    cfg = _step_config(case)
    model = DecodeStep(cfg, case["batch"], torch.device("cuda"), n_distinct=1, seed=seed, prepack=case["prepack"])
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    tokens = torch.randint(0, cfg.vocab, (case["batch"],), generator=gen, device="cuda")
    return {"kind": "step", "model": model, "tokens": tokens, "pos": case["context"] - 1}


def prepare(case, seed):
    if case["kind"] == "step":
        return _prepare_step(case, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)

    def weight(n, k, dtype):
        return QMatMul(QTensor.quantize(normal(n, k) * 0.02, DTYPES[dtype]))

    if case["kind"] == "proj":
        matrix = weight(case["n"], case["k"], case["dtype"])
        return {"kind": "proj", "matrix": matrix.prepack() if case["prepack"] else matrix, "x": normal(case["rows"], case["k"])}
    d, ff, n_experts = case["d"], case["ff"], case["experts"]
    w13, w2 = (case["w13"], case["w2"]) if case["kind"] == "moe" else ("q80", "q80")
    experts = [Mlp(weight(ff, d, w13), weight(d, ff, w2), weight(ff, d, w13)) for _ in range(n_experts)]
    router = normal(n_experts, d) * 0.02
    if case["kind"] == "moe":
        block = MlpOrMoe.moe(case["top_k"], router, experts)
    else:
        fs = case["ff_shared"]
        shared = Mlp(weight(fs, d, w13), weight(d, fs, w2), weight(fs, d, w13))
        block = MlpOrMoe.moe(case["top_k"], router, experts, norm_topk_prob=False, shared_expert=shared, shared_expert_gate=normal(d) * 0.02)
    if case["prepack"]:
        block.prepack()
    return {"kind": case["kind"], "block": block, "x": normal(case["rows"], d), "norm": 1.0 + 0.1 * normal(d) if case.get("layer") else None}


def run(state):
    if state["kind"] == "proj":
        return state["matrix"].forward(state["x"])
    if state["kind"] == "step":
        model = state["model"]
        logits = model.forward(state["tokens"], state["pos"])
        return {"logits": logits, "k_cache": model.k_cache, "v_cache": model.v_cache}
    if state["norm"] is not None:
        return state["block"].forward_layer(state["x"], state["norm"], 1e-5)
    return state["block"].forward(state["x"])


def _block_work(rows, d, ff, n_experts, top_k, w13, w2):
    active = n_experts * (1.0 - (1.0 - top_k / n_experts) ** rows)  # experts that get a row, on average
    weights = active * (2 * d * ff * BYTES_PER_WEIGHT[w13] + d * ff * BYTES_PER_WEIGHT[w2])
    return weights + 4 * n_experts * d + 8 * rows * d, 2.0 * rows * (top_k * 3 * d * ff + n_experts * d)


def work(case):
    kind = case["kind"]
    if kind == "proj":
        n, k, rows = case["n"], case["k"], case["rows"]
        return {"bytes": n * k * BYTES_PER_WEIGHT[case["dtype"]] + 4 * rows * (n + k), "flops": 2.0 * rows * n * k}
    if kind == "moe":
        b, f = _block_work(case["rows"], case["d"], case["ff"], case["experts"], case["top_k"], case["w13"], case["w2"])
        return {"bytes": b, "flops": f}
    if kind == "fine":
        b, f = _block_work(case["rows"], case["d"], case["ff"], case["experts"], case["top_k"], "q80", "q80")
        shared = 3 * case["d"] * case["ff_shared"]
        return {"bytes": b + shared * BYTES_PER_WEIGHT["q80"], "flops": f + 2.0 * case["rows"] * shared}
    cfg, rows = _step_config(case), case["batch"]
    d, hd = cfg.d_model, cfg.head_dim
    b, f = _block_work(rows, d, cfg.d_ff, cfg.n_expert, cfg.n_expert_used, "q4k", "q6k")
    attn = d * hd * (2 * cfg.n_head + 2 * cfg.n_kv_head)
    cache = 2 * rows * cfg.n_kv_head * case["context"] * hd
    b += attn * BYTES_PER_WEIGHT["q4k"] + 4 * cache + cfg.vocab * d * BYTES_PER_WEIGHT["q6k"] + 4 * rows * (d + cfg.vocab)
    f += 2.0 * rows * (attn + cfg.vocab * d) + 2.0 * cache * cfg.n_head / cfg.n_kv_head
    return {"bytes": b, "flops": f}


def tolerance(case):
    # Four times what another order of the f32 sums shows (measured over the listed and some drawn cases).
    if case["kind"] == "proj":
        # exact integer block sums; only the order of the f32 sums over the blocks differs (3.4e-7), and the scale
        # of a block may be applied to either factor first
        return {"rel": 1e-5}
    if case["kind"] == "moe":
        # the hidden rows are quantized to int8 before the second product: a last-bit difference of a hidden value
        # moves an int8 value by a step now and then (1.6e-4)
        return {"rel": 6e-4}
    if case["kind"] == "fine":
        return {"rel": 1.3e-3}  # the same, and f16 operands in the second product of large batches (3.2e-4)
    # five quantizations of activations in a row, each of which turns last-bit differences into steps: 7e-3 (7e-2 for
    # the worst value) between two orders of the attention's sums
    return {"rel": 0.03, "max": 0.3}
