"""Performance cases of the decode layer: what a serving program calls, over the sizes it calls it with.

Every case is one call of a public operator of ``mega_kernel_qwen36`` on inputs that are already on the GPU.
Sizes are those of the two configurations in ``mega_kernel_qwen36/config.py`` (35B-A3B: mixture of experts, 27B:
dense), of their tensor-parallel slices, and of the repository's small single-precision MoE example.  ``listed()``
gives the fixed cases, ``draw(rng)`` further ones of the same ranges.
"""

import math
import os
import sys

import torch

# the package lives in a folder of its own; the repository's root is the working folder
sys.path.insert(0, os.path.abspath("mega-kernel-3.6_b200"))

import mega_kernel_qwen36 as mk  # noqa: E402

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
ELEM = {"bf16": 2, "f16": 2, "f32": 4}

MOE = {  # hidden, experts, top_k, intermediate (routed and shared alike)
    "35b": (2048, 256, 8, 512),
    "small": (256, 16, 4, 128),
}
HEADS = {  # query heads, KV heads, head_dim, hidden
    "35b": (16, 2, 256, 2048),
    "27b": (24, 4, 256, 5120),
}
DENSE_27B = (5120, 17408)
LINEAR_VALUE_HEADS = {"35b": 32, "27b": 48}
LINEAR_KEY_HEADS, LINEAR_DIM = 16, 128
VOCABULARY = 248320


def listed():
    return [
        # one user: every layer of every token is one such call, so its latency is the token rate
        {"name": "moe_35b_b1", "op": "moe", "shape": "35b", "batch": 1, "dtype": "bf16"},
        # a small server's batch: eight tokens meet about 58 different experts
        {"name": "moe_35b_b8", "op": "moe", "shape": "35b", "batch": 8, "dtype": "bf16"},
        # a busy server's batch: most experts have a token, many have several
        {"name": "moe_35b_b32", "op": "moe", "shape": "35b", "batch": 32, "dtype": "bf16"},
        # the repository's small example in single precision: all latency
        {"name": "moe_small_f32_b1", "op": "moe", "shape": "small", "batch": 1, "dtype": "f32"},
        # the dense model's feed-forward for one user, and for a batch of eight
        {"name": "dense_27b_b1", "op": "dense", "slices": 1, "batch": 1, "dtype": "bf16"},
        {"name": "dense_27b_b8", "op": "dense", "slices": 1, "batch": 8, "dtype": "bf16"},
        # one long conversation
        {"name": "attention_35b_32k", "op": "attention", "shape": "35b", "batch": 1, "context": 32768, "dtype": "bf16"},
        # several conversations of an ordinary, odd length
        {"name": "attention_27b_b6_3001", "op": "attention", "shape": "27b", "batch": 6, "context": 3001, "dtype": "f16"},
        # one recurrent step for one user, the state updated where it lies: the smallest call of a decode step
        {"name": "linear_step_35b_b1", "op": "linear", "shape": "35b", "batch": 1, "steps": 1, "inplace": True, "dtype": "bf16"},
        # tokens that are known beforehand (a prompt's tail, a draft being checked) run through the recurrence in one call
        {"name": "linear_64_steps_35b_b8", "op": "linear", "shape": "35b", "batch": 8, "steps": 64, "inplace": False, "dtype": "bf16"},
        # the last call of a decode step: logits over the vocabulary and the next tokens
        {"name": "lm_head_35b_b4", "op": "projection", "role": "lm_head", "shape": "35b", "slices": 1, "batch": 4, "dtype": "bf16"},
        # a whole full-attention layer of the dense model: norm, q|k|v, rotary, cache append, attention, output projection, feed-forward
        {"name": "layer_27b_b3_5000", "op": "layer", "shape": "27b", "ffn": True, "batch": 3, "context": 5000, "capacity": 8192, "dtype": "bf16"},
    ]


def _log_int(rng, low, high):
    """Whole numbers from low to high, evenly spread over their logarithm."""
    return min(high, max(low, int(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng):
    op = rng.choice(["moe", "moe", "dense", "attention", "attention", "linear", "linear", "projection", "layer"])
    dtype = rng.choice(["bf16", "bf16", "bf16", "f16"])
    if op == "moe":
        shape = rng.choice(["35b", "35b", "35b", "small"])
        if shape == "small":
            return {"op": op, "shape": shape, "batch": _log_int(rng, 1, 16), "dtype": rng.choice(["f32", dtype])}
        return {"op": op, "shape": shape, "batch": _log_int(rng, 1, 32), "dtype": dtype}
    if op == "dense":  # the whole layer or one tensor-parallel rank's slice of it
        return {"op": op, "slices": rng.choice([1, 1, 2, 4, 8]), "batch": _log_int(rng, 1, 16), "dtype": dtype}
    if op == "attention":
        batch = _log_int(rng, 1, 16)
        return {"op": op, "shape": rng.choice(["35b", "27b"]), "batch": batch, "context": _log_int(rng, 40, min(65536, 131072 // batch)),
                "dtype": dtype}
    if op == "linear":
        shape, inplace = rng.choice(["35b", "27b"]), rng.random() < 0.5
        if rng.random() < 0.6:
            return {"op": op, "shape": shape, "batch": _log_int(rng, 1, 32), "steps": 1, "inplace": inplace, "dtype": dtype}
        return {"op": op, "shape": shape, "batch": _log_int(rng, 1, 8), "steps": _log_int(rng, 2, 128), "inplace": inplace, "dtype": dtype}
    if op == "projection":
        role, shape = rng.choice(["qkv", "out", "lm_head"]), rng.choice(["35b", "27b"])
        slices = (1 if shape == "35b" else 4) * rng.choice([1, 2]) if role == "lm_head" else 1
        # the operator holds the tokens on chip: 64 KB of them
        return {"op": op, "role": role, "shape": shape, "slices": slices, "batch": _log_int(rng, 1, 8 if shape == "35b" else 4), "dtype": dtype}
    shape = rng.choice(["35b", "27b"])
    context = _log_int(rng, 100, 12000)
    capacity = context + rng.choice([0, rng.randrange(1, 4096)])
    return {"op": op, "shape": shape, "ffn": shape == "27b" and rng.random() < 0.5, "batch": _log_int(rng, 1, 4), "context": context,
            "capacity": capacity, "dtype": dtype}


def _projection_sizes(case):
    """in_features, out_features, fused norm, residual, arg-max."""
    hq, hkv, d, hidden = HEADS[case["shape"]]
    if case["role"] == "qkv":
        return hidden, (hq + 2 * hkv) * d, True, False, False
    if case["role"] == "out":
        return hq * d, hidden, False, True, False
    return hidden, VOCABULARY // case["slices"], True, False, True


class _Inputs:
    """Seeded tensors on the GPU with the distributions that the layers meet: weights of spread 0.02, norm weights
    near one, activations and cache entries of spread one, recurrent state of spread 0.1."""

    def __init__(self, dtype, seed):
        self.dtype, self.gen = dtype, torch.Generator(device="cuda")
        self.gen.manual_seed(seed)

    def normal(self, *size, std=1.0, mean=0.0, dtype=None):
        return torch.empty(size, dtype=dtype or self.dtype, device="cuda").normal_(mean, std, generator=self.gen)

    def weight(self, *size):
        return self.normal(*size, std=0.02)

    def norm(self, n):
        return self.normal(n, std=0.05, mean=1.0)

    def unit(self, *size):
        t = self.normal(*size, dtype=torch.float32)
        return (t / t.norm(dim=-1, keepdim=True)).to(self.dtype)

    def gate(self, *size):
        return torch.sigmoid(self.normal(*size, dtype=torch.float32))


def prepare(case, seed):
    """(function, arguments, keywords, buffers that the call updates)"""
    make = _Inputs(DTYPES[case["dtype"]], seed)
    op, batch = case["op"], case["batch"]
    if op == "moe":
        h, e, k, i = MOE[case["shape"]]
        weights = mk.MoeWeights(make.norm(h), make.weight(e, h), make.weight(e, i, h), make.weight(e, i, h), make.weight(e, h, i),
                                make.weight(i, h), make.weight(i, h), make.weight(h, i))
        return mk.moe_decode, (make.normal(batch, h), weights), {"top_k": k}, ()
    if op == "dense":
        h, i = DENSE_27B[0], DENSE_27B[1] // case["slices"]
        return mk.dense_ffn_decode, (make.normal(batch, h), _dense_weights(make, h, i)), {}, ()
    if op == "attention":
        hq, hkv, d, _ = HEADS[case["shape"]]
        t = case["context"]
        return mk.full_attention_decode, (mk.FullAttentionInputs(make.normal(batch, hq, d), make.normal(batch, t, hkv, d),
                                                                 make.normal(batch, t, hkv, d)),), {}, ()
    if op == "linear":
        hk, hv, d = LINEAR_KEY_HEADS, LINEAR_VALUE_HEADS[case["shape"]], LINEAR_DIM
        state = make.normal(batch, hv, d, d, std=0.1, dtype=torch.float32)
        lead = (batch,) if case["steps"] == 1 else (case["steps"], batch)
        q, k, v = make.unit(*lead, hk, d), make.unit(*lead, hk, d), make.normal(*lead, hv, d)
        decay, beta = make.gate(*lead, hv), make.gate(*lead, hv)
        if case["steps"] == 1:
            return mk.linear_attention_decode_gated, (q, k, v, state), {"decay_per_head": decay, "beta_per_head": beta,
                                                                        "inplace": case["inplace"]}, ()
        return mk.linear_attention_decode_steps, (q, k, v, state), {"decay_per_step": decay, "beta_per_step": beta,
                                                                    "inplace": case["inplace"]}, ()
    if op == "projection":
        n_in, n_out, norm, residual, argmax = _projection_sizes(case)
        return mk.linear_decode, (make.normal(batch, n_in), make.weight(n_out, n_in)), {
            "norm_weight": make.norm(n_in) if norm else None, "residual": make.normal(batch, n_out) if residual else None,
            "return_argmax": argmax}, ()
    hq, hkv, d, h = HEADS[case["shape"]]
    position, capacity = case["context"] - 1, case["capacity"]
    angle = position * 1e7 ** (-torch.arange(32, dtype=torch.float32, device="cuda") / 32)
    block = mk.AttentionBlockInputs(
        input_norm_weight=make.norm(h), qkv_weight=make.weight((hq + 2 * hkv) * d, h), out_weight=make.weight(h, hq * d),
        k_cache=make.normal(batch, capacity, hkv, d), v_cache=make.normal(batch, capacity, hkv, d), position=position,
        query_heads=hq, kv_heads=hkv, head_dim=d, cos=angle.cos().repeat(2), sin=angle.sin().repeat(2), rotary_dim=64)
    hidden, caches = make.normal(batch, h), (block.k_cache, block.v_cache)
    if not case["ffn"]:
        return mk.attention_block_decode, (hidden, block), {}, caches
    return mk.decode_layer, (3, hidden), {"dense_ffn": _dense_weights(make, *DENSE_27B), "attention_block": block}, caches


def _dense_weights(make, h, i):
    return mk.DenseFfnWeights(make.norm(h), make.weight(i, h), make.weight(i, h), make.weight(h, i))


def run(state):
    function, arguments, keywords, updated = state
    result = function(*arguments, **keywords)
    if isinstance(result, mk.DecodeLayerResult):
        result = (result.hidden, result.attention_output)
    return (result, *updated) if updated else result


def work(case):
    op, b, e = case["op"], case["batch"], ELEM[case["dtype"]]
    if op == "moe":
        h, experts, k, i = MOE[case["shape"]]
        # experts with at least one token, on average over inputs
        distinct = experts * (1 - (1 - k / experts) ** b)
        return {"bytes": ((distinct + 1) * 3 * i * h + experts * h + h + 2 * b * h) * e + b * k * 12,
                "flops": 2 * b * ((k + 1) * 3 * i * h + experts * h)}
    if op == "dense":
        return _dense_work(b, DENSE_27B[1] // case["slices"], e)
    if op == "attention":
        return _attention_work(case, b, e)
    if op == "linear":
        hv, d, steps = LINEAR_VALUE_HEADS[case["shape"]], LINEAR_DIM, case["steps"]
        per_step = b * ((2 * LINEAR_KEY_HEADS + 2 * hv) * d * e + 2 * hv * 4)
        return {"bytes": 2 * b * hv * d * d * 4 + steps * per_step, "flops": steps * b * hv * (5 * d * d + d)}
    if op == "projection":
        n_in, n_out, norm, residual, _ = _projection_sizes(case)
        return _projection_work(n_in, n_out, b, e, norm, residual)
    hq, hkv, d, h = HEADS[case["shape"]]
    parts = [_projection_work(h, (hq + 2 * hkv) * d, b, e, True, False), _attention_work(case, b, e),
             _projection_work(hq * d, h, b, e, False, True)]
    if case["ffn"]:
        parts.append(_dense_work(b, DENSE_27B[1], e))
    return {"bytes": sum(p["bytes"] for p in parts), "flops": sum(p["flops"] for p in parts)}


def _dense_work(b, i, e):
    h = DENSE_27B[0]
    return {"bytes": (3 * i * h + h + 2 * b * h) * e, "flops": 6 * b * i * h}


def _attention_work(case, b, e):
    hq, hkv, d, _ = HEADS[case["shape"]]
    return {"bytes": b * (2 * case["context"] * hkv * d + 2 * hq * d) * e, "flops": 4 * b * hq * d * case["context"]}


def _projection_work(n_in, n_out, b, e, norm, residual):
    return {"bytes": (n_out * n_in + b * n_in + b * n_out * (2 if residual else 1) + (n_in if norm else 0)) * e, "flops": 2 * b * n_in * n_out}


def tolerance(case):
    """Outputs are rounded to the tensors' type once; sums are in single precision.  Router choices are whole numbers
    that may swap where two logits are equal up to that precision."""
    rel = {"bf16": 1e-2, "f16": 2e-3, "f32": 1e-5}[case["dtype"]]
    if case["op"] == "moe":
        return {"rel": rel, "differ": 0.01}
    return {"rel": rel}
