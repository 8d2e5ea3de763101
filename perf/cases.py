"""The work that a user of this library has it do, as cases that can be timed and compared.

Every operator is called through its public ``run(...)`` on the inputs of the benchmark
configurations (``ako4x_b200.workloads``): the sizes are those configurations' own, the sizes of
the tests, and generic ones between them. ``listed()`` holds twelve points of the ranges and
``draw()`` gives any other: one more call of one operator, from a single row or token up to the
largest configuration. Sequence lengths are ragged: they belong to a case, so that its work is
known, and only the values depend on the seed.
"""
import math
import random

import torch

from ako4x_b200 import (dsa_attention, dsa_indexer, fp8_quantize, gdn_decode, gdn_prefill, gemm, gqa_decode,
                        mla_decode, mla_prefill, moe, rmsnorm)
from ako4x_b200 import workloads as W

DEVICE = "cuda"
TOPK = 2048
EXPERTS, LOCAL_EXPERTS = 256, 32
HIDDEN, INTER = 7168, 2048
GEMM_N, GEMM_K = 2048, 4096


def listed():
    return [
        # Normalising the heads of a few tokens in a decode step: one launch, nothing to amortise it.
        {"name": "rmsnorm_rows64", "op": "rmsnorm", "rows": 64},
        # One user's chat at a few hundred tokens of context: the smallest decode attention call.
        {"name": "gqa_decode_b1", "op": "gqa_decode", "batch": 1, "max_len": 547},
        # A serving batch of decode attention with ragged contexts up to 8192 tokens.
        {"name": "gqa_decode_b64", "op": "gqa_decode", "batch": 64, "max_len": 8192},
        # The same for latent attention.
        {"name": "mla_decode_b32", "op": "mla_decode", "batch": 32, "max_len": 8192},
        # A prefill step over eight ragged prompts, some of them behind a cached prefix: the
        # largest case.
        {"name": "mla_prefill_b8", "op": "mla_prefill", "batch": 8, "max_q": 2048, "max_kv": 8192},
        # One token of one sequence at the longest context: index scores, selection and sparse
        # attention, by the two plug-ins one after the other.
        {"name": "dsa_decode_t1", "op": "dsa", "tokens": 1, "ctx": 32768, "chained": False},
        # A chunk of a long prompt through the same path, by the call that chains the two.
        {"name": "dsa_prefill_t512", "op": "dsa", "tokens": 512, "ctx": 32768, "chained": True},
        # Experts of a decode batch: bound by the weights that the batch touches.
        {"name": "moe_t128", "op": "moe", "tokens": 128, "skew": 0.0, "offset": 0, "bias": "fp32", "activations": "fp8"},
        # Experts of a prefill step, the benchmark's headline size.
        {"name": "moe_t8192", "op": "moe", "tokens": 8192, "skew": 0.0, "offset": 0, "bias": "fp32", "activations": "fp8"},
        # Linear attention, one token for each of 16 sequences: reads and writes the states.
        {"name": "gdn_decode_b16", "op": "gdn_decode", "batch": 16, "state": True},
        # Linear attention over eight ragged prompts.
        {"name": "gdn_prefill_n8", "op": "gdn_prefill", "sequences": 8, "max_len": 2048, "state": True},
        # A projection of a mid-sized batch with an odd number of rows.
        {"name": "gemm_m969", "op": "gemm", "rows": 969, "dtype": "float16"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw(rng):
    op = rng.choice(["rmsnorm", "gqa_decode", "mla_decode", "mla_prefill", "dsa", "moe", "gdn_decode", "gdn_prefill",
                     "gemm"])
    if op == "rmsnorm":
        return {"op": op, "rows": _log_int(rng, 1, 520128)}
    if op == "gqa_decode":
        return {"op": op, "batch": _log_int(rng, 1, 256), "max_len": _log_int(rng, 16, 8192)}
    if op == "mla_decode":
        return {"op": op, "batch": _log_int(rng, 1, 128), "max_len": _log_int(rng, 16, 8192)}
    if op == "mla_prefill":
        max_q = _log_int(rng, 1, 2048)
        return {"op": op, "batch": rng.randint(1, 8), "max_q": max_q, "max_kv": _log_int(rng, max_q, 8192)}
    if op == "dsa":
        tokens = _log_int(rng, 1, 512)
        return {"op": op, "tokens": tokens, "ctx": _log_int(rng, 2048, 32768), "chained": rng.random() < 0.5}
    if op == "moe":
        return {"op": op, "tokens": _log_int(rng, 1, 8192), "skew": rng.choice([0.0, 0.0, 0.5]),
                "offset": LOCAL_EXPERTS * rng.randrange(EXPERTS // LOCAL_EXPERTS),
                "bias": rng.choice(["fp32", "bf16"]), "activations": rng.choice(["fp8", "bf16"])}
    if op == "gdn_decode":
        return {"op": op, "batch": _log_int(rng, 1, 256), "state": rng.random() < 0.8}
    if op == "gdn_prefill":
        n = _log_int(rng, 1, 64)
        return {"op": op, "sequences": n, "max_len": _log_int(rng, 1, 8192 // n), "state": rng.random() < 0.5}
    return {"op": op, "rows": _log_int(rng, 1, 16294), "dtype": rng.choice(["float16", "bfloat16"])}


def _cost(case):
    w = work(case)
    return max(w["bytes"] / 6e12, w["flops"] / 1.6e15)


def draw(rng):
    largest = max(_cost(c) for c in listed())
    while True:
        case = _draw(rng)
        if _cost(case) <= largest:
            return case


def _lens(case, lo, hi, count, what):
    """`count` lengths, uniform in [lo, hi]: a property of the case."""
    key = [what] + ["%s=%s" % (k, case[k]) for k in sorted(case) if k != "name"]
    rng = random.Random(" ".join(key))
    return [rng.randint(lo, hi) for _ in range(count)]


def _decode_lens(case):
    least = max(1, case["max_len"] // (64 if case["op"] == "gqa_decode" else 16))
    return _lens(case, least, case["max_len"], case["batch"], "kv")


def _prefill_lens(case):
    q = _lens(case, max(1, case["max_q"] // 128), case["max_q"], case["batch"], "q")
    kv = [_lens(case, n, case["max_kv"], 1, "kv%d" % i)[0] for i, n in enumerate(q)]
    return q, kv


def _gdn_lens(case):
    return _lens(case, max(1, case["max_len"] // 64), case["max_len"], case["sequences"], "seq")


def prepare(case, seed):
    op = case["op"]
    if op == "rmsnorm":
        a = W.make_rmsnorm(case["rows"], shape_id=seed, device=DEVICE)
    elif op == "gqa_decode":
        a = W.make_gqa_decode(case["batch"], shape_id=seed, device=DEVICE, lens=_decode_lens(case))
    elif op == "mla_decode":
        a = W.make_mla_decode(case["batch"], shape_id=seed, device=DEVICE, lens=_decode_lens(case))
    elif op == "mla_prefill":
        q, kv = _prefill_lens(case)
        a = W.make_mla_prefill(case["batch"], shape_id=seed, device=DEVICE, q_lens=q, kv_lens=kv)
    elif op == "dsa":
        a = W.make_dsa_indexer(case["tokens"], max(case["ctx"], case["tokens"]), shape_id=seed, device=DEVICE)
        pages = a["k_index_cache_fp8"].shape[0]
        none = torch.empty((case["tokens"], 0), dtype=torch.int32, device=DEVICE)
        b = W.make_dsa_attention(case["tokens"], case["ctx"], none, pages, shape_id=seed, device=DEVICE)
        del b["sparse_indices"]
        a.update(b)
    elif op == "moe":
        a = W.make_moe(case["tokens"], shape_id=seed, device=DEVICE, num_local_experts=LOCAL_EXPERTS,
                       local_expert_offset=case["offset"], skew=case["skew"])
        if case["bias"] == "bf16":
            a["routing_bias"] = a["routing_bias"].to(torch.bfloat16)
        if case["activations"] == "bf16":
            g = torch.Generator(device=DEVICE)
            g.manual_seed(seed)
            x = torch.randn((case["tokens"], HIDDEN), generator=g, device=DEVICE)
            a["hidden_states"], a["hidden_states_scale"] = x.to(torch.bfloat16), None
    elif op == "gdn_decode":
        a = W.make_gdn_decode(case["batch"], shape_id=seed, device=DEVICE, with_state=case["state"])
    elif op == "gdn_prefill":
        a = W.make_gdn_prefill(_gdn_lens(case), shape_id=seed, device=DEVICE, with_state=case["state"])
    else:
        a = W.make_gemm(case["rows"], shape_id=seed, device=DEVICE, n=GEMM_N, k=GEMM_K, dtype=getattr(torch, case["dtype"]))
    return {"op": op, "chained": case.get("chained", False), "args": list(a.values())}


RUN = {"rmsnorm": rmsnorm.run, "gqa_decode": gqa_decode.run, "mla_decode": mla_decode.run,
       "mla_prefill": mla_prefill.run, "gdn_decode": gdn_decode.run, "gdn_prefill": gdn_prefill.run, "gemm": gemm.run}


def run(state):
    op, a = state["op"], state["args"]
    if op == "dsa":
        if state["chained"]:
            return dsa_indexer.run_with_attention(*a)
        index, (q_nope, q_pe, ckv, kpe, sm_scale) = a[:5], a[5:]
        (topk,) = dsa_indexer.run(*index)
        o, lse = dsa_attention.run(q_nope, q_pe, ckv, kpe, topk, sm_scale)
        return o, lse, topk
    if op == "moe":
        if a[3] is None:
            x, scale = fp8_quantize.quantize_1x128(a[2])
            return moe.run(a[0], a[1], x, scale, *a[4:])
        return moe.run(*a)
    return RUN[op](*a)


def _expected_touched(n, draws):
    """How many of n equally likely items `draws` picks touch."""
    return n * (1.0 - (1.0 - 1.0 / n) ** draws)


def work(case):
    op = case["op"]
    if op == "rmsnorm":
        n = case["rows"]
        return {"bytes": n * 512 + 256, "flops": n * 128 * 4}
    if op == "gqa_decode":
        b, keys = case["batch"], sum(_decode_lens(case))
        return {"bytes": keys * (4096 + 4) + b * (2 * 8192 + 128), "flops": keys * 32 * 128 * 4}
    if op == "mla_decode":
        b, keys = case["batch"], sum(_decode_lens(case))
        return {"bytes": keys * (1152 + 4) + b * (16 * (576 + 512) * 2 + 64), "flops": keys * 34816}
    if op == "mla_prefill":
        q, kv = _prefill_lens(case)
        pairs = sum(n * (m - n) + n * (n + 1) // 2 for n, m in zip(q, kv))   # (query, visible key)
        return {"bytes": sum(kv) * (1152 + 4) + sum(q) * (16 * (576 + 512) * 2 + 64), "flops": pairs * 34816}
    if op == "dsa":
        t, ctx = case["tokens"], max(case["ctx"], case["tokens"])
        chosen = sum(min(TOPK, ctx - t + 1 + i) for i in range(t))
        pairs = sum(ctx - t + 1 + i for i in range(t))
        keys = min(ctx, _expected_touched(ctx, chosen)) if t > 1 else chosen
        return {"bytes": ctx * 132 + t * (8192 + 256) + t * TOPK * 4 + keys * 1152 + t * (16 * (576 + 512) * 2 + 64),
                "flops": pairs * 64 * 128 * 2 + chosen * 34816}
    if op == "moe":
        t = case["tokens"]
        pairs = t * 8 * LOCAL_EXPERTS / EXPERTS
        experts = _expected_touched(LOCAL_EXPERTS, pairs)
        act = t * HIDDEN * (2 if case["activations"] == "bf16" else 1) + t * HIDDEN // 128 * 4
        return {"bytes": experts * 3 * HIDDEN * INTER + act + t * EXPERTS * 4 + t * HIDDEN * 2,
                "flops": pairs * 6 * HIDDEN * INTER}
    if op == "gdn_decode":
        b = case["batch"]
        return {"bytes": b * (8 * 128 * 128 * 4 * (2 if case["state"] else 1) + 2 * (512 * 2 + 1024 * 2 + 16)),
                "flops": b * 8 * 128 * 128 * 6}
    if op == "gdn_prefill":
        lens = _gdn_lens(case)
        t, n = sum(lens), len(lens)
        return {"bytes": t * 2 * (512 * 2 + 1024 * 2 + 16) + n * 8 * 128 * 128 * 4 * (2 if case["state"] else 1),
                "flops": t * 8 * 128 * 128 * 6}
    m = case["rows"]
    return {"bytes": 2 * (m * GEMM_K + GEMM_N * GEMM_K + m * GEMM_N), "flops": 2 * m * GEMM_N * GEMM_K}


def tolerance(case):
    """bf16 results (and bf16 attention probabilities, or an activation of bf16 accuracy between two
    FP8 products) everywhere but in the fp32 outputs beside them, which are of the same sums."""
    op = case["op"]
    if op in ("rmsnorm", "gdn_decode", "gdn_prefill"):
        return {"rel": 4e-3}
    if op == "gemm":
        return {"rel": 1e-3 if case["dtype"] == "float16" else 4e-3}
    if op == "dsa":
        return {"rel": 1e-2, "differ": 0.01}   # a tie of fp32 sums may go either way
    return {"rel": 1e-2}
