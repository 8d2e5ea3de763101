"""Paged GQA decode (32 query heads, 8 KV heads, head_dim 128, bf16).

Same signature and return convention as the reference plug-in
``run(q, k_cache, v_cache, kv_indptr, kv_indices, sm_scale) -> (o, lse)``
(reference/gqa-paged-decode-h32-kv8-d128-ps1/variants/triton_pdl_grid_dispatch/kernel.py:420-532).
"""
from . import _cabi


def run(q, k_cache, v_cache, kv_indptr, kv_indices, sm_scale):
    return _cabi.native().gqa_decode(q, k_cache, v_cache, kv_indptr, kv_indices, sm_scale)
