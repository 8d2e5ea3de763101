"""Gated Delta Net prefill (4 q/k heads, 8 v heads, head size 128, k-last fp32 state), sequences
packed along the token axis.

Same signature as the reference plug-in ``run(q, k, v, state, A_log, a, dt_bias, b, cu_seqlens,
scale)`` (reference/gdn-prefill/variants/cuda_graph_v5/kernel.py:1333): returns ``(output bf16
[T, 8, 128], new_state fp32 [num_seqs, 8, 128, 128])``; ``state=None`` means zeros, ``scale`` of
None or 0 means 1/sqrt(128).
"""
from . import _cabi


def run(q, k, v, state, A_log, a, dt_bias, b, cu_seqlens, scale, _chunked=True):
    return _cabi.native().gdn_prefill(q, k, v, state, A_log, a, dt_bias, b, cu_seqlens, scale, _chunked)
