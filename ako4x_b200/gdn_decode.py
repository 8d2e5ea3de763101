"""Gated Delta Net decode (4 q/k heads, 8 v heads, head size 128, k-last fp32 state).

Same signature as the reference plug-in ``run(q, k, v, state, A_log, a, dt_bias, b, scale)``
(reference/gdn-decode/variants/cuda_bv32_register_resident/kernel.py:456-523): returns
``(output bf16 [B, 1, 8, 128], new_state fp32 [B, 8, 128, 128])``; ``state=None`` means zeros,
``scale`` of None or 0 means 1/sqrt(128).
"""
from . import _cabi


def run(q, k, v, state, A_log, a, dt_bias, b, scale):
    return _cabi.native().gdn_decode(q, k, v, state, A_log, a, dt_bias, b, scale)
