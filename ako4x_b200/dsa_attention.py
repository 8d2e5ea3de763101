"""DSA sparse MLA attention (16 heads, ckv 512, kpe 64, bf16; keys chosen per token by index).

Same signature and return convention as the reference plug-in
``run(q_nope, q_pe, ckv_cache, kpe_cache, sparse_indices, sm_scale) -> (o, lse)``
(reference/dsa-sparse-attention/variants/hybrid_pdl_v2/kernel.py:557-626).
"""
from . import _cabi


def run(q_nope, q_pe, ckv_cache, kpe_cache, sparse_indices, sm_scale):
    return _cabi.native().dsa_attention(q_nope, q_pe, ckv_cache, kpe_cache, sparse_indices, sm_scale)
