"""Paged MLA decode (16 heads, ckv 512, kpe 64, bf16).

Same signature and return convention as the reference plug-in
``run(q_nope, q_pe, ckv_cache, kpe_cache, kv_indptr, kv_indices, sm_scale) -> (o, lse)``
(reference/mla-paged-decode-h16-ckv512-kpe64-ps1/variants/triton_split_kv_2d_reduce_pdl_rw2/kernel.py:369-435).
"""
from . import _cabi


def run(q_nope, q_pe, ckv_cache, kpe_cache, kv_indptr, kv_indices, sm_scale):
    return _cabi.native().mla_decode(q_nope, q_pe, ckv_cache, kpe_cache, kv_indptr, kv_indices, sm_scale)
