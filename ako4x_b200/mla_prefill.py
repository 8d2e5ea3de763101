"""Causal paged MLA prefill (16 heads, ckv 512, kpe 64, bf16, ragged batch).

Same signature and return convention as the reference plug-in
``run(q_nope, q_pe, ckv_cache, kpe_cache, qo_indptr, kv_indptr, kv_indices, sm_scale) -> (o, lse)``
(reference/mla-paged-prefill-causal-h16-ckv512-kpe64-ps1/variants/
iter6-triton-split-K-grid-pid0-kvsplit/submission_no_cache.py:537-692). No host read of the
indptr arrays takes place: the launch geometry depends on shapes only.
"""
from . import _cabi


def run(q_nope, q_pe, ckv_cache, kpe_cache, qo_indptr, kv_indptr, kv_indices, sm_scale):
    return _cabi.native().mla_prefill(q_nope, q_pe, ckv_cache, kpe_cache, qo_indptr, kv_indptr, kv_indices, sm_scale)
