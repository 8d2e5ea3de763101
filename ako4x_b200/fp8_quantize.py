"""The producers in front of the operator set: the FP8 activation quantiser that makes the MoE's
``hidden_states`` / ``hidden_states_scale`` pair and the writer of the indexer's paged index-K cache
(rule and layouts: reference/moe-fp8-block-scale/variants/fused_routing_v2/kernel.py:495-503 and
reference/dsa-topk-indexer/variants/v8_radix_bt256/kernel.py:562, 621-625)."""
from . import _cabi


def quantize_1x128(x):
    """bf16 [rows, cols] -> (e4m3 [rows, cols], fp32 scales [cols/128, rows]); cols % 128 == 0."""
    return _cabi.native().quantize_1x128(x)


def index_k_cache_write(k, slot_mapping, k_index_cache):
    """Stores bf16 index keys [tokens, 128] into the paged cache (any view with 8448 bytes per page) at
    global slots ``slot_mapping`` (int32, page * 64 + slot; -1 skips the token). In place."""
    _cabi.native().index_k_cache_write(k, slot_mapping, k_index_cache)
    return k_index_cache
