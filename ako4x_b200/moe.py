"""FP8 block-scale MoE with DeepSeek-V3 grouped routing (256 experts, top-8 of the 4 best of 8
groups; hidden 7168, intermediate 2048; the local experts of one expert-parallel rank).

Same signature and return convention as the reference plug-in
``run(routing_logits, routing_bias, hidden_states, hidden_states_scale, gemm1_weights,
gemm1_weights_scale, gemm2_weights, gemm2_weights_scale, local_expert_offset,
routed_scaling_factor) -> out``
(reference/moe-fp8-block-scale/variants/fused_routing_v2/kernel.py:509-667).
"""
import torch

from . import _cabi

HIDDEN = 7168
INTER = 2048
NUM_EXPERTS = 256


def _scalar(v):
    return v.item() if torch.is_tensor(v) else v


def run(routing_logits, routing_bias, hidden_states, hidden_states_scale, gemm1_weights,
        gemm1_weights_scale, gemm2_weights, gemm2_weights_scale, local_expert_offset,
        routed_scaling_factor, _check_status=False):
    out = _cabi.native().moe(routing_logits, routing_bias, hidden_states, hidden_states_scale, gemm1_weights,
                             gemm1_weights_scale, gemm2_weights, gemm2_weights_scale, local_expert_offset,
                             routed_scaling_factor, _check_status)
    if _check_status:
        out, ws = out
        off = _cabi.lib().ako4x_moe_fp8_block_scale_status_offset(hidden_states.shape[0])
        code = int(ws[off:off + 4].view(torch.int32).item())   # synchronises: tests only
        if code != 0:
            raise _cabi.Ako4xError(f"moe: a bounded device wait gave up (status {code})")
    return out


def run_checked(*args):
    """``run`` followed by a read of the device status word (synchronises the stream)."""
    return run(*args, _check_status=True)


@torch.no_grad()
def ep_combine(rows, pos):
    """Expert-parallel combine: out[t] = bf16(sum over ranks, ascending, of rows[pos[t, g]])."""
    tokens, world = pos.shape
    cols = rows.shape[1]
    if rows.dtype != torch.bfloat16 or pos.dtype != torch.int32:
        raise _cabi.Ako4xError("ep_combine: rows bf16 [n, cols], pos int32 [tokens, world]")
    out = torch.empty((tokens, cols), dtype=torch.bfloat16, device=pos.device)
    rows_c, pos_c = rows.contiguous(), pos.contiguous()
    st = _cabi.lib().ako4x_moe_ep_combine(
        _cabi.ptr(rows_c) if rows.numel() else None, _cabi.ptr(pos_c),
        _cabi.ptr(out), tokens, world, cols, _cabi.stream())
    del rows_c, pos_c
    _cabi.check(st, "ako4x_moe_ep_combine")
    return out


@torch.no_grad()
def ds_routing(routing_logits, routing_bias, routed_scaling_factor):
    """The routing stage alone: (topk_ids int32 [tokens,8] ascending, topk_weights fp32 [tokens,8])."""
    tokens = routing_logits.shape[0]
    dev = routing_logits.device
    ids = torch.empty((tokens, 8), dtype=torch.int32, device=dev)
    w = torch.empty((tokens, 8), dtype=torch.float32, device=dev)
    lg, rb = routing_logits.contiguous(), routing_bias.contiguous()
    st = _cabi.lib().ako4x_moe_ds_routing(
        _cabi.ptr(lg), _cabi.ptr(rb),
        1 if routing_bias.dtype == torch.bfloat16 else 0, float(_scalar(routed_scaling_factor)),
        _cabi.ptr(ids), _cabi.ptr(w), tokens, _cabi.stream())
    del lg, rb
    _cabi.check(st, "ako4x_moe_ds_routing")
    return ids, w
