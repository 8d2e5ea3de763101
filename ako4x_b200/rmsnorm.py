"""bf16 RMSNorm, hidden size 128.

Same signature as the reference plug-in ``run(hidden_states, weight)``
(reference/rmsnorm-h128/variants/triton_tiered_rows/kernel.py:261-278).
"""
import torch

from . import _cabi


def run(hidden_states: torch.Tensor, weight: torch.Tensor) -> torch.Tensor:
    return _cabi.native().rmsnorm(hidden_states, weight)
