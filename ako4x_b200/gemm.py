"""Dense GEMM ``C = A @ B.T`` (definition ``gemm_n2048_k4096``: A [M, 4096], B [2048, 4096], fp16).

``run(A, B) -> C`` is the signature of the reference family (reference/gemm-n2048-k4096/README.md,
whose best implementation is ``torch.matmul(A, B.T)``). fp16 or bf16 operands, fp32 accumulation
on tcgen05 tensor cores, output in the operand type. N must be a multiple of 256, K of 64.
"""
import torch

from . import _cabi


def run(A: torch.Tensor, B: torch.Tensor) -> torch.Tensor:
    return _cabi.native().gemm(A, B)
