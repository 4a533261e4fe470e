"""Drop-in for the reference module of the same name (its ``triton_fuse_silu_backward``,
operators/triton_fuse_lora_silu_hadamard_backward_kernels.py:152-178)."""
from .._lib import host


def triton_fuse_silu_backward(xa1, b1, q1, s1, xa2, b2, q2, s2, grad_o, quantize_bit=8):
    """De-quantizes the saved gate/up main branches, recomputes the forward and returns
    (o, grad_gate, grad_up), each [B, M, N] bf16."""
    return host.silu_backward(xa1, b1, q1, s1, xa2, b2, q2, s2, grad_o, quantize_bit)
