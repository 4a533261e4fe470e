"""Drop-in for the reference module of the same name (its ``triton_fuse_silu_forward``,
operators/triton_fuse_lora_silu_hadamard_forward_kernels.py:152-181).  The name is kept so
the reference's layers can import it unchanged; the kernel behind it is CUDA (libhyc.so)."""
from .._lib import host


def triton_fuse_silu_forward(xa1, b1, x1, s1, xa2, b2, x2, s2, quantize_bit=8):
    """q1 = quant(x1, s1), q2 = quant(x2, s2), o = silu(x1 + xa1 @ b1) * (x2 + xa2 @ b2).
    xa*: [B, M, R] ; b*: [R, N] ; x*: [B, M, N] ; s*: [1, N].  -> (q1, q2, o)."""
    return host.silu_forward(xa1, b1, x1, s1, xa2, b2, x2, s2, quantize_bit)
