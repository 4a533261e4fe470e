"""Drop-in for the wrappers of the reference's ``operators/rope_kernels.py`` (:81-131): rotary embedding in
the rotate-half form on ``[batch, seq_len, n_heads, head_dim]`` tensors, own sm_100a kernel."""
import torch

from .._lib import host

BF16 = torch.bfloat16
ROPE_GROUP_SIZE = 4


def calculate_settings(n):
    """Launch hints of the reference (block size = next power of two, warps by size).  Returned so that callers
    that pass them back to ``rope_backward`` keep working; this implementation ignores them."""
    block = 1 << max(0, int(n) - 1).bit_length()
    if block > 65536:
        raise RuntimeError("Cannot launch with a feature dim of %d: the maximum block size is 65536." % n)
    warps = 4
    if block >= 32768:
        warps = 32
    elif block >= 8192:
        warps = 16
    elif block >= 2048:
        warps = 8
    return block, warps


def _rope(x, cos, sin, backward, inplace=False):
    return host.rope(x, cos, sin, backward, inplace)


def rope_forward(x, cos, sin):
    """x [batch, seq_len, n_heads, head_dim] -> rotated tensor of the same shape (a new tensor; the input is
    left as it is, where the reference rotates a contiguous copy in place)."""
    return _rope(x, cos, sin, False)


def rope_backward(dy, cos, sin, n_groups=None, BLOCK_SIZE=None, num_warps=None):
    """Gradient of ``rope_forward``: the same rotation with the sine negated."""
    return _rope(dy, cos, sin, True)


def rope_inplace(x, cos, sin, backward=False):
    """Rotates a contiguous bf16 ``[batch, seq_len, n_heads, head_dim]`` tensor in place (no allocation)."""
    if x.dtype != BF16 or not x.is_contiguous():
        raise ValueError("rope_inplace needs a contiguous bf16 tensor")
    return _rope(x, cos, sin, backward, inplace=True)
