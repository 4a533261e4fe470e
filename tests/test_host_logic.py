"""Host-side logic that needs no device: the calibration running mean, checks before any launch."""
import pathlib
import re

import pytest
import torch

from hyc_lora_release_b200.operators.compress_function import (
    head_to_hidden_shape, hidden_to_head_shape, update_dict)


def test_update_dict_matches_reference(golden):
    d = golden["update_dict"]
    old = {"outlier_channel_index": None, "scale": None}
    for it, new in enumerate(d["history"]):
        old = update_dict(old, {k: v.clone() for k, v in new.items()}, it)
    assert torch.equal(old["outlier_channel_index"], d["final"]["outlier_channel_index"])
    assert torch.equal(old["scale"], d["final"]["scale"])


def test_head_hidden_roundtrip():
    x = torch.arange(2 * 3 * 8, dtype=torch.float32).reshape(2, 3, 8)
    assert torch.equal(head_to_hidden_shape(hidden_to_head_shape(x, 4)), x)


def test_rows_of_no_columns_are_an_error():
    """An integer division by zero in native code would end the process, not raise."""
    from hyc_lora_release_b200.operators import compress_function as cf, rmsnorm_kernels as rn, softmax_kernels as sk
    none, one = torch.zeros(2, 3, 4, 0), torch.zeros(1)
    for call in (lambda: sk.softmax_backward(none, none), lambda: cf.compression_softmax_topk(none, 0.05),
                 lambda: rn.rmsnorm_forward_save(none, one, 1e-5, 4, one, None, one),
                 lambda: rn.rmsnorm_backward_packed(none, one, one, None, None, one, one, 4)):
        with pytest.raises(ValueError, match="empty"):
            call()


def test_tensor_memory_is_taken_after_the_wait():
    """A kernel that may start before the one in front of it has ended takes no tensor memory until that one has: the kernel in
    front may still want some, and would wait for good.  Read from the sources, since a failure would hang the GPU."""
    csrc = pathlib.Path(__file__).resolve().parent.parent / "hyc_lora_release_b200" / "csrc"
    seen = 0
    for path in sorted(csrc.glob("*.cu*")):
        text = path.read_text()
        for at in [m.start() for m in re.finditer(r"tcgen05\.alloc", text)]:
            function = max(text.rfind("\n" + word, 0, at) for word in ("__global__", "__device__", "template", "static", "inline"))
            assert re.search(r"^ *pdl_wait\(\);", text[function:at], re.M), f"{path.name}: tensor memory before pdl_wait()"
            seen += 1
    assert seen >= 4


@pytest.mark.gpu
def test_error_codes_become_hyc_errors():
    """A code that the library returns is a HycError on both paths to it."""
    from hyc_lora_release_b200._lib import HycError
    from hyc_lora_release_b200.operators import compress_function as cf
    with pytest.raises(HycError, match="hyc_softmax_topk_compress"):
        cf.compression_softmax_topk(torch.zeros(1, 1, 8, 72, device="cuda"), 0.05)
