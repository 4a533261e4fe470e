"""The weight records and the plan of the fused layer on the CPU: what they cache of the adapters, and when it is renewed."""
import os
import sys
import types

import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
from layer_case import CONFIG, build, modules  # noqa: E402

ADAPTERS = ("q", "k", "v", "o", "gate", "up", "down")


@pytest.fixture()
def bound():
    """-> (layer, bind(): binds the weights as a call of the layer does, the seven projections)"""
    from hyc_lora_release_b200.layer import FusedLlamaLayerIntraInterFullFuse
    case = build("mistral")
    mods = modules(case, "cpu")
    layer = FusedLlamaLayerIntraInterFullFuse()
    layer.set_hyclora_config(types.SimpleNamespace(q_bit=4, **CONFIG))
    norms = case["p"]["norm_w1"], case["p"]["norm_w2"]
    return layer, lambda: layer._bind(*norms, mods), mods


def test_padded_factors_are_no_part_of_a_graph(bound):
    layer, bind, _ = bound
    with torch.enable_grad():
        aw, mw, _ = bind()
    for record in (aw, mw):
        for name, t in record.padded().items():
            assert not t.requires_grad and t.grad_fn is None, name
