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


def _padded(layer):
    return {**layer._weights[1].padded(), **layer._weights[2].padded()}


@pytest.mark.parametrize("change", ["data", "in place", "view"])
def test_padded_factors_follow_the_adapters(bound, change):
    """A record bound after the change is the measure: ``.data`` replaced (the version stays), written in place (the storage
    stays), another view of the same storage (both stay)."""
    from hyc_lora_release_b200.layer import FusedLlamaLayerIntraInterFullFuse
    layer, bind, mods = bound
    bind()
    before = {k: t.clone() for k, t in _padded(layer).items()}
    for i, name in enumerate(ADAPTERS):
        for j in (1, 2):
            w = mods[name][j].default.weight
            if change == "data":
                w.data = w.data + 1 + i
            elif change == "in place":
                with torch.no_grad():
                    w.add_(1 + i)
            else:
                w.data = w.data.as_strided(w.shape, (1, w.shape[0]))
    assert not layer._plan.fresh()
    bind()
    assert layer._plan.fresh()
    got = _padded(layer)
    case_layer = FusedLlamaLayerIntraInterFullFuse()
    case_layer.set_hyclora_config(layer.hyclora_config)
    case_layer._bind(layer._weights[1].norm_w, layer._weights[2].norm_w, mods)
    for k, t in _padded(case_layer).items():
        assert torch.equal(got[k], t) and not torch.equal(got[k], before[k]), k


def test_replaced_adapter_memory_is_not_handed_out_again(bound):
    """The address of a factor identifies it only while its memory is held."""
    layer, bind, mods = bound
    bind()
    ws = [mods[n][j].default.weight for n in ADAPTERS for j in (1, 2)]
    old = {w.data_ptr() for w in ws}
    for w in ws:
        w.data = torch.zeros_like(w.data)
    later = [torch.empty_like(w) for w in ws for _ in range(20)]
    assert not old & {t.data_ptr() for t in later}


@pytest.mark.parametrize("heads,d,kv", [(4, 128, 4), (2, 128, 2), (8, 128, 2), (4, 64, 2), (4, 128, 0), (0, 128, 2), (4, 128, 3), (4, 256, 1)])
def test_head_geometry_is_checked_against_the_projections(heads, d, kv):
    """4 query and 2 key/value heads of 128 are what the weights hold; the check comes before anything is launched."""
    from hyc_lora_release_b200._lib import host
    H, t = 512, lambda *s: torch.zeros(*s, dtype=torch.bfloat16)
    w = [t(H), t(512, H), t(256, H), t(256, H), t(512, 16), t(256, 16), t(256, 16), t(3, H, 16)]
    with pytest.raises(RuntimeError, match="head"):
        host.attn_forward_map(t(1, 8, H), w, [t(1)] * 7, t(8, 128), t(8, 128), None, heads, d, kv, 4, 1e-5, torch.zeros(1, dtype=torch.int32))
    with pytest.raises(RuntimeError, match="head"):
        host.attn_backward_map(t(8, 512), t(1, 4, 8, 8), [], 0, [t(8, 1)] * 9, w[4:7], t(8, 128), t(8, 128), 1, 8, heads, d, kv, 4, None, 0, 0,
                               torch.zeros(1, dtype=torch.int32))


@pytest.mark.parametrize("how", ["deepcopy", "file"])
def test_a_bound_layer_can_be_copied_and_saved(bound, how):
    import copy
    import io
    layer, bind, mods = bound
    bind()
    layer.iteration = 7
    if how == "deepcopy":
        other = copy.deepcopy(layer)
    else:
        f = io.BytesIO()
        torch.save(layer, f)
        f.seek(0)
        other = torch.load(f, weights_only=False)
    assert other.iteration == 7 and layer._plan is not None
    norms = layer._weights[1].norm_w, layer._weights[2].norm_w
    other._bind(*norms, mods)
    assert other._plan.fresh() and other._plan is not layer._plan


@pytest.mark.parametrize("with_plan", [True, False])
@pytest.mark.parametrize("what", ["weight", "adapter type", "adapter rank", "o bias", "down bias"])
def test_a_parameter_that_stops_fitting_is_refused(bound, what, with_plan):
    """The parameters are the same objects; what ``.data`` holds has become something that the layer refuses."""
    layer, bind, mods = bound
    biased = ("o", "down") if with_plan else ("o", "down", "q")
    for n in biased:
        base = mods[n][0]
        base.bias = torch.nn.Parameter(torch.zeros(base.weight.shape[0], dtype=torch.bfloat16), requires_grad=False)
    bind()
    assert (layer._plan is not None) == with_plan
    bind()
    p = {"weight": mods["up"][0].weight, "adapter type": mods["k"][1].default.weight, "adapter rank": mods["k"][1].default.weight,
         "o bias": mods["o"][0].bias, "down bias": mods["down"][0].bias}[what]
    p.data = p.data[:8] if what == "adapter rank" else p.data.float()
    with pytest.raises(NotImplementedError):
        bind()


def _bad(t, how):
    return {"rows": lambda: t[:-8], "columns": lambda: t[:, :-8].contiguous(), "type": lambda: t.float(),
            "strides": lambda: t.t().contiguous().t()}[how]()


@pytest.mark.parametrize("how", ["rows", "columns", "type", "strides"])
@pytest.mark.parametrize("which", [1, 2, 3, 4, 5, 6])
def test_projections_and_factors_that_do_not_fit_are_refused(which, how):
    """The kernels read weights and factors by address: a matrix of another size, type or (weights) layout is an error before
    anything is launched.  A factor of other strides is copied, so it gets as far as the check for the device."""
    from hyc_lora_release_b200._lib import host
    H, I, t, st = 512, 1024, lambda *s: torch.zeros(*s, dtype=torch.bfloat16), torch.zeros(1, dtype=torch.int32)
    match = "CUDA" if which > 3 and how == "strides" else "expected|head|projection"
    w = [t(H), t(512, H), t(256, H), t(256, H), t(512, 16), t(256, 16), t(256, 16), t(3, H, 16)]
    w[which] = _bad(w[which], how)
    with pytest.raises(RuntimeError, match=match):
        host.attn_forward_map(t(1, 8, H), w, [t(1), t(H), t(H), t(512), t(256), t(256), t(512)], t(8, 128), t(8, 128), None, 4, 128, 2, 4, 1e-5, st)
    if which in (1, 2):
        w = [t(H), t(I, H), t(I, H), t(H, I), t(I, 16), t(I, 16), t(2, H, 16), t(I, 64), t(H, 64)]
        w[which] = _bad(w[which], how)
        with pytest.raises(RuntimeError, match="expected"):
            host.mlp_forward(t(1, 8, H), w, [t(1), t(H), t(H), t(I), t(I)], None, 4, 1e-5, st)
        w = [t(H, I), t(I, 16), t(I, 16), t(H, 16), t(64, I)]
        w[0] = _bad(w[0], how)
        with pytest.raises(RuntimeError, match="expected"):
            host.mlp_backward_lora(t(8, H), w, [t(1)] * 8, 4, st)


@pytest.mark.parametrize("which", [3, 4, 5])
def test_scales_of_another_length_are_refused(which):
    from hyc_lora_release_b200._lib import host
    H, t, st = 512, lambda *s: torch.zeros(*s, dtype=torch.bfloat16), torch.zeros(1, dtype=torch.int32)
    w = [t(H), t(512, H), t(256, H), t(256, H), t(512, 16), t(256, 16), t(256, 16), t(3, H, 16)]
    stats = [t(1), t(H), t(H), t(512), t(256), t(256), t(512)]
    stats[which] = t(1)
    with pytest.raises(ValueError, match="per-channel scale"):
        host.attn_forward_map(t(1, 8, H), w, stats, t(8, 128), t(8, 128), None, 4, 128, 2, 4, 1e-5, st)
    if which < 5:
        w = [t(H), t(1024, H), t(1024, H), t(H, 1024), t(1024, 16), t(1024, 16), t(2, H, 16), t(1024, 64), t(H, 64)]
        stats = [t(1), t(H), t(H), t(1024), t(1024)]
        stats[which] = t(1)
        with pytest.raises(ValueError, match="per-channel scale"):
            host.mlp_forward(t(1, 8, H), w, stats, None, 4, 1e-5, st)
