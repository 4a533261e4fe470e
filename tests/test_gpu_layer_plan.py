"""The calibrated layer through its plan (one native call forward, one backward) on the GPU."""
import os
import sys
import types

import pytest
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
from test_gpu_layer import BF16, DEV, _Holder, _base  # noqa: E402
from test_oracle_layer import layer_problem  # noqa: E402

pytestmark = pytest.mark.gpu
NAMES = ("q", "k", "v", "o", "gate", "up", "down")


class Problem:
    """A calibrated layer with its modules and inputs.  ``seed`` fixes the frozen weights and the inputs."""

    def __init__(self, B=1, M=128, heads=4, kv=2, d=128, I=512, q=4, map_mode="topk", seed=5, bias=(), mask=None):
        from hyc_lora_release_b200.layer import FusedLlamaLayerIntraInterFullFuse
        g = torch.Generator().manual_seed(seed)
        self.geometry = heads, d, kv
        x, p, cos, sin, own_mask = layer_problem(g, B, M, heads * d, heads, d, kv, I)
        self.x, self.cos, self.sin, self.mask = x.to(DEV), cos.to(DEV), sin.to(DEV), own_mask.to(DEV) if mask is None else mask
        self.gy = torch.randn(x.shape, generator=g).to(BF16).to(DEV)
        self.norms = p["norm_w1"].to(DEV), p["norm_w2"].to(DEV)
        self.mods = {n: (_base(p["w" + n].t().to(DEV), 0.1 * torch.ones(p["w" + n].shape[1], dtype=BF16) if n in bias else None),
                         _Holder(p["a" + n].t().to(DEV)), _Holder(p["b" + n].t().to(DEV))) for n in NAMES}
        self.config = types.SimpleNamespace(use_hyclora=True, iteration_threshold=2, softmax_outlier_ratio=0.05,
                                            layernorm_outlier_ratio=0.01, q_bit=q, softmax_map_mode=map_mode)
        self.layer = FusedLlamaLayerIntraInterFullFuse()
        self.layer.set_hyclora_config(self.config)
        for _ in range(2):
            self.step()

    def lora(self):
        return [self.mods[n][j].default.weight for n in NAMES for j in (1, 2)]

    def forward(self, x, layer=None, mods=None, mask=None):
        mods = mods or self.mods
        args = [x, self.norms[0], None, self.cos, self.sin]
        for n in ("q", "k", "v", "o"):
            args += list(mods[n])
        args += [self.norms[1], None]
        for n in ("gate", "up", "down"):
            args += list(mods[n])
        return (layer or self.layer)(*args, self.mask if mask is None else mask, *self.geometry)

    def step(self, layer=None, x=None):
        """-> [y, grad_x, the fourteen adapter gradients]"""
        x = (self.x if x is None else x).detach().requires_grad_(True)
        y = self.forward(x, layer)
        return [y.detach(), *torch.autograd.grad(y, [x, *self.lora()], self.gy)]

    def fresh_layer(self):
        """A layer that has seen none of the earlier steps but has their statistics."""
        from hyc_lora_release_b200.layer import FusedLlamaLayerIntraInterFullFuse
        layer = FusedLlamaLayerIntraInterFullFuse()
        layer.set_hyclora_config(self.config)
        for mine, theirs in ((layer.attn_state, self.layer.attn_state), (layer.mlp_state, self.layer.mlp_state)):
            mine.iteration = theirs.iteration
            mine.static_value = {k: dict(v) for k, v in theirs.static_value.items()}
        return layer


def _same(got, want):
    return all(torch.equal(a, b) for a, b in zip(got, want, strict=True))


@pytest.mark.parametrize("shape", [dict(), dict(map_mode="prune", q=2), dict(B=2, M=200, map_mode="prune", kv=4, q=8), dict(M=320, q=8),
                                   dict(B=3, M=8, map_mode="prune"), dict(M=264, map_mode="prune", heads=6), dict(M=64, bias=("o", "down")),
                                   dict(heads=8, kv=4, d=64, M=136, map_mode="prune"), dict(heads=8, d=64, kv=8, M=128), dict(M=1088, map_mode="topk"),
                                   dict(B=2, M=256, map_mode="prune"), dict(M=768, map_mode="prune", heads=8, kv=2, q=2), dict(B=2, M=192)])
def test_plan_equals_the_stepwise_path(shape):
    """The step-wise path is what the oracle tests hold; the plan runs the same launches: equal bits, also after the adapters
    have changed between two steps."""
    p = Problem(**shape)
    for _ in range(2):
        assert p.layer._steady()
        got = p.step()
        p.layer.keep_saved = True
        want = p.step()
        p.layer.keep_saved = False
        assert _same(got, want) and _same(got, p.step(layer=p.fresh_layer()))
        with torch.no_grad():
            for i, w in enumerate(p.lora()):
                w.mul_(1 + 0.1 * i)
    p.layer.raise_on_device_errors()


def _masks(kind, B, heads, M):
    """Additive masks whose rows of tiles end at different places: per batch entry, per head, with a gap, or nowhere."""
    i = torch.arange(M, device=DEV)
    dead = i[None] > i[:, None]
    if kind == "padded":         # the entries of a batch are of different lengths: the last keys of each are ruled out
        length = torch.tensor([M - 200 * b for b in range(B)], device=DEV)
        dead = (dead[None] | (i[None, None] >= length[:, None, None]))[:, None]
    elif kind == "heads":        # heads look back different distances
        back = torch.tensor([M, 130, 300, 64][:heads], device=DEV)
        dead = (dead[None] | (i[None] < i[:, None] - back[:, None, None]))[None]
    elif kind == "gap":          # a tile in the middle of the rows is ruled out
        dead = (dead & (i[:, None] >= 256) | ((i >= 128) & (i < 256))[None])[None, None]
    else:                        # "open": nothing is ruled out but a few keys
        dead = (i < 5).expand(M, M)[None, None]
    return torch.zeros(dead.shape, dtype=BF16, device=DEV).masked_fill(dead, torch.finfo(BF16).min)


@pytest.mark.parametrize("map_mode", ["topk", "prune"])
@pytest.mark.parametrize("kind,B,heads,kv", [("padded", 2, 4, 2), ("heads", 1, 4, 4), ("heads", 2, 4, 2), ("gap", 1, 4, 2), ("open", 1, 2, 2)])
def test_plan_equals_the_stepwise_path_for_any_mask(kind, B, heads, kv, map_mode):
    """The plan leaves what the mask rules out of the map unwritten, the step-wise path writes zeros there: equal bits, also where
    the memory that the maps get holds NaN."""
    M = 512
    p = Problem(B=B, M=M, heads=heads, kv=kv, map_mode=map_mode, mask=_masks(kind, B, heads, M))
    p.layer.keep_saved = True
    want = p.step()
    p.layer.keep_saved = False
    for _ in range(2):
        used = [torch.full((B, heads, M, M), float("nan"), dtype=BF16, device=DEV) for _ in range(8)]
        del used
        assert _same(p.step(), want) and all(bool(t.isfinite().all()) for t in want)
    p.layer.raise_on_device_errors()


@pytest.mark.parametrize("stepwise", [False, True])
@pytest.mark.parametrize("M", [100, 4104])
def test_lengths_outside_the_softmax_kernels_are_refused(M, stepwise):
    from hyc_lora_release_b200._lib import HycError
    p = Problem(heads=2, map_mode="prune")
    p.layer.keep_saved = stepwise
    x = torch.zeros(1, M, 256, dtype=BF16, device=DEV)
    p.cos, p.sin = torch.ones(M, 128, dtype=BF16, device=DEV), torch.zeros(M, 128, dtype=BF16, device=DEV)
    with pytest.raises(HycError, match="shape"):
        p.forward(x, mask=torch.zeros(1, 1, M, M, dtype=BF16, device=DEV))


@pytest.mark.parametrize("map_mode", ["topk", "prune"])
@pytest.mark.parametrize("stepwise", [False, True])
def test_step_captured_after_eager_steps(map_mode, stepwise):
    """Eager steps on the default stream, then the capture of a step on another one: what the layer keeps between steps must
    not tie a later step to the stream of an earlier one.  The replay on other inputs equals the eager step bit for bit."""
    p = Problem(map_mode=map_mode)
    p.layer.keep_saved = stepwise             # the step-wise path
    for _ in range(3):
        p.step()
    torch.manual_seed(0)
    other = torch.randn(p.x.shape, device=DEV).to(BF16)
    want = p.step(x=other)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        p.step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    x = p.x.clone()
    with torch.cuda.graph(graph):
        got = p.step(x=x)
    x.copy_(other)
    graph.replay()
    torch.cuda.synchronize()
    assert _same(got, want)


def test_hook_that_updates_adapters_in_place():
    """An update of the adapters inside ``on_lora_grads`` counts as one: the next step uses the new factors everywhere."""
    p = Problem()
    p.step()
    seen = []

    def hook(grads):
        named = p.layer.named_lora_weights()
        with torch.no_grad():
            for name, grad in grads.items():
                before = named[name]._version
                named[name].add_(grad.reshape(named[name].shape), alpha=0.5)
                seen.append(named[name]._version > before)
    p.layer.on_lora_grads = hook
    p.step()
    p.layer.on_lora_grads = None
    assert len(seen) == 14 and all(seen)
    assert _same(p.step(), p.step(layer=p.fresh_layer()))


def test_backward_after_another_adapter_was_bound():
    """The backward pass of a step goes by the factors of its own forward pass, also when these have changed and the layer
    has been called with other adapters in between."""
    def run(switch):
        p = Problem()
        x = p.x.detach().requires_grad_(True)
        y = p.forward(x)
        with torch.no_grad():
            for w in p.lora():
                w.mul_(1.5)
        if switch:
            other = {n: (m[0], _Holder(3 * m[1].default.weight), _Holder(3 * m[2].default.weight)) for n, m in p.mods.items()}
            with torch.no_grad():
                p.forward(p.x, mods=other)
        return torch.autograd.grad(y, [x, *p.lora()], p.gy)
    assert _same(run(True), run(False))


def test_hook_of_the_mlp_half_that_changes_the_attention_half():
    """Both paths take the attention half's factors as the hook left them."""
    def run(stepwise):
        p = Problem()
        p.layer.keep_saved = stepwise

        def hook(grads):
            if "grad_ag" in grads:
                with torch.no_grad():
                    for w in p.lora()[:8]:
                        w.mul_(1.5)
        p.layer.on_lora_grads = hook
        return p.step()
    assert _same(run(False), run(True))


@pytest.mark.parametrize("stepwise", [False, True])
@pytest.mark.parametrize("what", ["mask", "cos", "q", "k", "v", "o", "gate", "up", "down", "q scale", "o scale", "gate scale"])
def test_tensor_on_another_device_is_refused(what, stepwise):
    """A tensor on the host is an error of the call, never an address that a kernel reads."""
    p = Problem()
    p.layer.keep_saved = stepwise
    x, mask, attn, mlp = p.x, p.mask, p.layer.attn_state.static_value, p.layer.mlp_state.static_value
    if what == "mask":
        mask = mask.cpu()
    elif what == "cos":
        p.cos, p.sin = p.cos.cpu(), p.sin.cpu()
    elif what.endswith(" scale"):
        entry = {**attn, **mlp}[what.split()[0]]
        entry["scale"] = entry["scale"].cpu()
    else:
        p.mods[what][0].cpu()
    with pytest.raises(RuntimeError, match="device|CUDA"):
        p.forward(x, mask=mask)
    assert int(p.layer._status.item()) == 0


def test_outlier_indices_may_lie_on_the_host():
    p = Problem()
    want = p.step()
    for entry in (p.layer.attn_state.static_value["x"], p.layer.mlp_state.static_value["x_medium"]):
        entry["outlier_channel_index"] = entry["outlier_channel_index"].cpu()
    assert _same(p.step(), want)


@pytest.mark.parametrize("stepwise", [False, True])
def test_head_geometry_and_scale_that_do_not_fit_are_refused(stepwise):
    p = Problem()
    p.layer.keep_saved = stepwise
    want = p.step()
    fits = p.geometry
    for geometry in ((4, 128, 4), (2, 128, 2), (4, 64, 2), (4, 128, 0)):
        p.geometry = geometry
        with pytest.raises(RuntimeError, match="head"):
            p.forward(p.x)
    p.geometry = fits
    entry = p.layer.attn_state.static_value["o"]
    scale = entry["scale"]
    entry["scale"] = scale.reshape(-1)[:1]
    with pytest.raises(ValueError, match="per-channel scale"):
        p.forward(p.x)
    entry["scale"] = scale
    # (a failed call may have advanced one half: what counts is that the launches of a right call are unharmed)
    p.layer.iteration = 10
    assert _same(p.step(), want)


def _at_offset(t, n):
    """A copy of ``t`` that starts n elements behind a 16-byte boundary."""
    flat = torch.empty(t.numel() + n, dtype=t.dtype, device=t.device)[n:]
    return flat.copy_(t.reshape(-1)).view(t.shape)


@pytest.mark.parametrize("n", [1, 2, 4])
def test_misaligned_scale_of_o_is_refused(n):
    from hyc_lora_release_b200._lib import HycError
    p = Problem()
    entry = p.layer.attn_state.static_value["o"]
    entry["scale"] = _at_offset(entry["scale"].to(BF16), n)
    with pytest.raises(HycError, match="align"):
        p.forward(p.x)


@pytest.mark.parametrize("stepwise", [False, True])
@pytest.mark.parametrize("n", [2, 4])
def test_adapters_off_a_16_byte_boundary(n, stepwise):
    """Adapters that are slices of a flat buffer: the same step, bit for bit."""
    p = Problem()
    p.layer.keep_saved = stepwise
    want = p.step()
    for w in p.lora():
        w.data = _at_offset(w.data, n)
    assert _same(p.step(), want)


def test_statistics_written_behind_the_version_counter():
    """Statistics that the kernels read as a converted copy (here fp32) count as they are at the call."""
    p = Problem()
    for state in (p.layer.attn_state, p.layer.mlp_state):
        for entry in state.static_value.values():
            if entry.get("scale") is not None:
                entry["scale"] = entry["scale"].float()
    before = p.step()
    for state in (p.layer.attn_state, p.layer.mlp_state):
        for entry in state.static_value.values():
            if entry.get("scale") is not None:
                entry["scale"].data.mul_(2)
    after = p.step()
    assert not _same(after, before) and _same(after, p.step(layer=p.fresh_layer()))


def test_norm_weights_and_scales_of_another_length_are_refused():
    from hyc_lora_release_b200.operators import rmsnorm_kernels as rk
    x, w, s = torch.randn(8, 256, device=DEV).to(BF16), torch.ones(256, dtype=BF16, device=DEV), torch.ones(1, 256, dtype=BF16, device=DEV)
    for ww, sx, sy in ((w[:128], s, s), (w, s[:, :64], s), (w, s, s[:, :64])):
        with pytest.raises(ValueError, match="entries"):
            rk.rmsnorm_forward_save(x, ww, 1e-5, 4, sx, None, sy)
    _, rstd, _, q, _ = rk.rmsnorm_forward_save(x, w, 1e-5, 4, s, None, s)
    for ww, sx in ((w[:128], s), (w, s[:, :64])):
        with pytest.raises(ValueError, match="entries"):
            rk.rmsnorm_backward_packed(x, q, sx, None, None, ww, rstd, 4)


@pytest.mark.parametrize("stepwise", [False, True])
def test_replay_follows_the_adapters_and_leaves_eager_steps_alone(stepwise):
    """Adapters updated in place between replays count in the next one, and a step that runs after a capture does not read what
    the capture only recorded (nothing was replayed in between)."""
    p = Problem()
    p.layer.keep_saved = stepwise

    def update(f):
        with torch.no_grad():
            for i, w in enumerate(p.lora()):
                w.mul_(f + 0.05 * i)
    p.step()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        p.step()
    torch.cuda.current_stream().wait_stream(side)
    update(1.1)                               # the copies of the adapters are out of date when the capture begins
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = p.step()
    assert _same(p.step(), p.step(layer=p.fresh_layer()))
    for f in (0.9, 1.2):
        update(f)
        graph.replay()
        want = p.step(layer=p.fresh_layer())
        assert _same(got, want) and _same(p.step(), want)
