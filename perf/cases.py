"""Performance cases of the framework: the work a fine-tuning program has it do, through its public entry points.

Kinds of case:
  layer    one fused decoder layer, forward + backward through the module and autograd, after calibration: what a
           model runs once per layer and training step (geometries of Llama-2-7B and Mistral-7B, LoRA rank 16 on all
           seven projections, frozen weights in bf16 or as 4-bit block-wise codes, the probability map kept by the
           global threshold ("prune", the default) or as per-row top-k + 4-bit groups ("topk"))
  mlp      the MLP half alone, forward + backward (``mlp.mlp_forward`` / ``mlp.mlp_backward``)
  map      the per-row top-k form of a probability map: save, restore, restore fused with the softmax backward
  prune    the threshold-pruned form of a probability map: save and restore, as a sparse tensor with the list's length
           read by the host ("sparse") or in buffers of a fixed capacity ("static")
  channel  per-channel quantize-and-pack and back: with outlier channels, plain, or with zero points
  silu     the fused LoRA-SiLU-Hadamard operators on their own, forward + backward
"""
import math
import types

import torch

from hyc_lora_release_b200 import mlp
from hyc_lora_release_b200.layer import FusedLlamaLayerIntraInterFullFuse
from hyc_lora_release_b200.operators import compress_function as cf
from hyc_lora_release_b200.operators.triton_fuse_lora_silu_hadamard_backward_kernels import triton_fuse_silu_backward
from hyc_lora_release_b200.operators.triton_fuse_lora_silu_hadamard_forward_kernels import triton_fuse_silu_forward

BF16 = torch.bfloat16
R = 16                                   # LoRA rank
HEAD = 128                               # head size of both geometries
HIDDEN, HEADS = 4096, 32
KV_HEADS = {"llama": 32, "mistral": 8}
INTER = {"llama": 11008, "mistral": 14336}
PROJ = ("q", "k", "v", "o", "gate", "up", "down")


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # one layer of a Llama-2-7B step on one long sequence, 4-bit saves, top-k map: the training step of the benchmark
        dict(name="layer-llama-1x2048-topk", kind="layer", model="llama", batch=1, seq=2048, q=4, map="topk", weights="bf16"),
        # a full micro-batch on the grouped-heads geometry, the default form of the map: the largest step of the list
        dict(name="layer-mistral-4x1024-prune", kind="layer", model="mistral", batch=4, seq=1024, q=4, map="prune", weights="bf16"),
        # padded instruction batch of an odd length, 2-bit saves
        dict(name="layer-llama-2x696-prune", kind="layer", model="llama", batch=2, seq=696, q=2, map="prune", weights="bf16"),
        # one short prompt with 4-bit frozen weights and 8-bit saves: latency, launches and host work decide
        dict(name="layer-llama-1x128-nf4", kind="layer", model="llama", batch=1, seq=128, q=8, map="prune", weights="nf4"),
        # MLP half at the two benchmark shapes
        dict(name="mlp-llama-4x512-q4", kind="mlp", model="llama", batch=4, seq=512, q=4),
        dict(name="mlp-mistral-1x8192-q8", kind="mlp", model="mistral", batch=1, seq=8192, q=8),
        # attention-map compression of the benchmark, and rows that are not a power of two long
        dict(name="map-4x32x512-q4", kind="map", batch=4, heads=32, rows=512, cols=512, q=4, ratio=0.05),
        dict(name="map-1x32x320-q2", kind="map", batch=1, heads=32, rows=320, cols=320, q=2, ratio=0.02),
        # the reference's sparse-tensor form of the same map at an odd length
        dict(name="prune-2x32x696-sparse", kind="prune", batch=2, heads=32, seq=696, ratio=0.05, form="sparse"),
        # activation saves: the smallest call (a few dozen tokens) and the largest (a micro-batch of the widest tensor)
        dict(name="channel-1x37x4096-q8", kind="channel", batch=1, seq=37, n=4096, q=8, form="plain", ratio=0.0),
        dict(name="channel-1x8192x14336-q4", kind="channel", batch=1, seq=8192, n=14336, q=4, form="outlier", ratio=0.01),
        # the stand-alone fused operators on a ragged token count
        dict(name="silu-1x1100x11008-q4", kind="silu", batch=1, seq=1100, n=11008, q=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("layer", "layer", "layer", "mlp", "mlp", "map", "prune", "channel", "channel", "silu"))
    q = rng.choice((2, 4, 4, 8))
    if kind == "layer":
        form = rng.choice(("prune", "topk"))
        step = 8 if form == "prune" else 64          # what the two forms ask of the sequence length
        while True:
            b, m = rng.choice((1, 1, 2, 3, 4)), step * max(1, _log(rng, 64, 2048) // step)
            if b * m <= 4096 and b * m * m <= 4 * 1024 * 1024:
                break
        return dict(kind=kind, model=rng.choice(("llama", "mistral")), batch=b, seq=m, q=q, map=form,
                    weights=rng.choice(("bf16", "bf16", "nf4")))
    if kind == "mlp":
        t = _log(rng, 32, 8192)
        b = rng.choice((1, 1, 2, 4))
        return dict(kind=kind, model=rng.choice(("llama", "mistral")), batch=b, seq=max(1, t // b), q=q)
    if kind == "map":
        s = 64 * rng.choice((1, 2, 3, 4, 5, 8, 8, 11, 16, 16, 23, 32))
        b, h = rng.choice((1, 2, 4)), rng.choice((8, 32))
        while b * h * s * s > 1 << 27:
            b, h = max(1, b // 2), h if b > 1 else h // 2
        return dict(kind=kind, batch=b, heads=h, rows=s, cols=s, q=q, ratio=rng.choice((0.01, 0.02, 0.05)))
    if kind == "prune":
        s = 8 * max(1, _log(rng, 64, 2048) // 8)
        b, h = rng.choice((1, 2, 4)), rng.choice((8, 32))
        while b * h * s * s > 1 << 27:
            b, h = max(1, b // 2), h if b > 1 else h // 2
        return dict(kind=kind, batch=b, heads=h, seq=s, ratio=rng.choice((0.01, 0.05, 0.1)), form=rng.choice(("sparse", "static")))
    if kind == "channel":
        t = _log(rng, 16, 8192)
        b = rng.choice((1, 1, 2, 4))
        form = rng.choice(("outlier", "outlier", "plain", "zero_point"))
        return dict(kind=kind, batch=b, seq=max(1, t // b), n=rng.choice((1024, 4096, 4096, 5120, 11008, 14336)), q=q,
                    form=form, ratio=rng.choice((0.005, 0.01)) if form == "outlier" else 0.0)
    return dict(kind=kind, batch=rng.choice((1, 2)), seq=_log(rng, 16, 2048), n=rng.choice((1024, 4096, 11008, 14336)), q=q)


# ------------------------------------------------------------------ what the program has before the call

class _Draws:
    """Random tensors on the GPU from one seed."""

    def __init__(self, seed):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.g = torch.Generator(device=self.dev).manual_seed(seed)

    def normal(self, *shape, scale=1.0):
        return (torch.randn(*shape, generator=self.g, device=self.dev) * scale).to(BF16)

    def uniform(self, *shape, bound=1.0):
        return ((torch.rand(*shape, generator=self.g, device=self.dev) * 2 - 1) * bound).to(BF16)

    def outlier_channels(self, n, ratio):
        k = int(n * ratio)
        idx = torch.randperm(n, generator=self.g, device=self.dev)[:k]
        amp = 15 + 25 * torch.rand(k, generator=self.g, device=self.dev)
        return idx, amp

    def activation(self, b, m, n, idx, amp):
        """N(0, 1) with a few strong channels, as decoder activations have them."""
        x = torch.randn(b, m, n, generator=self.g, device=self.dev)
        x[:, :, idx] *= amp
        return x.to(BF16)

    def causal_map(self, b, h, rows, cols):
        """Softmax of causally masked N(0, 1) * 3 logits."""
        mask = torch.full((rows, cols), float("-inf"), device=self.dev).triu(1)
        out = torch.empty((b, h, rows, cols), dtype=BF16, device=self.dev)
        for i in range(b):
            out[i] = torch.softmax(3 * torch.randn(h, rows, cols, generator=self.g, device=self.dev) + mask, -1)
        return out


def _nf4_table(dev):
    """Sixteen quantiles of a standard normal, scaled to [-1, 1], with a zero among them."""
    pos = torch.special.ndtri(torch.linspace(0.9677083, 0.5, 9, dtype=torch.float64)[:-1])
    neg = -torch.special.ndtri(torch.linspace(0.9677083, 0.5, 8, dtype=torch.float64)[:-1])
    t = torch.cat([neg, torch.zeros(1, dtype=torch.float64), pos]).sort().values
    return (t / t.abs().max()).float().to(dev)


def _nf4_weight(w):
    """The weight as packed 4-bit codes with the quant state that describes them (blocks of 64)."""
    table = _nf4_table(w.device)
    blocks = w.float().view(-1, 64)
    absmax = blocks.abs().amax(1).clamp_(min=1e-12)
    codes = torch.bucketize(blocks / absmax[:, None], (table[1:] + table[:-1]) / 2).to(torch.uint8).view(-1)
    p = torch.nn.Parameter(((codes[0::2] << 4) | codes[1::2]).view(-1, 1), requires_grad=False)
    p.quant_state = types.SimpleNamespace(shape=tuple(w.shape), code=table, blocksize=64, dtype=BF16, quant_type="nf4",
                                          nested=False, absmax=absmax, state2=None, offset=None)
    return p


class _Base(torch.nn.Module):
    """A frozen projection."""

    def __init__(self, weight):
        super().__init__()
        self.weight = weight if isinstance(weight, torch.nn.Parameter) else torch.nn.Parameter(weight, requires_grad=False)
        self.bias = None


class _Adapter(torch.nn.Module):
    """One LoRA factor as a PEFT module dictionary holds it."""

    def __init__(self, weight):
        super().__init__()
        self.default = torch.nn.Module()
        self.default.weight = torch.nn.Parameter(weight)


def _prepare_layer(c, d):
    b, m, h, kv, inter = c["batch"], c["seq"], HIDDEN, KV_HEADS[c["model"]], INTER[c["model"]]
    dims = dict(q=(h, h), k=(kv * HEAD, h), v=(kv * HEAD, h), o=(h, h), gate=(inter, h), up=(inter, h), down=(h, inter))
    mods = {}
    for n in PROJ:
        out, inp = dims[n]
        w = d.normal(out, inp, scale=0.02)
        mods[n] = (_Base(_nf4_weight(w) if c["weights"] == "nf4" else w), _Adapter(d.uniform(R, inp, bound=inp ** -0.5)),
                   _Adapter(d.normal(out, R, scale=0.02)))
    idx, amp = d.outlier_channels(h, 0.005)
    pos = torch.arange(m, dtype=torch.float32, device=d.dev)
    inv = 1.0 / (10000.0 ** (torch.arange(0, HEAD, 2, dtype=torch.float32, device=d.dev) / HEAD))
    emb = torch.cat([torch.outer(pos, inv)] * 2, -1)
    mask = torch.full((m, m), torch.finfo(BF16).min, device=d.dev).triu(1).to(BF16).reshape(1, 1, m, m)
    layer = FusedLlamaLayerIntraInterFullFuse()
    layer.set_hyclora_config(types.SimpleNamespace(use_hyclora=True, iteration_threshold=5, softmax_outlier_ratio=0.05,
                                                   layernorm_outlier_ratio=0.005, q_bit=c["q"], softmax_map_mode=c["map"]))
    rest = [1 + d.normal(h, scale=0.1), None, emb.cos().to(BF16), emb.sin().to(BF16)]
    for n in PROJ[:4]:
        rest += mods[n]
    rest += [1 + d.normal(h, scale=0.1), None]
    for n in PROJ[4:]:
        rest += mods[n]
    rest += [mask, HEADS, HEAD, kv]
    with torch.no_grad():
        for _ in range(5):                           # the calibration iterations of a run
            layer(d.activation(b, m, h, idx, amp), *rest)
    lora = [mods[n][j].default.weight for n in PROJ for j in (1, 2)]
    return dict(layer=layer, rest=rest, lora=lora, x=d.activation(b, m, h, idx, amp).requires_grad_(True), gy=d.normal(b, m, h))


def _prepare_mlp(c, d):
    b, m, h, inter = c["batch"], c["seq"], HIDDEN, INTER[c["model"]]
    w = mlp.MLPWeights(norm_w=1 + d.normal(h, scale=0.1), wg=d.normal(inter, h, scale=0.02), wu=d.normal(inter, h, scale=0.02),
                       wd=d.normal(h, inter, scale=0.02), ag=d.uniform(R, h, bound=h ** -0.5), bg=d.normal(inter, R, scale=0.02),
                       au=d.uniform(R, h, bound=h ** -0.5), bu=d.normal(inter, R, scale=0.02),
                       ad=d.uniform(R, inter, bound=inter ** -0.5), bd=d.normal(h, R, scale=0.02))
    idx, amp = d.outlier_channels(h, 0.005)
    state = mlp.MLPState(q_bit=c["q"], layernorm_outlier_ratio=0.005)
    status = torch.zeros(1, dtype=torch.int32, device=d.dev)
    for _ in range(5):
        mlp.mlp_forward(d.activation(b, m, h, idx, amp), w, state, status=status)
    return dict(w=w, mlp_state=state, status=status, x=d.activation(b, m, h, idx, amp), gy=d.normal(b, m, h))


def _prepare_channel(c, d):
    b, m, n, q = c["batch"], c["seq"], c["n"], c["q"]
    idx, amp = d.outlier_channels(n, max(c["ratio"], 0.005))
    calib, x = d.activation(b, m, n, idx, amp), d.activation(b, m, n, idx, amp)
    if c["form"] == "outlier":
        o_idx, scale = cf.get_statistics_channel_base(calib, c["ratio"], q, "per-channel")
        return dict(x=x, static={"outlier_channel_index": o_idx, "scale": scale})
    if c["form"] == "zero_point":
        scale, zp = cf.get_statistics_only_quant_zero_point(calib, q, "per-channel")
        return dict(x=x, static={"scale": scale, "zero_point": zp})
    return dict(x=x, static={"scale": cf.get_statistics_only_quant(calib, q, "per-channel")})


def _prepare_silu(c, d):
    b, m, n, q = c["batch"], c["seq"], c["n"], c["q"]
    x1, x2 = d.normal(b, m, n), d.normal(b, m, n)
    return dict(xa1=d.normal(b, m, R), b1=d.normal(n, R, scale=0.02).t(), x1=x1, s1=cf.get_statistics_only_quant(x1, q, "per-channel"),
                xa2=d.normal(b, m, R), b2=d.normal(n, R, scale=0.02).t(), x2=x2, s2=cf.get_statistics_only_quant(x2, q, "per-channel"),
                g=d.normal(b, m, n))


def prepare(case, seed):
    d, kind = _Draws(seed), case["kind"]
    if kind == "layer":
        state = _prepare_layer(case, d)
    elif kind == "mlp":
        state = _prepare_mlp(case, d)
    elif kind == "map":
        a = d.causal_map(case["batch"], case["heads"], case["rows"], case["cols"])
        state = dict(a=a, g=d.normal(*a.shape))
    elif kind == "prune":
        a = d.causal_map(case["batch"], case["heads"], case["seq"], case["seq"])
        thr = cf.get_statistics_softmax(a[:1, :4], case["ratio"])
        state = dict(a=a, outlier=thr, threshold=float(thr))
    elif kind == "channel":
        state = _prepare_channel(case, d)
    else:
        state = _prepare_silu(case, d)
    state["case"] = case
    return state


# ------------------------------------------------------------------ one pass

def run(state):
    c = state["case"]
    kind, q = c["kind"], c.get("q")
    if kind == "layer":
        y = state["layer"](state["x"], *state["rest"])
        return [y.detach(), *torch.autograd.grad(y, [state["x"]] + state["lora"], state["gy"])]
    if kind == "mlp":
        y, saved = mlp.mlp_forward(state["x"], state["w"], state["mlp_state"], status=state["status"])
        g = mlp.mlp_backward(state["gy"], saved, state["w"], status=state["status"])
        return [y] + [g["grad_" + n] for n in ("x", "ag", "bg", "au", "bu", "ad", "bd")]
    if kind == "map":
        m = cf.compression_softmax_topk(state["a"], c["ratio"], q)
        return [*m.tensors(), m.to_dense(), m.softmax_backward(state["g"], scale=HEAD ** -0.5)]
    if kind == "prune":
        if c["form"] == "sparse":
            m, _ = cf.compression_pack_softmax_base(state["a"], c["ratio"], 5, 5, {"outlier": state["outlier"]})
            return [m._nnz(), cf.decompression_softmax(m)]       # the list's length and the map it stands for
        m = cf.compression_softmax_static(state["a"], state["threshold"], ratio=c["ratio"])
        return [m.nnz, m.to_dense()]
    if kind == "channel":
        if c["form"] == "outlier":
            o, codes, idx, scale = cf.compression_pack_channel_base(state["x"], c["ratio"], q, "per-channel", 5, 5, state["static"])
            return [o, codes, cf.outlier_addition_fuse_decompression_dequantization(codes, scale, o, idx, q)]
        if c["form"] == "zero_point":
            codes, scale, zp = cf.compression_pack_quant_zp_base(state["x"], q, "per-channel", 5, 5, state["static"])
            return [codes, cf.decompression_dequantization_with_zero_point(codes, scale, zp, q)]
        codes, scale = cf.compression_pack_quant_base(state["x"], q, "per-channel", 5, 5, state["static"])
        return [codes, cf.decompression_dequantization(codes, scale, q)]
    s = state
    q1, q2, o = triton_fuse_silu_forward(s["xa1"], s["b1"], s["x1"], s["s1"], s["xa2"], s["b2"], s["x2"], s["s2"], q)
    return [q1, q2, o, *triton_fuse_silu_backward(s["xa1"], s["b1"], q1, s["s1"], s["xa2"], s["b2"], q2, s["s2"], s["g"], q)]


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """Bytes: every input (weights included) once, every output once.  Operations: the products of the pass; the
    attention products over the causal half of the map."""
    c, kind, q = case, case["kind"], case.get("q", 0)
    if kind in ("layer", "mlp"):
        t, h, inter = c["batch"] * c["seq"], HIDDEN, INTER[c["model"]]
        mlp_w, attn_w = 3 * h * inter, 0
        adapters = R * (3 * h + 3 * inter)
        flops = 4 * t * mlp_w + 6 * t * adapters
        if kind == "layer":
            kv = KV_HEADS[c["model"]] * HEAD
            attn_w = 2 * h * h + 2 * h * kv
            more = R * (6 * h + 2 * kv)
            adapters += more
            # scores and P V forward, four such products backward, each 2 x (seq^2 / 2) x head per head
            flops += 4 * t * attn_w + 6 * t * more + 6 * c["batch"] * HEADS * HEAD * c["seq"] ** 2
        per_weight = 0.5 + 4 / 64 if c.get("weights") == "nf4" else 2
        return {"bytes": (mlp_w + attn_w) * per_weight + 4 * adapters + 2 * 4 * t * h, "flops": flops}
    if kind == "map":
        rows, s = c["batch"] * c["heads"] * c["rows"], c["cols"]
        saved = rows * (s * q // 8 + 3 * (s // 64) + 4 * int(s * c["ratio"]))
        return {"bytes": 2 * rows * s * 4 + saved, "flops": 0}
    if kind == "prune":
        n = c["batch"] * c["heads"] * c["seq"] ** 2
        return {"bytes": 2 * n * 2 + n * c["ratio"] * (10 if c["form"] == "sparse" else 4), "flops": 0}
    n = c["batch"] * c["seq"] * c["n"]
    if kind == "channel":
        return {"bytes": n * (2 + q / 8 + 2) + 2 * c["batch"] * c["seq"] * int(c["n"] * c["ratio"]), "flops": 0}
    return {"bytes": n * ((4 + 2 * q / 8 + 2) + (2 + 6)), "flops": 2 * 4 * c["batch"] * c["seq"] * R * c["n"]}


def tolerance(case):
    kind = case["kind"]
    if kind in ("prune", "channel"):
        return "exact"                   # stored values, indices, codes and what is rebuilt from them
    if kind == "map":
        return {"rel": 5e-3}             # the save is whole numbers and copies; the softmax backward ends in bf16
    if kind == "silu":
        return {"rel": 5e-3, "differ": 0.0}
    # gradients come from codes of computed tensors: where a last-bit difference of a bf16 value lies on the edge between
    # two codes, the restored value moves by a whole quantizer step (the coarser, the fewer bits)
    if kind == "mlp":
        return {"rel": 2e-2 if case["q"] == 2 else 1e-2}
    return {"rel": 2e-2}
