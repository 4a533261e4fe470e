"""4-bit block-wise frozen weights: the CPU statement of the storage format (oracle/nf4.py), the CUDA de-quantizer
against it bit for bit, and the fused layer driven with such weights against the same layer driven with the
de-quantized matrices.  (The library whose format this is, bitsandbytes 0.43.2, is not present: parity with it is
unpinned, see oracle/nf4.py.)"""
import types

import pytest
import torch

from oracle import nf4 as onf4

BF16 = torch.bfloat16


def test_format_statement_round_trip():
    """Nibble order, block maxima and the nested form, on the CPU."""
    table = onf4.normal_float_table()
    assert table.numel() == 16 and float(table[0]) == -1.0 and float(table[-1]) == 1.0 and float(table[7]) == 0.0
    assert bool((table[1:] > table[:-1]).all())
    g = torch.Generator().manual_seed(3)
    w = (torch.randn(48, 64, generator=g) * 0.02).to(BF16)
    packed, qs = onf4.quantize_4bit(w, table, blocksize=64)
    assert packed.shape == (48 * 64 // 2, 1) and packed.dtype == torch.uint8 and qs.absmax.numel() == 48
    # element 0 sits in the HIGH nibble of byte 0
    first = int(packed[0, 0])
    blk0 = float(qs.absmax[0])
    assert abs(float(table[first >> 4]) * blk0 - float(w.reshape(-1)[0])) <= 0.2 * blk0
    back = onf4.ref_dequantize_4bit(packed, qs)
    assert back.shape == w.shape and back.dtype == BF16
    err = (back.float() - w.float()).abs().max() / w.float().abs().max()
    assert float(err) < 0.2                      # half the widest gap of the table, relative to a block maximum
    # exact at the block maxima and at zero
    z = torch.zeros(2, 64); z[0, 5] = 1.5; z[1, 9] = -0.25
    pz, qz = onf4.quantize_4bit(z.to(BF16), table, blocksize=64)
    bz = onf4.ref_dequantize_4bit(pz, qz).float()
    assert float(bz[0, 5]) == 1.5 and float(bz[1, 9]) == -0.25 and float(bz.abs().sum()) == 1.75
    # nested: the maxima come back within the resolution of the 8-bit table
    pn, qn = onf4.quantize_4bit(w, table, blocksize=64, nested=True, blocksize2=16)
    assert qn.absmax.dtype == torch.uint8 and qn.state2.absmax.numel() == 3
    m = onf4.block_maxima(qn)
    assert float((m - qs.absmax).abs().max()) < 0.05 * float(qs.absmax.max())


@pytest.mark.gpu
@pytest.mark.parametrize("shape,blocksize,nested", [((64, 64), 64, False), ((256, 1024), 64, False), ((300, 130), 64, False),
                                                   ((128, 512), 128, True), ((96, 4096), 64, True), ((7, 6), 2, False)])
def test_dequantizer_matches_the_format_statement(shape, blocksize, nested):
    from hyc_lora_release_b200 import nf4
    table = onf4.normal_float_table()
    g = torch.Generator().manual_seed(shape[0] + shape[1])
    w = (torch.randn(*shape, generator=g) * 0.03).to(BF16)
    packed, qs = onf4.quantize_4bit(w, table, blocksize=blocksize, nested=nested, blocksize2=32)
    want = onf4.ref_dequantize_4bit(packed, qs)
    got = nf4.dequantize_nf4(packed.cuda(), qs)
    assert got.shape == tuple(shape) and got.dtype == BF16
    assert torch.equal(got.cpu(), want)
    # a parameter that carries its quant state, as the reference's modules hold it
    p = torch.nn.Parameter(packed.cuda(), requires_grad=False)
    p.quant_state = qs
    assert nf4.is_quantized(p) and torch.equal(nf4.dequantize_nf4(p).cpu(), want)


@pytest.mark.gpu
def test_layer_with_4bit_frozen_weights():
    """The layer module with 4-bit frozen weights gives bit for bit what it gives with the de-quantized matrices
    (of 256 rows: a launch de-quantizes them, the same kernels run on the same values), and it does not keep the bf16 matrices between
    the passes."""
    from hyc_lora_release_b200 import nf4
    from hyc_lora_release_b200.layer import FusedLlamaLayerIntraInterFullFuse
    from test_gpu_layer import layer_problem, _Holder, _base
    DEV = "cuda"
    g = torch.Generator().manual_seed(77)
    B, M, heads, d, kv, I, q = 2, 128, 4, 128, 2, 1024, 4
    H = heads * d
    x, p, cos, sin, mask = layer_problem(g, B, M, H, heads, d, kv, I)
    table = onf4.normal_float_table()
    cfg = types.SimpleNamespace(use_hyclora=True, iteration_threshold=5, softmax_outlier_ratio=0.05,
                                layernorm_outlier_ratio=0.01, q_bit=q, softmax_map_mode="prune")
    n1 = torch.nn.Parameter(p["norm_w1"].to(DEV), requires_grad=False)
    n2 = torch.nn.Parameter(p["norm_w2"].to(DEV), requires_grad=False)
    gy = torch.randn(B, M, H, generator=g).to(BF16).to(DEV)
    names = ("q", "k", "v", "o", "gate", "up", "down")
    quant = {}
    for i, n in enumerate(names):
        w = p["w" + n].t().contiguous()                       # [out, in]
        quant[n] = onf4.quantize_4bit(w, table, blocksize=64, nested=(i % 2 == 1), blocksize2=64)

    def run(four_bit):
        mods = {}
        for n in names:
            packed, qs = quant[n]
            if four_bit:
                base = torch.nn.Module()
                base.weight = torch.nn.Parameter(packed.to(DEV), requires_grad=False)
                base.weight.quant_state = qs
                base.bias = None
            else:
                base = _base(onf4.ref_dequantize_4bit(packed, qs).to(DEV))
            mods[n] = (base, _Holder(p["a" + n].t().to(DEV)), _Holder(p["b" + n].t().to(DEV)))
        layer = FusedLlamaLayerIntraInterFullFuse()
        layer.set_hyclora_config(cfg)
        layer.check_kernel_status = True
        outs = []
        for it in range(7):
            xin = x.to(DEV).requires_grad_(True)
            args = [xin, n1, None, cos.to(DEV), sin.to(DEV)]
            for n in ("q", "k", "v", "o"):
                args += list(mods[n])
            args += [n2, None]
            for n in ("gate", "up", "down"):
                args += list(mods[n])
            y = layer(*args, mask.to(DEV), heads, d, kv)
            for m3 in mods.values():
                m3[1].default.weight.grad = None
                m3[2].default.weight.grad = None
            y.backward(gy)
            outs.append((y.detach().clone(), xin.grad.clone(), [m3[k].default.weight.grad.clone() for m3 in mods.values() for k in (1, 2)]))
        return layer, outs

    layer4, o4 = run(True)
    layer16, o16 = run(False)
    for (y4, gx4, gl4), (y16, gx16, gl16) in zip(o4, o16):
        assert torch.equal(y4, y16) and torch.equal(gx4, gx16)
        assert all(torch.equal(a, b) for a, b in zip(gl4, gl16))
    aw, mw, _ = layer4._weights[1:]
    assert isinstance(aw.wq, nf4.QuantizedWeight) and isinstance(mw.wd, nf4.QuantizedWeight)
    assert "_pad" in vars(aw) and "_pad" in vars(mw)          # the scratch of the passes came back to the records


# which of a layer's products (q k v, o, gate and up, down, their backward products) decode their weights on the way in, by the SMs they fill
PRODUCTS = ("qkv", "o", "gateup", "down", "graddown", "gradx gu", "grado", "gradx qkv")


@pytest.mark.gpu
@pytest.mark.parametrize("B,M,heads,kv,I,inside", [
    (1, 128, 4, 2, 1024, ()), (1, 128, 32, 32, 11008, set(PRODUCTS) - {"o"}), (3, 40, 32, 32, 11008, set(PRODUCTS) - {"o"}),
    (1, 64, 24, 8, 9472, {"gateup", "down", "graddown", "gradx gu", "gradx qkv"}), (1, 64, 38, 2, 11008, set(PRODUCTS) - {"qkv", "o"})])
@pytest.mark.parametrize("coded,nested", [("q k v o gate up down", ""), ("q k v o gate up down", "q k v o gate up down"), ("q v gate down", "v down"), ("k o up", "k")])
def test_short_layers_with_4bit_frozen_weights(B, M, heads, kv, I, inside, coded, nested):
    """Up to 128 rows the products of a calibrated layer decode their weights where that pays, called and in a capture (``inside``): bit for bit
    the layer with the de-quantized matrices, with one- and two-level scales and with some projections plain (gate and up then count as
    matrices in the forward pass)."""
    from hyc_lora_release_b200 import nf4
    from hyc_lora_release_b200._lib import lib
    from hyc_lora_release_b200.layer import FusedLlamaLayerIntraInterFullFuse
    from test_gpu_layer import _Holder, _base
    d, R = 128, 16
    H, D, Dkv, T = heads * d, heads * d, kv * d, B * M
    g = torch.Generator(device="cuda").manual_seed(H + T + len(coded))
    rn = lambda *s, scale=1.0: (torch.randn(*s, generator=g, device="cuda") * scale).to(BF16)
    fixed, gate_up, down = 2, 16, 32
    want = {"qkv": (fixed, D + 2 * Dkv, H), "o": (fixed, H, D + 64), "gateup": (gate_up, I, H), "down": (0, H, I + 64), "graddown": (down, I, H + 64),
            "gradx gu": (0, H, 2 * I + 64), "grado": (0, D, H + 64), "gradx qkv": (0, H, D + 2 * Dkv + 64)}
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert {n for n in PRODUCTS if lib.hyc_nf4_product_pays(want[n][0], T, *want[n][1:], 1)} == set(inside)
        assert {n for n in PRODUCTS if lib.hyc_nf4_product_pays(want[n][0], T, *want[n][1:], 0)} == set(inside) | set(PRODUCTS) - {"qkv", "o"}
    shapes = dict(q=(D, H), k=(Dkv, H), v=(Dkv, H), o=(H, D), gate=(I, H), up=(I, H), down=(H, I))
    table = onf4.normal_float_table().cuda()
    base4, base16, lora = {}, {}, {}
    for n, (rows, cols) in shapes.items():
        num = rows * cols
        qs = types.SimpleNamespace(shape=(rows, cols), code=table, blocksize=64, dtype=BF16, nested=n in nested.split())
        if qs.nested:
            qs.absmax = torch.randint(0, 256, (num // 64,), generator=g, dtype=torch.uint8, device="cuda")
            qs.state2 = types.SimpleNamespace(code=torch.linspace(0, 1, 256), blocksize=256, absmax=(torch.rand((num // 64 + 255) // 256, generator=g, device="cuda") + 0.5) * 0.03)
            qs.offset = 0.01
        else:
            qs.absmax = (torch.rand(num // 64, generator=g, device="cuda") + 0.5) * 0.03
        packed = torch.nn.Parameter(torch.randint(0, 256, (num // 2, 1), generator=g, dtype=torch.uint8, device="cuda"), requires_grad=False)
        packed.quant_state = qs
        base16[n] = _base(nf4.dequantize_nf4(packed))
        base4[n] = base16[n]
        if n in coded.split():
            base4[n] = torch.nn.Module()
            base4[n].weight, base4[n].bias = packed, None
        lora[n] = _Holder(rn(R, cols, scale=cols ** -0.5)), _Holder(rn(rows, R, scale=0.05))
    norms = [torch.nn.Parameter(1 + rn(H, scale=0.1), requires_grad=False) for _ in range(2)]
    fr = torch.outer(torch.arange(M, dtype=torch.float32), 1.0 / (10000.0 ** (torch.arange(0, d, 2, dtype=torch.float32) / d)))
    emb = torch.cat([fr, fr], dim=-1)
    cos, sin = emb.cos().to(BF16).cuda(), emb.sin().to(BF16).cuda()
    mask = torch.full((M, M), torch.finfo(BF16).min).triu(1).to(BF16).reshape(1, 1, M, M).cuda()
    x, gy = rn(B, M, H), rn(B, M, H)

    def run(base):
        layer = FusedLlamaLayerIntraInterFullFuse()
        layer.set_hyclora_config(types.SimpleNamespace(use_hyclora=True, iteration_threshold=1, softmax_outlier_ratio=0.05, layernorm_outlier_ratio=0.01,
                                                       q_bit=4, softmax_map_mode="prune"))
        layer.attn_state.prune_capacity_margin = 4.0      # (few batches for the 64 lists of the saved map: they fill unevenly)
        factors = [h.default.weight for n in lora for h in lora[n]]
        xin = x.clone().requires_grad_(True)

        def step():
            args = [xin, norms[0], None, cos, sin]
            for n in shapes:
                args += ([norms[1], None] if n == "gate" else []) + [base[n], *lora[n]]
            y = layer(*args, mask, heads, d, kv)
            return [y, *torch.autograd.grad(y, [xin] + factors, gy)]

        outs = [[t.detach().clone() for t in step()] for _ in range(3)]
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            step()
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                kept = step()
        graph.replay()
        torch.cuda.synchronize()
        layer.raise_on_device_errors()
        return outs + [[t.detach().clone() for t in kept]]

    for a, b in zip(run(base4), run(base16)):
        assert all(bool(torch.isfinite(t).all()) for t in a) and all(torch.equal(s, t) for s, t in zip(a, b))
