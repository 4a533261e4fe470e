"""The attention kernels (probabilities + P V + codes, and the backward pass from the restored map) against the separate
steps with the same rounding points, at the edges of their 128-row tiles.

Tolerances: reference and kernel share every inner rounding to bf16, so apart from the few elements whose fp32 sums fall
on different sides of a rounding edge a result differs by its own rounding, at most 2^-8 of the value; the probabilities
differ where a score does (bf16 scores of size 8: a step of 2^-5 in the exponent, 3 % of one entry), bounded in norm."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF16 = torch.bfloat16


def _mask(kind, g, B, h, M):
    low = torch.finfo(BF16).min
    causal = torch.full((M, M), low).triu(1).reshape(1, 1, M, M)
    if kind == "causal":
        return causal.to(BF16).to(DEV)
    if kind == "padded":                       # the first quarter of sample 0 is padding: rows there attend to nothing
        m = causal.repeat(B, 1, 1, 1)
        m[0, :, :, :M // 4] = low
        return m.to(BF16).to(DEV)
    if kind == "heads":
        return (torch.randn(B, h, M, M, generator=g) * 2).to(BF16).to(DEV)
    if kind == "inf":
        return causal.masked_fill(causal < 0, float("-inf")).to(BF16).to(DEV)
    return None


def _rel(x, y):
    return float((x.double() - y.double()).norm() / y.double().norm())


@pytest.mark.parametrize("B,M,h,kv,kind,q", [(1, 128, 1, 1, None, 4), (1, 8, 2, 2, "causal", 8), (2, 200, 4, 2, "causal", 2),
                                             (1, 256, 2, 1, "causal", 4), (2, 392, 2, 2, "padded", 4), (1, 520, 3, 3, "heads", 4),
                                             (1, 136, 4, 2, "heads", 8), (1, 1096, 2, 2, "inf", 4), (1, 4096, 1, 1, "causal", 4)])
def test_attention_forward_backward(B, M, h, kv, kind, q):
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    from hyc_lora_release_b200.operators import compress_function as cf
    g = torch.Generator().manual_seed(M + h)
    d, n = 128, h // kv
    rn = lambda *s: torch.randn(*s, generator=g).to(BF16).to(DEV)
    qx, kx, vx, go = rn(B, M, h * d), rn(B, M, kv * d), rn(B, M, kv * d), rn(B, M, h * d)
    mask, scale = _mask(kind, g, B, h, M), 1 / math.sqrt(d)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    a, o = torch.full((B, h, M, M), float("nan"), dtype=BF16, device=DEV), torch.empty((B, M, h * d), dtype=BF16, device=DEV)
    osc, oc = torch.full((h * d,), 0.2, dtype=BF16, device=DEV), torch.empty((B, M, h * d * q // 8), dtype=torch.uint8, device=DEV)
    cls, cb, ch, strides = None, 0, 0, (0, 0, 0)
    if mask is not None:
        nb, nh = mask.shape[:2]
        strides = (0 if nb == 1 else mask.stride(0), 0 if nh == 1 else mask.stride(1), mask.stride(2))
        cls = torch.empty(lib.hyc_attn_mask_class_bytes(nb, nh, M), dtype=torch.uint8, device=DEV)
        check(lib.hyc_attn_mask_class(ptr(mask), *strides, nb, nh, M, ptr(cls), stream_of(qx)), "class")
        cb, ch = (0 if nb == 1 else nh), (0 if nh == 1 else 1)
    check(lib.hyc_attn_fwd_tcgen05(ptr(qx), ptr(kx), ptr(vx), B, M, h, kv, d, scale, ptr(mask), *strides, ptr(cls), cb, ch, ptr(a), ptr(o),
                                   ptr(osc), ptr(oc), q, ptr(st), stream_of(qx)), "fwd")
    assert int(st.item()) == 0
    heads = lambda t, m: t.view(B, M, m, d).transpose(1, 2).repeat_interleave(h // m, 1)
    hid = lambda t: t.transpose(1, 2).reshape(B, M, -1)
    qh, kh, vh, gh = heads(qx, h).float(), heads(kx, kv).float(), heads(vx, kv).float(), heads(go, h).float()
    t = ((qh @ kh.transpose(-1, -2)).to(BF16).float() * scale).to(BF16)
    if mask is not None:
        t = t + mask
    ref = torch.softmax(t.float(), -1)
    assert bool(torch.isfinite(a).all()) and _rel(a, ref) < 2 ** -8
    # the rest on the emitted tensors: o, its codes, and the gradients from a pruned map
    assert _rel(o, hid(a.float() @ vh)) < 2 ** -8
    assert torch.equal(oc, cf.compression_quantization(o, osc.view(1, -1), q))
    p = torch.where(a > 0.01, a, torch.zeros_like(a))
    da = (gh @ vh.transpose(-1, -2)).to(BF16)
    ds = ((da.float() - (p * da).float().sum(-1, keepdim=True)) * p.float()).to(BF16)
    ds = (ds.float() * scale).to(BF16)
    group = lambda x: x.view(B, kv, n, M, d).sum(2)
    want = (hid(ds.float() @ kh), hid(group(ds.float().transpose(-1, -2) @ qh)), hid(group(p.float().transpose(-1, -2) @ gh)))
    got = [torch.full_like(x, float("nan")) for x in (qx, kx, vx)]
    gs = torch.empty_like(a)
    check(lib.hyc_attn_bwd_tcgen05(ptr(qx), ptr(kx), ptr(vx), ptr(go), ptr(p), ptr(gs), B, M, h, kv, d, scale, ptr(cls), cb, ch,
                                   ptr(got[0]), ptr(got[1]), ptr(got[2]), ptr(st), stream_of(qx)), "bwd")
    assert int(st.item()) == 0
    for x, y in zip(got, want):
        assert bool(torch.isfinite(x).all()) and _rel(x, y) < 2 ** -8
    # shapes outside the kernels are refused before any launch
    assert lib.hyc_attn_fwd_tcgen05(ptr(qx), ptr(kx), ptr(vx), B, M, h, kv, 64, scale, None, 0, 0, 0, None, 0, 0, None, ptr(o), None, None,
                                    q, ptr(st), stream_of(qx)) == -8


@pytest.mark.parametrize("case", ["levels", "lowest", "nan"])
def test_rows_without_a_passing_or_a_finite_entry(case):
    """Rows masked everywhere, with masks of two levels (the higher one takes all) and with the type's lowest value next to -inf
    (equal shares of the former), and NaN scores that fill whole quarters of a row's tile (the whole row is NaN, as in a
    softmax): the probabilities of the reference."""
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    g = torch.Generator().manual_seed(11)
    B, M, h, d = 1, 264, 2, 128
    rn = lambda *s: torch.randn(*s, generator=g).to(BF16).to(DEV)
    qx, kx, vx = rn(B, M, h * d), rn(B, M, h * d), rn(B, M, h * d)
    mask = torch.zeros(1, 1, M, M)
    if case == "levels":
        mask[..., :M // 2, :] = -2e30
        mask[..., :M // 2, ::3] = -4e30
        mask[..., :M // 2, 200:] = -8e30
    elif case == "lowest":
        mask[..., :M // 2, :] = float("-inf")
        mask[..., :M // 2, 40:200] = torch.finfo(BF16).min
    else:
        kx[:, 32:96, :d] = float("nan")          # head 0
    mask = mask.to(BF16).to(DEV)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    a, o = torch.zeros((B, h, M, M), dtype=BF16, device=DEV), torch.empty((B, M, h * d), dtype=BF16, device=DEV)
    cls = torch.empty(lib.hyc_attn_mask_class_bytes(1, 1, M), dtype=torch.uint8, device=DEV)
    check(lib.hyc_attn_mask_class(ptr(mask), 0, 0, M, 1, 1, M, ptr(cls), stream_of(qx)), "class")
    check(lib.hyc_attn_fwd_tcgen05(ptr(qx), ptr(kx), ptr(vx), B, M, h, h, d, 1 / math.sqrt(d), ptr(mask), 0, 0, M, ptr(cls), 0, 0, ptr(a), ptr(o),
                                   None, None, 4, ptr(st), stream_of(qx)), "fwd")
    assert int(st.item()) == 0
    heads = lambda t: t.view(B, M, h, d).transpose(1, 2).float()
    t = ((heads(qx) @ heads(kx).transpose(-1, -2)).to(BF16).float() / math.sqrt(d)).to(BF16) + mask
    ref = torch.softmax(t.float(), -1)
    assert torch.equal(a.isnan(), ref.isnan())
    assert _rel(a.nan_to_num(), ref.nan_to_num()) < 2 ** -8


@pytest.mark.parametrize("B,M,h,kv,kind", [(1, 8, 1, 1, None), (2, 136, 4, 2, "causal"), (1, 264, 2, 1, "padded"), (1, 1096, 2, 2, "causal")])
def test_map_up_to_the_columns_that_are_reported(B, M, h, kv, kind):
    """With row_cols the map is the same up to those columns, nothing is written behind them and zeros would have been."""
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    g = torch.Generator().manual_seed(M)
    d, scale = 128, 128 ** -0.5
    rn = lambda *s: torch.randn(*s, generator=g).to(BF16).to(DEV)
    qx, kx, vx = rn(B, M, h * d), rn(B, M, kv * d), rn(B, M, kv * d)
    mask, st = _mask(kind, g, B, h, M), torch.zeros(1, dtype=torch.int32, device=DEV)
    cls, cb, strides = None, 0, (0, 0, 0)
    if mask is not None:
        nb = mask.shape[0]
        cb, strides = 0 if nb == 1 else 1, (0 if nb == 1 else mask.stride(0), 0, mask.stride(2))
        cls = torch.empty(lib.hyc_attn_mask_class_bytes(nb, 1, M), dtype=torch.uint8, device=DEV)
        check(lib.hyc_attn_mask_class(ptr(mask), *strides, nb, 1, M, ptr(cls), stream_of(qx)), "class")
    maps, outs = [torch.full((B, h, M, M), -1.0, dtype=BF16, device=DEV) for _ in range(2)], [torch.empty_like(qx) for _ in range(2)]
    cols = torch.empty(B * h * M, dtype=torch.int16, device=DEV)
    fwd = (ptr(qx), ptr(kx), ptr(vx), B, M, h, kv, d, scale, ptr(mask), *strides, ptr(cls), cb, 0)
    check(lib.hyc_attn_fwd_tcgen05(*fwd, ptr(maps[0]), ptr(outs[0]), None, None, 4, ptr(st), stream_of(qx)), "fwd")
    check(lib.hyc_attn_fwd_cols_tcgen05(*fwd, ptr(maps[1]), ptr(cols), ptr(outs[1]), None, None, 4, ptr(st), stream_of(qx)), "fwd")
    inside = (torch.arange(M, device=DEV)[None] < cols[:, None]).view(B, h, M, M)
    assert int(st.item()) == 0 and torch.equal(*outs)
    assert torch.equal(maps[0][inside], maps[1][inside]) and bool((maps[0][~inside] == 0).all()) and bool((maps[1][~inside] == -1).all())
    if kind == "causal":
        assert torch.equal(cols.view(B * h, M)[0], ((torch.arange(M) // 128 + 1) * 128).clamp(max=M).to(torch.int16).to(DEV))
