"""The launches that take several operands at once (q, k and v rebuilt from their codes, the rotary embedding of q and k, up
to four 4-bit weights) against the single forms, bit for bit: row remainders, grouped heads, both types of the
tables, weights with a tail and block sizes of their own."""
import ctypes

import pytest
import torch

from oracle import nf4 as onf4

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF16 = torch.bfloat16


def _tables(M, d, dtype):
    pos = torch.arange(M + 3, dtype=torch.float32)
    inv = 1.0 / (10000.0 ** (torch.arange(0, d, 2, dtype=torch.float32) / d))
    emb = torch.cat([torch.outer(pos, inv)] * 2, dim=-1)
    return emb.cos().to(dtype).to(DEV), emb.sin().to(dtype).to(DEV)


def _arr(ts):
    return (ctypes.c_void_p * len(ts))(*[t.data_ptr() for t in ts])


@pytest.mark.parametrize("table", [BF16, torch.float32])
@pytest.mark.parametrize("B,M,heads,kv,q", [(1, 1, 1, 1, 4), (1, 17, 4, 2, 8), (3, 37, 5, 1, 2), (2, 200, 32, 8, 4)])
def test_rebuild_qkv(B, M, heads, kv, q, table):
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    from hyc_lora_release_b200.operators import compress_function as cf, rope_kernels as rk
    g = torch.Generator().manual_seed(M + q)
    T, d = B * M, 128
    n = (heads * d, kv * d, kv * d)
    cos, sin = _tables(M, d, table)
    codes = [torch.randint(0, 256, (T, w * q // 8), generator=g).to(torch.uint8).to(DEV) for w in n]
    scales = [(0.05 + torch.rand(w, generator=g)).to(BF16).to(DEV) for w in n]
    xas = [torch.randn(T, 16, generator=g).to(BF16).to(DEV) for _ in n]
    bts = [torch.randn(w, 16, generator=g).to(BF16).to(DEV) for w in n]
    ys = [torch.full((T, w), float("nan"), dtype=BF16, device=DEV) for w in n]
    check(lib.hyc_rebuild_qkv(_arr(codes), _arr(scales), _arr(xas), _arr(bts), _arr(ys), (ctypes.c_int * 3)(*n), ptr(cos), ptr(sin), cos.stride(0),
                              1 if table == torch.float32 else 0, T, M, q, stream_of(cos)), "hyc_rebuild_qkv")
    for i, (c, s, xa, bt, y) in enumerate(zip(codes, scales, xas, bts, ys)):
        want = cf.decompression_dequantization_lora_add(c.view(1, T, -1), s.view(1, -1), xa.view(1, T, 16), bt.t(), q)
        if i < 2:
            want = rk.rope_forward(want.view(B, M, -1, d), cos, sin)
        assert torch.equal(y, want.reshape(T, -1)), "qkv"[i]


@pytest.mark.parametrize("table", [BF16, torch.float32])
@pytest.mark.parametrize("B,M,heads,kv,d", [(1, 1, 1, 1, 16), (3, 37, 5, 1, 64), (2, 200, 32, 8, 128), (1, 9, 70, 70, 128)])
@pytest.mark.parametrize("backward", [False, True])
def test_rope_pair(B, M, heads, kv, d, table, backward):
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    from hyc_lora_release_b200.operators import rope_kernels as rk
    g = torch.Generator().manual_seed(M + d)
    cos, sin = _tables(M, d, table)
    x0, x1 = (torch.randn(B, M, h, d, generator=g).to(BF16).to(DEV) for h in (heads, kv))
    one = rk.rope_backward if backward else rk.rope_forward
    want = one(x0, cos, sin), one(x1, cos, sin)
    check(lib.hyc_rope_pair(ptr(x0), heads, ptr(x1), kv, ptr(cos), ptr(sin), cos.stride(0), 1 if table == torch.float32 else 0, B * M, M, d,
                            1 if backward else 0, stream_of(x0)), "hyc_rope_pair")
    assert torch.equal(x0, want[0]) and torch.equal(x1, want[1])


class Nf4Job(ctypes.Structure):
    _fields_ = [("packed", ctypes.c_void_p), ("code16", ctypes.c_void_p), ("absmax", ctypes.c_void_p), ("absmax_q", ctypes.c_void_p),
                ("code256", ctypes.c_void_p), ("absmax2", ctypes.c_void_p), ("out", ctypes.c_void_p), ("numel", ctypes.c_int64),
                ("blocksize", ctypes.c_int), ("blocksize2", ctypes.c_int), ("offset", ctypes.c_float)]


@pytest.mark.parametrize("parts", [[((7, 6), 2, False)], [((300, 130), 64, False), ((128, 512), 128, True)],
                                   [((96, 4096), 64, True), ((5, 2), 64, False), ((33, 62), 24, False)],
                                   [((64, 64), 4096, False), ((31, 66), 32, True), ((256, 1024), 64, False), ((1, 2), 2, True)]])
def test_nf4_weights_in_one_launch(parts):
    from hyc_lora_release_b200._lib import check, lib, stream_of
    table = onf4.normal_float_table()
    jobs, keep, want = (Nf4Job * len(parts))(), [], []
    for j, (shape, blocksize, nested) in zip(jobs, parts):
        g = torch.Generator().manual_seed(shape[0])
        packed, qs = onf4.quantize_4bit((torch.randn(*shape, generator=g) * 0.03).to(BF16), table, blocksize=blocksize, nested=nested, blocksize2=24)
        want.append(onf4.ref_dequantize_4bit(packed, qs))
        t = [packed.to(DEV), qs.code.to(DEV), qs.absmax.to(DEV), torch.zeros(shape, dtype=BF16, device=DEV)]
        j.packed, j.code16, j.out, j.numel, j.blocksize, j.blocksize2 = t[0].data_ptr(), t[1].data_ptr(), t[3].data_ptr(), t[3].numel(), blocksize, 1
        if nested:
            t += [qs.state2.code.to(DEV), qs.state2.absmax.to(DEV)]
            j.absmax_q, j.code256, j.absmax2, j.blocksize2, j.offset = t[2].data_ptr(), t[4].data_ptr(), t[5].data_ptr(), 24, float(qs.offset)
        else:
            j.absmax = t[2].data_ptr()
        keep.append(t)
    check(lib.hyc_dequant_nf4_many(len(parts), jobs, stream_of(keep[0][0])), "hyc_dequant_nf4_many")
    for t, w in zip(keep, want):
        assert torch.equal(t[3].cpu(), w)


@pytest.mark.parametrize("nested", [False, True])
@pytest.mark.parametrize("blocksize,packed_off,out_off", [(64, 0, 0), (64, 4, 0), (64, 0, 8), (48, 8, 16), (16, 0, 0), (8, 0, 0), (4096, 8, 16)])
def test_nf4_lanes_of_sixteen_and_of_eight(blocksize, packed_off, out_off, nested):
    """16 elements per lane where they share a scale and the tensors start on 8 and 32 bytes, eight elsewhere: the same values."""
    from hyc_lora_release_b200._lib import check, lib, stream_of
    g = torch.Generator().manual_seed(blocksize + packed_off)
    w = (torch.randn(3, 1024 * 5 + 62, generator=g) * 0.03).to(BF16)
    packed, qs = onf4.quantize_4bit(w, onf4.normal_float_table(), blocksize=blocksize, nested=nested, blocksize2=32)
    want = onf4.ref_dequantize_4bit(packed, qs).flatten()
    n = want.numel()
    p = torch.zeros(packed.numel() + 16, dtype=torch.uint8, device=DEV)
    p[packed_off:packed_off + packed.numel()] = packed.flatten().to(DEV)
    out = torch.full((n + 48,), -3.0, dtype=BF16, device=DEV)
    t = [qs.code.to(DEV), qs.absmax.to(DEV)] + ([qs.state2.code.to(DEV), qs.state2.absmax.to(DEV)] if nested else [])
    v = lambda x: ctypes.c_void_p(x.data_ptr())
    check(lib.hyc_dequant_nf4(ctypes.c_void_p(p.data_ptr() + packed_off), v(t[0]), None if nested else v(t[1]), v(t[1]) if nested else None,
                              v(t[2]) if nested else None, v(t[3]) if nested else None, 32, float(qs.offset) if nested else 0.0, n, blocksize,
                              ctypes.c_void_p(out.data_ptr() + 2 * out_off), stream_of(out)), "hyc_dequant_nf4")
    got = out.cpu()
    assert torch.equal(got[out_off:out_off + n], want)
    assert (got[:out_off] == -3.0).all() and (got[out_off + n:] == -3.0).all()
