"""Products that decode their 4-bit weights on the way in: the same bits as de-quantizing first, at the edges of the row tile, with K
shared by one, two and four CTAs, an odd number of k-blocks, one- and two-level scales, and next to operands that are bf16.  (The C entries; a
layer that takes them: test_nf4.py.)"""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16 = "cuda", torch.bfloat16


class Codes(ctypes.Structure):
    _fields_ = [(n, ctypes.c_void_p) for n in ("packed", "code16", "absmax", "absmax_q", "code256", "absmax2")] + [
        ("blocksize", ctypes.c_int), ("blocksize2", ctypes.c_int), ("offset", ctypes.c_float)]


def _weight(g, rows, cols, block, nested):
    """-> (codes, the bf16 matrix they stand for, what has to stay alive)"""
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    n = rows * cols
    packed = torch.randint(0, 256, (n // 2,), generator=g, dtype=torch.uint8).to(DEV)
    code = torch.randn(16, generator=g).to(DEV)
    absmax = (torch.rand(n // block, generator=g) * 0.1 + 0.01).to(DEV)
    q, code2, absmax2 = None, None, None
    if nested:
        q = torch.randint(0, 256, (n // block,), generator=g, dtype=torch.uint8).to(DEV)
        code2 = torch.rand(256, generator=g).to(DEV)
        absmax2 = (torch.rand((n // block + 255) // 256, generator=g) * 0.1 + 0.01).to(DEV)
    out = torch.empty(rows, cols, dtype=BF16, device=DEV)
    check(lib.hyc_dequant_nf4(ptr(packed), ptr(code), None if nested else ptr(absmax), ptr(q), ptr(code2), ptr(absmax2), 256, 0.02, n, block, ptr(out),
                              stream_of(out)), "dequant")
    c = Codes(ptr(packed), ptr(code), None if nested else ptr(absmax), ptr(q), ptr(code2), ptr(absmax2), block, 256, 0.02)
    assert lib.hyc_nf4_product_supported(ctypes.byref(c), 128, cols) == 1 and lib.hyc_nf4_product_supported(ctypes.byref(c), 129, cols) == 0
    return c, out, (packed, code, absmax, q, code2, absmax2)


def _ptrs(ts):
    return (ctypes.c_void_p * len(ts))(*[t.data_ptr() if t is not None else None for t in ts])


@pytest.mark.parametrize("T", [1, 63, 64, 65, 127, 128])
@pytest.mark.parametrize("K,block,nested", [(64, 64, False), (320, 64, True), (2048, 128, True), (4096, 64, False)])
@pytest.mark.parametrize("b_is_kn", [0, 1])
def test_segments(T, K, block, nested, b_is_kn):
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    g = torch.Generator().manual_seed(T + K + b_is_kn)
    rn = lambda *s: torch.randn(*s, generator=g).to(BF16).to(DEV)
    N = 512
    # two coded operands and a bf16 one behind them
    ks = (K, 192, 64)
    shape = lambda k: (k, N) if b_is_kn else (N, k)
    w = [_weight(g, *shape(k), block, nested) for k in ks[:2]]
    last, a, res = rn(*shape(64)), [rn(T, k) for k in ks], rn(T, N)
    st, kk = torch.zeros(1, dtype=torch.int32, device=DEV), (ctypes.c_int * 3)(*ks)
    want, got = torch.empty(T, N, dtype=BF16, device=DEV), torch.full((T, N), float("nan"), dtype=BF16, device=DEV)
    check(lib.hyc_gemm_segments_tcgen05(3, _ptrs(a), _ptrs([w[0][1], w[1][1], last]), kk, T, N, b_is_kn, ptr(res), ptr(want), ptr(st), stream_of(want)), "bf16")
    codes = (Codes * 3)(w[0][0], w[1][0], Codes())
    check(lib.hyc_gemm_segments_nf4_tcgen05(3, _ptrs(a), _ptrs([None, None, last]), codes, kk, T, N, b_is_kn, ptr(res), ptr(got), ptr(st), stream_of(got)), "nf4")
    assert int(st.item()) == 0 and torch.equal(got, want)


@pytest.mark.parametrize("T,q", [(1, 4), (65, 2), (128, 8)])
def test_projections(T, q):
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    g = torch.Generator().manual_seed(T)
    rn = lambda *s, sc=1.0: (torch.randn(*s, generator=g) * sc).to(BF16).to(DEV)
    H, I, st = 448, 512, torch.zeros(1, dtype=torch.int32, device=DEV)
    x, s1, s2 = rn(T, H), rn(I).abs() + 0.1, rn(I).abs() + 0.1
    xa, bt = [rn(T, 16) for _ in range(3)], [rn(I, 16, sc=.1) for _ in range(3)]
    gate, up = _weight(g, I, H, 64, False), _weight(g, I, H, 64, True)
    stream = stream_of(x)

    def gateup(coded):
        o = [torch.empty(T, I * q // 8, dtype=torch.uint8, device=DEV) for _ in range(2)] + [torch.empty(T, I, dtype=BF16, device=DEV)]
        w = [ctypes.byref((Codes * 2)(gate[0], up[0]))] if coded else [ptr(gate[1]), ptr(up[1])]
        f = lib.hyc_mlp_gateup_fwd_nf4_tcgen05 if coded else lib.hyc_mlp_gateup_fwd_tcgen05
        check(f(ptr(x), *w, T, H, I, ptr(xa[0]), ptr(bt[0]), 16, 1, ptr(xa[1]), ptr(bt[1]), 16, 1, ptr(s1), ptr(s2), *[ptr(t) for t in o], None, None, q,
                ptr(st), stream), "gateup")
        return o

    assert all(torch.equal(a, b) for a, b in zip(gateup(True), gateup(False)))
    # three weights side by side, the middle one bf16
    ns = (512, 256, 256)
    ws = [_weight(g, n, H, 64, False) for n in ns]
    sc = [rn(n).abs() + 0.1 for n in ns]

    def linears(coded):
        qo = [torch.empty(T, n * q // 8, dtype=torch.uint8, device=DEV) for n in ns]
        y = [torch.empty(T, n, dtype=BF16, device=DEV) for n in ns]
        tail = [(ctypes.c_int * 3)(*ns), _ptrs(xa), _ptrs(bt), _ptrs(sc), _ptrs(qo), _ptrs(y), q, ptr(st), stream]
        if coded:
            check(lib.hyc_linears_lora_save_fwd_nf4_tcgen05(ptr(x), T, H, 3, _ptrs([None, ws[1][1], None]), (Codes * 3)(ws[0][0], Codes(), ws[2][0]), *tail), "nf4")
        else:
            check(lib.hyc_linears_lora_save_fwd_tcgen05(ptr(x), T, H, 3, _ptrs([w[1] for w in ws]), *tail), "bf16")
        return qo + y

    assert all(torch.equal(a, b) for a, b in zip(linears(True), linears(False)))
    # backward of the down projection
    down, gy, gd, ad = _weight(g, H, I, 64, True), rn(T, H), rn(T, 64), rn(64, I, sc=.1)
    q1, q2 = [torch.randint(0, 256, (T, I * q // 8), generator=g, dtype=torch.uint8).to(DEV) for _ in range(2)]

    def graddown(coded):
        o = [torch.empty(T, I, dtype=BF16, device=DEV) for _ in range(3)]
        f = lib.hyc_mlp_graddown_bwd_nf4_tcgen05 if coded else lib.hyc_mlp_graddown_bwd_tcgen05
        check(f(ptr(gy), ctypes.byref(down[0]) if coded else ptr(down[1]), T, H, I, ptr(gd), ptr(ad), 64, ptr(xa[0]), ptr(bt[0]), 16, 1, ptr(xa[1]), ptr(bt[1]),
                16, 1, ptr(q1), ptr(s1), ptr(q2), ptr(s2), None, None, 0, *[ptr(t) for t in o], q, ptr(st), stream), "graddown")
        return o

    assert all(torch.equal(a, b) for a, b in zip(graddown(True), graddown(False)))
    assert int(st.item()) == 0


@pytest.mark.parametrize("T", [1, 128, 129, 300])
def test_no_codes(T):
    """Operands that are all bf16: the namesake's result, at any number of rows; a weight of codes behind 128 rows is refused."""
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    g = torch.Generator().manual_seed(T)
    rn = lambda *s: torch.randn(*s, generator=g).to(BF16).to(DEV)
    K, N, q = 192, 256, 4
    st, kk = torch.zeros(1, dtype=torch.int32, device=DEV), (ctypes.c_int * 2)(K, 64)
    a, b, out = [rn(T, K), rn(T, 64)], [rn(N, K), rn(N, 64)], [torch.full((T, N), float("nan"), dtype=BF16, device=DEV) for _ in range(2)]
    stream = stream_of(out[0])
    check(lib.hyc_gemm_segments_tcgen05(2, _ptrs(a), _ptrs(b), kk, T, N, 0, None, ptr(out[0]), ptr(st), stream), "bf16")
    check(lib.hyc_gemm_segments_nf4_tcgen05(2, _ptrs(a), _ptrs(b), (Codes * 2)(), kk, T, N, 0, None, ptr(out[1]), ptr(st), stream), "nf4")
    assert torch.equal(*out)
    xa, bt, sc = [rn(T, 16) for _ in b], [rn(N, 16) for _ in b], [rn(N).abs() + 0.1 for _ in b]
    w = [b[0], rn(N, K)]

    def linears(f, *codes):
        qo, y = [torch.empty(T, N * q // 8, dtype=torch.uint8, device=DEV) for _ in w], [torch.empty(T, N, dtype=BF16, device=DEV) for _ in w]
        check(f(ptr(a[0]), T, K, 2, _ptrs(w), *codes, (ctypes.c_int * 2)(N, N), _ptrs(xa), _ptrs(bt), _ptrs(sc), _ptrs(qo), _ptrs(y), q, ptr(st), stream), "linears")
        return qo + y

    assert all(torch.equal(x, y) for x, y in zip(linears(lib.hyc_linears_lora_save_fwd_tcgen05), linears(lib.hyc_linears_lora_save_fwd_nf4_tcgen05, (Codes * 2)())))
    if T > 128:
        w4 = _weight(g, N, K, 64, False)
        coded = (Codes * 2)(w4[0], Codes())
        assert lib.hyc_gemm_segments_nf4_tcgen05(2, _ptrs(a), _ptrs([None, b[1]]), coded, kk, T, N, 0, None, ptr(out[1]), ptr(st), stream) != 0
    assert int(st.item()) == 0
