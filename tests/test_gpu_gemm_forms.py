"""The forms of the GEMM kernels that depend on the shape: clusters that split K (few rows), pairs and half-width column
tiles, and several weights in one launch, at the edges of their ranges.

Tolerance: fp32 sums of K products carry at most K * 2^-24 * (|A| |B|) of rounding, and every rounding to bf16 adds
2^-8 (half a unit of an 8-bit significand) of the value it rounds."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF16 = torch.bfloat16


def _rn(g, *shape, scale=1.0):
    return (torch.randn(*shape, generator=g) * scale).to(BF16).to(DEV)


@pytest.mark.parametrize("M", [1, 64, 65, 128, 129, 255, 256, 257, 640, 641])
@pytest.mark.parametrize("N,K,K2", [(256, 4096, 0), (256, 1984, 64), (1024, 1024, 1024), (4352, 2048, 64)])
@pytest.mark.parametrize("b_is_kn", [False, True])
def test_gemm_splits_and_tiles(M, N, K, K2, b_is_kn):
    from hyc_lora_release_b200 import mlp
    g = torch.Generator().manual_seed(M + N + K)
    a, a2 = _rn(g, M, K), (_rn(g, M, K2) if K2 else None)
    shape = (lambda k: (k, N)) if b_is_kn else (lambda k: (N, k))
    b, b2 = _rn(g, *shape(K), scale=0.05), (_rn(g, *shape(K2), scale=0.05) if K2 else None)
    res = _rn(g, M, N)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    d = mlp.gemm(a, b, b_is_kn=b_is_kn, a2=a2, b2=b2, residual=res, status=st)
    assert int(st.item()) == 0
    op = (lambda t: t.double()) if b_is_kn else (lambda t: t.double().t())
    main, mag = a.double() @ op(b), a.double().abs() @ op(b).abs()
    if K2:
        main, mag = main + a2.double() @ op(b2), mag + a2.double().abs() @ op(b2).abs()
    want = main + res.double()
    bound = (K + K2) * 2.0 ** -24 * mag + 2.0 ** -8 * (main.abs() + want.abs()) * 1.01
    assert bool(((d.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("T", [1, 100, 128, 200, 300])
@pytest.mark.parametrize("ns", [(512, 256, 256), (256, 256), (768,)])
def test_projections_in_one_launch(T, ns):
    """Outputs and codes of several weights at once against each weight on its own (another split of K may round a
    main branch the other way: its code then moves by one step, counted)."""
    from hyc_lora_release_b200 import mlp
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    g = torch.Generator().manual_seed(T + len(ns))
    K, q = 2048, 4
    x = _rn(g, T, K)
    ws, bs = [_rn(g, n, K, scale=0.03) for n in ns], [_rn(g, n, 16, scale=0.05) for n in ns]
    xas = [_rn(g, T, 16) for _ in ns]
    scs = [torch.full((n,), 0.2 + 0.1 * i, dtype=BF16, device=DEV) for i, n in enumerate(ns)]
    ys = [torch.full((T, n), float("nan"), dtype=BF16, device=DEV) for n in ns]
    qs = [torch.zeros((T, n * q // 8), dtype=torch.uint8, device=DEV) for n in ns]
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    arr = lambda ts: (ctypes.c_void_p * len(ns))(*[t.data_ptr() for t in ts])
    check(lib.hyc_linears_lora_save_fwd_tcgen05(ptr(x), T, K, len(ns), arr(ws), (ctypes.c_int * len(ns))(*ns), arr(xas), arr(bs),
                                                arr(scs), arr(qs), arr(ys), q, ptr(st), stream_of(x)), "linears")
    for w, b, xa, sc, y, codes in zip(ws, bs, xas, scs, ys, qs):
        y1, q1, _ = mlp.linear_lora_save(x, w, None, b, sc, q, xa=xa, status=st)
        assert int(st.item()) == 0
        main, mag = x.double() @ w.double().t(), x.double().abs() @ w.double().abs().t()
        lora = xa.double() @ b.double().t()
        bound = K * 2.0 ** -24 * mag + 2.0 ** -8 * (main.abs() + lora.abs() + (main + lora).abs()) * 1.01 + 1e-6
        assert bool(((y.double() - main - lora).abs() <= bound).all())
        flips = ((codes ^ q1) != 0).double().mean()
        assert float(flips) < 2e-3 and bool(((y.double() - y1.double()).abs() <= 2 * bound).all())


def _lora_b(g, n, transposed):
    """-> (the [n, 16] factor, the tensor that is passed, its column stride, its rank stride)"""
    b = _rn(g, n, 16, scale=0.3)
    if transposed:
        t = b.t().contiguous()
        return b, t, 1, n
    return b, b, 16, 1


@pytest.mark.parametrize("T", [129, 256, 300, 700, 1500])
@pytest.mark.parametrize("I,q,transposed", [(256, 4, False), (1280, 2, True), (2816, 8, False)])
def test_lora_terms_of_the_pair_form(T, I, q, transposed):
    """Gate/up forward and grad_down backward with LoRA terms as large as the main branches (a term in the wrong row or
    column is an error of the order of the result), wide and half-width tiles, a ragged last row block, both layouts of B.
    Forward and backward round to bf16 at most eight times on the way from exact products, each at most 2^-8 of the value:
    2-norm of the difference below 8 * 2^-8 of the result's."""
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    g = torch.Generator().manual_seed(T + I)
    H = 512
    x, wg, wu = _rn(g, T, H), _rn(g, I, H, scale=0.04), _rn(g, I, H, scale=0.04)
    xa1, xa2 = _rn(g, T, 16), _rn(g, T, 16)
    (b1, p1, c1, r1), (b2, p2, c2, r2) = _lora_b(g, I, transposed), _lora_b(g, I, transposed)
    s = torch.full((I,), 0.25 if q > 2 else 1.0, dtype=BF16, device=DEV)
    q1, q2 = (torch.zeros(T, I * q // 8, dtype=torch.uint8, device=DEV) for _ in range(2))
    o, m1, m2, had, gg, gu = (torch.full((T, I), float("nan"), dtype=BF16, device=DEV) for _ in range(6))
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    check(lib.hyc_mlp_gateup_fwd_tcgen05(ptr(x), ptr(wg), ptr(wu), T, H, I, ptr(xa1), ptr(p1), c1, r1, ptr(xa2), ptr(p2), c2, r2, ptr(s), ptr(s),
                                         ptr(q1), ptr(q2), ptr(o), ptr(m1), ptr(m2), q, ptr(st), stream_of(x)), "gateup")
    assert int(st.item()) == 0

    def near(got, want):
        assert float((got.double() - want).norm()) <= 8 * 2.0 ** -8 * float(want.norm())
    l1, l2 = xa1.double() @ b1.double().t(), xa2.double() @ b2.double().t()
    near(m1, x.double() @ wg.double().t())
    near(m2, x.double() @ wu.double().t())
    near(o, torch.nn.functional.silu(m1.double() + l1) * (m2.double() + l2))

    wd, gy = _rn(g, H, I, scale=0.04), _rn(g, T, H)
    from hyc_lora_release_b200.operators import compress_function as cf
    d1, d2 = (cf.decompression_dequantization(c.view(1, T, -1), s.view(1, 1, -1), q).view(T, I).double() for c in (q1, q2))
    check(lib.hyc_mlp_graddown_bwd_tcgen05(ptr(gy), ptr(wd), T, H, I, None, None, 0, ptr(xa1), ptr(p1), c1, r1, ptr(xa2), ptr(p2), c2, r2,
                                           ptr(q1), ptr(s), ptr(q2), ptr(s), None, None, 0, ptr(had), ptr(gg), ptr(gu), q, ptr(st),
                                           stream_of(x)), "graddown")
    assert int(st.item()) == 0
    y1, y2, gd = d1 + l1, d2 + l2, gy.double() @ wd.double()
    sig = torch.sigmoid(y1)
    near(had, y1 * sig * y2)
    near(gu, gd * y1 * sig)
    near(gg, gd * y2 * sig * (1 + y1 * (1 - sig)))


@pytest.mark.parametrize("N,K", [(512, 4096), (1024, 8192), (256, 12288)])
def test_fixed_order_does_not_depend_on_the_rows(N, K):
    """A row's sum is the same bits whatever else is computed with it, on every form that the row count selects."""
    from hyc_lora_release_b200 import mlp
    g = torch.Generator().manual_seed(K)
    a, a2, b, b2, res = _rn(g, 700, K), _rn(g, 700, 64), _rn(g, N, K, scale=0.02), _rn(g, N, 64, scale=0.1), _rn(g, 700, N)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    run = lambda M, **kw: mlp.gemm(a[:M], b, a2=a2[:M], b2=b2, residual=res[:M], status=st, **kw)
    whole = run(700, fixed_order=True)
    for M in (1, 64, 128, 129, 256, 257, 512):
        assert torch.equal(run(M, fixed_order=True), whole[:M]), M
    assert int(st.item()) == 0


def test_o_projection_does_not_depend_on_the_rows():
    """The o projection of the layer at a hidden size whose K is as long as a down projection's: x_medium, which is quantized
    next, is the same bits (the library's LoRA-A product aside: its factor is zero here)."""
    from hyc_lora_release_b200._lib import host
    g = torch.Generator().manual_seed(3)
    H = 8192
    wo, zero, bo = _rn(g, H, H, scale=0.01), torch.zeros(H, 64, dtype=BF16, device=DEV), _rn(g, H, 64)
    x, o = _rn(g, 1, 300, H), _rn(g, 300, H)
    st, sc = torch.zeros(1, dtype=torch.int32, device=DEV), torch.ones(H, dtype=BF16, device=DEV)
    run = lambda M: host.attn_forward_out(x[:, :M], o[:M], wo, zero, bo, sc, None, None, 4, st)[0]
    whole = run(300)
    for M in (64, 128, 200, 256):
        assert torch.equal(run(M), whole[:, :M]), M


@pytest.mark.parametrize("T", [40, 100, 300])
@pytest.mark.parametrize("offset", [1, 2, 4])
def test_lora_factors_at_any_address(T, offset):
    """LoRA-B factors that start at an odd element, or off a 16-byte boundary (slices of a flat buffer): the same bits."""
    from hyc_lora_release_b200 import mlp
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    g = torch.Generator().manual_seed(T)
    H, I, q = 512, 4352, 4
    x, wg, wu, wd, gy = _rn(g, T, H), _rn(g, I, H, scale=0.04), _rn(g, I, H, scale=0.04), _rn(g, H, I, scale=0.04), _rn(g, T, H)
    xa, b, s = _rn(g, T, 16), _rn(g, I, 16, scale=0.3), torch.full((I,), 0.25, dtype=BF16, device=DEV)
    flat = torch.empty(b.numel() + offset, dtype=BF16, device=DEV)[offset:]
    moved = flat.copy_(b.reshape(-1)).view(I, 16)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)

    def run(b):
        q1, q2 = (torch.zeros(T, I * q // 8, dtype=torch.uint8, device=DEV) for _ in range(2))
        o, had, gg, gu = (torch.zeros((T, I), dtype=BF16, device=DEV) for _ in range(4))
        check(lib.hyc_mlp_gateup_fwd_tcgen05(ptr(x), ptr(wg), ptr(wu), T, H, I, ptr(xa), ptr(b), 16, 1, ptr(xa), ptr(b), 16, 1, ptr(s), ptr(s),
                                             ptr(q1), ptr(q2), ptr(o), None, None, q, ptr(st), stream_of(x)), "gateup")
        check(lib.hyc_mlp_graddown_bwd_tcgen05(ptr(gy), ptr(wd), T, H, I, None, None, 0, ptr(xa), ptr(b), 16, 1, ptr(xa), ptr(b), 16, 1,
                                               ptr(q1), ptr(s), ptr(q2), ptr(s), None, None, 0, ptr(had), ptr(gg), ptr(gu), q, ptr(st),
                                               stream_of(x)), "graddown")
        return [o, q1, q2, had, gg, gu, *mlp.linear_lora_save(x, wg, None, b, s, q, xa=xa, status=st)]
    assert all(torch.equal(u, v) for u, v in zip(run(moved), run(b)))
    assert int(st.item()) == 0
