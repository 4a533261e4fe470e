"""Rank-16 products with a large operand (both directions from one read) at the edges of the 128 x 128 tiles and of the
regions a block takes, against fp64.

Tolerance: fp32 sums of K products carry at most K * 2^-24 * (|A| |B|), the rounding to bf16 2^-8 of the value."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BF16 = torch.bfloat16


class Job(ctypes.Structure):
    _fields_ = [("x", ctypes.c_void_p), ("ldx", ctypes.c_int64), ("w", ctypes.c_void_p * 3), ("ld_w", ctypes.c_int64),
                ("y", ctypes.c_void_p * 3), ("ld_y", ctypes.c_int64), ("xa", ctypes.c_void_p), ("ld_xa", ctypes.c_int64),
                ("z", ctypes.c_void_p), ("n", ctypes.c_int), ("n_w", ctypes.c_int), ("y_pad", ctypes.c_int), ("z_transposed", ctypes.c_int)]


def _close(got, a, b):
    want, mag = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    bound = a.shape[1] * 2.0 ** -24 * mag + 2.0 ** -8 * want.abs() * 1.01 + 1e-30
    return bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("T", [1, 63, 64, 65, 200, 1024, 4097])
@pytest.mark.parametrize("ns", [(8,), (256, 264), (512, 128, 1000), (4352,)])
@pytest.mark.parametrize("n_w,with_z", [(0, True), (1, True), (1, False), (3, False), (2, True)])
def test_products(T, ns, n_w, with_z):
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    g = torch.Generator().manual_seed(T + sum(ns))
    rn = lambda *s: torch.randn(*s, generator=g).to(BF16).to(DEV)
    jobs, keep = (Job * len(ns))(), []
    for i, n in enumerate(ns):
        x = rn(T, n + 8)[:, :n]                                   # a row stride of its own
        ws = [rn(n, 16) for _ in range(n_w)]
        y = torch.full((T, 64), float("nan"), dtype=BF16, device=DEV)
        xa, tr = rn(T, 64), i % 2
        z = torch.full((16, n) if tr else (n, 16), float("nan"), dtype=BF16, device=DEV) if with_z else None
        j = jobs[i]
        j.x, j.ldx, j.n, j.n_w, j.ld_w, j.ld_y, j.y_pad = x.data_ptr(), n + 8, n, n_w, 16, 64, 64 - 16 * n_w if n_w else 0
        for k, w in enumerate(ws):
            j.w[k], j.y[k] = w.data_ptr(), y.data_ptr() + 32 * k
        if with_z:
            j.xa, j.ld_xa, j.z, j.z_transposed = xa.data_ptr(), 64, z.data_ptr(), tr
        keep.append((x, ws, y, xa, z, tr))
    nbytes = lib.hyc_skinny_workspace_bytes(len(ns), jobs, T)
    work = torch.empty(nbytes // 4, dtype=torch.float32, device=DEV)
    st = torch.zeros(1, dtype=torch.int32, device=DEV)
    check(lib.hyc_skinny_products(len(ns), jobs, T, ptr(work), nbytes, ptr(st), stream_of(work)), "skinny")
    assert int(st.item()) == 0
    for x, ws, y, xa, z, tr in keep:
        for k, w in enumerate(ws):
            assert _close(y[:, 16 * k:16 * k + 16], x, w)
        if ws:
            assert bool((y[:, 16 * len(ws):] == 0).all())
        if z is not None:
            assert _close(z.t() if tr else z, x.t(), xa[:, :16])
    assert lib.hyc_skinny_products(len(ns), jobs, T, ptr(work), nbytes - 4, ptr(st), stream_of(work)) == -5
