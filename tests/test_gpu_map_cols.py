"""Probability maps whose rows end early: the save and restore kernels that do not touch what lies behind the rows' ends,
against the whole-row kernels on the same map with zeros there."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _map(maps, M, kind, seed):
    """-> (map with NaN behind the rows' ends, the same with zeros there, row_cols)"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    unit = 128 if M > 64 else 64
    r = torch.arange(M, device="cuda")
    if kind == "causal":
        cols = ((r // unit + 1) * unit).clamp(max=M).repeat(maps)
    elif kind == "whole":
        cols = torch.full((maps * M,), M, device="cuda")
    else:      # any multiple of 64 (M itself among them), none as well
        cols = (torch.randint(0, M // 64 + 2, (maps * M,), generator=g, device="cuda") * 64).clamp(max=M)
        if kind != "any":
            cols[0] = M if kind == "any, the first whole" else 0
    a = torch.softmax(3 * torch.randn(maps * M, M, generator=g, device="cuda"), -1).to(torch.bfloat16)
    behind = torch.arange(M, device="cuda")[None] >= cols[:, None]
    return a.masked_fill(behind, float("nan")), a.masked_fill(behind, 0.0), cols.to(torch.int16), behind


def _call(name, *args):
    from hyc_lora_release_b200._lib import lib, check, stream_of
    args = [ctypes.c_void_p(x.data_ptr()) if isinstance(x, torch.Tensor) else x for x in args]
    check(getattr(lib, name)(*args, stream_of(torch.empty(0, device="cuda"))), name)


def _topk_buffers(rows, M, k, q):
    e = lambda *s, dt: torch.empty(*s, dtype=dt, device="cuda")
    return [e(rows, k, dt=torch.bfloat16), e(rows, k, dt=torch.int16), e(rows, M * q // 8, dt=torch.uint8), e(rows, M // 64, dt=torch.bfloat16),
            e(rows, M // 64, dt=torch.int8)]


@pytest.mark.parametrize("kind", ["causal", "whole", "any, the first empty", "any, the first whole"])      # (the first row decides on the order)
@pytest.mark.parametrize("M,k,q", [(64, 3, 4), (128, 6, 2), (192, 9, 4), (192, 10, 8), (448, 22, 4), (704, 35, 4), (704, 0, 2), (1024, 51, 4),
                                   (1984, 99, 2), (2048, 102, 4), (2048, 128, 8)])
def test_topk_rows_that_end_early(M, k, q, kind):
    from hyc_lora_release_b200._lib import lib
    assert lib.hyc_softmax_topk_cols_supported(M, k) == 1
    maps = 3
    a, dense, cols, behind = _map(maps, M, kind, M + k)
    rows = maps * M
    whole, early = _topk_buffers(rows, M, k, q), _topk_buffers(rows, M, k, q)
    _call("hyc_softmax_topk_compress", dense, rows, M, k, *whole, q)
    _call("hyc_softmax_topk_compress_cols", a, rows, M, cols, k, *early, q)
    for w, e in zip(whole, early):
        assert torch.equal(w.view(torch.uint8), e.view(torch.uint8))
    val, col, codes, scale, zp = whole
    full = torch.empty(rows, M, dtype=torch.bfloat16, device="cuda")
    _call("hyc_softmax_topk_restore", val, col, k, codes, scale, zp, rows, M, full, q)
    out = torch.full_like(full, -7.0)
    _call("hyc_softmax_topk_restore_cols", val, col, k, codes, scale, zp, rows, M, cols, out, q)
    assert torch.equal(out, full.masked_fill(behind, -7.0))


@pytest.mark.parametrize("beyond", [64, 320, 65535 - 704])
@pytest.mark.parametrize("M,q", [(192, 2), (704, 4), (1984, 8), (512, 4)])
@pytest.mark.parametrize("kind", ["any, the first empty", "any, the first whole"])
def test_row_ends_beyond_the_row_are_its_end(M, q, beyond, kind):
    """A reported end above M counts as M: no group behind the row is read or written, in the middle of the buffers or after them."""
    maps, k = 2, 5
    rows = maps * M
    a, dense, cols, behind = _map(maps, M, kind, M)
    too_far = torch.where(cols.int() == M, torch.minimum(cols.int() + beyond, torch.full_like(cols.int(), 65535)), cols.int()).to(torch.uint16)
    assert bool((cols == M).any())
    fill = lambda bufs: [t.view(torch.uint8).fill_(0xa5).view(t.dtype) for t in bufs]
    exact, far = fill(_topk_buffers(rows, M, k, q)), fill(_topk_buffers(rows + 64, M, k, q))
    _call("hyc_softmax_topk_compress_cols", a, rows, M, cols, k, *exact, q)
    _call("hyc_softmax_topk_compress_cols", a, rows, M, too_far, k, *far, q)
    for e, f in zip(exact, far):
        e, f = e.flatten().view(torch.uint8), f.flatten().view(torch.uint8)
        assert torch.equal(e, f[:e.numel()]) and bool((f[e.numel():] == 0xa5).all())
    out = [torch.full((rows + 8, M), -7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    for o, c in zip(out, (cols, too_far)):
        val, col, codes, scale, zp = exact
        _call("hyc_softmax_topk_restore_cols", val, col, k, codes, scale, zp, rows, M, c, o, q)
    assert torch.equal(*out) and bool((out[1][rows:] == -7.0).all())


def test_topk_lists_that_do_not_fit_are_refused():
    from hyc_lora_release_b200._lib import lib
    assert lib.hyc_softmax_topk_cols_supported(2048, 129) == 0      # two lists of a warp need 258 staged entries
    assert lib.hyc_softmax_topk_cols_supported(4096, 10) == 0 and lib.hyc_softmax_topk_cols_supported(96, 4) == 0


@pytest.mark.parametrize("kind", ["causal", "whole", "any"])
@pytest.mark.parametrize("M,maps,thr", [(256, 3, 0.01), (768, 2, 0.004), (1024, 2, 0.003), (2048, 1, 0.002), (4096, 1, 0.001), (256, 2, -1.0)])
def test_pruned_rows_that_end_early(M, maps, thr, kind):
    g = torch.Generator(device="cuda").manual_seed(M)
    numel = maps * M * M
    r = torch.arange(M, device="cuda")
    if kind == "causal":
        cols = ((r // 128 + 1) * 128).clamp(max=M).repeat(maps)
    elif kind == "whole":
        cols = torch.full((maps * M,), M, device="cuda")
    else:
        cols = torch.randint(0, M // 8 + 1, (maps * M,), generator=g, device="cuda") * 8
    a = torch.softmax(3 * torch.randn(maps * M, M, generator=g, device="cuda"), -1).to(torch.bfloat16)
    behind = torch.arange(M, device="cuda")[None] >= cols[:, None]
    dense = a.masked_fill(behind, 0.0)
    a = a.masked_fill(behind, float("inf"))
    cols = cols.to(torch.int16)
    from hyc_lora_release_b200._lib import lib
    words = torch.empty(2 * numel, dtype=torch.int32, device="cuda")
    directory = torch.empty(lib.hyc_softmax_prune_tiled_directory_bytes(numel) // 4, dtype=torch.int32, device="cuda")
    nnz = torch.empty(1, dtype=torch.int64, device="cuda")
    _call("hyc_softmax_prune_tiled_cols", a, numel, M, cols, thr, words, words.numel(), directory, nnz)
    want = torch.where((dense > torch.tensor(thr, dtype=torch.bfloat16)) & (dense != 0), dense, torch.zeros_like(dense))
    assert int(nnz) == int((want != 0).sum())
    out = torch.full_like(dense, -7.0)
    _call("hyc_softmax_prune_tiled_restore_cols", words, words.numel(), directory, M, cols, out, numel)
    assert torch.equal(out, want.masked_fill(behind, -7.0))
    _call("hyc_softmax_prune_tiled_restore", words, words.numel(), directory, out, numel)
    assert torch.equal(out, want)
    assert lib.hyc_softmax_prune_tiled_restore_cols(None, 0, ctypes.c_void_p(directory.data_ptr()), M - 8, ctypes.c_void_p(cols.data_ptr()),
                                                    ctypes.c_void_p(out.data_ptr()), numel, None) == -3


@pytest.mark.parametrize("thr", [0.25, -1.0])
@pytest.mark.parametrize("numel", [8, 1024, 4096 + 8, 3 * 4096 + 1000])
def test_ordered_list_at_any_density(numel, thr):
    """The ordered fill packs four trips of a warp at once: none, one entry per lane, whole lanes, everything, and ends."""
    from hyc_lora_release_b200._lib import lib
    i = torch.arange(numel, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(numel)
    for keep in (i < 0, i % 8 == 7, i // 8 % 32 == 5, i >= 0, i // 256 % 4 == 2, torch.rand(numel, generator=g, device="cuda") < 0.3):
        # (what is dropped is a zero or, where the threshold allows it, below it)
        a = torch.where(keep, 0.5 + (i % 61).float() / 128, torch.where(i % 2 == 0, 0.0, -2.0)).to(torch.bfloat16)
        ws = torch.empty(lib.hyc_softmax_prune_workspace_bytes(numel) // 8 + 1, dtype=torch.int64, device="cuda")
        _call("hyc_softmax_prune_count", a, numel, thr, ws, ws.numel() * 8)
        n = int(ws[0])
        idx, val = torch.empty(max(n, 1), dtype=torch.int64, device="cuda"), torch.empty(max(n, 1), dtype=torch.bfloat16, device="cuda")
        _call("hyc_softmax_prune_fill", a, numel, thr, ws, idx, val, n)
        want = keep.nonzero().flatten()
        assert n == want.numel() and torch.equal(idx[:n], want) and torch.equal(val[:n], a[want])
