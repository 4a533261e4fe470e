"""Rank-16 products whose partial sums are many results of few partials each (a block per SM and more), next to the same X in fewer rows,
where they are added up the other way; against fp64.  Tolerance: as for the products themselves, K * 2^-24 * (|A| |B|) and one rounding."""
import pytest
import torch

from test_gpu_skinny import BF16, DEV, Job, _close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,ns", [(1100, (11008, 11008, 11008)), (2048, (11008, 264, 8192)), (4097, (2304, 2304, 2304)), (130, (14336, 14336))])
def test_sums(T, ns):
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    g = torch.Generator(device=DEV).manual_seed(T)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV).to(BF16)
    jobs, keep = (Job * len(ns))(), []
    for i, n in enumerate(ns):
        x, w, xa, y = rn(T, n), rn(n, 16), rn(T, 16), torch.full((T, 64), float("nan"), dtype=BF16, device=DEV)
        z = torch.full((16, n) if i == 1 else (n, 16), float("nan"), dtype=BF16, device=DEV)
        j = jobs[i]
        j.x, j.ldx, j.n, j.n_w, j.ld_w, j.ld_y, j.y_pad = x.data_ptr(), n, n, 1, 16, 64, 48
        j.w[0], j.y[0], j.xa, j.ld_xa, j.z, j.z_transposed = w.data_ptr(), y.data_ptr(), xa.data_ptr(), 16, z.data_ptr(), int(i == 1)
        keep.append((x, w, xa, y, z))
    nbytes = lib.hyc_skinny_workspace_bytes(len(ns), jobs, T)
    work, st = torch.full((nbytes // 4,), float("nan"), device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    check(lib.hyc_skinny_products(len(ns), jobs, T, ptr(work), nbytes, ptr(st), stream_of(work)), "skinny")
    assert int(st.item()) == 0
    for i, (x, w, xa, y, z) in enumerate(keep):
        assert _close(y[:, :16], x, w) and bool((y[:, 16:] == 0).all())
        assert _close(z.t() if i == 1 else z, x.t(), xa)
