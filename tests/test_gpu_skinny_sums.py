"""Rank-16 products whose partial sums are many results of few partials each (up to sixteen, a block per SM and more: a thread per result),
on both sides of that line, where they are added up the other way; against fp64.  Tolerance: as for the products themselves, K * 2^-24 *
(|A| |B|) and one rounding."""
import pytest
import torch

from test_gpu_skinny import BF16, DEV, Job, _close

pytestmark = pytest.mark.gpu


def _sums(T, ns, n_w, sms):
    """-> (partials of a result at most, blocks of 256 results, workspace bytes) of the regions that the launch picks: of R x C tiles each,
    by their rounds on the SMs."""
    tiles, rows, best = [-(-n // 128) for n in ns], -(-T // 128), None
    for R in range(1, min(rows + 1, 14)):
        for C in range(1, max(tiles) + 1):
            if R + max(n_w) * C <= 14 and R * max(n_w) + C <= 32:
                regions = sum(-(-rows // R) * -(-t // C) for t in tiles)
                cost = -(-regions // sms) * (R * C + 6) * 4096 + regions * (R + C)
                if best is None or cost < best[0]:
                    best = (cost, -(-rows // R), [-(-t // C) for t in tiles])
    _, r, c = best
    return (max([r] + [k for k, w in zip(c, n_w) if w]), len(ns) * -(-max(4 * (w * T + n) for n, w in zip(ns, n_w)) // 256),
            64 * sum(w * k * T + r * n for n, w, k in zip(ns, n_w, c)))


# the form of the MLP backward pass: two results and one of each kind, the last one transposed; 16 and 17 partials; 148 and 147 blocks
@pytest.mark.parametrize("T,ns,n_w,few", [
    (1100, (11008, 11008, 11008), (1, 1, 1), True), (2048, (11008, 264, 8192), (1, 1, 1), False), (4097, (2304, 2304, 2304), (1, 1, 1), True),
    (130, (14336, 14336), (1, 1), False), (2048, (11008, 11008, 11008), (1, 1, 0), True), (389, (14336, 14336), (1, 1), True),
    (384, (4352, 4352), (1, 1), False), (5376, (4096,), (1,), True), (5253, (4096,), (1,), False)])
def test_sums(T, ns, n_w, few):
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    g = torch.Generator(device=DEV).manual_seed(T)
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV).to(BF16)
    jobs, keep, turned = (Job * len(ns))(), [], 2 if 0 in n_w else 1
    for i, n in enumerate(ns):
        x, w, xa, y = rn(T, n), rn(n, 16), rn(T, 16), torch.full((T, 64), float("nan"), dtype=BF16, device=DEV)
        z = torch.full((16, n) if i == turned else (n, 16), float("nan"), dtype=BF16, device=DEV)
        j = jobs[i]
        j.x, j.ldx, j.n, j.n_w, j.ld_w, j.ld_y, j.y_pad = x.data_ptr(), n, n, n_w[i], 16, 64, 48
        j.xa, j.ld_xa, j.z, j.z_transposed = xa.data_ptr(), 16, z.data_ptr(), int(i == turned)
        if n_w[i]:
            j.w[0], j.y[0] = w.data_ptr(), y.data_ptr()
        keep.append((x, w, xa, y, z))
    nbytes, sms = lib.hyc_skinny_workspace_bytes(len(ns), jobs, T), torch.cuda.get_device_properties(0).multi_processor_count
    parts, blocks, planned = _sums(T, ns, n_w, sms)
    assert nbytes == planned and (sms != 148 or (parts <= 16 and blocks >= sms) == few)
    work, st = torch.full((nbytes // 4,), float("nan"), device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    check(lib.hyc_skinny_products(len(ns), jobs, T, ptr(work), nbytes, ptr(st), stream_of(work)), "skinny")
    assert int(st.item()) == 0
    for i, (x, w, xa, y, z) in enumerate(keep):
        if n_w[i]:
            assert _close(y[:, :16], x, w) and bool((y[:, 16:] == 0).all())
        assert _close(z.t() if i == turned else z, x.t(), xa)
