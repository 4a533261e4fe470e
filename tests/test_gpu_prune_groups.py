"""The ordered prune at the edges of the tiles of 4096 elements, of the groups of eight that a block counts, and of the 2048 groups that the
scan takes at a time.  Indices and values are copies: exact."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16, TILE = "cuda", torch.bfloat16, 4096


@pytest.mark.parametrize("numel", [1, TILE, 8 * TILE - 1, 8 * TILE, 8 * TILE + 1, 17 * TILE + 5, 1024 * 8 * TILE + 3, 2048 * 8 * TILE + 8 * TILE + 1])
@pytest.mark.parametrize("thr", [0.99, -0.5])
def test_prune(numel, thr):
    from hyc_lora_release_b200._lib import host
    g = torch.Generator(device=DEV).manual_seed(numel)
    a = torch.randn(numel, generator=g, device=DEV).to(BF16)
    a[::3] = 0
    want = torch.nonzero((a > torch.tensor(thr, dtype=BF16, device=DEV)) & (a != 0)).flatten()
    for thr_dev in (None, torch.tensor([thr], device=DEV)):
        m = host.prune_sparse(a, thr, thr_dev)
        assert torch.equal(m.indices()[0], want) and torch.equal(m.values(), a[want])
