"""Results that share an allocation: each is a contiguous tensor of its own on a 256-byte boundary, none reaches into another, and what is
written through one is seen by no other."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16 = "cuda", torch.bfloat16


def _apart(ts):
    spans = sorted((t.data_ptr(), t.data_ptr() + t.numel() * t.element_size()) for t in ts if t.numel())
    assert all(t.is_contiguous() and t.data_ptr() % 256 == 0 for t in ts if t.numel())
    assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
    copies = [t.clone() for t in ts]
    for i, t in enumerate(ts):
        t.view(-1).view(torch.uint8).fill_(0x55)
        assert all(torch.equal(x.view(torch.uint8), c.view(torch.uint8)) for j, (x, c) in enumerate(zip(ts, copies)) if j > i)


@pytest.mark.parametrize("rows,S,ratio,q", [(1, 64, 0.0, 2), (3, 320, 0.02, 4), (257, 512, 0.05, 8)])
def test_topk(rows, S, ratio, q):
    from hyc_lora_release_b200.operators import compress_function as cf
    a = torch.softmax(torch.randn(1, 1, rows, S, device=DEV), -1).to(BF16)
    m = cf.compression_softmax_topk(a, ratio, q)
    assert m.q.shape == (rows, S * q // 8) and m.val.shape == (rows, int(S * ratio)) and m.q.dtype == torch.uint8 and m.val.dtype == BF16
    _apart(list(m.tensors()))


@pytest.mark.parametrize("T,N,k,q", [(1, 32, 0, 2), (37, 4096, 20, 8), (130, 96, 3, 4)])
def test_norm(T, N, k, q):
    from hyc_lora_release_b200._lib import host
    x, w, s = torch.randn(1, T, N, device=DEV).to(BF16), torch.ones(N, dtype=BF16, device=DEV), torch.full((1, N), 0.3, dtype=BF16, device=DEV)
    idx = torch.arange(k, device=DEV)
    y, rstd, xo, xq, xnq = host.rmsnorm_save(x, w, 1e-5, q, s, idx, s)
    assert rstd.shape == (T,) and rstd.dtype == torch.float32 and xo.shape == (1, T, k) and xq.shape == xnq.shape == (1, T, N * q // 8)
    assert host.rmsnorm_save(x, w, 1e-5, q, s, idx, None)[4] is None
    _apart([y, rstd, xo, xq, xnq])
