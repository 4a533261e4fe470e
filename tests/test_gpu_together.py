"""Results that one call makes several of: each is a contiguous tensor on a 256-byte boundary, none reaches into another, and what is written
through one is seen by no other.  What a caller gets hold of has a storage of its own: keeping one result keeps no other."""
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


def _alone(ts):
    assert all(t.untyped_storage().nbytes() == t.numel() * t.element_size() for t in ts)


def test_operators_own_what_they_return():
    from hyc_lora_release_b200.operators import compress_function as cf
    from hyc_lora_release_b200.operators.rmsnorm_kernels import rmsnorm_forward_save
    a = torch.softmax(torch.randn(1, 2, 64, 128, device=DEV) * 4, -1).to(BF16)
    _alone(cf.compression_softmax_topk(a, 0.05, 4).tensors())
    m = cf.compression_softmax_static(a, 0.05, capacity=a.numel())
    _alone([m.words, m.directory, m.nnz])
    dense, nnz = m.to_dense(), m.nnz
    del m                                        # the count stays, the words go
    assert int(nnz.item()) == int((dense != 0).sum())
    x, s = torch.randn(1, 5, 64, device=DEV).to(BF16), torch.full((64,), 0.3, dtype=BF16, device=DEV)
    _alone(rmsnorm_forward_save(x, torch.ones(64, dtype=BF16, device=DEV), 1e-5, 4, s, torch.arange(3, device=DEV), s))


def test_halves_own_what_they_return():
    """The records of the two halves and the gradients of the attention half, through the calls that hand them out."""
    from hyc_lora_release_b200.attention import AttnState, attention_backward, attention_forward
    from hyc_lora_release_b200.mlp import MLPState, MLPWeights, mlp_forward
    from test_gpu_layer import _attn_weights, layer_problem
    g = torch.Generator().manual_seed(5)
    B, M, heads, d, kv, I = 1, 128, 4, 128, 2, 512
    x, p, cos, sin, mask = layer_problem(g, B, M, heads * d, heads, d, kv, I)
    x, cos, sin, mask = (t.to(DEV) for t in (x, cos, sin, mask))
    t = lambda n: p[n].t().contiguous().to(DEV)
    aw = _attn_weights(p)
    mw = MLPWeights(norm_w=p["norm_w2"].to(DEV), wg=t("wgate"), wu=t("wup"), wd=t("wdown"), ag=t("agate"), bg=t("bgate"), au=t("aup"), bu=t("bup"),
                    ad=t("adown"), bd=t("bdown"))
    sa, sm = AttnState(iteration_threshold=1), MLPState(iteration_threshold=1)
    for _ in range(2):                           # the second is a steady one
        y, fa = attention_forward(x, aw, sa, cos, sin, mask, heads, d, kv)
        _, fm = mlp_forward(y, mw, sm)
    _alone([fa[n] for n in ("rstd", "x_o", "x_q", "xn_q", "q_q", "k_q", "v_q")] + [fm[n] for n in ("rstd", "xm_o", "xm_q", "xn_q", "gate_q", "up_q")])
    ga = attention_backward(torch.randn_like(y), fa, aw)
    _alone([ga[n] for n in ("grad_q", "grad_k", "grad_v")])
