"""Backward of the attention kernels with more items than blocks: what a block works on one after the other is what blocks of their own
make of it.  The sums of an item do not depend on the others, so the results are the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV, BF16 = "cuda", torch.bfloat16


@pytest.mark.parametrize("B,M,h,kv", [(5, 264, 40, 40), (7, 384, 32, 16), (3, 128, 148, 148), (2, 200, 40, 40), (2, 128, 149, 149)])
@pytest.mark.parametrize("form", ["none", "causal", "dead keys"])
def test_items(B, M, h, kv, form):
    from hyc_lora_release_b200._lib import check, lib, ptr, stream_of
    g, d = torch.Generator(device=DEV).manual_seed(B + M), 128
    rn = lambda *s: torch.randn(*s, generator=g, device=DEV).to(BF16)
    q, k, v, go = rn(B, M, h * d), rn(B, M, kv * d), rn(B, M, kv * d), rn(B, M, h * d)
    i = torch.arange(M, device=DEV)
    keep = torch.ones(M, M, dtype=torch.bool, device=DEV) if form == "none" else (i[:, None] >= i[None] if form == "causal" else (i < 128)[None].expand(M, M))
    p = (torch.softmax(rn(B, h, M, M).float(), -1) * keep).to(BF16)
    st, cls = torch.zeros(1, dtype=torch.int32, device=DEV), None
    if form != "none":
        mask = torch.zeros(1, 1, M, M, dtype=BF16, device=DEV).masked_fill(~keep, torch.finfo(BF16).min)
        cls = torch.empty(lib.hyc_attn_mask_class_bytes(1, 1, M), dtype=torch.uint8, device=DEV)
        check(lib.hyc_attn_mask_class(ptr(mask), 0, 0, M, 1, 1, M, ptr(cls), stream_of(q)), "cls")

    def backward(q, k, v, go, p):
        out, gs = [torch.full_like(x, float("nan")) for x in (q, k, v)], torch.empty_like(p)
        check(lib.hyc_attn_bwd_tcgen05(ptr(q), ptr(k), ptr(v), ptr(go), ptr(p), ptr(gs), q.shape[0], M, h, kv, d, d ** -0.5, ptr(cls), 0, 0, *[ptr(x) for x in out],
                                       ptr(st), stream_of(q)), "bwd")
        return out

    whole = backward(q, k, v, go, p)
    assert int(st.item()) == 0
    for b in range(B):
        for x, y in zip(whole, backward(q[b:b + 1], k[b:b + 1], v[b:b + 1], go[b:b + 1], p[b:b + 1])):
            assert bool(torch.isfinite(y).all()) and torch.equal(x[b:b + 1], y)
    assert int(st.item()) == 0
