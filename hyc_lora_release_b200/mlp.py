"""MLP half of the HyC-LoRA fused decoder layer on the tcgen05 kernels.

Mirrors the MLP part of ``FusedLlamaLayerIntraInterFullFuseFunc.forward/backward``
(models/llama/fused_llama_layer_intra_inter_full_fuse.py:203-252 and :359-396; the Mistral
twin is identical for this part) with plain bf16 frozen weights:

  forward : RMSNorm -> save x (outlier channels + per-channel codes) -> gate/up GEMMs with the
            quantizer, LoRA add, SiLU and Hadamard in the GEMM epilogue -> save x_norm codes ->
            down GEMM with LoRA add and residual in the epilogue;
  backward: grad_down GEMM with the de-quantize / recompute / SiLU-Hadamard backward in the
            epilogue -> LoRA gradients -> grad_x GEMM (gate and up accumulated in one tile) ->
            RMSNorm backward on the restored x.

Only packed codes, scales, the outlier slab, the rank-16 LoRA activations and rstd are kept
between the two passes.  Weights use the nn.Linear layout ([out, in]); the LoRA factors are
``lora_A.weight`` [r, in] and ``lora_B.weight`` [out, r].
"""
from dataclasses import dataclass, field
from typing import Optional

import torch

from ._lib import HycError, check, host, lib, ptr, require_cuda, stream_of
from .operators import compress_function as cf
from .operators.rmsnorm_kernels import rmsnorm_forward

BF16 = torch.bfloat16
_KERNEL_STATUS = {1: "TMA producer wait timed out", 2: "MMA issuer wait timed out", 3: "epilogue wait timed out"}


def _status_tensor(device):
    return torch.zeros(1, dtype=torch.int32, device=device)


def check_status(status, what):
    """Raise if a bounded wait inside a tcgen05 kernel gave up (synchronises)."""
    v = int(status.item())
    if v != 0:
        raise HycError("%s: %s" % (what, _KERNEL_STATUS.get(v, "status %d" % v)))


def _lora(xa, bt, ld_col, ld_r):
    if xa is None:
        return [None, None, 0, 0]
    return [ptr(xa), ptr(bt), ld_col, ld_r]


def gemm(a, b, *, b_is_kn=False, a2=None, b2=None, a3=None, b3=None, lora0=None, lora1=None, residual=None,
         status=None, fixed_order=False):
    """D = a @ op(b) (+ a2 @ op(b2)) (+ a3 @ op(b3)) (+ LoRA terms) (+ residual) on the tcgen05 kernel.

    a [M,K] bf16; b [N,K] (b_is_kn=False) or [K,N] (b_is_kn=True), both row-major.
    fixed_order: the order of summation does not depend on M (for results that are quantized, or feed what is).
    lora = (xa [M,16], bt, ld_col, ld_r): adds xa @ Bt^T with Bt(col, r) = bt[col*ld_col + r*ld_r]."""
    require_cuda(a, b)
    M, K = a.shape
    N = b.shape[1] if b_is_kn else b.shape[0]
    K2 = 0 if a2 is None else a2.shape[1]
    K3 = 0 if a3 is None else a3.shape[1]
    d = torch.empty((M, N), dtype=BF16, device=a.device)
    st = status if status is not None else _status_tensor(a.device)
    l0 = _lora(*lora0) if lora0 else [None, None, 0, 0]
    l1 = _lora(*lora1) if lora1 else [None, None, 0, 0]
    check(lib.hyc_gemm_bf16_tcgen05(ptr(a), ptr(b), M, N, K, (1 if b_is_kn else 0) | (2 if fixed_order else 0), ptr(a2), ptr(b2), K2,
                                    ptr(a3), ptr(b3), K3, *l0, *l1, ptr(residual), ptr(d), ptr(st), stream_of(a)),
          "hyc_gemm_bf16_tcgen05")
    return d


def lora_a_products(x2, stacked):
    """x2 [T, K] times several LoRA-A factors at once: ``stacked`` [n, K, r] holds their transposes; one batched library
    call whose left operand is the same x2 for every batch (stride 0), -> [n, T, r], each [T, r] contiguous.  Measured
    on a B200, x2 [2048, 4096]: 9.5 us for three factors against 20.5 us as three products."""
    return torch.bmm(x2.unsqueeze(0).expand(stacked.shape[0], -1, -1), stacked)


def linear_lora_save(x, w, a, b, scale, q_bit, *, want_main=False, status=None, xa=None):
    """A LoRA projection with the save of its main branch in the GEMM epilogue (steady state of the q/k/v/o
    projections): x [T,K], w [N,K], a = lora_A.weight [r,K], b = lora_B.weight [N,r], scale [N] ->
    (y [T,N], q_main [T, N*q_bit/8], xa [T,r][, main])."""
    require_cuda(x, w, a, b, scale)
    T, K = x.shape
    N = w.shape[0]
    if xa is None:
        xa = (x @ a.t()).contiguous()
    dev = x.device
    y = torch.empty((T, N), dtype=BF16, device=dev)
    qm = torch.empty((T, N * q_bit // 8), dtype=torch.uint8, device=dev)
    main = torch.empty((T, N), dtype=BF16, device=dev) if want_main else None
    st = status if status is not None else _status_tensor(dev)
    sc = scale.to(BF16).reshape(-1).contiguous()
    check(lib.hyc_linear_lora_save_fwd_tcgen05(ptr(x), ptr(w), T, K, N, ptr(xa), ptr(b.contiguous()), b.shape[1], 1,
                                               ptr(sc), ptr(qm), ptr(y), ptr(main), q_bit, ptr(st), stream_of(x)),
          "hyc_linear_lora_save_fwd_tcgen05")
    return (y, qm, xa, main) if want_main else (y, qm, xa)


def lora_grad_a(q, scale, gm, r2, q_bit):
    """out [r2, H] = gm[:, :r2]^T @ dequant(q, scale), the packed activation de-quantized inside the kernel.
    q [T, H*q_bit/8] uint8, scale [H] bf16, gm [T, >= r2] bf16 (row stride a multiple of 8)."""
    return host.lora_grad_a(q, scale, gm, r2, q_bit)


def contents_key(tensors):
    """Equal keys: the tensors hold what they held, as long as an alias of each is kept beside the key (``_pad_of`` of the
    weight records; without it another tensor's storage may come to lie at the old address), and what was made of them
    was made in the same stream capture (a replay makes again only what was recorded) or outside of one."""
    return (host.capture_of(tensors[0]), *((t.data_ptr(), t._version, t.shape, t.stride(), t.dtype) for t in tensors))


@dataclass
class MLPWeights:
    """Frozen bf16 weights ([out, in]) and LoRA factors of one MLP."""
    norm_w: torch.Tensor   # [H]
    wg: torch.Tensor       # [I, H]
    wu: torch.Tensor       # [I, H]
    wd: torch.Tensor       # [H, I]
    ag: torch.Tensor       # gate lora_A.weight [r, H]
    bg: torch.Tensor       # gate lora_B.weight [I, r]
    au: torch.Tensor
    bu: torch.Tensor
    ad: torch.Tensor       # down lora_A.weight [r, I]
    bd: torch.Tensor       # down lora_B.weight [H, r]
    bias_d: Optional[torch.Tensor] = None    # bias of the down projection ([H] bf16) or None; no gradient

    @torch.no_grad()      # as part of a graph they would keep the adapters' AccumulateGrad nodes, and with them the stream of
    def padded(self):     # the step that made them, alive: a later step could not be captured on another stream
        """LoRA factors zero-padded to a K of 64 so that a rank-16 product can ride along a GEMM as one more
        K block (built once per optimizer step; a few hundred KB):
          ad_rows  [64, I]  rows 0..15 = Ad            (second operand of grad_down's LoRA part, [K, N])
          ad_cols  [I, 64]  columns 0..15 = Ad^T       (projects hadamard to the padded down LoRA activation)
          bd_cols  [H, 64]  columns 0..15 = Bd         (second operand of the down projection's LoRA part, [N, K])
          agu_rows [64, H]  rows 0..15 = Ag, 16..31 = Au (second operand of grad_x's LoRA part, [K, N])
        and the transposed factors of the rank-16 products:
          agu_t    [2, H, r]  Ag^T, Au^T  (x_norm @ both in one call)"""
        ts = (self.ag, self.au, self.ad, self.bd, self.bg, self.bu)
        key = contents_key(ts)
        if getattr(self, "_pad_key", None) != key:
            r, I = self.ad.shape
            H = self.bd.shape[0]
            dev, dt = self.ad.device, self.ad.dtype
            ad_rows = torch.zeros(64, I, dtype=dt, device=dev); ad_rows[:r] = self.ad
            bd_cols = torch.zeros(H, 64, dtype=dt, device=dev); bd_cols[:, :r] = self.bd
            agu_rows = torch.zeros(64, H, dtype=dt, device=dev); agu_rows[:r] = self.ag; agu_rows[r:2 * r] = self.au
            agu_t = torch.stack((self.ag.t(), self.au.t())).contiguous()      # [2, H, r]
            self._pad = dict(ad_rows=ad_rows, ad_cols=ad_rows.t().contiguous(), bd_cols=bd_cols, agu_rows=agu_rows,
                             agu_t=agu_t)
            self._pad_key, self._pad_of = key, [t.detach() for t in ts]
        return self._pad


@dataclass
class MLPState:
    """Calibration state of the MLP part of a layer (the reference keeps the same entries in
    ``static_value``, fused_llama_layer_intra_inter_full_fuse.py:557-570)."""
    iteration: int = 0
    iteration_threshold: int = 5
    q_bit: int = 4
    layernorm_outlier_ratio: float = 0.005
    static_value: dict = field(default_factory=lambda: {
        'x_medium': {'outlier_channel_index': None, 'scale': None},
        'x_norm_2': {'scale': None}, 'gate': {'scale': None}, 'up': {'scale': None}})


def mlp_forward(x_medium, w: MLPWeights, state: MLPState, eps=1e-5, status=None):
    """-> (x_out [B,M,H], saved tuple).  Advances the calibration state like the layer does."""
    require_cuda(x_medium)
    B, M, H = x_medium.shape
    st = status if status is not None else _status_tensor(x_medium.device)
    q, sv = state.q_bit, state.static_value
    if state.iteration < state.iteration_threshold:
        x_out, saved = _mlp_forward_calibrating(x_medium, w, state, eps, st)
    else:
        # steady state: the norm, the save of its input (codes + outlier channels) and the save of its output are one
        # pass over x_medium, then gate/up and down; one call into the native host path for the whole sequence
        pad = w.padded()
        xm, xn_scale = sv['x_medium'], sv['x_norm_2']['scale']
        x_out, rstd, xm_o, xm_q, xn_q, q1, q2, gs, us, gu_xa, down_xa64 = host.mlp_forward(
            x_medium, [w.norm_w, w.wg, w.wu, w.wd, w.bg, w.bu, pad["agu_t"], pad["ad_cols"], pad["bd_cols"]],
            [xm['outlier_channel_index'], xm['scale'], xn_scale, sv['gate']['scale'], sv['up']['scale']], w.bias_d, q, eps, st)
        saved = dict(rstd=rstd, xm_o=xm_o, xm_q=xm_q, xm_scale=xm['scale'], xm_idx=xm['outlier_channel_index'], xn_q=xn_q,
                     xn_scale=xn_scale, gate_q=q1, gate_scale=gs, up_q=q2, up_scale=us, gate_xa=gu_xa[0], up_xa=gu_xa[1],
                     gu_xa=gu_xa, down_xa=down_xa64[:, :16], q_bit=q, shape=(B, M, H))
    state.iteration += 1
    return x_out, saved


def _mlp_forward_calibrating(x_medium, w, state, eps, st):
    """A calibration iteration: every save takes its statistics from the finished tensor."""
    require_cuda(x_medium, w.wg, w.wu, w.bg, w.bu)
    B, M, H = x_medium.shape
    T, I, q, it, thd = B * M, w.wg.shape[0], state.q_bit, state.iteration, state.iteration_threshold
    sv, dev = state.static_value, x_medium.device
    x_norm, _, rstd, _, _ = rmsnorm_forward(x_medium, w.norm_w, eps)
    xm_o, xm_q, xm_idx, xm_scale = cf.compression_pack_channel_base(x_medium, state.layernorm_outlier_ratio, q, 'per-channel', it, thd,
                                                                    sv['x_medium'])
    xn2 = x_norm.reshape(T, H)
    gu_xa = lora_a_products(xn2, w.padded()["agu_t"])                # x_norm @ Ag^T and x_norm @ Au^T in one call
    gate_xa, up_xa = gu_xa[0], gu_xa[1]
    q1 = torch.empty((B, M, I * q // 8), dtype=torch.uint8, device=dev)
    q2 = torch.empty((B, M, I * q // 8), dtype=torch.uint8, device=dev)
    had = torch.empty((T, I), dtype=BF16, device=dev)

    def gateup(s1, s2, m1=None, m2=None):
        check(lib.hyc_mlp_gateup_fwd_tcgen05(
            ptr(xn2), ptr(w.wg), ptr(w.wu), T, H, I,
            ptr(gate_xa), ptr(w.bg), 16, 1, ptr(up_xa), ptr(w.bu), 16, 1,
            ptr(s1), ptr(s2), ptr(q1), ptr(q2), ptr(had), ptr(m1), ptr(m2), q, ptr(st), stream_of(x_medium)),
            "hyc_mlp_gateup_fwd_tcgen05")

    # the scales depend on the finished main branches, so the GEMM runs twice (the first pass only materialises
    # gate_main / up_main)
    ones = torch.ones(I, dtype=BF16, device=dev)
    m1 = torch.empty((B, M, I), dtype=BF16, device=dev)
    m2 = torch.empty((B, M, I), dtype=BF16, device=dev)
    gateup(ones, ones, m1, m2)
    gate_scale = cf.get_statistics_only_quant(m1, q, 'per-channel')
    up_scale = cf.get_statistics_only_quant(m2, q, 'per-channel')
    del m1, m2
    gs = gate_scale.to(BF16).reshape(-1).contiguous()
    us = up_scale.to(BF16).reshape(-1).contiguous()
    gateup(gs, us)
    xn_q, xn_scale = cf.compression_pack_quant_base(x_norm, q, 'per-channel', it, thd, sv['x_norm_2'])
    pad = w.padded()
    down_xa64 = had @ pad["ad_cols"]               # [T, 64]: the LoRA-A activation of the down projection, zero-padded
    # down = hadamard @ Wd^T + down_xa @ Bd^T (one more K block) + residual
    x_out = gemm(had, w.wd, a2=down_xa64, b2=pad["bd_cols"], residual=x_medium.reshape(T, H).to(BF16).contiguous(), status=st)
    if w.bias_d is not None:
        x_out += w.bias_d.to(BF16)
    sv['x_medium'] = cf.update_dict(sv['x_medium'], {'outlier_channel_index': xm_idx, 'scale': xm_scale}, it)
    sv['x_norm_2'] = cf.update_dict(sv['x_norm_2'], {'scale': xn_scale}, it)
    sv['gate'] = cf.update_dict(sv['gate'], {'scale': gate_scale}, it)
    sv['up'] = cf.update_dict(sv['up'], {'scale': up_scale}, it)
    saved = dict(rstd=rstd, xm_o=xm_o, xm_q=xm_q, xm_scale=xm_scale, xm_idx=xm_idx, xn_q=xn_q, xn_scale=xn_scale,
                 gate_q=q1, gate_scale=gs, up_q=q2, up_scale=us, gate_xa=gate_xa, up_xa=up_xa, gu_xa=gu_xa,
                 down_xa=down_xa64[:, :16], q_bit=q, shape=(B, M, H))
    return x_out.reshape(B, M, H), saved


def mlp_backward(grad_out, saved, w: MLPWeights, status=None, on_lora_grads=None):
    """-> dict(grad_x, grad_ag, grad_bg, grad_au, grad_bu, grad_ad, grad_bd); LoRA gradients in the
    layout of the weights they belong to ([r, in] / [out, r]).  ``on_lora_grads(dict)`` (optional) is called
    as soon as the six LoRA gradients are enqueued, before the grad_x GEMM and the RMSNorm backward: the
    place to start their all-reduce so that it overlaps the rest of the pass."""
    B, M, H = saved['shape']
    T, q = B * M, saved['q_bit']
    dev = grad_out.device
    st = status if status is not None else _status_tensor(dev)
    g = grad_out.to(BF16).reshape(T, H).contiguous()
    pad = w.padded()
    gu_xa = saved.get('gu_xa')
    if gu_xa is None:
        gu_xa = torch.stack((saved['gate_xa'], saved['up_xa']))
    # grad_down GEMM with the SiLU-Hadamard backward in its epilogue, then the six LoRA gradients: the rank-16 products of
    # grad_gate, grad_up and hadamard from one read of each, the A side of gate and up in one pass over the packed
    # x_norm, de-quantized in shared memory
    had, ggu, gm64, grad_bd, grad_ad, ga, grad_bgu = host.mlp_backward_lora(
        g, [w.wd, w.bg, w.bu, w.bd, pad["ad_rows"]],
        [saved['gate_q'], saved['gate_scale'], saved['up_q'], saved['up_scale'], gu_xa, saved['down_xa'], saved['xn_q'],
         saved['xn_scale']], q, st)
    grads = dict(grad_ag=ga[:16], grad_bg=grad_bgu[0], grad_au=ga[16:32], grad_bu=grad_bgu[1], grad_ad=grad_ad, grad_bd=grad_bd)
    if on_lora_grads is not None:
        on_lora_grads(dict(grads))
    # grad wrt x_norm (gate, up and LoRA products accumulate in one tensor-memory tile), then the RMSNorm backward
    # straight from the saved form of x_medium with the residual gradient added in the same pass
    grad_x = host.mlp_backward_x(g, ggu, gm64, [w.wg, w.wu, pad["agu_rows"], w.norm_w],
                                 [saved['xm_q'], saved['xm_scale'], saved['xm_o'], saved['xm_idx'], saved['rstd']],
                                 [B, M, H], q, st)
    return dict(grads, grad_x=grad_x, hadamard=had, g_gate=ggu[0], g_up=ggu[1])
