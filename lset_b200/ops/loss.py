"""Similarity product for the contrastive losses.

``similarity(q, k)`` returns the fp32 score matrix ``q · kᵀ``. For bf16 CUDA inputs the forward and
both gradient products run on the tcgen05 GEMM (no transposes: the passage-gradient product
consumes the score gradient and the queries as MN-major operands); elsewhere it is a plain matmul.
Replaces the cuBLAS matmul of lset/losses/infonce.py:20 and lset/losses/contrastive.py:22.
"""
from __future__ import annotations

import ctypes

import torch

from . import _native as nv
from .gemm import matmul_abt


class _Similarity(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k):
        ctx.save_for_backward(q, k)
        return matmul_abt(q, k, out_dtype=torch.float32)

    @staticmethod
    def backward(ctx, ds):
        q, k = ctx.saved_tensors
        Q, K = ds.shape
        # bf16 copy of the score gradient with a row stride that is a multiple of 8 elements
        Kp = (K + 7) // 8 * 8
        Qp = (Q + 7) // 8 * 8
        g = torch.zeros(Qp, Kp, dtype=torch.bfloat16, device=ds.device)
        g[:Q, :K] = ds
        dq = dk = None
        if ctx.needs_input_grad[0]:
            kp = k if Kp == K else torch.cat([k, k.new_zeros(Kp - K, k.shape[1])])
            dq = matmul_abt(g[:Q], kp, b_mn=True)                     # [Q, D] = g · k
        if ctx.needs_input_grad[1]:
            qp = q if Qp == Q else torch.cat([q, q.new_zeros(Qp - Q, q.shape[1])])
            dk = matmul_abt(g, qp, a_mn=True, b_mn=True)[:K]          # [K, D] = gᵀ · q
        return dq, dk


def similarity(q: torch.Tensor, k: torch.Tensor) -> torch.Tensor:
    """fp32 ``[Q, K]`` scores of ``q [Q, D]`` against ``k [K, D]``."""
    native = (nv.use_native(q, k) and q.dtype == torch.bfloat16 and k.dtype == torch.bfloat16
              and q.shape[1] % 8 == 0 and k.shape[0] % 8 == 0)
    if native:
        return _Similarity.apply(q.contiguous(), k.contiguous())
    return q.float() @ k.float().t()


# ------------------------------------------------------------------------------------------------
# Backward of the streaming losses in column panels.
#
# The probability gradient W = (softmax - target) * coef is needed as a bf16 operand of two more
# products (dQ = W · K, dK = Wᵀ · Q). It is never held as a whole [Q, K] matrix: the passages are
# walked in panels of columns, the panel's W is recomputed from the saved row LSE, dK of the panel
# is complete after one product, and dQ accumulates over the panels in fp32. A panel's W is capped
# at PANEL_BYTES (half of the 126 MB L2, so the two products that read it find it there); score
# matrices below the cap take a single panel. Extra memory: the cap plus the fp32 accumulator of dQ. (One
# native call, lb_loss_bwd; across ranks dist/xrank_loss.py.)
# ------------------------------------------------------------------------------------------------
PANEL_BYTES = 64 << 20
PANEL_MIN_COLS = 1024       # narrower panels leave the dK product too few tiles


def panel_cols(M: int, N: int) -> int:
    """Columns per panel for M query rows: as many as fit PANEL_BYTES of bf16, a multiple of 256
    (the loss kernels' column tile; keeps label rows 16-byte aligned), at least PANEL_MIN_COLS."""
    Mp = (M + 7) // 8 * 8
    cols = max(PANEL_MIN_COLS, (PANEL_BYTES // (2 * Mp)) // 256 * 256)
    return min(N, cols)


# ------------------------------------------------------------------------------------------------
# Streaming losses: scores never materialise in fp32; see csrc/gemm/loss.h. One native call each way.
# ------------------------------------------------------------------------------------------------
class LbLoss(ctypes.Structure):      # csrc/gemm/loss.h
    _fields_ = [("q", ctypes.c_void_p), ("k", ctypes.c_void_p), ("ldq", ctypes.c_longlong),
                ("ldk", ctypes.c_longlong), ("M", ctypes.c_int), ("N", ctypes.c_int), ("D", ctypes.c_int),
                ("inv_temperature", ctypes.c_float), ("target_offset", ctypes.c_longlong),
                ("labels", ctypes.c_void_p), ("ld_labels", ctypes.c_longlong), ("tw", ctypes.c_void_p),
                ("ld_tw", ctypes.c_longlong), ("row_scale", ctypes.c_void_p), ("row_w", ctypes.c_void_p),
                ("loss_mode", ctypes.c_int), ("loss_scale", ctypes.c_float),
                ("scratch", ctypes.c_void_p), ("lse", ctypes.c_void_p), ("loss", ctypes.c_void_p),
                ("grad", ctypes.c_void_p), ("grad_scale", ctypes.c_float), ("panel", ctypes.c_int),
                ("W", ctypes.c_void_p), ("ldw", ctypes.c_longlong), ("dq", ctypes.c_void_p),
                ("dq32", ctypes.c_void_p), ("dk", ctypes.c_void_p), ("status", ctypes.c_void_p),
                ("stream", ctypes.c_void_p)]


_lib = None


def _library():
    global _lib
    if _lib is None:
        lib = nv.load()
        lib.lb_infonce_scratch_floats.restype = ctypes.c_longlong
        lib.lb_infonce_scratch_floats.argtypes = [ctypes.c_int, ctypes.c_int]
        lib.lb_loss_fwd.argtypes = lib.lb_loss_bwd.argtypes = [ctypes.c_void_p]
        _lib = lib
    return _lib


def _loss_struct(q, k, inv_t, target_offset=0, labels8=None, tw=None, row_scale=None, row_w=None,
                 mode=0) -> LbLoss:
    p = LbLoss()
    p.q, p.k, p.ldq, p.ldk = q.data_ptr(), k.data_ptr(), q.stride(0), k.stride(0)
    p.M, p.D = q.shape
    p.N = k.shape[0]
    p.inv_temperature, p.target_offset = inv_t, target_offset
    if labels8 is not None:
        p.labels, p.ld_labels = labels8.data_ptr(), labels8.stride(0)
        p.row_scale, p.row_w, p.loss_mode = row_scale.data_ptr(), row_w.data_ptr(), mode
        if tw is not None:
            p.tw, p.ld_tw = tw.data_ptr(), tw.stride(0)
    p.status, p.stream = nv.status_word(q.device).data_ptr(), nv.stream_ptr()
    return p


def _loss_fwd(p: LbLoss, q, loss_scale: float):
    """``(loss [], lse [M])``."""
    lib = _library()
    scr = torch.empty(lib.lb_infonce_scratch_floats(p.M, (p.N + 7) // 8 * 8), dtype=torch.float32,
                      device=q.device)
    lse = torch.empty(p.M, dtype=torch.float32, device=q.device)
    loss = torch.empty((), dtype=torch.float32, device=q.device)
    p.scratch, p.lse, p.loss, p.loss_scale = scr.data_ptr(), lse.data_ptr(), loss.data_ptr(), loss_scale
    nv.check_rc(lib.lb_loss_fwd(ctypes.addressof(p)), "lb_loss_fwd")
    nv.count_launch(2)
    return loss, lse


def _loss_bwd(p: LbLoss, q, k, lse, grad, grad_scale: float, need_dq: bool, need_dk: bool):
    """``(dq, dk)``, in panels of columns of at most ``PANEL_BYTES`` of probability gradient."""
    step = panel_cols(p.M, p.N)
    grad = grad if grad.dtype == torch.float32 else grad.float()
    ldw = (step + 7) // 8 * 8
    W = torch.empty(p.M, ldw, dtype=torch.bfloat16, device=q.device)
    dq = torch.empty(p.M, p.D, dtype=torch.bfloat16 if step >= p.N else torch.float32,
                     device=q.device) if need_dq else None
    dk = torch.empty(p.N, p.D, dtype=torch.bfloat16, device=q.device) if need_dk else None
    p.lse, p.grad, p.grad_scale = lse.data_ptr(), grad.data_ptr(), grad_scale
    p.panel, p.W, p.ldw = step, W.data_ptr(), ldw
    if need_dq:
        p.dq = dq.data_ptr()
        if step < p.N:
            p.dq32 = dq.data_ptr()
    p.dk = dk.data_ptr() if need_dk else None
    nv.check_rc(_library().lb_loss_bwd(ctypes.addressof(p)), "lb_loss_bwd")
    nv.count_launch((1 + need_dq + need_dk) * ((p.N + step - 1) // step))
    if need_dq and step < p.N:
        dq = dq.to(q.dtype)
    return dq, dk


class _FusedInfoNCE(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, inv_t, target_offset, denom):
        loss, lse = _loss_fwd(_loss_struct(q, k, inv_t, target_offset), q, 1.0 / denom)
        ctx.save_for_backward(q, k, lse)
        ctx.meta = (inv_t, target_offset, denom)
        return loss

    @staticmethod
    def backward(ctx, g):
        q, k, lse = ctx.saved_tensors
        inv_t, target_offset, denom = ctx.meta
        dq, dk = _loss_bwd(_loss_struct(q, k, inv_t, target_offset), q, k, lse, g, inv_t / denom,
                           ctx.needs_input_grad[0], ctx.needs_input_grad[1])
        return dq, dk, None, None, None


def fused_infonce_supported(q, k) -> bool:
    return (nv.use_native(q, k) and q.dtype == torch.bfloat16 and k.dtype == torch.bfloat16
            and q.shape[1] % 8 == 0 and k.shape[0] % 8 == 0 and q.shape[1] == k.shape[1])


def fused_infonce(q, k, temperature: float, target_offset: int = 0, denom: float | None = None):
    """``sum_r CE(q_r · Kᵀ / T, r + target_offset) / denom`` (``denom`` defaults to the number of
    queries) on the streaming tcgen05 kernels. ``temperature`` must be a Python float."""
    denom = float(denom if denom is not None else q.shape[0])
    return _FusedInfoNCE.apply(q.contiguous(), k.contiguous(), 1.0 / float(temperature),
                               int(target_offset), denom)


# ------------------------------------------------------------------------------------------------
# Streaming label-matrix loss (multi-positive NCE / soft-label cross-entropy): the [Q, K] scores
# exist only as tensor-core accumulators.
# ------------------------------------------------------------------------------------------------
class _FusedLabelLoss(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, labels8, tw, row_scale, row_w, inv_t):
        loss, lse = _loss_fwd(_loss_struct(q, k, inv_t, 0, labels8, tw, row_scale, row_w), q, 1.0)
        ctx.save_for_backward(q, k, lse, labels8, row_scale, row_w, *([tw] if tw is not None else []))
        ctx.inv_t = inv_t
        return loss

    @staticmethod
    def backward(ctx, g):
        q, k, lse, labels8, row_scale, row_w, *rest = ctx.saved_tensors
        p = _loss_struct(q, k, ctx.inv_t, 0, labels8, rest[0] if rest else None, row_scale, row_w)
        dq, dk = _loss_bwd(p, q, k, lse, g, ctx.inv_t, ctx.needs_input_grad[0], ctx.needs_input_grad[1])
        return dq, dk, None, None, None, None, None


def fused_label_loss_supported(q, k) -> bool:
    return (nv.use_native(q, k) and q.dtype == torch.bfloat16 and k.dtype == torch.bfloat16
            and q.shape[1] % 8 == 0 and q.shape[1] == k.shape[1])


_LABEL_KINDS = {torch.float32: 0, torch.int64: 1, torch.int32: 2, torch.int8: 3, torch.bool: 3}


def _label_prep(labels, kind: int, Kp: int):
    """``(int8 labels [Q, Kp], row_scale [Q], row_w [Q])`` of a 0/1/-1 label matrix in one launch."""
    Q, K = labels.shape
    dev = labels.device
    lab8 = torch.empty(Q, Kp, dtype=torch.int8, device=dev)
    stats = torch.empty(2 * Q + 2, dtype=torch.float32, device=dev)     # two words of counters behind
    at = stats.data_ptr()
    rc = nv.load().lb_label_prep(
        nv.c_void_p(labels.data_ptr()), nv.c_int(kind), nv.c_ll(labels.stride(0)), nv.c_int(Q),
        nv.c_int(K), nv.c_int(Kp), nv.c_void_p(lab8.data_ptr()), nv.c_void_p(at),
        nv.c_void_p(at + 4 * Q), nv.c_void_p(at + 8 * Q), nv.c_void_p(nv.stream_ptr()))
    nv.check_rc(rc, "lb_label_prep")
    nv.count_launch()
    return lab8, stats[:Q], stats[Q:2 * Q]


def fused_label_loss(q, k, labels, temperature: float, scores=None):
    """Label-matrix contrastive loss on the streaming kernels. ``labels [Q, K]``: 1 positive,
    0 negative, negative values ignored. Without ``scores``: multi-positive NCE
    ``mean_q(LSE_valid(s_q) − mean_{p ∈ pos(q)} s_qp)``; with ``scores``: soft-label cross-entropy
    against ``scores / sum(scores)`` over the non-ignored columns. Queries without a positive (or
    with a zero score sum) are skipped, as in lset/losses/contrastive.py:22-53. No host sync."""
    Q, K = labels.shape
    dev = q.device
    Kp = (K + 31) // 32 * 32
    kind = _LABEL_KINDS.get(labels.dtype)
    if (scores is None and kind is not None and labels.device == dev and Q > 0 and K > 0
            and (K == 1 or labels.stride(1) == 1)):
        lab8, row_scale, row_w = _label_prep(labels, kind, Kp)
        return _FusedLabelLoss.apply(q.contiguous(), k.contiguous(), lab8, None,
                                     row_scale, row_w, 1.0 / float(temperature))
    lab8 = torch.full((Q, Kp), -1, dtype=torch.int8, device=dev)
    lab8[:, :K].copy_(labels)           # converts in the copy: no fp32 [Q, K] temporary
    labels = lab8[:, :K]
    any_valid = labels.max(dim=1).values >= 0      # row statistics without [Q, K] temporaries
    tw = None
    if scores is not None:
        tw = torch.zeros(Q, Kp, dtype=torch.float32, device=dev)
        tw[:, :K] = scores.to(dev, torch.float32)
        torch.nan_to_num_(tw, nan=0.0, posinf=0.0, neginf=0.0)   # "no teacher score": target 0
        tw[:, :K].masked_fill_(labels < 0, 0.0)
        tsum = tw.sum(dim=1)
        keep = (tsum > 0) & any_valid
        row_scale = 1.0 / tsum.clamp(min=1e-12)
    else:
        n_pos = labels.clamp(min=0).sum(dim=1, dtype=torch.int32)   # labels are -1 / 0 / 1 here
        keep = (n_pos > 0) & any_valid
        row_scale = 1.0 / n_pos.clamp(min=1).float()
    keepf = keep.float()
    row_w = keepf / keepf.sum().clamp(min=1.0)
    return _FusedLabelLoss.apply(q.contiguous(), k.contiguous(), lab8, tw,
                                 row_scale.contiguous(), row_w.contiguous(),
                                 1.0 / float(temperature))


# ------------------------------------------------------------------------------------------------
# Multi-positive NCE (every positive against the query's negatives only), and the int8-label
# "soft" / "cross" cross-entropies: the three loss types of lset/kernels/loss.py:1051-1089.
# ------------------------------------------------------------------------------------------------
def reference_switches_to_fused(num_queries: int, num_docs: int, loss_type: str = "multi") -> bool:
    """Sizes from which the reference replaces its eager label-matrix loss by its fused kernel, and
    with it the loss definition (lset/kernels/loss.py:37-55). Used only to keep the *semantics*
    aligned with the reference at every batch size; speed is not the criterion here."""
    if loss_type == "multi":
        return num_queries >= 2048 or (num_queries >= 1024 and num_docs >= 4096)
    return num_queries >= 2048 and num_docs >= 4096


def _pad_labels_int8(labels):
    Q, K = labels.shape
    Kp = (K + 31) // 32 * 32
    lab8 = torch.full((Q, Kp), -1, dtype=torch.int8, device=labels.device)
    lab8[:, :K].copy_(labels)
    return lab8


class _FusedMpNce(torch.autograd.Function):
    """loss = mean_{valid q} mean_{p ∈ pos(q)} softplus(LSE_{n ∈ neg(q)} s_qn − s_qp)."""

    @staticmethod
    def forward(ctx, q, k, labels8, pos_qi, pos_di, inv_t):
        M, N, dev = q.shape[0], k.shape[0], q.device
        ones = torch.ones(M, dtype=torch.float32, device=dev)
        zeros = torch.zeros(M, dtype=torch.float32, device=dev)
        _, neg_lse = _loss_fwd(_loss_struct(q, k, inv_t, 0, labels8, None, ones, zeros, mode=1), q, 1.0)
        lab = labels8[:, :N]
        num_pos = (lab > 0).sum(dim=1)
        has_neg = (lab == 0).any(dim=1)
        valid = ((num_pos > 0) & has_neg).float()
        denom = valid.sum().clamp(min=1.0)
        num_pos_f = num_pos.clamp(min=1).float()
        # scores of the positive pairs: P row dot products (P is a few per query)
        pos_scores = (q[pos_qi].float() * k[pos_di].float()).sum(dim=1) * inv_t
        gap = neg_lse[pos_qi] - pos_scores
        per_pos = torch.nn.functional.softplus(gap)
        q_sum = torch.zeros(M, dtype=torch.float32, device=dev).index_add_(0, pos_qi, per_pos)
        loss = ((q_sum / num_pos_f) * valid).sum() / denom
        aux = torch.zeros(M, dtype=torch.float32, device=dev).index_add_(0, pos_qi,
                                                                          torch.sigmoid(gap))
        row_w = valid / (denom * num_pos_f)
        ctx.save_for_backward(q, k, labels8, neg_lse, aux, row_w)
        ctx.inv_t = inv_t
        return loss

    @staticmethod
    def backward(ctx, g):
        q, k, labels8, neg_lse, aux, row_w = ctx.saved_tensors
        p = _loss_struct(q, k, ctx.inv_t, 0, labels8, None, aux, row_w, mode=1)
        dq, dk = _loss_bwd(p, q, k, neg_lse, g, ctx.inv_t, ctx.needs_input_grad[0],
                           ctx.needs_input_grad[1])
        return dq, dk, None, None, None, None


def fused_dense_loss(q, k, labels, scale: float, loss_type: str = "multi", pos_qi=None,
                     pos_di=None, pos_counts=None):
    """The reference's fused dense embedding loss (lset/kernels/loss.py:1051-1089) on the streaming
    tcgen05 kernels. ``labels [Q, K]`` int8-valued: > 0 positive (the value is the soft label for
    "soft" / "cross"), 0 negative, < 0 ignored. ``scale`` = 1 / temperature (Python float).

    * ``"multi"``: multi-positive NCE, ``mean_q mean_{p} softplus(LSE_neg(q) − s_qp)`` over queries
      that have a positive and a negative.
    * ``"soft"``:  ``mean_q (LSE_valid(q) − Σ_k (l_qk / Σ l_q) s_qk)`` over queries with Σ l_q > 0.
    * ``"cross"``: ``mean_q (Σ l_q · LSE_valid(q) − Σ_k l_qk s_qk)``.
    ``pos_qi`` / ``pos_di`` (indices of the positive pairs, as the collator provides them) avoid a
    ``nonzero`` on the label matrix; ``pos_counts`` is accepted for signature parity."""
    del pos_counts
    if loss_type not in ("multi", "soft", "cross"):
        raise ValueError(f"unknown loss_type {loss_type!r}")
    lab8 = _pad_labels_int8(labels.to(q.device))
    K = labels.shape[1]
    q, k = q.contiguous(), k.contiguous()
    if loss_type == "multi":
        if pos_qi is None or pos_di is None:
            pos_qi, pos_di = (lab8[:, :K] > 0).nonzero(as_tuple=True)
        return _FusedMpNce.apply(q, k, lab8, pos_qi.to(q.device).long(), pos_di.to(q.device).long(),
                                 float(scale))
    lab = lab8[:, :K]
    label_sum = lab.clamp(min=0).sum(dim=1).float()
    keep = (label_sum > 0).float()
    row_scale = 1.0 / label_sum.clamp(min=1e-9)
    row_w = keep / keep.sum().clamp(min=1.0)
    if loss_type == "cross":
        row_w = row_w * label_sum     # Σl·LSE − Σ l·s  =  Σl · (LSE − Σ (l/Σl)·s)
    return _FusedLabelLoss.apply(q, k, lab8, None, row_scale.contiguous(), row_w.contiguous(),
                                 float(scale))
