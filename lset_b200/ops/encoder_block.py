"""Whole post-LayerNorm encoder block (BERT / XLM-R) forward and backward in two native calls.

Op by op a block is eight launches forward and about thirty backward, each with an autograd node and
a foreign call of its own: at the batch sizes such encoders are used with, the host needs several
times longer to issue them than the GPU to run them. ``run`` hands the sequence to
``lb_encoder_fwd`` / ``lb_encoder_bwd`` (``csrc/block/block.cu``), as ``ops/block.py`` does for the
decoder block; autograd sees one node. Forward values have the bits of the op-by-op path, except in
passes declared to be inference (``ops.block.inference_pass``), whose products may be summed in
pieces; bias gradients are added to their fp32 accumulators without a rounding to bf16 in between.

Taken for blocks of plain bf16 ``Linear`` layers with biases (fused or separate query / key / value)
on the GPU; everything else (tensor parallelism, 8-bit layers, adapters, selective activation
checkpointing, wrapped, hooked or subclassed submodules) keeps the op-by-op path.

Replaces the Python block of the reference (lset/models/encoder/bert/model.py:53-142).
"""
from __future__ import annotations

import ctypes
import math

import torch
from torch.nn.modules.module import _has_any_global_hook

from . import _ac
from . import _native as nv
from ._grads import main_grad_of
from .block import (LbBlockIO, LbLinear, LbProjection, LbStreamCtx, Plan, Watch, _arena_size, _fp, _vp,
                    _work_arena, may_split, node_inputs, records_nothing, unhooked)
from .runtime_options import enabled, options as _rt


class LbEncoderDesc(ctypes.Structure):
    _fields_ = [("H", ctypes.c_int), ("heads", ctypes.c_int), ("hd", ctypes.c_int),
                ("I", ctypes.c_int), ("eps", ctypes.c_float), ("softmax_scale", ctypes.c_float),
                ("ln1_w", _vp), ("ln1_b", _vp), ("ln2_w", _vp), ("ln2_b", _vp),
                ("ln1_wgrad", _fp), ("ln1_bgrad", _fp), ("ln2_wgrad", _fp), ("ln2_bgrad", _fp),
                ("qkv", LbProjection), ("o_proj", LbLinear), ("in_", LbLinear), ("out", LbLinear),
                ("bias", _vp * 6), ("bias_grad", _fp * 6)]


_lib = None
calls = 0     # blocks taken by the runner (for tests)


def _library():
    global _lib
    if _lib is None:
        lib = nv.load()
        for fn in (lib.lb_encoder_saved_bytes, lib.lb_encoder_work_bytes):
            fn.restype, fn.argtypes = ctypes.c_size_t, [_vp, ctypes.c_int]
        for fn in (lib.lb_encoder_fwd, lib.lb_encoder_bwd):
            fn.argtypes = [_vp, _vp, _vp]
        _lib = lib
    return _lib


def _modules(block):
    att, mlp = block.attention, block.mlp
    qkv = [att.qkv_proj] if att.fused_qkv else [att.query, att.key, att.value]
    return qkv, att.dense, mlp.dense_in, mlp.dense_out, att.LayerNorm, mlp.LayerNorm


def _plain(m) -> bool:
    from ..models.layers import Linear

    return (type(m) is Linear and m.bias is not None and "forward" not in m.__dict__
            and not hasattr(m, "_tp_kind") and not m._forward_hooks and not m._forward_pre_hooks
            and not m._backward_hooks and not m._backward_pre_hooks
            and m.weight.dtype == torch.bfloat16 and m.bias.dtype == torch.bfloat16
            and m.weight.is_cuda and m.bias.is_cuda
            and m.weight.is_contiguous() and m.bias.is_contiguous()
            and m.weight.shape[0] % 8 == 0 and m.weight.shape[1] % 8 == 0)


class EncoderPlan(Plan):
    """The tensors that feed the descriptor (``desc``: its sizes); addresses are read on every call."""

    def __init__(self, block):
        self.ok = False
        self.signature = self._signature(block)
        if self.signature is None:
            return
        qkv, o, fin, fout, ln1, ln2 = _modules(block)
        att = block.attention
        H, hd = o.weight.shape[0], att.head_dim
        if hd not in (64, 128) or att.num_heads * hd != H or H % 8:
            return
        if not all(_plain(m) for m in qkv + [o, fin, fout]):
            return
        if any(m.weight.shape != (3 * H // len(qkv), H) for m in qkv):
            return
        if any(m.bias.shape != m.weight.shape[:1] for m in qkv + [o, fin, fout]):
            return
        if (o.weight.shape != (H, H) or fin.weight.shape[1] != H
                or fout.weight.shape != (H, fin.weight.shape[0])):
            return
        for ln in (ln1, ln2):
            if (type(ln) is not torch.nn.LayerNorm or ln.weight is None or ln.bias is None
                    or ln.weight.dtype != torch.bfloat16 or ln.bias.dtype != torch.bfloat16
                    or not ln.weight.is_cuda or ln.eps != ln1.eps
                    or ln.weight.shape != (H,) or ln.bias.shape != (H,)
                    or not ln.weight.is_contiguous() or not ln.bias.is_contiguous()
                    or ln._forward_hooks or ln._forward_pre_hooks or ln._backward_hooks
                    or ln._backward_pre_hooks or "forward" in ln.__dict__):
                return
        d = LbEncoderDesc()
        d.H, d.heads, d.hd, d.I = H, att.num_heads, hd, fin.weight.shape[0]
        d.eps, d.softmax_scale = float(ln1.eps), 1.0 / math.sqrt(hd)
        d.qkv.n, d.qkv.width = len(qkv), 3 * H
        self.desc = d
        self.linears = [*enumerate(qkv), (3, o), (4, fin), (5, fout)]
        part = d.qkv.part
        for i, m in self.linears:
            dst = (part[0], part[1], part[2], d.o_proj, d.in_, d.out)[i]
            dst.n_out, dst.k_in = m.weight.shape
            dst.ldw = m.weight.stride(0)
        self.norms = [(ln1, "ln1"), (ln2, "ln2")]
        self.params = [p for ln, _ in self.norms for p in (ln.weight, ln.bias)]
        self.params += [p for _, m in self.linears for p in (m.weight, m.bias)]
        self.weights = [ln.weight for ln, _ in self.norms] + [m.weight for _, m in self.linears]
        self.ok = True

    @staticmethod
    def _signature(block):
        """Changes when a submodule is wrapped, replaced, hooked, moved, cast or given other
        data (looked up in the modules' dicts, see ``BlockPlan._signature``)."""
        att, mlp = block._modules["attention"], block._modules["mlp"]
        am, mm = att._modules, mlp._modules
        mods = (am["qkv_proj"],) if att.fused_qkv else (am["query"], am["key"], am["value"])
        mods += (am["dense"], mm["dense_in"], mm["dense_out"], am["LayerNorm"], mm["LayerNorm"])
        sig = []
        for m in mods:
            d = m.__dict__
            p = d["_parameters"]
            w, b = p.get("weight"), p.get("bias")
            if w is None or b is None:
                return None
            # (``.data`` of a parameter can be exchanged under the same object)
            sig.append((id(m), type(m), id(w), id(b), "forward" in d, w.dtype, w.device, w.shape,
                        w.is_contiguous(), b.dtype, b.device, b.shape, b.is_contiguous(), d.get("eps"),
                        len(d["_forward_hooks"]), len(d["_forward_pre_hooks"]),
                        len(d["_backward_hooks"]), len(d["_backward_pre_hooks"])))
        return sig

    def fill(self, grads: dict) -> LbEncoderDesc:
        """A descriptor of its own for the call (another thread may be in a pass of the same block),
        with the tensors' present addresses; ``grads`` as in ``BlockPlan.fill``. (Sizes are part of
        the signature; of a pass without gradients the accumulators stay null.)"""
        d = LbEncoderDesc.from_buffer_copy(self.desc)
        part, bias = d.qkv.part, d.bias
        (l1, _), (l2, _) = self.norms
        d.ln1_w, d.ln1_b = l1.weight.data_ptr(), l1.bias.data_ptr()
        d.ln2_w, d.ln2_b = l2.weight.data_ptr(), l2.bias.data_ptr()
        slots = (part[0], part[1], part[2], d.o_proj, d.in_, d.out)
        for i, m in self.linears:
            slots[i].w = m.weight.data_ptr()
            bias[i] = m.bias.data_ptr()
        if grads:
            for ln, name in self.norms:
                setattr(d, name + "_wgrad", grads.get(id(ln.weight)))
                setattr(d, name + "_bgrad", grads.get(id(ln.bias)))
            for i, m in self.linears:
                slots[i].wgrad = grads.get(id(m.weight))
                d.bias_grad[i] = grads.get(id(m.bias))
        return d


def plan_of(block):
    plan = block.__dict__.get("_lb_plan")
    if plan is None or plan.signature is None or plan.signature != plan._signature(block):
        plan = EncoderPlan(block)
        block.__dict__["_lb_plan"] = plan
    return plan if plan.ok else None


_types = None


def _own_forwards(block) -> bool:
    """Whether calling the block's two halves would run the forwards that the runner stands for."""
    global _types
    if _types is None:
        from ..models.bert import BertAttention, BertMLP

        _types = (BertAttention, BertMLP)
    mods = block._modules
    att, mlp = mods["attention"], mods["mlp"]
    if type(att) is not _types[0] or type(mlp) is not _types[1] or _has_any_global_hook():
        return False
    for m in (att, mlp):
        d = m.__dict__
        if ("forward" in d or d["_forward_hooks"] or d["_forward_pre_hooks"]
                or d["_backward_hooks"] or d["_backward_pre_hooks"]):
            return False
    return True


def usable(block, x, ctx) -> bool:
    if not (x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2 and x.shape[0] > 0):
        return False
    if _ac._active is not None or not enabled("block_runner") or _rt.attention_backend == "sdpa":
        return False
    if not enabled("fused_layernorm") or not _own_forwards(block):
        return False
    plan = plan_of(block)
    return plan is not None and x.shape[1] == plan.desc.H and ctx.pos.shape[0] == x.shape[0]


def _stream_struct(ctx, plan: EncoderPlan, device, training: bool) -> LbStreamCtx:
    d = plan.desc
    grad = torch.is_grad_enabled()
    split = may_split(training)
    key = ("_lb_enc", grad, split, d.hd, d.H)
    hit = ctx.tables.get(key)
    if hit is not None:
        return hit
    ap = ctx.plan
    ptf, capf, tile = ap.fwd_tiles(d.heads, d.heads, d.hd)
    ptq, capq = ap.tiles(128) if grad else (None, 0)
    s = LbStreamCtx()
    s.T, s.packed = int(ctx.pos.shape[0]), int(ap.cu_seqlens is not None)
    s.seq_start, s.seq_end = ap.seq_start.data_ptr(), ap.seq_end.data_ptr()
    s.plan_f, s.cap_f, s.tile_f = ptf.data_ptr(), capf, tile
    s.plan_q = s.plan_kv = nv.ptr(ptq) or None      # one query head per KV head: the same tiles
    s.cap_q = s.cap_kv = capq
    s.status = nv.status_word(device).data_ptr()
    # partial sums of the backward's norms: the struct's own, as its backward comes later than other
    # callers' passes, which would grow or write a shared buffer
    sums = None
    if grad:
        sums = torch.empty(2 * _library().lb_norm_bwd_partial_rows() * 2 * d.H, dtype=torch.float32,
                           device=device)
        s.norm_scratch = sums.data_ptr()
    s.may_split = int(split)
    # what the attention of short sequences is chosen by (0: not known)
    s.n_seq, s.max_len = ap.seq_start.numel(), getattr(ap, "max_seqlen", 0)
    s._keep = (ctx.pos, ap, ptf, ptq, sums)
    ctx.tables[key] = s
    return s


class _EncoderBlockFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, plan, sctx, stream_ctx, *params):
        global calls
        lib = _library()
        d = plan.fill({})
        x = x if x.is_contiguous() else x.contiguous()
        T, H = x.shape
        nbytes = lib.lb_encoder_saved_bytes(ctypes.addressof(d), T)
        saved = torch.empty(_arena_size(nbytes), dtype=torch.uint8, device=x.device)
        out = torch.empty_like(x)
        io = LbBlockIO()
        io.branch, io.out, io.saved = x.data_ptr(), out.data_ptr(), saved.data_ptr()
        sctx.stream = nv.stream_ptr()
        rc = lib.lb_encoder_fwd(ctypes.addressof(d), ctypes.addressof(sctx), ctypes.addressof(io))
        if rc != 0:
            nv.check_rc(rc, "lb_encoder_fwd")
        nv.count_launch(io.launches)
        calls += 1
        # the weights, for autograd to see that the backward reads what the forward read
        ctx.save_for_backward(x, saved, *plan.weights)
        ctx.plan, ctx.sctx, ctx.stream_ctx = plan, sctx, stream_ctx
        return out

    @staticmethod
    def backward(ctx, d_out):
        lib = _library()
        x, saved = ctx.saved_tensors[:2]
        plan, sctx = ctx.plan, ctx.sctx
        T, H = x.shape
        d_out = d_out.to(x.dtype).contiguous()
        # weight gradients go straight into the sharding runtime's fp32 accumulators; a parameter
        # without one gets a temporary that is returned to autograd
        grads, temps = {}, []
        for p in plan.params:
            mg = main_grad_of(p) if p.requires_grad else None
            temp = None
            if p.requires_grad and mg is None:
                mg = temp = torch.zeros(p.shape, dtype=torch.float32, device=x.device)
            temps.append(temp)
            if mg is not None:
                grads[id(p)] = mg.data_ptr()
        d = plan.fill(grads)
        work = _work_arena(lib.lb_encoder_work_bytes(ctypes.addressof(d), T), x.device)
        dx = torch.empty_like(x)
        io = LbBlockIO()
        io.branch, io.saved, io.work = x.data_ptr(), saved.data_ptr(), work.data_ptr()
        io.d_out, io.dx = d_out.data_ptr(), dx.data_ptr()
        sctx.stream = nv.stream_ptr()
        rc = lib.lb_encoder_bwd(ctypes.addressof(d), ctypes.addressof(sctx), ctypes.addressof(io))
        if rc != 0:
            nv.check_rc(rc, "lb_encoder_bwd")
        nv.count_launch(io.launches)
        pgrads = tuple(None if t is None else t.to(p.dtype) for t, p in zip(temps, plan.params))
        return (dx, None, None, None) + pgrads


def run(block, x, ctx):
    plan = block.__dict__["_lb_plan"]     # ``usable`` has just accepted it
    sctx = _stream_struct(ctx, plan, x.device, block.training)
    return _EncoderBlockFn.apply(x, plan, sctx, ctx, *node_inputs(plan.params))


class _Inference(Plan):
    """What a pass without derivatives keeps of one block (see ``ops.block._Inference``)."""

    def __init__(self, block, plan):
        qkv, o, fin, fout, ln1, ln2 = _modules(block)
        att, mlp = block.attention, block.mlp
        names = ("qkv_proj",) if att.fused_qkv else ("query", "key", "value")
        names = [(att, n) for n in names + ("dense", "LayerNorm")] + [
            (mlp, n) for n in ("dense_in", "dense_out", "LayerNorm")]
        self.modules = [(owner._modules, n, owner._modules[n], owner._modules[n].__dict__)
                        for owner, n in names]
        self.halves, self.eps, self.norms = (att, mlp), ln1.eps, (ln1.__dict__, ln2.__dict__)
        self.fused = att.fused_qkv
        self.plan = plan
        self.watch = Watch([(m, p) for _, _, m, _ in self.modules for p in ("weight", "bias")])
        d = self.desc = plan.fill({})
        self.addr = ctypes.addressof(d)
        self.sizes = (d.heads, d.I)      # what the size of the block's activations follows from

    def same(self, block) -> bool:
        mods = block._modules
        if (mods["attention"] is not self.halves[0] or mods["mlp"] is not self.halves[1]
                or self.halves[0].fused_qkv != self.fused):
            return False
        for where, name, m, d in self.modules:
            if where.get(name) is not m or not unhooked(d) or "_tp_kind" in d:
                return False
        return (self.norms[0]["eps"] == self.eps and self.norms[1]["eps"] == self.eps
                and self.watch.same())


def _inference_of(block):
    kept = block.__dict__.get("_lb_inference")
    if kept is not None and kept.same(block):
        return kept
    plan = plan_of(block)
    if plan is None:
        return None
    kept = block.__dict__["_lb_inference"] = _Inference(block, plan)
    return kept


def run_inference(block_type, layers, x, ctx):
    """The blocks of a pass without derivatives (see ``ops.block.run_inference``); returns ``(how many,
    x)``."""
    if not (records_nothing() and x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2
            and x.is_contiguous() and x.shape[0] > 0 and ctx.pos.shape[0] == x.shape[0]):
        return 0, x
    if (_ac._active is not None or _rt.attention_backend == "sdpa" or _has_any_global_hook()
            or not enabled("block_runner") or not enabled("fused_layernorm")):
        return 0, x
    global calls
    lib = _library()
    T, H = x.shape
    io, key, sizes, outs, n, launches = LbBlockIO(), None, None, None, 0, 0
    io_at = ctypes.addressof(io)
    for block in layers:
        d = block.__dict__
        if type(block) is not block_type or not unhooked(d) or not _own_forwards(block):
            break
        kept = _inference_of(block)
        if kept is None or kept.desc.H != H:
            break
        k = (kept.desc.hd, d["training"])
        if k != key:
            key = k
            sctx = _stream_struct(ctx, kept.plan, x.device, d["training"])
            sctx.stream = nv.stream_ptr()
            sctx_at = ctypes.addressof(sctx)
        if kept.sizes != sizes:
            sizes = kept.sizes
            arena = torch.empty(_arena_size(lib.lb_encoder_saved_bytes(kept.addr, T)),
                                dtype=torch.uint8, device=x.device)
            io.saved = arena.data_ptr()
        if outs is None:
            outs = torch.empty_like(x), torch.empty_like(x)
        out = outs[n & 1]
        io.branch, io.out = x.data_ptr(), out.data_ptr()
        io.chained = int(n > 0)
        rc = lib.lb_encoder_fwd(kept.addr, sctx_at, io_at)
        if rc != 0:
            nv.check_rc(rc, "lb_encoder_fwd")
        launches += io.launches
        x = out
        n += 1
    if n:
        nv.count_launch(launches)
        calls += n
    return n, x
