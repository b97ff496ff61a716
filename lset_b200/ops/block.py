"""Whole-decoder-block forward and backward in two native calls.

A pre-norm decoder block is a fixed sequence of about a dozen kernel launches forward and two dozen
backward. Issued op by op from Python (one ``autograd.Function`` and one foreign call per launch)
the host needs longer to enqueue them than the GPU needs to run them. ``run`` hands the whole
sequence to the library's block runner (``csrc/block/block.cu``): Python allocates the outputs and
one activation arena, fills three small structs and makes one call; autograd sees one node per
block. The kernels, their order and their arguments are those of the op-by-op path, so both paths
produce the same numbers.

Taken for blocks whose projections are plain bf16 ``Linear`` layers (fused, or separate) or LoRA
wrappers around them, without biases. Tensor-parallel blocks on a token-sharded stream (sequence
parallelism with the fused all-gather / reduce-scatter GEMMs, fused QKV and gate-up weights, packed
batches) are taken too: the runner then issues the gathered and the reduced GEMMs and their device
barriers itself, on the symmetric buffers of the group's ``SPState``, in the order the op-by-op
path uses. Everything else (all-reduce tensor parallelism, FP8 / NF4 layers, Gemma's sandwich
norms, selective activation checkpointing, CPU tensors) keeps the op-by-op path.

Replaces the Python block of the reference (lset/models/decoder/qwen3/block.py:23-68).
"""
from __future__ import annotations

import contextlib
import ctypes
import math
import threading

import torch

from torch.nn.modules.module import _has_any_global_hook

from . import _ac
from . import _native as nv
from ._grads import main_grad_of
from .runtime_options import enabled, options as _rt

_vp, _fp, _ip = ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p


class LbLinear(ctypes.Structure):
    _fields_ = [("w", _vp), ("wgrad", _fp), ("lora_a", _vp), ("lora_b", _vp),
                ("lora_a_grad", _fp), ("lora_b_grad", _fp), ("ldw", ctypes.c_longlong),
                ("n_out", ctypes.c_int), ("k_in", ctypes.c_int), ("lora_r", ctypes.c_int),
                ("lora_scale", ctypes.c_float)]


class LbProjection(ctypes.Structure):
    _fields_ = [("part", LbLinear * 3), ("n", ctypes.c_int), ("width", ctypes.c_int)]


class LbBlockDesc(ctypes.Structure):
    _fields_ = [("H", ctypes.c_int), ("Hq", ctypes.c_int), ("Hk", ctypes.c_int),
                ("hd", ctypes.c_int), ("I", ctypes.c_int), ("causal", ctypes.c_int),
                ("act_kind", ctypes.c_int), ("qk_norm", ctypes.c_int), ("eps", ctypes.c_float),
                ("w_off", ctypes.c_float), ("softmax_scale", ctypes.c_float),
                ("ln1_w", _vp), ("ln1_wgrad", _fp), ("ln2_w", _vp), ("ln2_wgrad", _fp),
                ("qn_w", _vp), ("qn_wgrad", _fp), ("kn_w", _vp), ("kn_wgrad", _fp),
                ("qkv", LbProjection), ("gate_up", LbProjection), ("o_proj", LbLinear),
                ("down", LbLinear)]


class LbStreamCtx(ctypes.Structure):
    _fields_ = [("T", ctypes.c_int), ("packed", ctypes.c_int), ("cos", _fp), ("sin", _fp),
                ("pos", _vp), ("pos_i64", ctypes.c_int), ("seq_start", _ip), ("seq_end", _ip),
                ("plan_f", _ip), ("cap_f", ctypes.c_int), ("tile_f", ctypes.c_int),
                ("plan_q", _ip), ("cap_q", ctypes.c_int), ("plan_kv", _ip),
                ("cap_kv", ctypes.c_int), ("status", _ip), ("norm_scratch", _fp),
                ("rope_scratch", _fp), ("wg_tmp", _fp), ("stream", _vp),
                ("may_split", ctypes.c_int), ("n_seq", ctypes.c_int), ("max_len", ctypes.c_int)]


class LbTpCtx(ctypes.Structure):
    _fields_ = [("world", ctypes.c_int), ("rank", ctypes.c_int), ("rows", ctypes.c_int),
                ("reserved", ctypes.c_int), ("ag_peers", _vp * 2), ("ag_local", _vp * 2),
                ("ag_flags", _vp), ("ag_counter", _vp), ("rs_peers", _vp * 2),
                ("rs_local", _vp * 2), ("pads", _vp), ("bar_limit_ns", ctypes.c_ulonglong),
                ("ag_epoch", ctypes.c_uint), ("ag_calls", ctypes.c_uint),
                ("rs_epoch", ctypes.c_uint), ("bar_epoch", ctypes.c_uint)]


class LbBlockIO(ctypes.Structure):
    _fields_ = [("branch", _vp), ("residual", _vp), ("out", _vp), ("res_out", _vp),
                ("saved", _vp), ("d_out", _vp), ("d_res_out", _vp), ("dx", _vp), ("work", _vp),
                ("tp", _vp), ("fewer_launches", ctypes.c_int), ("launches", ctypes.c_int),
                ("chained", ctypes.c_int)]


_lib = None
calls = {"dp": 0, "tp": 0}   # block forwards taken by the runner, by stream layout (for tests)


def _library():
    global _lib
    if _lib is None:
        lib = nv.load()
        lib.lb_block_saved_bytes.restype = ctypes.c_size_t
        lib.lb_block_work_bytes.restype = ctypes.c_size_t
        for fn in (lib.lb_block_fwd, lib.lb_block_bwd):
            fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
        lib.lb_block_saved_bytes.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int,
                                             ctypes.c_void_p]
        lib.lb_block_work_bytes.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p]
        lib.lb_block_fwd_launches.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int,
                                              ctypes.c_void_p]
        lib.lb_block_bwd_launches.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p]
        _lib = lib
    return _lib


def _arena_size(nbytes: int) -> int:
    """``nbytes`` rounded up to the next size of a geometric series (eight sizes per octave, at
    most 12.5 % more). Packed batches differ in token count from step to step; with exact sizes
    every batch longer than all before it makes the caching allocator ask the driver for one new
    block per decoder block (a stall of up to several hundred milliseconds on a busy host), with
    rounded sizes that happens a few times at the start of a run and then no more."""
    if nbytes <= (1 << 20):
        return max(nbytes, 1)
    top = 1 << (nbytes.bit_length() - 1)       # largest power of two <= nbytes
    step = top >> 3
    return (nbytes + step - 1) // step * step


def _work_arena(nbytes: int, device) -> torch.Tensor:
    """Temporary storage of one block's backward. Each call has its own: passes of other streams run
    at the same time, and the allocator hands blocks of one stream's passes the same memory."""
    return torch.empty(_arena_size(nbytes), dtype=torch.uint8, device=device)


# --------------------------------------------------------------------------- eligibility
def _plain_linear(m) -> bool:
    from ..models.layers import Linear

    return (type(m) is Linear and m.bias is None and "forward" not in m.__dict__
            and not hasattr(m, "_tp_kind") and m.weight.dtype == torch.bfloat16
            and m.weight.is_cuda and m.weight.stride(-1) == 1)


def _sp_linear(m, kind: str, st) -> bool:
    """A bias-free bf16 ``Linear`` that ``apply_tp`` wrapped for the token-sharded stream."""
    from ..models.layers import Linear

    return (type(m) is Linear and m.bias is None and getattr(m, "_tp_kind", None) == kind
            and getattr(m, "_sp_state", None) is st and m.weight.dtype == torch.bfloat16
            and m.weight.is_cuda and m.weight.stride(-1) == 1)


def _linear_parts(m):
    """``(weight, lora_A weight or None, lora_B weight or None, scale)`` for a supported projection
    module, else None."""
    if _plain_linear(m):
        return m.weight, None, None, 0.0
    base = getattr(m, "base_linear", None)
    if base is not None and hasattr(m, "lora_A") and _plain_linear(base):
        a, b = m.lora_A, m.lora_B
        drop = getattr(m, "dropout", None)
        if (_plain_linear(a) and _plain_linear(b) and m.r % 8 == 0
                and (isinstance(drop, torch.nn.Identity) or not m.training)):
            return base.weight, a.weight, b.weight, float(m.scale)
    return None


def _no_plan():
    return None


class Plan:
    """Kept in its block's ``__dict__``. A copy or a pickle of the model is without it (the descriptor
    holds addresses) and makes its own."""

    def __reduce__(self):
        return _no_plan, ()


class BlockPlan(Plan):
    """What the runner needs to know about one ``DecoderBlock``: which tensors feed which field of
    the descriptor. Pointers are re-read on every call (parameters may be re-homed into flat
    buffers after the plan was made)."""

    def __init__(self, block):
        att, mlp, tr = block.self_attn, block.mlp, block.traits
        self.ok = False
        self.signature = self._signature(block)
        if tr.sandwich_norms or att.head_dim not in (64, 128):
            return
        if att.num_heads % att.num_kv_heads or (att.num_heads // att.num_kv_heads) not in (1, 2, 4, 8):
            return
        qkv_mods = [att.qkv_proj] if att.fused_qkv else [att.q_proj, att.k_proj, att.v_proj]
        gu_mods = [mlp.gate_up_proj] if mlp.fused_gate_up else [mlp.gate_proj, mlp.up_proj]
        mods = qkv_mods + [att.o_proj] + gu_mods + [mlp.down_proj]
        # tensor parallelism on a token-sharded stream: every projection carries the group's state
        self.sp = getattr(att.o_proj, "_sp_state", None)
        if self.sp is not None:
            kinds = ("colwise", "rowwise", "colwise", "rowwise")
            if len(mods) != 4 or not all(_sp_linear(m, k, self.sp) for m, k in zip(mods, kinds)):
                return
            parts = [(m.weight, None, None, 0.0) for m in mods]
        else:
            parts = [_linear_parts(m) for m in mods]
        if any(p is None for p in parts):
            return
        self.qkv, self.o = parts[:len(qkv_mods)], parts[len(qkv_mods)]
        self.gate_up, self.down = parts[len(qkv_mods) + 1:-1], parts[-1]
        self.ln1, self.ln2 = block.input_layernorm, block.post_attention_layernorm
        self.qn = att.q_norm.weight if att.q_norm is not None else None
        self.kn = att.k_norm.weight if att.k_norm is not None else None
        hd = att.head_dim
        H = self.ln1.weight.shape[0]
        width = sum(p[0].shape[0] for p in self.qkv)
        if width % ((att.num_heads // att.num_kv_heads + 2) * hd):
            return
        Hk = width // ((att.num_heads // att.num_kv_heads + 2) * hd)
        Hq = Hk * (att.num_heads // att.num_kv_heads)
        I = sum(p[0].shape[0] for p in self.gate_up) // 2
        if H % 8 or I % 8 or self.down[0].shape[1] != I or self.o[0].shape[1] != Hq * hd:
            return
        if len(self.gate_up) == 2 and self.gate_up[0][0].shape[0] != I:
            return
        if len(self.qkv) == 3 and [p[0].shape[0] for p in self.qkv] != [Hq * hd, Hk * hd, Hk * hd]:
            return
        for w in (self.ln1.weight, self.ln2.weight, self.qn, self.kn):
            if w is not None and (w.dtype != torch.bfloat16 or not w.is_cuda):
                return
        d = LbBlockDesc()
        d.H, d.Hq, d.Hk, d.hd, d.I = H, Hq, Hk, hd, I
        d.causal = int(att.causal)
        d.act_kind = {"swiglu": 0, "geglu": 1}[mlp.kind]
        d.qk_norm = int(self.qn is not None)
        d.eps, d.w_off = float(self.ln1.eps), float(self.ln1.w_off)
        d.softmax_scale = float(att.softmax_scale if att.softmax_scale is not None
                                else 1.0 / math.sqrt(hd))
        d.qkv.n, d.qkv.width = len(self.qkv), width
        d.gate_up.n, d.gate_up.width = len(self.gate_up), 2 * I
        self.desc = d
        self.rope = (hd, att.rope_theta, att.rope_scaling)
        # every trainable tensor, in the order the autograd node lists them
        self.params = []
        for w in (self.ln1.weight, self.ln2.weight, self.qn, self.kn):
            if w is not None:
                self.params.append(w)
        for p in self.qkv + [self.o] + self.gate_up + [self.down]:
            self.params.extend(t for t in p[:3] if t is not None)
        self._launches = {}
        self.ok = True

    @staticmethod
    def _signature(block):
        """Changes when a projection, a norm or a weight is wrapped, replaced, moved or cast after the
        plan was made (which keeps them alive: an id stands for one object). (Modules and parameters
        are looked up in their dicts: attribute access on a module costs more than the rest of this,
        which runs for every block of every pass.)"""
        att, mlp = block._modules["self_attn"], block._modules["mlp"]
        am, mm = att._modules, mlp._modules
        mods = ((am["qkv_proj"],) if att.fused_qkv else (am["q_proj"], am["k_proj"], am["v_proj"]))
        mods += (am["o_proj"],)
        mods += ((mm["gate_up_proj"],) if mlp.fused_gate_up else (mm["gate_proj"], mm["up_proj"]))
        sig = []
        for m in mods + (mm["down_proj"],):
            d = m.__dict__
            w = d["_parameters"].get("weight")
            if w is None:
                w = m.weight
            sig.append((id(m), type(m), id(w), "forward" in d, id(d.get("_sp_state")), w.dtype, w.device,
                        d["training"]))
        bm = block._modules
        for m in (bm["input_layernorm"], bm["post_attention_layernorm"], am.get("q_norm"), am.get("k_norm")):
            if m is not None:
                sig.append((id(m), id(m.__dict__["_parameters"].get("weight"))))
        return sig

    def still_valid(self, block) -> bool:
        return self.signature == self._signature(block)

    # ------------------------------------------------------------------ descriptor
    @staticmethod
    def _fill_linear(dst: LbLinear, part, grads) -> None:
        w, a, b, scale = part
        dst.w = w.data_ptr()
        dst.ldw = w.stride(0)
        dst.n_out, dst.k_in = w.shape
        if grads:            # (of a pass without gradients the accumulators stay null)
            dst.wgrad = grads.get(id(w))
        if a is not None:
            dst.lora_a, dst.lora_b = a.data_ptr(), b.data_ptr()
            dst.lora_a_grad, dst.lora_b_grad = grads.get(id(a)), grads.get(id(b))
            dst.lora_r, dst.lora_scale = a.shape[0], scale

    def fill(self, grads: dict) -> LbBlockDesc:
        """A descriptor of its own for the call (another thread may be in a pass of the same block),
        with the tensors' present addresses. ``grads`` maps ``id(param)`` to the address of its fp32
        gradient accumulator (absent = no weight gradient wanted)."""
        d = LbBlockDesc.from_buffer_copy(self.desc)
        ln1, ln2 = self.ln1.weight, self.ln2.weight
        d.ln1_w, d.ln2_w = ln1.data_ptr(), ln2.data_ptr()
        if self.qn is not None:
            d.qn_w, d.kn_w = self.qn.data_ptr(), self.kn.data_ptr()
        if grads:
            d.ln1_wgrad, d.ln2_wgrad = grads.get(id(ln1)), grads.get(id(ln2))
            if self.qn is not None:
                d.qn_wgrad, d.kn_wgrad = grads.get(id(self.qn)), grads.get(id(self.kn))
        for i, p in enumerate(self.qkv):
            self._fill_linear(d.qkv.part[i], p, grads)
        for i, p in enumerate(self.gate_up):
            self._fill_linear(d.gate_up.part[i], p, grads)
        self._fill_linear(d.o_proj, self.o, grads)
        self._fill_linear(d.down, self.down, grads)
        return d


def node_inputs(params):
    """The parameters an autograd node lists: those of a pass that records no derivatives are left
    out (each costs the call a look at its wrapper)."""
    if torch.is_grad_enabled() or torch.autograd.forward_ad._current_level >= 0:
        return params
    return ()


def plan_of(block):
    plan = block.__dict__.get("_lb_plan")
    if plan is None or not plan.still_valid(block):
        plan = BlockPlan(block)
        block.__dict__["_lb_plan"] = plan
    return plan if plan.ok else None


_types = None


def _own_forwards(block) -> bool:
    """Whether calling the block's two halves would run the forwards that the runner stands for."""
    global _types
    if _types is None:
        from ..models.layers import Attention, GatedMLP

        _types = (Attention, GatedMLP)
    mods = block._modules
    att, mlp = mods["self_attn"], mods["mlp"]
    return (type(att) is _types[0] and type(mlp) is _types[1]
            and "forward" not in att.__dict__ and "forward" not in mlp.__dict__)


def usable(block, branch, ctx) -> bool:
    """True when this call can go through the block runner."""
    if not (branch.is_cuda and branch.dtype == torch.bfloat16 and branch.dim() == 2):
        return False
    if _ac._active is not None or not enabled("block_runner") or _rt.attention_backend == "sdpa":
        return False
    for name in ("fused_rmsnorm", "fused_residual_rmsnorm", "fused_qk_norm_rope"):
        if not enabled(name):
            return False
    if not _own_forwards(block):
        return False
    plan = plan_of(block)
    if plan is None:
        return False
    if plan.sp is None:
        if ctx.pos.shape[0] != branch.shape[0]:  # a token-sharded stream needs the group's state
            return False
    elif not _sp_ready(plan.sp, branch, ctx):
        return False
    if torch.is_grad_enabled() and plan.desc.hd > 128:
        return False
    return True


# --------------------------------------------------------------------------- token-sharded stream
def _sp_ready(st, branch, ctx) -> bool:
    """The runner drives the fused tensor-parallel GEMMs only on peer memory with bf16
    accumulators and the device barrier, for packed batches."""
    st.bind(branch.device)
    if not (st.fused and st.rs_bf16 and enabled("tp_block_runner")):
        return False
    if ctx.plan.cu_seqlens is None or branch.shape[0] * st.world < ctx.pos.shape[0]:
        return False
    return st.token().pad is not None


def _tp_struct(st, rows: int, H: int):
    """The group's symmetric buffers and counters as the runner's struct, plus what to advance
    after the call. Buffers are created (a rendezvous of the group) on first use or growth; every
    rank gets here with the same shapes."""
    buf, rs, tok = st.ag_buf(rows, H), st.rs_buf(rows, H), st.token()
    fl = buf.flags(rows)
    t = LbTpCtx()
    t.world, t.rank, t.rows = st.world, st.rank, rows
    keep = []
    for i in range(2):
        a, b = buf.x_sym[i].c_ptr_array(), rs.slot_ptrs(i, rows, H)
        keep += [a, b]
        t.ag_peers[i] = ctypes.cast(a, ctypes.c_void_p)
        t.rs_peers[i] = ctypes.cast(b, ctypes.c_void_p)
        t.ag_local[i] = buf.x_sym[i].local.data_ptr()
        t.rs_local[i] = rs.acc[i].local.data_ptr()
    t.ag_flags, t.ag_counter = fl[0].data_ptr(), buf.counter.data_ptr()
    pads = tok.pad.c_ptr_array()
    keep.append(pads)
    t.pads = ctypes.cast(pads, ctypes.c_void_p)
    t.bar_limit_ns = tok.limit_ns
    t.ag_epoch, t.ag_calls = st._ag_epoch[H], fl[1]
    t.rs_epoch, t.bar_epoch = rs.epoch, tok.epoch
    t._keep = keep
    return t, (st, H, fl, rs, tok)


def _tp_advance(state) -> None:
    """Each runner call makes two uses of the publication area and of the accumulators and passes
    four barriers (see ``LbTpCtx`` in csrc/block/block.h)."""
    st, H, fl, rs, tok = state
    st._ag_epoch[H] += 2
    fl[1] += 2
    rs.epoch += 2
    tok.epoch += 4


# --------------------------------------------------------------------------- order of summation
_thread = threading.local()


@contextlib.contextmanager
def inference_pass():
    """The forwards of this thread within it are for their results alone: no later pass with gradients
    has to reproduce their bits. Their products may then be summed in pieces, which is faster with few
    tokens, and how many pieces depends on the number of tokens."""
    before = getattr(_thread, "inference", False)
    _thread.inference = True
    try:
        yield
    finally:
        _thread.inference = before


def may_split(training: bool) -> bool:
    """Whether products may be summed in pieces: in passes declared to be inference (torch's inference
    mode declares it too) of a model in evaluation mode. Other passes without gradients keep the order
    of those with gradients: a checkpoint or a cached-gradient step recomputes what they computed."""
    return (not training and not torch.is_grad_enabled()
            and (getattr(_thread, "inference", False) or torch.is_inference_mode_enabled()))


# --------------------------------------------------------------------------- stream context
def _stream_struct(ctx, plan: BlockPlan, device, training: bool) -> LbStreamCtx:
    """The per-forward struct, cached on the Python stream context (all blocks share it). The
    backward's tile lists are built for a pass that records gradients only."""
    d = plan.desc
    grad = torch.is_grad_enabled()
    split = may_split(training)
    key = ("_lb", grad, split, d.hd, d.Hq // d.Hk, plan.rope[1], id(plan.rope[2]))
    hit = ctx.tables.get(key)
    if hit is not None:
        return hit
    lib = _library()
    cos, sin = ctx.rope(*plan.rope)
    ap = ctx.plan
    G = d.Hq // d.Hk
    ptf, capf, tile = ap.fwd_tiles(d.Hq, d.Hk, d.hd)
    ptq, capq = ap.tiles(128 // G) if grad else (None, 0)
    ptk, capk = ap.tiles(128) if grad else (None, 0)
    s = LbStreamCtx()
    s.T, s.packed = int(ctx.pos.shape[0]), int(ap.cu_seqlens is not None)
    s.cos, s.sin = cos.data_ptr(), sin.data_ptr()
    s.pos, s.pos_i64 = ctx.pos.data_ptr(), int(ctx.pos.dtype == torch.int64)
    s.seq_start, s.seq_end = ap.seq_start.data_ptr(), ap.seq_end.data_ptr()
    s.plan_f, s.cap_f, s.tile_f = ptf.data_ptr(), capf, tile
    s.plan_q, s.cap_q, s.plan_kv, s.cap_kv = nv.ptr(ptq) or None, capq, nv.ptr(ptk) or None, capk
    s.status = nv.status_word(device).data_ptr()
    # partial sums of the backward's norms: the struct's own, as its backward comes later than other
    # callers' passes, which would grow or write a shared buffer
    sums = None
    if grad:
        norm, rope = 2 * lib.lb_norm_bwd_partial_rows() * d.H, lib.lb_rope_bwd_partial_rows() * 2 * d.hd
        sums = torch.empty(norm + rope + 2 * d.hd, dtype=torch.float32, device=device)
        s.norm_scratch = sums.data_ptr()
        s.rope_scratch = sums.data_ptr() + 4 * norm
        s.wg_tmp = sums.data_ptr() + 4 * (norm + rope)
    s.stream = 0
    s.may_split = int(split)
    # what the attention of short sequences is chosen by (0: not known)
    s.n_seq, s.max_len = ap.seq_start.numel(), getattr(ap, "max_seqlen", 0)
    # keep the tensors the struct points to alive as long as the struct
    s._keep = (cos, sin, ctx.pos, ap, ptf, ptq, ptk, sums)
    ctx.tables[key] = s
    return s


# --------------------------------------------------------------------------- autograd node
class _BlockFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, branch, residual, plan, sctx, stream_ctx, *params):
        lib = _library()
        dev = branch.device
        d = plan.fill({})
        T, H = branch.shape
        branch = branch if branch.is_contiguous() else branch.contiguous()
        if residual is not None and not residual.is_contiguous():
            residual = residual.contiguous()
        has_res = residual is not None
        # token-sharded stream: T is this rank's row count and the struct names the group's buffers
        tp, tp_state = _tp_struct(plan.sp, T, H) if plan.sp is not None else (None, None)
        tp_ptr = ctypes.addressof(tp) if tp is not None else None
        nbytes = lib.lb_block_saved_bytes(ctypes.addressof(d), T, int(has_res), tp_ptr)
        saved = torch.empty(_arena_size(nbytes), dtype=torch.uint8, device=dev)
        out = torch.empty(T, H, dtype=branch.dtype, device=dev)
        res_out = torch.empty(T, H, dtype=branch.dtype, device=dev)
        io = LbBlockIO()
        io.tp = tp_ptr
        io.branch, io.residual = branch.data_ptr(), (residual.data_ptr() if has_res else None)
        io.out, io.res_out, io.saved = out.data_ptr(), res_out.data_ptr(), saved.data_ptr()
        sctx.stream = nv.stream_ptr()
        rc = lib.lb_block_fwd(ctypes.addressof(d), ctypes.addressof(sctx), ctypes.addressof(io))
        if rc != 0:
            nv.check_rc(rc, "lb_block_fwd")
        if tp is not None:
            _tp_advance(tp_state)
        calls["tp" if tp is not None else "dp"] += 1
        n = plan._launches.get(("f", sctx.packed))
        if n is None:
            n = lib.lb_block_fwd_launches(ctypes.addressof(d), ctypes.addressof(sctx), int(has_res),
                                          tp_ptr)
            plan._launches[("f", sctx.packed)] = n
        nv.count_launch(n - io.fewer_launches)
        ctx.save_for_backward(branch, residual, saved, res_out)
        ctx.plan, ctx.sctx, ctx.stream_ctx = plan, sctx, stream_ctx
        return out, res_out

    @staticmethod
    def backward(ctx, d_out, d_res_out):
        lib = _library()
        branch, residual, saved, res_out = ctx.saved_tensors
        plan, sctx = ctx.plan, ctx.sctx
        dev = branch.device
        T, H = branch.shape
        if d_out is None:
            d_out = torch.zeros(T, H, dtype=branch.dtype, device=dev)
        d_out = d_out if d_out.is_contiguous() else d_out.contiguous()
        if d_res_out is not None and not d_res_out.is_contiguous():
            d_res_out = d_res_out.contiguous()
        # weight gradients go straight into the sharding runtime's fp32 accumulators; a parameter
        # without one gets a temporary that is returned to autograd
        grads, temps = {}, []
        for p in plan.params:
            if not p.requires_grad:
                temps.append(None)
                continue
            mg = main_grad_of(p)
            if mg is None:
                mg = torch.zeros(p.shape, dtype=torch.float32, device=dev)
                temps.append(mg)
            else:
                temps.append(None)
            grads[id(p)] = mg.data_ptr()
        d = plan.fill(grads)
        tp, tp_state = _tp_struct(plan.sp, T, H) if plan.sp is not None else (None, None)
        tp_ptr = ctypes.addressof(tp) if tp is not None else None
        work = _work_arena(lib.lb_block_work_bytes(ctypes.addressof(d), T, tp_ptr), dev)
        dx = torch.empty(T, H, dtype=branch.dtype, device=dev)
        io = LbBlockIO()
        io.tp = tp_ptr
        io.branch = branch.data_ptr()
        io.residual = residual.data_ptr() if residual is not None else None
        io.res_out, io.saved = res_out.data_ptr(), saved.data_ptr()
        io.d_out = d_out.data_ptr()
        io.d_res_out = d_res_out.data_ptr() if d_res_out is not None else None
        io.dx, io.work = dx.data_ptr(), work.data_ptr()
        sctx.stream = nv.stream_ptr()
        rc = lib.lb_block_bwd(ctypes.addressof(d), ctypes.addressof(sctx), ctypes.addressof(io))
        if rc != 0:
            nv.check_rc(rc, "lb_block_bwd")
        if tp is not None:
            _tp_advance(tp_state)
        key = ("b", sctx.packed, len(grads))
        n = plan._launches.get(key)
        if n is None:
            n = lib.lb_block_bwd_launches(ctypes.addressof(d), ctypes.addressof(sctx), tp_ptr)
            plan._launches[key] = n
        nv.count_launch(n - io.fewer_launches)
        pgrads = tuple(None if t is None else t.to(p.dtype) for t, p in zip(temps, plan.params))
        return (dx, dx if residual is not None else None, None, None, None) + pgrads


def run(block, branch, residual, ctx):
    """``(mlp_out, residual_out)`` of one decoder block, as ``DecoderBlock.forward`` returns them, for
    a block that ``usable`` has just accepted."""
    plan = block.__dict__["_lb_plan"]
    sctx = _stream_struct(ctx, plan, branch.device, block.training)
    return _BlockFn.apply(branch, residual, plan, sctx, ctx, *node_inputs(plan.params))


# --------------------------------------------------------------------------- passes without derivatives
def records_nothing() -> bool:
    """Whether this pass is for its results alone, as torch sees it: no derivatives of any kind, no
    transform, no trace to which a call behind torch's back would be missing."""
    return (not torch.is_grad_enabled() and torch.autograd.forward_ad._current_level < 0
            and torch._C._functorch.peek_interpreter_stack() is None
            and not torch.jit.is_tracing() and not torch.compiler.is_compiling())


def unhooked(d: dict) -> bool:
    """``d``: the ``__dict__`` of a module. Whether calling it runs its class's forward alone."""
    return not ("forward" in d or d["_forward_hooks"] or d["_forward_pre_hooks"]
                or d["_backward_hooks"] or d["_backward_pre_hooks"])


class Watch:
    """Tensors (parameters by module and name) as a descriptor was filled from them; ``same`` looks at
    each of them: at a parameter that was replaced, and at data exchanged under one."""

    def __init__(self, params):
        self.items = []
        for owner, name in params:
            t = owner._parameters[name]
            self.items.append((owner._parameters, name, t, t.data_ptr(), t.dtype, t.shape, t.stride()))

    def same(self) -> bool:
        for where, name, t, ptr, dtype, shape, stride in self.items:
            if (where.get(name) is not t or t.data_ptr() != ptr or t.dtype != dtype
                    or t.shape != shape or t.stride() != stride):
                return False
        return True


class _Inference(Plan):
    """What a pass without derivatives keeps of one block: the descriptor, filled in, and what to look
    at before it is used again. Never changed once made: another thread may be in a pass with it."""

    def __init__(self, block, plan):
        att, mlp = block.self_attn, block.mlp
        qkv = [(att, n) for n in (("qkv_proj",) if att.fused_qkv else ("q_proj", "k_proj", "v_proj"))]
        gu = [(mlp, n) for n in (("gate_up_proj",) if mlp.fused_gate_up else ("gate_proj", "up_proj"))]
        names = qkv + [(att, "o_proj")] + gu + [(mlp, "down_proj")]
        self.modules = [(owner._modules, n, owner._modules[n], owner._modules[n].__dict__)
                        for owner, n in names]
        norms = [block.input_layernorm, block.post_attention_layernorm]
        if plan.qn is not None:
            norms += [att.q_norm, att.k_norm]
        # (a weight may be a buffer, or computed by its module: such a block is called by itself)
        self.ok = (plan.sp is None and all(_plain_linear(m) for _, _, m, _ in self.modules)
                   and all("weight" in m._parameters for m in norms + [m for _, _, m, _ in self.modules]))
        if not self.ok:
            return
        self.halves = (att, mlp, *norms[:2], att._modules.get("q_norm"), att._modules.get("k_norm"))
        self.fused = att.fused_qkv, mlp.fused_gate_up
        self.plan = plan
        self.watch = Watch([(m, "weight") for m in norms] + [(m, "weight") for _, _, m, _ in self.modules])
        d = self.desc = plan.fill({})
        self.addr = ctypes.addressof(d)
        # all that the size of the block's activations and its number of launches follow from
        self.sizes = (d.Hq, d.Hk, d.hd, d.I, d.qk_norm, d.qkv.n, d.gate_up.n)

    def same(self, block) -> bool:
        mods = block._modules
        att, mlp = mods["self_attn"], mods["mlp"]
        am = att._modules
        if (att, mlp, mods["input_layernorm"], mods["post_attention_layernorm"]) != self.halves[:4]:
            return False
        if (am.get("q_norm"), am.get("k_norm")) != self.halves[4:]:
            return False
        if (att.fused_qkv, mlp.fused_gate_up) != self.fused:
            return False
        for where, name, m, d in self.modules:
            if (where.get(name) is not m or "forward" in d or "_tp_kind" in d
                    or d["_parameters"].get("bias") is not None):
                return False
        return self.watch.same()


def _inference_of(block):
    kept = block.__dict__.get("_lb_inference")
    if kept is not None and kept.ok and kept.same(block):
        return kept
    plan = plan_of(block)
    if plan is None:
        return None
    kept = _Inference(block, plan)
    block.__dict__["_lb_inference"] = kept
    return kept if kept.ok else None


def run_inference(block_type, layers, branch, ctx):
    """The blocks of a pass without derivatives, one after the other, with one activation arena and one
    pair of stream buffers for all of them and no autograd node each. Takes the blocks from the first on
    that are plain ones; returns ``(how many, branch, residual)``."""
    if not (records_nothing() and branch.is_cuda and branch.dtype == torch.bfloat16
            and branch.dim() == 2 and branch.is_contiguous() and branch.shape[0] > 0
            and ctx.pos.shape[0] == branch.shape[0]):
        return 0, branch, None
    if _ac._active is not None or _rt.attention_backend == "sdpa" or _has_any_global_hook():
        return 0, branch, None
    for name in ("block_runner", "fused_rmsnorm", "fused_residual_rmsnorm", "fused_qk_norm_rope"):
        if not enabled(name):
            return 0, branch, None
    lib = _library()
    dev = branch.device
    T, H = branch.shape
    io, sctx, key, sizes, out, residual, n, launches = LbBlockIO(), None, None, None, None, None, 0, 0
    io_at = ctypes.addressof(io)
    x = branch
    for block in layers:
        d = block.__dict__
        if type(block) is not block_type or not unhooked(d) or not _own_forwards(block):
            break
        kept = _inference_of(block)
        if kept is None or kept.desc.H != H:
            break
        plan = kept.plan
        k = (plan.desc.hd, plan.desc.Hq // plan.desc.Hk, plan.rope[1], id(plan.rope[2]), d["training"])
        if k != key:
            key = k
            sctx = _stream_struct(ctx, plan, dev, d["training"])
            sctx.stream = nv.stream_ptr()
            sctx_at = ctypes.addressof(sctx)
        if kept.sizes != sizes:
            sizes = kept.sizes
            arena = torch.empty(_arena_size(lib.lb_block_saved_bytes(kept.addr, T, 1, None)),
                                dtype=torch.uint8, device=dev)
            io.saved = arena.data_ptr()
            per_block = lib.lb_block_fwd_launches(kept.addr, sctx_at, 1, None)
        if out is None:
            out, res = torch.empty_like(branch), torch.empty_like(branch)
            io.out, io.res_out = out.data_ptr(), res.data_ptr()
        # (a block has read its inputs before it writes its outputs: from the second one on they are
        # the same buffers)
        io.branch = x.data_ptr()
        io.residual = residual.data_ptr() if residual is not None else None
        io.chained = int(n > 0)
        rc = lib.lb_block_fwd(kept.addr, sctx_at, io_at)
        if rc != 0:
            nv.check_rc(rc, "lb_block_fwd")
        launches += per_block - io.fewer_launches
        x, residual = out, res
        n += 1
    if n:
        nv.count_launch(launches)
        calls["dp"] += n
    return n, x, residual
