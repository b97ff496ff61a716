"""Host side of the block runners: what their structs point to, and which blocks they take."""
import copy
import ctypes
import pickle
from types import SimpleNamespace

import pytest
import torch

from lset_b200.ops import block as dec_ops
from lset_b200.ops import encoder_block as enc_ops

LIB = SimpleNamespace(lb_norm_bwd_partial_rows=lambda: 8, lb_rope_bwd_partial_rows=lambda: 8)


class Plan:
    """Stands for an ``AttnPlan``, whose tile lists are made on the device."""

    cu_seqlens = seq_start = seq_end = torch.zeros(2, dtype=torch.int32)

    def tiles(self, tokens):
        return torch.zeros(8, dtype=torch.int32), 2

    def fwd_tiles(self, heads, kv_heads, head_dim):
        return (*self.tiles(128), 128)


def _stream_struct(ops, monkeypatch, training=True):
    monkeypatch.setattr(ops, "_library", lambda: LIB)
    word = torch.zeros(1, dtype=torch.int32)
    monkeypatch.setattr(ops.nv, "status_word", lambda device=None: word)
    table = torch.zeros(4, 4)
    ctx = SimpleNamespace(plan=Plan(), pos=torch.zeros(5, dtype=torch.int64), tables={},
                          rope=lambda *a: (table, table))
    plan = SimpleNamespace(desc=SimpleNamespace(H=16, hd=64, heads=2, Hq=2, Hk=1), rope=(64, 1e4, None))
    return ops._stream_struct(ctx, plan, torch.device("cpu"), training)


@pytest.mark.parametrize("ops", [enc_ops, dec_ops])
def test_stream_struct_owns_the_buffers_of_the_backward(ops, monkeypatch):
    """The backward comes later than other callers' passes: a buffer that one of them may replace
    or write is not what the struct can point to."""
    structs = [_stream_struct(ops, monkeypatch) for _ in range(2)]
    # (partial rows of two norms, each of a weight and, in an encoder, a bias)
    sizes = ([("norm_scratch", 2 * 8 * 2 * 16)] if ops is enc_ops else
             [("norm_scratch", 2 * 8 * 16), ("rope_scratch", 8 * 2 * 64), ("wg_tmp", 2 * 64)])
    taken = []
    for s in structs:
        for name, n in sizes:
            a = ctypes.cast(getattr(s, name), ctypes.c_void_p).value
            assert any(torch.is_tensor(t) and t.data_ptr() <= a
                       and a + 4 * n <= t.data_ptr() + t.nbytes for t in s._keep), name
            assert all(a + 4 * n <= lo or hi <= a for lo, hi in taken), name
            taken.append((a, a + 4 * n))
    with torch.no_grad():
        assert not _stream_struct(ops, monkeypatch).norm_scratch


@pytest.mark.parametrize("ops", [enc_ops, dec_ops])
def test_only_passes_declared_to_be_inference_are_summed_in_pieces(ops, monkeypatch):
    """What a checkpoint or a cached-gradient step computes without gradients is recomputed with them,
    in evaluation mode too: the same order of summation."""
    def splits(training):
        return bool(_stream_struct(ops, monkeypatch, training).may_split)

    with torch.no_grad():
        assert not splits(False) and not splits(True)
        with dec_ops.inference_pass():
            assert splits(False) and not splits(True)
            with dec_ops.inference_pass():
                pass
            assert splits(False)
        assert not splits(False)
    with torch.inference_mode():
        assert splits(False) and not splits(True)
    with dec_ops.inference_pass():
        assert not splits(False)          # gradients are recorded


class _Accepted(RuntimeError):
    pass


@pytest.fixture
def decide(monkeypatch):
    """``usable`` on the CPU: everything but the device is real."""
    def plan_of(block):
        raise _Accepted

    def call(ops, block, ctx):
        monkeypatch.setattr(ops, "plan_of", plan_of)
        x = SimpleNamespace(is_cuda=True, dtype=torch.bfloat16, shape=(5, 128), dim=lambda: 2)
        try:
            assert ops.usable(block, x, ctx) is False
            return False
        except _Accepted:      # everything that is looked at before the plan is accepted
            return True
    return call


def _bert_block():
    from lset_b200.models.bert import BertBlock
    from lset_b200.models.configs import BertConfig

    return BertBlock(BertConfig(vocab_size=8, hidden_size=128, intermediate_size=256,
                                num_hidden_layers=1, num_attention_heads=2))


def _subclass(m):
    m.__class__ = type("Own", (type(m),), {"forward": lambda self, x, *a: x})


def _patched(m):
    m.forward = lambda x, *a: x


def _hooked(m):
    m.register_forward_hook(lambda *a: None)


def _decoder_block():
    from lset_b200.models import Qwen3Config
    from lset_b200.models.decoder import Qwen3Decoder

    return Qwen3Decoder(Qwen3Config(vocab_size=8, hidden_size=128, intermediate_size=256,
                                    num_hidden_layers=1, num_attention_heads=2,
                                    num_key_value_heads=1, head_dim=64)).layers[0]


@pytest.mark.parametrize("half", ["self_attn", "mlp"])
@pytest.mark.parametrize("change", [_subclass, _patched])
def test_decoder_blocks_with_a_forward_of_their_own_are_not_taken(decide, half, change):
    block = _decoder_block()
    assert decide(dec_ops, block, None)
    change(getattr(block, half))
    assert not decide(dec_ops, block, None)


@pytest.mark.parametrize("half", ["attention", "mlp"])
@pytest.mark.parametrize("change", [_subclass, _patched, _hooked])
def test_encoder_blocks_with_a_forward_of_their_own_are_not_taken(decide, half, change):
    block = _bert_block()
    assert decide(enc_ops, block, None)
    change(getattr(block, half))
    assert not decide(enc_ops, block, None)


def test_encoder_block_with_another_mlp_or_under_a_global_hook_is_not_taken(decide):
    block = _bert_block()
    handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    try:
        assert not decide(enc_ops, block, None)
    finally:
        handle.remove()
    assert decide(enc_ops, block, None)
    block.mlp = torch.nn.Linear(128, 128)      # no dense_in
    assert not decide(enc_ops, block, None)


@pytest.mark.parametrize("make,plan,name", [(_bert_block, enc_ops.EncoderPlan, "dense_in"),
                                            (_decoder_block, dec_ops.BlockPlan, "down_proj")])
def test_signature_sees_a_linear_that_became_another_class(make, plan, name):
    block = make()
    before = plan._signature(block)
    assert plan._signature(block) == before
    _subclass(getattr(block.mlp, name))        # as the 8-bit conversion does
    assert plan._signature(block) != before


def _encoder_plan():
    block, plan = _bert_block(), enc_ops.EncoderPlan.__new__(enc_ops.EncoderPlan)
    qkv, o, fin, fout, ln1, ln2 = enc_ops._modules(block)
    plan.desc = enc_ops.LbEncoderDesc()
    plan.linears = list(enumerate(qkv + [o, fin, fout]))
    plan.norms = [(ln1, "ln1"), (ln2, "ln2")]
    return plan, fout.weight, lambda d: d.out


def _decoder_plan():
    block, plan = _decoder_block(), dec_ops.BlockPlan.__new__(dec_ops.BlockPlan)
    plan.desc = dec_ops.LbBlockDesc()
    plan.ln1, plan.ln2, plan.qn, plan.kn = block.input_layernorm, block.input_layernorm, None, None
    parts = [(m.weight, None, None, 0.0) for m in (block.self_attn.q_proj, block.self_attn.o_proj,
                                                   block.mlp.up_proj, block.mlp.down_proj)]
    plan.qkv, plan.o, plan.gate_up, plan.down = parts[:1], parts[1], parts[2:3], parts[3]
    return plan, block.mlp.down_proj.weight, lambda d: d.down


@pytest.mark.parametrize("make", [_encoder_plan, _decoder_plan])
def test_every_call_has_a_descriptor_of_its_own(make):
    """A forward in one thread does not clear the gradient addresses that another thread's backward
    has just filled in."""
    plan, w, linear = make()
    backward = plan.fill({id(w): 4096})
    forward = plan.fill({})
    assert linear(backward).wgrad and not linear(forward).wgrad
    assert ctypes.cast(linear(backward).wgrad, ctypes.c_void_p).value == 4096
    assert linear(backward).w == linear(forward).w == w.data_ptr()
    assert not linear(plan.desc).w


def test_backward_passes_that_overlap_do_not_share_their_temporary_storage():
    a, b = (dec_ops._work_arena(3 << 20, torch.device("cpu")) for _ in range(2))
    assert a.numel() >= 3 << 20
    assert a.data_ptr() + a.numel() <= b.data_ptr() or b.data_ptr() + b.numel() <= a.data_ptr()


@pytest.mark.parametrize("make,plan", [(_bert_block, _encoder_plan), (_decoder_block, _decoder_plan)])
@pytest.mark.parametrize("copied", [copy.deepcopy, lambda m: pickle.loads(pickle.dumps(m))])
def test_a_block_that_has_run_can_be_copied_and_pickled(make, plan, copied):
    block = make()
    block.__dict__["_lb_plan"] = plan()[0]      # as after a pass on the GPU
    other = copied(block)
    assert other.__dict__["_lb_plan"] is None
    for a, b in zip(block.parameters(), other.parameters()):
        assert torch.equal(a, b)


class _OnDevice(torch.Tensor):
    is_cuda = True


def _qwen(norms):
    d = dec_ops.LbBlockDesc()
    d.H, d.Hq, d.Hk, d.hd, d.I, d.qk_norm = 128, 2, 1, 64, 256, norms
    return d


def _bert(heads):
    d = enc_ops.LbEncoderDesc()
    d.H, d.heads, d.hd, d.I = 128, heads, 128 // heads, 256
    return d


@pytest.mark.parametrize("ops,descs", [(dec_ops, [_qwen(0), _qwen(1), _qwen(0)]), (enc_ops, [_bert(1), _bert(2)])])
def test_every_block_of_an_inference_pass_has_room_for_its_activations(ops, descs, monkeypatch):
    """Blocks of a stack need not be alike: q/k norms and heads have statistics of their own in the arena."""
    desc_type, arenas, fits = type(descs[0]), [], []

    def need(addr, T, *_):
        d = desc_type.from_address(addr)
        return T * (d.heads if ops is enc_ops else 8 + d.qk_norm * (d.Hq + d.Hk)) * 4

    def forward(addr, sctx, io):
        at = dec_ops.LbBlockIO.from_address(io).saved
        fits.append(any(a.data_ptr() == at and need(addr, 5) <= a.numel() for a in arenas))
        return 0

    def arena(n, *a, **kw):
        arenas.append(torch.zeros(n, dtype=torch.uint8))
        return arenas[-1]

    name = "lb_encoder" if ops is enc_ops else "lb_block"
    lib = SimpleNamespace(lb_block_fwd_launches=lambda *a: 1,
                          **{name + "_saved_bytes": need, name + "_fwd": forward})
    kept = []
    for d in descs:     # as a pass fills them in
        monkeypatch.setattr(ops, "Watch", lambda params: None)
        monkeypatch.setattr(ops, "_plain_linear", lambda m: True, raising=False)
        plan = SimpleNamespace(fill=lambda grads, d=d: d, desc=d, rope=(64, 1e4, None), sp=None, qn=None)
        kept.append(ops._Inference(_bert_block() if ops is enc_ops else _decoder_block(), plan))
    blocks = torch.nn.ModuleList(torch.nn.Identity() for _ in descs)
    monkeypatch.setattr(ops, "_library", lambda: lib)
    monkeypatch.setattr(ops, "_own_forwards", lambda block: True)
    monkeypatch.setattr(ops, "_inference_of", lambda block: kept[list(blocks).index(block)])
    monkeypatch.setattr(ops, "_stream_struct", lambda *a: dec_ops.LbStreamCtx())
    monkeypatch.setattr(ops.nv, "stream_ptr", lambda: 0)
    monkeypatch.setattr(ops, "torch", SimpleNamespace(**{**vars(torch), "empty": arena}))
    x = torch.zeros(5, 128, dtype=torch.bfloat16).as_subclass(_OnDevice)
    with torch.no_grad():
        done, *_ = ops.run_inference(torch.nn.Identity, blocks, x, SimpleNamespace(pos=torch.zeros(5)))
    assert done == len(descs) and fits == [True] * len(descs)


def _decoder_inference(block, monkeypatch):
    monkeypatch.setattr(dec_ops, "_plain_linear", lambda m: True)
    plan = SimpleNamespace(fill=lambda grads: _qwen(0), desc=_qwen(0), rope=(64, 1e4, None), sp=None, qn=None)
    return dec_ops._Inference(block, plan)


@pytest.mark.parametrize("name", ["mlp.down_proj", "input_layernorm"])
def test_a_block_with_a_weight_that_is_no_parameter_is_called_by_itself(name, monkeypatch):
    block = _decoder_block()
    assert _decoder_inference(block, monkeypatch).ok
    m = block.get_submodule(name)
    w = m.weight.detach()
    del m.weight
    m.register_buffer("weight", w)
    assert not _decoder_inference(block, monkeypatch).ok


def test_what_is_kept_of_a_block_sees_a_projection_that_is_gone(monkeypatch):
    block = _decoder_block()
    kept = _decoder_inference(block, monkeypatch)
    assert kept.same(block)
    block.self_attn.fused_qkv = True
    assert not kept.same(block)
    block.self_attn.fused_qkv = False
    del block.self_attn.q_proj
    assert not kept.same(block)
