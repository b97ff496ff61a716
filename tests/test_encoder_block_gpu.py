"""The native encoder-block runner against the op-by-op path of the same blocks."""
import pytest
import torch

from lset_b200.dist.sharded import ParamStore
from lset_b200.models.bert import BertEncoder
from lset_b200.models.configs import BertConfig
from lset_b200.ops import _native as nv
from lset_b200.ops import encoder_block as enc_ops
from lset_b200.ops.runtime_options import configure

pytestmark = pytest.mark.gpu


def _model(H, heads, I, fused, layers=2):
    torch.manual_seed(3)
    model = BertEncoder(BertConfig(vocab_size=512, hidden_size=H, intermediate_size=I,
                                   num_hidden_layers=layers, num_attention_heads=heads,
                                   max_position_embeddings=2048), fused_projections=fused)
    for n, p in model.named_parameters():
        if p.dim() > 1 or n.endswith("bias"):
            torch.nn.init.normal_(p, std=0.05)
    return model.cuda().to(torch.bfloat16)


def _inputs(lens, padded):
    g = torch.Generator().manual_seed(1)
    if padded:
        S = max(lens)
        mask = torch.zeros(len(lens), S, dtype=torch.long)
        for i, n in enumerate(lens):
            mask[i, :n] = 1
        return dict(input_ids=torch.randint(0, 512, (len(lens), S), generator=g).cuda(),
                    attention_mask=mask.cuda())
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32).cuda()
    pos = torch.cat([torch.arange(n) for n in lens]).cuda()
    return dict(input_ids=torch.randint(0, 512, (sum(lens),), generator=g).cuda(),
                position_ids=pos, cu_seqlens=cu, max_seqlen=max(lens))


def _run(model, inputs, on, backward=True):
    configure(block_runner=on)
    try:
        for p in model.parameters():
            p.grad = None
        out = model(**inputs)["hidden_states"]
        mask = inputs.get("attention_mask")
        out = out if mask is None else out * mask[..., None].to(out.dtype)
        if backward:
            torch.manual_seed(9)
            (out.float() * torch.randn(out.shape, device="cuda")).sum().backward()
        nv.check_status()
        return out.detach()
    finally:
        configure(block_runner=True)


@pytest.mark.parametrize("H,heads,I", [(128, 2, 256), (768, 12, 3072), (256, 2, 520)])
@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("lens,padded", [([1, 33, 128, 64, 5], False), ([300, 700, 2000, 1500], False),
                                         ([40, 7, 129], True)])
def test_runner_matches_the_op_path(H, heads, I, fused, lens, padded):
    model, inputs = _model(H, heads, I, fused), _inputs(lens, padded)
    before = enc_ops.calls
    got = _run(model, inputs, True)
    assert enc_ops.calls == before + len(model.layers)
    grads = {n: p.grad.clone() for n, p in model.named_parameters()}
    want = _run(model, inputs, False)
    assert torch.equal(got, want)
    for n, p in model.named_parameters():
        # sums of a few bf16 terms in another order, through two blocks. A key bias moves all of a
        # row's scores alike: its gradient is zero but for the rounding of the terms, which are of
        # the size of the value bias's.
        a, b = grads[n].float(), p.grad.float()
        size = dict(model.named_parameters())[n.replace("key.bias", "value.bias")].grad.float()
        assert (a - b).norm().item() < 2e-2 * size.norm().item(), n
    with torch.no_grad():        # contractions may be split then: another order of summation
        model.eval()
        assert torch.allclose(_run(model, inputs, True, False).float(), want.float(), atol=6e-2)


def test_runner_adds_to_main_grads_and_skips_frozen_parameters():
    model = _model(128, 2, 256, False)
    model.layers[0].attention.dense.weight.requires_grad_(False)
    model.layers[1].mlp.LayerNorm.bias.requires_grad_(False)
    store = ParamStore(model, device=torch.device("cuda"))
    inputs = _inputs([20, 70, 9], False)
    flats = []
    for on in (True, False):
        store.zero_grad()
        _run(model, inputs, on)
        store.finish_backward()
        flats.append([g.flat_grad.clone() for g in store.groups])
    assert model.layers[0].attention.dense.weight.grad is None
    for a, b in zip(*flats):
        assert (a - b).norm().item() < 2e-2 * b.norm().item() + 1e-6


@pytest.mark.parametrize("trained", ["embeddings", "norms", "attention.dense.", "layers.0.", "query",
                                     "mlp.dense_in", "mlp.dense_out"])
@pytest.mark.parametrize("T", [300, 700])
def test_gradients_below_frozen_parameters(T, trained):
    """Which launches follow each other in the backward depends on what trains: with the linears
    frozen the activation's gradient comes right behind the GEMM that writes its input, which at
    these sizes lets the next launch start early. Same bounds as above; every pass the same."""
    model, inputs = _model(768, 12, 3072, False), _inputs([T // 3, T - T // 3], False)
    for n, p in model.named_parameters():
        p.requires_grad_(trained in n or (trained == "norms" and "LayerNorm" in n))
    grads = []
    for on in (True, True, True, False):
        _run(model, inputs, on)
        grads.append({n: p.grad.float() for n, p in model.named_parameters() if p.requires_grad})
    assert grads[0]
    for n, want in grads[-1].items():
        # (the key bias has no gradient but rounding, see above)
        size = grads[-1].get(n.replace("key.bias", "value.bias"), want).norm().item()
        for got in grads[:-1]:
            assert (got[n] - want).norm().item() < 2e-2 * size, n


def test_copy_of_a_model_that_has_run():
    import copy

    model, inputs = _model(128, 2, 256, False), _inputs([20, 9], False)
    want = _run(model, inputs, True)
    before = enc_ops.calls
    assert torch.equal(_run(copy.deepcopy(model), inputs, True), want)
    assert enc_ops.calls == before + len(model.layers)


def test_eval_passes_with_and_without_gradients_have_the_same_bits():
    model, inputs = _model(768, 12, 3072, False).eval(), _inputs([9, 20, 3], False)
    with torch.no_grad():
        first = model(**inputs)["hidden_states"]
    assert torch.equal(first, model(**inputs)["hidden_states"])
    nv.check_status()


def test_passes_of_models_of_different_width_interleaved(monkeypatch):
    """The wider model's pass, between the narrower one's two, asks for larger buffers."""
    from lset_b200.ops import norm

    models = [_model(128, 2, 256, False), _model(768, 12, 3072, False)]
    inputs = _inputs([20, 70, 9], False)
    want = []
    for m in models:
        _run(m, inputs, True)
        want.append({n: p.grad for n, p in m.named_parameters()})
        for p in m.parameters():
            p.grad = None
    monkeypatch.setattr(norm, "_scratch", {})
    outs = [m(**inputs)["hidden_states"] for m in models]
    held = [torch.full((1 << k,), 3.0, device="cuda") for k in range(8, 22) for _ in range(4)]
    for m, out in zip(models, outs):
        torch.manual_seed(9)
        (out.float() * torch.randn(out.shape, device="cuda")).sum().backward()
    nv.check_status()
    assert all((t == 3.0).all() for t in held)      # nobody else's memory was written
    for m, grads in zip(models, want):
        for n, p in m.named_parameters():
            size = grads[n.replace("key.bias", "value.bias")].float().norm().item()
            assert (p.grad.float() - grads[n].float()).norm().item() < 2e-2 * size, n


def test_hooked_or_replaced_submodules_keep_the_op_path():
    model, inputs = _model(128, 2, 256, False), _inputs([20, 9], False)
    seen = []
    model.layers[0].mlp.register_forward_hook(lambda *a: seen.append(1))
    model.layers[1].attention.dense = torch.nn.Linear(128, 128).cuda().to(torch.bfloat16)
    before = enc_ops.calls
    _run(model, inputs, True)
    assert enc_ops.calls == before and seen


def test_data_exchanged_under_the_same_parameter():
    """Other storage, another eps: what the runner has looked at once is looked at again."""
    model, inputs = _model(128, 2, 256, False), _inputs([20, 9], False)
    _run(model, inputs, True)
    before = enc_ops.calls
    layers = model.layers
    w = layers[0].mlp.dense_in.weight
    w.data = w.data.t().contiguous().t()               # same values, column by column in memory
    got = _run(model, inputs, True)
    assert enc_ops.calls == before + len(layers) - 1   # that block goes op by op
    assert torch.allclose(got.float(), _run(model, inputs, False).float(), atol=6e-2)
    w.data = w.data.contiguous()
    for layer in layers:
        layer.attention.LayerNorm.eps = layer.mlp.LayerNorm.eps = 0.5
    before = enc_ops.calls
    got = _run(model, inputs, True)
    assert enc_ops.calls == before + len(layers)
    assert torch.allclose(got.float(), _run(model, inputs, False).float(), atol=6e-2)


@pytest.mark.parametrize("name", ["attention.query", "mlp.dense_out", "attention.LayerNorm"])
def test_weights_changed_in_place_before_the_backward_are_refused(name):
    """The backward reads the weights of the forward: autograd refuses others, as op by op."""
    model, inputs = _model(128, 2, 256, False), _inputs([20, 9], False)
    for on in (True, False):
        configure(block_runner=on)
        try:
            out = model(**inputs)["hidden_states"]
            with torch.no_grad():
                model.layers[1].get_submodule(name).weight.mul_(2)
            with pytest.raises(RuntimeError, match="modified by an inplace operation"):
                out.float().sum().backward()
        finally:
            configure(block_runner=True)


@pytest.mark.parametrize("T,parts", [(1, (64, 0, 0)), (700, (768, 768, 768)), (5000, (72, 0, 0))])
def test_bias_grad(T, parts):
    import ctypes

    N = sum(parts)
    dy = torch.randn(T, N, device="cuda").to(torch.bfloat16)
    outs = [torch.full((n,), 2.0, device="cuda") for n in parts]
    vp = ctypes.c_void_p
    rc = nv.load().lb_bias_grad(vp(dy.data_ptr()), ctypes.c_longlong(N), T, *parts,
                                *[vp(o.data_ptr() if o.numel() else 0) for o in outs],
                                vp(nv.stream_ptr()))
    assert rc == 0
    ref = dy.double().sum(0) + 2
    # fp32 sums of T terms
    assert (torch.cat(outs).double() - ref).abs().max().item() < T * 2 ** -23 * 8


@pytest.mark.parametrize("T", [4096, 4097, 8191, 20000])
def test_bias_grad_sums_in_a_fixed_order(T):
    """Pass after pass the same bits, from one chunk of rows to a cluster of eight."""
    import ctypes

    N = 776
    dy = torch.randn(T, N, device="cuda").to(torch.bfloat16)
    vp, outs = ctypes.c_void_p, []
    for _ in range(20):
        out = torch.zeros(N, device="cuda")
        assert nv.load().lb_bias_grad(vp(dy.data_ptr()), ctypes.c_longlong(N), T, N, 0, 0,
                                      vp(out.data_ptr()), vp(0), vp(0), vp(nv.stream_ptr())) == 0
        outs.append(out)
    assert all(torch.equal(o, outs[0]) for o in outs)
    assert (outs[0].double() - dy.double().sum(0)).abs().max().item() < T * 2 ** -23 * 8


def test_norms_that_share_weights_both_add_to_their_gradients():
    model, inputs = _model(128, 2, 256, False), _inputs([9, 20, 3], False)
    for layer in model.layers:
        first, second = layer.attention.LayerNorm, layer.mlp.LayerNorm
        second.weight, second.bias = first.weight, first.bias
    _run(model, inputs, False)
    want = {n: p.grad.float() for n, p in model.named_parameters()}
    before = enc_ops.calls
    _run(model, inputs, True)
    assert enc_ops.calls == before + len(model.layers)
    for n, p in model.named_parameters():
        size = want[n.replace("key.bias", "value.bias")].norm().item()
        assert (p.grad.float() - want[n]).norm().item() < 2e-2 * size, n
