"""Varlen attention kernels against the fp32 eager oracle (ragged sequences, GQA, both masks)."""
import pytest
import torch

from lset_b200.ops import _native as nv
from lset_b200.ops.attention import AttnPlan, attention_ref, varlen_attention

pytestmark = pytest.mark.gpu


def _make(lens, Hq, Hk, hd, fused=False, seed=0):
    torch.manual_seed(seed)
    T = sum(lens)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")
    if fused:
        qkv = torch.randn(T, Hq + 2 * Hk, hd, device="cuda").to(torch.bfloat16)
        q, k, v = qkv[:, :Hq], qkv[:, Hq:Hq + Hk], qkv[:, Hq + Hk:]
    else:
        q = torch.randn(T, Hq, hd, device="cuda").to(torch.bfloat16)
        k = torch.randn(T, Hk, hd, device="cuda").to(torch.bfloat16)
        v = torch.randn(T, Hk, hd, device="cuda").to(torch.bfloat16)
    return q, k, v, cu, AttnPlan(cu, max(lens), T)


CASES = [
    ([64], 2, 2, 128), ([128], 2, 1, 128), ([17, 200, 64, 333], 4, 2, 128),
    ([40, 512, 129, 1], 16, 8, 128), ([300, 77], 8, 2, 128), ([250, 31], 8, 1, 128),
    ([100, 260], 4, 4, 64), ([90, 130], 2, 1, 256),
]


@pytest.mark.parametrize("lens,Hq,Hk,hd", CASES)
@pytest.mark.parametrize("causal", [True, False])
def test_forward(lens, Hq, Hk, hd, causal):
    q, k, v, cu, plan = _make(lens, Hq, Hk, hd)
    o = varlen_attention(q, k, v, plan, causal)
    nv.check_status()
    ref = attention_ref(q.float(), k.float(), v.float(), cu, causal)
    err = (o.float() - ref).abs().max().item()
    assert err < 3e-2, err


def test_forward_fused_qkv_views():
    q, k, v, cu, plan = _make([70, 190, 33], 16, 8, 128, fused=True)
    o = varlen_attention(q, k, v, plan, True)
    nv.check_status()
    ref = attention_ref(q.float(), k.float(), v.float(), cu, True)
    assert (o.float() - ref).abs().max().item() < 3e-2


@pytest.mark.parametrize("lens,Hq,Hk,hd", CASES)
@pytest.mark.parametrize("causal", [True, False])
def test_backward(lens, Hq, Hk, hd, causal):
    q, k, v, cu, plan = _make(lens, Hq, Hk, hd, seed=1)
    q.requires_grad_(); k.requires_grad_(); v.requires_grad_()
    o = varlen_attention(q, k, v, plan, causal)
    g = torch.randn_like(o)
    o.backward(g)
    nv.check_status()
    qr, kr, vr = (t.detach().float().requires_grad_() for t in (q, k, v))
    ref = attention_ref(qr, kr, vr, cu, causal)
    ref.backward(g.float())
    for name, a, b in (("dq", q.grad, qr.grad), ("dk", k.grad, kr.grad), ("dv", v.grad, vr.grad)):
        err = (a.float() - b).abs().max().item()
        scale = b.abs().max().item() + 1e-6
        assert err / scale < 3e-2, (name, err, scale)


@pytest.mark.parametrize("left", [True, False])
def test_padded_plan(left):
    torch.manual_seed(3)
    B, S, Hq, Hk, hd = 3, 96, 4, 2, 128
    lens = [96, 40, 7]
    mask = torch.zeros(B, S, dtype=torch.long, device="cuda")
    for b, L in enumerate(lens):
        if left:
            mask[b, S - L:] = 1
        else:
            mask[b, :L] = 1
    plan = AttnPlan.from_mask(mask)
    q = torch.randn(B * S, Hq, hd, device="cuda").to(torch.bfloat16)
    k = torch.randn(B * S, Hk, hd, device="cuda").to(torch.bfloat16)
    v = torch.randn(B * S, Hk, hd, device="cuda").to(torch.bfloat16)
    o = varlen_attention(q, k, v, plan, True)
    nv.check_status()
    ref = attention_ref(q.float(), k.float(), v.float(), plan.seq_start, True, seq_end=plan.seq_end)
    assert (o.float() - ref).abs().max().item() < 3e-2


def test_stream_padded_past_the_last_sequence():
    """A packed stream padded to a fixed token budget: the tokens behind the last sequence belong
    to no sequence. Their output and gradient rows are cleared (no kernel writes them), and what
    they hold on input does not reach the rows of real tokens."""
    lens, pad = [70, 190, 33], 150
    Hq, Hk, hd = 8, 4, 128
    q, k, v, cu, plan = _make(lens, Hq, Hk, hd, seed=5)
    T = sum(lens)
    big = lambda h: (torch.randn(pad, h, hd, device="cuda") * 50).to(torch.bfloat16)  # noqa: E731
    qp, kp, vp = (torch.cat([t, big(t.shape[1])]).requires_grad_() for t in (q, k, v))
    plan_p = AttnPlan(cu, max(lens), T + pad)
    q.requires_grad_(); k.requires_grad_(); v.requires_grad_()
    o = varlen_attention(q, k, v, plan, True)
    g = torch.randn_like(o)
    o.backward(g)
    # poison the allocator's free blocks so that "never written" shows up as garbage
    junk = torch.full((T + pad, Hq, hd), float("nan"), device="cuda", dtype=torch.bfloat16)
    del junk
    op = varlen_attention(qp, kp, vp, plan_p, True)
    op.backward(torch.cat([g, torch.zeros(pad, Hq, hd, device="cuda", dtype=g.dtype)]))
    nv.check_status()
    assert torch.equal(op[:T], o) and not op[T:].any()
    for a, b in ((qp.grad, q.grad), (kp.grad, k.grad), (vp.grad, v.grad)):
        assert torch.equal(a[:T], b) and not a[T:].any()


@pytest.mark.parametrize("Hq,Hk,hd", [(2, 2, 128), (4, 2, 128), (8, 2, 64), (8, 1, 128), (3, 3, 64)])
@pytest.mark.parametrize("causal", [True, False])
@pytest.mark.parametrize("scale", [None, -0.2, 0.0])
def test_forward_tile_edges(Hq, Hk, hd, causal, scale):
    """Sequences that end on, before and behind the edges of the two-tile kernel: its 32-column
    chunks, 128-token KV blocks and query tiles of 128 / G tokens, one tile or two; long ones whose
    running maximum keeps moving; a scale that is not positive.

    Output and LSE are fp32 sums over bf16 probabilities rounded once (2^-9) and bf16 outputs
    (2^-9): 2^-8 of a value, against the 2-norm of the result."""
    G = Hq // Hk
    qt = 128 // G
    lens = [1, qt - 1, qt, qt + 1, 2 * qt, 2 * qt + 1, 31, 33, 127, 128, 129, 257, 640]
    q, k, v, cu, plan = _make(lens, Hq, Hk, hd, seed=1)
    k = (k.float() * torch.linspace(0.2, 4, k.shape[0], device="cuda")[:, None, None]).to(k.dtype)
    o = varlen_attention(q, k, v, plan, causal, scale)
    nv.check_status()
    ref = attention_ref(q.float(), k.float(), v.float(), cu, causal, scale)
    assert ((o.float() - ref).norm() / ref.norm()).item() < 2 ** -8
    again = varlen_attention(q, k, v, plan, causal, scale)   # the work counter was put back
    assert torch.equal(o, again)


def test_padded_plan_clears_the_gradient_rows_of_padding():
    """Rows of a padded batch that belong to no sequence get zero gradients, not what the buffers
    held before: the projections sum over all rows."""
    B, S, H, hd = 3, 96, 2, 64
    mask = torch.zeros(B, S, dtype=torch.long, device="cuda")
    for i, n in enumerate((40, 7, 96)):
        mask[i, :n] = 1
    plan = AttnPlan.from_mask(mask)
    q, k, v = (torch.randn(B * S, H, hd, device="cuda").to(torch.bfloat16).requires_grad_()
               for _ in range(3))
    o = varlen_attention(q, k, v, plan, False)
    junk = [torch.full((B * S, H, hd), float("nan"), device="cuda", dtype=torch.bfloat16)
            for _ in range(8)]
    del junk
    o.backward(torch.randn_like(o))
    nv.check_status()
    pad = mask.reshape(-1) == 0
    for t in (q, k, v):
        assert not t.grad[pad].any() and t.grad[~pad].abs().max() > 0


@pytest.mark.parametrize("Hq,Hk,hd", [(2, 2, 128), (4, 2, 128), (8, 2, 64), (8, 1, 128), (3, 3, 64)])
@pytest.mark.parametrize("causal", [True, False])
def test_forward_of_the_one_tile_kernel(Hq, Hk, hd, causal, monkeypatch):
    """The kernel that short sequences take, on the sequences and with the bound of
    ``test_forward_tile_edges``, and on a stream with rows behind the last sequence."""
    test_forward_tile_edges(Hq, Hk, hd, causal, -0.2)
    monkeypatch.setattr(AttnPlan, "_one_tile", lambda *a: True)
    test_forward_tile_edges(Hq, Hk, hd, causal, None)
    test_forward_tile_edges(Hq, Hk, hd, causal, -0.2)
    test_stream_padded_past_the_last_sequence()


def test_short_sequences_take_the_one_tile_kernel():
    def tile(n, length, Hq, Hk, hd, longest=0):
        cu = torch.arange(n + 1, dtype=torch.int32, device="cuda") * length
        return AttnPlan(cu, longest or length, n * length).fwd_tiles(Hq, Hk, hd)[2]

    assert tile(256, 30, 12, 12, 64) == 128 and tile(256, 64, 12, 12, 64) == 128
    assert tile(256, 65, 12, 12, 64) == 256
    assert tile(256, 64, 16, 8, 128) == 64 and tile(256, 65, 16, 8, 128) == 128
    assert tile(256, 57, 16, 8, 128, 90) == 64 and tile(256, 58, 16, 8, 128, 90) == 128
    assert tile(256, 128, 16, 16, 128) == 128
    assert tile(1, 30, 16, 8, 128) == 128          # fewer sequences than SMs
    assert tile(256, 300, 4, 4, 256) == 128


@pytest.mark.parametrize("Hq,Hk,hd", [(4, 2, 128), (3, 3, 64)])
@pytest.mark.parametrize("one_tile", [False, True])
@pytest.mark.parametrize("spans", [[(0, 40), (50, 96), (0, 0), (90, 96)], [(0, 0), (0, 0), (3, 96)],
                                   [(0, 96), (0, 96)], [(0, 96), (0, 7), (0, 0), (0, 0)], [(0, 0)]])
def test_kernels_clear_the_rows_of_no_sequence(Hq, Hk, hd, one_tile, spans, monkeypatch):
    """Padding left, right and between, rows without a token first, last and next to each other: the
    kernels write every row of buffers that hold garbage, zeros where there is no sequence."""
    from lset_b200.ops.attention import _native_bwd, _native_fwd

    if one_tile:
        monkeypatch.setattr(AttnPlan, "_one_tile", lambda *a: True)
    torch.manual_seed(0)
    S, scale = 96, hd ** -0.5
    mask = torch.zeros(len(spans), S, dtype=torch.long, device="cuda")
    for row, (a, b) in zip(mask, spans):
        row[a:b] = 1
    T, live = mask.numel(), mask.reshape(-1) > 0
    plan = AttnPlan.from_mask(mask)
    q, k, v, do = (torch.randn(T, h, hd, device="cuda").to(torch.bfloat16) for h in (Hq, Hk, Hk, Hq))
    want, _ = _native_fwd(q, k, v, plan, True, scale)      # into zeros
    nan = lambda t, *a, **kw: torch.full_like(t, float("nan"))  # noqa: E731
    monkeypatch.setattr(torch, "zeros", lambda *s, **kw: torch.full(s, float("nan"), **kw))
    o, lse = _native_fwd(q, k, v, plan, True, scale)
    monkeypatch.undo()
    assert torch.equal(o, want) and not o[~live].any()
    grads = [[f(t) for t in (q, k, v)] for f in (torch.zeros_like, nan)]
    for g in grads:
        _native_bwd(do, q, k, v, o, lse, plan, True, scale, *g)
    nv.check_status()
    for a, b in zip(*grads):
        assert torch.equal(a, b) and not b[~live].any() and not b[live].isnan().any()
