"""The attention of short sequences, with q's and k's norms and rotation in it, against the kernels it
stands in for: the rotation and an fp32 softmax attention of its outputs."""
import math

import pytest
import torch

from lset_b200.ops import _native as nv
from lset_b200.ops.attention import AttnPlan, attention_ref
from lset_b200.ops.rope import qk_norm_rope

pytestmark = pytest.mark.gpu


def _rand(*shape):
    return torch.randn(*shape, device="cuda").to(torch.bfloat16)


@pytest.mark.parametrize("Hq,Hk,hd,causal,rotate,norm", [
    (4, 2, 128, 1, True, True), (2, 2, 128, 0, True, False), (3, 3, 64, 0, False, False),
    (8, 1, 64, 1, True, True), (2, 1, 128, 0, False, False)])
@pytest.mark.parametrize("lens,tail,max_len", [
    ([1], 0, 1), ([15, 16, 17], 3, 17), ([64, 0, 63, 33], 0, 64), ([65, 130, 7], 2, 64), ([200], 1, 200)])
def test_short_attention(Hq, Hk, hd, causal, rotate, norm, lens, tail, max_len):
    torch.manual_seed(len(lens))
    T, W = sum(lens) + tail, (Hq + 2 * Hk) * hd
    qkv, pos = _rand(T, W), torch.randint(0, 300, (T,), device="cuda")
    cu = torch.tensor([0] + lens, device="cuda").cumsum(0).to(torch.int32)
    cos, sin = (f(torch.rand(300, hd // 2, device="cuda") * 6) for f in (torch.cos, torch.sin))
    qw, kw = _rand(hd) * 0.2 + 1, _rand(hd) * 0.2 + 1
    q, k, v = (t.unflatten(1, (-1, hd)) for t in qkv.split((Hq * hd, Hk * hd, Hk * hd), 1))
    qr, kr = q, k
    if rotate:
        qr, kr = qk_norm_rope(q, k, *((qw, kw) if norm else (None, None)), cos, sin, pos)
    scale = 1 / math.sqrt(hd)
    want = attention_ref(qr.float(), kr.float(), v.float(), cu, bool(causal), scale)
    plan, cap = AttnPlan(cu, max(lens), T).tiles(128 // (Hq // Hk))
    out = torch.full((T, Hq, hd), 7.0, device="cuda", dtype=torch.bfloat16)
    p = lambda t: nv.c_void_p(t.data_ptr() if t is not None else 0)  # noqa: E731
    rc = nv.load().lb_attn_short(
        p(q), p(k), p(v), nv.c_ll(W), p(qw if norm else None), p(kw if norm else None),
        p(cos if rotate else None), p(sin if rotate else None), p(pos if rotate else None), nv.c_int(1),
        p(cu), p(cu[1:]), p(plan), nv.c_int(cap), p(out), nv.c_ll(Hq * hd), nv.c_int(T),
        nv.c_int(len(lens)), nv.c_int(max_len), nv.c_int(Hq), nv.c_int(Hk), nv.c_int(hd),
        nv.c_float(1e-6), nv.c_float(0.0), nv.c_float(scale), nv.c_int(causal), nv.c_void_p(nv.stream_ptr()))
    assert rc == 0
    # probabilities and the output are rounded to bf16 (2^-9 each of values up to the largest v)
    err = (out.float() - want).abs().max().item()
    assert err < 2 * 2 ** -9 * v.float().abs().max().item(), err
    assert not out[sum(lens):].any()
    nv.check_status()


@pytest.mark.parametrize("B,max_len,hd,rotation,want", [
    (18, 64, 128, 1, 1), (19, 64, 128, 1, 0), (4, 65, 128, 1, 0), (500, 64, 64, 0, 1), (1, 65, 64, 0, 0),
    (1, 24, 256, 1, 0), (0, 24, 64, 0, 0), (1, 0, 64, 0, 0)])
def test_which_calls_are_short(B, max_len, hd, rotation, want):
    """16 query heads on 148 SMs: two CTAs an SM with rotation."""
    args = [nv.c_int(x) for x in (B, max_len, 16, 8, hd, rotation)]
    assert bool(nv.load().lb_attn_short_ok(*args)) == bool(want)
    assert not nv.load().lb_attn_short_ok(*args[:2], nv.c_int(6), nv.c_int(2), *args[4:])


@pytest.mark.parametrize("padded", [False, True])
@pytest.mark.parametrize("heads,kv_heads,head_dim", [(4, 2, 128), (4, 4, 64)])
def test_passes_declared_inference_run_it(heads, kv_heads, head_dim, padded):
    """Against the same pass not declared so, which runs the rotation and the tile kernels: per layer the
    probabilities, the attention's output and the sums of its projection are rounded differently, 2^-9 each
    of values that the next layer's norm may amplify: 2^-6 for two layers. A launch a layer is saved."""
    from lset_b200.models import Qwen3Config
    from lset_b200.models.decoder import Qwen3Decoder
    from lset_b200.ops.block import inference_pass

    torch.manual_seed(2)
    cfg = Qwen3Config(vocab_size=512, hidden_size=256, intermediate_size=512, num_hidden_layers=2,
                      num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=head_dim)
    model = Qwen3Decoder(cfg, fused_projections=True).cuda().to(torch.bfloat16).eval()
    lens = [9, 33, 1]
    if padded:
        mask = torch.zeros(3, 33, dtype=torch.long, device="cuda")
        for i, n in enumerate(lens):
            mask[i, 33 - n:] = 1
        inputs = dict(input_ids=torch.randint(0, 512, (3, 33), device="cuda"), attention_mask=mask)
    else:
        cu = torch.tensor([0, 9, 42, 43], dtype=torch.int32, device="cuda")
        inputs = dict(input_ids=torch.randint(0, 512, (43,), device="cuda"), cu_seqlens=cu, max_seqlen=33,
                      position_ids=torch.cat([torch.arange(n, device="cuda") for n in lens]))
    with torch.no_grad():
        before = nv.launches()
        want = model(**inputs)["hidden_states"].float()
        between = nv.launches()
        with inference_pass():
            got = model(**inputs)["hidden_states"].float()
    assert (between - before) - (nv.launches() - between) >= 2
    assert torch.isfinite(got).all()
    if padded:
        want, got = want[mask.bool()], got[mask.bool()]
    assert ((got - want).norm() / want.norm()).item() < 2 ** -6
    nv.check_status()
