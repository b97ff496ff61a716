"""Row-wise sm_100a kernels against their eager PyTorch oracles (forward and backward)."""
import pytest
import torch

from lset_b200.ops import _native as nv
from lset_b200.ops import activation as A
from lset_b200.ops import embedding as E
from lset_b200.ops import norm as N
from lset_b200.ops import pooling as P
from lset_b200.ops import rope as R

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def _r(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(BF)


def _close(a, b, tol=2e-2, name=""):
    err = (a.float() - b.float()).abs().max().item()
    ref = b.float().abs().max().item() + 1e-6
    assert err / ref < tol, f"{name}: err {err:.4g} ref {ref:.4g}"


def _grads(fn, inputs, gout):
    leaves = [t.detach().clone().requires_grad_() for t in inputs]
    out = fn(*leaves)
    outs = out if isinstance(out, tuple) else (out,)
    gs = gout if isinstance(gout, tuple) else (gout,)
    torch.autograd.backward([o for o in outs if o is not None], [g for g in gs])
    return outs, [l.grad for l in leaves]


def _f32(fn):
    """Run an oracle in fp32 on fp32 copies of bf16 inputs (less rounding noise in the reference)."""
    return fn


@pytest.mark.parametrize("N_,H", [(300, 1024), (1000, 2560), (77, 4096), (513, 768), (64, 128), (9, 8192)])
@pytest.mark.parametrize("w_off", [0.0, 1.0])
def test_rms_norm(N_, H, w_off):
    x, w, g = _r(N_, H), _r(H, scale=0.5), _r(N_, H)
    (y,), gr = _grads(lambda a, b: N.rms_norm(a, b, 1e-6, w_off), [x, w], g)
    (yr,), grr = _grads(lambda a, b: N.rms_norm_ref(a, b, 1e-6, w_off), [x.float(), w.float()], g.float())
    nv.check_status()
    _close(y, yr, name="y")
    _close(gr[0], grr[0], name="dx")
    _close(gr[1], grr[1], 3e-2, name="dw")


@pytest.mark.parametrize("N_,H", [(300, 1024), (1000, 2560), (130, 4096)])
def test_residual_rms_norm(N_, H):
    r, x, w = _r(N_, H), _r(N_, H), _r(H, scale=0.5)
    g1, g2 = _r(N_, H), _r(N_, H)
    (y, nr), gr = _grads(lambda a, b, c: N.residual_rms_norm(a, b, c, 1e-6), [r, x, w], (g1, g2))
    (yr, nrr), grr = _grads(lambda a, b, c: N.residual_rms_norm_ref(a, b, c, 1e-6),
                            [r.float(), x.float(), w.float()], (g1.float(), g2.float()))
    _close(y, yr, name="y"); _close(nr, nrr, name="nr")
    _close(gr[0], grr[0], name="dr"); _close(gr[1], grr[1], name="dx"); _close(gr[2], grr[2], 3e-2, name="dw")


@pytest.mark.parametrize("N_,H", [(200, 768), (1000, 1024), (33, 2560)])
def test_double_residual_rms_norm(N_, H):
    r, a, w1, w2 = _r(N_, H), _r(N_, H), _r(H, scale=0.3), _r(H, scale=0.3)
    g1, g2 = _r(N_, H), _r(N_, H)
    (out, nr), gr = _grads(lambda p, q, u, v: N.double_residual_rms_norm(p, q, u, v, 1e-6, 1.0),
                           [r, a, w1, w2], (g1, g2))
    (outr, nrr), grr = _grads(lambda p, q, u, v: N.double_residual_rms_norm_ref(p, q, u, v, 1e-6, 1.0),
                              [t.float() for t in (r, a, w1, w2)], (g1.float(), g2.float()))
    _close(out, outr, name="y"); _close(nr, nrr, name="nr")
    _close(gr[0], grr[0], name="dr"); _close(gr[1], grr[1], 3e-2, name="da")
    _close(gr[2], grr[2], 4e-2, name="dw1"); _close(gr[3], grr[3], 4e-2, name="dw2")


@pytest.mark.parametrize("N_,H", [(300, 768), (1000, 1024), (64, 384)])
@pytest.mark.parametrize("res", [False, True])
def test_layer_norm(N_, H, res):
    x, w, b, g = _r(N_, H), _r(H, scale=0.5), _r(H, scale=0.5), _r(N_, H)
    if res:
        r, g2 = _r(N_, H), _r(N_, H)
        (y, nr), gr = _grads(lambda a, c, d, e: N.residual_layer_norm(a, c, d, e, 1e-12), [r, x, w, b], (g, g2))
        (yr, nrr), grr = _grads(lambda a, c, d, e: N.residual_layer_norm_ref(a, c, d, e, 1e-12),
                                [t.float() for t in (r, x, w, b)], (g.float(), g2.float()))
        _close(nr, nrr, name="nr")
    else:
        (y,), gr = _grads(lambda c, d, e: N.layer_norm(c, d, e, 1e-12), [x, w, b], g)
        (yr,), grr = _grads(lambda c, d, e: N.layer_norm_ref(c, d, e, 1e-12),
                            [t.float() for t in (x, w, b)], g.float())
    _close(y, yr, name="y")
    for i, (a_, b_) in enumerate(zip(gr, grr)):
        _close(a_, b_, 3e-2, name=f"grad{i}")


@pytest.mark.parametrize("Hq,Hk,hd", [(16, 8, 128), (32, 8, 128), (12, 12, 64), (4, 1, 256)])
@pytest.mark.parametrize("do_norm", [True, False])
def test_qk_norm_rope(Hq, Hk, hd, do_norm):
    T = 333
    qkv = _r(T, Hq + 2 * Hk, hd)
    q, k = qkv[:, :Hq], qkv[:, Hq:Hq + Hk]
    qw = _r(hd, scale=0.5) if do_norm else None
    kw = _r(hd, scale=0.5) if do_norm else None
    pos = torch.randint(0, 700, (T,), device="cuda")
    cos, sin = R.rope_tables(hd, 1024, 1e6, "cuda")
    gq, gk = _r(T, Hq, hd), _r(T, Hk, hd)
    ins = [q, k] + ([qw, kw] if do_norm else [])
    f = (lambda a, b, c, d: R.qk_norm_rope(a, b, c, d, cos, sin, pos)) if do_norm else \
        (lambda a, b: R.qk_norm_rope(a, b, None, None, cos, sin, pos))
    fr = (lambda a, b, c, d: R.qk_norm_rope_ref(a, b, c, d, cos, sin, pos)) if do_norm else \
        (lambda a, b: R.qk_norm_rope_ref(a, b, None, None, cos, sin, pos))
    (qo, ko), gr = _grads(f, ins, (gq, gk))
    (qr, kr), grr = _grads(fr, [t.float() for t in ins], (gq.float(), gk.float()))
    nv.check_status()
    _close(qo, qr, name="q"); _close(ko, kr, name="k")
    for i, (a_, b_) in enumerate(zip(gr, grr)):
        _close(a_, b_, 3e-2, name=f"grad{i}")


@pytest.mark.parametrize("kind", ["swiglu", "geglu"])
def test_glu(kind):
    gu, g = _r(500, 2 * 3072), _r(500, 3072)
    (y,), gr = _grads(lambda a: A.glu(a, kind), [gu], g)
    (yr,), grr = _grads(lambda a: A.glu_ref(a[:, :3072], a[:, 3072:], kind), [gu.float()], g.float())
    _close(y, yr); _close(gr[0], grr[0])


def test_gelu():
    x, g = _r(100, 3072), _r(100, 3072)
    (y,), gr = _grads(A.gelu, [x], g)
    (yr,), grr = _grads(torch.nn.functional.gelu, [x.float()], g.float())
    _close(y, yr); _close(gr[0], grr[0])


def test_normalize_and_gather():
    x, g = _r(1500, 1024), _r(1500, 1024)
    (y,), gr = _grads(P.normalize, [x], g)
    (yr,), grr = _grads(lambda a: torch.nn.functional.normalize(a, dim=-1), [x.float()], g.float())
    _close(y, yr); _close(gr[0], grr[0])
    idx = torch.tensor([5, 17, 1499, 0, 700], device="cuda")
    g2 = _r(5, 1024)
    (y2,), gr2 = _grads(lambda a: P.gather_normalize(a, idx), [x], g2)
    (y2r,), gr2r = _grads(lambda a: torch.nn.functional.normalize(a[idx], dim=-1), [x.float()], g2.float())
    _close(y2, y2r); _close(gr2[0], gr2r[0])


@pytest.mark.parametrize("strategy", ["last_token", "cls", "mean", "weighted_mean"])
def test_packed_pool(strategy):
    lens = [5, 130, 64, 1, 300]
    T = sum(lens)
    cu = torch.tensor([0, 5, 135, 199, 200, 500], dtype=torch.int32, device="cuda")
    h, g = _r(T, 768), _r(5, 768)
    (y,), gr = _grads(lambda a: P.packed_pool(a, cu, strategy), [h], g)
    (yr,), grr = _grads(lambda a: P.packed_pool(a, cu, strategy), [h.float()], g.float())
    _close(y, yr); _close(gr[0], grr[0])


def test_embedding():
    tab = _r(1000, 1024).requires_grad_()
    ids = torch.randint(0, 1000, (7, 33), device="cuda")
    out = E.embedding(ids, tab)
    assert torch.equal(out, tab.detach()[ids])
    g = _r(7, 33, 1024)
    out.backward(g)
    ref = torch.zeros(1000, 1024, device="cuda").index_add_(0, ids.reshape(-1), g.reshape(-1, 1024).float())
    _close(tab.grad, ref)
    pos_tab, typ_tab = _r(64, 1024), _r(2, 1024)
    pos = torch.arange(33, device="cuda")[None]
    typ = torch.zeros(7, 33, dtype=torch.long, device="cuda")
    out3 = E.embedding(ids, tab.detach(), extra=((pos, pos_tab), (typ, typ_tab)))
    ref3 = tab.detach()[ids].float() + pos_tab[pos].float() + typ_tab[typ].float()
    _close(out3, ref3)


def test_bounded_wait_times_out_with_status_and_context_survives():
    import ctypes

    lib = nv.load()
    flag = torch.zeros(1, dtype=torch.int32, device="cuda")      # nothing ever sets it
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    waited = torch.zeros(1, dtype=torch.int64, device="cuda")
    rc = lib.lb_bounded_wait_probe(ctypes.c_void_p(flag.data_ptr()), ctypes.c_uint(1),
                                   ctypes.c_ulonglong(200_000_000), ctypes.c_void_p(status.data_ptr()),
                                   ctypes.c_void_p(waited.data_ptr()),
                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    torch.cuda.synchronize()
    assert status.item() == 4 and 0.15e9 < waited.item() < 2e9
    flag.fill_(1)                                                 # a set flag returns at once
    status.zero_()
    lib.lb_bounded_wait_probe(ctypes.c_void_p(flag.data_ptr()), ctypes.c_uint(1),
                              ctypes.c_ulonglong(200_000_000), ctypes.c_void_p(status.data_ptr()),
                              ctypes.c_void_p(waited.data_ptr()),
                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert status.item() == 0 and waited.item() < 50_000_000
    assert torch.ones(4, device="cuda").sum().item() == 4.0       # the context is still usable


def test_device_barrier_single_gpu_forms():
    """The device barrier on one GPU: a one-rank group passes at once; a two-rank group whose peer
    never announces runs into the bounded wait and reports the peer-timeout status (nothing hangs,
    the context stays usable). The peer's pad is a second local buffer, so no other GPU is involved."""
    import ctypes

    lib = nv.load()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    mine = torch.zeros(64, dtype=torch.int32, device="cuda")
    peer = torch.zeros(64, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    pads1 = (ctypes.c_void_p * 1)(mine.data_ptr())
    for epoch in (1, 2, 3):
        rc = lib.lb_device_barrier(pads1, ctypes.c_int(1), ctypes.c_int(0), ctypes.c_uint(epoch),
                                   ctypes.c_ulonglong(200_000_000),
                                   ctypes.c_void_p(status.data_ptr()), stream)
        assert rc == 0
    torch.cuda.synchronize()
    assert status.item() == 0 and mine[0].item() == 3
    pads2 = (ctypes.c_void_p * 2)(mine.data_ptr(), peer.data_ptr())
    mine.zero_()
    rc = lib.lb_device_barrier(pads2, ctypes.c_int(2), ctypes.c_int(0), ctypes.c_uint(1),
                               ctypes.c_ulonglong(200_000_000), ctypes.c_void_p(status.data_ptr()),
                               stream)
    assert rc == 0
    torch.cuda.synchronize()
    assert status.item() == 4                      # kStatusTimeoutPeer
    assert mine[0].item() == 1 and peer[0].item() == 1   # this rank did announce to both pads
    mine[1] = 2                                    # the "peer" is already one barrier ahead
    status.zero_()
    lib.lb_device_barrier(pads2, ctypes.c_int(2), ctypes.c_int(0), ctypes.c_uint(2),
                          ctypes.c_ulonglong(200_000_000), ctypes.c_void_p(status.data_ptr()), stream)
    torch.cuda.synchronize()
    assert status.item() == 0
    assert torch.ones(4, device="cuda").sum().item() == 4.0


def test_poll_status_raises_one_call_late_without_blocking():
    """The training loop's non-blocking status check: the value seen is the one copied by the
    previous call; a non-zero status raises and clears the word."""
    word = nv.status_word(torch.device("cuda", torch.cuda.current_device()))
    word.zero_()
    nv.poll_status()
    nv.poll_status()                       # still clean
    word.fill_(4)                          # what a kernel that gave up waiting for a peer writes
    nv.poll_status()                       # copies the 4 ...
    with pytest.raises(nv.NativeError):
        nv.poll_status()                   # ... and the next call sees it
    torch.cuda.synchronize()
    assert word.item() == 0
    nv.poll_status()
    nv.poll_status()


@pytest.mark.gpu
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("H", [8, 64, 136, 768, 1024, 2560])
def test_segment_mean_chunk_edges(H, weighted):
    """Segments around the 32 tokens a thread has in flight (per token subset), and empty ones."""
    from lset_b200.ops.pooling import segment_mean

    subsets = max(1, min(32, 256 // (H // 8)))
    whole = 32 * subsets
    lens = [1, 0, subsets, whole - 1, whole, whole + 1, 2 * whole - subsets, 2 * whole + 3]
    cu = torch.tensor([0] + lens).cumsum(0).int().cuda()
    x = torch.randn(sum(lens), H, generator=torch.Generator().manual_seed(H)).bfloat16().cuda()
    got = segment_mean(x, cu, weighted).double()
    for m, n in enumerate(lens):
        seg = x[int(cu[m]):int(cu[m + 1])].double()
        w = torch.arange(1, n + 1, device="cuda").double() if weighted else torch.ones(n).double().cuda()
        if n == 0:
            assert torch.equal(got[m], torch.zeros_like(got[m]))
            continue
        want = (w[:, None] * seg).sum(0) / w.sum()
        # one rounding to bf16, and fp32 sums of n terms in any order
        tol = want.abs() * 2.0 ** -8 + n * 2.0 ** -23 * (w[:, None] * seg.abs()).sum(0) / w.sum()
        assert ((got[m] - want).abs() <= tol + 1e-30).all(), (m, n)


@pytest.mark.gpu
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("H", [8, 64, 136, 1024, 2560])
def test_segment_mean_of_many_or_short_segments(H, weighted):
    """These have a kernel of their own: the sums of the other one, in its order from 64 columns up."""
    from lset_b200.ops.pooling import segment_mean

    lens = [1, 0, 3, 40, 17, 33, 100]
    one = torch.randn(sum(lens), H, generator=torch.Generator().manual_seed(H)).bfloat16().cuda()
    few = segment_mean(one, torch.tensor([0] + lens).cumsum(0).int().cuda(), weighted)
    cu = torch.tensor([0] + lens * 90).cumsum(0).int().cuda()
    many = segment_mean(one.repeat(90, 1), cu, weighted).view(90, len(lens), H)
    assert torch.equal(many, many[:1].expand_as(many))
    if H >= 64:
        assert torch.equal(many[0], few)
    ref = torch.stack([(s.double() * (torch.arange(1, n + 1, device="cuda").double()[:, None]
                                      if weighted else 1)).sum(0)
                       / max(1.0, n * (n + 1) / 2 if weighted else n)
                       for n, s in zip(lens, one.split(lens))])
    # one rounding to bf16 and fp32 sums of at most 100 terms
    assert ((many[0].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-4).all()
    short = segment_mean(one[:20], torch.tensor([0, 1, 1, 5, 20]).int().cuda(), weighted)
    if H >= 64:
        assert torch.equal(short[0], few[0])


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [1, 4])
@pytest.mark.parametrize("H", [64, 136, 1024, 2560])
def test_rms_norm_takes_a_weight_that_starts_anywhere(H, offset):
    """A slice of a flat buffer that does not start at a 16-byte boundary; the same bits."""
    from lset_b200.ops.norm import residual_rms_norm, rms_norm

    g = torch.Generator().manual_seed(H)
    x, r = (torch.randn(37, H, generator=g).bfloat16().cuda() for _ in range(2))
    flat = torch.randn(H + offset, generator=g).bfloat16().cuda()
    w = flat[offset:]
    assert w.data_ptr() % 16 != 0
    assert torch.equal(rms_norm(x, w), rms_norm(x, w.clone()))
    for a, b in zip(residual_rms_norm(r, x, w), residual_rms_norm(r, x, w.clone())):
        assert torch.equal(a, b)


@pytest.mark.parametrize("Hq,Hk,hd", [(16, 8, 128), (5, 1, 64), (3, 1, 256)])
@pytest.mark.parametrize("norm", [True, False])
def test_rope_of_few_and_of_many_tokens_has_the_same_bits(Hq, Hk, hd, norm):
    """Few tokens are cut into groups of heads, and their backward has lanes of its own; values and input
    gradients of a token do not depend on how many there are. Weight gradients: fp32 sums."""
    from lset_b200.ops.rope import qk_norm_rope

    torch.manual_seed(hd)
    T, parts = 16000, [1, 33, 4000, 11966]      # more than 3 * 148 * 4096 / hd / 2 of them: many
    q, k = (torch.randn(T, h, hd, device="cuda").to(torch.bfloat16) for h in (Hq, Hk))
    gq, gk = torch.randn_like(q), torch.randn_like(k)
    ws = [(torch.rand(hd, device="cuda") + 0.5).to(torch.bfloat16).requires_grad_() for _ in range(2)]
    cos, sin = torch.randn(512, hd // 2, device="cuda"), torch.randn(512, hd // 2, device="cuda")
    pos = torch.randint(0, 512, (T,), device="cuda")

    def run(rows):
        a, b = q[rows].clone().requires_grad_(), k[rows].clone().requires_grad_()
        out = qk_norm_rope(a, b, *(ws if norm else (None, None)), cos, sin, pos[rows])
        for w in ws:
            w.grad = None
        torch.autograd.backward(out, (gq[rows], gk[rows]))
        return [*(o.detach() for o in out), a.grad, b.grad], [w.grad.double() for w in ws if norm]

    whole, wsum = run(slice(0, T))
    total, at = [0.0, 0.0], 0
    for n in parts:
        part, wg = run(slice(at, at + n))
        for x, y in zip(part, whole):
            assert torch.equal(x, y[at:at + n]), n
        total = [a + b for a, b in zip(total, wg)]
        at += n
    assert at == T
    for a, b in zip(total, wsum):      # four bf16 roundings of the parts' sums
        assert ((a - b).norm() / b.norm()).item() < 4 * 2 ** -8


@pytest.mark.parametrize("op", ["swiglu", "geglu", "rms"])
def test_rows_of_many_have_the_bits_of_few(op):
    """Walks that go round the grid several times, and end within a round; widths that fill no wave of
    vectors. A row's values and input gradients do not depend on how many rows there are."""
    torch.manual_seed(0)
    T, H = (6401, 3080) if op != "rms" else (4801, 1000)    # above 64 * 256 * 148 vectors; 6 * 148 * 4 rows
    x, g, g2 = _r(T, H if op == "rms" else 2 * H), _r(T, H), _r(T, H)
    w, r = _r(H, scale=0.5), _r(T, H)

    def run(rows):
        if op == "rms":
            outs, gr = _grads(lambda a, b, c: N.residual_rms_norm(a, b, c, 1e-6), [r[rows], x[rows], w],
                              (g[rows], g2[rows]))
            return [*outs, *gr[:2]]
        outs, gr = _grads(lambda a: A.glu(a, op), [x[rows]], g[rows])
        return [*outs, *gr]

    whole, at = run(slice(0, T)), 0
    for n in (1, 3, 700, T - 704):
        for a, b in zip(run(slice(at, at + n)), whole):
            assert torch.equal(a, b[at:at + n]), n
        at += n


@pytest.mark.parametrize("N_,H", [(1, 1032), (700, 1032), (3000, 1032), (2, 2056), (2500, 2056)])
def test_rms_norm_weight_gradient_is_summed_in_one_order(N_, H):
    """Bits of a training step (the gradient norm, and through the clip coefficient every weight): six partial rows
    an SM, each of them the sums of its rows (two at a time up to 2048 columns), then every 32nd partial row,
    then those. bf16 products are exact in fp32."""
    torch.manual_seed(H)
    x, dy, w = _r(N_, H), _r(N_, H), _r(H, scale=0.5)
    rstd, dx = torch.rand(N_, device="cuda") + 0.5, torch.empty_like(x)
    lib = nv.load()
    scratch = torch.empty(lib.lb_norm_bwd_partial_rows() * H, device="cuda")
    dw = torch.empty(H, device="cuda")
    p = lambda t: nv.c_void_p(t.data_ptr())  # noqa: E731
    assert lib.lb_rms_norm_bwd(p(dy), nv.c_void_p(0), p(x), p(w), p(rstd), p(dx), p(scratch), p(dw), nv.c_int(1),
                               nv.c_int(0), nv.c_int(N_), nv.c_int(H), nv.c_float(0.0),
                               nv.c_void_p(nv.stream_ptr())) == 0
    rows = 2 if H <= 2048 else 1
    ctas = min((N_ + rows - 1) // rows, 6 * torch.cuda.get_device_properties(0).multi_processor_count)
    terms = dy.float() * (x.float() * rstd[:, None]).to(torch.bfloat16).float()
    terms = torch.nn.functional.pad(terms, (0, 0, 0, -N_ % (ctas * rows))).view(-1, ctas, rows, H)
    part = torch.zeros(ctas, rows, H, device="cuda")
    for t in terms:
        part += t
    part = torch.nn.functional.pad(part.sum(1), (0, 0, 0, -ctas % 32)).view(-1, 32, H)
    groups = torch.zeros(32, H, device="cuda")
    for t in part:
        groups += t
    want = torch.zeros(H, device="cuda")
    for t in groups:
        want += t
    assert torch.equal(dw, want)


@pytest.mark.parametrize("T,Hq,Hk,hd", [(1, 2, 1, 128), (3000, 16, 8, 128), (2500, 5, 2, 64), (10000, 2, 1, 128),
                                        (5000, 3, 1, 256)])
def test_rope_weight_gradients_are_summed_in_one_order(T, Hq, Hk, hd):
    """As for the norms: groups of lanes walk over units of heads (four of q's and k's in a row of few tokens, else
    all of a token), a partial row has the groups of 16 tokens (of 128 columns), then every 32nd partial row, then
    those. Without a rotation the terms are products of bf16 values, exact in fp32."""
    torch.manual_seed(T)
    H, dev = Hq + Hk, "cuda"
    x, dy, dx = _r(T, H * hd), _r(T, H * hd), torch.empty(T, H * hd, device=dev, dtype=torch.bfloat16)
    qw, kw, rstd = _r(hd), _r(hd), torch.rand(T, H, device=dev) + 0.5
    rq, rk = rstd[:, :Hq].contiguous(), rstd[:, Hq:].contiguous()
    cos, sin = torch.ones(1, hd // 2, device=dev), torch.zeros(1, hd // 2, device=dev)
    pos = torch.zeros(T, dtype=torch.int32, device=dev)
    lib = nv.load()
    scratch = torch.empty(lib.lb_rope_bwd_partial_rows() * 2 * hd, device=dev)
    dw = torch.empty(2, hd, device=dev)
    p = lambda t, at=0: nv.c_void_p(t.data_ptr() + 2 * at)  # noqa: E731
    ld, k_at = nv.c_ll(H * hd), Hq * hd
    assert lib.lb_qk_norm_rope_bwd(
        p(dy), ld, p(dy, k_at), ld, p(x), ld, p(x, k_at), ld, p(qw), p(kw), p(cos), p(sin), p(pos), nv.c_int(0),
        nv.c_int(1), p(rq), p(rk), p(dx), ld, p(dx, k_at), ld, p(scratch), p(dw), nv.c_int(1), nv.c_int(0),
        nv.c_int(T), nv.c_int(Hq), nv.c_int(Hk), nv.c_int(hd), nv.c_float(0.0), nv.c_int(1),
        nv.c_void_p(nv.stream_ptr())) == 0
    sms, groups = torch.cuda.get_device_properties(0).multi_processor_count, 2048 // hd
    unit = 4 if T < 3 * sms * groups // 2 else H
    parts = -(-H // unit)
    rows = min(-(-T * parts // groups), 4 * sms)
    terms = dy.view(T, H, hd).float() * (x.view(T, H, hd).float() * rstd[..., None]).to(torch.bfloat16).float()
    terms = torch.nn.functional.pad(terms, (0, 0, 0, parts * unit - H)).view(T * parts, unit, hd)
    is_k = (torch.arange(parts * unit, device=dev) >= Hq).view(parts, unit).repeat(T, 1)[..., None]
    extra = -T * parts % (rows * groups)
    for kind, got in ((False, dw[0]), (True, dw[1])):
        t = torch.where(is_k == kind, terms, 0.0)
        t = torch.nn.functional.pad(t, (0, 0, 0, 0, 0, extra)).view(-1, rows, groups, unit, hd)
        acc = torch.zeros(rows, groups, hd, device=dev)
        for step in t:
            for j in range(unit):
                acc += step[:, :, j]
        part = torch.zeros(rows, hd, device=dev)
        for j in range(groups):
            part += acc[:, j]
        part = torch.nn.functional.pad(part, (0, 0, 0, -rows % 32)).view(-1, 32, hd)
        sums, want = torch.zeros(32, hd, device=dev), torch.zeros(hd, device=dev)
        for q in part:
            sums += q
        for q in sums:
            want += q
        assert torch.equal(got, want), kind
