"""The GEMM for few tokens (``lb_gemm_small``): one to three weights side by side, along the output
columns, the contraction or the output rows, split over clusters or not, against fp64 products."""
import ctypes

import pytest
import torch

from lset_b200.ops import _native as nv

pytestmark = pytest.mark.gpu
_vp, _ll, _ci = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int
N_PARTS, K_PARTS, M_PARTS = 0, 1, 2


class SmallGemm(ctypes.Structure):      # LbSmallGemm of csrc/gemm/gemm_small.h
    _fields_ = [("A", _vp), ("B", _vp * 3), ("C", _vp * 3), ("lda", _ll), ("ldb", _ll * 3),
                ("ldc", _ll * 3), ("M", _ci), ("N", _ci), ("K", _ci), ("ext", _ci * 3),
                ("nparts", _ci), ("mode", _ci), ("a_mn", _ci), ("b_mn", _ci), ("out_fp32", _ci),
                ("bias", _vp * 3), ("glu_h", _vp), ("ld_h", _ll), ("glu_kind", _ci),
                ("b_ready", _ci), ("may_split", _ci), ("bn", _ci), ("splits", _ci), ("status", _vp), ("stream", _vp)]


def _call(a, bs, cs, M, N, K, ext, mode, a_mn=0, b_mn=0, fp32=0, bias=(), h=None, bn=0, splits=0, kind=0, scale=None):
    g = SmallGemm()
    g.A, g.lda = a.data_ptr(), a.stride(0)
    for i, b in enumerate(bs):
        g.B[i], g.ldb[i] = b.data_ptr(), b.stride(0)
    for i, c in enumerate(cs):
        g.C[i], g.ldc[i] = c.data_ptr(), c.stride(0)
    for i, e in enumerate(ext):
        g.ext[i] = e
    for i, b in enumerate(bias):
        g.bias[i] = b.data_ptr()
    g.M, g.N, g.K, g.nparts, g.mode = M, N, K, len(ext), mode
    g.a_mn, g.b_mn, g.out_fp32, g.bn, g.splits = a_mn, b_mn, fp32, bn, splits
    if h is not None:
        g.glu_h, g.ld_h, g.glu_kind = h.data_ptr(), h.stride(0), kind
    g.status, g.stream = nv.status_word(a.device).data_ptr(), nv.stream_ptr()
    if scale is not None:
        return nv.load().lb_gemm_small_scaled(ctypes.byref(g), ctypes.c_float(scale))
    return nv.load().lb_gemm_small(ctypes.byref(g))


def _rand(*shape):
    return torch.randn(*shape, device="cuda").to(torch.bfloat16)


def _rel(x, ref):
    return ((x.double() - ref).norm() / ref.norm()).item()


def _columns(c, ext):
    at, out = 0, []
    for e in ext:
        out.append(c[:, at:at + e])
        at += e
    return out


FORMS = [(bn, s) for bn in (64, 128) for s in (1, 2, 8)] + [(0, 0)]
ROUND = 2 ** -8   # one rounding to bf16 (2^-9 at most, less in the 2-norm)


@pytest.mark.parametrize("T", [1, 33, 128, 257])
@pytest.mark.parametrize("ext,K", [([72], 64), ([128, 64, 136], 200), ([768, 768, 768], 2048)])
def test_parts_along_the_columns(T, ext, K):
    torch.manual_seed(T)
    a, bs, bias = _rand(T, K), [_rand(e, K) for e in ext], [_rand(e) for e in ext]
    ref = a.double() @ torch.cat(bs).double().t()
    for bn, s in FORMS:
        c = torch.full((T, sum(ext)), float("nan"), device="cuda", dtype=torch.bfloat16)
        assert _call(a, bs, _columns(c, ext), T, sum(ext), K, ext, N_PARTS, bn=bn, splits=s) == 0
        assert _rel(c, ref) < ROUND, (bn, s)
        assert _call(a, bs, _columns(c, ext), T, sum(ext), K, ext, N_PARTS, bias=bias, bn=bn,
                     splits=s) == 0
        assert _rel(c, ref + torch.cat(bias).double()) < ROUND, (bn, s)
    nv.check_status()


@pytest.mark.parametrize("T,N", [(1, 8), (7, 16), (100, 56), (127, 120), (300, 16)])
def test_operands_with_fewer_rows_than_a_tile(T, N):
    """Loaded as they are: what lies below them in shared memory is read by no one. Not finite here,
    from the product before."""
    K = 1024
    bad = torch.full((256, K), float("nan"), device="cuda", dtype=torch.bfloat16)
    junk = torch.empty(256, 128, device="cuda", dtype=torch.bfloat16)
    a, b = _rand(T, K), _rand(N, K)
    ref = a.double() @ b.double().t()
    for bn, s in FORMS:
        for _ in range(2):      # 2 x 148 CTAs and more: every SM's shared memory
            assert _call(bad, [bad.repeat(80, 1)], [junk.new_empty(256, 20480)], 256, 20480, K, [20480],
                         N_PARTS, bn=64, splits=1) == 0
        c = torch.full((T, N), float("nan"), device="cuda", dtype=torch.bfloat16)
        assert _call(a, [b], [c], T, N, K, [N], N_PARTS, bn=bn, splits=s) == 0
        assert _rel(c, ref) < ROUND, (bn, s)
    nv.check_status()


@pytest.mark.parametrize("T", [1, 128, 257])
@pytest.mark.parametrize("ext,N", [([64], 72), ([128, 64, 192], 200), ([3072, 3072], 1024)])
def test_parts_along_the_contraction(T, ext, N):
    torch.manual_seed(T)
    a, bs = _rand(T, sum(ext)), [_rand(e, N) for e in ext]
    ref = a.double() @ torch.cat(bs).double()
    for bn, s in FORMS:
        c = torch.full((T, N), float("nan"), device="cuda", dtype=torch.bfloat16)
        assert _call(a, bs, [c], T, N, sum(ext), ext, K_PARTS, b_mn=1, bn=bn, splits=s) == 0
        # every product and every sum is rounded once
        assert _rel(c, ref) < (2 * len(ext) - 1) * ROUND, (bn, s)
        apart = [torch.empty(T, N, device="cuda", dtype=torch.bfloat16) for _ in ext]
        for x, b, e, out in zip(_columns(a, ext), bs, ext, apart):
            assert _call(x, [b], [out], T, N, e, [N], N_PARTS, b_mn=1, bn=bn, splits=1) == 0
        for x in apart[1:]:
            apart[0] += x
        assert torch.equal(c, apart[0]), (bn, s)
    nv.check_status()


@pytest.mark.parametrize("T", [1, 64, 300])
@pytest.mark.parametrize("ext,N", [([72], 64), ([128, 64, 136], 200)])
def test_parts_along_the_rows_add_to_fp32(T, ext, N):
    torch.manual_seed(T)
    a, b = _rand(T, sum(ext)), _rand(T, N)
    ref = a.double().t() @ b.double() + 3
    for bn, s in FORMS:
        cs = [torch.full((e, N), 3.0, device="cuda") for e in ext]
        assert _call(a, [b], cs, sum(ext), N, T, ext, M_PARTS, a_mn=1, b_mn=1, fp32=1, bn=bn,
                     splits=s) == 0
        # fp32 sums of at most 300 products, one more addition
        assert _rel(torch.cat(cs), ref) < 300 ** 0.5 * 2 ** -23, (bn, s)
    nv.check_status()


@pytest.mark.parametrize("T,I", [(1, 40), (130, 1152), (32, 3072)])
@pytest.mark.parametrize("keep", [True, False])
def test_gated_pair(T, I, keep):
    K = 1024
    torch.manual_seed(I)
    a, w = _rand(T, K), [_rand(I, K) * 0.05, _rand(I, K) * 0.05]
    gate, up = (a.double() @ x.double().t() for x in w)
    want = torch.nn.functional.silu(gate) * up
    for bn, s in FORMS:
        gu = torch.full((T, 2 * I), float("nan"), device="cuda", dtype=torch.bfloat16)
        h = torch.full((T, I), float("nan"), device="cuda", dtype=torch.bfloat16)
        assert _call(a, w, [gu[:, :I], gu[:, I:]] if keep else [], T, 2 * I, K, [I, I], N_PARTS,
                     h=h, bn=bn, splits=s) == 0
        # both factors are rounded (2^-9 each, the gate's amplified by at most 1.1 through SiLU),
        # then their product
        assert _rel(h, want) < 2 * ROUND, (bn, s)
        if keep:
            assert _rel(gu, torch.cat([gate, up], 1)) < ROUND
        else:
            assert torch.isnan(gu).all()
    nv.check_status()


@pytest.mark.parametrize("T,N,K", [(1, 8, 64), (65, 72, 1096), (130, 3072, 768)])
@pytest.mark.parametrize("keep,biased", [(True, True), (False, True), (False, False)])
def test_gelu_of_a_product(T, N, K, keep, biased):
    """The bits of the product and a GELU of its own."""
    from lset_b200.ops.activation import gelu

    torch.manual_seed(N)
    a, b, bias = _rand(T, K), _rand(N, K) * 0.05, [_rand(N)] if biased else ()
    for bn, s in [*FORMS, (64 | 64 << 16, 1), (32 | 64 << 16, 4)]:
        u, c, h = (torch.full((T, N), 3.0, device="cuda", dtype=torch.bfloat16) for _ in range(3))
        assert _call(a, [b], [u], T, N, K, [N], N_PARTS, bias=bias, bn=bn, splits=s) == 0
        assert _call(a, [b], [c] if keep else [], T, N, K, [N], N_PARTS, bias=bias, h=h, kind=2, bn=bn,
                     splits=s) == 0
        assert torch.equal(h, gelu(u)), (bn, s)
        assert torch.equal(c, u) if keep else (c == 3).all()
    nv.check_status()


@pytest.mark.parametrize("T", [1, 130, 5000])
@pytest.mark.parametrize("ext,b_mn", [([16, 16, 16], 0), ([8, 64], 0), ([16], 1)])
def test_scaled_products_are_rounded_before_and_after(T, ext, b_mn):
    K = 512
    a, bs = _rand(T, K), [_rand(K, e) if b_mn else _rand(e, K) for e in ext]
    for bn, s in [*FORMS, (64 | 64 << 16, 1)]:
        c, d = ([torch.full((T, e), 3.0, device="cuda", dtype=torch.bfloat16) for e in ext] for _ in range(2))
        assert _call(a, bs, c, T, sum(ext), K, ext, N_PARTS, b_mn=b_mn, bn=bn, splits=s) == 0
        assert _call(a, bs, d, T, sum(ext), K, ext, N_PARTS, b_mn=b_mn, bn=bn, splits=s, scale=0.3) == 0
        for x, y in zip(c, d):
            assert torch.equal(y, (x.float() * 0.3).to(torch.bfloat16)), (bn, s)
    nv.check_status()


@pytest.mark.parametrize("T", [1, 63, 65, 200])
@pytest.mark.parametrize("N,K", [(8, 64), (72, 1096), (1024, 200)])
def test_tiles_of_64_rows(T, N, K):
    """64 x 64 and 64 x 32 tiles: the bits of the 128 x 64 tiles, in every form that takes them; the
    longest contraction goes round the operand ring more than once."""
    torch.manual_seed(T)
    a, b, w = _rand(T, K), _rand(N, K), [_rand(64, N), _rand(K - K % 64, N)]
    wide, bias, x = _rand(T, 64 + K - K % 64), _rand(N), _rand(T, N)

    def both(run, out):
        want = out()
        assert run(want, 64) == 0
        for tile in (64 | 64 << 16, 32 | 64 << 16):
            got = out()
            assert run(got, tile) == 0
            assert torch.equal(got, want), tile & 0xffff

    bf = lambda *s: lambda: torch.full(s, 3.0, device="cuda", dtype=torch.bfloat16)
    both(lambda c, t: _call(a, [b], [c], T, N, K, [N], N_PARTS, bias=[bias], bn=t, splits=1), bf(T, N))
    both(lambda c, t: _call(a, [b, b], [], T, 2 * N, K, [N, N], N_PARTS, h=c, bn=t, splits=1), bf(T, N))
    both(lambda c, t: _call(wide, w, [c], T, N, wide.shape[1], [64, K - K % 64], K_PARTS, b_mn=1, bn=t,
                            splits=2), bf(T, N))
    both(lambda c, t: _call(a, [x], [c], K, N, T, [K], M_PARTS, a_mn=1, b_mn=1, fp32=1, bn=t, splits=1),
         lambda: torch.full((K, N), 3.0, device="cuda"))
    # a split sum: fp32 pieces, one rounding
    c = bf(T, N)()
    assert _call(a, [b], [c], T, N, K, [N], N_PARTS, bn=32 | 64 << 16, splits=4) == 0
    assert _rel(c, a.double() @ b.double().t()) < ROUND
    nv.check_status()


def test_shapes_it_does_not_take():
    a, b, c = _rand(8, 64), _rand(16, 64), _rand(8, 16)
    assert _call(a, [b], [c], 8, 12, 64, [12], N_PARTS) == -3          # columns not a multiple of 8
    assert _call(a, [_rand(40, 16), _rand(24, 16)], [c], 8, 16, 64, [40, 24], K_PARTS,
                 b_mn=1) == -3                                          # a k-block over two weights
    assert _call(a, [b], [c.float()], 8, 16, 64, [16], N_PARTS, fp32=1) == -3
    assert _call(a, [b, b], [], 8, 32, 64, [16, 16], N_PARTS, h=c, kind=2) == -3    # GELU of one product


@pytest.mark.parametrize("T,N,K", [(40, 1024, 2048), (304, 768, 3072), (1000, 2048, 1024)])
@pytest.mark.parametrize("a_mn,b_mn", [(0, 0), (0, 1), (1, 1)])
def test_unsplit_it_has_the_bits_of_the_tile_kernels(T, N, K, a_mn, b_mn):
    from lset_b200.ops.gemm import matmul_abt

    torch.manual_seed(T)
    a = _rand(K, T) if a_mn else _rand(T, K)
    b = _rand(K, N) if b_mn else _rand(N, K)
    dtype = torch.float32 if a_mn else torch.bfloat16
    before = nv.load().lb_gemm_use_2cta(-1)
    out = {}
    for on in (0, 1):
        nv.load().lb_gemm_use_2cta(on)
        out[on] = torch.zeros(T, N, device="cuda", dtype=dtype)
        matmul_abt(a, b, a_mn=bool(a_mn), b_mn=bool(b_mn), out=out[on], accumulate=bool(a_mn))
    nv.load().lb_gemm_use_2cta(before)
    assert torch.equal(out[0], out[1])
    for bn in (64, 128):         # the kernel itself: what the dispatch above takes is the model's choice
        c = torch.zeros_like(out[0])
        assert _call(a, [b], [c], T, N, K, [N], N_PARTS, a_mn=a_mn, b_mn=b_mn, fp32=a_mn, bn=bn,
                     splits=1) == 0
        assert torch.equal(c, out[0]), bn
    nv.check_status()


@pytest.mark.parametrize("T,I,K", [(256, 256, 64), (257, 264, 200), (700, 1160, 1024)])
@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("keep", [True, False])
def test_gated_pair_on_cta_pairs(T, I, K, kind, keep):
    """``lb_gemm_glu_2cta`` has the bits of the two products and the activation kernel."""
    from lset_b200.ops.gemm import matmul_abt

    torch.manual_seed(T)
    lib, a, w = nv.load(), _rand(T, K), _rand(2 * I, K) * 0.1
    gu = matmul_abt(a, w)
    want = torch.empty(T, I, device="cuda", dtype=torch.bfloat16)
    stream = _vp(nv.stream_ptr())
    assert lib.lb_glu_fwd(_ci(kind), _vp(gu.data_ptr()), _vp(gu.data_ptr() + 2 * I), _ll(2 * I),
                          _vp(want.data_ptr()), _ll(I), _ll(T), _ci(I), stream) == 0
    got, h = torch.full_like(gu, float("nan")), torch.full_like(want, float("nan"))
    ptr = got.data_ptr() if keep else 0
    assert lib.lb_gemm_glu_2cta(
        _vp(a.data_ptr()), _vp(w.data_ptr()), _vp(w.data_ptr() + 2 * I * K), _vp(ptr),
        _vp(ptr + 2 * I if keep else 0), _vp(h.data_ptr()), _ci(T), _ci(I), _ci(K), _ll(K), _ll(K),
        _ll(2 * I), _ll(I), _ci(kind), _vp(nv.status_word(a.device).data_ptr()), stream) == 0
    nv.check_status()
    assert torch.equal(h, want)
    assert torch.equal(got, gu) if keep else torch.isnan(got).all()


@pytest.mark.parametrize("M,N,T,half", [(2560, 9728, 5157, 2688), (768, 768, 5096, 2560), (16, 12288, 4096, 2048)])
def test_weight_gradients_over_many_tokens_keep_their_two_pieces(M, N, T, half):
    """Bits of a training step: the first ``half`` of the tokens (whole k-blocks of the kernel's) and the others,
    each summed by itself. (Three pieces and more are added up as they come.)"""
    from lset_b200.ops.gemm import matmul_abt

    torch.manual_seed(T)
    dy, x = _rand(T, M), _rand(T, N)

    def grad(rows):
        out = torch.zeros(M, N, device="cuda")
        return matmul_abt(dy[rows], x[rows], a_mn=True, b_mn=True, out=out, accumulate=True, splits=0)

    assert torch.equal(grad(slice(0, T)), grad(slice(0, half)).add_(grad(slice(half, T))))
    nv.check_status()


@pytest.mark.parametrize("ext,N,T,whole", [
    ([2048, 1024, 1024], 1024, 9096, True), ([2048, 1024, 1024], 1024, 12096, False),
    ([768, 256, 256], 768, 13096, True), ([768, 256, 256], 768, 14096, False),
    ([2048, 512, 512], 2048, 5096, True), ([768, 768, 768], 768, 11096, True)])
def test_which_joint_weight_gradients_are_summed_whole(ext, N, T, whole):
    lib, g = nv.load(), SmallGemm()
    g.A = g.B[0] = 4096
    g.lda, g.ldb[0] = sum(ext), N
    for i, e in enumerate(ext):
        g.C[i], g.ldc[i], g.ext[i] = 4096, N, e
    g.M, g.N, g.K, g.nparts, g.mode = sum(ext), N, T, len(ext), M_PARTS
    g.a_mn = g.b_mn = g.out_fp32 = 1
    plan, tile = lib.lb_gemm_small_plan, lib.lb_gemm_tile_cost
    plan.restype = tile.restype = ctypes.c_double
    cost = plan(ctypes.byref(g), ctypes.byref(_ci()), ctypes.byref(_ci()))
    apart = sum(tile(_ci(e), _ci(N), _ci(T), _ci(1), _ci(0)) for e in ext)
    assert (0 <= cost < apart) == whole
