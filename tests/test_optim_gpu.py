"""The optimiser kernels over lists of buffers, against the same update in 64 bits."""
import ctypes

import pytest
import torch

from lset_b200.dist.sharded import LbOptGroup
from lset_b200.ops import _native as nv

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[1], [4096, 3, 8193], [5 + 97 * i for i in range(95)]])
def test_lists_of_buffers(sizes):
    """Buffers of one element, of a chunk, of remainders, and more of them than a launch takes."""
    torch.manual_seed(len(sizes))
    lib, n = nv.load(), len(sizes)
    p, g, m = ([torch.randn(k, device="cuda") for k in sizes] for _ in range(3))
    v = [torch.rand(k, device="cuda") + 0.1 for k in sizes]
    low = [torch.zeros(k, device="cuda", dtype=torch.bfloat16) for k in sizes]
    groups = (LbOptGroup * n)()
    for i, e in enumerate(groups):
        e.p, e.g, e.m, e.v, e.p_bf16 = (t[i].data_ptr() for t in (p, g, m, v, low))
        e.n, e.slot = sizes[i], i % 2
    scratch = torch.empty(lib.lb_sumsq_scratch_floats(nv.c_int(n)), device="cuda")
    out = torch.empty(2, device="cuda")
    stream = nv.c_void_p(nv.stream_ptr())
    assert lib.lb_sumsq_groups(groups, nv.c_int(n), nv.c_void_p(scratch.data_ptr()),
                               nv.c_void_p(out.data_ptr()), stream) == 0
    for slot in (0, 1):     # fp32 sums of positive terms, in chunks
        want = sum(float(x.double().square().sum()) for x in g[slot::2])
        assert abs(out[slot].item() - want) <= 1e-5 * want
    lr, b1, b2, eps, wd, step = 1e-2, 0.9, 0.99, 1e-8, 0.1, 3
    want = []
    for a, b, c, d in zip(p, g, m, v):
        a, b, c, d = (t.double() for t in (a, b, c, d))
        c = b1 * c + (1 - b1) * b
        d = b2 * d + (1 - b2) * b * b
        a = a * (1 - lr * wd) - lr / (1 - b1 ** step) * c / ((d / (1 - b2 ** step)).sqrt() + eps)
        want.append((a, c, d))
    f = nv.c_float
    assert lib.lb_adamw_groups(groups, nv.c_int(n), f(lr), f(b1), f(b2), f(eps), f(wd), f(1 - b1 ** step),
                               f((1 - b2 ** step) ** 0.5), f(1.0), ctypes.c_void_p(0), nv.c_int(1), stream) == 0
    for i, (a, c, d) in enumerate(want):     # a dozen fp32 roundings of values of order one
        for got, ref in ((p[i], a), (m[i], c), (v[i], d)):
            assert torch.allclose(got.double(), ref, rtol=2e-6, atol=2e-6)
        assert torch.equal(low[i], p[i].to(torch.bfloat16))
        assert not g[i].any()


def _sums_of_squares(lib, tensors, slots):
    groups = (LbOptGroup * len(tensors))()
    for e, t, slot in zip(groups, tensors, slots):
        e.g, e.n, e.slot = t.data_ptr(), t.numel(), slot
    n = nv.c_int(len(tensors))
    scratch = torch.empty(lib.lb_sumsq_scratch_floats(n), device="cuda")
    out = torch.empty(2, device="cuda")
    assert lib.lb_sumsq_groups(groups, n, nv.c_void_p(scratch.data_ptr()), nv.c_void_p(out.data_ptr()),
                               nv.c_void_p(nv.stream_ptr())) == 0
    return out.cpu()


def test_sums_of_squares_are_added_buffer_by_buffer():
    """Bits of the gradient norm, hence of every clipped step: the sum of each buffer by itself (whatever else
    is in the list), one after the other."""
    torch.manual_seed(0)
    lib = nv.load()
    tensors = [torch.randn(5 + 7919 * i, device="cuda") for i in range(60)]
    tensors += [torch.randn(5_000_003, device="cuda"), torch.randn(8, device="cuda")]
    slots = [int(i % 5 == 2) for i in range(len(tensors))]
    want = torch.zeros(2)
    for t, slot in zip(tensors, slots):
        want[slot] += _sums_of_squares(lib, [t], [slot])[slot]
    assert torch.equal(_sums_of_squares(lib, tensors, slots), want)
