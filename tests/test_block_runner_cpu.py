"""Host side of the block runners: what their structs point to, and which blocks they take."""
import ctypes
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


def _stream_struct(ops, monkeypatch, training=True):
    monkeypatch.setattr(ops, "_library", lambda: LIB)
    word = torch.zeros(1, dtype=torch.int32)
    monkeypatch.setattr(ops.nv, "status_word", lambda device=None: word)
    table = torch.zeros(4, 4)
    ctx = SimpleNamespace(plan=Plan(), pos=torch.zeros(5, dtype=torch.int64), tables={},
                          rope=lambda *a: (table, table))
    plan = SimpleNamespace(desc=SimpleNamespace(H=16, hd=64, Hq=2, Hk=1), rope=(64, 1e4, None))
    return ops._stream_struct(ctx, plan, torch.device("cpu"), training)


@pytest.mark.parametrize("ops", [enc_ops, dec_ops])
def test_stream_struct_owns_the_buffers_of_the_backward(ops, monkeypatch):
    """The backward comes later than other callers' passes: a buffer that one of them may replace
    or write is not what the struct can point to."""
    structs = [_stream_struct(ops, monkeypatch) for _ in range(2)]
    sizes = ([("norm_scratch", 8 * 2 * 16), ("wg_tmp", 2 * 16)] if ops is enc_ops else
             [("norm_scratch", 8 * 16), ("rope_scratch", 8 * 2 * 64), ("wg_tmp", 2 * 64)])
    for name, n in sizes:
        at = [ctypes.cast(getattr(s, name), ctypes.c_void_p).value for s in structs]
        for a, s in zip(at, structs):
            assert any(torch.is_tensor(t) and t.data_ptr() <= a
                       and a + 4 * n <= t.data_ptr() + t.nbytes for t in s._keep), name
        assert abs(at[0] - at[1]) >= 4 * n, name
    with torch.no_grad():
        assert not _stream_struct(ops, monkeypatch).norm_scratch
