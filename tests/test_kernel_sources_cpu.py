"""Rules of the CUDA sources that no compiler checks."""
import re
from pathlib import Path

import lset_b200

CSRC = Path(lset_b200.__file__).parent / "csrc"
TEXTS = {p: p.read_text() for p in sorted(CSRC.rglob("*.cu*")) if "_build" not in p.parts}


def _functions(text):
    """Texts of the functions of a file, each from the line after the last closing brace in column
    zero to its own."""
    return re.split(r"\n}[^\n]*\n", text)


def _kernel_body(name):
    for text in TEXTS.values():
        for fn in _functions(text):
            if re.search(r"__global__[^;{]*\b" + name + r"\(", fn):
                return fn
    raise AssertionError(f"no kernel {name}")


def test_kernels_launched_as_programmatic_dependents_wait():
    """A kernel launched with ``launch_pdl`` may start while the one in front of it still runs: it
    has to wait for that kernel's results, and only then let the next one start."""
    names = set()
    for text in TEXTS.values():
        for fn in _functions(text):
            if "launch_pdl(" in fn:
                found = re.findall(r"\b\w+_kernel\b", fn)
                assert found, fn[:200]
                names.update(found)
    assert {"gelu_fwd_kernel", "gelu_bwd_kernel", "gemm_small_kernel", "qk_rope_bwd_kernel",
            "attn_fwd_pair_kernel", "rms_fwd_kernel"} <= names
    for name in sorted(names):
        body = _kernel_body(name)
        assert "pdl_wait();" in body, name
        assert 0 <= body.find("pdl_wait();") < body.find("pdl_trigger();"), name


def test_lanes_of_the_load_warp_of_dkv_agree_on_their_waits():
    """Every wait is bounded, and may run out in some lanes only: all 32 take part in the shuffles
    behind it, so they have to leave the loops together."""
    body = _kernel_body("attn_dkv_kernel")
    loads = body[body.index("if (warp == kDkvMath / 32) {"):
                 body.index("if (warp == kDkvMath / 32 + 1) {")]
    per_item, per_step = loads.split("i < steps && ok;")
    waits = re.findall(r"(.*)mbar_wait\(", per_item)
    assert len(waits) == 2 and all(w.endswith("__all_sync(0xffffffffu, ") for w in waits)
    # lanes that left the inner loop meet the others behind it
    behind = per_step[per_step.index("unsigned drawn"):]
    assert behind.index("ok = __all_sync(0xffffffffu, ok);") < behind.index("__shfl_sync")


def test_every_thread_of_the_small_gemm_waits_before_it_stores():
    """The loading and the issuing warp store results too, and a cluster barrier of the aligned form
    wants whole warps, which the loops in front of it do not leave together."""
    body = _kernel_body("gemm_small_kernel")
    joined = body[:body.index("sum and store")].rsplit("\n  }\n", 1)[1]    # behind the warps' roles
    assert "pdl_wait();" in joined
    text = next(t for t in TEXTS.values() if "void cluster_sync_()" in t)
    barrier = text[text.index("void cluster_sync_()"):]
    assert barrier.index("__syncwarp();") < barrier.index("barrier.cluster.arrive")
