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
            if "return launch_pdl(" in fn:
                found = re.findall(r"\b\w+_kernel\b", fn)
                assert found, fn[:200]
                names.update(found)
    assert {"gelu_fwd_kernel", "gelu_bwd_kernel", "gemm_small_kernel", "qk_rope_bwd_kernel",
            "attn_fwd_pair_kernel", "rms_fwd_kernel"} <= names
    for name in sorted(names):
        body = _kernel_body(name)
        assert "pdl_wait();" in body, name
        assert 0 <= body.find("pdl_wait();") < body.find("pdl_trigger();"), name
