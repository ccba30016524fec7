"""Functions of the native implementation that return a status consume the CUDA error they
report, so a caller that drops the status reports success for a launch that failed.  Read
from the source: a launch that fails on purpose is no test for a GPU."""
import re
from pathlib import Path

CSRC = Path(__file__).parent.parent / "ecs_mhd_2d_b200" / "csrc"


def _source(name):
    return re.sub(r"//[^\n]*", "", (CSRC / name).read_text())


def _dropped(src, names):
    """Calls of `names` that are statements of their own."""
    call = re.compile(r"(?<=[;{})])\s*(?:else\s+)?(\w+)(?:<[^;(]*>)?\([^;]*;")
    return [m.group(0).strip() for m in call.finditer(src) if m.group(1) in names]


def test_no_status_is_dropped():
    src = _source("impl.cuh")
    names = set(re.findall(r"static int (\w+)\(", src)) | {"cuda_err", "grow"}
    assert {"rk4_chain", "rk4_setup", "fx_chain", "adj_chain", "integrate_rk4", "residual"} <= names
    assert _dropped(src, names) == []


def test_no_launch_wrapper_is_void_over_a_status():
    """A void function that calls one with a status has nowhere to put it."""
    src = _source("impl.cuh")
    names = set(re.findall(r"static int (\w+)\(", src))
    for m in re.finditer(r"static (?:void|const cplx<R>\*) (\w+)\([^;{]*\)\s*\{", src):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(src[end], 0)
            end += 1
        called = set(re.findall(r"\b(\w+)\(", src[m.end():end])) & names
        assert not called - {"fx_scheme"}, (m.group(1), called)
