"""A kernel that lets its successor start does so after it has waited for its predecessor: a
grid that triggers while it still waits admits a further grid of waiting CTAs, which then
fill the SMs unevenly.  Read from the kernels' source."""
import re
from pathlib import Path

CSRC = Path(__file__).parent.parent / "ecs_mhd_2d_b200" / "csrc"


def test_trigger_follows_the_wait():
    seen = 0
    for path in sorted(CSRC.glob("kernels*.cuh")):
        calls = re.findall(r"\bpdl_(wait|trigger)\(\);", re.sub(r"//[^\n]*", "", path.read_text()))
        for i, call in enumerate(calls):
            if call == "trigger":
                seen += 1
                assert i > 0 and calls[i - 1] == "wait", (path.name, i)
    assert seen >= 8
