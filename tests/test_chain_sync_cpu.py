"""Kernels that write another CTA's shared memory: CUDA allows it only while that CTA runs,
so a cluster barrier has to come before the first pass.  Read from the kernels' source,
because a run on hardware does not show a missing barrier reliably."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).parent.parent / "ecs_mhd_2d_b200" / "csrc"
BARRIER = re.compile(r"\b(?:cluster_barrier\(\)|cl\.sync\(\))")


def _functions():
    """(name, body) of every function of the kernel headers, comments taken out."""
    out = []
    for path in sorted(CSRC.glob("kernels*.cuh")):
        src = re.sub(r"//[^\n]*|__(?:launch_bounds|cluster_dims)__\([^)]*\)", "", path.read_text())
        for m in re.finditer(r"^(?:static )?(?:__global__|__device__)[^;{]*?(\w+)\([^;{]*\)\s*\{", src, re.M):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(src[end], 0)
                end += 1
            out.append((m.group(1), src[m.start():m.end()].startswith("__global__"), src[m.end():end - 1]))
    return out


def _remote_writers(functions):
    """Functions that map a peer's shared memory, themselves or through what they call."""
    names = {name for name, _, body in functions if "map_shared_rank" in body}
    while True:
        call = re.compile(r"\b(?:%s)\s*[<(]" % "|".join(sorted(names)))
        more = {name for name, _, body in functions if call.search(body)} - names
        if not more:
            return names
        names |= more


def _before_first_pass(body, names):
    """The part of a kernel's body before its outermost statement with a remote write."""
    first = re.search(r"\bmap_shared_rank\b|\b(?:%s)\s*[<(]" % "|".join(sorted(names)), body).start()
    depth, start = 0, 0
    for i, ch in enumerate(body[:first]):
        depth += {"{": 1, "}": -1, "(": 1, ")": -1}.get(ch, 0)
        if depth == 0 and ch in ";}":
            start = i + 1
    return body[:start]


FUNCTIONS = _functions()
WRITERS = _remote_writers(FUNCTIONS)
CHAINS = [(name, body) for name, kernel, body in FUNCTIONS if kernel and re.fullmatch(r"k_\w+_chain", name)]


def test_every_chain_is_seen():
    assert {n for n, _ in CHAINS} == {"k_tan_chain", "k_rk4_chain", "k_fx_chain", "k_adj_chain", "k_tdj_chain", "k_rk43_chain"}
    assert {n for n, _ in CHAINS} <= WRITERS


@pytest.mark.parametrize("name,body", CHAINS, ids=[n for n, _ in CHAINS])
def test_cluster_barrier_before_the_first_pass(name, body):
    assert BARRIER.search(_before_first_pass(body, WRITERS)), name


def test_cluster_sum_waits_for_its_peers():
    body = next(b for n, _, b in FUNCTIONS if n == "cluster_sum2")
    assert BARRIER.search(body[:body.index("map_shared_rank")])
