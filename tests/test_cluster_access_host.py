"""Another block's shared memory may be touched only once that block is known to run: every function that turns an address
into another block's has to have passed a barrier of the whole cluster first."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "silicon-violetto_b200" / "csrc"
REMOTE = re.compile(r"\b(sc_remote|map_to_rank|cluster_addr)\(")
WAIT = re.compile(r"\b(sc_)?cluster_sync\(\)|barrier\.cluster\.wait")
HELPERS = {"sc_remote", "map_to_rank", "cluster_addr"}


def functions(text):
    """(name, body) of every function definition outside any other."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"(?:__global__|__device__)[^;{}]*?(\w+)\s*\(", text):
        if m.group(1) in ("__launch_bounds__", "__cluster_dims__", "__align__"):
            head = re.compile(r"(?:__launch_bounds__|__cluster_dims__|__align__)\s*\((?:[^()]|\([^()]*\))*\)|\s+|(\w+)\s*(\(?)")
            at, name = m.start(1), None
            while name is None:
                h = head.match(text, at)
                if h is None:
                    break
                if h.group(1) and h.group(2):
                    name = h.group(1)
                at = h.end()
            if name is None:
                continue
        else:
            name = m.group(1)
        start = text.find("{", m.end())
        semi = text.find(";", m.end())
        if start < 0 or 0 <= semi < start:
            continue
        depth, i = 0, start
        while True:
            depth += (text[i] == "{") - (text[i] == "}")
            i += 1
            if depth == 0:
                break
        yield name, text[start:i]


def all_functions():
    return [(p.name, n, b) for p in sorted(CSRC.glob("*.cu*")) for n, b in functions(p.read_text()) if n not in HELPERS and REMOTE.search(b)]


def test_the_search_finds_the_kernels_that_exchange():
    found = {n for _, n, _ in all_functions()}
    assert {"stats_kernel", "gemm_kernel", "sample_cluster_kernel", "sc_scan", "sc_inverse_cdf_rest"} <= found, found
    assert len({f for f, _, _ in all_functions()}) >= 6


@pytest.mark.parametrize("file,name,body", all_functions(), ids=lambda v: v if len(v) < 60 else "")
def test_a_cluster_barrier_comes_before_the_first_access_to_another_block(file, name, body):
    wait = WAIT.search(body)
    assert wait and wait.start() < REMOTE.search(body).start(), f"{file}: {name} reaches into another block before any cluster barrier"
