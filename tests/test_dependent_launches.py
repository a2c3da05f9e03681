"""Kernels launched as programmatic dependents may run while the kernels
before them still write.  What those write they must not declare as read-only
for their own lifetime (const ... __restrict__) nor read by __ldg.  Read from
the sources; no GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(
    __file__))), "inovesa_gb300", "csrc")

# kernel: its parameters that a kernel before it in the chain may be writing
CHAIN = {
    "k_rotation": ["in"], "k_kick_y": ["in", "offsets"],
    "k_kick_x": ["in", "offsets"], "k_kick_y4": ["in", "offsets"],
    "k_kick_table": ["offsets"], "k_kick_x4": ["in", "shtab", "wtab"],
    "k_fp": ["in"], "k_fp4": ["in"], "k_dynrf": [],
    "k_project_x": ["data"], "k_project_y": ["data"],
    "k_integrate": ["proj64"], "k_normalize": ["data", "filling"],
    "k_moments": ["proj", "filling"], "k_wake": ["proj"], "k_csr": ["proj"],
    # the batch's maps kernels beside k_bwake
    "k_bmaps1": ["wake", "factor"], "k_bstrip": ["rinfo"],
}
# tables that stand before any chain begins (and the density that k_bmaps1
# reads, complete before k_bwake lets it start)
TABLES = {"qv", "ws", "wtab", "tw", "d4", "w4", "src"}


def sources():
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as h:
                out[f] = re.sub(r"//[^\n]*", "", h.read())
    return out


def kernel(name):
    """(parameters, body) of a __global__ function."""
    for text in sources().values():
        m = re.search(r"\b%s\(([^)]*)\)\s*\{" % name, text)
        if m and "__global__" in text[max(0, m.start() - 160):m.start()]:
            depth, i = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(text[i], 0)
                i += 1
            return [p.strip() for p in m[1].split(",")], text[m.end():i]
    raise AssertionError(name)


@pytest.mark.parametrize("name", sorted(CHAIN))
def test_chain_reads_are_ordinary(name):
    params, body = kernel(name)
    for want in CHAIN[name]:
        (p,) = [q for q in params if re.search(r"\b%s$" % want, q)]
        assert not ("const" in p and "__restrict__" in p), p
        assert not re.search(r"__ldg\(\s*(reinterpret_cast<[^>]*>\(\s*)?%s\b"
                             % want, body), (name, want)
    if name != "k_bmaps1":
        for arg in re.findall(
                r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\(\s*)?(\w+)", body):
            assert arg in TABLES - {"src"}, (name, arg)


def test_every_dependent_launch_is_listed():
    names = set()
    for text in sources().values():
        for m in re.finditer(r"pdl_launch\(\s*([^,]*),", text):
            names |= set(re.findall(r"k_\w+", m[1]))
    assert names and names <= set(CHAIN) | {"kernel"}, names
