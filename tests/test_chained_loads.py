"""Kernels launched as programmatic dependents (csrc/snntc_launch.cuh) are on the SMs while the kernel in front of them may
still be writing what they read. The read-only path -- __ldg, ld.global.nc, or any load through a `const T* __restrict__`
kernel parameter -- is defined for memory that nobody writes during the whole life of a kernel, so such a kernel must not
use it. Checked on the sources: a race is not a thing to provoke on a GPU."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "snntc_2023_b200", "csrc")
READ_ONLY = re.compile(r"__ldg\s*\(|\bld\.global\.nc|const\s+\w+(?:\s+\w+)?\s*\*\s*__restrict__|\b__ldc[gs]\s*\(")


def _strip_comments(text):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def _kernels(text):
    """(name, header and body) of every __global__ function of a source text."""
    for m in re.finditer(r"__global__", text):
        attributes = {"__launch_bounds__", "__cluster_dims__"}
        name = next(n for n in re.finditer(r"(\w+)\s*\(", text[m.end():]) if n.group(1) not in attributes).group(1)
        depth, end = 0, text.index("{", m.end())
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        yield name, text[m.start():end]


def _sources():
    return sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def test_the_scan_sees_the_kernels():
    """Every kernel that is launched as a dependent is found, and begins with the wait."""
    launched, found = set(), {}
    for f in _sources():
        text = _strip_comments(open(os.path.join(CSRC, f)).read())
        launched |= set(re.findall(r"launch_chained\(\s*(\w+_kernel)", text))
        found.update(_kernels(text))
    launched.add("snn_walk_ring_kernel")      # handed to launch_chained as an argument
    assert len(launched) > 25 and launched <= set(found), sorted(launched - set(found))
    for name in launched:
        assert "chain_wait();" in found[name], name


@pytest.mark.parametrize("source", _sources())
def test_no_read_only_loads_in_chained_kernels(source):
    text = _strip_comments(open(os.path.join(CSRC, source)).read())
    if source == "snntc_launch.cuh":          # where ld_readonly is defined: the one exception, held to its rule below
        text = text.replace("return __ldg(p);", "", 1)
    unchained = set(re.findall(r"\b(\w+_kernel)(?:<[\w, ]+>)?\s*<<<", text))
    for name, body in _kernels(text):
        if name in unchained and "chain_wait" not in body:
            text = text.replace(body, "")     # launched in plain stream order: nothing in front of it is still running
    assert not READ_ONLY.findall(text), [m.group(0) for m in READ_ONLY.finditer(text)]


def test_the_read_only_path_only_where_nothing_is_still_running():
    """Kernels that read by ld_readonly are launched in plain stream order, never as dependents; every kernel that lets its
    successor onto the SMs early has waited for its own predecessor first."""
    for f in _sources():
        text = _strip_comments(open(os.path.join(CSRC, f)).read())
        chained = set(re.findall(r"launch_chained\(\s*(\w+_kernel)", text)) | {"snn_walk_ring_kernel"}
        plain = set(re.findall(r"\b(\w+_kernel)(?:<[\w, ]+>)?\s*<<<", text))
        for name, body in _kernels(text):
            if "chain_next" in body:
                assert body.index("chain_wait();") < body.index("chain_next();"), name
            if "ld_readonly" in body:
                assert name in plain and name not in chained, name
