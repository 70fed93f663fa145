"""Kernels that are brought up before their predecessor has ended (no GPU).

The compiler may move a read-only load at a known address ahead of
``grid_wait()``, where it would see what was there before the predecessor
wrote.  So a kernel launched with ``launch_dependent``, and the headers its
bond and node phases come from, hold no ``__restrict__`` pointer and no
read-only load, and it waits once, outside any branch, before it reads or
writes memory.
"""
import pathlib
import re

import pytest

CSRC = (pathlib.Path(__file__).resolve().parent.parent
        / "probabilistic_peridynamics_gb300" / "csrc")
READ_ONLY = re.compile(r"__restrict__|__ldg\b|ld\.global\.nc|\bldg_[a-z]")
KERNELS = {(path.name, name) for path in CSRC.glob("*.cu")
           for name in re.findall(r"launch_dependent\((k_\w+)",
                                  path.read_text())}


def _code(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def _body(text, kernel):
    """Parameters and body of the kernel's definition."""
    at = re.search(r"__global__[^;{]*?\b" + kernel + r"\(", text).end()
    start = text.index("{", at)
    depth, end = 0, start
    while True:
        depth += {"{": 1, "}": -1}.get(text[end], 0)
        end += 1
        if depth == 0:
            return text[at:start], text[start:end]


def test_there_are_such_kernels():
    assert {name for _, name in KERNELS} >= {"k_fused_f64", "k_pair_bonds",
                                             "k_pair_nodes"}


@pytest.mark.parametrize("file,kernel", sorted(KERNELS))
def test_no_read_only_loads(file, kernel):
    parameters, body = _body(_code(CSRC / file), kernel)
    assert READ_ONLY.findall(parameters + body) == []
    before, wait, after = body.partition("grid_wait();")
    assert wait and "grid_wait" not in after
    assert before.count("{") - before.count("}") == 1
    assert "return" not in before and "[" not in before.replace(
        "extern __shared__ double s_stack[]", "")


@pytest.mark.parametrize("header", ["pp_bond_f64.cuh", "pp_fused.cuh",
                                    "pp_pairs.cuh"])
def test_headers(header):
    assert READ_ONLY.findall(_code(CSRC / header)) == []
