"""Kernels that are launched behind one another without waiting for the end of
the launch before (launch_chained, csrc/engine.hpp): each waits (chain_wait)
before it reads anything, and takes no `__restrict__` pointer - the qualifier
lets the compiler read through the path that assumes nobody writes the data
while the kernel is resident, which the launch before still does."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "idefix_gb300", "csrc")


def _sources():
    out = {}
    for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*")) + glob.glob(os.path.join(CSRC, "*.hpp"))):
        with open(p) as f:
            out[os.path.basename(p)] = re.sub(r"//[^\n]*", "", f.read())
    return out


def _kernels(text):
    """(name, head up to the body, body) of every __global__ definition"""
    for m in re.finditer(r"__global__", text):
        brace = text.find("{", m.end())
        semi = text.find(";", m.end())
        if brace < 0 or 0 <= semi < brace:
            continue  # a declaration
        head = text[m.end():brace]
        depth, end = 0, brace
        while True:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
            if depth == 0:
                break
        name = re.findall(r"\b(ke?_\w+)\s*\(", head)
        if name:
            yield name[0], head, text[brace + 1:end - 1]


SOURCES = _sources()
KERNELS = {n: (h, b) for t in SOURCES.values() for n, h, b in _kernels(t)}
WAITING = sorted(n for n, (_, b) in KERNELS.items() if "chain_wait()" in b)


def _launched():
    names = set()
    for t in SOURCES.values():
        names |= set(re.findall(r"launch_chained\(\s*[\w.>-]+,\s*(ke?_\w+)", t))
        names |= set(re.findall(r"launch_kernel\(\s*[\w.>-]+,\s*[\w.>-]+,\s*(ke?_\w+)", t))
        names |= set(re.findall(r"IDFX_CHAIN_DE?\(\s*(ke?_\w+)", t))
    return names


def test_the_chained_kernels_are_found():
    assert len(WAITING) >= 15 and _launched() and _launched() <= set(WAITING)


@pytest.mark.parametrize("name", WAITING)
def test_chained_kernel_reads_coherently_after_its_wait(name):
    head, body = KERNELS[name]
    assert "__restrict__" not in head
    before = [s.strip() for s in body[:body.index("chain_wait()")].split(";")]
    for s in before:  # declarations of shared memory and types alone
        assert s == "" or re.match(r"(extern\s+)?__shared__|constexpr|using", s), s
