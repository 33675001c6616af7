"""Kernels that may start before their predecessor in the stream has ended: they wait for it before they read, and
nothing in them lets the compiler take what the predecessor writes for constant (const __restrict__ arguments and
__ldg go through the read-only path, which holds for data that no one writes during the kernel's whole life).
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpsdyn_b200", "csrc")


def bracket(text, i, pair):
    """The index behind the bracket that closes the one at i."""
    depth = 0
    for j in range(i, len(text)):
        depth += (text[j] == pair[0]) - (text[j] == pair[1])
        if depth == 0:
            return j + 1
    raise ValueError("open bracket")


def functions(text):
    """(name, arguments, body, whether a kernel) of every device function of a source."""
    for m in re.finditer(r"__(?:global|device)__", text):
        end = text.find("{", m.end())
        head = re.sub(r"__(?:launch_bounds|cluster_dims|align)__\s*\((?:[^()]|\([^()]*\))*\)", "", text[m.end():end])
        name = re.search(r"(\w+)\s*\(", head)
        if end < 0 or ";" in head or not name:
            continue
        yield name.group(1), head[name.end() - 1:], text[end:bracket(text, end, "{}")], m.group() == "__global__"


SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", SOURCES)
def test_chained_kernels_wait_and_read_plainly(name):
    text = source(name)
    found = {f: (a, b) for f, a, b, _ in functions(text)}
    waits = {f for f, (_, b) in found.items() if re.search(r"\b(join_stream|await_predecessor)\(\)", b)}
    for kernel in set(re.findall(r"launch_chained\(st,\s*(\w+)", text)):
        assert kernel in waits, f"{kernel} is launched early and does not wait"
        # with the functions of the same source that it calls
        todo, seen = [kernel], set()
        while todo:
            f = todo.pop()
            seen.add(f)
            args, body = found[f]
            assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", args), f"{kernel}: read-only argument of {f}"
            assert "__ldg(" not in body and "ld.global.nc" not in body, f"{kernel}: read-only load in {f}"
            todo += [g for g in found if g not in seen and g not in todo and re.search(r"\b%s\s*(<[^;{}()]*>)?\(" % g, body)]
