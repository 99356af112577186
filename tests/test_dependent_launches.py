"""Kernels that launch_after starts run while the kernel before them still writes: each
waits for it first, and nothing that they execute loads through the read-only path
(__ldg, ld.global.nc, or a __restrict__ pointer, from which the compiler may choose it),
which wants memory that nobody writes while the kernel lives.  Read from the sources."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fluid-simulation_gb300", "csrc")
READ_ONLY = re.compile(r"__ldg\b|\bld\.global\.nc\b|__restrict__")


def source(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def functions(text):
    """{name: [argument lists and bodies]} of the functions defined in a source text."""
    found = {}
    for m in re.finditer(r"\b(\w+)\s*\(", text):
        if m.group(1) in ("if", "for", "while", "switch", "return", "sizeof", "__launch_bounds__", "asm", "volatile"):
            continue
        depth, i = 1, m.end()
        while depth and i < len(text):
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        tail = re.match(r"\s*(const\s*)?(:[^{;]*)?\{", text[i:])
        if not tail:
            continue
        depth, j = 1, i + tail.end()
        while depth and j < len(text):
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        found.setdefault(m.group(1), []).append(text[m.start():j])
    return found


def dependent_kernels():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        for name in sorted(set(re.findall(r"\blaunch_after\(\s*(\w+)", source(path)))):
            yield os.path.basename(path), name


KERNELS = list(dependent_kernels())


def test_there_are_some():
    assert len(KERNELS) >= 16 and ("fl_g2p.cu", "k_g2p") in KERNELS


@pytest.mark.parametrize("file,kernel", KERNELS)
def test_waits_first_and_loads_plainly(file, kernel):
    text = source(os.path.join(CSRC, file)) + "".join(source(p) for p in glob.glob(os.path.join(CSRC, "*.cuh")))
    defined = functions(text)
    body = defined[kernel][0]
    statements = body[body.index("{") + 1:].lstrip()
    assert statements.startswith("after_previous();")
    seen, todo = set(), [kernel]
    while todo:
        name = todo.pop()
        if name in seen:
            continue
        seen.add(name)
        for code in defined[name]:
            assert not READ_ONLY.search(code), (kernel, name)
            todo += [n for n in set(re.findall(r"\b(\w+)\b", code)) if n in defined]
