"""Loads of the kernels that are launched before their predecessor has ended.

A kernel launched with launch_chained() (csrc/launch.cuh) is resident while
the kernel before it still writes, so its inputs are not read-only for its
lifetime: the non-coherent path (``__ldg``, ``ldg3``) is closed to it, and so
is ``__restrict__`` on a pointer that it reads, which lets the compiler choose
that path and move the load over the wait.  Read from the sources: a wrong
load need not show in a run.
"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "cross-denoiser_b200", "csrc")
FILES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    text = re.sub(r"/\*.*?\*/", " ", text, flags=re.S)
    text = re.sub(r"//[^\n]*", " ", text)
    return re.sub(r"CD_DEV float3 ldg3\(.*?\n}", " ", text, flags=re.S)   # the helper's own definition


def kernels(text):
    """(name, parameters, body, start, end) of every __global__ function defined in text."""
    out = []
    for m in re.finditer(r"__global__", text):
        brace = text.index("{", m.end())
        head = text[m.end():brace]
        if ";" in head:
            continue
        depth, i = 1, brace + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        head = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", " ", head)
        name, params = re.match(r"\s*void\s+(\w+)\s*\((.*)\)\s*$", head, re.S).groups()
        out.append((name, params, text[brace:i], m.start(), i))
    return out


CHAINED_FILES = [f for f in FILES if f.endswith(".cu") and "launch_chained(" in source(f)]


def test_there_are_chained_kernels():
    assert len(CHAINED_FILES) >= 7


@pytest.mark.parametrize("name", CHAINED_FILES + [f for f in FILES if f.endswith(".cuh")])
def test_no_non_coherent_load(name):
    text = source(name)
    rest = text
    for _, _, body, start, end in reversed(kernels(text)):
        if "chain_wait();" not in body:       # starts after its predecessor's end: any load will do
            rest = rest[:start] + rest[end:]
    for bad in (r"__ldg\(", r"\bldg3\(", r"ld\.global\.nc", r"\bconst\b[^,;(){}]*\*\s*__restrict__"):
        assert not re.search(bad, rest), f"{name}: {re.search(bad, rest).group(0)!r} in chained code"


@pytest.mark.parametrize("name", CHAINED_FILES)
def test_restrict_marks_outputs_only(name):
    """A __restrict__ parameter of a chained kernel is written, never read in place."""
    for kernel, params, body, _, _ in kernels(source(name)):
        if "chain_wait();" not in body:
            continue
        for p in re.findall(r"__restrict__\s*(\w+)", params):
            reads = re.findall(rf"(?<![\w.>]){p}\s*\[[^\]]*\]\s*(?!\s*=[^=])", body)
            assert not reads, f"{name}: {kernel} reads its __restrict__ parameter {p}: {reads}"


@pytest.mark.parametrize("name", CHAINED_FILES)
def test_wait_comes_before_every_pointer_parameter(name):
    """chain_wait() stands in every kernel launched by name with launch_chained(),
    and no pointer parameter is used before it."""
    text = source(name)
    found = {k: (params, body) for k, params, body, _, _ in kernels(text)}
    for k in re.findall(r"launch_chained\(\s*(\w+_kernel)\b", text):
        assert "chain_wait();" in found[k][1], f"{name}: {k} is launched chained and never waits"
    for k, (params, body) in found.items():
        if "chain_wait();" not in body:
            continue
        before = body[:body.index("chain_wait();")]
        for p in re.findall(r"\*\s*(?:__restrict__\s*)?(\w+)", params):
            assert not re.search(rf"\b{p}\b", before), f"{name}: {k} uses {p} before its wait"
