"""Loads of the step's chained kernels, read from the source.

A kernel that is launched with programmatic stream serialization may start
while the kernel before it still writes; only after chain_begin()'s wait is the
memory its own.  `__ldg` and pointers that a kernel takes as `__restrict__`
promise that nobody writes the memory for as long as the kernel lives, which
lets the compiler load through the non-coherent path, or before the wait.
Chained kernels therefore begin with chain_begin() and make no such promise.
"""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "n-body-2d_b200" / "csrc"
FILES = ["k_sort.cu", "k_tree.cu", "k_force32.cu", "k_force64.cu", "k_allpairs.cu"]


def _kernels(text):
    """(name, parameters, body) of the file's kernels."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?"
                         r"(\w+)\(([^)]*)\)\s*\{", text):
        depth, end = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            end += 1
        yield m.group(1), m.group(2), text[m.end():end - 1]


def _launched_chained(text):
    """Kernel names that the file gives to chain_launch (by name, or through a
    function pointer picked just before)."""
    names = {m.group(1) for m in re.finditer(r"__global__[^;{]*?(\w+)\([^)]*\)\s*\{", text)}
    calls = " ".join(re.findall(r"chain_launch\([^;]*;", text))
    calls += " ".join(re.findall(r"auto\* \w*kernel = [^;]*;", text))
    return {n for n in names if re.search(rf"\b{n}\b", calls)}


@pytest.mark.parametrize("name", FILES)
def test_chained_kernels_wait_first_and_load_plainly(name):
    text = (CSRC / name).read_text()
    chained = [k for k in _kernels(text) if "chain_begin();" in k[2]]
    assert chained
    assert _launched_chained(text) <= {k[0] for k in chained}
    for kernel, params, body in chained:
        assert re.match(r"\s*(?:nb::)?chain_begin\(\);", body), f"{kernel} does not wait first"
        assert "__restrict__" not in params, f"{kernel} promises memory that the chain writes"
    code = re.sub(r"//[^\n]*", "", text)
    assert not re.search(r"__ldg\b|ld\.global\.nc", code), f"{name}: a non-coherent load"
