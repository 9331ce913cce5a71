"""Kernels that start before the kernel ahead has ended (they call pdl_wait) read what that one writes.
A `const T* __restrict__` parameter lets the compiler load through the read-only path, which is defined
only for data that nothing writes while the kernel is resident: such parameters may only be what no
kernel of the chain writes.  Read from the sources; no GPU is needed."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "neon_b200" / "csrc"
CONSTANT = {"inv", "mask"}  # written before the chain starts, never within it
OUTPUT = {"k_csr_spmv": {"q"}}  # only written by the kernel


def _close(text, i):
    """The place behind the bracket that closes the one opened just before i."""
    depth = 1
    while depth:
        depth += {"(": 1, "{": 1, ")": -1, "}": -1}.get(text[i], 0)
        i += 1
    return i


def _kernels(text):
    """(name, parameters, body) of every __global__ function."""
    for m in re.finditer(r"__global__\s+void\b", text):
        at = re.compile(r"\s*(\w+)\s*\(").match(text, m.end())
        if at.group(1) == "__launch_bounds__":
            at = re.compile(r"\s*(\w+)\s*\(").match(text, _close(text, at.end()))
        end = _close(text, at.end())
        body = text.index("{", end)
        yield at.group(1), text[at.end():end], text[body:_close(text, body + 1)]


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.cu*")))
def test_early_kernels_have_no_restricted_vectors(source):
    text = re.sub(r"//[^\n]*", "", (CSRC / source).read_text())
    for name, params, body in _kernels(text):
        if "pdl_wait()" not in body:
            continue
        restricted = set(re.findall(r"__restrict__\s+(\w+)", params))
        assert restricted <= CONSTANT | OUTPUT.get(name, set()), name
        for q in OUTPUT.get(name, ()):
            assert re.search(r"const[^,]*\b%s\b" % q, params) is None
            assert re.findall(r"\b%s\b(?!\[\w+\] = )" % q, body) == []


def test_the_early_kernels_are_found():
    found = {name for p in CSRC.glob("*.cu*")
             for name, _, body in _kernels(re.sub(r"//[^\n]*", "", p.read_text()))
             if "pdl_wait()" in body}
    assert {"k_csr_spmv", "k_xr", "k_p", "k_mf_apply", "k_mf_gather", "k_mf_xr", "k_mf_p",
            "k_element"} <= found
