"""Kernels of a chain of overlapping launches (chain.cuh) read what the kernel before them writes by
ordinary loads.  Read-only loads (`__ldg`, `ld.global.nc`, and `const ... __restrict__` parameters, whose
loads a compiler may turn into such) are for memory that nothing writes during the kernel's life; in a
chain only the matrix is that.  Checked in the sources, since a run that goes right shows nothing."""
import glob
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "vhci_b200", "csrc")
MATRIX = {"rowptr", "col", "val", "diag"}  # complete before the chain that multiplies by it begins


def _strip(src):
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", src, flags=re.S)


def _functions(src, head):
    """(name, parameters, body) of every function whose declaration matches `head`."""
    for m in re.finditer(head + r"[^;{}]*?\b(\w+)\s*\(", src):
        if m.group(1) == "__launch_bounds__":
            m = re.compile(r"\)\s*(\w+)\s*\(").search(src, m.end())
        i = m.end()
        depth = 1
        while depth:
            depth += {"(": 1, ")": -1}.get(src[i], 0)
            i += 1
        params = src[m.end():i - 1]
        j = k = src.index("{", i)
        depth = 0
        while True:
            depth += {"{": 1, "}": -1}.get(src[k], 0)
            k += 1
            if depth == 0:
                break
        yield m.group(1), params, src[j:k]


def _read_only(params, body):
    """What the function reads through the read-only path: parameter names and load addresses."""
    found = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params))
    found |= set(re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\(\s*)?(\w+)", body))
    if re.search(r"\.nc\b", body):
        found.add("ld.global.nc")
    return found


def _chained():
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        src = _strip(open(path).read())
        for name, params, body in _functions(src, r"__global__\s+void"):
            if "chain_wait()" in body:
                out.append((os.path.basename(path) + ":" + name, params, body))
    return out


CHAINED = _chained()


def test_every_chained_launch_is_covered():
    launched = set()
    for path in glob.glob(os.path.join(CSRC, "*.cu")):
        src = _strip(open(path).read())
        launched |= set(re.findall(r"launch_chained\(\s*(\w+)", src))
    assert launched == {name.split(":")[1] for name, _, _ in CHAINED} and len(launched) >= 15


@pytest.mark.parametrize("name,params,body", CHAINED, ids=[c[0] for c in CHAINED])
def test_chained_kernel_loads(name, params, body):
    assert _read_only(params, body) <= MATRIX


def test_helpers_of_chained_kernels():
    """The row product reads the vector block, and load4 the tall operand, by ordinary loads."""
    src = _strip(open(os.path.join(CSRC, "rowprod.cuh")).read())
    (name, params, body), = [f for f in _functions(src, r"__device__ __forceinline__ void") if f[0] == "row_product"]
    assert _read_only(params, body) <= MATRIX
    src = _strip(open(os.path.join(CSRC, "k_proj.cu")).read())
    (name, params, body), = [f for f in _functions(src, r"__device__ __forceinline__ void") if f[0] == "load4"]
    assert not _read_only(params, body)
