"""Kernels that start while the launch before them still runs (programmatic dependents) read what that
launch writes with plain loads: the read-only path (__ldg, const __restrict__ parameters) is for data
that nobody writes during the kernel, and no wait orders it."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "dumux_gb300", "csrc")
# finished before the chain of Krylov kernels starts: the matrix, its mask, factor and pivots
READ_ONLY = re.compile(r"(a\.)?(A|LU|Lf|Dinv|mask|nbmask)\b|p\b|reinterpret_cast<const (float4|double2)\*>\(p\)")


def _chained_kernels():
    found = []
    for name in sorted(os.listdir(CSRC)):
        if not name.endswith(".cu"):
            continue
        text = open(os.path.join(CSRC, name)).read()
        names = set(re.findall(r"launchChained\((\w+)", text)) - {"void"}
        if "cudaLaunchAttributeProgrammaticStreamSerialization" in text:
            names |= {k for k in ("lanePackApply", "stencilPackApply", "stencilPlaneApply", "amgClusterCycle",
                                  "laneWaveKernel", "laneRingKernel") if re.search(r"__global__[^;{]*\b%s\(" % k, text)}
        for k in sorted(names):
            m = re.search(r"__global__[^;{]*?\b%s\((.*?)\)\s*\{(.*?)\n\}" % k, text, re.S)
            assert m, (name, k)
            found.append((name, k, m.group(1), m.group(2)))
    return found


@pytest.mark.parametrize("unit,kernel,params,body", _chained_kernels(), ids=lambda v: v if len(v) < 30 else "")
def test_operands_written_inside_the_chain_are_read_with_plain_loads(unit, kernel, params, body):
    for p in params.split(","):
        assert not ("const" in p and "__restrict__" in p), p
    assert not re.search(r"const \w+\* ?__restrict__", body)
    for arg in re.findall(r"__ldg\(([^;]*)", body):
        assert READ_ONLY.match(arg), arg


def test_vector_loads_of_the_krylov_kernels_do_not_take_the_read_only_path():
    text = open(os.path.join(CSRC, "linalg.cu")).read()
    body = re.search(r"void ldVec\(const T\* p, T\* o\)\s*\{(.*?)\n\}", text, re.S).group(1)
    assert "__ldg" not in body
