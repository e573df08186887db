"""Kernels launched with programmatic stream serialization live while the kernel before them still writes: their source may
not promise the compiler read-only memory for what such a kernel writes (the reason stands at pdl_wait in common.cuh)."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mgpt_b200", "csrc")
FILES = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))

# Non-coherent loads of operands that another kernel of the same call separates from their writer.
SEPARATED = {
    "decode.cu": {"p.b0[", "p.b1["},                                        # biases: router and plan lie between
    "gemm_tc.cu": {"b4 + q", "chunk0 + q", "p.gather_pos", "reinterpret_cast<const uint4*>(p.gather_src"},
    "router_tc.cu": {"p.br +"},                                             # router_copies_kernel reads it first
}


def _code(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_no_kernel_parameter_promises_read_only_memory(path):
    for m in re.finditer(r"__global__[^{;]*\{", _code(path)):
        assert "__restrict__" not in m.group(0), " ".join(m.group(0).split())[:120]


@pytest.mark.parametrize("path", FILES, ids=os.path.basename)
def test_non_coherent_loads_are_of_separated_operands(path):
    allowed = SEPARATED.get(os.path.basename(path), set())
    for m in re.finditer(r"__ldg\(([^;\n]*)", _code(path)):
        assert any(m.group(1).startswith(a) for a in allowed), m.group(0)
    if os.path.basename(path) != "decode.cu":                               # its weight stream
        assert "ld.global.nc" not in _code(path)
