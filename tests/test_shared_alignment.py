"""Shared arrays that the kernels access by 64-bit or 128-bit loads and stores are
declared with that alignment: a plain array of 4-byte elements has only theirs,
and where the compiler places it is not a property of the source."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "heavyrt_gb300" / "csrc"
WIDE = {"float4": 16, "uint4": 16, "int4": 16, "float2": 8, "uint2": 8, "unsigned long long": 8, "uint64_t": 8}
DECL = re.compile(r"__shared__\s+(__align__\(\d+\)\s+)?([\w ]+?)\s+(\w+)\s*\[")
CAST = re.compile(r"reinterpret_cast<\s*(?:const\s+)?([\w ]+?)\s*\*\s*>\(\s*(\w+)\s*[+)]")


def _too_narrow(text):
    declared = {}
    for align, kind, name in DECL.findall(text):
        given = int(re.search(r"\d+", align).group()) if align else WIDE.get(kind.strip(), 4)
        declared[name] = min(given, declared.get(name, given))
    return [(name, kind) for kind, name in CAST.findall(text) if name in declared and WIDE.get(kind, 0) > declared[name]]


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu*")), ids=lambda p: p.name)
def test_wide_access_needs_a_wide_array(path):
    assert _too_narrow(path.read_text()) == []


def test_the_check_sees_a_plain_array():
    body = "reinterpret_cast<float4*>(s_raw)[q] = x;"
    assert _too_narrow("__shared__ float s_raw[12]; " + body) == [("s_raw", "float4")]
    assert _too_narrow("__shared__ float4 s_raw[3]; " + body) == []
    assert _too_narrow("__shared__ __align__(16) float s_raw[12]; " + body) == []
