"""An array is read or written in place only where all of it is reached: the
comparison of the attributes of its first and last byte, on the host, with the
answers that the runtime gives for arrays that are page-locked or allocated as a
whole, in their first part only, in two blocks, or on two devices; and the
callers, which ask for the array's length."""
import re
import subprocess
from pathlib import Path

from heavyrt_gb300 import native_build

CSRC = Path(__file__).resolve().parents[1] / "heavyrt_gb300" / "csrc"

SOURCE = r"""
#include <cstdio>
#include "input_range.h"

static cudaPointerAttributes at(cudaMemoryType type, int device, uintptr_t address)
{
  cudaPointerAttributes a = {};
  a.type = type;
  a.device = device;
  a.devicePointer = (void*)address;
  return a;
}

int main()
{
  using hrt::api::same_block;
  const auto H = cudaMemoryTypeHost, D = cudaMemoryTypeDevice, U = cudaMemoryTypeUnregistered;
  std::printf("%d%d%d%d%d%d%d%d%d\n", same_block(at(H, 0, 4096), at(H, 0, 5095), 1000),  // whole
              same_block(at(D, 0, 4096), at(D, 0, 5095), 1000),                           // whole
              same_block(at(H, 0, 4096), at(H, 0, 4096), 1),                              // one byte
              same_block(at(H, 0, 4096), at(U, 0, 0), 1000),                              // locked in part
              same_block(at(H, 0, 4096), at(H, 0, 9191), 1000),                           // two mappings
              same_block(at(D, 0, 4096), at(U, 0, 0), 1000),                              // past the allocation
              same_block(at(D, 0, 4096), at(D, 1, 5095), 1000),                           // another device's
              same_block(at(D, 0, 4096), at(H, 0, 5095), 1000),                           // another kind
              same_block(at(H, 0, 0), at(H, 0, 0), 1));                                   // not mapped
  return 0;
}
"""


def test_the_whole_array_decides(tmp_path):
    src = tmp_path / "range.cpp"
    src.write_text(SOURCE)
    include = Path(native_build._nvcc()).resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-I", str(CSRC), "-I", str(include), str(src), "-o",
                    str(tmp_path / "range")], check=True)
    out = subprocess.run([str(tmp_path / "range")], check=True, capture_output=True, text=True).stdout
    assert out.strip() == "111000000"


def test_every_caller_gives_a_length():
    seen = 0
    for path in sorted(CSRC.glob("*.cu*")):
        for name, args in re.findall(r"\b(mapped_host|input_in_place)\(([^;]*?)\)\s*(?:[:);]|\?)", path.read_text()):
            want = 2 if name == "mapped_host" else 3
            assert args.count(",") >= want - 1, (path.name, name, args)
            seen += 1
    assert seen >= 8
