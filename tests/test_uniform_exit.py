"""A kernel whose own waits set the error word must not let its threads leave on that word one by one: the
word may change between the reads of two warps, and the warps that stay would wait for those that left at the
next counted barrier. Such kernels vote (__syncthreads_or) or let one thread read it for all. Read from the
sources, as the race itself would hang a GPU."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "libxstream_b200" / "csrc"


def kernels(text: str):
    """(name, body) of every __global__ function."""
    for m in re.finditer(r"__global__[^;{]*?\b(xs_\w+)\s*\([^;{]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), text[m.end():i]


def lone_exits(body: str) -> list[str]:
    return re.findall(r"if \(0 != \*\(volatile (?:const )?unsigned\*\)(?:err|abort)\) return", body)


FILES = sorted(CSRC.glob("*.cu"))


@pytest.mark.parametrize("path", FILES, ids=[p.name for p in FILES])
def test_waiting_kernels_leave_together(path):
    for name, body in kernels(path.read_text()):
        if re.search(r"mbar_wait\(", body):
            assert not lone_exits(body), name


def test_the_reader_finds_the_kernels():
    found = {name for p in FILES for name, _ in kernels(p.read_text())}
    assert {"xs_smm_tile_kernel", "xs_smm_staged_kernel", "xs_smm_uni_kernel", "xs_ozaki_gemm_kernel", "xs_ozs_smm_kernel"} <= found
    assert lone_exits("if (0 != *(volatile const unsigned*)err) return;")
