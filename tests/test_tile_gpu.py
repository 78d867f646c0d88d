"""GPU parity of the tile stack kernel, which takes untuned stacks of at least 7e5 DMMA steps: block sizes
at the edges of its warp tiles and panels, both ways of staging an operand, blocks that start 8 bytes
past a 16-byte boundary, segments over many chunks, the DBM record format. Reference: the CPU oracle.
Tolerance: an entry of a C block is a sum of at most S*k products of magnitude up to 1, accumulated in
FP64 in another order than the oracle's; the relative max-norm error per block of the other stack
tests (1e-13) covers 450 roundings of 2^-52 of the largest entry."""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import oracle
from libxstream_b200 import workloads as W
from test_kernel_choice import TILE, kind

pytestmark = pytest.mark.gpu

TOL = 1e-13


def run(A, stream, case, shift=0, alpha=None):
    """C of the device path, the pools starting `shift` doubles into their buffers."""
    pad = np.zeros(shift)
    a = A.DevBuf.from_array(np.concatenate([pad, case.a]), stream)
    b = A.DevBuf.from_array(np.concatenate([pad, case.b_rowmajor()]), stream)
    size = case.nc * case.m * case.n
    c = A.DevBuf(8 * (size + shift))
    c.zero(stream)
    st = case.stack + shift
    if alpha is None:
        s = A.DevBuf.from_array(st.astype(np.int32), stream)
        assert A.process(s, case.S, a, b, c, case.m, case.n, case.k, stream) == 0
    else:
        rec = np.empty((case.S, 6), np.int32)
        rec[:, :3] = (case.m, case.n, case.k)
        rec[:, 3:] = st - 1
        s = A.DevBuf.from_array(rec, stream)
        fmt = case.m | case.n << 8 | case.k << 16
        assert A.lib().libxstream_b200_dbm_launch(stream.handle, ctypes.c_double(alpha), case.S, fmt, None, s.ptr, a.ptr, b.ptr,
                                                  c.ptr) == 0
    out = c.download(np.zeros(size + shift), stream)
    stream.sync()
    for x in (a, b, c, s):
        x.free()
    return out[shift:]


def reference(case, alpha=1.0):
    ref = np.zeros(case.nc * case.m * case.n)
    oracle.smm(case.stack, case.a, case.b, ref, case.m, case.n, case.k, b_rowmajor=False, threads=oracle.max_threads())
    return alpha * ref


def steps(m, n, k):
    return -(-m // 8) * -(-n // 8) * -(-k // 4)


# one warp per block, two, four, nine and ten; odd and even sides, multiples of 8 and 16 (padded staging of
# one or both operands), k below, at and above a group of 16 indices, k over several panels
SHAPES = [(17, 29, 11), (7, 65, 30), (32, 32, 32), (33, 33, 33), (40, 40, 40), (45, 45, 45), (48, 48, 13), (16, 45, 17), (64, 64, 64),
          (65, 72, 15), (72, 72, 16), (80, 73, 3), (80, 80, 80), (24, 24, 24), (64, 26, 9), (30, 50, 150), (9, 10, 20)]


@pytest.mark.parametrize("shape", SHAPES, ids=[f"{m}x{n}x{k}" for m, n, k in SHAPES])
@pytest.mark.parametrize("shift", [0, 1])
def test_shapes(acc, shape, shift):
    A, stream = acc
    m, n, k = shape
    S = int(7.2e5 / steps(m, n, k)) + 3
    case = W.stack_case(m, n, k, S, 60, 50, 90, seed=m + 100 * n + 10000 * k)
    got = run(A, stream, case, shift)
    assert oracle.block_relerr(got, reference(case), m * n) <= TOL


# one DMMA step per panel, tiles of 4 x 4 on two padded operands, a team of two 4 x 4 tiles over several panels
@pytest.mark.parametrize("m,n,k,S", [(69, 28, 3, 20100), (64, 64, 64, 1600), (54, 29, 73, 1400), (23, 22, 5, 40100)])
def test_more_shapes(acc, m, n, k, S):
    A, stream = acc
    assert kind(m, n, k, S) == TILE
    case = W.stack_case(m, n, k, S, 60, 50, 90, seed=S)
    assert oracle.block_relerr(run(A, stream, case, 1), reference(case), m * n) <= TOL


def test_the_tile_kernel_runs_them(acc):
    """The stacks of this file, but for two shapes of test_shapes that run faster on the register kernel at that size."""
    others = {s for s in SHAPES if kind(*s, int(7.2e5 / steps(*s)) + 3) != TILE}
    assert others == {(64, 64, 64), (80, 73, 3)}
    assert kind(45, 45, 45, 3000) == kind(40, 33, 24, 8000) == TILE


@pytest.mark.parametrize("nc,zipf", [(1, 0.0), (3, 1.1), (2900, 0.0)])
def test_segments(acc, nc, zipf):
    """One C block over every chunk (two levels of piece sums), few blocks, more blocks than chunks; equal
    results from call to call."""
    A, stream = acc
    case = W.stack_case(45, 45, 45, 3000, 40, 40, nc, seed=nc, zipf_s=zipf)
    got = run(A, stream, case)
    assert oracle.block_relerr(got, reference(case), 45 * 45) <= TOL
    assert np.array_equal(got, run(A, stream, case))


def test_dbm_records(acc):
    A, stream = acc
    case = W.stack_case(40, 33, 24, 8000, 60, 50, 200, seed=3)
    got = run(A, stream, case, alpha=-1.5)
    assert oracle.block_relerr(got, reference(case, -1.5), 40 * 33) <= TOL


def test_wait_limit_reports_an_error(acc):
    """Waits that may not wait: the call ends with the device error word set, nothing hangs."""
    A, stream = acc
    lib = A.lib()
    case = W.stack_case(45, 45, 45, 3000, 40, 40, 50, seed=8)
    lib.libxstream_b200_set_wait_limit(1)
    try:
        a, b = A.DevBuf.from_array(case.a, stream), A.DevBuf.from_array(case.b_rowmajor(), stream)
        s, c = A.DevBuf.from_array(case.stack, stream), A.DevBuf(8 * case.nc * 45 * 45)
        c.zero(stream)
        assert A.process(s, case.S, a, b, c, 45, 45, 45, stream) == 0
        assert lib.c_dbcsr_acc_stream_sync(stream.handle) != 0
        assert lib.libxstream_b200_device_error(0) & 16
    finally:
        lib.libxstream_b200_set_wait_limit(0)
        lib.c_dbcsr_acc_clear_errors()
    for x in (a, b, c, s):
        x.free()
    assert oracle.block_relerr(run(A, stream, case), reference(case), 45 * 45) <= TOL
