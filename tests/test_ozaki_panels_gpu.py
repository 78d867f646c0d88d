"""GPU parity of the scheme-1 Ozaki GEMM at the edges of its tiles and digit panels (rows 128, columns 64,
k 32; eight diagonals per launch) and of the Ozaki stack form's combine of a segment over many chunks.
Tolerance: the products are exact integers on both sides, only the FP64 order of at most 15 diagonal sums
differs from the oracle's order of 64 pair sums: 1e-14 of the largest entry covers 45 roundings."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from libxstream_b200 import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-14


@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (127, 63, 31), (128, 64, 32), (129, 65, 33), (257, 200, 100), (40, 513, 65)])
@pytest.mark.parametrize("trans", ["NN", "TT"])
@pytest.mark.parametrize("slices,trim", [(1, 0), (5, 0), (7, 6), (8, 0)])
def test_gemm_edges(acc, M, N, K, trans, slices, trim):
    A, stream = acc
    g = W.rng(M + 7 * N + 31 * K + slices)
    op_a, op_b, c0 = g.uniform(-1, 1, (M, K)), g.uniform(-1, 1, (K, N)), g.uniform(-1, 1, (M, N))
    op_a *= np.ldexp(1.0, g.integers(-20, 21, (M, 1)))
    a, b = (op_a.T if trans[0] == "T" else op_a), (op_b.T if trans[1] == "T" else op_b)
    da, db, dc = (A.DevBuf.from_array(x.ravel(order="F"), stream) for x in (a, b, c0))
    assert A.ozaki_gemm(trans[0], trans[1], M, N, K, 1.25, da, a.shape[0], db, b.shape[0], -0.5, dc, M, slices, trim, stream) == 0
    got = dc.download(np.zeros(M * N), stream)
    stream.sync()
    for x in (da, db, dc):
        x.free()
    ref = np.zeros(M * N)
    oracle.ozaki_gemm(op_a.ravel(order="F"), op_b.ravel(order="F"), ref, M, N, K, slices, 2 * (slices - 1) - trim)
    ref = (1.25 * ref.reshape((M, N), order="F") - 0.5 * c0)
    got = got.reshape((M, N), order="F")
    scale = np.maximum(np.abs(ref).max(axis=1, keepdims=True), np.abs(c0).max(axis=1, keepdims=True))
    assert np.max(np.abs(got - ref) / scale) <= TOL


@pytest.mark.parametrize("M,N,K", [(8, 16, 64), (9, 17, 1300), (3, 40, 2000), (100, 5, 700), (130, 48, 40), (121, 49, 1000), (128, 1, 17000)])
@pytest.mark.parametrize("slices,trim", [(1, 0), (2, 0), (3, 2), (4, 3), (8, 0)])
def test_gemm_small_panels(acc, M, N, K, slices, trim):
    """Panels of fewer rows or columns than a tile, several k blocks per stage and a last stage that is not full."""
    test_gemm_edges(acc, M, N, K, "NT", slices, trim)


@pytest.mark.parametrize("m,n,k", [(16, 16, 16), (33, 20, 40)])
def test_stack_segment_over_many_chunks(acc, m, n, k):
    """One C block takes every entry, and a few blocks take many chunks each."""
    A, stream = acc
    for nc in (1, 3):
        case = W.stack_case(m, n, k, 6000, 50, 40, nc, seed=nc, zipf_s=0.0)
        bufs = [A.DevBuf.from_array(x, stream) for x in (case.stack, case.a, case.b_rowmajor(), np.zeros(nc * m * n))]
        s, a, b, c = bufs
        assert A.process_ozaki(s, case.S, m, n, k, a, case.na, b, case.nb, c, 8, 0, stream) == 0
        got = c.download(np.zeros(nc * m * n), stream)
        stream.sync()
        for x in bufs:
            x.free()
        ref = np.zeros(nc * m * n)
        oracle.smm(case.stack, case.a, case.b, ref, m, n, k, b_rowmajor=False)
        # 8 slices keep every bit of entries within 2^-3 of their row's largest; dropped bits are below 2^-52
        # of it, twice per product, and add up over S*k products
        assert oracle.block_relerr(got, ref, m * n) <= 1e-13
