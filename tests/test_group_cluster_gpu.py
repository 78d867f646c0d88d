"""GPU parity of stacks at the edges of the one-cluster grouping's two forms (32768 and 65536 entries; one
pass up to 2048 block positions, several above) and of back-to-back calls on one stream, whose grouping
starts before the call ahead of it ends. Tolerance as for the other stack tests (1e-13 per block)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from libxstream_b200 import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-13


@pytest.mark.parametrize("S", [32768, 32769, 50001, 65536, 65537])
@pytest.mark.parametrize("nc,zipf", [(1, 0.0), (1500, 1.1), (9000, 0.0)])
def test_group_forms(acc, S, nc, zipf):
    A, stream = acc
    case = W.stack_case(4, 6, 5, S, 300, 300, nc, seed=S + nc, zipf_s=zipf)
    bufs = [A.DevBuf.from_array(x, stream) for x in (case.stack, case.a, case.b_rowmajor(), np.zeros(nc * 24))]
    s, a, b, c = bufs
    assert A.process(s, S, a, b, c, 4, 6, 5, stream) == 0
    got = c.download(np.zeros(nc * 24), stream)
    stream.sync()
    ref = np.zeros(nc * 24)
    oracle.smm(case.stack, case.a, case.b, ref, 4, 6, 5, b_rowmajor=False, threads=oracle.max_threads())
    assert oracle.block_relerr(got, ref, 24) <= TOL
    for x in bufs:
        x.free()


def test_calls_back_to_back(acc):
    """Calls that each read what the one before wrote (C of one call is A of the next), nothing waited for
    between them: the early start of a grouping may not let any of them read too soon."""
    A, stream = acc
    m = 13
    case = W.stack_case(m, m, m, 3000, 64, 64, 64, seed=5)
    size = 64 * m * m
    pools = [A.DevBuf.from_array(case.a / 64, stream)] + [A.DevBuf(8 * size) for _ in range(6)]
    for p in pools[1:]:
        p.zero(stream)
    b, s = A.DevBuf.from_array(case.b_rowmajor(), stream), A.DevBuf.from_array(case.stack, stream)
    for i in range(6):
        assert A.process(s, case.S, pools[i], b, pools[i + 1], m, m, m, stream) == 0
    got = pools[6].download(np.zeros(size), stream)
    stream.sync()
    x = case.a / 64
    for _ in range(6):
        y = np.zeros(size)
        oracle.smm(case.stack, x, case.b, y, m, m, m, b_rowmajor=False)
        x = y
    # six products in a row: each adds at most its own 1e-13 of the largest entry of its result
    assert np.max(np.abs(got - x)) <= 6 * TOL * np.max(np.abs(x))
    for p in pools + [b, s]:
        p.free()
