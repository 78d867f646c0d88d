"""The tile kernel's plan, on the CPU: panels cover k exactly and the ring they need fits the shared memory that
the plan asks for, for every k an int holds. Sizes that pass 2^31 or 2^32 bytes must not wrap to small ones."""
from __future__ import annotations

import ctypes

import pytest

from libxstream_b200 import lib

SMEM_MAX = 227 * 1024


class Plan(ctypes.Structure):
    _fields_ = [(f, ctypes.c_int) for f in ("mt", "nt", "T", "nteam", "nsub_n", "Q", "pk", "npan", "R", "ctas", "nchunks", "L", "rem")] + [
        ("smem", ctypes.c_size_t)]


def geometry(m, n, k):
    pl = Plan()
    return pl if lib().xs_tile_geometry(m, n, k, ctypes.byref(pl)) == 0 else None


def check(m, n, k):
    pl = geometry(m, n, k)
    if pl is None:
        return False
    assert (pl.npan - 1) * pl.pk < k <= pl.npan * pl.pk
    assert pl.npan == 1 or pl.pk % (4 * pl.Q) == 0
    ring = pl.nteam * pl.R * 8 * min(pl.pk, k) * (m + n)
    assert ring < pl.smem <= SMEM_MAX // pl.ctas, (m, n, k, pl.npan, pl.pk, pl.smem)
    assert pl.T * 64 * pl.mt * pl.nt >= m * n and pl.T * pl.nteam <= 10
    return True


SIDES = [(1, 1), (8, 8), (13, 7), (48, 48), (16, 45), (23, 23), (45, 45), (56, 56), (64, 64), (64, 26), (72, 9), (80, 73), (80, 80)]


@pytest.mark.parametrize("m,n", SIDES)
def test_any_k(m, n):
    ks = {1, 3, 4, 15, 16, 17, 63, 64, 80, 100, 1000, 12345, 10**6, 2**31 - 1, 2**31 - 17}
    for side in (m, n, m + 2, n + 2, m + n, 2 * (m + n)):  # k at which some product passes a power of two
        for bits in range(28, 34):
            ks |= {2**bits // side // f + d for f in (1, 8, 16) for d in range(-9, 10)}
    ks = sorted(k for k in ks if 0 < k < 2**31)
    assert any([check(m, n, k) for k in ks])


def test_shapes_that_wrapped():
    """Whole blocks of these k were planned as one panel of a few kilobytes."""
    for m, n, k in [(45, 45, 11930466)] + [(56, 56, k) for k in range(9586975, 9586995)]:
        assert check(m, n, k)
        assert geometry(m, n, k).npan > 1


def test_blocks_beyond_ten_warps_are_refused():
    for m, n in [(640, 8), (6400, 1), (81, 81), (1 << 20, 1 << 11)]:
        assert geometry(m, n, 8) is None


@pytest.mark.parametrize("m,n,k", [(46, 13, 5), (9, 39, 8), (7, 72, 7), (12, 70, 3), (32, 76, 5), (64, 64, 5), (77, 64, 7), (74, 58, 6),
                                   (71, 78, 3), (16, 32, 64), (32, 4, 64), (16, 9, 45), (64, 75, 6), (13, 16, 9)])
def test_panels_with_too_little_work_are_refused(m, n, k):
    """Shapes measured slower than on the register kernel: few DMMA instructions per warp and panel, one team per SM,
    padded columns for one or two warps."""
    assert geometry(m, n, k) is None


@pytest.mark.parametrize("m,n,k", [(45, 45, 45), (64, 64, 64), (17, 29, 11), (32, 32, 32), (45, 26, 22), (13, 22, 9), (23, 22, 5), (48, 45, 9),
                                   (69, 28, 3), (80, 80, 80), (54, 29, 73), (72, 72, 16), (40, 33, 24), (9, 10, 20), (77, 76, 4), (13, 32, 35), (22, 32, 16), (4, 78, 8), (37, 16, 18)])
def test_shapes_measured_faster_are_taken(m, n, k):
    pl = geometry(m, n, k)
    assert pl is not None and pl.T * pl.nteam * pl.ctas >= 8
