"""Device memory that the scheme-1 GEMM asks for: the digits of A and B, with rows and columns rounded up to what the
tensor cores take, not to whole tiles when there are only a few of them."""
from __future__ import annotations

import ctypes

import pytest

from libxstream_b200 import lib


@pytest.mark.parametrize("M,N,K,slices", [(1, 1, 10**8, 7), (8, 16, 10**7, 8), (1, 4096, 10**5, 7), (4096, 1, 10**5, 7), (130, 65, 10**6, 3)])
def test_scratch_of_thin_products(M, N, K, slices):
    lib().xs_ozaki_gemm_scratch_bytes.restype = ctypes.c_size_t
    got = lib().xs_ozaki_gemm_scratch_bytes(M, N, K, slices)
    rows = M + 7 if M < 128 else M + 127
    cols = N + 15 if N < 64 else N + 63
    assert slices * (M + N) * K <= got <= slices * (rows + cols) * (K + 31) + 8 * (M + N) + 8192
