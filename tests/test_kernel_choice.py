"""Which kernel a stack runs on: the tile kernel for large untuned stacks, also beside a record that the on-line tuner
wrote for smaller ones; a record of the caller's runs as it says."""
from __future__ import annotations

import ctypes
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

from libxstream_b200 import lib

REGISTER, STAGED, FMA, TILE = 0, 1, 2, 3
DEFAULT, TUNED = 0, 1  # where parameters come from


class Params(ctypes.Structure):
    _fields_ = [(f, ctypes.c_int) for f in ("chunk", "mt", "nt", "kp", "generic", "wpb", "sorted", "tile")]


def lookup(m, n, k, S):
    p, source = Params(), ctypes.c_int(-1)
    lib().xs_params_lookup_ex(3, m, n, k, S, ctypes.byref(p), ctypes.byref(source))
    return p, source.value


def kind(m, n, k, S):
    return lib().xs_smm_kernel_kind(S, m, n, k, ctypes.byref(lookup(m, n, k, S)[0]))


def record(m, n, k, mt, nt, kp, tile):
    lib().xs_params_set.argtypes = [ctypes.c_int] * 4 + [ctypes.c_void_p, ctypes.c_double]
    assert lib().xs_params_set(3, m, n, k, ctypes.byref(Params(0, mt, nt, kp, 0, 4, 0, tile)), 0.0) == 0


def test_records_keep_what_they_say_about_the_tile_kernel():
    try:
        assert lookup(45, 45, 45, 100)[0].tile == 1
        record(45, 45, 45, 3, 3, 2, 1)  # as the on-line tuner writes it
        assert lookup(45, 45, 45, 100)[0].tile == 1
        assert lib().libxstream_b200_set_params(45, 45, 45, 0, 3, 3, 2, 4) == 0
        assert lookup(45, 45, 45, 100)[0].tile == 0
    finally:
        lib().libxstream_b200_clear_params()


@pytest.mark.gpu
def test_kinds(acc):
    assert kind(45, 45, 45, 3000) == TILE and kind(45, 45, 45, 1000) == REGISTER  # 7e5 DMMA steps are 1621 entries
    assert kind(23, 23, 23, 3000) == kind(23, 23, 23, 300000) == STAGED
    assert kind(46, 13, 5, 100000) == REGISTER  # 12 DMMA instructions per warp and panel
    assert [kind(64, 64, 64, S) for S in (1100, 1200, 5900, 6000, 65536, 65537)] == [REGISTER, TILE, TILE, REGISTER, REGISTER, TILE]
    for shape, most in (((32, 50, 8), 32768), ((16, 42, 15), 32768), ((24, 32, 15), 65536)):  # one short panel, padded columns
        assert kind(*shape, most) == TILE and kind(*shape, most + 1) == REGISTER
    assert kind(45, 45, 45, 2000000) == TILE  # in parts
    try:
        record(45, 45, 45, 3, 3, 2, 1)
        assert kind(45, 45, 45, 3000) == TILE and kind(45, 45, 45, 1000) == REGISTER
        record(45, 45, 45, 3, 3, 2, 0)
        assert kind(45, 45, 45, 3000) == REGISTER
        record(6, 6, 18, 1, 1, -1, 1)
        assert kind(6, 6, 18, 40000) == FMA
    finally:
        lib().libxstream_b200_clear_params()


AUTOTUNED = """
import json, sys
sys.path[:0] = [%(root)r, %(tests)r]
from libxstream_b200 import acc as A, workloads as W
from test_kernel_choice import kind, lookup
A.init()
stream = A.Stream("tuned")
def call(m, n, k, S):
    c = W.stack_case(m, n, k, S, 40, 40, 30, seed=S)
    b = [A.DevBuf.from_array(x, stream) for x in (c.stack, c.a, c.b_rowmajor())]
    out = A.DevBuf(8 * c.nc * m * n)
    out.zero(stream)
    assert A.process(b[0], S, b[1], b[2], out, m, n, k, stream) == 0
    stream.sync()
call(40, 33, 24, 8000)  # a tile kernel stack first: nothing is tuned
large = lookup(40, 33, 24, 8000)[1]
call(40, 33, 24, 300)   # then a small one: tuned
call(45, 45, 45, 300)
print(json.dumps({"large": large, "sources": [lookup(40, 33, 24, 300)[1], lookup(45, 45, 45, 300)[1]],
                  "small": [kind(40, 33, 24, 300), kind(45, 45, 45, 300)],
                  "kinds": [kind(40, 33, 24, 8000), kind(45, 45, 45, 3000)]}))
"""


@pytest.mark.gpu
def test_tuning_does_not_take_the_tile_kernel_away(acc):
    """The on-line tuner, which times the other kernels, in a process of its own (its switch is read once)."""
    here = Path(__file__).resolve().parent
    env = dict(os.environ, LIBXSTREAM_B200_AUTOTUNE="1", LIBXSTREAM_B200_MLP="0", LIBXSTREAM_B200_NOBUILD="1")
    proc = subprocess.run([sys.executable, "-c", AUTOTUNED % {"root": str(here.parent), "tests": str(here)}], env=env,
                          capture_output=True, text=True, timeout=600)
    assert proc.returncode == 0, proc.stderr[-2000:]
    out = json.loads(proc.stdout.splitlines()[-1])
    assert out["large"] == DEFAULT and out["sources"] == [TUNED, TUNED]
    assert out["kinds"] == [TILE, TILE] and TILE not in out["small"]
