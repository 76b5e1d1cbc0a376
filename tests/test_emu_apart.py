"""The two-launch step of small patches (tile.cuh's APART forms, 7 x 7 and
14 x 13 tiles) on the host against the oracle, bit for bit: the tiles' sizes
and one cell around them, thin patches, and the options its update runs."""
import ctypes
import subprocess

import numpy as np
import pytest

from dclaw_b200 import workloads as W
from dclaw_b200.params import CParams

from ._emu import CSRC, HERE
from .test_emu_parity import VARIANTS

SRC, LIB = HERE / "emu_apart.cpp", HERE / "libemu_apart.so"
TILES = [(7, 7), (14, 13)]
_dp = ctypes.POINTER(ctypes.c_double)


@pytest.fixture(scope="module")
def apart():
    if not LIB.exists() or any(d.stat().st_mtime > LIB.stat().st_mtime for d in [SRC, *CSRC.glob("*.cuh")]):
        subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fno-fast-math", "-fPIC", "-shared",
                        str(SRC), "-o", str(LIB)], check=True)
    fn = ctypes.CDLL(str(LIB)).emu_run_apart
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.POINTER(CParams), ctypes.c_int, ctypes.c_int, ctypes.c_double, ctypes.c_double, _dp, _dp,
                   ctypes.c_int, ctypes.c_double, _dp, _dp, ctypes.c_int, ctypes.c_int]

    def run(p, q, b, dx, dy, nsteps, dt, tile):
        q, b = (np.ascontiguousarray(a, dtype=np.float64).copy() for a in (q, b))
        dts, cfls = np.zeros(nsteps), np.zeros(nsteps)
        st = fn(ctypes.byref(p.to_c()), q.shape[2], q.shape[1], dx, dy, q.ctypes.data_as(_dp), b.ctypes.data_as(_dp),
                nsteps, dt, dts.ctypes.data_as(_dp), cfls.ctypes.data_as(_dp), *tile)
        return dict(q=q, dt=dts, cfl=cfls, status=st)

    return run


def _cmp(oracle, apart, p, q, b, dx, n, dt, tile):
    want = oracle.run(p, q, b, dx, dx, n, dt, libm="portable")
    got = apart(p, q, b, dx, dx, n, dt, tile)
    assert want["status"] == got["status"] == 0
    assert np.array_equal(want["q"], got["q"])
    assert np.array_equal(want["dt"], got["dt"]) and np.array_equal(want["cfl"], got["cfl"])


@pytest.mark.parametrize("tile", TILES, ids=["7x7", "14x13"])
@pytest.mark.parametrize("shape", [(2, 2), (3, 17), (17, 3), (7, 7), (8, 6), (6, 8), (13, 14), (14, 15), (12, 13),
                                   (27, 29), (2, 60), (60, 2)])
def test_sizes(oracle, apart, tile, shape):
    c = W.random_field_case(n=128, dx=0.5, seed=4)
    my, mx = shape
    j, i = np.unravel_index(np.argmax(c.q[0]), c.q[0].shape)
    j0, i0 = min(max(0, j - my // 2), 128 - my), min(max(0, i - mx // 2), 128 - mx)
    q, b = c.q[:, j0:j0 + my, i0:i0 + mx], c.b[j0:j0 + my, i0:i0 + mx]
    assert q[0].max() > 0.0
    _cmp(oracle, apart, c.params, q, b, c.dx, 10, c.dt_initial, tile)


@pytest.mark.parametrize("tile", TILES, ids=["7x7", "14x13"])
@pytest.mark.parametrize("variant", ["default", *sorted(set(VARIANTS) - {"src2m2"})])
def test_variants(oracle, apart, variant, tile):
    """(src2method 2 always steps over the tile lists.)"""
    c = W.slope_runout(n=48)
    p = c.params.replace(**VARIANTS.get(variant, {}))
    _cmp(oracle, apart, p, c.q, c.b, c.dx, 25, c.dt_initial, tile)
