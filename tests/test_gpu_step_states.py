"""Every path of the step on the states that its ordinary flows do not show:
a NaN far from the flow, no wet cell at all, buffers that hold something else
where the step has to write zeros, a captured graph.

PATHS: 7 x 7 tiles, 14 x 13 tiles in two launches, the tile lists, and the
lists with src2method 2's own src2. mx * my is odd for some, so that a plane
and a row range start on either half of a 16-byte line, where the lists'
zeros go out in bulk copies.
"""
import ctypes

import numpy as np
import pytest
import torch

from dclaw_b200 import _lib
from dclaw_b200.params import DClawParams
from dclaw_b200.solver import PatchStepper

from .test_gpu_step_paths import DX, flow

pytestmark = pytest.mark.gpu
PATHS = [(64, 40, 0), (31, 27, 0), (200, 198, 0), (201, 199, 0), (450, 320, 0), (901, 261, 0), (33, 31, 2), (260, 141, 2)]
IDS = [f"{mx}x{my}" + (f"_src2method{k}" if k else "") for mx, my, k in PATHS]
NOT_ZERO = 7.25


def params(k):
    return DClawParams(src2method=2, alphamethod=1) if k == 2 else DClawParams(src2method=k)


def stepper(q, b, p, log=False):
    st = PatchStepper(torch.tensor(q, device="cuda"), torch.tensor(b, device="cuda"), p, DX, DX, branch_log=log)
    st.init_clock(0.02)
    return st


def one_mass(mx, my, p):
    """A flow in one corner, the rest dry."""
    q, b = flow(mx, my, p, seed=5)
    x, y = np.meshgrid(np.arange(mx), np.arange(my))
    near = (x < max(6, mx // 5)) & (y < max(6, my // 5))
    h = np.where(near, 1.0 + 0.2 * np.sin(0.3 * x), 0.0)
    q = np.stack([h, 2.0 * h, -1.0 * h, 0.6 * h, 0.7 * p.rho_f * p.grav * h])
    return q, b


@pytest.mark.parametrize("path", PATHS, ids=IDS)
@pytest.mark.parametrize("where", ["dry", "last"])
@pytest.mark.parametrize("field", [0, 4])
def test_nan_far_from_the_flow(path, where, field):
    mx, my, k = path
    p = params(k)
    q, b = one_mass(mx, my, p)
    j, i = (my - 1, mx - 1) if where == "last" else (my // 2, (3 * mx) // 4)
    assert q[0, j, i] == 0.0
    q[field, j, i] = np.nan
    st = stepper(q, b, p)
    st.step(1)
    assert st.status() == 3


@pytest.mark.parametrize("path", PATHS, ids=IDS)
def test_all_dry_writes_zeros(path):
    mx, my, k = path
    p = params(k)
    _, b = one_mass(mx, my, p)
    st = stepper(np.zeros((5, my, mx)), b, p)
    for _ in range(3):
        st.qb.fill_(NOT_ZERO)
        st.step(1)
        assert torch.count_nonzero(st.state()) == 0
    c = st.read_clock()
    assert c.status == 0 and c.cfl == 0.0 and c.nsteps == 3


@pytest.mark.parametrize("path", PATHS, ids=IDS)
def test_every_cell_is_written(path):
    mx, my, k = path
    p = params(k)
    q, b = one_mass(mx, my, p)
    st, want = stepper(q, b, p), stepper(q, b, p, log=True)
    for _ in range(4):
        st.qb.fill_(NOT_ZERO)
        want.qb.fill_(NOT_ZERO)
        st.step(1)
        want.step(1)
        assert torch.equal(st.state(), want.state())
    assert torch.equal(st.clock[:4], want.clock[:4]) and st.status() == 0


@pytest.mark.parametrize("path", PATHS, ids=IDS)
def test_graph_replay_on_every_path(path):
    mx, my, k = path
    p = params(k)
    q, b = flow(mx, my, p, seed=8)
    eager, st = stepper(q, b, p), stepper(q, b, p)
    eager.step(12)
    st.capture(4)
    st.replay(3)
    assert torch.equal(eager.state(), st.state())
    assert torch.equal(eager.clock[:4], st.clock[:4]) and st.read_clock().nsteps == 12


@pytest.mark.parametrize("size", [(33, 41), (201, 140), (450, 331)], ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("k", [0, 2])
@pytest.mark.parametrize("wet", [True, False])
def test_row_range_is_written_and_no_other(size, k, wet):
    mx, my = size
    p = params(k)
    q, b = one_mass(mx, my, p)
    if not wet:
        q[:] = 0.0
    lib, g = _lib.load(), _lib.load().dclaw_rows_granule()
    want = stepper(q, b, p, log=True)
    want.step(1)
    for first in range(1, my + 1, g):
        for count in sorted({g, my - first + 1}):
            if first + count - 1 > my:
                continue
            st = stepper(q, b, p)
            st.qb.fill_(NOT_ZERO)
            _lib.check(lib.dclaw_step_rows(_lib.ptr(st.qa), _lib.ptr(st.qb), _lib.ptr(st.b), mx, my, DX, DX,
                                           ctypes.byref(st.cp), _lib.ptr(st.clock), _lib.ptr(st.work), st.work_bytes,
                                           first, count, _lib.stream_ptr()), "rows")
            rows = slice(first - 1, first - 1 + count)
            assert torch.equal(st.qb[:, rows], want.state()[:, rows])
            st.qb[:, rows] = NOT_ZERO
            assert bool((st.qb == NOT_ZERO).all())
