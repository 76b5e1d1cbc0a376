"""The step's paths against each other, bit for bit.

dclaw_step takes small patches through k_records and k_tile_apart (over 7 x 7
tiles while all of them have a place on the SMs), larger ones through the tile lists (src2method 2 always, with k_src2_quad_list), and every
patch with a branch log through the full-grid kernels, which the oracle tests
cover; the patch calls run the staged kernels. The sizes are those where a path can go
wrong: the smallest patches, one cell around a tile and around a CTA of the
staged kernels, thin ones, and both sides of the line between the first two.
"""
import numpy as np
import pytest
import torch

from dclaw_b200.params import DClawParams
from dclaw_b200.patch import MBC, Patch
from dclaw_b200.solver import PatchStepper
from dclaw_b200.workloads import state_from

pytestmark = pytest.mark.gpu
DX = 1.0


def flow(mx, my, p, seed=0):
    """A few moving masses on a rough slope, dry between them."""
    rng = np.random.default_rng(seed)
    x, y = np.meshgrid(np.arange(mx) + 0.5, np.arange(my) + 0.5)
    b = 0.4 * (mx - x) + 0.3 * np.sin(0.7 * x) * np.cos(0.5 * y) + 0.05 * rng.standard_normal((my, mx))
    h, u, v = np.zeros((my, mx)), np.zeros((my, mx)), np.zeros((my, mx))
    m = np.full((my, mx), 0.6)
    for _ in range(5):
        cx, cy, r = rng.uniform(0, mx), rng.uniform(0, my), rng.uniform(2.0, 0.25 * min(max(mx, my), 80) + 3.0)
        k = np.maximum(rng.uniform(0.3, 2.0) * (1.0 - ((x - cx) ** 2 + (y - cy) ** 2) / r**2), 0.0)
        u, v = np.where(k > h, rng.uniform(-2, 5), u), np.where(k > h, rng.uniform(-3, 3), v)
        m = np.where(k > h, rng.uniform(0.5, 0.68), m)
        h = np.maximum(h, k)
    return state_from(h, m, p, rng.uniform(0.4, 1.0), h * u, h * v), b


SIZES = [(2, 2), (3, 17), (14, 13), (15, 14), (29, 27), (64, 40), (7, 700), (316, 316), (317, 316), (5, 20011), (1201, 90)]
OPTIONS = [{}, dict(src2method=2, alphamethod=1), dict(bc=("extrap", "extrap"), limiter=1, friction_forcing=True, manning_coefficient=0.03),
           dict(order=1, transverse_waves=0, src2method=1), dict(src2method=-1, limiter=2, speed_limit=3.0)]


def params(o):
    o = dict(o)
    bc = o.pop("bc", None)
    return DClawParams(**o, **({} if bc is None else dict(bc_lower=bc, bc_upper=bc)))


@pytest.mark.parametrize("size", SIZES, ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("k", range(len(OPTIONS)))
def test_step_equals_full_grid(size, k):
    p = params(OPTIONS[k])
    q, b = flow(*size, p, seed=k)
    q, b = torch.tensor(q, device="cuda"), torch.tensor(b, device="cuda")
    got = []
    for log in (False, True):
        st = PatchStepper(q, b, p, DX, DX, branch_log=log)
        st.init_clock(0.02)
        st.step(3)
        got.append((st.state().clone(), st.clock[:4].clone(), st.status()))
    assert got[0][2] == got[1][2] == 0
    assert torch.equal(got[0][0], got[1][0])
    assert torch.equal(got[0][1], got[1][1])


def test_small_patch_reports_nan():
    p = DClawParams()
    q, b = flow(30, 20, p)
    q[4, 3, 2] = np.nan
    st = PatchStepper(torch.tensor(q, device="cuda"), torch.tensor(b, device="cuda"), p, DX, DX)
    st.init_clock(0.02)
    st.step(1)
    assert st.status() != 0


@pytest.mark.parametrize("size", [(7, 7), (8, 6), (6, 15), (50, 48), (119, 119), (119, 126), (2, 2072), (2, 2073)],
                         ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("k", [0, 2, 3])
def test_tiny_tiles_equal_full_grid(size, k):
    """Patches over 7 x 7 tiles: one cell around a tile, and both sides of the
    296 tiles (two on each of 148 SMs) above which the 14 x 13 ones are taken."""
    test_step_equals_full_grid(size, k)


@pytest.mark.parametrize("size", [(2, 2), (3, 129), (127, 5), (125, 30), (60, 61)], ids=lambda s: f"{s[0]}x{s[1]}")
@pytest.mark.parametrize("k", range(len(OPTIONS)))
def test_patch_calls_equal_step(size, k):
    p = params(OPTIONS[k])
    mx, my = size
    q, b = flow(mx, my, p, seed=10 + k)
    q, b = torch.tensor(q, device="cuda"), torch.tensor(b, device="cuda")
    st = PatchStepper(q, b, p, DX, DX, branch_log=True)
    st.init_clock(0.02, fixed_dt=True)
    st.step(2)
    pt = Patch(p, mx, my)
    qp, aux = (torch.zeros(n, my + 2 * MBC, mx + 2 * MBC, dtype=torch.float64, device="cuda") for n in (5, 6))
    qp[:, MBC:-MBC, MBC:-MBC] = q
    aux[0, MBC:-MBC, MBC:-MBC] = b
    for _ in range(2):
        pt.bc2amr(qp)
        pt.setaux(aux)
        pt.b4step2(qp, aux, DX, DX)
        cfl = pt.step2(qp, aux, DX, DX, 0.02)
        pt.src2(qp, aux, DX, DX, 0.0, 0.02)
    assert torch.equal(qp[:, MBC:-MBC, MBC:-MBC], st.state())
    assert cfl == float(st.clock[2])


@pytest.mark.parametrize("size", [(3, 2), (31, 17), (100, 15), (380, 380), (400, 400), (900, 260)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_adjoint_equals_host_build(size):
    """Few and many activity blocks (the reverse solves of the two directions
    share a launch up to 600), ragged ones, and cells at rest beside moving
    ones, which alone carry calc_taudir's and setvars' adjoints."""
    from dclaw_b200.adjoint import StepAdjoint

    from ._adj import Adj

    p = DClawParams()
    q, b = flow(*size, p, seed=3)
    q[1:3, :, : size[0] // 2] = 0.0
    lam = np.random.default_rng(4).standard_normal(q.shape)
    want, _ = Adj().vjp(p, q, b, DX, DX, 0.02, lam)
    adj = StepAdjoint(torch.tensor(b, device="cuda"), p, DX, DX)
    got = torch.empty(q.shape, dtype=torch.float64, device="cuda")
    adj.vjp(torch.tensor(q, device="cuda"), torch.tensor([0.02], dtype=torch.float64, device="cuda"),
            torch.tensor(lam, device="cuda"), got, torch.zeros(4, dtype=torch.float64, device="cuda"))
    adj.check_status()
    assert np.array_equal(got.cpu().numpy(), want)
