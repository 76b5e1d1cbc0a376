"""The line between the step's two-launch path and its tile lists.

A patch leaves the two-launch path above 100 000 cells, above five 14 x 13
tiles an SM, and where it is one tile wide above three. Drawn in cells alone the
line left thin patches, which have many tiles for their cells, on a path that
was a fifth slower for them.
"""
import pytest
import torch
from cuda.bindings import driver

from dclaw_b200.params import DClawParams
from dclaw_b200.solver import PatchStepper

from .test_gpu_step_paths import DX, flow

pytestmark = pytest.mark.gpu
TX, TY = 14, 13
TWO_LAUNCHES, LISTS = 2, 5


def launches_per_step(st):
    """Nodes of a captured step (every node is a launch)."""
    st.step(2)
    g, s = torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=s):
        st.step(2)
    err, _, n = driver.cuGraphGetNodes(driver.CUgraph(g.raw_cuda_graph()))
    assert err == driver.CUresult.CUDA_SUCCESS and n % 2 == 0
    return n // 2


def line_size(name, over, nsm):
    """(mx, my) at the line on nsm SMs, or (over = 1) one cell beyond it."""
    return {
        "column": (5, TY * 3 * nsm + over),
        "full column": (TX, TY * 3 * nsm + over),
        "row": (TX * 3 * nsm + over, 3),
        "two columns": (TX + 1, TY * (5 * nsm // 2) + over),
        "two rows": (TX * (5 * nsm // 2) + over, TY + 1),
        "cells": (316 + over, 316),
    }[name]


@pytest.mark.parametrize("over", [0, 1])
@pytest.mark.parametrize("name", ["column", "full column", "row", "two columns", "two rows", "cells"])
def test_line(name, over):
    mx, my = line_size(name, over, torch.cuda.get_device_properties(0).multi_processor_count)
    p = DClawParams()
    q, b = flow(mx, my, p, seed=6)
    q, b = torch.tensor(q, device="cuda"), torch.tensor(b, device="cuda")
    st, want = PatchStepper(q, b, p, DX, DX), PatchStepper(q, b, p, DX, DX, branch_log=True)
    for s in (st, want):
        s.init_clock(0.02)
        s.step(2)
    assert torch.equal(st.state(), want.state()) and torch.equal(st.clock[:4], want.clock[:4])
    assert launches_per_step(st) == (LISTS if over else TWO_LAUNCHES)


@pytest.mark.parametrize("size", [(5, 20000), (20, 5000), (20000, 5)], ids=lambda s: f"{s[0]}x{s[1]}")
def test_thin_patches_step_over_the_lists(size):
    p = DClawParams()
    q, b = flow(*size, p, seed=7)
    st = PatchStepper(torch.tensor(q, device="cuda"), torch.tensor(b, device="cuda"), p, DX, DX)
    st.init_clock(0.02)
    assert launches_per_step(st) == LISTS
