"""EnsembleStepper from device arenas: the arenas' shapes are checked."""
import numpy as np
import pytest
import torch

from dclaw_b200.ensemble import EnsembleStepper, Member
from dclaw_b200.params import DClawParams

pytestmark = pytest.mark.gpu


def members():
    p = DClawParams()
    rng = np.random.default_rng(2)
    out = []
    for mx, my in ((20, 9), (33, 17)):
        h = np.where(rng.random((my, mx)) < 0.4, 1.0, 0.0)
        out.append(Member(np.stack([h, h, -h, 0.6 * h, 5e3 * h]), 0.1 * rng.random((my, mx)), p, 1.0, 1.0, 0.02))
    return out


def test_arenas_are_copied():
    a = EnsembleStepper(members())
    c = EnsembleStepper(members(), q=a.qa, bed=a.bed)
    assert torch.equal(a.qa, c.qa) and torch.equal(a.bed, c.bed) and a.qa.data_ptr() != c.qa.data_ptr()
    a.step(2)
    c.step(2)
    assert torch.equal(a.qa, c.qa)


@pytest.mark.parametrize("which", ["q", "bed"])
@pytest.mark.parametrize("bad", ["one", "scalar", "short", "long"])
def test_wrong_shapes_are_refused(which, bad):
    a = EnsembleStepper(members())
    n = (a.qa if which == "q" else a.bed).numel()
    t = {"one": torch.zeros(1), "scalar": torch.zeros(()), "short": torch.zeros(n - 1), "long": torch.zeros(n + 1)}[bad]
    with pytest.raises(ValueError, match="arena"):
        EnsembleStepper(members(), **{which: t.double().cuda()})
