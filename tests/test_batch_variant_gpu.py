"""The launch shape of an ensemble that is not tuned follows the ensemble's sizes: not what the
context ran before, and not the shape for grids a hundred times larger."""
import numpy as np
import pytest

from thesiscode_b200 import configs
from thesiscode_b200.batch import batch_info, batch_rk4
from thesiscode_b200.panel_velocity import Context

pytestmark = pytest.mark.gpu


def variant(precision, levels, before=None):
    ctx = Context(0, precision)
    if before is not None:
        w = configs.gaussian(level=before, delta=0.02)
        ctx.velocity(1, w.xV[:64], w.xA, w.zetaA, w.areaA)
    batch_rk4(ctx, configs.batched_gaussians(count=3, seed=2, levels=levels), 0.01, 1, graph=False, autotune=False)
    v = batch_info(ctx)["variant"]
    ctx.close()
    return v


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_calls_before_do_not_choose_the_shape(gpu, precision):
    assert len({variant(precision, (2, 3), before) for before in (None, 3, 5)}) == 1


@pytest.mark.parametrize("precision,want", [("fp64", (6, 7)), ("fp32c", (1, 12))])
def test_shape_by_the_largest_member(gpu, precision, want):
    """Below 12,288 panels and from there on, as single runs choose it."""
    assert (variant(precision, (2, 4)), variant(precision, (3, 5))) == want


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
def test_members_equal_runs_of_their_own(gpu, precision):
    """Members on both sides of the frame search's 16 tiles (2,048 targets of 128): each within
    rounding of its own single run."""
    ws = configs.batched_gaussians(count=6, seed=3, levels=(1, 2, 3, 4))
    alone = [w.copy() for w in ws]
    ctx = Context(0, precision)
    ctx.set_deltas(0.02, 0.02, 0.02)
    ctx.set_omega(2.0)
    batch_rk4(ctx, ws, 0.01, 1, graph=False, autotune=False)
    tol = 1e-12 if precision == "fp64" else 1e-6
    for w, a in zip(ws, alone):
        ctx.rk4_step(a.xA, a.zetaA, a.areaA, a.xV, np.zeros((0, 3)), 0.01, 1)
        assert np.abs(w.xA - a.xA).max() <= tol and np.abs(w.xV - a.xV).max() <= tol
    ctx.close()
