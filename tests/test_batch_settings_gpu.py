"""A batch on a context whose settings changed since its last batch of the same shapes.

The plan and the captured steps of a batch are kept while its shapes stay. What the steps
depend on besides - the visiting order, omega, delta, the precision, the launch shape asked
for - may change between two calls; each call gives, bit for bit, what a fresh context with
those settings gives (the same kernels on the same inputs)."""
import ctypes

import numpy as np
import pytest

from thesiscode_b200 import _native as N
from thesiscode_b200 import configs
from thesiscode_b200.batch import batch_info, batch_rk4
from thesiscode_b200.panel_velocity import Context

pytestmark = pytest.mark.gpu
BASE = dict(order=N.TC_ORDER_HILBERT, omega=2.0, delta=0.01, precision="fp64", variant=None)
PRECISION = {"fp64": N.TC_FP64, "fp32c": N.TC_FP32C}


def apply(ctx, s):
    N.call("tc_set_precision", ctx.handle, PRECISION[s["precision"]])
    N.call("tc_set_target_order", ctx.handle, s["order"])
    ctx.set_omega(s["omega"])
    ctx.set_deltas(s["delta"], s["delta"], s["delta"])
    if s["variant"] is not None:
        N.call("tc_set_pair_variant", ctx.handle, PRECISION[s["precision"]], s["variant"])


def step(ctx, graph):
    ws = configs.batched_gaussians(count=4, seed=6, levels=(1, 2, 3))
    rng = np.random.default_rng(3)
    for w in ws:  # stored in no order, so that a visiting order matters
        mix = rng.permutation(w.nA)
        w.xA, w.zetaA, w.areaA = w.xA[mix].copy(), w.zetaA[mix].copy(), w.areaA[mix].copy()
    tke = batch_rk4(ctx, ws, 0.01, 2, graph=graph, autotune=False)
    return [tke] + [v for w in ws for v in (w.xA, w.zetaA, w.xV)]


def fresh(s, graph):
    ctx = Context(0, s["precision"])
    apply(ctx, s)
    out = step(ctx, graph)
    info = batch_info(ctx)
    ctx.close()
    return out, info


CHANGES = [dict(order=N.TC_ORDER_GIVEN), dict(omega=5.0), dict(delta=0.05), dict(precision="fp32c"),
           dict(precision="fp32c", variant=12), dict(variant=6)]


@pytest.mark.parametrize("graph", [True, False])
@pytest.mark.parametrize("change", CHANGES, ids=str)
def test_changed_settings_reach_the_next_batch(gpu, change, graph):
    """Settings A, then B, then A again on one context, which keeps its plan."""
    a, b = dict(BASE), dict(BASE, **change)
    if "variant" in change:  # what the library chooses by itself, set back by its number
        a["variant"] = fresh(a, graph)[1]["variant"]
    want = {0: fresh(a, graph), 1: fresh(b, graph)}
    ctx = Context(0, "fp64")
    for which, s in ((0, a), (1, b), (0, a)):
        apply(ctx, s)
        for _ in range(2):  # the second of each replays the captured steps
            got = step(ctx, graph)
            for g, w in zip(got, want[which][0]):
                np.testing.assert_array_equal(g, w)
        assert batch_info(ctx) == want[which][1]
    ctx.close()


def test_tuning_asked_for_later(gpu):
    """A batch run without tuning does not keep a later call from tuning."""
    ctx = Context(0, "fp32c")
    ws = configs.batched_gaussians(count=4, seed=6, levels=(2, 3))
    ctx.set_omega(2.0)
    n0 = ctypes.c_longlong()

    def launches(autotune):
        N.call("tc_stats", ctx.handle, 1, None, None, None, None)
        batch_rk4(ctx, [w.copy() for w in ws], 0.01, 1, graph=False, autotune=autotune)
        N.call("tc_stats", ctx.handle, 1, None, ctypes.byref(n0), None, None)
        return n0.value

    plain = launches(False)
    assert launches(True) > plain  # the candidates' launches
    assert launches(True) == plain  # tuned once
    ctx.close()
