"""The one-CTA visiting order of dense local target sets: the same order, at the same cost."""
import ctypes
import statistics

import numpy as np
import pytest
from test_small_order_gpu import sphere_keys

from thesiscode_b200 import _native as N
from thesiscode_b200 import configs
from thesiscode_b200.panel_velocity import Context

pytestmark = pytest.mark.gpu


def targets(m, spread, seed=1):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((m, 3)) if spread is None else np.array([0.3, -0.5, 0.8]) + spread * rng.standard_normal((m, 3))
    return np.ascontiguousarray(X / np.linalg.norm(X, axis=1, keepdims=True))


@pytest.mark.parametrize("m", [33, 1024, 1025, 8191, 16384])
@pytest.mark.parametrize("spread", [0.0, 1e-6, 1e-4, 1e-2, 0.3])
def test_order_of_clusters(gpu, m, spread):
    """Points in one key, in a few cells of the sphere, in a region: the stable sort's order."""
    w = configs.gaussian(level=2, delta=0.02)
    X = targets(m, spread)
    order = np.argsort(sphere_keys(X), kind="stable")
    got = []
    for mode, pts in ((N.TC_ORDER_HILBERT, X), (N.TC_ORDER_GIVEN, np.ascontiguousarray(X[order]))):
        ctx = Context(0, "fp32c")
        ctx.set_deltas(*w.deltas)
        N.call("tc_set_target_order", ctx.handle, mode)
        got.append(ctx.velocity(N.TC_VERTEX, pts, w.xA, w.zetaA, w.areaA)[0])
        ctx.close()
    np.testing.assert_array_equal(got[0][order], got[1])


@pytest.mark.parametrize("m", [4096, 16384])
def test_cost_does_not_depend_on_where_the_points_are(gpu, m):
    """A sum over 20 sources is mostly the order. All targets in one place may take twice the
    time of targets all over the sphere (the sort's work is the same; atomics and memory
    see other addresses)."""
    import torch

    w = configs.gaussian(level=0, delta=0.02)
    ms = {}
    for spread in (None, 1e-4):
        ctx = Context(0, "fp32c")
        ctx.set_deltas(0.02, 0.02, 0.02)
        N.call("tc_set_stream", ctx.handle, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        dev = [torch.from_numpy(v).cuda() for v in (targets(m, spread), w.xA, w.zetaA, w.areaA)]
        u = torch.zeros((m, 3), dtype=torch.float64, device="cuda")
        p = [ctypes.c_void_p(t.data_ptr()) for t in dev + [u]]
        times = []
        for _ in range(20):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record()
            N.call("tc_bs_velocity_device", ctx.handle, N.TC_VERTEX, p[0], m, p[1], p[2], p[3], w.nA, 0, m, p[4], None)
            e[1].record()
            torch.cuda.synchronize()
            times.append(e[0].elapsed_time(e[1]))
        ctx.close()
        ms[spread] = statistics.median(times[5:])
    assert ms[1e-4] <= 2.0 * ms[None], ms
