"""The FP64 pair kernel's frame and wide forms against the oracle.

A CTA whose targets lie within 0.85 of their middle sums in its own frame, others in global
coordinates; targets are sorted where that pays. The cases cross the sizes of the target tiles
(128, 384, 512 to 1,024) and of the source tile (256), targets in grid order, shuffled, in one
small patch (frame form always) and in two opposite patches (wide form always), the self pair
under a visiting order, and every compiled shape.

Bound: both sides round the denominator to at most 8 ulps of 1 (oracle: six roundings; frame
form: the rotated products), 9e-16, and D >= delta^2 / 1 = 2.5e-3 with delta 0.05, so a term
is off by at most 4e-13 of itself and the sum by less, since the terms' errors are independent:
1e-12 of the largest velocity, the FP64 path's stated bound."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from thesiscode_b200 import _native as N
from thesiscode_b200 import configs
from thesiscode_b200.panel_velocity import Context

pytestmark = pytest.mark.gpu
TOL = 1e-12


def points(kind, m, seed):
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((m, 3))
    if kind == "patch":
        x = np.array([0.4, -0.7, 0.6]) + 0.02 * x
    elif kind == "poles":
        x = np.where(np.arange(m)[:, None] % 2 == 0, 1.0, -1.0) * np.array([0.1, 0.2, 0.97]) + 0.02 * x
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    return x * rng.uniform(1.0 - 1e-6, 1.0 + 1e-6, (m, 1))  # off the sphere, as RK4 leaves them


def check(ctx, cls, X, x, z, a, rows, tol=TOL):
    dX, _ = ctx.velocity(cls, X, x, z, a)
    ref = O.rows(cls, rows, X, x, z, a, delta=0.05, nthreads=8)
    err = np.abs(dX[rows] - ref).max() / np.abs(ref).max()
    assert err <= tol, err
    return dX


@pytest.mark.parametrize("kind", ["sphere", "patch", "poles"])
@pytest.mark.parametrize("m,n", [(1, 1), (127, 255), (129, 257), (383, 256), (385, 513), (769, 1000), (3071, 15)])
def test_forms_at_tile_edges(gpu, kind, m, n):
    ctx = Context(0, "fp64")
    ctx.set_deltas(0.05, 0.05, 0.05)
    rng = np.random.default_rng(n)
    x, X = points("sphere", n, 1), points(kind, m, 2)
    check(ctx, N.TC_VERTEX, X, x, rng.standard_normal(n), rng.uniform(0.5, 1.5, n) / n, np.arange(m, dtype=np.int32))
    if m > 1:  # the targets as sources: the self pair is left out
        check(ctx, N.TC_ACTIVE, None, X, rng.standard_normal(m), np.full(m, 1.0 / m), np.arange(m, dtype=np.int32))
    ctx.close()


@pytest.mark.parametrize("cls", [N.TC_ACTIVE, N.TC_VERTEX])
def test_sorted_and_given_order(gpu, cls):
    """Large enough to be sorted (2e8 pairs): both orders, and shuffled input, within the bound."""
    w = configs.jet(level=5, delta=0.05)
    rng = np.random.default_rng(5)
    mix = rng.permutation(w.nA)
    xA, zA, aA = (np.ascontiguousarray(v[mix]) for v in (w.xA, w.zetaA, w.areaA))
    rows = np.sort(rng.choice(w.nV, 300, replace=False)).astype(np.int32)
    for mode in (N.TC_ORDER_HILBERT, N.TC_ORDER_GIVEN):
        ctx = Context(0, "fp64")
        ctx.set_deltas(0.05, 0.05, 0.05)
        N.call("tc_set_target_order", ctx.handle, mode)
        check(ctx, cls, None if cls == N.TC_ACTIVE else w.xV, xA, zA, aA, rows)
        ctx.close()


def test_every_shape_on_compact_and_scattered_targets(gpu):
    cnt = ctypes.c_int()
    N.call("tc_pair_variant_count", N.TC_FP64, ctypes.byref(cnt))
    rng = np.random.default_rng(9)
    x, z = points("sphere", 1537, 3), rng.standard_normal(1537)
    a = np.full(1537, 1.0 / 1537)
    for v in range(cnt.value):
        for kind in ("patch", "sphere"):
            X = points(kind, 9000, 4)
            ctx = Context(0, "fp64")
            ctx.set_deltas(0.05, 0.05, 0.05)
            N.call("tc_set_pair_variant", ctx.handle, N.TC_FP64, v)
            check(ctx, N.TC_VERTEX, X, x, z, a, np.arange(0, 9000, 31, dtype=np.int32))
            check(ctx, N.TC_ACTIVE, None, x, z, a, np.arange(0, 1537, 7, dtype=np.int32))
            ctx.close()


def test_a_bad_target_spoils_its_own_row_only(gpu):
    """Device arrays are not scanned: a NaN or infinite target leaves the others as they are."""
    import torch

    x, X = points("sphere", 700, 6), points("patch", 5000, 7)
    rng = np.random.default_rng(8)
    z, a = rng.standard_normal(700), np.full(700, 1.0 / 700)
    ctx = Context(0, "fp64")
    ctx.set_deltas(0.05, 0.05, 0.05)
    out = []
    for bad in (False, True):
        Y = X.copy()
        if bad:
            Y[1234] = np.nan
            Y[4000, 1] = np.inf
        dev = [torch.from_numpy(v).cuda() for v in (Y, x, z, a)]
        u = torch.zeros((5000, 3), dtype=torch.float64, device="cuda")
        p = [ctypes.c_void_p(t.data_ptr()) for t in dev + [u]]
        N.call("tc_bs_velocity_device", ctx.handle, N.TC_VERTEX, p[0], 5000, p[1], p[2], p[3], 700, 0, 5000, p[4], None)
        torch.cuda.synchronize()
        out.append(u.cpu().numpy())
    ctx.close()
    fine = np.ones(5000, bool)
    fine[[1234, 4000]] = False
    assert np.all(np.isnan(out[1][~fine]).any(axis=1))
    scale = np.abs(out[0]).max()
    assert np.abs(out[1][fine] - out[0][fine]).max() <= TOL * scale
