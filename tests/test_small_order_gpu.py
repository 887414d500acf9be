"""Visiting orders of small target sets: the one-CTA order is the device-wide sort's.

The FP32C sum visits its targets in the order of their sphere keys, so the same targets give
the same partial tiles, and bit for bit the same velocities, whichever sort ordered them.
tc_rk4_stage_range and tc_bs_velocity take the one-CTA order up to 16,384 targets a class; a
caller that sorts its targets by the same order beforehand and asks for TC_ORDER_GIVEN gets
the same tiles without any sort."""
import numpy as np
import pytest

from thesiscode_b200 import _native as N
from thesiscode_b200 import configs
from thesiscode_b200.panel_velocity import Context

pytestmark = pytest.mark.gpu

# cube faces along the curve and their (swap, flip u, flip v), as in sphere_order.cuh
RANK, SWAP, FLIP_U, FLIP_V, BITS = 0x1d850, 0x08, 0x16, 0x08, 14


def sphere_keys(x):
    """The 31-bit key of each point, restated from the construction in sphere_order.cuh."""
    keys = np.zeros(len(x), np.int64)
    for j, p in enumerate(x):
        a = np.abs(p)
        axis = 0 if a[0] >= a[1] and a[0] >= a[2] else 1 if a[1] >= a[2] else 2
        u, v = (p[1], p[2]) if axis == 0 else (p[0], p[2]) if axis == 1 else (p[0], p[1])
        face = 2 * axis + (1 if p[axis] < 0.0 else 0)
        if (SWAP >> face) & 1:
            u, v = v, u
        u = -u if (FLIP_U >> face) & 1 else u
        v = -v if (FLIP_V >> face) & 1 else v
        inv = 1.0 / abs(p[axis])
        n = 1 << BITS
        X, Y = (int(min(max((c * inv + 1.0) * 0.5 * n, 0.0), n - 1.0)) for c in (u, v))
        d, s = 0, n >> 1
        while s:
            rx, ry = int(bool(X & s)), int(bool(Y & s))
            d += s * s * ((3 * rx) ^ ry)
            if ry == 0:
                if rx == 1:
                    X, Y = n - 1 - X, n - 1 - Y
                X, Y = Y, X
            s >>= 1
        keys[j] = (((RANK >> (3 * face)) & 7) << (2 * BITS)) | d
    return keys


@pytest.mark.parametrize("m,spread", [(1, 2.0), (31, 2.0), (1025, 2.0), (8193, 2.0), (16384, 2.0),
                                      (16385, 2.0), (3000, 1e-3)])
def test_order_is_the_stable_sort_by_key(gpu, m, spread):
    """Sizes at the edges of the one-CTA order (16,384) and of its threads; and targets that
    all share a few cells."""
    w = configs.gaussian(level=3, delta=0.02)
    rng = np.random.default_rng(m)
    X = rng.standard_normal((m, 3)) if spread > 1.0 else np.array([0.3, -0.5, 0.8]) + spread * rng.standard_normal((m, 3))
    X[m // 2:m // 2 + 7] = X[m // 2]  # equal keys stay in index order
    X /= np.linalg.norm(X, axis=1, keepdims=True)
    order = np.argsort(sphere_keys(X), kind="stable")
    got = []
    for mode, pts in ((N.TC_ORDER_HILBERT, X), (N.TC_ORDER_GIVEN, np.ascontiguousarray(X[order]))):
        ctx = Context(0, "fp32c")
        ctx.set_deltas(*w.deltas)
        N.call("tc_set_target_order", ctx.handle, mode)
        got.append(ctx.velocity(N.TC_VERTEX, pts, w.xA, w.zetaA, w.areaA)[0])
        ctx.close()
    np.testing.assert_array_equal(got[0][order], got[1])


def test_stage_orders_of_three_classes(gpu):
    """One RK4 step with three classes, two of them small and one large, equals the same step
    with every class sorted by the caller."""
    w = configs.rh4(level=5, parity=True)
    out = []
    sets = [(w.xA, w.zetaA, w.areaA, w.xV, w.xQ)]
    o = [np.argsort(sphere_keys(x), kind="stable") for x in (w.xV, w.xQ)]
    sets.append((w.xA, w.zetaA, w.areaA, w.xV[o[0]], w.xQ[o[1]]))
    for xA, zA, aA, xV, xQ in sets:
        ctx = Context(0, "fp32c")
        ctx.set_omega(w.omega)
        ctx.set_deltas(*w.deltas)
        xA, zA, xV, xQ = xA.copy(), zA.copy(), xV.copy(), xQ.copy()
        ctx.rk4_step(xA, zA, aA, xV, xQ, w.dt, 1)
        ctx.close()
        out.append((xA, zA, xV, xQ))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    np.testing.assert_array_equal(out[0][1], out[1][1])
    np.testing.assert_array_equal(out[0][2][o[0]], out[1][2])
    np.testing.assert_array_equal(out[0][3][o[1]], out[1][3])
