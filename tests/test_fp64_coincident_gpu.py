"""FP64 sums whose targets lie on sources, with little or no smoothing.

A pair of equal points has no velocity, x_i x x_k = 0, wherever its denominator
1 - x.x + delta^2 is not rounded to 0 (there the reference's 0/0 is NaN, and so is the
library's sum, the denominator being the fused 1 - x.x + delta^2). With delta = 0 such a
denominator is rounding, 1e-17 to 1e-16, and its reciprocal must not reach the sum.

Bound: 1e-12 of the largest velocity, as in test_fp64_forms_gpu.py. The pairs of unequal
points have D >= h^2/2 >= 1e-5 (h: the closest such pair, 5e-3 at level 6), a denominator is
rounded to at most 9e-16, so a pair's velocity, at most G / (4 pi h) < 1e-3 of the field, is off
by 1e-10 of itself at most."""
import ctypes
from fractions import Fraction

import numpy as np
import pytest

from thesiscode_b200 import _native as N
from thesiscode_b200 import configs
from thesiscode_b200.panel_velocity import Context

pytestmark = pytest.mark.gpu
TOL = 1e-12


def device_sum(ctx, cls, X, x, z, a):
    """Device arrays: results are not scanned for NaN."""
    import torch

    m = len(x) if X is None else len(X)
    dev = [torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (x if X is None else X, x, z, a)]
    u = torch.zeros((m, 3), dtype=torch.float64, device="cuda")
    p = [ctypes.c_void_p(t.data_ptr()) for t in dev + [u]]
    if X is None:
        p[0] = None
    N.call("tc_bs_velocity_device", ctx.handle, cls, p[0], m, p[1], p[2], p[3], len(x), 0, m, p[4], None)
    torch.cuda.synchronize()
    return u.cpu().numpy()


def fused_denominator(p, delta):
    d = Fraction(float(1.0 + delta * delta))
    for c in p:
        d = Fraction(float(d - Fraction(float(c)) ** 2))
    return float(d)


def check(ctx, cls, X, x, z, a, delta, rows):
    """Rows of the sum against extended precision, pairs of equal points left out."""
    ctx.set_deltas(delta, delta, delta)
    got = device_sum(ctx, cls, X, x, z, a)[rows]
    P = (x if X is None else X)[rows]
    xl = x.astype(np.longdouble)
    want = np.zeros((len(rows), 3), np.longdouble)
    undefined = np.zeros(len(rows), bool)
    for j, p in enumerate(P):
        same = (x == p).all(axis=1)
        D = 1 - xl @ p.astype(np.longdouble) + np.longdouble(delta * delta)
        w = np.where(same, 0, (z * a) / np.where(same, 1, D))
        T = (w[:, None] * (xl - p)).sum(axis=0)
        want[j] = np.cross(p.astype(np.longdouble), T) / (-4 * np.longdouble(np.pi))
        if cls == N.TC_ACTIVE:
            same[rows[j]] = False
        undefined[j] = same.any() and fused_denominator(p, delta) == 0.0
    assert np.array_equal(np.isnan(got).any(axis=1), undefined)
    err = np.abs(got - want)[~undefined].max() / np.abs(want).max()
    assert err <= TOL, err
    return undefined


@pytest.mark.parametrize("level", [4, 6])
@pytest.mark.parametrize("cls", [N.TC_VERTEX, N.TC_PASSIVE])
def test_targets_on_panel_centres(gpu, level, cls):
    """Panel centres as targets, and the divided panels' centres, most of which are a child's."""
    w = configs.rh4(level=level, parity=True)
    X = w.xA if cls == N.TC_VERTEX else w.xQ
    on = (np.arange(len(X)) if cls == N.TC_VERTEX else
          np.flatnonzero(np.isin(X.view("V24").ravel(), np.ascontiguousarray(w.xA).view("V24").ravel())))
    rows = np.sort(np.random.default_rng(level).choice(on, 250, replace=False))
    ctx = Context(0, "fp64")
    undefined = check(ctx, cls, np.ascontiguousarray(X), w.xA, w.zetaA, w.areaA, 0.0, rows)
    assert 0 <= undefined.sum() < 200
    ctx.close()


@pytest.mark.parametrize("delta", [0.0, 1e-9, 1e-3, 0.0099, 0.01])
@pytest.mark.parametrize("variant", [None, 0, 1, 2, 3, 6, 7])
def test_every_shape(gpu, variant, delta):
    """Each launch shape, sources in no order, half of them up to 1e-9 off the sphere, and a
    number of sources that fills no tile."""
    w = configs.rh4(level=4, parity=True)
    rng = np.random.default_rng(4)
    mix = rng.permutation(w.nA)[:4999]
    x = w.xA[mix] * (1.0 + 1e-9 * rng.uniform(-1, 1, (len(mix), 1)) * (rng.random((len(mix), 1)) < 0.5))
    x = np.ascontiguousarray(x)
    z, a = w.zetaA[mix], w.areaA[mix]
    X = np.concatenate([w.xV, x[::3], x[::-2]])[np.argsort(np.concatenate([w.xV, x[::3], x[::-2]])[:, 2])]
    X = np.ascontiguousarray(np.concatenate([X, X, X, X]))  # at least 16 tiles of every shape
    rows = rng.choice(np.flatnonzero(np.isin(X.view("V24").ravel(), x.view("V24").ravel())), 150, replace=False)
    ctx = Context(0, "fp64")
    if variant is not None:
        N.call("tc_set_pair_variant", ctx.handle, N.TC_FP64, variant)
    check(ctx, N.TC_VERTEX, X, x, z, a, delta, np.sort(rows))
    ctx.close()


def test_two_panels_in_one_place(gpu):
    """TC_ACTIVE leaves out the panel itself, not another one at the same point."""
    w = configs.rh4(level=5, parity=True)
    rng = np.random.default_rng(5)
    twice = rng.choice(w.nA, 400, replace=False)
    x, z, a = (np.ascontiguousarray(np.concatenate([v, v[twice]])) for v in (w.xA, w.zetaA, w.areaA))
    ctx = Context(0, "fp64")
    check(ctx, N.TC_ACTIVE, None, x, z, a, 0.0, np.sort(np.concatenate([twice[:100], w.nA + np.arange(100, 200)])))
    ctx.close()
