"""FP32C shapes at the sizes where the automatic choice and the tiles change, against the oracle.

Targets cross the 192-, 256- and 384-target tiles, sources the 64-source segments, the 128- and
256-source tiles and the limits of the automatic shapes (12,288 and 131,072), few targets meet
many sources (launches of more chunks than a full grid's), and targets and sources sit off the
sphere as RK4 leaves them.

Bound: the offsets' rounding, eps rho / h with rho <= 1 the radius of a CTA's targets and h the
distance to the nearest source: sources are level-4 to level-7 panel centres and targets the
same grid's vertices, h >= 0.6 x the spacing sqrt(4 pi / n); 4 eps / h, eps = 2^-24, of the
largest velocity. An index error is off by a term, some 1/n of it or more."""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from thesiscode_b200 import _native as N
from thesiscode_b200 import configs
from thesiscode_b200.panel_velocity import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("level,n,m", [(4, 63, 1), (4, 129, 191), (4, 255, 193), (5, 12287, 257), (5, 12288, 383),
                                       (5, 12289, 2561), (7, 131071, 385), (7, 131072, 191), (7, 131073, 1153)])
def test_shapes_at_their_limits(gpu, level, n, m):
    w = configs.gaussian(level=level, delta=0.01)
    rng = np.random.default_rng(n + m)
    off = 1.0 + 1e-6 * rng.standard_normal((w.nA, 1))
    x = np.ascontiguousarray((w.xA * off)[:n])
    z, a = rng.standard_normal(n), w.areaA[:n].copy()
    X = np.ascontiguousarray(w.xV[rng.choice(w.nV, m, replace=False)] * (1.0 + 1e-6 * rng.standard_normal((m, 1))))
    rows = np.sort(rng.choice(m, min(m, 400), replace=False)).astype(np.int32)
    arows = np.sort(rng.choice(n, min(n, 200), replace=False)).astype(np.int32)
    tol = 4.0 * 2.0 ** -24 / (0.6 * np.sqrt(4.0 * np.pi / w.nA))
    ctx = Context(0, "fp32c")
    ctx.set_deltas(0.01, 0.01, 0.05)
    for cls, Y, d, r in ((N.TC_VERTEX, X, 0.01, rows), (N.TC_PASSIVE, X, 0.05, rows), (N.TC_ACTIVE, None, 0.01, arows)):
        dX, _ = ctx.velocity(cls, Y, x, z, a)
        ref = O.rows(cls, r, Y, x, z, a, delta=d, nthreads=8)
        err = np.abs(dX[r] - ref).max() / np.abs(ref).max()
        assert err <= tol, (cls, err, tol)
    ctx.close()


def test_automatic_shapes(gpu):
    """12 below 131,072 sources, 1 below 12,288; 0 from there (and 2, 6 and 7 in FP64)."""
    w = configs.gaussian(level=7, delta=0.01)
    got = []
    for prec, code in (("fp32c", N.TC_FP32C), ("fp64", N.TC_FP64)):
        ctx = Context(0, prec)
        for n, m in ((12287, 30000), (12288, 30000), (65535, 30000), (65536, 30000), (131071, 30000), (131072, 30000),
                     (131072, 24000), (131072, 6000)):
            ctx.velocity(N.TC_VERTEX, w.xV[:m], w.xA[:n], w.zetaA[:n], w.areaA[:n])
            v = ctypes.c_int()
            N.call("tc_get_pair_variant", ctx.handle, code, ctypes.byref(v))
            got.append(v.value)
        ctx.close()
    assert got == [1, 12, 12, 12, 12, 0, 0, 0, 6, 7, 7, 2, 2, 2, 7, 6]


@pytest.mark.parametrize("n,m", [(700, 5000), (131072, 1500)])
def test_a_bad_target_spoils_its_own_row_only(gpu, n, m):
    """Device arrays are not scanned. A NaN or infinite target shares its thread's reciprocals with
    another target and must not reach it: every other row stays within twice the bound of the
    rows without it (its CTA takes another origin, so they round differently)."""
    import torch

    w = configs.gaussian(level=7 if n > 100000 else 4, delta=0.02)
    x, a = w.xA[:n].copy(), w.areaA[:n].copy()
    rng = np.random.default_rng(8)
    z = rng.standard_normal(n)
    X = np.ascontiguousarray(configs.gaussian(level=5, delta=0.02).xV[:m])
    ctx = Context(0, "fp32c")
    ctx.set_deltas(0.02, 0.02, 0.02)
    out = []
    for bad in (False, True):
        Y = X.copy()
        if bad:
            Y[1234] = np.nan
            Y[400, 1] = np.inf
        dev = [torch.from_numpy(v).cuda() for v in (Y, x, z, a)]
        u = torch.zeros((m, 3), dtype=torch.float64, device="cuda")
        p = [ctypes.c_void_p(t.data_ptr()) for t in dev + [u]]
        N.call("tc_bs_velocity_device", ctx.handle, N.TC_VERTEX, p[0], m, p[1], p[2], p[3], n, 0, m, p[4], None)
        torch.cuda.synchronize()
        out.append(u.cpu().numpy())
    ctx.close()
    fine = np.ones(m, bool)
    fine[[1234, 400]] = False
    assert np.all(np.isnan(out[1][~fine]).any(axis=1)) and np.all(np.isfinite(out[1][fine]))
    tol = 4.0 * 2.0 ** -24 / (0.6 * np.sqrt(4.0 * np.pi / w.nA))
    assert np.abs(out[1][fine] - out[0][fine]).max() <= 2.0 * tol * np.abs(out[0]).max()
