"""tc_bs_velocity_device_noalloc in FP64 where the targets' order no longer fits its scratch.

Such a call runs in the stored order (slower, same sum); one that fits is sorted. Both agree
with the allocating entry point within 1e-13 of the largest velocity (the order of rounding
differs: 1,280 terms in sums of 256, each rounded to 1.1e-16 of a partial sum that the
largest velocity's scale bounds, delta 0.05)."""
import ctypes

import numpy as np
import pytest

from thesiscode_b200 import _native as N
from thesiscode_b200 import configs
from thesiscode_b200.panel_velocity import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1_200_000, 600_000])
def test_fp64_order_or_stored(gpu, m):
    import torch

    w = configs.gaussian(level=3, delta=0.05)
    rng = np.random.default_rng(m)
    X = rng.standard_normal((m, 3))
    X /= np.linalg.norm(X, axis=1, keepdims=True)
    assert 32 * w.nA + 24 * m < 32 << 20 and m * w.nA >= 2e8  # accepted, and worth an order
    assert (m * (24 + 4 + 3 * 4) > 32 << 20) == (m == 1_200_000)  # partial sums, order, keys
    ctx = Context(0, "fp64")
    ctx.set_deltas(0.05, 0.05, 0.05)
    dev = [torch.from_numpy(v).cuda() for v in (X, w.xA, w.zetaA, w.areaA)]
    p = [ctypes.c_void_p(t.data_ptr()) for t in dev]
    out = []
    for name in ("tc_bs_velocity_device", "tc_bs_velocity_device_noalloc"):
        u = torch.zeros((m, 3), dtype=torch.float64, device="cuda")
        N.call(name, ctx.handle, N.TC_VERTEX, p[0], m, p[1], p[2], p[3], w.nA, 0, m, ctypes.c_void_p(u.data_ptr()), None)
        torch.cuda.synchronize()
        out.append(u.cpu().numpy())
    ctx.close()
    assert np.abs(out[1] - out[0]).max() <= 1e-13 * np.abs(out[0]).max()
