"""Host-array calls through the page-locked staging buffer equal the device-array calls.

A call whose arrays take at most 512 KiB goes through one buffer once the context has made 16
such transfers, before that and where it is larger it copies array by array: the same steps on arrays around that limit, from and to host memory and device memory,
bit for bit. The buffer is reused: a second load before the first state is stored, and calls
of other sizes, leave nothing of the first behind."""
import ctypes

import numpy as np
import pytest

from thesiscode_b200 import _native as N
from thesiscode_b200.panel_velocity import Context

pytestmark = pytest.mark.gpu


def state(nA, nV, nQ, seed):
    rng = np.random.default_rng(seed)
    out = []
    for n in (nA, nV, nQ):
        x = rng.standard_normal((n, 3))
        out.append(np.ascontiguousarray(x / np.linalg.norm(x, axis=1, keepdims=True)))
    return out[0], rng.standard_normal(nA), np.full(nA, 4.0 * np.pi / max(nA, 1)), out[1], out[2]


def host_step(ctx, s, steps):
    xA, z, a, xV, xQ = (v.copy() for v in s)
    tke, ke = ctx.rk4_step(xA, z, a, xV, xQ, 0.01, steps)
    return [xA, z, xV, xQ, tke, ke]


def device_step(ctx, s, steps):
    import torch

    dev = [torch.from_numpy(v.copy()).cuda() for v in s]
    ke = torch.zeros(len(s[0]), dtype=torch.float64, device="cuda")
    tke = np.zeros(steps)
    p = [ctypes.c_void_p(t.data_ptr()) if t.numel() else None for t in dev + [ke]]
    N.call("tc_rk4_step_device", ctx.handle, p[0], p[1], p[2], len(s[0]), p[3], len(s[3]), p[4], len(s[4]), 0.01, steps,
           N.dptr(tke), p[5])
    torch.cuda.synchronize()
    return [dev[0].cpu().numpy(), dev[1].cpu().numpy(), dev[3].cpu().numpy(), dev[4].cpu().numpy(), tke, ke.cpu().numpy()]


def staging_context(prec, transfers=16):
    """A context after `transfers` small transfers; by then it has taken (or is about to take) the buffer."""
    ctx = Context(0, prec)
    s = state(3, 1, 0, 9)
    for _ in range(transfers):
        ctx.rk4_load(*s)
    return ctx


def test_the_buffer_is_taken_between_load_and_store(gpu):
    """Loads and stores on either side of the transfer from which on the buffer is used."""
    for transfers in (0, 13, 14, 15, 16, 17):
        ctx = staging_context("fp64", transfers)
        for seed in (1, 2):
            s = state(300, 100, 7, seed)
            ctx.rk4_load(*s)
            for a, b in zip(ctx.rk4_store(300, 100, 7), (s[0], s[1], s[3], s[4])):
                np.testing.assert_array_equal(a, b)
        ctx.close()


# doubles staged on the way in: 5 nA + 3 nV + 3 nQ, at most 65,536
@pytest.mark.parametrize("prec", ["fp64", "fp32c"])
@pytest.mark.parametrize("nA,nV,nQ", [(1, 0, 0), (257, 0, 3), (40, 1000, 0), (13107, 0, 0), (13106, 2, 0), (13106, 3, 0),
                                      (9000, 4000, 2845), (9000, 4000, 2846)])
def test_host_and_device_arrays_agree(gpu, prec, nA, nV, nQ):
    ctx = staging_context(prec)
    ctx.set_deltas(0.05, 0.05, 0.05)
    for seed, steps in ((1, 1), (2, 3)):
        s = state(nA, nV, nQ, seed)
        for a, b in zip(host_step(ctx, s, steps), device_step(ctx, s, steps)):
            np.testing.assert_array_equal(a, b)
    ctx.close()


def test_a_second_load_replaces_the_first(gpu):
    ctx = staging_context("fp64")
    first, second = state(300, 100, 7, 3), state(200, 50, 0, 4)
    ctx.rk4_load(*first)
    ctx.rk4_load(*second)
    got = ctx.rk4_store(200, 50, 0)
    for a, b in zip(got, (second[0], second[1], second[3], second[4])):
        np.testing.assert_array_equal(a, b)
    ctx.rk4_load(*first)
    got = ctx.rk4_store(300, 100, 7)
    for a, b in zip(got, (first[0], first[1], first[3], first[4])):
        np.testing.assert_array_equal(a, b)
    ctx.close()


def test_a_non_finite_result_is_reported_with_its_index(gpu):
    """Finite inputs whose step overflows: the result comes back, and the call says where."""
    ctx = staging_context("fp64")
    xA, z, a, xV, xQ = state(50, 0, 0, 5)
    z[:] = 1e300
    a[:] = 1e300
    with pytest.raises(N.TcError) as e:
        ctx.rk4_step(xA, z, a, xV, xQ, 0.01, 1)
    assert e.value.status == N.TC_ERR_NONFINITE and "xA (result) at index" in str(e.value)
    assert not np.all(np.isfinite(xA))
    ctx.close()


def test_adjoint_buffers_are_reused_across_sizes(gpu):
    """The buffers stay between calls: a large, a small and the large problem again give what
    fresh contexts give."""
    def run(ctx, n, seed):
        x, z, a, _, _ = state(n, 0, 0, seed)
        J, gz, gx = np.zeros(1), np.zeros(n), np.zeros((n, 3))
        N.call("tc_rk4_vjp", ctx.handle, N.dptr(x), N.dptr(z), N.dptr(a), n, 0.01, 3, 2, N.dptr(x), N.dptr(z), N.dptr(J),
               N.dptr(gz), N.dptr(gx))
        return J, gz, gx

    kept = Context(0, "fp64")
    kept.set_deltas(0.05, 0.05, 0.05)
    for n in (3000, 70, 3000):
        fresh = Context(0, "fp64")
        fresh.set_deltas(0.05, 0.05, 0.05)
        for a, b in zip(run(kept, n, n), run(fresh, n, n)):
            np.testing.assert_array_equal(a, b)
        fresh.close()
    kept.reset_rk4()
    kept.close()
