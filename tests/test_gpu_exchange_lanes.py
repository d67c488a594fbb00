"""The particle exchanges with four lanes to a particle and with one (fewer than
131,072 particles, or more): the same particles with one more far from them, so
that one call takes each form.

A particle's change is a sum of at most 400 terms (15 lists of cells that hold
fewer than 25 particles here) whose absolute values add up to less than twice the
largest value: the two orders of summation differ by less than 400 eps x 2 = 4.8e-5
of it."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def test_lane_forms_agree():
    import vortegrid_gb300 as vg
    n = 131071
    g = vg.GridGeom.make([-1.0] * 3, [2.0] * 3, [25, 33, 31])
    ctx = vg.Context(numerics=vg.NUMERICS_FAST)
    rng = np.random.default_rng(5)
    ps = np.zeros((n + 1, 4), np.float32)
    ps[:, :3] = rng.uniform(-0.999, 0.999, (n + 1, 3))
    ps[:, 3] = 0.02
    ps[n, :3] = 50.0  # outside the grid: in no list
    w = rng.normal(0, 1, (n + 1, 4)).astype(np.float32)
    d = rng.uniform(0.5, 2.0, n + 1).astype(np.float32)
    out = []
    for m in (n, n + 1):
        p, v, q = (torch.from_numpy(a[:m].copy()).cuda() for a in (ps, w, d))
        L, P = vg.lib(), vg._ptr
        ctx.check(L.vg_pse_device(ctx.h, ctypes.byref(g), P(p), P(v), m, 0.01, 0.02), "pse")
        ctx.check(L.vg_heat_pse_device(ctx.h, ctypes.byref(g), P(p), P(q), m, 0.01, 1.0, 0.02), "heat")
        ctx.synchronize()
        out.append((v.cpu().numpy()[:n], q.cpu().numpy()[:n]))
    for a, b, before in zip(out[0], out[1], (w[:n], d[:n])):
        assert np.abs(a - before).max() > 0
        assert np.abs(a - b).max() <= 4.8e-5 * np.abs(before).max()


@pytest.mark.parametrize("n3", [(25, 33, 31), (21, 22, 23), (13, 17, 15), (9, 9, 9)])
@pytest.mark.parametrize("sigma", [0.25, None])
def test_dense_cells(n3, sigma):
    """One lane to a particle list by list (dense cells) and in one loop, in a puff
    both: against four lanes, as above.  A sum of N terms, each at most 2 nu dt times
    twice the largest value, in two orders: N eps of what the terms' absolute values
    add up to, N = 15 lists of the fullest cell."""
    import vortegrid_gb300 as vg
    n, nu, dt = 131071, 0.01, 0.02
    g = vg.GridGeom.make([-1.0] * 3, [2.0] * 3, list(n3))
    ctx = vg.Context(numerics=vg.NUMERICS_FAST)
    rng = np.random.default_rng(sum(n3))
    ps = np.zeros((n + 1, 4), np.float32)
    ps[:, :3] = rng.uniform(-0.999, 0.999, (n + 1, 3)) if sigma is None else rng.normal(0, sigma, (n + 1, 3)).clip(-0.99, 0.99)
    ps[:, 3] = 0.02
    ps[n, :3] = 50.0
    w = rng.normal(0, 1, (n + 1, 4)).astype(np.float32)
    d = rng.uniform(0.5, 2.0, n + 1).astype(np.float32)
    cell = ((ps[:n, :3].astype(np.float64) + 1) / 2 * (np.array(n3) - 1)).astype(int) @ [1, n3[0], n3[0] * n3[1]]
    terms = 15 * np.bincount(cell).max()
    out = []
    for m in (n, n + 1):
        p, v, q = (torch.from_numpy(a[:m].copy()).cuda() for a in (ps, w, d))
        L, P = vg.lib(), vg._ptr
        ctx.check(L.vg_pse_device(ctx.h, ctypes.byref(g), P(p), P(v), m, nu, dt), "pse")
        ctx.check(L.vg_heat_pse_device(ctx.h, ctypes.byref(g), P(p), P(q), m, nu, 1.0, dt), "heat")
        ctx.synchronize()
        out.append((v.cpu().numpy()[:n], q.cpu().numpy()[:n]))
    for a, b, before in zip(out[0], out[1], (w[:n], d[:n])):
        assert np.abs(a - before).max() > 0
        bound = terms * np.finfo(np.float32).eps * max(1.0, terms * 2 * nu * dt * 2) * np.abs(before).max()
        assert np.abs(a - b).max() <= bound
