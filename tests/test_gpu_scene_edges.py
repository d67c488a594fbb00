"""Surface and fluid-body kernels where their tiles, blocks and groups end:
  * the signed-distance sweep's 16^3 tiles on grids of one tile or less, of a
    tile and one point, and ragged on every axis: bit-exact against the oracle;
  * the block sums of the fluid-body impulses over more blocks than one CTA
    has threads: the whole set's impulse is the sum of its parts'.
"""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def vg():
    import vortegrid_gb300 as vg
    vg.lib()
    return vg


@pytest.fixture(scope="module")
def ctx(vg):
    return vg.Context(numerics=vg.NUMERICS_REFERENCE)


@pytest.mark.parametrize("n", [(2, 2, 2), (16, 16, 16), (17, 16, 15), (16, 33, 17), (49, 3, 18), (5, 40, 70)])
def test_signed_distance_tiles(vg, ctx, oracle_lib, n):
    """Bit for bit: the tiles only reorder updates that do not depend on each other."""
    g = vg.GridGeom.make([-1.0, -0.5, 0.25], [2.0, 1.5, 3.0], list(n))
    og = oracle_lib.Geom.from12(g.as12(), g.points)
    rng = np.random.default_rng(sum(n))
    x = np.stack(np.meshgrid(*[np.linspace(-1, 1, k) for k in n[::-1]], indexing="ij"), -1)
    dens = np.full(g.capacity, 1.0, np.float32)
    field = 1.0 + np.where((x ** 2).sum(-1) < 0.6, 1.0, -0.5) + 0.1 * rng.standard_normal(x.shape[:3])
    dens[:field.size] = field.astype(np.float32).ravel()
    d = torch.from_numpy(dens).cuda()
    out = torch.zeros(g.capacity, dtype=torch.float32, device="cuda")
    ctx.check(vg.lib().vg_signed_distance_device(ctx.h, ctypes.byref(g), vg._ptr(d), 1.0, 1, vg._ptr(out)), "sdf")
    ctx.synchronize()
    ref = oracle_lib.signed_distance(og, dens, 1.0, 0)
    m = field.size
    assert np.array_equal(out.cpu().numpy()[:m].view(np.uint32), np.ascontiguousarray(ref[:m], np.float32).view(np.uint32))


def _tracers(n, seed):
    rng = np.random.default_rng(seed)
    ps = np.empty((n, 4), np.float32)
    ps[:, :3] = rng.uniform(-1, 1, (n, 3))
    ps[:, 3] = 0.01
    return torch.from_numpy(ps).cuda()


def _body(box, pos, vel, size, hollow=0.0):
    b = np.zeros(32, np.float32)
    b[0], b[1] = box, hollow
    b[2:5], b[5:8] = pos, vel
    b[8:11] = 0.3
    b[11:20] = np.eye(3).ravel()
    b[20:23] = size
    b[23] = 1.0
    return b


def _collide(vg, ctx, ps, vel, bodies):
    b = np.ascontiguousarray(bodies, np.float32)
    out = np.zeros((len(b), 6), np.float32)
    ctx.check(vg.lib().vg_collide_tracers_device(ctx.h, vg._ptr(b), len(b), vg._ptr(ps), vg._ptr(vel), None, len(ps),
                                                 vg._ptr(out)), "collide tracers")
    return out


@pytest.mark.parametrize("n", [1, 256 * 1024, 256 * 1024 + 1, 256 * 9000 + 77])
def test_body_sums_of_many_blocks(vg, ctx, n):
    """Tracers at rest and a sphere moving along x: every contact's x impulse
    has the same sign, so FP32 rounding of the sums stays relative to them.
    The blocks' partial sums are the same in both forms; two compensated sums
    (2 eps each), the tree in FP64 and the results' rounding (3 eps / 2) stay
    within 6 eps = 3.6e-7 of each other."""
    body = [_body(0, (0.1, 0, 0), (1, 0, 0), (0.7, 0, 0))]
    ps = _tracers(n, 1)
    ps[0, :3] = torch.tensor([0.3, 0.1, 0.0])
    cut = n // 512 * 256
    parts = np.zeros(6)
    for a, b in ((0, cut), (cut, n)):
        if b > a:
            p = ps[a:b].clone()
            parts += _collide(vg, ctx, p, torch.zeros_like(p), body)[0].astype(np.float64)
    whole = _collide(vg, ctx, ps, torch.zeros_like(ps), body)[0]
    assert abs(whole[0]) > 0 and abs(whole[0] - parts[0]) <= 3.6e-7 * abs(parts[0])


def _some_bodies(nb):
    """Moving spheres, solid boxes and hollow boxes by turns."""
    out = []
    for k in range(nb):
        at = (0.5 - 0.2 * k, 0.1 * k, -0.3 + 0.1 * k)
        kind = k % 3
        out.append(_body(0 if kind == 1 else 1, at, (0.5, 0.1 * k, -0.2),
                         (0.4, 0, 0) if kind == 1 else ((0.5, 0.7, 0.6) if kind == 0 else (1.9, 2.1, 2.0)),
                         hollow=1.0 if kind == 2 else 0.0))
    return out


@pytest.mark.parametrize("nb", [1, 2, 3, 4, 5, 9, 16])
def test_body_groups(vg, ctx, oracle_lib, nb):
    """Bodies are taken four to a launch: any number of them leaves vortons
    and tracers bit for bit as the oracle, also where a position or a velocity
    is infinite or NaN (a NaN's payload is not compared)."""
    n = 5000
    rng = np.random.default_rng(nb)
    pos = rng.uniform(-1.2, 1.2, (n, 3)).astype(np.float32)
    vel = rng.normal(0, 0.5, (n, 3)).astype(np.float32)
    w = rng.normal(0, 1.0, (n, 3)).astype(np.float32)
    for k, bad in enumerate((np.inf, -np.inf, np.nan)):
        pos[10 + k, k] = bad
        pos[20 + k, (k + 1) % 3] = bad
        vel[30 + k, k] = bad
    size = np.full(n, 0.03, np.float32)
    dens = rng.uniform(0.5, 2.0, n).astype(np.float32)
    bodies = np.stack(_some_bodies(nb))

    def same(got, ref):
        a, b = got.cpu().numpy(), np.asarray(ref, np.float32)
        a = a[:, :3] if a.ndim == 2 else a
        nan = np.isnan(b)
        assert np.array_equal(np.isnan(a), nan)
        assert np.array_equal(a[~nan].view(np.uint32), b[~nan].view(np.uint32))

    def quad(xyz, last=None):
        q = np.zeros((n, 4), np.float32)
        q[:, :3] = xyz
        if last is not None:
            q[:, 3] = last
        return torch.from_numpy(q).cuda()

    ps, v, a4, d = quad(pos, size), quad(vel), quad(w), torch.from_numpy(dens).cuda()
    out, cnt = np.zeros((nb, 9), np.float32), np.zeros(nb, np.uint64)
    ctx.check(vg.lib().vg_collide_vortons_device(ctx.h, vg._ptr(bodies), nb, vg._ptr(ps), vg._ptr(v), vg._ptr(a4),
                                                 vg._ptr(d), n, 1.0, 1.0, vg._ptr(out), vg._ptr(cnt)), "vortons")
    op, ov, ow, od, oout = oracle_lib.collide_vortons(pos, vel, w, size, dens, bodies)
    for got, ref in ((ps, op), (v, ov), (a4, ow), (d, od)):
        same(got, ref)
    assert np.array_equal(cnt.astype(np.float64), oout[:, 8].astype(np.float64))
    ps, v = quad(pos, size), quad(vel)
    out = np.zeros((nb, 6), np.float32)
    ctx.check(vg.lib().vg_collide_tracers_device(ctx.h, vg._ptr(bodies), nb, vg._ptr(ps), vg._ptr(v), vg._ptr(d), n,
                                                 vg._ptr(out)), "tracers")
    op, ov, _ = oracle_lib.collide_tracers(pos, vel, size, dens, bodies)
    same(ps, op)
    same(v, ov)


@pytest.mark.parametrize("scale", [1e-30, 1e-14, 1.0, 3e12])
def test_density_statistics_scales(vg, ctx, oracle_lib, scale):
    """The field statistics' sums in pairs of floats, and in FP64 where a square
    leaves the range of floats: signed distances against the oracle's, whose
    serial FP32 sums of 4,913 values are within 4,913 eps / 2 = 1.5e-4 of them
    (mean, and twice that in the mean of squares): the threshold, and with it a
    distance, within 1e-3 of its scale."""
    n = (17, 17, 17)
    g = vg.GridGeom.make([-1.0] * 3, [2.0] * 3, list(n))
    og = oracle_lib.Geom.from12(g.as12(), g.points)
    x = np.stack(np.meshgrid(*[np.linspace(-1, 1, k) for k in n], indexing="ij"), -1)
    dens = (scale * (1.0 + np.clip(0.8 - (x ** 2).sum(-1), -0.7, 0.7))).astype(np.float32).ravel()
    d = torch.from_numpy(dens).cuda()
    out = torch.zeros(g.capacity, dtype=torch.float32, device="cuda")
    ctx.check(vg.lib().vg_signed_distance_device(ctx.h, ctypes.byref(g), vg._ptr(d), float(np.float32(scale)), 0,
                                                 vg._ptr(out)), "sdf")
    ctx.synchronize()
    ref = np.asarray(oracle_lib.signed_distance(og, dens, float(np.float32(scale)), 0), np.float32)[:dens.size]
    got = out.cpu().numpy()[:dens.size]
    assert np.array_equal(np.isnan(got), np.isnan(ref))
    assert np.nanmax(np.abs(got - ref)) <= 1e-3 * np.nanmax(np.abs(ref))
