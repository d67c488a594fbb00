"""The FAST tree walk's forms: one or four lanes to a query, prepared or raw leaf
cells, and boundary points with odd x copied, on grids where each applies,
against a walk in float64 over the tree's own cells.

Vorticity along +z only and positive: every term of the z sum has the same
sign, so its rounding is relative to the sum.  A walk adds fewer than 64 cells of
each of at most 9 layers; with a term's own rounding (rsqrt 2 ulp, ten operations)
the FP32 sum differs by less than (576 + 12) eps = 7.1e-5."""
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


def vortons(n, seed):
    rng = np.random.default_rng(seed)
    ps = np.zeros((n, 4), np.float32)
    ps[:, :3] = rng.uniform(-0.6, 0.6, (n, 3))
    ps[:, 3] = 0.05
    w = np.zeros((n, 4), np.float32)
    w[:, 2] = rng.uniform(0.5, 2.0, n)
    return torch.from_numpy(ps).cuda(), torch.from_numpy(w).cuda()


def boundary(vg, ctx, g, ps, w, copy):
    out = torch.full((g.capacity, 3), -7.0, device="cuda")
    ctx.check(vg.lib().vg_boundary_vecpot_device(ctx.h, ctypes.byref(g), vg._ptr(ps), vg._ptr(w), len(ps), copy,
                                                 vg._ptr(out)), "boundary")
    ctx.synchronize()
    nx, ny, nz = g.points
    return out.cpu().numpy()[: nx * ny * nz].reshape(nz, ny, nx, 3)


def tree_cells(vg, ctx, g, ps, w):
    n = ctypes.c_size_t()
    L, P = vg.lib(), vg._ptr
    ctx.check(L.vg_tree_device(ctx.h, 0, ctypes.byref(g), P(ps), P(w), len(ps), None, 0, 1.0, 1.0, None, None, 0,
                               ctypes.byref(n)), "size")
    t = torch.zeros((n.value, 8), device="cuda")
    ctx.check(L.vg_tree_device(ctx.h, 0, ctypes.byref(g), P(ps), P(w), len(ps), None, 0, 1.0, 1.0, None, P(t), n.value,
                               ctypes.byref(n)), "tree")
    ctx.synchronize()
    return t.cpu().numpy().astype(np.float64)


def walk64(cells, g, q, kind):
    """The walk's sums in float64 for queries q [m, 3]: of each layer's cells below
    an open one, all that the query is not in (widened by 1e-4 cells)."""
    mn, ext = np.array([float(v) for v in g.min_corner]), np.array([float(v) for v in g.extent])
    layers = [np.array(g.points)]
    while layers[-1].prod() > 8:
        layers.append(np.maximum((layers[-1] - 1) // 2 + 1, 2))
    base = np.concatenate([[0], np.cumsum([a.prod() for a in layers])])
    out = np.zeros((len(q), 3))
    f0, fn = np.zeros((len(q), 3), int), np.ones((len(q), 3), int)
    live = np.ones(len(q), bool)
    for layer in range(len(layers) - 1, 0, -1):
        npc = layers[layer - 1]
        d = (npc - 1) // (layers[layer] - 1)
        cell = ext / (npc - 1)
        c0, cn = f0 * d, fn * d
        o0, on = np.zeros_like(f0), np.zeros_like(fn)
        if layer > 1:
            for a in range(3):
                for i in range(cn[:, a].max()):
                    ch = c0[:, a] + i
                    lo = mn[a] + ch * cell[a]
                    at = (i < cn[:, a]) & (q[:, a] >= lo - 1e-4 * cell[a]) & (q[:, a] < lo + 1.0001 * cell[a])
                    o0[:, a] = np.where(at & (on[:, a] == 0), ch, o0[:, a])
                    on[:, a] += at
        opened = (on > 0).all(1)
        for iz, iy, ix in np.ndindex(*cn.max(0)[::-1]):
            i = np.array([ix, iy, iz])
            ch = c0 + i
            use = live & (i < cn).all(1) & ~(opened & (ch >= o0).all(1) & (ch < o0 + on).all(1))
            k = base[layer - 1] + ch[:, 0] + npc[0] * (ch[:, 1] + npc[1] * ch[:, 2])
            c = cells[np.where(use, k, 0)]
            r = c[:, 3] / 2
            use = use & (r > 0)
            r = np.where(use, r, 1.0)
            dv = q - c[:, :3]
            d2 = (dv ** 2).sum(1)
            if kind == 0:
                law = np.minimum(d2 ** -0.5, 1 / r) ** 3
                term = np.cross(c[:, 4:7], dv) * law[:, None]
            else:
                term = c[:, 4:7] * np.where(d2 < r * r, d2 / r ** 3, d2 ** -0.5)[:, None]
            out += np.where(use[:, None], term * (2 / 3 * r ** 3)[:, None], 0.0)
        live &= opened
        f0, fn = np.where(opened[:, None], o0, f0), np.where(opened[:, None], on, fn)
    return out


# four lanes, prepared; four lanes, prepared; one lane, raw; thin: prepared; two points along x; four lanes, raw
@pytest.mark.parametrize("n3", [(9, 9, 9), (33, 32, 34), (60, 57, 51), (80, 3, 90), (2, 12, 12), (50, 48, 46)])
def test_boundary_forms(vg, n3):
    ps, w = vortons(3000, sum(n3))
    g = vg.GridGeom.make([-1.0] * 3, [2.0] * 3, list(n3))
    fast, ref = vg.Context(numerics=vg.NUMERICS_FAST), vg.Context(numerics=vg.NUMERICS_REFERENCE)
    a, b = boundary(vg, fast, g, ps, w, 0), boundary(vg, ref, g, ps, w, 0)
    face = np.ones(a.shape[:3], bool)
    face[1:-1, 1:-1, 1:-1] = False
    assert np.all(a[~face] == -7.0) and np.all(b[~face] == -7.0)
    some = np.argwhere(face)[::7]
    step = 2.0 / (np.array(n3) - 1.0)
    want = walk64(tree_cells(vg, fast, g, ps, w), g, -1.0 + some[:, ::-1] * step * (1 - 2.0 ** -22), 1)[:, 2]
    assert np.all(want > 0)
    assert np.all(np.abs(a[tuple(some.T)][:, 2] - want) <= 7.1e-5 * want)
    # odd x copied from the point before; the last x of inner rows zero where odd
    for got, plain, tol in ((boundary(vg, ref, g, ps, w, 1), b, 0.0), (boundary(vg, fast, g, ps, w, 1), a, 1.42e-4)):
        want = plain.copy()
        want[:, :, 1::2] = plain[:, :, 0:plain.shape[2] - plain.shape[2] % 2:2]
        if n3[0] % 2 == 0 and n3[0] > 2:
            want[1:-1, 1:-1, -1] = 0.0
        assert np.all(np.abs(got[face] - want[face])[:, 2] <= tol * np.abs(want[face][:, 2]))


@pytest.mark.parametrize("kind", [0, 1])
@pytest.mark.parametrize("m", [1, 33, 16383, 16384, 40000])
def test_query_forms(vg, kind, m):
    """Queries on one lane and on four, of raw and of prepared leaves."""
    ps, w = vortons(4000, m)
    rng = np.random.default_rng(m)
    q = np.zeros((m, 4), np.float32)
    q[:, :3] = rng.uniform(-1.0, 1.0, (m, 3))
    q[:, 0] += 3.0  # to one side: the terms of the velocity's y component have one sign, too
    qd = torch.from_numpy(q).cuda()
    comp = 1 if kind == 0 else 2
    for n3 in ((33, 33, 33), (65, 60, 58)):
        g = vg.GridGeom.make([-1.0] * 3, [2.0] * 3, list(n3))
        ctx = vg.Context(numerics=vg.NUMERICS_FAST)
        o, pts = torch.zeros((m, 4), device="cuda"), ctypes.c_size_t()
        ctx.check(vg.lib().vg_tree_device(ctx.h, kind, ctypes.byref(g), vg._ptr(ps), vg._ptr(w), len(ps), vg._ptr(qd),
                                          m, 1.0, 1.0, vg._ptr(o), None, 0, ctypes.byref(pts)), "tree")
        ctx.synchronize()
        some = slice(None, None, max(1, m // 97))
        want = walk64(tree_cells(vg, ctx, g, ps, w), g, q[some, :3].astype(np.float64), kind)[:, comp]
        assert np.all(want > 0)
        assert np.all(np.abs(o.cpu().numpy()[some, comp] - want) <= 7.1e-5 * want)
