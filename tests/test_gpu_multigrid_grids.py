"""Solves of several grids in turn on one context.  The cycles of the adaptive
solve are kept as graphs, the coarsest level's sine tables in a workspace that a
grid with larger tables moves: a grid solved again after it gives, bit for bit,
what a context gives that has solved no other."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def problem(n3):
    import vortegrid_gb300 as vg
    rng = np.random.default_rng(sum(n3))
    shape = n3[::-1] + (3,)
    start = torch.from_numpy(rng.normal(0, 1, shape).astype(np.float32)).cuda()
    rhs = torch.from_numpy(rng.normal(0, 50, shape).astype(np.float32)).cuda()
    return vg.GridGeom.make([-1.0, 0.0, 0.5], [(k - 1) / 64.0 for k in n3], list(n3)), start, rhs


def solve(ctx, grid, start, rhs):
    import vortegrid_gb300 as vg
    soln = start.clone()
    cyc, r0, r1 = ctypes.c_int(), ctypes.c_double(), ctypes.c_double()
    ctx.check(vg.lib().vg_multigrid_device(ctx.h, ctypes.byref(grid), vg._ptr(soln), vg._ptr(rhs), 1e-6, 50,
                                           ctypes.byref(cyc), ctypes.byref(r0), ctypes.byref(r1)), "multigrid")
    ctx.synchronize()
    assert 0 < cyc.value < 50 and r1.value <= 1e-6
    return soln


# tables of 16 KB, 131 KB and 54 KB; the largest grid's fields come first or last
@pytest.mark.parametrize("order", [((17, 17, 17), (129, 129, 129)), ((225, 161, 193), (129, 129, 129))])
@pytest.mark.parametrize("fp64", [0, 1])
def test_grids_in_turn(order, fp64):
    import vortegrid_gb300 as vg

    def context():
        c = vg.Context(numerics=vg.NUMERICS_FAST)
        c.check(vg.lib().vg_set_coarsest_fp64(c.h, fp64), "coarsest level")
        return c
    problems = [problem(n3) for n3 in order]
    alone = [solve(context(), *p) for p in problems]
    ctx = context()
    for _ in range(2):
        for p, want in zip(problems, alone):
            for _ in range(2):
                assert torch.equal(solve(ctx, *p).view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("n3,other", [((33, 33, 33), (25, 25, 25)), ((65, 49, 33), (17, 17, 17))])
def test_record_frames_around_another_solve(n3, other):
    """Frames of pinned records, replayed from a graph on a fixed schedule, with a
    solve of a grid with smaller tables between them: bit for bit the frames of
    pageable records, which always run directly."""
    import vortegrid_gb300 as vg
    from vortegrid_gb300 import workloads
    pos, w, s = workloads.ring(1500, seed=4)
    grid = vg.GridGeom.make([-1.5] * 3, [3.0] * 3, list(n3))
    g2, start, rhs = problem(other)
    out = []
    for pinned in (False, True):
        sim = vg.VortonSim(cfg=vg.default_config(fixed_grid=grid, device=0))
        sim.set_poisson_schedule(3, 1)
        v = vg.make_particles(pos, w, s)
        if pinned:
            keep = torch.empty(v.nbytes, dtype=torch.uint8, pin_memory=True)
            rec = keep.numpy().view(v.dtype)
            rec[...] = v
            v = rec
        frames = []
        for k in range(9):
            if k in (5, 7):
                x, cyc, r = start.clone(), ctypes.c_int(), ctypes.c_double()
                sim.check(vg.lib().vg_multigrid_device(sim.h, ctypes.byref(g2), vg._ptr(x), vg._ptr(rhs), 1e-6, 50,
                                                       ctypes.byref(cyc), ctypes.byref(r), ctypes.byref(r)), "multigrid")
            sim.UpdateAndEvolve(v, 1.0 / 60.0, k)
            frames.append(np.ascontiguousarray(v["velocity"]).copy())
        out.append(frames)
    for k, (a, b) in enumerate(zip(*out)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), k


@pytest.mark.parametrize("n3", [(33, 33, 33), (65, 65, 65)])
def test_norms_of_solves_from_zero(n3):
    """From a start and boundary of zeros the first residual is the right-hand side,
    so that both norms are the same number, as they are for a right-hand side of
    zeros: each solve by its own norms, whichever came before."""
    import vortegrid_gb300 as vg
    grid, _, rhs = problem(n3)
    zero = torch.zeros_like(rhs)
    ctx = vg.Context(numerics=vg.NUMERICS_FAST)
    want = None
    for _ in range(50):
        for b in (zero, rhs):
            soln, cyc, r0, r1 = zero.clone(), ctypes.c_int(-1), ctypes.c_double(-1), ctypes.c_double(-1)
            ctx.check(vg.lib().vg_multigrid_device(ctx.h, ctypes.byref(grid), vg._ptr(soln), vg._ptr(b), 1e-6, 50,
                                                   ctypes.byref(cyc), ctypes.byref(r0), ctypes.byref(r1)), "multigrid")
            if b is zero:
                assert cyc.value == 0 and r0.value == r1.value == 0.0 and not soln.any()
                continue
            assert cyc.value > 0 and r0.value == 1.0 and 0 < r1.value <= 1e-6
            want = soln.clone() if want is None else want
            assert torch.equal(soln.view(torch.int32), want.view(torch.int32))


# planes x components beyond what a launch has blocks in z; four planes to a thread of the sweeps, and one
@pytest.mark.parametrize("n3", [(17, 17, 22401), (5, 5, 22401)])
def test_long_box(n3):
    """The reported residual is the solution's own, in float64 (the stored floats'
    residual is half an ulp of each of the seven values)."""
    import vortegrid_gb300 as vg
    grid, start, rhs = problem(n3)
    x = solve(vg.Context(numerics=vg.NUMERICS_FAST), grid, start, rhs).double()
    h = [1.0 / float(grid.cell_spacing[a]) ** 2 for a in range(3)]
    c = x[1:-1, 1:-1, 1:-1]
    lap = (h[0] * (x[1:-1, 1:-1, :-2] + x[1:-1, 1:-1, 2:] - 2 * c) + h[1] * (x[1:-1, :-2, 1:-1] + x[1:-1, 2:, 1:-1] - 2 * c) +
           h[2] * (x[:-2, 1:-1, 1:-1] + x[2:, 1:-1, 1:-1] - 2 * c))
    b = rhs.double()[1:-1, 1:-1, 1:-1]
    stored = np.finfo(np.float32).eps * float(x.norm())
    assert float((b - lap).norm()) <= 1e-6 * float(b.norm()) + 4 * sum(h) * stored


@pytest.mark.parametrize("n3", [(65, 65, 65), (129, 65, 49), (193, 129, 129)])
def test_norms_of_whole_numbers(n3):
    """With unit cells and whole numbers the first residual is exact, and so are the sums
    of three of its squares (below 2^24).  The norm is told to a part in 10^13: 17
    additions to pairs of floats (2^-47 each), the blocks' sums in float64."""
    import vortegrid_gb300 as vg
    grid = vg.GridGeom.make([0.0] * 3, [float(k - 1) for k in n3], list(n3))
    rng = np.random.default_rng(sum(n3))
    shape = n3[::-1] + (3,)
    x0, b = rng.integers(-60, 61, shape), rng.integers(-1000, 1001, shape)
    c = x0[1:-1, 1:-1, 1:-1]
    lap = (x0[1:-1, 1:-1, :-2] + x0[1:-1, 1:-1, 2:] + x0[1:-1, :-2, 1:-1] + x0[1:-1, 2:, 1:-1] + x0[:-2, 1:-1, 1:-1] +
           x0[2:, 1:-1, 1:-1] - 6 * c)
    inner = b[1:-1, 1:-1, 1:-1]
    want = np.sqrt(float(((inner - lap) ** 2).sum())) / np.sqrt(float((inner ** 2).sum()))
    soln, rhs = (torch.from_numpy(a.astype(np.float32)).cuda() for a in (x0, b))
    ctx, cyc, r0, r1 = vg.Context(numerics=vg.NUMERICS_FAST), ctypes.c_int(), ctypes.c_double(), ctypes.c_double()
    ctx.check(vg.lib().vg_multigrid_device(ctx.h, ctypes.byref(grid), vg._ptr(soln), vg._ptr(rhs), 1e-6, 50,
                                           ctypes.byref(cyc), ctypes.byref(r0), ctypes.byref(r1)), "multigrid")
    assert abs(r0.value - want) <= 2e-13 * want


@pytest.mark.parametrize("n3", [(33, 33, 33), (65, 65, 65)])
def test_norms_out_of_range(n3):
    """A right-hand side whose squares are beyond the floats is refused, and the
    context solves the next one."""
    import vortegrid_gb300 as vg
    grid, start, rhs = problem(n3)
    ctx, cyc, r = vg.Context(numerics=vg.NUMERICS_FAST), ctypes.c_int(), ctypes.c_double()

    def status(x, b):
        st = vg.lib().vg_multigrid_device(ctx.h, ctypes.byref(grid), vg._ptr(x), vg._ptr(b), 1e-6, 50, ctypes.byref(cyc),
                                          ctypes.byref(r), ctypes.byref(r))
        ctx.synchronize()
        return st
    assert status(torch.zeros_like(rhs), rhs * 1e20) == 3  # VG_NONFINITE
    assert status(start.clone(), rhs) == 0
