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
