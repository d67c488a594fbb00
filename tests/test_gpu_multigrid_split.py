"""The adaptive multigrid solve over grids on which its split levels end in
different places: rows that fill whole groups of four places or not, two levels
and more, thin and long boxes, unequal spacings, boundary values and a start that
are not zero.

The solution of the seven-point equations is found by sine transforms in
float64.  With the reported residual r |b| (checked in float64), the error is
at most r |b| / lambda, lambda the operator's smallest eigenvalue in magnitude,
plus the rounding of the stored floats."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def operator(x, h):
    c = x[1:-1, 1:-1, 1:-1]
    return (h[0] * (x[1:-1, 1:-1, :-2] + x[1:-1, 1:-1, 2:] - 2 * c) + h[1] * (x[1:-1, :-2, 1:-1] + x[1:-1, 2:, 1:-1] - 2 * c) +
            h[2] * (x[:-2, 1:-1, 1:-1] + x[2:, 1:-1, 1:-1] - 2 * c))


def sine(n):
    k = np.arange(1, n + 1)
    return np.sqrt(2.0 / (n + 1)) * np.sin(np.pi * np.outer(k, k) / (n + 1))


@pytest.mark.parametrize("n3", [(65, 65, 65), (67, 69, 71), (97, 49, 33), (131, 67, 35), (161, 17, 77), (37, 129, 41),
                                (225, 33, 49)])
def test_adaptive_solve(n3):
    import vortegrid_gb300 as vg
    g = vg.GridGeom.make([-1.0, 0.0, 0.5], [2.0, 1.5, 1.0], list(n3))
    rng = np.random.default_rng(sum(n3))
    shape = n3[::-1] + (3,)
    x0 = rng.normal(0, 1, shape).astype(np.float32)
    b = rng.normal(0, 50, shape).astype(np.float32)
    h = [1.0 / float(g.cell_spacing[a]) ** 2 for a in range(3)]
    # exact: the boundary's terms to the right-hand side, sine transforms, the eigenvalues
    edge = x0.astype(np.float64)
    edge[1:-1, 1:-1, 1:-1] = 0.0
    n = [k - 2 for k in n3]
    S = [sine(k) for k in n]
    lam = [-4.0 * h[a] * np.sin(np.pi * np.arange(1, n[a] + 1) / (2 * (n[a] + 1))) ** 2 for a in range(3)]

    def spin(v):
        v = np.einsum("ix,zyxc->zyic", S[0], v, optimize=True)
        v = np.einsum("jy,zyxc->zjxc", S[1], v, optimize=True)
        return np.einsum("kz,zyxc->kyxc", S[2], v, optimize=True)
    inner = b[1:-1, 1:-1, 1:-1].astype(np.float64)
    exact = spin(spin(inner - operator(edge, h)) / (lam[0][:, None] + lam[1][:, None, None] + lam[2][:, None, None, None]))
    tol, smallest = 1e-6, abs(lam[0][0] + lam[1][0] + lam[2][0])
    ctx = vg.Context(numerics=vg.NUMERICS_FAST)
    soln, rhs = torch.from_numpy(x0.copy()).cuda(), torch.from_numpy(b).cuda()
    cyc, r0, r1 = ctypes.c_int(), ctypes.c_double(), ctypes.c_double()
    for _ in range(2):  # the second from replayed cycles
        soln.copy_(torch.from_numpy(x0))
        status = vg.lib().vg_multigrid_device(ctx.h, ctypes.byref(g), vg._ptr(soln), vg._ptr(rhs), tol, 50,
                                              ctypes.byref(cyc), ctypes.byref(r0), ctypes.byref(r1))
        ctx.synchronize()
        x = soln.cpu().numpy()
        bound = np.array(x0)
        bound[1:-1, 1:-1, 1:-1] = x[1:-1, 1:-1, 1:-1]
        assert np.array_equal(x.view(np.uint32), bound.view(np.uint32))  # the boundary is as it was
        norm = np.linalg.norm(inner)
        stored = np.finfo(np.float32).eps * np.linalg.norm(exact)
        res = np.linalg.norm(inner - operator(x.astype(np.float64), h))
        if n3 == (67, 69, 71):  # halves once, to a level too large for the exact solve: refused, nothing done
            assert status == 9 and np.array_equal(x, x0)
            continue
        # 161 x 17 x 77 (cells of 0.0125 by 0.094) stops at the cycle limit, with the residual that it has reached
        if status != 0:
            assert n3 == (161, 17, 77) and cyc.value == 50 and tol < r1.value < 0.1 * r0.value
        else:
            assert r1.value <= tol and 0 < cyc.value <= 50
        # the stored floats' own residual: half an ulp of each of the seven values
        assert abs(res - r1.value * norm) <= 4 * sum(h) * stored
        assert np.linalg.norm(x[1:-1, 1:-1, 1:-1] - exact) <= r1.value * norm / smallest + 2 * stored
