"""The stretch straight from the velocity grid: vortons of cells whose corners
all lie inside the grid take fixed offsets, the others select each corner's
neighbours.  A step's vorticity (direct velocity, no diffusion) against the
Jacobian grid's stretch (vg_stretch_device), bit for bit, on
grids with no inner cell, with one, and with both kinds along each axis."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n3", [(2, 2, 2), (3, 5, 4), (4, 4, 4), (4, 3, 9), (17, 4, 6), (33, 20, 27)])
def test_stretch_by_cells(n3):
    import vortegrid_gb300 as vg
    g = vg.GridGeom.make([-1.0, -1.5, -0.75], [2.0, 3.0, 1.5], list(n3))
    sim = vg.VortonSim(cfg=vg.default_config(velocity_technique=vg.VELOCITY_DIRECT, fixed_grid=g, enable_stretch=1,
                                             enable_diffusion=0, device=0))
    rng = np.random.default_rng(sum(n3))
    n = 3000
    ps, w = np.zeros((n, 4), np.float32), np.zeros((n, 4), np.float32)
    ps[:, :3] = rng.uniform(-0.999, 0.999, (n, 3)) * [1.0, 1.5, 0.75]
    ps[:, 3] = 0.1
    w[:, :3] = rng.normal(0, 1, (n, 3))
    ps, w = torch.from_numpy(ps).cuda(), torch.from_numpy(w).cuda()
    got = w.clone()
    sim.UpdateDevice(ps.clone(), got, torch.zeros_like(ps), 0.01, 0)
    vel, geom = ctypes.c_void_p(), vg.GridGeom()
    L, P = vg.lib(), vg._ptr
    sim.check(L.vg_get_velocity_grid_device(sim.h, ctypes.byref(vel), ctypes.byref(geom)), "grid")
    ref = w.clone()
    sim.check(L.vg_stretch_device(sim.h, ctypes.byref(geom), vel, P(ps), P(ref), n, ctypes.c_float(0.01)), "stretch")
    sim.synchronize()
    assert not torch.equal(ref, w)
    assert torch.equal(got.view(torch.int32), ref.view(torch.int32))
