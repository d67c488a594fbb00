"""Tracers gathered from the float4 copy of the step's velocity grid
(VortonSim.AdvectDevice, 2^18 tracers or more): positions and velocities bit
for bit those of vg_gather_advect_device on the three-float grid, for counts
that end within a warp and within a group of eight, on ragged grids, with
tracers outside the grid and not finite."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("np3,m", [((2, 2, 2), 262144), ((9, 33, 17), 262144 + 5), ((33, 2, 40), 262144 + 31),
                                   ((65, 64, 63), 262144 + 264)])
def test_points_gather(np3, m):
    import vortegrid_gb300 as vg
    grid = vg.GridGeom.make([-1.5, -1.0, -0.5], [3.0, 2.0, 1.0], list(np3))
    sim = vg.VortonSim(cfg=vg.default_config(velocity_technique=vg.VELOCITY_DIRECT, fixed_grid=grid, enable_stretch=0,
                                             enable_diffusion=0, device=0))
    rng = np.random.default_rng(m)

    def f4(xyz):
        o = np.zeros((len(xyz), 4), np.float32)
        o[:, :3] = xyz
        return torch.from_numpy(o).cuda()
    ps, w = f4(rng.uniform(-0.3, 0.3, (40, 3))), f4(rng.normal(0, 1, (40, 3)))
    ps[:, 3] = 0.1
    x = rng.uniform([-1.5, -1.0, -0.5], [1.5, 1.0, 0.5], (m, 3)).astype(np.float32)
    x[100:200] += 5.0
    x[300], x[301, 1], x[302, 2], x[m - 1] = np.nan, np.inf, -np.inf, 9.0
    trp = f4(x)
    trv = torch.ones_like(trp)
    sim.UpdateDevice(ps, w, torch.zeros_like(ps), 0.01, 0)
    ref_p, ref_v = trp.clone(), torch.ones_like(trv)
    vg3, geom = ctypes.c_void_p(), vg.GridGeom()
    sim.check(vg.lib().vg_get_velocity_grid_device(sim.h, ctypes.byref(vg3), ctypes.byref(geom)), "grid")
    L, P = vg.lib(), vg._ptr
    L.vg_gather_advect_device(sim.h, ctypes.byref(geom), vg3, P(ref_p), P(ref_v), m, 0.01)
    try:
        sim.AdvectDevice(trp, trv, 0.01)
    except Exception as e:  # tracers outside the grid are reported, as by any gather
        assert "grid" in str(e)
    torch.cuda.synchronize()
    for a, b in ((trp, ref_p), (trv, ref_v)):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
