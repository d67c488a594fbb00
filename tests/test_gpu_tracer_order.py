"""Tracers gathered from the float4 copy of the step's velocity grid in the order
of their cells, every other one so, and all in one cell: warps on either side of
the line between loads by thread and by eight lanes.  Positions and velocities bit
for bit those of vg_gather_advect_device on the three-float grid."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", ["cells", "pairs", "one cell"])
@pytest.mark.parametrize("np3,m", [((9, 33, 17), 262144 + 5), ((65, 64, 63), 262144 + 264)])
def test_points_gather_in_order(np3, m, order):
    import vortegrid_gb300 as vg
    L, P = vg.lib(), vg._ptr
    low, size = np.array([-1.5, -1.0, -0.5]), np.array([3.0, 2.0, 1.0])
    grid = vg.GridGeom.make(list(low), list(size), list(np3))
    sim = vg.VortonSim(cfg=vg.default_config(velocity_technique=vg.VELOCITY_DIRECT, fixed_grid=grid, enable_stretch=0,
                                             enable_diffusion=0, device=0))
    rng = np.random.default_rng(m)

    def f4(xyz):
        o = np.zeros((len(xyz), 4), np.float32)
        o[:, :3] = xyz
        return torch.from_numpy(o).cuda()
    ps, w = f4(rng.uniform(-0.3, 0.3, (40, 3))), f4(rng.normal(0, 1, (40, 3)))
    ps[:, 3] = 0.1
    x = rng.uniform(low, low + size, (m, 3)).astype(np.float32)
    cells = np.array(np3) - 1
    at = np.clip(((x.astype(np.float64) - low) / size * cells).astype(int), 0, cells - 1)
    s = x[np.argsort(at[:, 0] + cells[0] * (at[:, 1] + cells[1] * at[:, 2]), kind="stable")]
    if order == "pairs":
        s[1::2] = x[1::2]
    elif order == "one cell":
        s = np.float32([0.01, 0.02, 0.03]) + x * np.float32(1e-3)
    s[100:120] += 5.0
    s[300], s[301, 1], s[m - 1] = np.nan, np.inf, 9.0
    trp = f4(s)
    trv = torch.ones_like(trp)
    sim.UpdateDevice(ps, w, torch.zeros_like(ps), 0.01, 0)
    ref_p, ref_v = trp.clone(), torch.ones_like(trv)
    vg3, geom = ctypes.c_void_p(), vg.GridGeom()
    sim.check(L.vg_get_velocity_grid_device(sim.h, ctypes.byref(vg3), ctypes.byref(geom)), "grid")
    L.vg_gather_advect_device(sim.h, ctypes.byref(geom), vg3, P(ref_p), P(ref_v), m, 0.01)
    try:
        sim.AdvectDevice(trp, trv, 0.01)
    except vg.VgError as e:  # tracers outside the grid are reported, as by any gather
        assert "grid" in str(e)
    torch.cuda.synchronize()
    for a, b in ((trp, ref_p), (trv, ref_v)):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))
