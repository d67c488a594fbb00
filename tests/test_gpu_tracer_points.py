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


def _moving(mod, grid, n):
    """An effect on a grid: a puff whose velocity changes from frame to frame."""
    rng = np.random.default_rng(n)
    return mod.Effect((rng.normal(0, 0.12, (n, 3))).clip(-0.4, 0.4).astype(np.float32),
                      rng.normal(0, 8.0, (n, 3)).astype(np.float32), 0.05, grid)


@pytest.mark.parametrize("capture", ["batch", "caller"])
@pytest.mark.parametrize("cells", [32, 48])
def test_points_after_replayed_steps(capture, cells):
    """Frames replayed from graphs, the batch's own and one that the caller
    captured, each followed by an advection through the context's velocity grid:
    the velocities of that frame's grid, not of an earlier one's copy."""
    import vortegrid_gb300 as vg
    from vortegrid_gb300 import batch as mod
    grid = vg.GridGeom.make([-1.0] * 3, [2.0] * 3, [cells + 1] * 3)
    m, L, P = 262144 + 9, vg.lib(), vg._ptr
    rng = np.random.default_rng(cells)
    x = np.zeros((m, 4), np.float32)
    x[:, :3] = rng.uniform(-0.9, 0.9, (m, 3))
    x = torch.from_numpy(x).cuda()
    if capture == "batch":
        B = mod.Batch([_moving(mod, grid, 500)], streams=1)
        B.calibrate(0.02)
        ctx = vg.lib().vg_batch_context(B.h, 0)

        def frame():
            B.step(0.02)
            B.synchronize()
    else:
        e = _moving(mod, grid, 500)
        stream = torch.cuda.Stream()
        cfg = vg.default_config(velocity_technique=vg.VELOCITY_DIRECT, fixed_grid=grid, enable_stretch=0,
                                enable_diffusion=0, device=0)
        cfg.stream = stream.cuda_stream
        sim = vg.VortonSim(cfg=cfg)
        ps, w = torch.zeros((e.n, 4), device="cuda"), torch.zeros((e.n, 4), device="cuda")
        ps[:, :3], ps[:, 3], w[:, :3] = torch.from_numpy(e.pos), 0.1, torch.from_numpy(0.5 * e.vort)
        vel, graph = torch.zeros_like(ps), torch.cuda.CUDAGraph()
        ctx = sim.h
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            sim.UpdateAndEvolveDevice(ps, w, vel, 0.02)
            stream.synchronize()
            with torch.cuda.graph(graph, stream=stream):
                sim.UpdateAndEvolveDevice(ps, w, vel, 0.02)

        def frame():
            with torch.cuda.stream(stream):
                graph.replay()
            torch.cuda.synchronize()
    seen = []
    for _ in range(4):
        frame()
        g3, geom = ctypes.c_void_p(), vg.GridGeom()
        assert L.vg_get_velocity_grid_device(ctx, ctypes.byref(g3), ctypes.byref(geom)) == 0
        got = []
        for call in ("step", "grid"):
            p, v = x.clone(), torch.zeros_like(x)
            torch.cuda.synchronize()
            if call == "step":
                assert L.vg_advect_device(ctx, P(p), P(v), m, ctypes.c_float(0.02)) == 0
            else:
                assert L.vg_gather_advect_device(ctx, ctypes.byref(geom), g3, P(p), P(v), m, ctypes.c_float(0.02)) == 0
            assert L.vg_synchronize(ctx) == 0
            got.append((p, v))
        assert all(torch.equal(a.view(torch.int32), b.view(torch.int32)) for a, b in zip(*got))
        seen.append(got[0][1].cpu().numpy())
    assert not np.array_equal(seen[0], seen[1])  # the grid does change
