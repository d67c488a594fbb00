"""Cell lists (vg_partition_device) where the paths of the counting sort end:
cells of one vorton, at the largest size a thread counts (512), that a CTA
sorts (8,192) and beyond (one bitmap window is 262,144 indices), counts at the
edges of the scan's tiles (4,096) and chunks, vortons outside the grid and NaN.
Exact: whole numbers, compared with a stable sort by cell on the CPU."""
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
    return vg.Context()


def run(vg, ctx, n3, cells):
    """cells: the cell of each vorton, or -1 (outside) or -2 (NaN)."""
    g = vg.GridGeom.make([0.0] * 3, [float(k - 1) for k in n3], list(n3))
    pts = int(np.prod(n3))
    cells = np.asarray(cells, np.int64)
    n = len(cells)
    c = np.maximum(cells, 0)
    pos = np.zeros((n, 4), np.float32)
    pos[:, 0], pos[:, 1], pos[:, 2] = c % n3[0] + 0.25, c // n3[0] % n3[1] + 0.25, c // (n3[0] * n3[1]) + 0.25
    pos[cells == -1, 1] = -1e6
    pos[cells == -2, 2] = np.nan
    key = np.where(cells < 0, pts, cells)
    p = torch.from_numpy(pos).cuda()
    start = torch.full((pts + 2,), -1, dtype=torch.int32, device="cuda")
    items = torch.full((max(n, 1),), -1, dtype=torch.int32, device="cuda")
    for _ in range(2):
        ctx.check(vg.lib().vg_partition_device(ctx.h, ctypes.byref(g), vg._ptr(p), n, vg._ptr(start), vg._ptr(items)),
                  "partition")
    ctx.synchronize()
    expect = np.concatenate([[0], np.cumsum(np.bincount(key, minlength=pts + 1))])
    assert np.array_equal(start.cpu().numpy(), expect)
    assert np.array_equal(items.cpu().numpy()[:n], np.argsort(key, kind="stable"))


@pytest.mark.parametrize("n3", [(2, 2, 2), (15, 13, 21), (16, 16, 16), (17, 241, 1025)])
@pytest.mark.parametrize("n", [1, 33, 4096, 50001])
def test_scattered(vg, ctx, n3, n):
    rng = np.random.default_rng(n)
    cells = rng.integers(-2, int(np.prod(n3)), n)
    run(vg, ctx, n3, cells)


@pytest.mark.parametrize("sizes", [(512, 513), (1, 511, 2, 1025), (8192, 8193, 3), (4097, 20000, 8193, 700),
                                   (262145,), (300000, 513, 9000)])
def test_full_cells(vg, ctx, sizes):
    """Cells of the given sizes, their vortons interleaved, and as many outside the grid."""
    rng = np.random.default_rng(len(sizes))
    cells = np.concatenate([np.full(m, 3 + 7 * k) for k, m in enumerate(sizes)] + [np.full(max(sizes) // 2, -1)])
    run(vg, ctx, (9, 8, 7), rng.permutation(cells))


@pytest.mark.parametrize("sizes", [(100000,), (5000, 40000, 600, 8192, 513), (262144, 262145, 31, 8193), (1000003,)])
@pytest.mark.parametrize("shuffled", [False, True])
def test_large_cells(vg, ctx, sizes, shuffled):
    """Cells that bitmaps order, one window and many, their chunks of slots shared
    with other large cells, in index order and not, among scattered vortons."""
    rng = np.random.default_rng(sum(sizes))
    cells = np.concatenate([np.full(m, 5 + 11 * k) for k, m in enumerate(sizes)] + [rng.integers(100, 3000, 2000)])
    run(vg, ctx, (17, 15, 13), rng.permutation(cells) if shuffled else cells)


@pytest.mark.parametrize("others", [0, 900001])
def test_many_vortons(vg, ctx, others):
    """More than 2^20 vortons: large cells are sorted up to 8,192 vortons and ordered by bitmaps beyond."""
    rng = np.random.default_rng(others + 1)
    sizes = [513, 8192, 8193, 70000, 3000, 400000] + [9000] * 60
    cells = np.concatenate([np.full(m, 7 * k) for k, m in enumerate(sizes)] + [rng.integers(600, 60000, others),
                                                                              np.full(300000, -1)])
    assert len(cells) > 1 << 20
    run(vg, ctx, (65, 33, 31), rng.permutation(cells))


@pytest.mark.parametrize("sizes", [(96, 97, 128, 129), (256, 257, 512, 513), (1024, 1025, 2048, 2049), (4096, 4097, 8192),
                                   tuple(range(90, 135)) * 40, tuple(range(500, 525)) * 30,
                                   tuple(range(1010, 1040)) * 20, tuple(range(1900, 2200, 3)) * 8])
@pytest.mark.parametrize("shuffled", [False, True])
def test_sorted_cells(vg, ctx, sizes, shuffled):
    """Cells that a warp, a group of warps or a CTA sorts, at the edges of what a thread holds of
    them, one each and more than there are warps, groups and CTAs."""
    cells = np.repeat(3 * np.arange(len(sizes)), sizes)
    run(vg, ctx, (17, 25, 15), np.random.default_rng(len(cells)).permutation(cells) if shuffled else cells)
