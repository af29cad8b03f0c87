"""Tile lists, ranges and work order against the oracle where the listed
scenes do not go (B200 required).  All bit for bit."""
import numpy as np
import pytest

from splat_b200 import scene
from test_gpu_parity import check_view_against_oracle, gpu_raster, make, oracle_cam, oracle_opts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [8, 16, 32])
def test_full_lists_of_uneven_views(tile):
    """Full rectangle lists (tileCull = 0) of views whose tiles share warps:
    their ranges and the buckets of the work order are made together, so every
    tile has to be rasterised exactly once."""
    n = 3000
    params, sh = scene.surface_scene(n, seed=8, sh_deg=1, log_scale=(-3.5, 0.5))
    sizes = [(75, 53), (33, 97), (160, 90), (9, 7), (121, 40)]
    cams = [scene.ring_cameras(len(sizes), 4.0, 0.5, w, h, phase=0.2)[k] for k, (w, h) in enumerate(sizes)]
    rgbs = [scene.uniform_target(w, h, seed=20 + k) for k, (w, h) in enumerate(sizes)]
    opts = dict(shDeg=1, tile=tile, tileCull=0, maxBatch=len(sizes))
    t, targets, metas = make(params, sh, cams, rgbs, opts, radius=2.0)
    for _ in range(3):
        gpu_raster(t, range(len(sizes)), 3)
        for v in range(len(sizes)):
            check_view_against_oracle(t, oracle_opts(opts), oracle_cam(metas[v], v, len(sizes), 1), params, sh,
                                      targets, n, view=v)


@pytest.mark.parametrize("cull", [1, 0])
def test_lists_after_replayed_passes(cull):
    """The lists and counts read back belong to the pass that ran last, also
    when it replayed a captured graph: the tile size changes between passes,
    and with it the buffer of the sorted entries (one sort pass at tile 16 and
    32, two at tile 8) and whether entry values carry block bits (tile 16)."""
    n = 3000
    params, sh = scene.uniform_scene(n, seed=9, sh_deg=1)
    params.reshape(-1, 16)[:, 13] += 2.0  # enough donors for refine
    cam = scene.ring_cameras(1, 3.0, 0.0, 200, 150)[0]
    rgb = scene.uniform_target(200, 150, seed=30)
    t, targets, metas = make(params, sh, [cam], [rgb], dict(shDeg=1, tileCull=cull), radius=1.0)
    launches = {}
    for tile in [16, 8, 16, 32, 16, 8, 32, 8, 16]:
        opts = dict(shDeg=1, tile=tile, tileCull=cull)
        t.setRasterConfig(tile, 64)
        gpu_raster(t, [0], 3)
        g, _, _, _ = check_view_against_oracle(t, oracle_opts(opts), oracle_cam(metas[0], 0, 1, 1), params, sh, targets,
                                               n)
        assert launches.setdefault(tile, t._state().lastLaunches) == t._state().lastLaunches
    assert launches[8] == launches[16] + 1
    assert t.refine(iter([0.5] * 10**6).__next__)["maxTile"] == g["cnt"].max()


@pytest.mark.parametrize("budget", [0, 1])
def test_splats_billions_of_pixels_wide(budget):
    """Splats right of the image that reach more than 2^34 pixels to the left:
    every block column between is theirs, with the whole rows that the usual
    expansion writes and with the lane's own walk after a tile went over the
    entry budget."""
    W, H, n = 150, 70, 40
    rng = np.random.default_rng(12)
    f, z = 3.0e6, 0.06
    P = np.zeros((n, 16), np.float32)
    P[:, 0] = (rng.uniform(100.0, 130.0, n)) * z / f  # mean 25 to 55 pixels right of the image
    P[:, 1] = rng.uniform(-40.0, 40.0, n) * z / f
    P[:, 2] = z + 1.0e-3 * np.arange(n)
    P[:, 3:6] = [5.9, -12.0, -12.0]  # 1.8e10 by 307 pixels (sigma)
    P[:, 6] = 1.0
    P[:, 10:13] = rng.normal(0.0, 1.0, (n, 3))
    P[:, 13] = -2.0
    cam = dict(R=[1, 0, 0, 0, 1, 0, 0, 0, 1], t=[0, 0, 0], f=f, cx=W / 2, cy=H / 2, w=W, h=H)
    params, sh = P.reshape(-1), np.zeros(n * 9, np.float32)
    opts = dict(shDeg=1, **(dict(entriesCap=700) if budget else {}))
    t, targets, metas = make(params, sh, [cam], [scene.uniform_target(W, H, seed=5)], opts, radius=1.0)
    gpu_raster(t, [0], 3)
    g, _, _, b = check_view_against_oracle(t, oracle_opts(opts), oracle_cam(metas[0], 0, 1, 1), params, sh, targets, n)
    x0 = g["rect"][0::2] & 0xFFFF
    assert (x0[g["rect"][0::2] != 0xFFFFFFFF] > 0).any() and (g["img"].reshape(H, W, 4)[:16, 64:, 3] > 0.5).all()
    assert b["dropped"].any() == bool(budget)
