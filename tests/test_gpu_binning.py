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
