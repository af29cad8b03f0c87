"""The warp-per-block rasteriser against the oracle where it can go wrong
(B200 required): more composited entries in a block than its exponential
cache holds, pixels and whole blocks without a target, blocks cut by the
image's edge, colours large enough for the clamped sums, every tile size
(block bits at 16, cull tests at 32, whole tiles at 8), and one block per
tile group instead of the work queue.  All bit for bit."""
import numpy as np
import pytest

from splat_b200 import scene
from test_gpu_parity import check_view_against_oracle, deep_tile_scene, gpu_raster, make, oracle_cam, oracle_opts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bright", [0, 1])
@pytest.mark.parametrize("persistent", [0, 1])
@pytest.mark.parametrize("tile", [8, 16, 32])
def test_warp_raster_bitexact(tile, persistent, bright):
    W, H, n = 75, 53, 4000
    params, cam = deep_tile_scene(n, seed=3, W=W, H=H)
    rng = np.random.default_rng(tile + bright)
    sh = rng.normal(0.0, 0.05, n * 9).astype(np.float32)
    if bright:  # a tenth of the splats hundreds of times brighter than white
        sh.reshape(n, 9)[rng.choice(n, n // 10, replace=False)] *= 1.0e4
    rgb = scene.uniform_target(W, H, seed=6).reshape(H, W, 3)
    rgb[8:16, 16:24] = -1.0  # a block without targets
    rgb[rng.random((H, W)) < 0.1] = -1.0
    opts = dict(shDeg=1, tile=tile, persistent=persistent)
    t, targets, metas = make(params, sh, [cam], [rgb.reshape(-1)], opts, radius=1.0)
    gpu_raster(t, [0], 3)
    _, r, _, _ = check_view_against_oracle(t, oracle_opts(opts), oracle_cam(metas[0], 0, 1, 1), params, sh, targets, n)
    assert np.asarray(r["end"]).max() > 600  # far more than the 256 entries a warp's cache holds
    gpu_raster(t, [0], 1)                    # forward only: the same image
    check = make(params, sh, [cam], [rgb.reshape(-1)], dict(opts, tile=16), radius=1.0)[0]
    a, b = t.renderTrainCam(0), check.renderTrainCam(0)
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
