"""The warp-per-block rasteriser against the oracle where it can go wrong
(B200 required): more composited entries in a block than its exponential
cache holds, pixels and whole blocks without a target, blocks cut by the
image's edge, colours large enough for the clamped sums, every tile size
(block bits at 16, cull tests at 32, whole tiles at 8), and one block per
tile group instead of the work queue.  All bit for bit."""
import numpy as np
import pytest

from splat_b200 import scene
from oracle import oracle as O
from test_gpu_parity import (assert_bits, check_view_against_oracle, deep_tile_scene, gpu_raster, gpu_view, make,
                             oracle_cam, oracle_opts)

pytestmark = pytest.mark.gpu


# budget 60000: the entries' buffers cannot hold the cache, which gets its own
# allocation of 256 entries a warp; 768000: it lies in the buffers, 247 deep;
# 0 (12M entries): there, 1024 deep
@pytest.mark.parametrize("budget", [0, 60000, 768000])
@pytest.mark.parametrize("bright", [0, 1])
@pytest.mark.parametrize("persistent", [0, 1])
@pytest.mark.parametrize("tile", [8, 16, 32])
def test_warp_raster_bitexact(tile, persistent, bright, budget):
    W, H, n = 75, 53, 4000
    params, cam = deep_tile_scene(n, seed=3, W=W, H=H)
    rng = np.random.default_rng(tile + bright)
    sh = rng.normal(0.0, 0.05, n * 9).astype(np.float32)
    if bright:  # a tenth of the splats hundreds of times brighter than white
        sh.reshape(n, 9)[rng.choice(n, n // 10, replace=False)] *= 1.0e4
    rgb = scene.uniform_target(W, H, seed=6).reshape(H, W, 3)
    rgb[8:16, 16:24] = -1.0  # a block without targets
    rgb[rng.random((H, W)) < 0.1] = -1.0
    opts = dict(shDeg=1, tile=tile, persistent=persistent, **(dict(entriesCap=budget) if budget else {}))
    t, targets, metas = make(params, sh, [cam], [rgb.reshape(-1)], opts, radius=1.0)
    gpu_raster(t, [0], 3)
    _, r, _, b = check_view_against_oracle(t, oracle_opts(opts), oracle_cam(metas[0], 0, 1, 1), params, sh, targets, n)
    assert not b["dropped"].any() and np.asarray(r["end"]).max() > 600  # far more than 256 entries in a block
    assert_bits(t.renderTrainCam(0).reshape(-1), r["img"], "forward-only image")


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("tile", [8, 16, 32])
def test_infinite_colours_stay_where_they_composite(tile, variant):
    """A model may hold SH coefficients that are infinite, or so large that
    their sum is: a pixel that does not composite such a splat keeps its
    colour, and its gradients, in every part of the backward (cached entries
    and those past the cache, with pixels whose own loss is infinite beside
    finite ones).  The oracle visits only what a pixel composites."""
    W, H, n = 75, 53, 4000
    params, cam = deep_tile_scene(n, seed=4, W=W, H=H)
    P = params.reshape(-1, 16)
    rng = np.random.default_rng(tile)
    P[:, 0] = rng.uniform(-0.8, 0.8, n)  # wider and larger: no pixel composites more than a part of them
    P[:, 1] = rng.uniform(-0.5, 0.5, n)
    P[:, 3:6] += 0.8
    P[:, 13] += 0.7
    sh = rng.normal(0.0, 0.05, n * 9).astype(np.float32)
    wild = rng.choice(n, 24, replace=False)
    sh.reshape(n, 9)[wild[:8], ::4] = np.inf
    sh.reshape(n, 9)[wild[8:16], :] = rng.choice([-3.0e38, 3.0e38], (8, 9))
    sh.reshape(n, 9)[wild[16:], 0] = np.nan  # a colour of NaN is 0
    rgb = scene.uniform_target(W, H, seed=6).reshape(H, W, 3)
    rgb[rng.random((H, W)) < 0.1] = -1.0
    opts = dict(shDeg=1, tile=tile, backwardVariant=variant)
    t, targets, metas = make(params, sh, [cam], [rgb.reshape(-1)], opts, radius=1.0)
    o, c = oracle_opts(opts), oracle_cam(metas[0], 0, 1, 1)
    proj = O.project(o, c, params, sh, n)
    b = O.bin_tiles(o, c, proj, n)
    r = O.render(o, c, proj, b, targets, n, train=True, ncams=1, variant=variant)
    img = np.asarray(r["img"]).reshape(H, W, 4)
    bad = np.isinf(img[..., :3]).any(-1)
    assert 0.01 < bad.mean() < 0.5 and not np.isnan(img).any()
    assert np.asarray(r["end"]).max() > 300  # past the 256 entries a warp's cache holds
    gpu_raster(t, [0], 3)
    g = gpu_view(t, 0, metas[0], n, tile=tile)
    assert_bits(g["img"], r["img"], "image")
    assert_bits(g["finalT"], r["finalT"], "final transmittance")
    assert_bits(g["end"], r["end"], "end indices")
    assert_bits(g["gradP"], r["gradP"].reshape(-1, 16)[:, :10], "fixed-point screen-space gradients")
    assert_bits(t.renderTrainCam(0).reshape(-1), r["img"], "forward-only image")
