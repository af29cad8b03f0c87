"""Restarting training from a written model (B200 required).

gs_write_gaussians + gs_reset_moments + the iteration counter put a trainer
back in the state setup() leaves: the same steps then give the same
parameters, SH coefficients and Adam moments, bit for bit.  The benchmark
starts every timed segment this way."""
import numpy as np
import pytest

from splat_b200 import scene
from splat_b200.trainer import GSTrainer
from test_gpu_parity import assert_bits, config0, make

GS_E_INVALID = -1

pytestmark = pytest.mark.gpu


def test_write_and_reset_moments_restart_training_exactly():
    params, sh, cams, rgbs = config0()
    t, _, _ = make(params, sh, cams, rgbs, dict(shDeg=2), radius=1.0)

    def run():
        t.iter = 2000
        for _ in range(3):
            t.stepBatch([0])
        g = t.readGaussians()
        return g["data"].copy(), g["sh"].copy(), [x.copy() for x in t.readMoments()]

    p1, s1, m1 = run()
    assert not np.array_equal(p1, params)
    assert np.any(m1[0] != 0)
    # training on from here leaves other moments; the reset returns to setup's
    t.stepBatch([0])
    t.writeGaussians(params, sh)
    t.resetMoments()
    assert all(not np.any(x) for x in t.readMoments())
    p2, s2, m2 = run()
    assert_bits(p2, p1, "params after the restart")
    assert_bits(s2, s1, "SH after the restart")
    for a, b, name in zip(m2, m1, ("m", "v", "SH m", "SH v")):
        assert_bits(a, b, f"Adam {name} after the restart")


def test_second_setup_forgets_the_first_ones_raster():
    """setup() again with a smaller view: refine's tile telemetry covers no
    tile and the introspection calls have no raster until a pass has run."""
    import ctypes as C
    from splat_b200 import native as N
    n = 2000
    params, sh = scene.uniform_scene(n, seed=3, sh_deg=2)
    params.reshape(-1, 16)[:, 13] += 2.0
    t = None
    for w, h in [(640, 360), (64, 48)]:
        cam = dict(scene.ring_cameras(1, 3.0, 0.0, w, h)[0], imgIdx=0)
        images = [dict(tw=w, th=h, rgb=scene.uniform_target(w, h, seed=1))]
        first = t is None
        t = t or GSTrainer.create(dict(shDeg=2, maxSplats=2 * n))
        t.setup(dict(data=params, n=n, sh=sh), [cam], images, w, h, 1.0)
        if first:
            t.stepBatch([0])
            assert t.refine(iter([0.5] * 10**6).__next__)["maxTile"] > 0
        else:
            rect = np.zeros(n * 2, np.uint32)
            assert N.lib().gs_debug_records(t._h, 0, None, N.ptr(rect, C.c_uint32)) == GS_E_INVALID
            assert t.refine(iter([0.5] * 10**6).__next__)["maxTile"] == 0
            t.stepBatch([0])
            assert t._state().lastLaunches > 0
