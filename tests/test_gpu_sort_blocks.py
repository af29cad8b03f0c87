"""The sorts around the sizes where their blocks change (B200 required): a
quarter block, and the last size sorted in quarter blocks.  The static sort
(votes, 32-bit keys) against numpy's stable sort; the presort (its first pass
drops culled items) and the entry sort, both with the OR form, and refine's sort
of 64-bit keys against the oracle.  Exactly equal."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
import rigs
from splat_b200 import native as N
from splat_b200 import scene
from test_gpu_parity import assert_bits, check_view_against_oracle, gpu_raster, make, oracle_cam, oracle_opts

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [8, 16])
@pytest.mark.parametrize("n", [1023, 1024, 1025, 4097, 262143, 262144, 262145])
def test_sort_at_block_sizes(n, bits):
    import torch
    rng = np.random.default_rng(n + bits)
    k = rng.integers(0, 1 << bits, n).astype(np.uint32)
    k[: n // 3] = 7  # long runs of one digit
    v = np.arange(n, dtype=np.uint32)
    dk, dv = torch.from_numpy(k.view(np.int32)).cuda(), torch.from_numpy(v.view(np.int32)).cuda()
    torch.cuda.synchronize()
    N.check(N.lib().gs_sort_entries_static(C.c_void_p(dk.data_ptr()), C.c_void_p(dv.data_ptr()), n, bits, None))
    order = np.argsort(k, kind="stable")
    assert np.array_equal(dk.cpu().numpy().view(np.uint32), k[order])
    assert np.array_equal(dv.cpu().numpy().view(np.uint32), v[order])


@pytest.mark.parametrize("live", [1023, 1024, 1025, 4097, 262143, 262144, 262145])
def test_presort_and_entry_sort_at_block_sizes(live):
    """`live` visible splats, each inside one tile (so as many entries), and a
    tenth as many behind the camera between them, with equal depths among the
    visible ones."""
    W, H, n = 64, 48, live + live // 10 + 1
    rng = np.random.default_rng(live)
    P = np.zeros((n, 16), np.float32)
    behind = np.zeros(n, bool)
    behind[rng.choice(n, n - live, replace=False)] = True
    z = (3.0 + rng.integers(0, max(2, live // 3), n) / live).astype(np.float32)  # about three splats a depth
    tile = rng.integers(0, 12, n)
    P[:, 0] = (tile % 4 * 16 + rng.uniform(7.0, 9.0, n) - W / 2) / 64.0 * z
    P[:, 1] = (tile // 4 * 16 + rng.uniform(7.0, 9.0, n) - H / 2) / 64.0 * z
    P[:, 2] = np.where(behind, -z, z)
    P[:, 3:6] = -5.0
    P[:, 6] = 1.0
    P[:, 10:13] = rng.normal(0.0, 1.0, (n, 3))
    P[:, 13] = rng.uniform(1.0, 3.0, n)
    cam = dict(R=[1, 0, 0, 0, 1, 0, 0, 0, 1], t=[0, 0, 0], f=64.0, cx=W / 2, cy=H / 2, w=W, h=H)
    params, sh = P.reshape(-1), np.zeros(n * 9, np.float32)
    opts = dict(shDeg=1, maxSplats=n, maxBatch=1)
    t, targets, metas = make(params, sh, [cam], [scene.uniform_target(W, H, seed=2)], opts, radius=1.0)
    gpu_raster(t, [0], 3)
    o = dict(opts, entriesCap=max(12_000_000, 24 * n))
    _, _, _, b = check_view_against_oracle(t, oracle_opts(o), oracle_cam(metas[0], 0, 1, 1), params, sh, targets, n)
    assert len(b["ids"]) == live


@pytest.mark.parametrize("donors", [1023, 1024, 1025, 262143, 262144, 262145])
def test_donor_sort_at_block_sizes(donors):
    """refine with exactly `donors` donors, many of equal size: its splits pick
    from the quarter of the sorted list that holds the largest."""
    n, K = donors + 60, 3
    rng = np.random.default_rng(donors)
    params, sh = scene.uniform_scene(n, seed=5, sh_deg=1)
    P = params.reshape(-1, 16)
    P[:, 3:6] = (rng.integers(0, max(2, donors // 4), n) / donors - 4.0)[:, None]
    P[:, 13] = 1.0
    P[rng.choice(n, 60, replace=False), 13] = -6.0  # dead
    cap = n + 3000
    cam = scene.ring_cameras(1, 3.0, 0.0, 64, 48)[0]
    t, _, _ = make(params, sh, [cam], [scene.uniform_target(64, 48, seed=3)], dict(shDeg=1, maxSplats=cap, maxBatch=1),
                   radius=1.0)
    t.iter = 2000
    t.growLimit = min(cap, n + max(300, n // 100))
    z = lambda k: np.zeros(cap * k, np.float32)
    op, osh = z(16), z(3 * K)
    op[:n * 16], osh[:n * 3 * K] = params, sh
    r_cpu = O.refine(n, cap, op, z(16), z(16), osh, z(3 * K), z(3 * K), K, rigs.lcg(7), t.iter, 0.75 * 60000,
                     growLimit=t.growLimit)
    r_gpu = t.refine(rigs.lcg(7))
    assert (r_gpu["moved"], r_gpu["grown"], r_gpu["n"]) == (r_cpu["moved"], r_cpu["grown"], r_cpu["n"])
    assert r_cpu["moved"] >= 52 and r_cpu["grown"] >= 150
    g = t.readGaussians()
    assert_bits(g["data"], op[:r_gpu["n"] * 16], "params after refine")
    assert_bits(g["sh"], osh[:r_gpu["n"] * 3 * K], "SH after refine")
