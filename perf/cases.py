"""Cases of the training step's performance: what a program that trains a
Gaussian-splat model with this library has it do, through GSTrainer and the
C ABI (include/splat_b200.h).

Four kinds of pass:

* ``train``: a burst of optimiser steps between two snapshots -- plain steps
  (``stepOnce``, one view each, the camera picked by the trainer) or batched
  ones (``stepBatch``, several views per step) -- then the loss and the whole
  model, read into the caller's pinned buffers;
* ``cycle``: batched steps, then ``refine`` at the splat cap (relocation with
  opacity-weighted donors), then the loss and the model;
* ``eval``: the held-out views' evaluation passes (forward, loss, backward to
  the camera, no optimiser), statistics and camera gradients back;
* ``render``: a viewer's frame, forward only, into a pinned host image.

Scenes are the synthetic ones of splat_b200.scene (uniform cube; surface
scene, with a share of fine splats for dense detail), drawn on the GPU from
the seed; training targets are rendered from a perturbed copy of the model
(the cube's are uniform-random images).
"""
from __future__ import annotations

import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "splat.js_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from splat_b200 import native as N  # noqa: E402
from splat_b200 import scene  # noqa: E402
from splat_b200.trainer import GSTrainer  # noqa: E402

# view sizes of the uneven batch: captured photo sets rarely have one size
UNEVEN = [(640, 360), (960, 540), (1280, 720), (1280, 720), (1600, 900), (1920, 1080), (1920, 1080), (1920, 1080)]


def listed():
    return [
        # a new session's first seconds: a seed cloud at preview size, plain
        # colour; every launch and every host call shows
        dict(name="train_4k_sh0_259x199", kind="train", scene="uniform", n=4003, sh=0, w=259, h=199, views=1, cams=6,
             steps=6, uneven=False, tile=16, depth=64),
        # small object, one camera, random target: the smallest benchmark configuration
        dict(name="train_20k_256", kind="train", scene="uniform", n=20000, sh=2, w=256, h=256, views=1, cams=1,
             steps=12, uneven=False, tile=16, depth=64),
        # a phone capture early on: odd sizes, first SH band, two views a step
        dict(name="batch2_137k_sh1_801x603", kind="train", scene="surface", n=137219, sh=1, w=801, h=603, views=2,
             cams=7, steps=12, uneven=False, tile=16, depth=64),
        # the ordinary run: plain steps, half a million splats, 720p
        dict(name="train_500k_720p", kind="train", scene="surface", n=500000, sh=2, w=1280, h=720, views=1, cams=12,
             steps=24, uneven=False, tile=16, depth=64),
        # plain steps at the benchmark's size
        dict(name="train_1M_1080p", kind="train", scene="surface", n=1000000, sh=2, w=1920, h=1080, views=1, cams=8,
             steps=24, uneven=False, tile=16, depth=64),
        # the benchmark's batched step: eight 1080p views
        dict(name="batch8_1M_1080p", kind="train", scene="surface", n=1000000, sh=2, w=1920, h=1080, views=8, cams=8,
             steps=8, uneven=False, tile=16, depth=64),
        # eight views of uneven size in one step
        dict(name="batch8_1M_uneven", kind="train", scene="surface", n=1000000, sh=2, w=1920, h=1080, views=8, cams=8,
             steps=8, uneven=True, tile=16, depth=64),
        # the largest training: two million splats, a fifth of them fine, every SH band, four 1080p views
        dict(name="batch4_2M_sh3_1080p", kind="train", scene="fine", n=2000000, sh=3, w=1920, h=1080, views=4, cams=4,
             steps=8, uneven=False, tile=16, depth=256),
        # the refinement schedule at the splat cap
        dict(name="cycle_300k_sh3_720p", kind="cycle", scene="fine", n=300000, sh=3, w=1280, h=720, views=4, cams=8,
             steps=16, uneven=False, tile=16, depth=256),
        # metrics: held-out views evaluated between bursts
        dict(name="eval_1M_1080p", kind="eval", scene="surface", n=1000000, sh=2, w=1920, h=1080, views=1, cams=4,
             steps=4, uneven=False, tile=16, depth=64),
        # the viewer on a finished model, and on a small one
        dict(name="render_1M_1080p", kind="render", scene="surface", n=1000000, sh=2, w=1920, h=1080, views=1, cams=4,
             steps=1, uneven=False, tile=16, depth=64),
        dict(name="render_20k_256", kind="render", scene="uniform", n=20000, sh=2, w=256, h=256, views=1, cams=1,
             steps=1, uneven=False, tile=16, depth=64),
    ]


def draw(rng):
    """A case of the same ranges: 3k-2M splats, every SH degree, 160-1920
    pixel wide views of odd sizes, 1-8 views a step."""
    kind = rng.choices(["train", "batch", "cycle", "eval", "render"], [35, 30, 10, 10, 15])[0]
    n = int(round(3000 * (2000000 / 3000) ** rng.random()))
    w = int(round(160 * (1920 / 160) ** rng.random()))
    h = max(90, min(1080, int(round(w * rng.uniform(0.5, 0.8)))))
    sh = rng.choice([0, 1, 2, 2, 3, 3])
    views = rng.randint(2, 8 if n <= 1000000 else 4) if kind in ("batch", "cycle") else 1
    cams = views if kind != "train" else rng.randint(1, 8)
    # passes of at most about 100 ms: the step's time grows with splats and pixels
    est = 0.2 + views * (0.3e-6 * n + 0.8e-6 * w * h) + 1.0e-6 * n
    steps = 1 if kind == "render" else rng.randint(2, 4) if kind == "eval" else \
        max(4, min(16, int(100.0 / est), rng.randint(6, 24)))
    if kind == "eval":
        cams = steps
    surface = "fine" if sh == 3 else "surface"
    return dict(kind="train" if kind == "batch" else kind, scene="uniform" if n < 30000 else surface, n=n, sh=sh, w=w,
                h=h, views=views, cams=cams, steps=steps, uneven=False, tile=rng.choice([16] * 8 + [8, 32]),
                depth=rng.choice([64, 64, 128, 256]))


def _coefs(case):
    return 3 * scene.sh_rest_coefs(case["sh"])


def _model(case, gen):
    """(params n*16, sh n*3K) of the case's scene as float32 arrays: the
    distributions of splat_b200.scene, drawn on the GPU."""
    n, dev = case["n"], "cuda"

    def normal(mean, std, *shape):
        return torch.randn(*shape, generator=gen, device=dev, dtype=torch.float32) * std + mean

    def uniform(lo, hi, *shape):
        return torch.rand(*shape, generator=gen, device=dev, dtype=torch.float32) * (hi - lo) + lo

    P = torch.zeros(n, 16, device=dev)
    if case["scene"] == "uniform":
        P[:, 0:3] = uniform(-1.0, 1.0, n, 3)
        P[:, 3:6] = normal(-4.0, 0.5, n, 3)
    else:  # 60% on three planes, 30% on the unit sphere, 10% on a radius-20 shell
        per, sph = n // 5, (3 * n) // 10
        pos = torch.zeros(n, 3, device=dev)
        for axis in range(3):
            a, b = [k for k in range(3) if k != axis]
            pos[axis * per:(axis + 1) * per, a] = uniform(-2.0, 2.0, per)
            pos[axis * per:(axis + 1) * per, b] = uniform(-2.0, 2.0, per)
        d = normal(0.0, 1.0, n - 3 * per, 3)
        d = d / d.norm(dim=1, keepdim=True)
        d[sph:] *= 20.0
        pos[3 * per:] = d
        P[:, 0:3] = pos[torch.randperm(n, generator=gen, device=dev)]
        P[:, 3:6] = normal(-5.0, 0.7, n, 3)
        if case["scene"] == "fine":
            pick = uniform(0.0, 1.0, n) < 0.2
            P[:, 3:6] = torch.where(pick[:, None], normal(-7.0, 0.5, n, 3), P[:, 3:6])
    q = normal(0.0, 1.0, n, 4)
    P[:, 6:10] = q / q.norm(dim=1, keepdim=True)
    c = (0.5 + scene.SH_C0 * normal(0.0, 0.3, n, 3)).clamp(1e-4, 1 - 1e-4)
    P[:, 10:13] = torch.log(c / (1 - c))
    P[:, 13] = normal(0.0, 1.0, n)
    if case["kind"] == "cycle":  # a model under way: a tenth of the splats have faded out
        P[:, 13] = torch.where(uniform(0.0, 1.0, n) < 0.1, normal(-4.5, 0.3, n), P[:, 13])
    sh = normal(0.0, 0.05, n * _coefs(case))
    return P.reshape(-1), sh


def _cameras(case):
    sizes = UNEVEN if case["uneven"] else [(case["w"], case["h"])] * case["cams"]
    cams = []
    for k, (w, h) in enumerate(sizes):
        radius, height = (3.0, 0.0) if case["scene"] == "uniform" else (4.0, 0.5)
        c = scene.ring_cameras(len(sizes), radius, height, w, h)[k]
        c["imgIdx"] = k
        cams.append(c)
    return cams


def _options(case, views):
    return dict(shDeg=case["sh"], maxSplats=case["n"], maxBatch=views, tile=case["tile"], batchDepth=case["depth"],
                donorSampling=1 if case["kind"] == "cycle" else 0)


def _pinned(*shape):
    return torch.zeros(*shape, dtype=torch.float32, pin_memory=True)


def _targets(case, cams, P, sh, gen):
    """One float32 RGB image per camera."""
    if case["scene"] == "uniform":
        return [dict(tw=c["w"], th=c["h"], rgb=torch.rand(c["w"] * c["h"] * 3, generator=gen, device="cuda").cpu().numpy())
                for c in cams]
    noise = 0.02 * torch.randn(case["n"], 16, generator=gen, device="cuda")
    noise[:, 14:] = 0.0
    pp = (P + noise.reshape(-1)).cpu().numpy()
    ps = (sh + 0.02 * torch.randn(sh.numel(), generator=gen, device="cuda")).cpu().numpy()
    t = GSTrainer.create(_options(case, 1))
    t.setup(dict(data=pp, n=case["n"], sh=ps), [dict(cams[0], imgIdx=0)],
            [dict(tw=1, th=1, rgb=np.zeros(3, np.float32))], max(c["w"] for c in cams), max(c["h"] for c in cams), 4.0)
    images = []
    for c in cams:
        frame = _pinned(c["h"], c["w"], 4)
        t.renderView(c, frame.numpy())
        rgb = frame.cuda()[..., :3].clamp(0.0, 1.0).contiguous().reshape(-1).cpu().numpy()
        images.append(dict(tw=c["w"], th=c["h"], rgb=rgb))
    return images


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    P, sh = _model(case, gen)
    cams = _cameras(case)
    if case["kind"] == "render":  # a viewer has no training targets
        images = [dict(tw=1, th=1, rgb=np.zeros(3, np.float32)) for _ in cams]
    else:
        images = _targets(case, cams, P, sh, gen)
    t = GSTrainer.create(_options(case, case["views"]))
    t.setup(dict(data=P.cpu().numpy(), n=case["n"], sh=sh.cpu().numpy()), cams, images,
            max(c["w"] for c in cams), max(c["h"] for c in cams), 3.0 if case["scene"] == "uniform" else 4.0)
    t.iter = 3000  # every SH band active
    t.rand = random.Random(seed).random
    state = dict(case=case, trainer=t, cams=cams)
    if case["kind"] == "render":
        state["frame"] = _pinned(case["h"], case["w"], 4)
        state["next"] = 0
    elif case["kind"] in ("train", "cycle"):
        state["params"] = _pinned(case["n"] * 16)
        state["sh"] = _pinned(max(1, case["n"] * _coefs(case)))
    return state


def _fp(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_float))


def run(state):
    case, t = state["case"], state["trainer"]
    L, h = N.lib(), t._h
    if case["kind"] == "render":  # the viewer orbits: another camera each frame
        cam = state["cams"][state["next"] % len(state["cams"])]
        state["next"] += 1
        t.renderView(cam, state["frame"].numpy())
        return state["frame"]
    if case["kind"] == "eval":
        out = []
        for ci in range(case["steps"]):
            stats = (C.c_uint32 * 4)()
            grads = np.zeros((len(state["cams"]) + 1) * 8, np.int32)
            N.check(L.gs_eval_pass(h, ci, None, stats, N.ptr(grads, C.c_int32)), h)
            out.append(dict(stats=np.frombuffer(stats, np.uint32).astype(np.int64), camGrad=grads))
        return out
    nc = len(state["cams"])
    for k in range(case["steps"]):
        if case["views"] == 1:
            t.stepOnce()
        else:
            t.stepBatch([(k * case["views"] + j) % nc for j in range(case["views"])])
    out = {}
    if case["kind"] == "cycle":
        out["refine"] = t.refine()
    out["loss"] = t.readLoss()
    N.check(L.gs_read_gaussians(h, _fp(state["params"]), _fp(state["sh"]), None), h)
    out["params"], out["sh"] = state["params"], state["sh"]
    return out


def work(case):
    """Bytes: a step reads and writes every parameter, SH coefficient and both
    their moments once and reads its targets; a pass also writes out the model
    (or the frame).  Flops: 26 forward and 70 backward per splat that a pixel
    composites; a pixel's light is used up after about 40 splats of the
    scenes' mean opacity, and it is covered by n * footprint / pixels."""
    n, row = case["n"], (16 + _coefs(case)) * 4
    sizes = UNEVEN if case["uneven"] else [(case["w"], case["h"])] * case["views"]
    pix = sum(w * h for w, h in sizes)
    scale, dist = (-4.0, 3.0) if case["scene"] == "uniform" else (-5.0, 4.0)
    pairs = 0.0
    for w, h in sizes:
        sigma2 = (math.exp(scale) * 1.171875 * w / dist) ** 2 + 0.3
        pairs += w * h * min(40.0, n * math.pi * 7.0 * sigma2 / (w * h))
    if case["kind"] == "render":
        return dict(bytes=float(n * row + pix * 16), flops=26.0 * pairs)
    if case["kind"] == "eval":
        return dict(bytes=float(case["steps"] * (n * row + pix * 4)), flops=case["steps"] * 96.0 * pairs)
    return dict(bytes=float(case["steps"] * (6 * n * row + pix * 4) + n * row), flops=case["steps"] * 96.0 * pairs)


# ---- the frame in 64 bits (plain torch) ------------------------------------
def exact(case, seed):
    """render: the image, in double precision from the same float32 model.
    The training kinds have none: a step's gradients are defined as sums of
    per-pixel integers (each pixel's term truncated to 1/16384), and the other
    kinds' outputs are those integers."""
    if case["kind"] != "render":
        return None
    gen = torch.Generator("cuda").manual_seed(seed)
    P, sh = _model(case, gen)
    cam = _cameras(case)[0]
    return _image64(P.reshape(-1, 16).double(), sh.double(), case["sh"], cam)


def _basis64(v):
    x, y, z = v[:, 0], v[:, 1], v[:, 2]
    xx, yy, zz = x * x, y * y, z * z
    c1 = math.sqrt(3 / (4 * math.pi))
    c2 = math.sqrt(15 / (4 * math.pi))
    c20 = math.sqrt(5 / (16 * math.pi))
    c22 = math.sqrt(15 / (16 * math.pi))
    a, b, c, d, e = (math.sqrt(35 / (32 * math.pi)), math.sqrt(105 / (4 * math.pi)), math.sqrt(21 / (32 * math.pi)),
                     math.sqrt(7 / (16 * math.pi)), math.sqrt(105 / (16 * math.pi)))
    return torch.stack([-c1 * y, c1 * z, -c1 * x,
                        c2 * x * y, -c2 * y * z, c20 * (2 * zz - xx - yy), -c2 * x * z, c22 * (xx - yy),
                        -a * y * (3 * xx - yy), b * x * y * z, -c * y * (4 * zz - xx - yy),
                        d * z * (2 * zz - 3 * xx - 3 * yy), -c * x * (4 * zz - xx - yy), e * z * (xx - yy),
                        -a * x * (xx - yy)], 1)


def _image64(P, sh, deg, cam, eCut=4.5, aMin=0.0039, tile=16):
    dev, W, H, f = P.device, cam["w"], cam["h"], float(np.float32(cam["f"]))
    R = torch.tensor(np.float32(cam["R"]).astype(np.float64).reshape(3, 3), device=dev)
    tr = torch.tensor(np.float32(cam["t"]).astype(np.float64), device=dev)
    pc = P[:, :3] @ R.T + tr
    P, pc, sh = (x[pc[:, 2] >= 0.05] for x in (P, pc, sh.reshape(len(P), -1)))
    q = P[:, 6:10] / P[:, 6:10].norm(dim=1, keepdim=True)
    w, x, y, z = q.T
    Q = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)
    M = Q * torch.exp(P[:, 3:6].clamp(-12.0, 6.0))[:, None, :]
    iz = 1.0 / pc[:, 2:3]
    T0 = f * iz * R[0] - f * pc[:, 0:1] * iz * iz * R[2]
    T1 = f * iz * R[1] - f * pc[:, 1:2] * iz * iz * R[2]
    m0, m1 = torch.einsum("nk,nkj->nj", T0, M), torch.einsum("nk,nkj->nj", T1, M)
    va, vb, vc = (m0 * m0).sum(1), (m0 * m1).sum(1), (m1 * m1).sum(1)
    ad, cd = va + 0.3, vc + 0.3
    det = ad * cd - vb * vb
    opa = torch.sigmoid(P[:, 13].clamp(-9.0, 9.0)) * torch.sqrt(((va * vc - vb * vb) / det).clamp_min(0.0))
    mx, my = f * pc[:, 0] * iz[:, 0] + cam["cx"], f * pc[:, 1] * iz[:, 0] + cam["cy"]
    mid = 0.5 * (ad + cd)
    lam = mid + torch.sqrt((mid * mid - det).clamp_min(0.0))
    emax = torch.log((opa / aMin).clamp_min(1.0001)).clamp_max(eCut)
    rad = torch.minimum(torch.sqrt(2 * emax * lam), torch.full_like(lam, float(W)))
    col = torch.sigmoid(P[:, 10:13].clamp(-9.0, 9.0))
    if deg:
        K = scene.sh_rest_coefs(deg)
        v = P[:, :3] + R.T @ tr
        v = v / v.norm(dim=1, keepdim=True)
        col = (col + torch.einsum("nk,nck->nc", _basis64(v)[:, :K], sh.reshape(-1, 3, K))).clamp_min(0.0)
    keep = (opa >= aMin) & (mx + rad >= 0) & (my + rad >= 0) & (mx - rad <= W) & (my - rad <= H)
    order = torch.argsort(pc[:, 2].masked_fill(~keep, math.inf))[:int(keep.sum())]
    mx, my, rad, opa, col = mx[order], my[order], rad[order], opa[order], col[order]
    hA, hB, hC = (0.5 * cd / det)[order], (-vb / det)[order], (0.5 * ad / det)[order]
    # (tile, splat) entries, nearest first in each tile
    tx, ty = -(-W // tile), -(-H // tile)
    x0, x1 = ((((mx + s * rad) / tile).floor()).clamp(0, tx - 1).long() for s in (-1, 1))
    y0, y1 = ((((my + s * rad) / tile).floor()).clamp(0, ty - 1).long() for s in (-1, 1))
    cnt = (x1 - x0 + 1) * (y1 - y0 + 1)
    ids = torch.repeat_interleave(torch.arange(len(cnt), device=dev), cnt)
    k = torch.arange(len(ids), device=dev) - (cnt.cumsum(0) - cnt)[ids]
    wide = (x1 - x0 + 1)[ids]
    tid, by = torch.sort((y0[ids] + k // wide) * tx + x0[ids] + k % wide, stable=True)
    ids = ids[by]
    lens = torch.bincount(tid, minlength=tx * ty)
    starts = lens.cumsum(0) - lens
    img = torch.zeros(ty * tile, tx * tile, 4, dtype=torch.float64, device=dev)
    px = torch.arange(tile * tile, device=dev)
    tiles = torch.argsort(lens, descending=True)[:int((lens > 0).sum())]
    at = 0
    while at < len(tiles):  # tiles of about the same length together
        longest = int(lens[tiles[at]])
        ts = tiles[at:at + max(1, min(512, 60000 // longest))]
        at += len(ts)
        X = (ts % tx)[:, None] * tile + px % tile
        Y = (ts // tx)[:, None] * tile + px // tile
        T = torch.ones(len(ts), tile * tile, dtype=torch.float64, device=dev)
        acc = torch.zeros(len(ts), tile * tile, 3, dtype=torch.float64, device=dev)
        for base in range(0, longest, 1024):
            j = base + torch.arange(min(1024, longest - base), device=dev)
            ok = j < lens[ts][:, None]
            e = ids[torch.where(ok, starts[ts][:, None] + j, 0)]
            dx, dy = X[:, None, :] + 0.5 - mx[e][..., None], Y[:, None, :] + 0.5 - my[e][..., None]
            ee = (hA[e][..., None] * dx * dx + hB[e][..., None] * dx * dy + hC[e][..., None] * dy * dy).clamp_min(0.0)
            a = (opa[e][..., None] * torch.exp(-ee)).clamp_max(0.99)
            a = torch.where(ok[..., None] & (ee <= eCut) & (a >= aMin), a, 0.0)
            before = T[:, None, :] * torch.cat([torch.ones_like(a[:, :1]), (1 - a).cumprod(1)[:, :-1]], 1)
            a = torch.where(before >= 1e-4, a, 0.0)  # a pixel stops once its light is used up
            acc += torch.einsum("tep,tec->tpc", before * a, col[e])
            T = T * (1 - a).prod(1)
        img[Y, X, :3] = acc
        img[Y, X, 3] = 1.0 - T
    return img[:H, :W].contiguous()
