"""Integrate's brick plan (8^3 bricks a frame cannot change are not visited) vs the FP64
oracle, which visits every voxel (the last size takes the listed form, the others the
one-launch form): empty volumes and volumes full of old content, sizes that
are not multiples of a brick, cameras inside and outside, depths that are zero or not numbers;
and the flags it works from against flags rebuilt from the volume."""
import numpy as np
import pytest

import kf_oracle as O
from helpers import integrate_ambiguous, small_workload
from oglfusionkinectv2_b200 import GFusion, _lib as L

pytestmark = pytest.mark.gpu

STORAGES = [L.KF_STORAGE_F32F32, L.KF_STORAGE_F16U16, L.KF_STORAGE_RG16I]


def old_content(size, storage, seed):
    """Random values and weights in every voxel but a zero block."""
    nx, ny, nz = size
    rng = np.random.default_rng(seed)
    F = rng.uniform(-1, 1, (nz, ny, nx)).astype(np.float32)
    W = rng.integers(0, 30, (nz, ny, nx))
    F[: nz // 3], W[: nz // 3] = 0, 0
    if storage == L.KF_STORAGE_F32F32:
        planes = F, W.astype(np.float32)
    elif storage == L.KF_STORAGE_F16U16:
        planes = F.astype(np.float16), W.astype(np.uint16)
    else:
        planes = (F * 32766).astype(np.int16), W.astype(np.int16)
    return np.concatenate([p.ravel().view(np.uint8) for p in planes])


@pytest.mark.parametrize("storage", STORAGES)
@pytest.mark.parametrize("size", [(4, 5, 6), (33, 20, 17), (64, 64, 64), (100, 52, 41), (200, 163, 180)])
@pytest.mark.parametrize("full", [False, True])
def test_plan_matches_dense_oracle(storage, size, full):
    w = small_workload(3, size=64, storage=storage, quirks=L.KF_QUIRKS_TRACKING if size[0] != 64 else L.KF_QUIRKS_DEFAULT)
    w.config.volumeSize = size
    w.config.mu = max(0.03, 1.5 / min(size))
    g, o = GFusion(w.config, w.intrinsics), O.Oracle(w.config, w.intrinsics)
    if full:
        raw = old_content(size, storage, 5)
        for s in (g, o):
            s.setVolumeRaw(raw)
    outside, inside = w.poses[1].copy(), w.poses[2].copy()
    outside[:3, 3] -= 0.9 * outside[:3, 2]
    inside[:3, 3] += 0.8 * inside[:3, 2]
    holes = w.frame(2).astype(np.float32)
    holes[100:180, 40:300] = 0.0
    holes[:, 400:] = 0.0
    holes[300:340, 100:200] = np.nan
    for pose, f in ((w.poses[0], w.frame(0)), (outside, w.frame(1)), (inside, holes)):
        oldF, oldW = o.getVolume()
        g.setVolumeRaw(o.getVolumeRaw())  # the same content on both sides before every frame
        for s in (g, o):
            s.setPose(pose)
            s.depthToVertex(f)
            s.integrate()
        Fg, Wg = g.getVolume()
        Fo, Wo = o.getVolume()
        bad = (np.abs(Fg - Fo) > 1e-3) | (Wg != Wo)
        idx = np.nonzero(bad)
        amb = integrate_ambiguous(w.config, w.intrinsics, pose, np.asarray(f), oldF, oldW, idx)
        assert amb.all(), f"{(~amb).sum()} unexplained voxel mismatches"
    assert (Wo > 0).any()


@pytest.mark.parametrize("storage", STORAGES)
def test_kept_flags_match_rebuilt_flags(storage):
    """40 frames (across flag refreshes) of a camera that turns away and back: the flags a
    session keeps and flags rebuilt from its volume before every frame give the same bits."""
    w = small_workload(40, size=72, storage=storage, quirks=L.KF_QUIRKS_TRACKING)
    a, b = GFusion(w.config, w.intrinsics), GFusion(w.config, w.intrinsics)
    for k in range(40):
        pose = w.poses[k].copy()
        pose[:3, 3] += 0.3 * np.sin(0.4 * k) * pose[:3, 2]
        f = w.frame(k)
        b.setVolumeRaw(b.getVolumeRaw())
        for s in (a, b):
            s.setPose(pose)
            s.depthToVertex(f)
            s.integrate()
            s.raycast()
        if k % 8 == 7:
            np.testing.assert_array_equal(a.getVolumeRaw(), b.getVolumeRaw())
            np.testing.assert_array_equal(a.getVerts(), b.getVerts())
            np.testing.assert_array_equal(a.getNorms(), b.getNorms())


FAR = np.eye(4)
FAR[:3, 3] = -1e200, 0.0, -1e200  # finite, but beyond FP32: x / z of every voxel is inf / inf
MIXED = np.zeros((4, 4))  # not rigid: the inverse's first row is not a number, the others are
MIXED[:3, 0], MIXED[2, 2], MIXED[:, 3] = (1e200, -1e200, 0.0), 1.0, (1e200, 1e200, -1.0, 1.0)


@pytest.mark.parametrize("storage", STORAGES)
@pytest.mark.parametrize("size", [(33, 20, 17), (64, 64, 64), (170, 165, 161)])
@pytest.mark.parametrize("pose", [FAR, MIXED])
def test_positions_that_are_not_numbers(storage, size, pose):
    """A voxel whose u is not a number reads column 0 (v is row 212 here), and its distance is not
    a number either: not above -mu, hence zeroed, unless that pixel holds no depth."""
    w = small_workload(1, size=64, storage=storage)
    w.config.volumeSize = size
    g = GFusion(w.config, w.intrinsics)
    raw = old_content(size, storage, 7)
    f = np.full((424, 512), 900.0, np.float32)
    for d, expect in ((0.0, raw), (900.0, np.zeros_like(raw))):
        f[212, 0] = d
        g.setVolumeRaw(raw)
        g.setPose(pose)
        g.depthToVertex(f)
        g.integrate()
        np.testing.assert_array_equal(g.getVolumeRaw(), expect)


@pytest.mark.parametrize("storage", STORAGES)
def test_kept_flags_match_rebuilt_flags_in_the_listed_form(storage):
    """As above for 12,075 bricks, whose integrate takes the plan and its list; 20 frames, across a
    refresh of the flags."""
    w = small_workload(20, size=72, storage=storage, quirks=L.KF_QUIRKS_TRACKING)
    w.config.volumeSize = (200, 163, 180)
    a, b = GFusion(w.config, w.intrinsics), GFusion(w.config, w.intrinsics)
    for k in range(20):
        pose = w.poses[k].copy()
        pose[:3, 3] += 0.3 * np.sin(0.4 * k) * pose[:3, 2]
        f = w.frame(k)
        b.setVolumeRaw(b.getVolumeRaw())
        for s in (a, b):
            s.setPose(pose)
            s.depthToVertex(f)
            s.integrate()
            s.raycast()
        if k % 5 == 4:
            np.testing.assert_array_equal(a.getVolumeRaw(), b.getVolumeRaw())
            np.testing.assert_array_equal(a.getVerts(), b.getVerts())
            np.testing.assert_array_equal(a.getNorms(), b.getNorms())
