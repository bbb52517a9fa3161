"""The calls' kernels at the sizes where they change shape: the LM's warps
and CTAs, the mask of a pose, the inlier scan, the admission of mixed host arrays."""
import numpy as np
import pytest

from turboransac_b200 import (BundleOptions_cuda, Camera_cuda, CameraPose_cuda, RansacOptions_cuda, estimate_batch,
                              scenes)

pytestmark = pytest.mark.gpu


def quat_angle(a, b):
    a, b = np.asarray(a) / np.linalg.norm(a), np.asarray(b) / np.linalg.norm(b)
    return 4.0 * np.arcsin(0.5 * min(np.linalg.norm(a - b), np.linalg.norm(a + b)))


def cam_of(f):
    return Camera_cuda(1, 640, 480, list(f.K))


def options(**kw):
    return RansacOptions_cuda(max_iterations=64, max_reproj_error=4.0, **kw)


def page_locked(a):
    import torch
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    t.numpy()[:] = a
    return t.numpy()


def unaligned(a):
    """A contiguous copy that starts 8 bytes off a 16-byte boundary."""
    buf = np.empty(a.size + 2)
    start = 0 if buf.ctypes.data % 16 else 1
    out = buf[start:start + a.size].reshape(a.shape)
    out[:] = a
    assert out.ctypes.data % 16 == 8
    return out


LM_SIZES = [4, 31, 32, 33, 127, 129, 255, 257, 383, 384, 385, 511, 513, 767, 768, 769, 1025, 1537, 2999, 3000, 3001,
            4097]


def test_lm_shapes_alone_and_in_a_large_batch(ctx, oracle):
    """All right matches, so the LM works on n inliers: one CTA's warps and rounds and
    the cluster around their edges. Alone and among 130 frames: the same bits; the
    oracle's pose within the pose bar (1e-6)."""
    frames = [scenes.make_frame(n, 1.0, 0.3, 7000 + n) for n in LM_SIZES]
    many = frames + [scenes.make_frame(40 + 3 * i, 0.9, 0.5, 8000 + i) for i in range(130 - len(frames))]
    got = estimate_batch(ctx, many, options())
    few = estimate_batch(ctx, frames[:5], options())
    for i, f in enumerate(frames):
        st, pose, _ = ctx.estimate_absolute_pose(f.uv, f.xyz, cam_of(f), options(), BundleOptions_cuda(), seed=f.seed)
        np.testing.assert_array_equal(got[i]["q"], pose.q)
        np.testing.assert_array_equal(got[i]["t"], pose.t)
        if i < len(few):
            np.testing.assert_array_equal(few[i]["q"], pose.q)
            np.testing.assert_array_equal(few[i]["t"], pose.t)
        o = oracle.estimate(f.uv, f.xyz, f.K, 4.0, seed=f.seed, samples_per_round=64, threads=8)
        assert quat_angle(pose.q, o["q"]) < 1e-6 and np.abs(pose.t - o["t"]).max() < 1e-6


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("n", [7, 8, 31, 33, 255, 257, 3071, 3073, 20001])
def test_bundle_adjust_sizes(ctx, oracle, n, weighted):
    """Slices of 0 to 2501 points a CTA, odd row counts in the admission's pieces."""
    f = scenes.make_frame(n, 1.0, 0.5, 600 + n)
    rng = np.random.default_rng(n)
    w = rng.uniform(0.5, 2.0, n) if weighted else None
    q0 = oracle.rotmat_to_quat(f.R_gt) + 1e-3 * rng.standard_normal(4)
    q0, t0 = q0 / np.linalg.norm(q0), f.t_gt + 1e-2 * rng.standard_normal(3)
    kw = dict(weights=w, honor_options=True) if weighted else {}
    pose, st = ctx.bundle_adjust(f.uv, f.xyz, cam_of(f), CameraPose_cuda(q0, t0), BundleOptions_cuda(loss_scale=1.0, loss_type=3),
                                 **kw)
    oq, ot, _ = oracle.lm(f.uv, f.xyz, f.K, q0, t0, loss_scale=1.0, loss=0, weights=w)
    assert quat_angle(pose.q, oq) < 1e-6 and np.abs(pose.t - ot).max() < 1e-6


@pytest.mark.parametrize("layout", [np.ascontiguousarray, page_locked, unaligned],
                         ids=["pageable", "page-locked", "unaligned"])
@pytest.mark.parametrize("n", [1, 2, 15, 17, 255, 256, 257, 3276, 3277, 20001, 151553])
def test_mask_of_a_pose(ctx, oracle, n, layout):
    f = scenes.make_frame(max(n, 4), 0.5, 1.0, 40 + n)
    xn = np.ascontiguousarray(((f.uv - [f.K[2], f.K[3]]) / [f.K[0], f.K[1]])[:n])
    X = np.ascontiguousarray(f.xyz[:n])
    thr = 16.0 / (0.5 * (f.K[0] + f.K[1])) ** 2
    q = oracle.rotmat_to_quat(f.R_gt)
    m = ctx.get_inliers(CameraPose_cuda(q, f.t_gt), layout(xn), layout(X), thr)
    np.testing.assert_array_equal(m, oracle.get_inliers(q, f.t_gt, xn, X, thr))


@pytest.mark.parametrize("n", [3, 31, 33, 255, 2047, 2049, 16385, 65537, 262143, 262145, 300001])
def test_inlier_scan_sizes(ctx, oracle, n):
    """The mask of the RANSAC pose and its count (one turn of the scan and several)."""
    f = scenes.make_frame(n, 0.7, 0.5, 900 + n)
    st, pose, m = ctx.estimate_absolute_pose(f.uv, f.xyz, cam_of(f), options(), BundleOptions_cuda(), seed=f.seed,
                                             skip_refine=True)
    assert st.details["num_inliers"] == int(np.count_nonzero(m))
    xn = np.ascontiguousarray((f.uv - [f.K[2], f.K[3]]) / [f.K[0], f.K[1]])
    thr = 16.0 / (0.5 * (f.K[0] + f.K[1])) ** 2
    want = oracle.get_inliers(pose.q, pose.t, xn, f.xyz, thr)
    r = np.flatnonzero(np.asarray(m).astype(bool) != np.asarray(want).astype(bool))
    assert r.size == 0


def test_mixed_host_arrays(ctx):
    """One small host batch of pageable, page-locked and unaligned arrays, below and
    above the size at which page-locked ones are read in place: each frame as alone."""
    import copy
    frames, sizes = [], [3, 15, 16, 17, 64, 65, 3276, 3277, 8191, 12000, 64, 5000]
    for i, n in enumerate(sizes):
        f = copy.copy(scenes.make_frame(n, 0.8, 0.5, 300 + i))
        put = (np.ascontiguousarray, page_locked, unaligned)[i % 3]
        f.uv = put(f.uv)
        f.xyz = (page_locked if i % 4 == 1 else put)(f.xyz)
        frames.append(f)
    for f, r in zip(frames, estimate_batch(ctx, frames, options(), masks=True)):
        st, pose, one = ctx.estimate_absolute_pose(np.array(f.uv), np.array(f.xyz), cam_of(f), options(),
                                                   BundleOptions_cuda(), seed=f.seed)
        np.testing.assert_array_equal(r["q"], pose.q)
        np.testing.assert_array_equal(r["t"], pose.t)
        np.testing.assert_array_equal(r["inliers"].astype(bool), np.asarray(one).astype(bool))


ONE_PROCESSOR = """
import os
os.sched_setaffinity(0, {min(os.sched_getaffinity(0))})
import numpy as np
from turboransac_b200 import Context, RansacOptions_cuda, estimate_batch, scenes
ctx = Context(0, 1 << 30)
frames = [scenes.make_frame(30000, 0.6, 0.5, 50 + i) for i in range(%d)]
r = estimate_batch(ctx, frames, RansacOptions_cuda(max_iterations=64, max_reproj_error=4.0))
assert len(r) == len(frames) and all(x["num_inliers"] > 15000 for x in r)
"""


@pytest.mark.parametrize("frames", [1, 2, 5, 16])
def test_host_copies_without_helper_threads(frames):
    """A process bound to one processor has no helpers to copy for it: one frame, a
    small batch, an ingested one (6 MB) and one whose ingestion overlaps its run (19 MB)."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", ONE_PROCESSOR % frames], cwd=root, check=True, timeout=120)


def off_boundary(a):
    """Page-locked, 4 bytes off an 8-byte boundary (a view into packed records, say)."""
    import torch
    raw = torch.empty(a.nbytes + 8, dtype=torch.uint8, pin_memory=True).numpy()
    out = raw[4:4 + a.nbytes].view(np.float64).reshape(a.shape)
    out[:] = a
    assert out.ctypes.data % 8 == 4
    return out


@pytest.mark.parametrize("frames", [1, 3, 6])
def test_page_locked_arrays_off_their_boundary(ctx, oracle, frames):
    """Read from a staging copy, not in place: a frame alone, a small batch and an
    ingested one (7 MB), a pose's mask and a bundle adjustment."""
    import copy
    fr = [scenes.make_frame(30000, 0.6, 0.5, 70 + i) for i in range(frames)]
    odd = []
    for f in fr:
        g = copy.copy(f)
        g.uv, g.xyz = off_boundary(f.uv), off_boundary(f.xyz)
        odd.append(g)
    for a, b in zip(estimate_batch(ctx, fr, options()), estimate_batch(ctx, odd, options())):
        np.testing.assert_array_equal(a["q"], b["q"])
        np.testing.assert_array_equal(a["t"], b["t"])
    f = fr[0]
    xn = np.ascontiguousarray((f.uv - [f.K[2], f.K[3]]) / [f.K[0], f.K[1]])
    pose = CameraPose_cuda(oracle.rotmat_to_quat(f.R_gt), f.t_gt)
    thr = 16.0 / (0.5 * (f.K[0] + f.K[1])) ** 2
    np.testing.assert_array_equal(ctx.get_inliers(pose, off_boundary(xn), odd[0].xyz, thr),
                                  ctx.get_inliers(pose, xn, f.xyz, thr))
    p0, _ = ctx.bundle_adjust(f.uv, f.xyz, cam_of(f), pose, BundleOptions_cuda(loss_scale=1.0))
    p1, _ = ctx.bundle_adjust(odd[0].uv, odd[0].xyz, cam_of(f), pose, BundleOptions_cuda(loss_scale=1.0))
    np.testing.assert_array_equal(p0.q, p1.q)
    np.testing.assert_array_equal(p0.t, p1.t)
