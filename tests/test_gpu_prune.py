"""Two-pass scoring (k_prune): the default shape, which drops hypotheses after a
random prefix of the points, must select what the one-pass FP32 shape selects,
from the same samples, whatever the points' order and quality."""
import numpy as np
import pytest

from turboransac_b200 import BundleOptions_cuda, Camera_cuda, RansacOptions_cuda, scenes

pytestmark = pytest.mark.gpu

KEYS = ("samples", "rounds", "hypotheses", "best_sample", "best_solution", "ransac_inliers", "num_inliers", "model_score")


def points(case):
    n, w = case["n"], case["w"]
    f = scenes.make_frame(n, w, case.get("sigma", 1.0), 9000 + n)
    uv, xyz = f.uv.copy(), f.xyz.copy()
    order = {"sorted": np.argsort(~f.inlier_gt, kind="stable"), "reversed": np.argsort(f.inlier_gt, kind="stable"),
             "striped": np.argsort(np.arange(n) % 64, kind="stable")}.get(case.get("order"))
    if order is not None:
        uv, xyz = uv[order], xyz[order]
    if case.get("bad"):  # infinities and NaN among the points
        xyz[::97] = np.inf
        uv[5::89] = np.nan
    if case.get("copies"):  # every point many times: long runs of exact ties
        uv, xyz = uv[np.arange(n) % 50], xyz[np.arange(n) % 50]
    return f, np.ascontiguousarray(uv), np.ascontiguousarray(xyz)


CASES = [dict(n=1024, w=0.5), dict(n=1025, w=0.9), dict(n=1100, w=0.15, order="sorted"), dict(n=2047, w=0.3),
         dict(n=2049, w=0.6, order="reversed"), dict(n=4096, w=0.1), dict(n=5000, w=0.3, order="sorted"),
         dict(n=9999, w=0.05, order="reversed"), dict(n=16384, w=0.02), dict(n=20000, w=0.0),
         dict(n=20001, w=0.15, order="striped"), dict(n=30000, w=0.8, sigma=3.0), dict(n=50000, w=0.05, order="sorted"),
         dict(n=6000, w=0.4, bad=True), dict(n=6000, w=1.0, sigma=0.01), dict(n=3000, w=0.5, copies=True)]


@pytest.mark.parametrize("forced", [0, 20000], ids=["stop-rule", "forced"])
@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()))
def test_two_pass_selection_equals_one_pass(ctx, case, forced):
    f, uv, xyz = points(case)
    # Enough samples per round that the call scores in two passes.
    ro = RansacOptions_cuda(max_iterations=max(1000, -(-20_000_000 // (3 * case["n"] // 2)) + 1), max_reproj_error=4.0)
    cam = Camera_cuda(1, 640, 480, list(f.K))
    kw = dict(seed=f.seed, force_samples=forced)
    st, pose, inl = ctx.estimate_absolute_pose(uv, xyz, cam, ro, BundleOptions_cuda(), **kw)
    st1, pose1, inl1 = ctx.estimate_absolute_pose(uv, xyz, cam, ro, BundleOptions_cuda(), hyp_per_thread=4, **kw)
    for k in KEYS:
        assert st.details[k] == st1.details[k], k
    np.testing.assert_array_equal(inl, inl1)
    np.testing.assert_array_equal(pose.q, pose1.q)
    np.testing.assert_array_equal(pose.t, pose1.t)
