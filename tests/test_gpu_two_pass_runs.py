"""Two-pass scoring where it does run: the steps here hold more pairs than the line from
which a step is scored in two passes (4.5e7), the pairs scored say so, and the selection is
that of the FP32 shape, which scores every hypothesis on every point."""
import copy

import numpy as np
import pytest

from turboransac_b200 import Batch, RansacOptions_cuda, scenes

pytestmark = pytest.mark.gpu

KEYS = ("samples", "rounds", "hypotheses", "best_sample", "best_solution", "ransac_inliers", "num_inliers", "model_score")


def frame(n, w, order=None, bad=False):
    f = scenes.make_frame(n, w, 1.0, 9100 + n)
    if order == "sorted":
        k = np.argsort(~f.inlier_gt, kind="stable")
        f.uv, f.xyz = np.ascontiguousarray(f.uv[k]), np.ascontiguousarray(f.xyz[k])
    if bad:  # infinities and NaN among the points
        f.xyz[::97] = np.inf
        f.uv[5::89] = np.nan
    return f


def run(ctx, f, tune=False, **kw):
    """(results, pairs scored) of one run."""
    b = Batch(ctx, [copy.copy(f)], kw.pop("ro"), **kw)
    if tune:
        b.autotune(repeats=1)
    _, pairs = b.profile()
    (r,) = b.results()
    b.close()
    return r, pairs


def same(r, s):
    assert r["status"] == s["status"] == 0
    for k in KEYS:
        assert r[k] == s[k], k
    np.testing.assert_array_equal(r["q"], s["q"])
    np.testing.assert_array_equal(r["t"], s["t"])


# About 1.4 hypotheses a sample: 1e8 points against samples are some 1.4e8 pairs.
@pytest.mark.parametrize("n,w,kw", [(1024, 0.5, {}), (1025, 0.9, {}), (1100, 0.3, dict(order="sorted")), (2047, 0.3, {}),
                                    (2049, 0.6, dict(order="sorted")), (4096, 0.2, {}), (6000, 0.4, dict(bad=True)),
                                    (20001, 0.15, dict(order="sorted")), (50000, 0.8, {})])
def test_forced_samples_in_two_passes(ctx, n, w, kw):
    f = frame(n, w, **kw)
    ro, m = RansacOptions_cuda(max_iterations=1000, max_reproj_error=4.0), -(-100_000_000 // n)
    r, pairs = run(ctx, f, ro=ro, force_samples=m)
    s, all_pairs = run(ctx, f, ro=ro, force_samples=m, hyp_per_thread=4)
    assert all_pairs == r["hypotheses"] * n > 4.5e7
    assert pairs < 0.85 * all_pairs  # (a prefix of half the points at n = 1024, of less above)
    same(r, s)


@pytest.mark.parametrize("n,w,kw", [(5000, 0.1, {}), (9999, 0.08, dict(order="sorted")), (30000, 0.1, {}), (6000, 0.1, dict(bad=True))])
def test_rounds_in_two_passes(ctx, n, w, kw):
    """The stop rule's rounds: the first without a model, later ones bounded by the best so far."""
    f = frame(n, w, **kw)
    ro = RansacOptions_cuda(max_iterations=max(1000, -(-45_000_000 // n)), max_reproj_error=4.0)
    r, pairs = run(ctx, f, ro=ro)
    s, all_pairs = run(ctx, f, ro=ro, hyp_per_thread=4)
    assert r["rounds"] > 1 and pairs < 0.7 * r["hypotheses"] * n
    same(r, s)


@pytest.mark.parametrize("n", [1023, 1024, 5000])
def test_steps_below_the_line_are_scored_once(ctx, n):
    f = frame(n, 0.5)
    ro, m = RansacOptions_cuda(max_iterations=1000, max_reproj_error=4.0), 20_000_000 // n
    r, pairs = run(ctx, f, ro=ro, force_samples=m)
    assert pairs == r["hypotheses"] * n < 4.5e7
    s, _ = run(ctx, f, ro=ro, force_samples=m, hyp_per_thread=4)
    same(r, s)


@pytest.mark.parametrize("bad", [False, True])
def test_tuned_shape_repacks_the_points(ctx, bad):
    """autotune tries every shape on points staged for it, each in its own order, and
    leaves them as its winner reads them."""
    f = frame(6000, 0.3, bad=bad)
    ro = RansacOptions_cuda(max_iterations=8000, max_reproj_error=4.0)
    r, _ = run(ctx, f, ro=ro)
    s, _ = run(ctx, f, ro=ro, tune=True)
    same(r, s)
