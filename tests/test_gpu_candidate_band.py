"""The FP64 re-rank sees the FP64 best hypothesis where FP32 scores are far off: narrow
thresholds, distant outliers and near points in a deep scene.

A score's error is held against its bound, from which the band of re-ranked candidates is
made: s/65536 + 1/4, or 1.5 * 2^-22 / tau * min(sqrt(n s), n - s) if that is more. Then
pairs of hypotheses are looked for whose FP32 scores are in the wrong order by more than
s/16384 + 1, what the first part alone makes the band: of each the FP64 best has to win."""
import numpy as np
import pytest

from helpers import normalized, sq_thr
from turboransac_b200 import BundleOptions_cuda, Camera_cuda, RansacOptions_cuda, scenes

pytestmark = pytest.mark.gpu


def frame(case):
    n, px, f = case["n"], case["px"], case.get("f", 525.0)
    fr = scenes.make_frame(n, case["w"], px / 4, 11 + n, K=(f, f, 319.5, 239.5), threshold_px=px)
    rng = np.random.default_rng(3)
    if "far" in case:  # one outlier in a hundred is far away
        out = np.flatnonzero(~fr.inlier_gt)[:max(1, n // 100)]
        fr.xyz[out] += case["far"] * rng.standard_normal((len(out), 3))
    if "deep" in case:  # depths over two decades
        Xc = (fr.xyz @ fr.R_gt.T + fr.t_gt) * np.exp(rng.uniform(0, np.log(case["deep"]), n))[:, None]
        fr.xyz = np.ascontiguousarray((Xc - fr.t_gt) @ fr.R_gt)
    return fr


CASES = [dict(n=200000, w=0.95, px=0.25), dict(n=100000, w=0.95, px=0.5, f=2000.0),
         dict(n=100000, w=0.95, px=4.0, deep=100.0), dict(n=20000, w=0.8, px=4.0, far=1000.0),
         dict(n=20000, w=0.95, px=1.0, far=100.0)]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()))
def test_selection_where_fp32_scores_are_far_off(ctx, oracle, case):
    f = frame(case)
    px, m = case["px"], 600
    rng = np.random.default_rng(1)
    good = np.flatnonzero(f.inlier_gt)
    tr = np.stack([rng.choice(good, 3, replace=False) for _ in range(m)]).astype(np.int32)
    ids, _, s32, _ = ctx.debug_score_samples(f.uv, f.xyz, f.K, px, tr)
    o = oracle.ransac(normalized(f), f.xyz, sq_thr(f, px), dump=4 * m, replay=tr, force_samples=m, samples_per_round=m)
    np.testing.assert_array_equal(ids, o["hyp_ids"])
    s64, s32, sample = o["hyp_scores"] / sq_thr(f, px), s32.astype(np.float64), ids >> 2
    top = np.argsort(s64)[:200]
    part = 1.5 * 2.0 ** -22 / np.sqrt(sq_thr(f, px)) * np.minimum(np.sqrt(f.n * s64), f.n - s64)
    assert (np.abs(s32 - s64) <= np.maximum(s64 / 65536 + 0.25, part))[top].all()
    a, b = np.meshgrid(top, top, indexing="ij")  # a is the better one by FP64
    off = np.where((s64[a] < s64[b]) & (sample[a] != sample[b]), s32[a] - s32[b] - (s32[b] / 16384 + 1), -1.0)
    order = np.argsort(off, axis=None)[::-1]
    pairs, seen = [], set()
    for k in order[:2000]:
        i, j = a.flat[k], b.flat[k]
        if off.flat[k] <= 0.05 or len(pairs) == 8:
            break
        if sample[i] not in seen and sample[j] not in seen:
            pairs.append((sample[i], sample[j]))
            seen.update(pairs[-1])
    cam = Camera_cuda(1, 640, 480, [float(k) for k in f.K])
    ro, bo = RansacOptions_cuda(max_iterations=m, max_reproj_error=px), BundleOptions_cuda()
    for i, j in pairs:
        st, _, _ = ctx.estimate_absolute_pose(f.uv, f.xyz, cam, ro, bo, replay=tr[[j, i]], force_samples=2, skip_refine=True)
        both = np.flatnonzero((sample == i) | (sample == j))
        best = both[np.argmin(s64[both])]
        assert st.details["best_sample"] == int(sample[best] == i)
        np.testing.assert_allclose(st.details["model_score"], s64[best] * sq_thr(f, px), rtol=1e-9)
    # All of them at once, as one round (scored in two passes) and in rounds of 50.
    for kw in (dict(replay=tr, force_samples=m), dict(replay=tr)):
        ro.max_iterations = m if "force_samples" in kw else 50
        st, _, _ = ctx.estimate_absolute_pose(f.uv, f.xyz, cam, ro, bo, skip_refine=True, **kw)
        used = sample < st.details["samples"]
        best = np.flatnonzero(used)[np.argmin(s64[used])]
        assert st.details["best_sample"] == sample[best]
        np.testing.assert_allclose(st.details["model_score"], s64[best] * sq_thr(f, px), rtol=1e-9)
