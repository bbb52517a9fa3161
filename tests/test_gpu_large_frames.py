"""One host frame on both sides of the size from which it is ingested (16 MiB, 419431
points): the results of the same points in device memory, bit for bit, from pageable and
page-locked arrays, alone, submitted and kept as a batch; and the oracle's scores."""
import copy

import numpy as np
import pytest

from helpers import normalized, sq_thr
from turboransac_b200 import (Batch, BundleOptions_cuda, Camera_cuda, DeviceFrame, RansacOptions_cuda,
                              estimate_batch_device, estimate_batch_submit, scenes)

pytestmark = pytest.mark.gpu


def page_locked(a):
    import torch
    return torch.from_numpy(a).pin_memory().numpy()


@pytest.mark.parametrize("n", [419430, 419431, 1000001])
def test_one_large_host_frame(ctx, n):
    f = scenes.make_frame(n, 0.5, 1.0, 77)
    ro = RansacOptions_cuda(max_iterations=64, max_reproj_error=4.0)
    ro.seed = f.seed
    cam = Camera_cuda(1, 640, 480, [float(k) for k in f.K])
    (d,) = estimate_batch_device(ctx, [DeviceFrame(f)], ro)
    assert d["status"] == 0 and d["num_inliers"] > 0.4 * n
    g = copy.copy(f)
    g.uv, g.xyz = page_locked(f.uv), page_locked(f.xyz)
    for h in (f, g):
        st, pose, m = ctx.estimate_absolute_pose(h.uv, h.xyz, cam, ro, BundleOptions_cuda(), seed=f.seed)
        assert np.count_nonzero(m) == d["num_inliers"] and st.details["best_sample"] == d["best_sample"]
        np.testing.assert_array_equal(pose.q, d["q"])
        np.testing.assert_array_equal(pose.t, d["t"])
        (r,) = estimate_batch_submit(ctx, [h], ro).collect()
        np.testing.assert_array_equal(r["q"], d["q"])
    b = Batch(ctx, [f], ro)
    b.run()
    (r,) = b.results()
    b.close()
    np.testing.assert_array_equal(r["q"], d["q"])


@pytest.mark.parametrize("n", [419430, 419431])
def test_scores_of_one_large_host_frame(ctx, oracle, n):
    f = scenes.make_frame(n, 0.5, 1.0, 78)
    tr = oracle.sample_triples(f.seed, 0, 12, n)
    ids, _, s32, _ = ctx.debug_score_samples(f.uv, f.xyz, f.K, 4.0, tr)
    o = oracle.ransac(normalized(f), f.xyz, sq_thr(f), dump=48, replay=tr, force_samples=12, samples_per_round=12)
    np.testing.assert_array_equal(ids, o["hyp_ids"])
    s64 = o["hyp_scores"] / sq_thr(f)
    part = 1.5 * 2.0 ** -22 / np.sqrt(sq_thr(f)) * np.minimum(np.sqrt(n * s64), n - s64)
    assert (np.abs(s32 - s64) <= np.maximum(s64 / 65536 + 0.25, part)).all()
