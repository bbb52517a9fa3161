"""gpu_ms of a host call covers the call's whole device work: the points' preparation is
inside, as it is when the points come from device memory."""
import numpy as np
import pytest

from turboransac_b200 import (BundleOptions_cuda, Camera_cuda, DeviceFrame, RansacOptions_cuda, estimate_batch,
                              estimate_batch_device, scenes)

pytestmark = pytest.mark.gpu


def test_gpu_ms_covers_the_preparation(ctx):
    """One frame, the same steps: the interval of a call from host arrays holds the
    preparation (about 4 % of it here, repeated to 0.2 %), and may hold the ingestion."""
    f = scenes.make_frame(100000, 0.9, 1.0, 21)
    cam = Camera_cuda(1, 640, 480, [float(k) for k in f.K])
    ro = RansacOptions_cuda(max_iterations=64, max_reproj_error=4.0)
    d = [DeviceFrame(f)]
    host, batch, dev = [], [], []
    for _ in range(15):
        st, _, _ = ctx.estimate_absolute_pose(f.uv, f.xyz, cam, ro, BundleOptions_cuda(), seed=f.seed)
        host.append(st.details["gpu_ms"])
        batch.append(estimate_batch(ctx, [f], ro)[0]["gpu_ms"])
        dev.append(estimate_batch_device(ctx, d, ro)[0]["gpu_ms"])
    assert np.median(host[3:]) > 0.985 * np.median(dev[3:])
    assert np.median(batch[3:]) > 0.985 * np.median(dev[3:])
