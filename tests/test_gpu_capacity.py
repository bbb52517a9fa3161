"""What a workspace holds: samples of one round and points of one frame, which do not
shrink with what else is kept beside them."""
import numpy as np
import pytest

from turboransac_b200 import CameraPose_cuda, Context, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mib,samples,points", [(256, 40764, 715904), (512, 110669, 1943808)])
def test_samples_and_points_of_a_workspace(mib, samples, points):
    """Four hypotheses a sample, 288 bytes each of 30 % of the workspace, after the
    records of 1024 frames and their candidates; the rest of it points."""
    c = Context(0, mib << 20)
    f = scenes.make_frame(64, 1.0, 0.5, 3)
    tr = np.stack([np.arange(samples) % 62, np.arange(samples) % 62 + 1, np.full(samples, 63)], 1).astype(np.int32)
    ids, _, _, _ = c.debug_score_samples(f.uv, f.xyz, f.K, 4.0, tr)
    assert len(ids) > samples // 4
    x, X = np.zeros((points, 2)), np.tile([0.0, 0.0, 1.0], (points, 1))
    m = c.get_inliers(CameraPose_cuda(np.array([1.0, 0, 0, 0]), np.zeros(3)), x, X, 1.0)
    assert int(np.count_nonzero(m)) == points
    c.close()
