"""The LM's sums cross the lanes of a warp in FP64: a gradient whose large terms
cancel keeps a remainder 51 bits below them."""
import numpy as np
import pytest

from turboransac_b200 import BundleOptions_cuda, Camera_cuda, CameraPose_cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [(0, 16, 8, 1, 17), (4, 20, 12, 5, 21), (0, 16, 4, 1, 17), (2, 18, 10, 6, 22)])
def test_cancelling_terms_keep_fp64_bits(ctx, lanes):
    """32 points at (0, 0, 1) seen with f = 1 by the first of the cluster's eight CTAs (the
    others' points weigh nothing): residuals 1, B, C, -1, -B along x, with
    B = 2^-24 + 2^-47 and C = 2^-51, so that the x gradient is C exactly, in FP64 in any
    order, while 48 bits lose it. One damped step from the identity then moves t_x by
    -C / (2 W + lambda), W = 32 the weight; y has residuals of 1, so that the step is
    accepted and t_y moves by -32 / (2 W + lambda)."""
    n = 256
    X = np.tile([0.0, 0.0, 1.0], (n, 1))
    r = np.zeros((n, 2))
    b, c = 2.0 ** -24 + 2.0 ** -47, 2.0 ** -51
    r[list(lanes), 0] = [1.0, b, c, -1.0, -b]
    r[:32, 1] = 1.0
    w = np.zeros(n)
    w[:32] = 1.0
    opt = BundleOptions_cuda(max_iterations=1, loss_type=0, loss_scale=1.0, gradient_tol=0.0, step_tol=0.0,
                             initial_lambda=1.0)
    cam = Camera_cuda(1, 2, 2, [1.0, 1.0, 0.0, 0.0])
    pose, st = ctx.bundle_adjust(-r, X, cam, CameraPose_cuda(np.array([1.0, 0.0, 0.0, 0.0]), np.zeros(3)), opt,
                                 weights=w, honor_options=True)
    assert st["lm_iterations"] == 1 and st["lm_invalid_steps"] == 0
    np.testing.assert_allclose(pose.t[1], -32.0 / 65.0, rtol=1e-12)
    np.testing.assert_allclose(pose.t[0], -c / 65.0, rtol=1e-9)
