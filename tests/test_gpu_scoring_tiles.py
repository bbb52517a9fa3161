"""The tensor-core scoring kernel at the edges of its tiles: 64-point tiles (two
32-point halves), 128-hypothesis blocks (32 a warp) and chunks of one, two and all
tiles, against the oracle's FP64 scores of the same samples.

Tolerance: the candidates re-ranked in FP64 are those within thr/32768 + 1/2 of
the running minimum (scores in tau^2 units), which holds the FP64 best as long as
each FP32 score is within half of that, s/65536 + 1/4, of its FP64 score."""
import numpy as np
import pytest

from helpers import normalized, sq_thr
from turboransac_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunk", [0, 64, 128])
@pytest.mark.parametrize("n,samples", [(3, 1), (31, 20), (33, 21), (63, 22), (64, 85), (65, 87), (129, 300),
                                       (1023, 1), (4097, 640), (70001, 90)])
def test_scores_at_tile_edges(ctx, oracle, n, samples, chunk):
    f = scenes.make_frame(n, 0.5, 1.0, 4000 + n)
    tr = oracle.sample_triples(f.seed, 0, samples, n)
    ids, _, s32, _ = ctx.debug_score_samples(f.uv, f.xyz, f.K, 4.0, tr,
                                             shape={"points_per_iter": 128, "chunk_points": chunk})
    o = oracle.ransac(normalized(f), f.xyz, sq_thr(f), dump=4 * samples, replay=tr, force_samples=samples,
                      samples_per_round=samples)
    np.testing.assert_array_equal(ids, o["hyp_ids"])
    s64 = o["hyp_scores"] / sq_thr(f)
    err = np.abs(s32.astype(np.float64) - s64)
    assert (err <= s64 / 65536 + 0.25).all(), err.max()
