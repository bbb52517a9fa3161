"""The two rules of two-pass scoring, on the CPU: the staging order is a bijection
whose prefixes sample structured subsets like a uniform draw, and the bound that
drops a hypothesis holds on exact hypergeometric tails."""
import math

import numpy as np
import pytest

U64 = (1 << 64) - 1


def stage_position(n, seed):
    """The staging order of tbr_kernels.cuh (stage_position), for all points."""
    bits = (n - 1).bit_length()
    mask, sh = np.uint64((1 << bits) - 1), np.uint64((bits + 1) // 2)
    keys, z = [], seed & U64
    for _ in range(6):
        z = (z + 0x9E3779B97F4A7C15) & U64
        k = z
        k = ((k ^ (k >> 30)) * 0xBF58476D1CE4E5B9) & U64
        k = ((k ^ (k >> 27)) * 0x94D049BB133111EB) & U64
        k ^= k >> 31
        keys.append((np.uint64((k & 0xFFFFFFFF) | 1), np.uint64(k >> 32)))

    def walk(x):
        for m, a in keys:
            x = (x * m + a) & np.uint64(0xFFFFFFFF) & mask
            x = x ^ (x >> sh)
        return x

    x = walk(np.arange(n, dtype=np.uint64))
    while (x >= n).any():
        x[x >= n] = walk(x[x >= n])
    return x.astype(np.int64)


@pytest.mark.parametrize("n", [1024, 1025, 1537, 4095, 4097, 30000, 65537])
def test_staging_order_is_a_bijection(n):
    for seed in (0, 1, 0xDEADBEEF12345678):
        assert np.array_equal(np.sort(stage_position(n, seed)), np.arange(n))


@pytest.mark.parametrize("n,m", [(1537, 512), (5000, 1024), (20000, 1024)])
def test_prefix_counts_of_structured_subsets_are_hypergeometric(n, m):
    i = np.arange(n)
    subsets = [i < n // 10, i < n // 2, i % 16 == 0, (i // 64) % 8 == 0, (i & 256) > 0]
    for k, s in enumerate(subsets):
        count = s.sum()
        mean = m * count / n
        sd = math.sqrt(mean * (1 - count / n) * (n - m) / (n - 1))
        z = np.array([((stage_position(n, 1000 * k + t)[s] < m).sum() - mean) / sd for t in range(200)])
        # 200 draws of a unit variable: the mean within 4.5 / sqrt(200), the
        # deviation within 4.5 / sqrt(400) of 1, no draw beyond 5.5.
        assert abs(z.mean()) < 0.32 and abs(z.std() - 1) < 0.23 and abs(z).max() < 5.5


def kl(x, mu):
    a = x * math.log(x / mu) if x > 0 else 0.0
    return a + (1 - x) * (math.log1p(-x) - math.log1p(-mu))


@pytest.mark.parametrize("n,good,m", [(2000, 100, 512), (2000, 900, 512), (30000, 2000, 1024), (50000, 600, 4096)])
def test_bound_holds_on_hypergeometric_tails(n, good, m):
    """ln P(X <= k) <= -m KL(k/m || good/n) for the hypergeometric X, all k below the mean."""
    lg = math.lgamma
    ch = lambda a, b: lg(a + 1) - lg(b + 1) - lg(a - b + 1)  # noqa: E731
    mu, tail = good / n, -math.inf
    for k in range(int(m * mu)):
        if m - k > n - good:
            continue
        t = ch(good, k) + ch(n - good, m - k) - ch(n, m)
        tail = max(tail, t) + math.log1p(math.exp(min(tail, t) - max(tail, t))) if tail > -math.inf else t
        assert tail <= -m * kl(k / m, mu) + 1e-6
