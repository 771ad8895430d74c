"""The exact E-step's tiles (components in blocks of 64 per pair of lane
slots, dimensions in 64-byte chunks, 8 or 16 rows per warp, two kernels above
256 components) at their edges, against the C restatement.

Tolerance: a logit is a sum of D products of size at most L, so either side
carries at most (D + 8) u L of rounding error, and a posterior moves by the
difference of two logits' errors on each side plus K u from the normaliser."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [(1, 1, 1), (31, 2, 7), (64, 3, 65), (65, 16, 129), (100, 17, 33), (128, 64, 31), (129, 80, 64), (192, 82, 40),
         (200, 33, 9), (256, 128, 130), (257, 20, 70), (300, 130, 37), (520, 8, 50), (64, 24, 37893), (128, 12, 37893)]


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("K,D,N", CASES)
def test_estep_tiles(vl, restatement, K, D, N, dtype):
    vl.set_precision("exact")
    r = np.random.Generator(np.random.PCG64(K * 1000 + D))
    mu = r.standard_normal((K, D)).astype(dtype)
    cv = r.uniform(0.5, 2.0, (K, D)).astype(dtype)
    pr = r.dirichlet(np.ones(K)).astype(dtype)
    x = (mu[r.integers(0, K, N)] + 0.7 * r.standard_normal((N, D))).astype(dtype)
    q, ll = vl.get_gmm_data_posteriors(x, pr, mu, cv)
    ref, refll = restatement.posteriors(x, pr, mu, cv)[:2]
    u = 2.0 ** (-24 if dtype == np.float32 else -53)
    x64, mu64, cv64 = (a.astype(np.float64) for a in (x[:200], mu, cv))
    L = float((((x64[:, None, :] - mu64[None]) ** 2) / cv64[None]).sum(2).max()) + D
    tol = 4 * (D + 8) * u * L + 2 * K * u
    assert np.max(np.abs(q - ref)) <= tol
    assert abs(ll - refll) <= tol * max(abs(refll), N)
