"""Exact E-step on rows whose squares overflow the data type: a component far
from such a row has an infinite distance and posterior 0, one near it a finite
distance, and the components that pad K to the kernel's blocks must not show.
Against the C restatement in the same type.

Tolerance: as for the E-step's tiles, with a logit bounded by the largest finite
distance plus the constant's log-determinant."""
import numpy as np
import pytest

from oracle.oracle import FLAG_FAST, FLAG_IMPROVED

pytestmark = pytest.mark.gpu

# |x| = BIG overflows when squared; differences of BIG / 100 do not.
BIG = {np.float32: 1e20, np.float64: 1e155}


def _inputs(K, D, N, dtype):
    r = np.random.Generator(np.random.PCG64(K * 1000 + N))
    big = BIG[dtype]
    mu, cv = r.standard_normal((K, D)), r.uniform(0.5, 2.0, (K, D))
    far = np.arange(K)[-2:] if K > 2 else np.arange(K)[-1:]  # the far components, others around zero
    mu[far] = big * (1 + 1e-3 * r.standard_normal((len(far), D)))
    cv[far] = (big / 100) ** 2 * r.uniform(0.5, 2.0, (len(far), D))
    pr = r.uniform(0.5, 1.5, K)
    x = r.standard_normal((N, D))
    rows = np.arange(0, N, 3)
    x[rows] = big * (1 + 1e-2 * r.standard_normal((len(rows), D)))
    if K == len(far):
        x = x[rows]
    return x.astype(dtype), (pr / pr.sum()).astype(dtype), mu.astype(dtype), cv.astype(dtype), far


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("K,D,N", [(1, 5, 40), (3, 8, 70), (32, 7, 65), (64, 16, 40), (100, 12, 129), (150, 9, 70),
                                   (200, 20, 40), (256, 6, 33), (300, 10, 40), (20, 3, 37893), (100, 4, 37893)])
def test_overflowing_rows(vl, restatement, K, D, N, dtype):
    vl.set_precision("exact")
    x, pr, mu, cv, far = _inputs(K, D, N, dtype)
    with np.errstate(over="ignore"):
        assert np.isinf(x.max() * x.max())
    q, ll = vl.get_gmm_data_posteriors(x, pr, mu, cv)
    ref, refll = restatement.posteriors(x, pr, mu, cv)[:2]
    assert np.all(np.isfinite(ref)) and np.isfinite(refll)
    u = 2.0 ** (-24 if dtype == np.float32 else -53)
    with np.errstate(over="ignore"):
        dist = ((x[:200, None, :] - mu[None]) ** 2 / cv[None]).astype(np.float64).sum(2)
    L = float(dist[np.isfinite(dist)].max()) + float(np.abs(np.log(cv.astype(np.float64))).sum(1).max()) + 2 * D
    tol = 4 * (D + 8) * u * L + 2 * K * u
    assert np.max(np.abs(q - ref)) <= tol
    assert abs(ll - refll) <= tol * max(abs(refll), len(x))


@pytest.mark.parametrize("flags", [FLAG_IMPROVED, FLAG_IMPROVED | FLAG_FAST])
@pytest.mark.parametrize("K", [3, 100])
def test_encoding_of_overflowing_rows(vl, restatement, K, flags):
    vl.set_precision("exact")
    x, pr, mu, cv, far = _inputs(K, 8, 90, np.float32)
    enc, nt = vl.fisher_encode(x, mu, cv, pr, flags)
    ref, nref = restatement.fisher(x, mu, cv, pr, flags)
    assert np.all(np.isfinite(ref)) and nt == nref
    # Float statistics of 90 rows on either side, a signed square root of them:
    # an error of 90 u relative to the largest gives its square root.
    assert np.max(np.abs(enc - ref)) <= np.sqrt(90 * 2.0 ** -24) * np.max(np.abs(ref))
