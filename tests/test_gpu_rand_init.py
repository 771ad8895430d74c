"""Rand initialisation bit for bit at the edges of its kernels: the parallel
form of the sequential energy sum (tiles of 8192 terms, binade crossings,
exact ties, subnormal, zero and non-finite terms) and the row tiles of the
global variance.  NumPy's cumulative sums add strictly in order in the data
type, so they restate the reference's loops (vl/kmeans.c:588-649,
vl/gmm.c:1376-1413) for sizes the scalar restatement cannot reach."""
import numpy as np
import pytest

from oracle.oracle import MT19937, _l2_rows

pytestmark = pytest.mark.gpu


def _rand_init(x, K, seed, lanes):
    T = x.dtype.type
    N = x.shape[0]
    rng = MT19937(seed)
    with np.errstate(all="ignore"):
        mean = np.cumsum(x, axis=0, dtype=T)[-1] / T(N)
        ss = np.cumsum((x - mean) * (x - mean), axis=0, dtype=T)[-1]
        sigma = ss / T(N - 1) if N > 1 else np.zeros(x.shape[1], T)
        at = rng.uindex(N)
        mind = np.full(N, np.inf, T)
        centers = []
        for c in range(K):
            thresh = T(rng.real1())
            centers.append(x[at])
            if c + 1 == K:
                break
            dist = _l2_rows(x[at], x, lanes, T)
            mind = np.where(mind < dist, mind, dist)
            pre = np.cumsum(mind, dtype=T)
            hit = np.flatnonzero(pre >= T(thresh * pre[-1]))
            at = int(min(hit[0], N - 1)) if hit.size else N - 1
    return np.array(centers), sigma


def _data(kind, N, D, r):
    if kind == "normal":
        return r.standard_normal((N, D))
    if kind == "grid":  # small integers: exact ties and repeated rows
        return r.integers(0, 3, (N, D)) * 0.5
    if kind == "range":  # squares over the whole exponent range, subnormal ones among them
        return r.standard_normal((N, D)) * 10.0 ** r.uniform(-23, 6, (N, 1))
    if kind == "tiny":
        return r.standard_normal((N, D)) * 1e-22
    x = r.standard_normal((N, D))
    x[N // 2, 0] = np.inf if kind == "inf" else np.nan
    return x


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["normal", "grid", "range", "tiny", "inf", "nan"])
@pytest.mark.parametrize("N,D", [(1, 3), (7, 8), (128, 33), (8191, 1), (8192, 12), (8193, 5), (40001, 16)])
def test_rand_init_bits(vl, kind, N, D, dtype):
    K = min(N, 7)
    x = _data(kind, N, D, np.random.Generator(np.random.PCG64(N + D))).astype(dtype)
    f = dtype == np.float32
    lanes = (8 if f else 4) if vl.lib().vl_cpu_has_avx() else (4 if f else 2) if vl.lib().vl_cpu_has_sse2() else 1
    for seed in (3, 11):
        means, sigma = _rand_init(x, K, seed, lanes)
        g = vl.GMM(D, K, dtype)
        vl.rand_seed(seed)
        vl.lib().vl_gmm_init_with_rand_data(g._h, x.ctypes.data, N)
        assert np.array_equal(g.means, means, equal_nan=True)
        assert np.array_equal(g.covariances, np.tile(sigma, (K, 1)), equal_nan=True)
