"""The statistics over passing rows (chunks of 128 or 64 rows, pairs of
dimensions with single ones between 64 and 96, one or four components per
warp, 16-, 8- and 4-byte copies) at their edges, against the C restatement.

Tolerances: those of the exact path against the reference's own arithmetic,
2e-5 relative in float and 1e-10 in double (each sum holds at most a few
thousand terms, so float sums carry at most about 1e-4 of their largest
partial sum and typically 1e-6)."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL = {np.float32: 2e-5, np.float64: 1e-10}


def _model(K, D, dtype, seed):
    r = np.random.Generator(np.random.PCG64(seed))
    mu = r.standard_normal((K, D)).astype(dtype)
    cv = r.uniform(1.0, 3.0, (K, D)).astype(dtype)
    pr = r.dirichlet(np.full(K, 2.0)).astype(dtype)
    return r, pr, mu, cv


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("K,D,N", [(1, 1, 1), (3, 2, 127), (17, 63, 128), (16, 64, 129), (33, 65, 300), (20, 96, 65),
                                   (18, 97, 64), (40, 128, 2049), (62, 82, 500)])
def test_fisher_one_image(vl, restatement, K, D, N, dtype):
    vl.set_precision("exact")
    r, pr, mu, cv = _model(K, D, dtype, K * 1000 + D)
    x = (mu[r.integers(0, K, N)] + r.standard_normal((N, D))).astype(dtype)
    enc, nt = vl.fisher_encode(x, mu, cv, pr, 0)
    ref, nref = restatement.fisher(x, mu, cv, pr, 0)
    assert rel_err(enc, ref) < TOL[dtype]
    assert abs(nt - nref) <= (0 if dtype == np.float64 else max(1, 1e-3 * nref))


@pytest.mark.parametrize("K,D", [(64, 80), (62, 33), (130, 128), (60, 64)])
def test_fisher_many_images(vl, restatement, K, D):
    import torch
    r, pr, mu, cv = _model(K, D, np.float32, K + D)
    counts = r.integers(0, 300, 170)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    x = (mu[r.integers(0, K, off[-1])] + r.standard_normal((off[-1], D))).astype(np.float32)
    enc = torch.zeros((len(counts), 2 * K * D), device="cuda")
    nt = torch.zeros(len(counts), dtype=torch.int64, device="cuda")
    t = [torch.from_numpy(a).cuda() for a in (mu, cv, pr, x)]
    vl.fisher_encode_batch_device(enc, *t, off, 0, "exact", nt)
    for j in list(range(0, len(counts), 17)) + [int(counts.argmax())]:
        ref, nref = restatement.fisher(x[off[j]:off[j + 1]], mu, cv, pr, 0)
        assert rel_err(enc[j].cpu().numpy(), ref) < TOL[np.float32]
        assert abs(int(nt[j]) - nref) <= max(1, 1e-3 * nref)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("K,D,N", [(17, 70, 900), (66, 64, 40000), (16, 128, 257)])
def test_em_step(vl, restatement, K, D, N, dtype):
    vl.set_precision("exact")
    r, pr, mu, cv = _model(K, D, dtype, K + N)
    x = (mu[r.integers(0, K, N)] + r.standard_normal((N, D))).astype(dtype)
    g = vl.GMM(D, K, dtype)
    g.set_initialization("custom")
    g.set_means(mu); g.set_covariances(cv); g.set_priors(pr)
    g.set_max_num_iterations(1)
    g.set_covariance_lower_bound(1e-4)
    g.cluster(x)
    q, _ = restatement.posteriors(x, pr, mu, cv)
    out = restatement.maximization(q, x, pr, mu, cv, np.full(D, 1e-4))
    for got, ref in zip((g.priors, g.means, g.covariances), out):
        assert rel_err(got, ref) < TOL[dtype]


@pytest.mark.parametrize("flags", [0, 3])
@pytest.mark.parametrize("dtype,K,D,N", [(np.float64, 1604, 130, 40), (np.float32, 2, 3, 5000), (np.float64, 9, 7, 4097)])
def test_fisher_finalize_parts(vl, restatement, dtype, K, D, N, flags):
    """A vector too long for the blocks' shared memory, one shorter than the
    cluster, and images of several segments."""
    vl.set_precision("exact")
    r, pr, mu, cv = _model(K, D, dtype, K + D)
    x = (mu[r.integers(0, K, N)] + r.standard_normal((N, D))).astype(dtype)
    enc, _ = vl.fisher_encode(x, mu, cv, pr, flags)
    ref, _ = restatement.fisher(x, mu, cv, pr, flags)
    assert rel_err(enc, ref) < TOL[dtype]


@pytest.mark.parametrize("N", [1, 255, 256, 257, 64 * 256, 64 * 256 + 1, 129 * 256])
def test_em_slab_counts(vl, restatement, N):
    """Slab sums of 1, 2, 64, 65 and 129 slabs (rounds of 64), in double."""
    r, pr, mu, cv = _model(3, 11, np.float64, N)
    x = mu[r.integers(0, 3, N)] + r.standard_normal((N, 11))
    g = vl.GMM(11, 3, np.float64)
    g.set_initialization("custom")
    g.set_means(mu); g.set_covariances(cv); g.set_priors(pr)
    g.set_max_num_iterations(1)
    g.set_covariance_lower_bound(1e-4)
    g.cluster(x)
    q, _ = restatement.posteriors(x, pr, mu, cv)
    for got, ref in zip((g.priors, g.means, g.covariances), restatement.maximization(q, x, pr, mu, cv, np.full(11, 1e-4))):
        assert rel_err(got, ref) < TOL[np.float64]
