"""EM with the tensor-core M-step when an iteration writes no posterior rows:
the rows after the last iteration (reached or converged early), a restart that
needs them mid-way, and the same model again on held buffers.

Tolerances: posteriors of one E-step against another of the same parameters
are the same kernel's (equal); parameters against the exact path's are within
the FP32 mode's own distance from it on a few iterations, 1e-4."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _data(N, D, K, seed, spread=2.0):
    r = np.random.Generator(np.random.PCG64(seed))
    mu = spread * r.standard_normal((K, D))
    x = (mu[r.integers(0, K, N)] + r.standard_normal((N, D))).astype(np.float32)
    return x, mu.astype(np.float32)


def _em(vl, x, mu, precision, iters):
    import torch
    K, D = mu.shape
    g = vl.GMM(D, K, np.float32)
    g.set_initialization("custom")
    g.set_means(mu)
    g.set_covariances(np.full((K, D), 1.5, np.float32))
    g.set_priors(np.full(K, 1.0 / K, np.float32))
    g.set_covariance_lower_bound(1e-3)
    g.set_max_num_iterations(iters)
    t = torch.from_numpy(x).cuda()
    return g, g.em_device(t, precision), t


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
@pytest.mark.parametrize("iters", [0, 2, 60])
def test_posteriors_after_em(vl, precision, iters):
    import torch
    x, mu = _data(3001, 64, 16, 1)
    g, ll, t = _em(vl, x, mu + 0.3, precision, iters)
    if iters == 60:
        assert len(g.ll_trace) < 61  # converged before the limit
    p = [torch.from_numpy(v).cuda() for v in (g.priors, g.means, g.covariances)]
    q = torch.zeros((3001, 16), device="cuda")
    ll2 = vl.gmm_posteriors_device(q, *p, t, precision)
    assert ll2 == ll
    assert np.array_equal(g.posteriors, q.cpu().numpy())


@pytest.mark.parametrize("precision", ["fp32", "bf16"])
def test_restart_needs_rows(vl, precision):
    x, mu = _data(6000, 64, 8, 2, spread=0.4)
    mu[3] += 40.0  # empties at once and restarts at the third iteration
    exact, _, _ = _em(vl, x, mu, "exact", 4)
    g, _, _ = _em(vl, x, mu, precision, 4)
    assert exact.num_restarts >= 1 and g.num_restarts == exact.num_restarts
    tol = 1e-4 if precision == "fp32" else 1e-2
    for a, b in ((g.means, exact.means), (g.covariances, exact.covariances), (g.priors, exact.priors)):
        assert rel_err(a, b) < tol


def test_same_model_again(vl):
    x, mu = _data(5000, 128, 264, 3)
    g, ll, t = _em(vl, x, mu, "fp32", 3)
    first = (g.means, g.covariances, g.priors)
    g.set_means(mu)
    g.set_covariances(np.full(mu.shape, 1.5, np.float32))
    g.set_priors(np.full(len(mu), 1.0 / len(mu), np.float32))
    assert g.em_device(t, "fp32") == ll
    for a, b in zip(first, (g.means, g.covariances, g.priors)):
        assert np.array_equal(a, b)
