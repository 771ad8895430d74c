"""Exact Fisher encoding with very many components: above 32,752 the finalize
tabulates no factors (above about 116,000 the table would not fit in shared
memory), and above 1,048,560 a grid of 16 components per block has more than
65,535 rows.  Against the C restatement in
64 bits (its float sum of K exponentials in order is off by up to K u itself).

Tolerance (relative L2): a posterior carries a relative error of about
(D + 8) u L, with logits up to L = 60, and each element is a sum of at most 64
terms: 1e-4 in float, 1e-12 in double.  In float the signed square root is left
out: it would turn a posterior that rounding moves across the 1e-6 skip into 1e-3
of an element."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

TOL = {np.float32: 1e-4, np.float64: 1e-12}


@pytest.mark.parametrize("dtype,K,D,N,flags", [(np.float32, 32760, 1, 9, 2), (np.float64, 40000, 3, 20, 3),
                                               (np.float32, 131072, 2, 64, 0), (np.float32, 131072, 2, 64, 2),
                                               (np.float64, 131072, 1, 20, 3), (np.float64, 1100000, 1, 3, 3)])
def test_many_components(vl, restatement, dtype, K, D, N, flags):
    vl.set_precision("exact")
    r = np.random.Generator(np.random.PCG64(K + D))
    mu = (3 * r.standard_normal((K, D))).astype(dtype)
    cv = r.uniform(0.5, 2.0, (K, D)).astype(dtype)
    pr = r.uniform(0.5, 1.5, K)
    if K > 500000:
        pr[::5000] *= 2000.0  # the others are below the encoder's 1e-6
    pr = (pr / pr.sum()).astype(dtype)
    x = (mu[r.integers(0, K, N)] + r.standard_normal((N, D))).astype(dtype)
    enc, nt = vl.fisher_encode(x, mu, cv, pr, flags)
    ref, nref = restatement.fisher(*(v.astype(np.float64) for v in (x, mu, cv, pr)), flags)
    assert np.any(ref != 0)
    assert rel_err(enc, ref) < TOL[dtype]
    assert abs(nt - nref) <= max(1, 1e-3 * nref)
