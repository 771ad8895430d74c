"""GPU tests of the tensor-core statistics kernel's rings in each of its builds:
all features in a CTA with one or two tiles of components (stats_mt 1 and 2; a few
work items would otherwise split the features), the split build (stats_mt 0, few
items), and the padded build of 96 dimensions with rows of fewer floats.  The
rings' depths and the tiles order nothing, so all give the same bits; compared
with the FP64 C restatement (relative L2 error per Fisher vector: FP32 mode 1e-4,
BF16 mode 1e-3, as in the tensor-core parity tests)."""
import numpy as np
import pytest

from conftest import rel_err
from oracle.oracle import FLAG_IMPROVED

pytestmark = pytest.mark.gpu

TOL = {"fp32": 1e-4, "bf16": 1e-3}
LONG = [1, 31, 32, 33, 0, 1021, 5003]
# Items of 1 to 10 chunks of 32 rows: fewer than, as many as and more than a
# ring is deep, so that a loader leaves with all its copies in flight.
SHORT = [32 * c - c % 3 for c in range(1, 11)]


def _data(D, K, counts):
    from vlfeat_b200 import workloads as W
    pr, mu, cv = W.fv_gmm(K, D, seed=3)
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    return pr, mu, cv, offs, W.pca_like(int(offs[-1]), D, seed=4)


def _check(restatement, enc, pr, mu, cv, offs, x, tol, images):
    for j in images:
        e, _ = restatement.fisher(*(v.astype(np.float64) for v in (x[offs[j]:offs[j + 1]], mu, cv, pr)), FLAG_IMPROVED)
        assert np.all(enc[j] == 0) if offs[j] == offs[j + 1] else rel_err(enc[j], e) < tol, j


@pytest.mark.parametrize("mode", ["fp32", "bf16"])
@pytest.mark.parametrize("D,K,counts", [(64, 64, LONG), (80, 64, LONG), (80, 256, LONG), (128, 256, LONG),
                                        (64, 256, SHORT), (80, 256, SHORT), (128, 128, SHORT)])
def test_depths(vl, restatement, D, K, counts, mode):
    import torch
    pr, mu, cv, offs, x = _data(D, K, counts)
    g = [torch.from_numpy(np.ascontiguousarray(a)).to("cuda") for a in (mu, cv, pr)]
    xt = torch.from_numpy(x).to("cuda")
    first = None
    for mt in (1, 2, 0):
        for stages in (0, 2, 3, 4):
            p = vl.FisherPlan(D, K, offs, FLAG_IMPROVED, mode)
            p.set_gmm(*g)
            p.set_config(item_rows=4096, stats_mt=mt, stats_stages=stages)
            enc = torch.zeros((len(counts), 2 * K * D), device="cuda")
            p.execute(enc, xt)
            assert p.status() == 0
            out = enc.cpu().numpy()
            first = out if first is None else first
            assert np.array_equal(out, first), (mt, stages)
    _check(restatement, first, pr, mu, cv, offs, x, TOL[mode], range(len(counts)))


@pytest.mark.parametrize("mode", ["fp32", "bf16"])
@pytest.mark.parametrize("D,K", [(81, 64), (84, 256), (90, 128), (96, 256)])
def test_padded(vl, restatement, D, K, mode):
    """Enough images that every CTA has its own items, in the 96-dimension build."""
    import torch
    counts = np.random.Generator(np.random.PCG64(D)).integers(0, 400, 170)
    pr, mu, cv, offs, x = _data(D, K, counts)
    enc = torch.zeros((len(counts), 2 * K * D), device="cuda")
    t = [torch.from_numpy(np.ascontiguousarray(a)).to("cuda") for a in (mu, cv, pr, x)]
    vl.fisher_encode_batch_device(enc, *t, offs, FLAG_IMPROVED, mode)
    _check(restatement, enc.cpu().numpy(), pr, mu, cv, offs, x, TOL[mode], range(0, len(counts), 13))
