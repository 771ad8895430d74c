"""GPU test of the tensor-core statistics kernel's rings of x rows, operands and
q^T: images shorter than a chunk, and long enough to
go round each ring many times.  The rings' depths order nothing, so depths of 2,
3 and as many as fit give the same bits; the default is compared with the FP64
C restatement (relative L2 error per Fisher vector: FP32 mode 1e-4, BF16 mode
1e-3, as in the tensor-core parity tests)."""
import numpy as np
import pytest

from conftest import rel_err
from oracle.oracle import FLAG_IMPROVED

pytestmark = pytest.mark.gpu

TOL = {"fp32": 1e-4, "bf16": 1e-3}
COUNTS = np.array([1, 31, 32, 33, 0, 1021, 5003])


@pytest.mark.parametrize("mode", ["fp32", "bf16"])
@pytest.mark.parametrize("D,K", [(64, 64), (80, 64), (80, 256), (128, 256)])
def test_ring_depths(vl, restatement, D, K, mode):
    import torch
    from vlfeat_b200 import workloads as W
    pr, mu, cv = W.fv_gmm(K, D, seed=3)
    offs = np.concatenate([[0], np.cumsum(COUNTS)]).astype(np.int64)
    x = W.pca_like(int(offs[-1]), D, seed=4)
    g = [torch.from_numpy(np.ascontiguousarray(a)).to("cuda") for a in (mu, cv, pr)]
    xt = torch.from_numpy(x).to("cuda")
    out = []
    for stages in (0, 2, 3):
        p = vl.FisherPlan(D, K, offs, FLAG_IMPROVED, mode)
        p.set_gmm(*g)
        p.set_config(item_rows=4096, stats_stages=stages)
        enc = torch.zeros((len(COUNTS), 2 * K * D), device="cuda")
        p.execute(enc, xt)
        assert p.status() == 0
        out.append(enc.cpu().numpy())
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    for j in range(len(COUNTS)):
        e, _ = restatement.fisher(x[offs[j]:offs[j + 1]].astype(np.float64), mu.astype(np.float64),
                                  cv.astype(np.float64), pr.astype(np.float64), FLAG_IMPROVED)
        if COUNTS[j] == 0:
            assert np.all(out[0][j] == 0)
        else:
            assert rel_err(out[0][j], e) < TOL[mode], j
