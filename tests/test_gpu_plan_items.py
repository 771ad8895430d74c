"""The statistics' work items of small batches.  An explicit item_rows of a plan is
used as it is: an image's plain vector then has the same bits alone and among other
images (at a row offset that is a multiple of 8, the posterior image's row group),
and whatever larger value is given.  The default shortens items while they all run at
once, so the statistics' time has no step at any one row count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(vl, D, K, offs, flags, mode, x, **cfg):
    import torch
    from vlfeat_b200 import workloads as W
    pr, mu, cv = (torch.from_numpy(v).cuda() for v in W.fv_gmm(K, D, seed=3))
    p = vl.FisherPlan(D, K, offs, flags, mode)
    p.set_gmm(mu, cv, pr)
    if cfg:
        p.set_config(**cfg)
    enc = torch.zeros((len(offs) - 1, 2 * K * D), device="cuda")
    p.execute(enc, x)
    assert p.status() == 0
    return p, enc, (mu, cv, pr)


@pytest.mark.parametrize("mode", ["fp32", "bf16"])
@pytest.mark.parametrize("D,K,mt", [(80, 256, 0), (64, 64, 0), (128, 256, 1), (80, 256, 2)])
def test_explicit_item_rows(vl, D, K, mt, mode):
    import torch
    from vlfeat_b200 import workloads as W
    n, before, after = 3000, 4000, 2501
    x = torch.from_numpy(W.pca_like(before + n + after, D, seed=4)).cuda()
    alone = np.array([0, n], np.int64)
    batch = np.array([0, before, before + n, before + n + after], np.int64)
    xi = x[before:before + n].contiguous()
    out = {r: _plan(vl, D, K, alone, 0, mode, xi, item_rows=r, stats_mt=mt)[1][0] for r in (256, 4096, 16384)}
    among = {r: _plan(vl, D, K, batch, 0, mode, x, item_rows=r, stats_mt=mt)[1][1] for r in (256, 4096)}
    assert torch.equal(out[4096], out[16384])  # one item either way
    assert torch.equal(out[4096], among[4096]) and torch.equal(out[256], among[256])
    assert not torch.equal(out[256], out[4096])  # twelve items: other roundings


def test_config_round_trip_keeps_the_default(vl):
    """A saved configuration with the default rows stands for the built-in choice."""
    import torch
    from vlfeat_b200 import workloads as W
    x = torch.from_numpy(W.pca_like(3000, 80, seed=4)).cuda()
    offs = np.array([0, 3000], np.int64)
    p, enc, _ = _plan(vl, 80, 256, offs, 3, "fp32", x)
    saved = p.get_config()
    assert saved["item_rows"] == 8192
    assert torch.equal(_plan(vl, 80, 256, offs, 3, "fp32", x, **saved)[1], enc)


def test_no_step_in_time(vl):
    """Device time of the statistics of one image, K=256, D=80: 17 us up to 4,096
    rows and 84 at 4,097 when short items ended there.  Below twice per 500 rows."""
    import torch
    from vlfeat_b200 import workloads as W
    pr, mu, cv = (torch.from_numpy(v).cuda() for v in W.fv_gmm(256, 80, seed=3))
    x = torch.from_numpy(W.pca_like(9000, 80, seed=4)).cuda()
    enc = torch.zeros((1, 2 * 256 * 80), device="cuda")
    t = []
    for n in range(1000, 9001, 500):
        best = np.inf
        for i in range(6):
            vl.profile_reset()
            vl.profile_enable(True)
            vl.fisher_encode_batch_device(enc, mu, cv, pr, x[:n], np.array([0, n], np.int64), 3, "fp32")
            torch.cuda.synchronize()
            if i:
                best = min(best, vl.profile_read()["tc_stats_f16x3"][1])
            vl.profile_enable(False)
        t.append(best)
    vl.profile_reset()
    assert max(b / a for a, b in zip(t, t[1:])) < 2, t
