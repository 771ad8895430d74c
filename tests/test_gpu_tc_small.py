"""The tensor-core encoder on one image and on a few small ones: the shortest
items that run at once, features split over CTAs, the wide finalize, and the
two sides of the 4,096-row rule, against the C restatement in double.

Tolerance: the E-step's posteriors are within 4e-5 of FP64 (its own bound), so
the plain vectors are held to 5e-5 relative; term counts to a few terms at the
1e-6 skip."""
import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _case(K, D, counts, seed):
    from vlfeat_b200 import workloads as W
    pr, mu, cv = W.fv_gmm(K, D, seed=seed)
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    return pr, mu, cv, off, W.pca_like(int(off[-1]), D, seed=seed + 1)


@pytest.mark.parametrize("mode", ["fp32", "bf16"])
@pytest.mark.parametrize("K,D,counts", [
    (8, 64, [1]), (64, 64, [255]), (64, 80, [257]), (256, 80, [4096]), (256, 80, [4097]), (136, 128, [900]),
    (512, 128, [700]), (104, 33, [513]), (256, 96, [130]), (256, 64, [0, 5, 0, 300, 1]), (256, 80, [40] * 30),
    (1024, 64, [300, 2000])])
def test_small_batches(vl, restatement, mode, K, D, counts):
    import torch
    pr, mu, cv, off, x = _case(K, D, counts, K + D)
    enc = torch.zeros((len(counts), 2 * K * D), device="cuda")
    nt = torch.zeros(len(counts), dtype=torch.int64, device="cuda")
    t = [torch.from_numpy(a).cuda() for a in (mu, cv, pr, x)]
    vl.fisher_encode_batch_device(enc, *t, off, 0, mode, nt)
    assert vl.last_precision() == mode
    d = [a.astype(np.float64) for a in (x, mu, cv, pr)]
    for j in range(len(counts)):
        ref, nref = restatement.fisher(d[0][off[j]:off[j + 1]], *d[1:], 0)
        got = enc[j].cpu().numpy()
        if counts[j] == 0:
            assert np.all(got == 0) and int(nt[j]) == 0
            continue
        assert rel_err(got, ref) < (5e-5 if mode == "fp32" else 1e-3)
        assert abs(int(nt[j]) - nref) <= max(2, 1e-3 * nref)


def test_prior_below_floor_and_rerun(vl, restatement):
    """Skipped components in the centred constants, and the same bits again
    (the preparation's block counter is cleared by each call)."""
    import torch
    pr, mu, cv, off, x = _case(64, 80, [600], 5)
    pr[::3] = 1e-8
    enc = [torch.zeros((1, 2 * 64 * 80), device="cuda") for _ in range(3)]
    t = [torch.from_numpy(a).cuda() for a in (mu, cv, pr, x)]
    for e in enc:
        vl.fisher_encode_batch_device(e, *t, off, 0, "fp32")
    ref, _ = restatement.fisher(*[a.astype(np.float64) for a in (x, mu, cv, pr)], 0)
    assert rel_err(enc[0][0].cpu().numpy(), ref) < 5e-5
    assert torch.equal(enc[0], enc[1]) and torch.equal(enc[0], enc[2])


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("K,D", [(64, 1), (64, 12), (64, 16), (72, 20), (256, 81), (264, 84), (256, 96), (264, 96),
                                 (256, 97), (264, 100), (512, 36)])
def test_padded_rows(vl, restatement, K, D, shift):
    """Dimensions the kernels pad: rows read where they are (multiples of 4,
    16-byte aligned) or copied (others; shift moves the data by one float),
    alone and in clusters of blocks, against the C restatement in double."""
    import torch
    pr, mu, cv, off, x = _case(K, D, [700, 0, 333], K + D)
    buf = torch.zeros(x.size + 1, device="cuda")
    t = buf[shift:shift + x.size].view(x.shape)
    t.copy_(torch.from_numpy(x))
    p = [torch.from_numpy(a).cuda() for a in (mu, cv, pr)]
    d = [a.astype(np.float64) for a in (x, mu, cv, pr)]
    enc = torch.zeros((3, 2 * K * D), device="cuda")
    vl.fisher_encode_batch_device(enc, *p, t, off, 0, "fp32")
    assert vl.last_precision() == "fp32"
    for j in (0, 2):
        ref, _ = restatement.fisher(d[0][off[j]:off[j + 1]], *d[1:], 0)
        assert rel_err(enc[j].cpu().numpy(), ref) < 5e-5
    q = torch.zeros((len(x), K), device="cuda")
    ll = vl.gmm_posteriors_device(q, p[2], p[0], p[1], t, "fp32")
    assert vl.last_precision() == "fp32"
    rq, rll = restatement.posteriors(d[0], d[3], d[1], d[2])
    assert np.max(np.abs(q.cpu().numpy() - rq)) < 4e-5
    assert abs(ll - rll) < 4e-6 * abs(rll) + 1e-4 * len(x)
