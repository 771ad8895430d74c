"""VLAD's per-component chains of many images, several images a block: byte for byte
against the restatement where the last block has fewer images, soft images (left to
the streaming kernel) among hard ones; and what the kernel takes when every image is
soft and it has nothing to do."""
import numpy as np
import pytest

from oracle.oracle import vlad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("K,D,nimg,most", [(32, 33, 1190, 3), (64, 40, 2401, 2), (64, 9, 4001, 1), (16, 70, 6000, 0),
                                           (8, 34, 12001, 70)])
def test_images_per_block(vl, K, D, nimg, most, dtype):
    import torch
    r = np.random.Generator(np.random.PCG64(K * D + nimg))
    off = np.concatenate([[0], np.cumsum(r.integers(0, most + 1, nimg))]).astype(np.int64)
    n = int(off[-1])
    x, mu = r.standard_normal((n, D)).astype(dtype), r.standard_normal((K, D)).astype(dtype)
    a = np.zeros((n, K), dtype)
    a[np.arange(n), r.integers(0, K, n)] = 1
    soft = r.integers(0, max(n, 1), n // 5)
    a[soft, r.integers(0, K, len(soft))] = 0.5
    t = [torch.from_numpy(v).cuda() for v in (mu, x, a)]
    enc = torch.full((nimg, K * D), 7.0, dtype=t[0].dtype, device="cuda")
    vl.vlad_encode_batch_device(enc, *t, off, 1)
    enc = enc.cpu().numpy()
    for j in list(range(0, nimg, 61)) + list(range(nimg - 9, nimg)):
        ref = vlad(x[off[j]:off[j + 1]], mu, a[off[j]:off[j + 1]], 1)
        assert np.array_equal(enc[j], np.asarray(ref, dtype).ravel()), j


def test_time_of_soft_images(vl):
    """3,000 soft images, K=64: 21 us by blocks of eight warps, 105 by blocks of one
    with an image each.  At most 50."""
    import torch
    nimg, K, D = 3000, 64, 64
    off = np.arange(nimg + 1, dtype=np.int64) * 10
    x, mu = torch.randn((10 * nimg, D), device="cuda"), torch.randn((K, D), device="cuda")
    a = torch.zeros((10 * nimg, K), device="cuda")
    a[:, 3:5] = 0.5
    enc = torch.zeros((nimg, K * D), device="cuda")
    vl.vlad_encode_batch_device(enc, mu, x, a, off, 0)
    best = np.inf
    for _ in range(5):
        vl.profile_reset()
        vl.profile_enable(True)
        vl.vlad_encode_batch_device(enc, mu, x, a, off, 0)
        torch.cuda.synchronize()
        best = min(best, vl.profile_read()["vlad_group"][1])
        vl.profile_enable(False)
    vl.profile_reset()
    assert best < 0.05
