"""The image norm of VLAD, a sequential sum formed in parallel, byte for byte
against the restatement at its tiles' edges (8192 float or 4096 double terms,
a short image, an image of zeros) and with values over a wide range."""
import numpy as np
import pytest

from oracle.oracle import vlad

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("K,D,scale", [(1, 4, 0), (2, 64, 0), (64, 64, 3), (64, 128, 0), (65, 128, 6), (129, 64, 12),
                                       (300, 32, 0)])
def test_norm_bytes(vl, K, D, scale, dtype):
    import torch
    r = np.random.Generator(np.random.PCG64(K + D))
    counts = [0, 40, 3, 500]
    off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    n = int(off[-1])
    x = (r.standard_normal((n, D)) * 10.0 ** r.uniform(-scale, scale, (n, 1))).astype(dtype)
    mu = r.standard_normal((K, D)).astype(dtype)
    a = np.zeros((n, K), dtype)
    a[np.arange(n), r.integers(0, K, n)] = 1
    enc = torch.zeros((len(counts), K * D), dtype=torch.from_numpy(x).dtype, device="cuda")
    vl.vlad_encode_batch_device(enc, *[torch.from_numpy(v).cuda() for v in (mu, x, a)], off, 0)
    for j in range(len(counts)):
        ref = vlad(x[off[j]:off[j + 1]], mu, a[off[j]:off[j + 1]], 0)
        assert np.array_equal(enc[j].cpu().numpy(), np.asarray(ref, dtype).ravel())
