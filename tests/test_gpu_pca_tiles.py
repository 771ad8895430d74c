"""The tensor-core projection's output tiles (32 or 16 rows staged per warp, or
stored in place) and its search for the frames' images (one row or none per
image, many images per tile, few), against the float64 restatement: 1e-5
relative per descriptor, the projection's own bound; positions to 1e-6."""
import numpy as np
import pytest

from oracle.oracle import pca_project

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("din,m", [(128, 80), (128, 96), (128, 128), (64, 31), (128, 32)])
@pytest.mark.parametrize("counts", ["one", "tiny", "empty", "few", "none"])
@pytest.mark.parametrize("shift", [0, 1])
def test_tiles(vl, din, m, counts, shift):
    import torch
    r = np.random.Generator(np.random.PCG64(din + m))
    N = {"one": 131, "tiny": 40003, "empty": 5000, "few": 40003, "none": 1}[counts]
    c = {"one": [131], "tiny": None, "empty": [0, 0, 700, 0, 0, 4300, 0], "few": [20000, 3, 20000], "none": None}[counts]
    if counts == "tiny":
        cut = np.sort(r.integers(0, N + 1, 20000))
        c = np.diff(np.concatenate([[0], cut, [N]]))
    off = np.concatenate([[0], np.cumsum(c)]).astype(np.int64) if c is not None else None
    x = r.standard_normal((N, din)).astype(np.float32)
    P = r.standard_normal((m, din)).astype(np.float32)
    cen = r.standard_normal(din).astype(np.float32)
    frames = sizes = None
    ldo = m
    if off is not None:
        frames = (r.uniform(0, 500, (N, 2))).astype(np.float32)
        sizes = r.uniform(100, 600, (len(off) - 1, 2)).astype(np.float32)
        ldo += 2
    buf = torch.zeros(N * ldo + 1, device="cuda")
    out = buf[shift:shift + N * ldo].view(N, ldo)
    t = lambda a: None if a is None else torch.from_numpy(a).cuda()
    vl.pca_project_device(out, t(x), t(P), t(cen), True, t(frames), off, t(sizes))
    ref = pca_project(x, P, cen, True, frames, off, sizes)
    got = out.cpu().numpy().astype(np.float64)
    d = np.linalg.norm(got[:, :m] - ref[:, :m], axis=1) / np.linalg.norm(ref[:, :m], axis=1)
    assert d.max() < 1e-5
    if off is not None:
        assert np.abs(got[:, m:] - ref[:, m:]).max() < 1e-6
    assert float(buf[0]) == 0.0 or shift == 0
