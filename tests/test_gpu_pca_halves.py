"""The tensor-core projection where only some of a warp's rows store: output tiles
staged in halves of 16 rows (128 to 96 dimensions with positions), whole (80), or
stored in place (an output that is not 16-byte aligned), with the last tile ending
at each side of a half.  Against the float64 restatement (1e-5 relative per
descriptor, positions 1e-6, the projection's own bounds); memory behind the output
stays as it was."""
import numpy as np
import pytest

from oracle.oracle import pca_project

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,shift", [(96, 0), (80, 0), (96, 1), (33, 0)])
@pytest.mark.parametrize("N", [1, 15, 16, 17, 31, 33, 112, 127, 129, 149 * 128 + 17])
def test_last_tile(vl, m, shift, N):
    import torch
    r = np.random.Generator(np.random.PCG64(m + N))
    x = r.standard_normal((N, 128)).astype(np.float32)
    P = r.standard_normal((m, 128)).astype(np.float32)
    cen = r.standard_normal(128).astype(np.float32)
    off = np.array([0, N // 2, N], np.int64)
    frames = r.uniform(0, 500, (N, 2)).astype(np.float32)
    sizes = r.uniform(100, 600, (2, 2)).astype(np.float32)
    ldo = m + 2
    buf = torch.full((N * ldo + 64,), -7.0, device="cuda")
    out = buf[shift:shift + N * ldo].view(N, ldo)
    t = lambda a: torch.from_numpy(a).cuda()
    vl.pca_project_device(out, t(x), t(P), t(cen), True, t(frames), off, t(sizes))
    ref = pca_project(x, P, cen, True, frames, off, sizes)
    got = out.cpu().numpy().astype(np.float64)
    d = np.linalg.norm(got[:, :m] - ref[:, :m], axis=1) / np.linalg.norm(ref[:, :m], axis=1)
    assert d.max() < 1e-5 and np.abs(got[:, m:] - ref[:, m:]).max() < 1e-6
    assert bool((buf[:shift] == -7.0).all()) and bool((buf[shift + N * ldo:] == -7.0).all())
