"""GPU test of the k-means assignment of near ties (rows whose least two
distances agree to rounding): integer rows of small range, where many distances
are equal and the order in which the kd-tree search visits the centres decides,
and rows half way between two centres.  The expected digests (SHA-1 of every
row's centre, and the generator's next draw) are those of the search run for
each listed row from the root, with no shortcut; the distances follow the SIMD
width that the reference would pick, AVX here."""
import ctypes as C
import hashlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# name: rows, dimension, centres, range of the integers, type
CASES = {
    "line": (3001, 1, 7, 40, np.float32),
    "plane": (20011, 2, 130, 64, np.float32),
    "plane_d": (20011, 2, 130, 64, np.float64),
    "cube": (9001, 9, 256, 4, np.float32),
    "wide": (12007, 80, 256, 3, np.float32),
    "wide_d": (5003, 33, 100, 3, np.float64),
    "many": (24001, 12, 2100, 5, np.float32),  # tree and heap too large for shared memory
}
EXPECT = {
    "line": ("c7cd90cb980460d6", 2261367146),
    "plane": ("ece3f501a64f4059", 238034767),
    "plane_d": ("ece3f501a64f4059", 238034767),
    "cube": ("042ae37eef8620b8", 623455558),
    "wide": ("d612840129941a22", 1575415970),
    "wide_d": ("e6ead00163719909", 290547667),
    "many": ("47f5af42441a650c", 195366796),
}


def digest(vl, name):
    n, d, k, r, dt = CASES[name]
    rng = np.random.default_rng(11)
    x = rng.integers(0, r, size=(n, d)).astype(dt)
    x[n // 2:] = (x[n // 2:] + np.roll(x[n // 2:], 1, axis=0)) / 2
    m = vl.GMM(d, k, dt)
    m.set_covariance_lower_bound(1e-4)
    vl.rand_seed(5)
    vl._clear()
    vl.lib().vl_gmm_init_with_kmeans(m._h, np.ascontiguousarray(x).ctypes.data_as(C.c_void_p), n, None)
    assert vl.lib().vl_get_last_error() == 0, vl.lib().vl_get_last_error_message()
    nxt = vl.rand_uint32()
    a = np.argmax(m.posteriors, axis=1).astype(np.uint32)
    return hashlib.sha1(a.tobytes()).hexdigest()[:16], int(nxt)


@pytest.mark.parametrize("name", list(CASES))
def test_near_ties(vl, name):
    if not vl.lib().vl_cpu_has_avx():
        pytest.skip("the digests hold for the AVX distance order")
    vl.set_precision("exact")
    assert digest(vl, name) == EXPECT[name]
