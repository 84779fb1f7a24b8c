"""Statistics of dense networks in batches: every effect type, at word edges, empty
and full networks, and sizes whose scratch holds fewer statistics at a time than
the model has. Order-dependent float64 statistics are added in the reference's
order, so all values equal the CPU engine's but for pow (type 7, 17: both sides'
libraries are within a few units in the last place per term, n terms)."""
import numpy as np
import pytest

from cusna_gb300 import sim as G

pytestmark = pytest.mark.gpu

TYPES = [0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 19, 20, 21, 23, 24]
TYPES2 = [25, 26, 27, 28, 29, 30, 31, 22, 10, 12, 29]


@pytest.mark.parametrize("types", [TYPES, TYPES2], ids=["first", "second"])
@pytest.mark.parametrize("n", [3, 32, 33, 100, 880])
def test_every_statistic_matches_the_oracle(gpu_lib, port, types, n):
    r = np.random.default_rng(n)
    k = len(types)
    A = np.zeros((3 if n <= 100 else 1, n, n), np.uint8)
    A[0] = r.random((n, n)) < min(0.5, 5.0 / n)
    if n <= 100:
        A[1] = 1
    for a in A:
        np.fill_diagonal(a, 0)
    p1 = r.choice([0.0, 0.5, 1.0, 2.0], k)
    p2 = r.random(k)
    vmat = r.standard_normal((k, n))
    vmiss = (r.random((k, n)) < 0.1).astype(np.uint8)
    wtab = np.cumsum(r.random((k, n + 1)), axis=1)
    wtab[:, 0] = 0.0
    dyn = (r.random(k) < 0.3).astype(np.int32)
    vb = r.standard_normal(n)
    od0, id0 = r.integers(0, 9, n).astype(np.int32), r.integers(0, 9, n).astype(np.int32)
    args = (n, k, np.asarray(types, np.int32), p1, p2, vmat, vmiss, dyn, vb, od0, id0, wtab, 0)
    out = np.atleast_2d(G.network_stats(A, *args))
    for a, got in zip(A, out):
        ref = np.asarray(port.network_stats(a, *args))
        power = np.isin(types, (7, 17))
        np.testing.assert_array_equal(got[~power], ref[~power])
        np.testing.assert_allclose(got[power], ref[power], rtol=(n + 8) * 2.0 ** -52, atol=0)
