"""Lattice construction around the tile and class limits of its sort: pixel
counts on both sides of the sort's tiles (2048 entries) and of multiples of 4 (padding
pixels), every compile-time and run-time dimension, vertices only padding
touches; every table equal to the oracle's, and the splat lists through the
filter."""
import numpy as np
import pytest

from densecrf_ho_b200 import Permutohedral

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 3, 5, 6, 8, 9, 16])
@pytest.mark.parametrize("N", [1, 3, 4, 5, 682, 683, 1365, 4099])
def test_tables(N, d, oracle_mod):
    rng = np.random.default_rng(100 * d + N)
    f = (rng.standard_normal((N, d)) * 2 + 20).astype(np.float32)  # away from 0: padding has vertices of its own
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    a, b = lat.export(), orc.export()
    assert a["M"] == b["M"]
    for k in ("offset", "rank", "bary", "keys", "nbr"):
        assert np.array_equal(a[k], np.asarray(b[k]).reshape(a[k].shape)), k
    x = rng.standard_normal((N, 3)).astype(np.float32)
    assert np.array_equal(lat.compute(x), orc.compute(x))


def test_handle_rebuilt_smaller_and_larger(oracle_mod):
    lat = Permutohedral()
    for N, spread in ((3000, 1.0), (40, 5.0), (9000, 0.1), (1, 1.0)):
        rng = np.random.default_rng(N)
        f = (rng.standard_normal((N, 5)) * spread).astype(np.float32)
        orc = oracle_mod.OracleLattice(f)
        lat.init(f)
        x = rng.standard_normal((N, 21)).astype(np.float32)
        assert lat.M == orc.M and np.array_equal(lat.compute(x), orc.compute(x))
