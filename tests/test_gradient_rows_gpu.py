"""The lattice's feature gradient at label counts around the groups of four
that its slice takes, in every compile-time bound of the dimension, against
the oracle, bit for bit."""
import numpy as np
import pytest

from densecrf_ho_b200 import Permutohedral

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [1, 2, 5, 6, 9])
@pytest.mark.parametrize("L", [1, 2, 3, 4, 5, 8, 21])
def test_gradient_vs_oracle(L, d, oracle_mod):
    rng = np.random.default_rng(10 * d + L)
    N = 131  # one whole block of pixels and a short one
    f = (rng.standard_normal((N, d)) * 1.5).astype(np.float32)
    a, b = (rng.standard_normal((N, L)).astype(np.float32) for _ in range(2))
    got = Permutohedral().init(f).gradient(a, b)
    assert np.array_equal(got, oracle_mod.OracleLattice(f).gradient(a, b))
