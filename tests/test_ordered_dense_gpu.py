"""The ordered filter on both sides of the line between its quad and its dense
form (2^19 pixel-label values, at most two features, no long list), calls of
either form and plain and restricted filters on one handle, bit for bit against
the oracle."""
import numpy as np
import pytest

from densecrf_ho_b200 import Permutohedral, synth

pytestmark = pytest.mark.gpu


def _iterate(N, L, rng, spread):
    if spread:
        return rng.random((N, L)).astype(np.float32)
    q = rng.random((N, L)).astype(np.float32) * np.float32(0.08)
    q[np.arange(N), rng.integers(0, L, N)] = rng.random(N).astype(np.float32)
    return q


@pytest.mark.parametrize("W,H,L,d", [
    (64, 64, 128, 2), (64, 64, 129, 2), (158, 158, 21, 2), (160, 157, 21, 2), (420, 417, 3, 2), (512, 513, 2, 1),
])
def test_both_sides_of_the_line(W, H, L, d, oracle_mod):
    rng = np.random.default_rng(W + L)
    f = synth.gaussian_features(W, H, 3, 3) if d == 2 else (np.arange(W * H, dtype=np.float32) / 7)[:, None]
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    for spread in (False, True):
        q = _iterate(W * H, L, rng, spread)
        assert np.array_equal(lat.compute_upper_minus_lower_ord(q), orc.compute_ord(q))


def test_forms_and_filters_on_one_handle(oracle_mod):
    """Label counts that take the dense, the quad and the dense form in turn,
    with the plain filter, which shares the value buffers, between them."""
    W, H = 161, 160
    rng = np.random.default_rng(1)
    f = synth.gaussian_features(W, H, 3, 3)
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    for L in (21, 5, 33, 21):
        q = _iterate(W * H, L, rng, L == 33)
        assert np.array_equal(lat.compute(q), orc.compute(q))
        assert np.array_equal(lat.compute_upper_minus_lower_ord(q), orc.compute_ord(q))
