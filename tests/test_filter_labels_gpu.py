"""The plain filter and the feature gradient on both sides of the label count
where one pixel's row no longer fits a warp's tile (some 3050), bit for bit:
the filter against the oracle, the gradient of a single label among many zero
ones against the one of four labels."""
import numpy as np
import pytest

from densecrf_ho_b200 import Permutohedral, synth

pytestmark = pytest.mark.gpu


def _features(W, H, d, spread):
    rgb = synth.make_image(W, H, 21, 6)["rgb"]
    f = synth.bilateral_features(W, H, 50 * spread, 50 * spread, *[15 * spread] * 3, rgb)
    return np.ascontiguousarray(f[:, :d])


# one pixel; short lists; short, long and huge lists
@pytest.mark.parametrize("W,H,d,spread", [(1, 1, 5, 1), (13, 7, 5, 1), (11, 9, 2, 1), (61, 23, 5, 40)])
@pytest.mark.parametrize("L", [3050, 3056, 3057, 3073, 5000, 12001])
def test_filter_vs_oracle(W, H, d, spread, L, oracle_mod):
    f = _features(W, H, d, spread)
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    x = np.random.default_rng(L).standard_normal((W * H, L)).astype(np.float32)
    for rev in (False, True):
        assert np.array_equal(lat.compute(x, rev), orc.compute(x, rev))


@pytest.mark.parametrize("L", [3056, 3057, 13001])
def test_gradient_of_one_label_among_many(L):
    """All labels but one are zero in a and b: they add zeros, and the gradient
    is the one label's, which the call with four labels (three zero) gives."""
    f = _features(13, 7, 5, 1)
    lat = Permutohedral().init(f)
    rng = np.random.default_rng(L)
    v = rng.standard_normal((2, 13 * 7)).astype(np.float32)
    small, large = (np.zeros((2, 13 * 7, n), np.float32) for n in (4, L))
    small[:, :, 1] = v
    for k in (0, L // 2, L - 1):
        large[:] = 0
        large[:, :, k] = v
        assert np.array_equal(lat.gradient(large[0], large[1]), lat.gradient(small[0], small[1]))
