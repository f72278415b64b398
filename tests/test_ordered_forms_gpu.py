"""The single ordered filter on both sides of each line between its quad and its
dense form: few labels over long and huge lists, many vertices, many pixels; bit
for bit against the oracle."""
import numpy as np
import pytest

from densecrf_ho_b200 import Permutohedral, synth

pytestmark = pytest.mark.gpu


def _features(W, H, d, kind):
    if kind == "line":
        return (np.arange(W * H, dtype=np.float32) / 7)[:, None]
    if kind == "grid":
        return synth.gaussian_features(W, H, 3, 3)
    rgb = synth.make_image(W, H, 21, 5)["rgb"]
    if kind == "noisy":
        rgb = np.random.default_rng(0).integers(0, 256, size=rgb.shape).astype(np.uint8)
    s = 8 if kind == "wide" else 1  # wide: huge lists
    return np.ascontiguousarray(synth.bilateral_features(W, H, 50 * s, 50 * s, *[15 * s] * 3, rgb)[:, :d])


def _iterate(N, L, rng, spread):
    if spread:
        return rng.random((N, L)).astype(np.float32)
    q = rng.random((N, L)).astype(np.float32) * np.float32(0.08)
    q[np.arange(N), rng.integers(0, L, N)] = rng.random(N).astype(np.float32)
    return q


@pytest.mark.parametrize("W,H,d,kind,labels", [
    (257, 256, 5, "wide", (1, 2, 3, 4, 5, 8, 12, 13, 20, 21)),  # more than 2^16 pixels: every split of the long lists
    (256, 256, 5, "wide", (20, 21)),
    (513, 512, 5, "photo", (12, 13)),   # more than 2^18
    (257, 256, 3, "photo", (6, 20)),
    (97, 83, 5, "noisy", (1, 8, 9)),    # some 25 thousand vertices
    (61, 47, 5, "noisy", (1, 2, 3, 4)),
    (512, 513, 2, "grid", (1,)), (512, 512, 2, "grid", (1, 2)),
    (128, 128, 2, "grid", (19, 20)), (127, 129, 2, "grid", (19, 20, 28, 29)),
    (31, 7, 2, "grid", (28, 29, 161)), (61, 47, 1, "line", (29,)),
])
def test_both_sides_of_each_line(W, H, d, kind, labels, oracle_mod):
    f = _features(W, H, d, kind)
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    rng = np.random.default_rng(W + d)
    for L in labels:
        for spread in (False, True):
            q = _iterate(W * H, L, rng, spread)
            assert np.array_equal(lat.compute_upper_minus_lower_ord(q), orc.compute_ord(q))


def test_restricted_and_plain_between_the_forms(oracle_mod):
    """One handle: the restricted filter shares the dense form's bins, the plain
    filter the value buffers of both."""
    W, H = 257, 256
    f = _features(W, H, 5, "wide")
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    rng = np.random.default_rng(3)
    pI = np.sort(rng.choice(W * H, 500, replace=False)).astype(np.int32)
    for L in (4, 21, 4):
        q, rq, rq2 = _iterate(W * H, L, rng, False), _iterate(500, L, rng, True), _iterate(500, L, rng, True)
        alone = Permutohedral().init(f)
        want = alone.compute_upper_minus_lower_ord_restricted(rq, pI, q, True)
        want2 = alone.compute_upper_minus_lower_ord_restricted(rq2, pI, None, False)
        full, plain = orc.compute_ord(q), orc.compute(q)
        assert np.array_equal(lat.compute_upper_minus_lower_ord(q), full)
        assert np.array_equal(lat.compute_upper_minus_lower_ord_restricted(rq, pI, q, True), want)
        assert np.array_equal(lat.compute(q), plain)
        assert np.array_equal(lat.compute_upper_minus_lower_ord(q), full)
        assert np.array_equal(lat.compute_upper_minus_lower_ord_restricted(rq2, pI, None, False), want2)
