"""A handle that holds what it can do without (padded rows, a build's scratch,
the ordered filter's buffers) takes every other call, host buffers and a new
lattice included, within what the call took on a fresh handle."""
import numpy as np
import pytest

from densecrf_ho_b200 import DenseCRF2D, Permutohedral, device_memory_stats, set_device_memory_limit, synth

pytestmark = pytest.mark.gpu


def _held():
    return device_memory_stats()[0]


def _features(W, H, d, seed=5):
    rgb = synth.make_image(W, H, 21, seed)["rgb"]
    return synth.bilateral_features(W, H, 50, 50, 15, 15, 15, rgb) if d == 5 else synth.gaussian_features(W, H, 3, 3)


def _rows(N, L):
    return 16 * N * ((L + 3) // 4)


@pytest.mark.parametrize("d", [2, 5])
@pytest.mark.parametrize("what", ["compute", "ordered"])
def test_host_calls_after_other_label_counts(d, what):
    W, H = 97, 83
    f = _features(W, H, d)
    rng = np.random.default_rng(d)
    small, large = rng.random((W * H, 4)).astype(np.float32), rng.random((W * H, 21)).astype(np.float32)

    def call(lat):
        return lat.compute(large) if what == "compute" else lat.compute_upper_minus_lower_ord(large)

    lat = Permutohedral().init(f)
    lat.compute(small)
    lat.compute_upper_minus_lower_ord(small)
    before = _held()
    want = call(lat)
    took = _held() - before
    lat = Permutohedral().init(f)
    lat.compute(small)
    lat.compute_upper_minus_lower_ord(small)
    rows = _rows(W * H, 21) - _rows(W * H, 4) if what == "compute" else 0
    set_device_memory_limit(_held() + took - rows - _rows(W * H, 4))
    try:
        got = call(lat)
    finally:
        set_device_memory_limit(0)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("d", [2, 5])
def test_a_larger_lattice_on_a_handle_that_filtered(d):
    f, g = _features(61, 47, d), _features(97, 83, d, 6)
    x, y = (np.random.default_rng(d).random((n, 21)).astype(np.float32) for n in (61 * 47, 97 * 83))
    lat = Permutohedral().init(f)
    before = _held()
    lat.init(g)
    took = _held() - before  # without filters in between
    want = lat.compute(y)
    lat = Permutohedral().init(f)
    lat.compute(x)
    lat.compute_upper_minus_lower_ord(x)
    set_device_memory_limit(_held() + took - _rows(61 * 47, 21))
    try:
        lat.init(g)
    finally:
        set_device_memory_limit(0)
    assert np.array_equal(lat.compute(y), want)


def test_terms_and_solvers_after_a_solve():
    W, H, L = 61, 47, 21
    img = synth.make_image(W, H, L, 3)

    def make(solve):
        m = DenseCRF2D(W, H, L)
        m.setUnaryEnergy(img["unary"])
        m.addPairwiseBilateral(50.0, 50.0, 15.0, 15.0, 15.0, img["rgb"], 5.0)
        q = m.unary_init()
        if solve:
            m.qp_inference_super_pixels_non_convex(q)
        return m, q

    def more(m, q):
        m.addPairwiseGaussian(3.0, 3.0, 3.0)
        return m.lp_inference_prox_super_pixels(q, prox_max_iter=2, fw_max_iter=3)

    m, q = make(True)
    before = _held()
    want = more(m, q)
    took = _held() - before
    del m
    m, q = make(True)
    set_device_memory_limit(_held() + took - 2 * _rows(W * H, L))  # the new term's rows and the old one's
    try:
        got = more(m, q)
    finally:
        set_device_memory_limit(0)
    assert np.array_equal(got, want)
