"""The ordered filter's sparse quads at the edges of their ranges: label counts
around the mask words (6.4 labels each), the 8-label bin rows, the 32-label
blocks and the compile-time 21; iterates that reach no bin, one bin, every bin
and exact tenths; lattices of short, long and huge lists; bit for bit against
the oracle."""
import ctypes as C

import numpy as np
import pytest

from densecrf_ho_b200 import Permutohedral, lib, synth
from densecrf_ho_b200._lib import check

pytestmark = pytest.mark.gpu


def _features(W, H, spread):
    if spread == 0:
        return synth.gaussian_features(W, H, 3, 3)
    rgb = synth.make_image(W, H, 21, 6)["rgb"]
    return synth.bilateral_features(W, H, 50 * spread, 50 * spread, *[15 * spread] * 3, rgb)


def _iterate(kind, N, L, rng):
    if kind == "zero":
        return np.zeros((N, L), np.float32)
    if kind == "one":
        return np.ones((N, L), np.float32)
    if kind == "onehot":
        q = np.zeros((N, L), np.float32)
        q[np.arange(N), rng.integers(0, L, N)] = 1.0
        return q
    if kind == "solve":  # most values near 0, one larger one per pixel
        q = rng.random((N, L)).astype(np.float32) * np.float32(0.08)
        q[np.arange(N), rng.integers(0, L, N)] = rng.random(N).astype(np.float32)
        return q
    if kind == "tenths":
        return (rng.integers(0, 11, (N, L)) / 10).astype(np.float32)
    return rng.random((N, L)).astype(np.float32)


@pytest.mark.parametrize("kind", ["zero", "one", "onehot", "solve", "tenths", "uniform"])
@pytest.mark.parametrize("L", [1, 2, 6, 7, 8, 20, 21, 25, 26, 32, 33, 65])
def test_iterates_and_label_counts(L, kind, oracle_mod):
    rng = np.random.default_rng(L)
    for (W, H), spread in (((1, 1), 0), ((31, 3), 0), ((47, 31), 1), ((61, 47), 8)):
        f = _features(W, H, spread)
        lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
        q = _iterate(kind, W * H, L, rng)
        assert np.array_equal(lat.compute_upper_minus_lower_ord(q), orc.compute_ord(q))


@pytest.mark.parametrize("L", [21, 40])
def test_one_lattice_for_several_iterates(L, oracle_mod):
    """A dense call between two sparse ones on one handle: no quad or mask of
    an earlier call is taken for this one's, and the plain filter, which shares
    the value buffers, neither."""
    W, H = 97, 61
    f = _features(W, H, 1)
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    rng = np.random.default_rng(3)
    for kind in ("solve", "uniform", "zero", "solve", "onehot"):
        q = _iterate(kind, W * H, L, rng)
        assert np.array_equal(lat.compute_upper_minus_lower_ord(q), orc.compute_ord(q))
        assert np.array_equal(lat.compute(q), orc.compute(q))
    f2 = _features(W, H, 8)  # the handle rebuilt on other features
    lat.init(f2)
    q = _iterate("solve", W * H, L, rng)
    assert np.array_equal(lat.compute_upper_minus_lower_ord(q), oracle_mod.OracleLattice(f2).compute_ord(q))


def test_unaligned_pointers(oracle_mod):
    import torch
    W, H, L = 61, 47, 21
    f = _features(W, H, 1)
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    q = _iterate("solve", W * H, L, np.random.default_rng(4))
    n = q.size
    src, dst = torch.zeros(n + 1, device="cuda"), torch.zeros(n + 1, device="cuda")
    src[1:] = torch.from_numpy(q.ravel()).cuda()
    torch.cuda.synchronize()
    check(lib().dcrf_lattice_compute_ord_dev(lat._h, C.c_void_p(dst[1:].data_ptr()), C.c_void_p(src[1:].data_ptr()), L))
    torch.cuda.synchronize()
    assert np.array_equal(dst[1:].cpu().numpy().reshape(W * H, L), orc.compute_ord(q))
