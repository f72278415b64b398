"""The plain filter's row splat, padding pass and warp-tiled slice at the edges
of their tiles: pixel counts around the slice's 20-pixel tile, label counts
around the 4-label group and the 32-label ring, list lengths on both sides of
the short / long / huge limits, pointers that are not 16-byte aligned."""
import ctypes as C

import numpy as np
import pytest

from densecrf_ho_b200 import Permutohedral, lib, synth
from densecrf_ho_b200._lib import check

pytestmark = pytest.mark.gpu


def _features(W, H, spread, seed=5):
    rgb = synth.make_image(W, H, 21, seed)["rgb"]
    if spread == 0:
        return synth.gaussian_features(W, H, 3, 3)
    return synth.bilateral_features(W, H, 50 * spread, 50 * spread, *[15 * spread] * 3, rgb)


# (W, H), spread: 0 Gaussian (short lists), 1 bilateral (short and long), 8 and 40 nearly flat (huge lists)
@pytest.mark.parametrize("size,spread", [((1, 1), 0), ((19, 1), 1), ((20, 1), 0), ((21, 3), 1), ((61, 47), 8),
                                         ((97, 61), 40)])
@pytest.mark.parametrize("L", [1, 2, 3, 4, 20, 21, 31, 33, 64, 130])
def test_edges_bit_exact(size, spread, L, oracle_mod):
    W, H = size
    f = _features(W, H, spread)
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    x = np.random.default_rng(L).standard_normal((W * H, L)).astype(np.float32)
    for rev in (False, True):
        assert np.array_equal(lat.compute(x, rev), orc.compute(x, rev))


@pytest.mark.parametrize("L", [5, 21])
def test_unaligned_pointers_bit_exact(L, oracle_mod):
    import torch
    W, H = 61, 47
    f = _features(W, H, 8)
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    x = np.random.default_rng(L).standard_normal((W * H, L)).astype(np.float32)
    ref = orc.compute(x)
    n = W * H * L
    for a in (0, 1):
        for b in (0, 1):  # input / output 0 or 4 bytes past a 16-byte boundary
            src, dst = torch.zeros(n + 1, device="cuda"), torch.zeros(n + 1, device="cuda")
            src[a:a + n] = torch.from_numpy(x.ravel()).cuda()
            torch.cuda.synchronize()
            check(lib().dcrf_lattice_compute_dev(lat._h, C.c_void_p(dst[b:].data_ptr()),
                                                 C.c_void_p(src[a:].data_ptr()), L, 0))
            torch.cuda.synchronize()
            assert np.array_equal(dst[b:b + n].cpu().numpy().reshape(W * H, L), ref)
