"""The ordered filter over wide label ranges: both sides of the line between the
staged and the warp-per-32-labels bins (96 labels), counts that no shared-memory
tile holds, and counts past 2^20; bit for bit against the oracle, or against
the same lattice's filter of 21 of the labels, which do not mix."""
import ctypes as C

import numpy as np
import pytest

from densecrf_ho_b200 import Permutohedral, lib, synth
from densecrf_ho_b200._lib import check

pytestmark = pytest.mark.gpu


def _features(W, H, d, spread):
    rgb = synth.make_image(W, H, 21, 6)["rgb"]
    f = synth.bilateral_features(W, H, 50 * spread, 50 * spread, *[15 * spread] * 3, rgb)
    return np.ascontiguousarray(f[:, :d])


def _iterate(N, L, rng, spread):
    q = rng.random((N, L)).astype(np.float32)
    if not spread:
        q *= np.float32(0.08)
        q[np.arange(N), rng.integers(0, L, N)] = rng.random(N).astype(np.float32)
    return q


# 1x1; short lists; short, long and huge lists
@pytest.mark.parametrize("W,H,d,spread", [(1, 1, 5, 1), (31, 7, 5, 1), (29, 11, 3, 1), (61, 47, 5, 8)])
@pytest.mark.parametrize("L", [95, 96, 97, 128, 129, 454, 455, 1000])
def test_label_counts_vs_oracle(W, H, d, spread, L, oracle_mod):
    rng = np.random.default_rng(L)
    f = _features(W, H, d, spread)
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    for wide in (False, True):
        q = _iterate(W * H, L, rng, wide)
        assert np.array_equal(lat.compute_upper_minus_lower_ord(q), orc.compute_ord(q))


@pytest.mark.parametrize("L", [(1 << 20) + 5])
def test_many_labels_vs_their_columns(L):
    import torch
    f = np.array([[0.1, 0.2, 0.3], [3.1, -2.0, 0.7]], np.float32)
    lat = Permutohedral().init(f)
    x = torch.rand(2, L, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    out = torch.empty_like(x)
    torch.cuda.synchronize()

    def call(dst, src, n):
        check(lib().dcrf_lattice_compute_ord_dev(lat._h, C.c_void_p(dst.data_ptr()), C.c_void_p(src.data_ptr()), n))
        torch.cuda.synchronize()

    call(out, x, L)
    for k in (0, L // 2, L - 21):
        xs = x[:, k:k + 21].contiguous()
        ref = torch.empty_like(xs)
        torch.cuda.synchronize()
        call(ref, xs, 21)
        assert torch.equal(out[:, k:k + 21], ref)


def test_unaligned_pointers():
    import torch
    W, H, L = 31, 7, 333
    f = _features(W, H, 5, 1)
    lat = Permutohedral().init(f)
    q = torch.from_numpy(_iterate(W * H, L, np.random.default_rng(2), True)).cuda()
    n = q.numel()
    src, dst, ref = torch.zeros(n + 1, device="cuda"), torch.zeros(n + 1, device="cuda"), torch.empty_like(q)
    src[1:] = q.reshape(-1)
    torch.cuda.synchronize()
    check(lib().dcrf_lattice_compute_ord_dev(lat._h, C.c_void_p(ref.data_ptr()), C.c_void_p(q.data_ptr()), L))
    check(lib().dcrf_lattice_compute_ord_dev(lat._h, C.c_void_p(dst[1:].data_ptr()), C.c_void_p(src[1:].data_ptr()), L))
    torch.cuda.synchronize()
    assert torch.equal(dst[1:].view_as(q), ref)
