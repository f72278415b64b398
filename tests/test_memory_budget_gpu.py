"""The padded rows of the plain filter are an aid, not a need: a call that has no
memory for them, or whose handle holds them when another buffer finds none,
gives the same bits without them.  The budgets are what the same call took
without one, less a byte (its last allocation is refused) and less all rows."""
import ctypes as C

import numpy as np
import pytest

from densecrf_ho_b200 import (DenseCRF2D, DenseCRF2DBatch, Permutohedral, device_memory_stats, lib,
                              set_device_memory_limit, synth)
from densecrf_ho_b200._lib import check

pytestmark = pytest.mark.gpu


def _held():
    return device_memory_stats()[0]


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _rows(N, L):
    return 16 * N * ((L + 3) // 4)


def _same_within(make, call, rows):
    """call(handle) without a budget, then on fresh handles within less."""
    h = make()
    before = _held()
    want = call(h)
    took = _held() - before
    del h
    for budget in (took - 1, took - rows):
        h = make()
        set_device_memory_limit(_held() + budget)
        try:
            got = call(h)
        finally:
            set_device_memory_limit(0)
        del h
        assert all(np.array_equal(a, b) for a, b in zip(got, want))


def _features(W, H, spread):
    if spread == 0:
        return synth.gaussian_features(W, H, 3, 3)
    rgb = synth.make_image(W, H, 21, 5)["rgb"]
    return synth.bilateral_features(W, H, 50 * spread, 50 * spread, *[15 * spread] * 3, rgb)


def _filter(lat, x, entry, *args):
    import torch
    out = torch.full_like(x, float("nan"))
    torch.cuda.synchronize()
    check(entry(lat._h, _ptr(out), _ptr(x), x.shape[1], *args))
    torch.cuda.synchronize()
    return out.cpu().numpy()


# short lists; short and long; short, long and huge
@pytest.mark.parametrize("W,H,spread", [(61, 47, 0), (61, 47, 1), (97, 61, 40)])
@pytest.mark.parametrize("L", [3, 5, 21, 32, 33, 70, 3100])
def test_filter(W, H, spread, L):
    import torch
    f = _features(W, H, spread)
    x = torch.randn(W * H, L, generator=torch.Generator(device="cuda").manual_seed(L), device="cuda")
    for rev in (0, 1):
        _same_within(lambda: Permutohedral().init(f),
                     lambda lat: [_filter(lat, x, lib().dcrf_lattice_compute_dev, rev)], _rows(W * H, L))


@pytest.mark.parametrize("L", [5, 21])
def test_ordered_filter_on_a_handle_that_holds_rows(L):
    import torch
    W, H = 161, 120
    f = _features(W, H, 0)
    x = torch.rand(W * H, L, generator=torch.Generator(device="cuda").manual_seed(L), device="cuda")
    entry = lib().dcrf_lattice_compute_ord_dev
    lat = Permutohedral().init(f)
    before = _held()
    want = _filter(lat, x, entry)
    took = _held() - before
    lat = Permutohedral().init(f)
    before = _held()
    _filter(lat, x, lib().dcrf_lattice_compute_dev, 0)
    set_device_memory_limit(before + took)  # the ordered filter's own, none of the rows
    try:
        got = _filter(lat, x, entry)
    finally:
        set_device_memory_limit(0)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("W,H,L", [(61, 47, 21), (61, 47, 6), (120, 90, 21)])
def test_qp(W, H, L):
    img = synth.make_image(W, H, L, 3)

    def make():
        m = DenseCRF2D(W, H, L)
        m.setUnaryEnergy(img["unary"])
        m.addPairwiseGaussian(3.0, 3.0, 3.0)
        m.addPairwiseBilateral(50.0, 50.0, 15.0, 15.0, 15.0, img["rgb"], 5.0)
        m.unary_init()
        return m

    q = make().unary_init()
    _same_within(make, lambda m: [m.qp_inference_super_pixels_non_convex(q) for _ in range(2)], 2 * _rows(W * H, L))


def _batch(sizes, L, unary, rgb):
    b = DenseCRF2DBatch(sizes, L)
    check(lib().dcrf_batch_set_unary_dev(b._h, _ptr(unary)))
    b.addPairwiseGaussian(3.0, 3.0, 3.0)
    b.addPairwiseBilateral(50.0, 50.0, 15.0, 15.0, 15.0, rgb, 5.0)
    return b


@pytest.mark.parametrize("L", [4, 21])
@pytest.mark.parametrize("what", ["qp", "meanfield"])
def test_batch(what, L):
    import torch
    sizes = [(61, 47), (40, 30), (97, 61)]
    N = sum(w * h for w, h in sizes)
    gen = torch.Generator(device="cuda").manual_seed(L)
    unary, grad = (torch.randn(N, L, generator=gen, device="cuda") for _ in range(2))
    init = torch.softmax(-unary, 1).contiguous()
    rgb = np.concatenate([synth.make_image(w, h, 21, i)["rgb"].reshape(-1, 3) for i, (w, h) in enumerate(sizes)])
    out, grad_u, iters = torch.empty_like(unary), torch.empty_like(unary), C.c_int(30)
    torch.cuda.synchronize()

    def qp(b):
        check(lib().dcrf_batch_qp_dev(b._h, _ptr(init), _ptr(out), C.byref(iters), None))
        torch.cuda.synchronize()
        return [out.cpu().numpy()]

    def meanfield(b):
        gw = np.zeros(2)
        check(lib().dcrf_batch_meanfield_dev(b._h, 4, _ptr(out)))
        check(lib().dcrf_batch_meanfield_backward_dev(b._h, _ptr(grad), _ptr(grad_u), gw.ctypes.data_as(C.c_void_p)))
        torch.cuda.synchronize()
        return [out.cpu().numpy(), grad_u.cpu().numpy(), gw]

    _same_within(lambda: _batch(sizes, L, unary, rgb), {"qp": qp, "meanfield": meanfield}[what], 2 * _rows(N, L))
