"""Threads that filter with different label counts at the same time: the shared
memory a kernel may use is an attribute of the kernel, not of the call, and one
thread's call must not lower it under another's.  Every call succeeds with the
bits that the same call gives alone."""
import ctypes as C
import threading

import numpy as np
import pytest

from densecrf_ho_b200 import DenseCRF2D, Permutohedral, lib, synth
from densecrf_ho_b200._lib import check

pytestmark = pytest.mark.gpu


def _together(calls, wants, times):
    failed, start = [], threading.Barrier(len(calls))

    def work(call, want):
        start.wait()
        for _ in range(times):
            try:
                if not np.array_equal(call(), want):
                    raise AssertionError("other bits")
            except Exception as e:  # noqa: BLE001 - handed to the test's thread
                failed.append(e)
                return

    threads = [threading.Thread(target=work, args=a) for a in zip(calls, wants)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[0]


@pytest.mark.parametrize("counts", [(100, 200, 300, 400), (5, 21, 40, 97)])
def test_filters(counts):
    """Some thousand ordered filters a thread, queued back to back: a call's
    window is a microsecond or so."""
    import torch
    W, H = 5, 3
    f = synth.bilateral_features(W, H, 50, 50, 15, 15, 15, synth.make_image(W, H, 21, 6)["rgb"])
    calls = []
    for L in counts:
        q = torch.from_numpy(np.random.default_rng(L).random((W * H, L)).astype(np.float32)).cuda()
        lat, out = Permutohedral().init(f), torch.empty_like(q)
        args = (lat._h, C.c_void_p(out.data_ptr()), C.c_void_p(q.data_ptr()), L)

        def call(lat=lat, q=q, out=out, args=args, entry=lib().dcrf_lattice_compute_ord_dev):
            for _ in range(200):
                check(entry(*args))
            return lat.compute_upper_minus_lower_ord(q.cpu().numpy())  # waits for the calls before it

        calls.append(call)
    torch.cuda.synchronize()
    _together(calls, [c() for c in calls], 25)


def test_lp_slices_of_different_sizes():
    """One and two labels with two terms of 13 to 16 features each: the ordered
    slice's largest blocks, on both sides of the opt-in."""
    W, H = 23, 17
    rng = np.random.default_rng(1)
    calls = []
    for L, d in ((1, 13), (1, 16), (1, 14), (2, 16)):
        m = DenseCRF2D(W, H, L)
        m.setUnaryEnergy(rng.random((W * H, L)).astype(np.float32))
        for _ in range(2):
            m.addPairwiseEnergy(rng.standard_normal((W * H, d)).astype(np.float32), 1.0)
        q = m.unary_init()
        calls.append(lambda m=m, q=q: m.lp_inference_prox_super_pixels(q, prox_max_iter=1, fw_max_iter=2))
    _together(calls, [c() for c in calls], 40)
