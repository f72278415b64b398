"""meanfield_backward with grad_U over grad_Q, wholly or shifted by some rows or
values: the same bits as with buffers of their own."""
import ctypes as C

import numpy as np
import pytest

from densecrf_ho_b200 import DenseCRF2DBatch, lib, synth
from densecrf_ho_b200._lib import check

pytestmark = pytest.mark.gpu


def _ptr(t):
    return C.c_void_p(t.data_ptr())


# steps 0: the softmax's adjoint alone
@pytest.mark.parametrize("steps", [0, 3])
@pytest.mark.parametrize("L", [2, 5, 21])
def test_overlapping_gradients(L, steps):
    import torch
    sizes = [(61, 47), (97, 61)]
    N = sum(w * h for w, h in sizes)
    gen = torch.Generator(device="cuda").manual_seed(L)
    unary, grad = (torch.randn(N, L, generator=gen, device="cuda") for _ in range(2))
    rgb = np.concatenate([synth.make_image(w, h, 21, i)["rgb"].reshape(-1, 3) for i, (w, h) in enumerate(sizes)])
    b = DenseCRF2DBatch(sizes, L)
    check(lib().dcrf_batch_set_unary_dev(b._h, _ptr(unary)))
    b.addPairwiseGaussian(3.0, 3.0, 3.0)
    b.addPairwiseBilateral(50.0, 50.0, 15.0, 15.0, 15.0, rgb, 5.0)
    out = torch.empty_like(unary)
    check(lib().dcrf_batch_meanfield_dev(b._h, steps, _ptr(out)))

    def backward(gq, gu):
        w = np.zeros(2)
        torch.cuda.synchronize()
        check(lib().dcrf_batch_meanfield_backward_dev(b._h, _ptr(gq), _ptr(gu), w.ctypes.data_as(C.c_void_p)))
        torch.cuda.synchronize()
        return gu.cpu().numpy().copy(), w

    want_u, want_w = backward(grad.clone(), torch.empty_like(grad))
    for shift in (0, 1, L, 40 * L, 33 * L + 1):  # of grad_U from grad_Q, in values, either way
        for back in (False, True):
            room = torch.empty(N * L + shift, device="cuda")
            q, u = (shift, 0) if back else (0, shift)
            gq, gu = room[q:q + N * L], room[u:u + N * L]
            gq.copy_(grad.view(-1))
            got_u, got_w = backward(gq, gu)
            assert np.array_equal(got_u.reshape(N, L), want_u) and np.array_equal(got_w, want_w)
