"""The batched QP's elementwise kernels where their loops divide: images whose
rows start off a 16-byte boundary, tiles cut short, images of fewer elements
than one stride of the reductions and of more than the four that go together
-- against the single-image solver, bit for bit."""
import numpy as np
import pytest

from densecrf_ho_b200 import DenseCRF2D, DenseCRF2DBatch, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    [(1, 1), (127, 113), (3, 1), (128, 116)],  # below and above 296 * 256 * 4 elements of 21 labels
    [(160, 181), (31, 1), (65, 2)],
])
def test_ragged_batch_equals_single_solves(sizes):
    imgs = [synth.make_image(w, h, 21, 5 + i) for i, (w, h) in enumerate(sizes)]

    def terms(m, rgb):
        m.addPairwiseGaussian(3.0, 3.0, 3.0)
        m.addPairwiseBilateral(50.0, 50.0, 15.0, 15.0, 15.0, rgb, 5.0)

    b = DenseCRF2DBatch(sizes, 21)
    b.setUnaryEnergy(np.concatenate([im["unary"] for im in imgs]))
    terms(b, np.concatenate([im["rgb"] for im in imgs]))
    out, st = b.qp_inference_super_pixels_non_convex(b.unary_init(), max_iter=5, stats=True)
    for i, ((w, h), im) in enumerate(zip(sizes, imgs)):
        m = DenseCRF2D(w, h, 21)
        m.setUnaryEnergy(im["unary"])
        terms(m, im["rgb"])
        o, s = m.qp_inference_super_pixels_non_convex(m.unary_init(), max_iter=5, stats=True)
        assert np.array_equal(b.split(out)[i], o), i
        assert st[i].iterations == s.iterations and st[i].energy == s.energy
