"""The LP on images of many vertices with few entries each: its ordered filters'
forms for few labels and very short lists, against the oracle."""
import numpy as np
import pytest

from densecrf_ho_b200 import DenseCRF2D, synth

pytestmark = pytest.mark.gpu


# the last: some 90 thousand vertices, where the terms filter one by one up to 4 labels
@pytest.mark.parametrize("W,H,L", [(w, h, n) for w, h in ((64, 48), (97, 61)) for n in (2, 3, 6, 7, 16, 21)] +
                         [(224, 160, n) for n in (2, 4, 5)])
def test_noisy_image_vs_oracle(W, H, L, oracle_mod):
    img = dict(synth.make_image(W, H, L, 4))
    img["rgb"] = np.random.default_rng(L).integers(0, 256, size=img["rgb"].shape).astype(np.uint8)
    m = DenseCRF2D(W, H, L)
    m.setUnaryEnergy(img["unary"])
    m.addPairwiseGaussian(3.0, 3.0, 3.0)
    m.addPairwiseBilateral(50.0, 50.0, 15.0, 15.0, 15.0, img["rgb"], 5.0)
    om = oracle_mod.build_model(oracle_mod.OracleModel, img)
    q = om.unary_init()
    got = m.lp_inference_prox_super_pixels(q, prox_max_iter=2, fw_max_iter=3)
    want, _ = om.lp(q, prox_max_iter=2, fw_max_iter=3)
    # the same arithmetic but for the dual gap's sums (FP64 here, the reference's float there)
    assert (got.argmax(1) == want.argmax(1)).mean() >= 0.999


def test_terms_one_by_one_with_cliques(oracle_mod):
    W, H, L = 224, 160, 3
    img = dict(synth.make_image(W, H, L, 4))
    img["rgb"] = np.random.default_rng(1).integers(0, 256, size=img["rgb"].shape).astype(np.uint8)
    off, idx = np.array([0, 400, 900], np.int32), np.arange(900, dtype=np.int32)
    w, c = np.array([1.0, 2.0], np.float32), np.array([5.0, 3.0], np.float32)
    m = DenseCRF2D(W, H, L)
    m.setUnaryEnergy(img["unary"])
    m.addPairwiseGaussian(3.0, 3.0, 3.0)
    m.addPairwiseBilateral(50.0, 50.0, 15.0, 15.0, 15.0, img["rgb"], 5.0)
    m.setCliques(off, idx, w, c)
    om = oracle_mod.build_model(oracle_mod.OracleModel, img)
    om.set_cliques(off, idx, w, c)
    q = om.unary_init()
    got = m.lp_inference_prox_super_pixels(q, prox_max_iter=2, fw_max_iter=3)
    want, _ = om.lp(q, prox_max_iter=2, fw_max_iter=3)
    assert (got.argmax(1) == want.argmax(1)).mean() >= 0.999


def test_a_second_solve_gives_the_same_bits():
    """... its graphs and buffers kept from the first."""
    W, H, L = 224, 160, 4
    img = dict(synth.make_image(W, H, L, 4))
    img["rgb"] = np.random.default_rng(1).integers(0, 256, size=img["rgb"].shape).astype(np.uint8)
    m = DenseCRF2D(W, H, L)
    m.setUnaryEnergy(img["unary"])
    m.addPairwiseGaussian(3.0, 3.0, 3.0)
    m.addPairwiseBilateral(50.0, 50.0, 15.0, 15.0, 15.0, img["rgb"], 5.0)
    q = m.unary_init()
    first = m.lp_inference_prox_super_pixels(q, prox_max_iter=3, fw_max_iter=6)
    assert np.array_equal(m.lp_inference_prox_super_pixels(q, prox_max_iter=3, fw_max_iter=6), first)
