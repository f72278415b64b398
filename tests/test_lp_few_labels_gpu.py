"""The LP on images of many vertices with few entries each: its ordered filters'
forms for few labels and very short lists, against the oracle."""
import numpy as np
import pytest

from densecrf_ho_b200 import DenseCRF2D, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H", [(64, 48), (97, 61)])
@pytest.mark.parametrize("L", [2, 3, 6, 7, 16, 21])
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
