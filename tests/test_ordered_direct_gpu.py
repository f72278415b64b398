"""The ordered slice on both sides of the line between one thread per element
and the staged form (fewer than 8 labels, or 2^17 pixel-label values), one
term and the LP's two, bit for bit."""
import numpy as np
import pytest

from densecrf_ho_b200 import DenseCRF2D, Permutohedral, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d", [2, 5])
@pytest.mark.parametrize("W,H,L", [(128, 128, 8), (129, 128, 8), (79, 79, 21), (80, 80, 21), (200, 101, 7)])
def test_both_forms_vs_oracle(W, H, L, d, oracle_mod):
    rng = np.random.default_rng(W + L)
    if d == 2:
        f = synth.gaussian_features(W, H, 3, 3)
    else:
        f = synth.bilateral_features(W, H, 50, 50, 15, 15, 15, synth.make_image(W, H, 21, 6)["rgb"])
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    for spread in (False, True):
        q = rng.random((W * H, L)).astype(np.float32)
        if not spread:
            q *= np.float32(0.08)
            q[np.arange(W * H), rng.integers(0, L, W * H)] = rng.random(W * H).astype(np.float32)
        assert np.array_equal(lat.compute_upper_minus_lower_ord(q), orc.compute_ord(q))


@pytest.mark.parametrize("W,H", [(79, 79), (80, 80)])
def test_lp_labels_vs_oracle(W, H, oracle_mod):
    """Both forms inside the LP: at most a label in a thousand differs, where
    the dual gap's sums, which the oracle adds one after the other, round a
    step length differently."""
    img = synth.make_image(W, H, 21, 3)
    orc = oracle_mod.build_model(oracle_mod.OracleModel, img)
    m = DenseCRF2D(W, H, 21)
    m.setUnaryEnergy(img["unary"])
    m.addPairwiseGaussian(3.0, 3.0, 3.0)
    m.addPairwiseBilateral(50.0, 50.0, 15.0, 15.0, 15.0, img["rgb"], 5.0)
    Q = orc.unary_init()
    a = m.lp_inference_prox_super_pixels(Q, prox_max_iter=3, fw_max_iter=4)
    b, _ = orc.lp(Q, prox_max_iter=3, fw_max_iter=4)
    assert (m.currentMap(a) == orc.current_map(b)).mean() >= 0.999
