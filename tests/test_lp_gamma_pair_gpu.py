"""The LP's first two qp-gamma iterations inside the step that forms Y,
against the path that launches them one by one (which a tolerance of 1e30 and
above takes), bit for bit, and the iteration counts either takes -- at pixel
counts around the 32-pixel tile, with and without cliques, launch by launch
and through the iteration graph."""
import numpy as np
import pytest

from densecrf_ho_b200 import DenseCRF2D, synth

pytestmark = pytest.mark.gpu


def _model(W, H, cliques):
    img = synth.make_image(W, H, 21, 4)
    m = DenseCRF2D(W, H, 21)
    m.setUnaryEnergy(img["unary"])
    m.addPairwiseGaussian(3.0, 3.0, 3.0)
    m.addPairwiseBilateral(50.0, 50.0, 15.0, 15.0, 15.0, img["rgb"], 5.0)
    if cliques:
        N = W * H
        cut = np.unique([0, N // 3, N // 2, N])
        m.setCliques(cut.astype(np.int32), np.arange(N, dtype=np.int32),
                     np.full(len(cut) - 1, 3.0, np.float32), np.full(len(cut) - 1, 5.0, np.float32))
    return m


@pytest.mark.parametrize("cliques", [False, True])
@pytest.mark.parametrize("W,H", [(1, 1), (31, 1), (33, 1), (43, 3), (40, 30)])
def test_pair_vs_single_iterations(W, H, cliques):
    m = _model(W, H, cliques)
    Q = m.unary_init()

    def run(qp_max_iter, qp_tol):
        out, st = m.lp_inference_prox_super_pixels(Q, prox_max_iter=2, fw_max_iter=3, qp_max_iter=qp_max_iter,
                                                   qp_tol=qp_tol, stats=True)
        return out, st.gamma_iters / st.inner_iters, st.energy

    single = run(2, 1e30)  # second test passes: two iterations, launched singly
    for other in (run(2, 0.0), run(1000, 1e29)):
        assert np.array_equal(other[0], single[0]) and other[1:] == single[1:] and other[1] == 2
    first = run(1, 0.0)
    assert first[1] == 1
    unbounded = run(1000, np.inf)  # the first test passes already
    assert np.array_equal(unbounded[0], first[0]) and unbounded[1:] == first[1:]
    assert run(5, 0.0)[1] <= 5 and run(3, -1.0)[1] == 3
