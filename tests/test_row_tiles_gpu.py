"""The row-tiled softmax kernels of the 21-label path (mean-field iterations,
their adjoint, the initial Q) against the general-label kernels' definition, at
pixel counts around the 32-pixel tile and with several images per batch."""
import numpy as np
import pytest

from densecrf_ho_b200 import DenseCRF2D, DenseCRF2DBatch, synth

pytestmark = pytest.mark.gpu


def _softmax64(x):
    e = np.exp(x - x.max(1, keepdims=True))
    return e / e.sum(1, keepdims=True)


# one float rounding per exp, sum term and quotient of values in [0, 1]
TOL = 21 * 2.0 ** -23


@pytest.mark.parametrize("sizes", [[(1, 1)], [(31, 1)], [(32, 1)], [(33, 1)], [(127, 1), (129, 1), (5, 7)]])
def test_meanfield_without_terms(sizes):
    """No pairwise term: Q_1 = Q_0 = softmax(-U), and the adjoint of one step is
    dU = -(Q o (g - <g, Q>)) of Q_1 (Q_0 does not reach the output)."""
    L = 21
    b = DenseCRF2DBatch(sizes, L)
    rng = np.random.default_rng(3)
    U = rng.standard_normal((b.N, L)).astype(np.float32)
    g = rng.standard_normal((b.N, L)).astype(np.float32)
    b.setUnaryEnergy(U)
    Q = _softmax64(-U.astype(np.float64))
    assert np.abs(b.unary_init() - Q).max() < TOL
    q1 = b.meanfield(1)
    assert np.abs(q1 - Q).max() < TOL
    gu, gw = b.meanfield_backward(g)
    ref = -(Q * (g - (g * Q).sum(1, keepdims=True)))
    assert np.abs(gu - ref).max() < 8 * TOL  # |g| < 4.5: Q's error times g, twice
    assert len(gw) == 0


@pytest.mark.parametrize("W,H", [(1, 1), (31, 1), (33, 1), (40, 30)])
def test_unary_init(W, H):
    img = synth.make_image(W, H, 21, 2)
    m = DenseCRF2D(W, H, 21)
    m.setUnaryEnergy(img["unary"])
    assert np.abs(m.unary_init() - _softmax64(-img["unary"].astype(np.float64))).max() < TOL
