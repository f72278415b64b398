"""Handles made and destroyed in numbers and from several threads: the pool of
page-locked slots behind the models' read-backs, and solves before and after the
first solve's loop becomes a graph."""
import threading

import numpy as np
import pytest

from densecrf_ho_b200 import DenseCRF2D, lib, synth
from densecrf_ho_b200._lib import check

pytestmark = pytest.mark.gpu


def _model(img):
    m = DenseCRF2D(img["W"], img["H"], 21)
    m.setUnaryEnergy(img["unary"])
    m.addPairwiseGaussian(3.0, 3.0, 3.0)
    m.addPairwiseBilateral(50.0, 50.0, 15.0, 15.0, 15.0, img["rgb"], 5.0)
    return m


def test_more_models_than_one_slab_and_release():
    img = synth.make_image(16, 12, 21, 1)
    ref = None
    for _ in range(2):
        models = [_model(img) for _ in range(70)]  # a slab holds 64
        for m in models[::7]:
            q = m.qp_inference_super_pixels_non_convex(m.unary_init())
            ref = q if ref is None else ref
            assert np.array_equal(q, ref)
        del models, m
        check(lib().dcrf_release_cached_memory())


def test_models_from_threads():
    img = synth.make_image(24, 18, 21, 2)
    m = _model(img)
    ref = m.qp_inference_super_pixels_non_convex(m.unary_init())
    bad = []

    def work():
        for _ in range(6):
            t = _model(img)
            if not np.array_equal(t.qp_inference_super_pixels_non_convex(t.unary_init()), ref):
                bad.append(1)

    ts = [threading.Thread(target=work) for _ in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad


def test_repeated_solves_equal_the_first(oracle_mod):
    """Eager first solve, then the graph, then again after a model change."""
    img = synth.make_image(48, 33, 21, 3)
    m, om = _model(img), oracle_mod.build_model(oracle_mod.OracleModel, img)
    Q = om.unary_init()
    ref = om.qp(Q)[0]
    for _ in range(3):
        assert np.array_equal(m.qp_inference_super_pixels_non_convex(Q), ref)
    u = np.ascontiguousarray(img["unary"][::-1])
    m.setUnaryEnergy(u)
    fresh = _model(dict(img, unary=u))
    for _ in range(2):
        assert np.array_equal(m.qp_inference_super_pixels_non_convex(Q),
                              fresh.qp_inference_super_pixels_non_convex(Q))
