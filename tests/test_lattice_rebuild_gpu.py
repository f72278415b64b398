"""What a lattice handle may keep when it is initialised again, and what not: the
splat stored by the restricted ordered filter belongs to the former lattice
(DCRF_E_STATE until a store call on the new one), an initialisation or a store
call that is refused leaves none behind, and the handle works afterwards; bit
for bit against the oracle."""
import numpy as np
import pytest

from densecrf_ho_b200 import DCRFError, Permutohedral, device_memory_stats, set_device_memory_limit, synth

pytestmark = pytest.mark.gpu

E_STATE, E_NOMEM = 4, 5


def _features(W, H, seed):
    return synth.bilateral_features(W, H, 50, 50, 15, 15, 15, synth.make_image(W, H, 21, seed)["rgb"])


def _inputs(N, L, seed):
    rng = np.random.default_rng(seed)
    pI = np.sort(rng.choice(N, N // 3, replace=False)).astype(np.int32)
    q = rng.random((N, L)).astype(np.float32)
    return pI, q, rng.random((pI.size, L)).astype(np.float32)


def _code(call):
    with pytest.raises(DCRFError) as e:
        call()
    return e.value.code


def test_stored_splat_ends_with_its_lattice(oracle_mod):
    lat = Permutohedral().init(_features(40, 30, 1))
    pI, q, rq = _inputs(40 * 30, 21, 1)
    lat.compute_upper_minus_lower_ord_restricted(rq, pI, q, store=True)
    f = _features(30, 20, 2)  # fewer pixels: every buffer is large enough
    lat.init(f)
    pI, q, rq = _inputs(30 * 20, 21, 2)
    assert _code(lambda: lat.compute_upper_minus_lower_ord_restricted(rq, pI, store=False)) == E_STATE
    want = oracle_mod.RestrictedOrd(lat.export(), 5).compute(rq, pI, q, True)
    assert np.array_equal(lat.compute_upper_minus_lower_ord_restricted(rq, pI, q, store=True), want)
    assert np.array_equal(lat.compute_upper_minus_lower_ord_restricted(rq, pI, store=False), want)


def test_refused_store_call_leaves_no_splat():
    lat = Permutohedral().init(_features(40, 30, 1))
    pI, q, rq = _inputs(40 * 30, 21, 1)
    want = lat.compute_upper_minus_lower_ord_restricted(rq, pI, q, store=True)
    pL, qL, rqL = _inputs(40 * 30, 400, 3)
    set_device_memory_limit(device_memory_stats()[0] + (20 << 20))
    try:
        assert _code(lambda: lat.compute_upper_minus_lower_ord_restricted(rqL, pL, qL, store=True)) == E_NOMEM
    finally:
        set_device_memory_limit(0)
    assert _code(lambda: lat.compute_upper_minus_lower_ord_restricted(rq, pI, store=False)) == E_STATE
    assert np.array_equal(lat.compute_upper_minus_lower_ord_restricted(rq, pI, q, store=True), want)


def test_refused_initialisation_leaves_no_lattice(oracle_mod):
    small, large = _features(40, 30, 1), _features(320, 240, 2)
    lat = Permutohedral().init(small)
    q = np.random.default_rng(4).random((40 * 30, 21)).astype(np.float32)
    lat.compute(q)
    for room in (4, 16):  # MiB beyond what is held: the features fit, the build, which needs some 60, does not
        set_device_memory_limit(device_memory_stats()[0] + (room << 20))
        try:
            assert _code(lambda: lat.init(large)) == E_NOMEM
        finally:
            set_device_memory_limit(0)
        assert _code(lambda: lat.compute(q)) == E_STATE
        lat.init(small)
        assert np.array_equal(lat.compute(q), oracle_mod.OracleLattice(small).compute(q))
