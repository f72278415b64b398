"""A call that fails leaves the next one alone: a filter of more labels than the
device has memory for ends with DCRF_E_NOMEM on the host, before any launch,
and the same handle's next filters give the oracle's bits, whether the failed
call was its first or had value buffers to give up."""
import ctypes as C

import numpy as np
import pytest

from densecrf_ho_b200 import DCRFError, Permutohedral, device_memory_stats, lib, set_device_memory_limit, synth
from densecrf_ho_b200._lib import check

pytestmark = pytest.mark.gpu

E_NOMEM = 5


@pytest.mark.parametrize("entry", ["compute", "compute_ord"])
def test_valid_call_after_a_refused_one(entry, oracle_mod):
    import torch
    W, H, L = 40, 30, 21
    f = synth.bilateral_features(W, H, 50, 50, 15, 15, 15, synth.make_image(W, H, 21, 6)["rgb"])
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    assert lat.M > 200
    q = np.random.default_rng(1).random((W * H, L)).astype(np.float32)
    t = torch.zeros(1, device="cuda")  # never touched: the value buffers come first
    p = C.c_void_p(t.data_ptr())
    huge = 300_000_000  # 16 bytes a vertex and four labels: 240 GB and more
    with pytest.raises(DCRFError) as e:
        if entry == "compute":
            check(lib().dcrf_lattice_compute_dev(lat._h, p, p, huge, 0))
        else:
            check(lib().dcrf_lattice_compute_ord_dev(lat._h, p, p, huge))
    assert e.value.code == E_NOMEM
    assert np.array_equal(lat.compute(q), orc.compute(q))
    assert np.array_equal(lat.compute_upper_minus_lower_ord(q), orc.compute_ord(q))


# MiB that the large call may take beyond what is held: its staging, the bins,
# the first value buffer or only the second one is refused
@pytest.mark.parametrize("entry,room", [("compute", r) for r in (0, 15, 30, 50, 75, 90)] +
                         [("compute_ord", r) for r in (0, 30, 45, 100, 700, 900, 1200)])
def test_handle_whose_buffers_could_not_grow(entry, room, oracle_mod):
    W, H = 40, 30
    f = synth.bilateral_features(W, H, 50, 50, 15, 15, 15, synth.make_image(W, H, 21, 6)["rgb"])
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    rng = np.random.default_rng(2)
    small, large = (rng.random((W * H, n)).astype(np.float32) for n in (21, 4000))
    call, want = ((lat.compute, orc.compute) if entry == "compute"
                  else (lat.compute_upper_minus_lower_ord, orc.compute_ord))
    assert np.array_equal(call(small), want(small))
    set_device_memory_limit(device_memory_stats()[0] + (room << 20))
    try:
        with pytest.raises(DCRFError) as e:
            call(large)
        assert e.value.code == E_NOMEM
    finally:
        set_device_memory_limit(0)
    assert np.array_equal(call(small), want(small))
