"""A plain filter whose value rows number more than 2^31 16-byte groups: 1000
labels over some nine million vertices, value buffers of 38 GB each.  The
labels do not mix, so the same lattice's filter of 21 of them, whose rows are
far below the line, gives the expected bits; the last pixels' vertices are the
last of the value buffer."""
import ctypes as C

import pytest

from densecrf_ho_b200 import Permutohedral, lib
from densecrf_ho_b200._lib import check

pytestmark = pytest.mark.gpu


def test_rows_past_two_to_the_31_groups():
    import torch
    N, d, L = 560_000, 16, 1000
    torch.cuda.empty_cache()
    check(lib().dcrf_release_cached_memory())
    if torch.cuda.mem_get_info()[0] < 140 << 30:
        pytest.skip("needs 140 GB of free device memory")
    gen = torch.Generator(device="cuda").manual_seed(1)
    f = 40.0 * torch.randn(N, d, generator=gen, device="cuda")  # spread out: next to no vertex shared
    x = torch.rand(N, L, generator=gen, device="cuda")
    out = torch.empty_like(x)
    lat = Permutohedral()
    torch.cuda.synchronize()
    check(lib().dcrf_lattice_init_dev(lat._h, C.c_void_p(f.data_ptr()), d, N))
    try:
        M = C.c_int()
        check(lib().dcrf_lattice_info(lat._h, C.byref(M), None, None))
        assert (M.value + 1) * (L // 4) >= 1 << 31
        check(lib().dcrf_lattice_compute_dev(lat._h, C.c_void_p(out.data_ptr()), C.c_void_p(x.data_ptr()), L, 0))
        torch.cuda.synchronize()
        for k in (0, L - 21):
            xs = x[:, k:k + 21].contiguous()
            ref = torch.empty_like(xs)
            torch.cuda.synchronize()
            check(lib().dcrf_lattice_compute_dev(lat._h, C.c_void_p(ref.data_ptr()), C.c_void_p(xs.data_ptr()), 21, 0))
            torch.cuda.synchronize()
            assert torch.equal(out[:, k:k + 21], ref)
    finally:
        del lat, x, out
        torch.cuda.empty_cache()
        check(lib().dcrf_release_cached_memory())
