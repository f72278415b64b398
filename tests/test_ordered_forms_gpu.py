"""The single ordered filter on both sides of each line between its quad and its
dense form: few labels over long and huge lists, many vertices, many pixels; bit
for bit against the oracle."""
import ctypes as C

import numpy as np
import pytest

from densecrf_ho_b200 import Permutohedral, device_memory_stats, lib, set_device_memory_limit, synth
from densecrf_ho_b200._lib import DCRFError, check

pytestmark = pytest.mark.gpu

DCRF_E_NOMEM = 5


def _features(W, H, d, kind):
    if kind == "line":
        return (np.arange(W * H, dtype=np.float32) / 7)[:, None]
    if kind == "grid":
        return synth.gaussian_features(W, H, 3, 3)
    rgb = synth.make_image(W, H, 21, 5)["rgb"]
    if kind == "noisy":
        rgb = np.random.default_rng(0).integers(0, 256, size=rgb.shape).astype(np.uint8)
    if kind == "half":  # noise beside one colour: many vertices and long lists
        rgb = np.random.default_rng(0).integers(0, 256, size=(H, W, 3)).astype(np.uint8)
        rgb[:, W // 2:] = 100
        rgb = rgb.reshape(-1, 3)
    s = 8 if kind == "wide" else 1  # wide: huge lists
    return np.ascontiguousarray(synth.bilateral_features(W, H, 50 * s, 50 * s, *[15 * s] * 3, rgb)[:, :d])


def _iterate(N, L, rng, spread):
    if spread:
        return rng.random((N, L)).astype(np.float32)
    q = rng.random((N, L)).astype(np.float32) * np.float32(0.08)
    q[np.arange(N), rng.integers(0, L, N)] = rng.random(N).astype(np.float32)
    return q


@pytest.mark.parametrize("W,H,d,kind,labels", [
    (257, 256, 5, "wide", (1, 2, 3, 4, 5, 8, 12, 13, 20, 21)),  # more than 2^16 pixels: every split of the long lists
    (256, 256, 5, "wide", (20, 21)),
    (513, 512, 5, "photo", (12, 13)),   # more than 2^18
    (257, 256, 3, "photo", (6, 20)),
    (97, 83, 5, "noisy", (1, 2, 6, 7, 12, 16, 17, 21, 33)),  # some 25 thousand vertices of few entries
    (200, 150, 5, "noisy", (1, 3, 4, 16, 17)),               # and 77 thousand
    (61, 47, 5, "noisy", (1, 2, 3, 4)), (31, 7, 3, "noisy", (1, 6, 7)),
    (512, 513, 2, "grid", (1,)), (512, 512, 2, "grid", (1, 2)),
    (128, 128, 2, "grid", (19, 20)), (127, 129, 2, "grid", (19, 20, 28, 29)),
    (31, 7, 2, "grid", (28, 29, 161)), (61, 47, 1, "line", (29,)),
])
def test_both_sides_of_each_line(W, H, d, kind, labels, oracle_mod):
    f = _features(W, H, d, kind)
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    rng = np.random.default_rng(W + d)
    for L in labels:
        for spread in (False, True):
            q = _iterate(W * H, L, rng, spread)
            assert np.array_equal(lat.compute_upper_minus_lower_ord(q), orc.compute_ord(q))


def test_restricted_and_plain_between_the_forms(oracle_mod):
    """One handle: the restricted filter shares the dense form's bins, the plain
    filter the value buffers of both."""
    W, H = 257, 256
    f = _features(W, H, 5, "wide")
    lat, orc = Permutohedral().init(f), oracle_mod.OracleLattice(f)
    rng = np.random.default_rng(3)
    pI = np.sort(rng.choice(W * H, 500, replace=False)).astype(np.int32)
    for L in (4, 21, 4):
        q, rq, rq2 = _iterate(W * H, L, rng, False), _iterate(500, L, rng, True), _iterate(500, L, rng, True)
        alone = Permutohedral().init(f)
        want = alone.compute_upper_minus_lower_ord_restricted(rq, pI, q, True)
        want2 = alone.compute_upper_minus_lower_ord_restricted(rq2, pI, None, False)
        full, plain = orc.compute_ord(q), orc.compute(q)
        assert np.array_equal(lat.compute_upper_minus_lower_ord(q), full)
        assert np.array_equal(lat.compute_upper_minus_lower_ord_restricted(rq, pI, q, True), want)
        assert np.array_equal(lat.compute(q), plain)
        assert np.array_equal(lat.compute_upper_minus_lower_ord(q), full)
        assert np.array_equal(lat.compute_upper_minus_lower_ord_restricted(rq2, pI, None, False), want2)


def _dev_filter(lat, x, entry, *args):
    import torch
    out = torch.full_like(x, float("nan"))
    torch.cuda.synchronize()
    check(entry(lat._h, C.c_void_p(out.data_ptr()), C.c_void_p(x.data_ptr()), x.shape[1], *args))
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _block(n):  # device blocks: powers of two split in quarters
    p = 512
    while p < n:
        p *= 2
    return p if p == 512 else -(-n // (p // 4)) * (p // 4)


@pytest.mark.parametrize("W,H,kind,L", [(97, 83, "noisy", 21), (97, 83, "photo", 21), (161, 120, "grid", 5),
                                        (97, 83, "half", 40), (97, 83, "half", 100)])
def test_without_memory_for_the_quads(W, H, kind, L):
    """Budgets below what a call of the quad form's range takes: the same bits or
    no memory, and never the latter where the dense form has room."""
    import torch
    N = W * H
    f = _features(W, H, 2 if kind == "grid" else 5, kind)
    x = torch.rand(N, L, generator=torch.Generator(device="cuda").manual_seed(L), device="cuda")
    entry = lib().dcrf_lattice_compute_ord_dev
    lat = Permutohedral().init(f)
    before = device_memory_stats()[0]
    want = _dev_filter(lat, x, entry)
    took = device_memory_stats()[0] - before
    dense = 2 * _block(80 * (lat.M + 1) * L) + _block(8 * N * L)
    del lat
    for budget in [took * k // 24 for k in range(25)] + [dense, took - 1]:
        lat = Permutohedral().init(f)
        set_device_memory_limit(device_memory_stats()[0] + budget)
        try:
            for _ in range(2):
                assert np.array_equal(_dev_filter(lat, x, entry), want)
        except DCRFError as e:
            assert e.code == DCRF_E_NOMEM and budget < dense
        finally:
            set_device_memory_limit(0)
        assert np.array_equal(_dev_filter(lat, x, entry), want)
        del lat


@pytest.mark.parametrize("W,H,kind,L", [(257, 256, "wide", 4), (257, 256, "wide", 21), (200, 150, "noisy", 3)])
def test_captured_in_a_caller_s_graph(W, H, kind, L):
    """A call captured on the lattice's stream and replayed on other values."""
    import torch
    f = _features(W, H, 5, kind)
    gen = torch.Generator(device="cuda").manual_seed(L)
    x, y = (torch.rand(W * H, L, generator=gen, device="cuda") for _ in range(2))
    entry = lib().dcrf_lattice_compute_ord_dev
    lat = Permutohedral().init(f)
    wants = [_dev_filter(lat, v, entry) for v in (x, y)]
    sp = C.c_void_p()
    check(lib().dcrf_lattice_stream(lat._h, C.byref(sp)))
    src, out = x.clone(), torch.empty_like(x)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.ExternalStream(sp.value), capture_error_mode="thread_local"):
        check(entry(lat._h, C.c_void_p(out.data_ptr()), C.c_void_p(src.data_ptr()), L))
    for v, want in zip((y, x), wants[::-1]):
        src.copy_(v)
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(out.cpu().numpy(), want)
    graph.reset()


def test_threads_with_lattices_of_their_own():
    """Both forms from several threads at once, each with its handle."""
    import threading

    import torch
    f, g = _features(257, 256, 5, "wide"), _features(97, 83, 5, "noisy")
    entry = lib().dcrf_lattice_compute_ord_dev
    jobs = []
    for L, feat in ((2, f), (12, f), (21, f), (1, g), (21, g)):
        x = torch.rand(len(feat), L, device="cuda", generator=torch.Generator(device="cuda").manual_seed(L))
        lat = Permutohedral().init(feat)
        jobs.append((lat, x, _dev_filter(lat, x, entry)))
    bad = []

    def work(lat, x, want):
        for _ in range(20):
            if not np.array_equal(_dev_filter(lat, x, entry), want):
                bad.append(x.shape)

    threads = [threading.Thread(target=work, args=j) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
