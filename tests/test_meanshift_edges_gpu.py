"""The mode search at the edges of its work split -- images of fewer pixels
than a warp holds, runs of candidates shorter and longer than a step, windows
that hold the whole image, flat and noisy colours -- against the same
procedure written out in Python doubles, bit for bit."""
import ctypes as C
import math

import numpy as np
import pytest

from densecrf_ho_b200 import _lib

f32 = np.float32


def _luv(c):
    r, g, b = (float(v) for v in c)
    x = 0.4125 * r + 0.3576 * g + 0.1804 * b
    y = 0.2125 * r + 0.7154 * g + 0.0721 * b
    z = 0.0193 * r + 0.1192 * g + 0.9502 * b
    l0 = y / 255.0
    L = f32(116.0 * math.pow(l0, 1.0 / 3.0) - 16.0) if l0 > 0.008856 else f32(903.3 * l0)
    den = x + 15 * y + 3 * z
    up, vp = (4 * x / den, 9 * y / den) if den != 0 else (4.0, 9.0 / 15.0)
    thirteen = float(f32(13) * L)
    return L, f32(thirteen * (up - 0.19784977571475)), f32(thirteen * (vp - 0.46834507665248))


def _oracle(rgb, W, H, s, r):
    N, ss, sr = W * H, f32(s), f32(r)
    pts = [[float(f32(i % W) / ss), float(f32(i // W) / ss)] + [float(v / sr) for v in _luv(rgb[i])] for i in range(N)]
    smin = min(p[2] for p in pts)
    cell = lambda y: (int(y[0]) + 1, int(y[1]) + 1, int(y[2] - smin) + 1)  # noqa: E731
    grid = {}
    for i in range(N - 1, -1, -1):
        grid.setdefault(cell(pts[i]), []).append(pts[i])
    hi = 80.0 / float(sr)

    def shift(y):
        c, sums, n = cell(y), [0.0] * 5, 0
        for a in (-1, 0, 1):
            for b in (-1, 0, 1):
                for d in (-1, 0, 1):
                    for p in grid.get((c[0] + a, c[1] + b, c[2] + d), ()):
                        e = [p[j] - y[j] for j in range(5)]
                        if not e[0] * e[0] + e[1] * e[1] < 1.0:
                            continue
                        lum = 4.0 * e[2] * e[2] if y[2] > hi else e[2] * e[2]
                        if lum + e[3] * e[3] + e[4] * e[4] < 1.0:
                            sums = [sums[j] + p[j] for j in range(5)]
                            n += 1
        return [sums[j] / float(n) - y[j] for j in range(5)] if n else [0.0] * 5

    out = np.zeros((N, 3), f32)
    for i in range(N):
        y, it = list(pts[i]), 1
        m = shift(y)
        mv = 0.0
        for v in m:
            mv += v * v
        while mv >= 0.01 and it < 100:
            y = [y[j] + m[j] for j in range(5)]
            m = shift(y)
            mv = (m[0] * m[0] + m[1] * m[1]) * float(ss) * float(ss)
            mv += (m[2] * m[2] + m[3] * m[3] + m[4] * m[4]) * float(sr) * float(sr)
            it += 1
        y = [y[j] + m[j] for j in range(5)]
        out[i] = [f32(v * float(sr)) for v in y[2:]]
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("W,H,s,r,kind", [
    (1, 1, 8, 8.0, "noise"), (3, 1, 1, 5.0, "noise"), (1, 9, 2, 6.5, "flat"), (7, 5, 3, 8.0, "steps"),
    (17, 9, 1, 12.0, "noise"), (13, 11, 40, 8.0, "steps"), (33, 8, 4, 30.0, "noise"), (16, 16, 5, 7.0, "bright"),
])
def test_mode_search_vs_written_out(W, H, s, r, kind):
    rng = np.random.default_rng(W * 100 + H)
    N = W * H
    if kind == "flat":
        rgb = np.full((N, 3), 77, np.uint8)
    elif kind == "noise":
        rgb = rng.integers(0, 256, (N, 3), dtype=np.uint8)
    elif kind == "steps":
        rgb = (np.repeat((np.arange(N) // 6 * 40 % 256)[:, None], 3, 1) + rng.integers(0, 6, (N, 3))).clip(0, 255).astype(np.uint8)
    else:  # around the level from which the L distance counts four-fold
        rgb = rng.integers(180, 256, (N, 3), dtype=np.uint8)
    rgb = np.ascontiguousarray(rgb)
    out = np.zeros((N, 3), f32)
    _lib.check(_lib.lib().dcrf_meanshift_filter(rgb.ctypes.data_as(C.c_void_p), W, H, s, C.c_float(r),
                                                out.ctypes.data_as(C.c_void_p)))
    assert np.array_equal(out, _oracle(rgb, W, H, s, r))
