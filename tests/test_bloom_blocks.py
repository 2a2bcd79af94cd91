"""The bloom chain's taps from one block of texels (kpt_post.cu TapAxis, large
levels) against the taps read one by one, in single precision on the CPU: the
same bits at every pixel that takes the block, and which pixels those are."""

import numpy as np
import pytest

F = np.float32


def _position(n, m):
    return np.arange(n, dtype=F) / F(n) * F(m)


def _lerp(a, b, t):
    return a + t * (b - a)


def _one_by_one(img, px, py):
    """textureReadBilinear at every (py, px), indices clamped."""
    h, w = img.shape
    x, y = px.astype(np.int32), py.astype(np.int32)
    ws, wt = (px - x.astype(F))[None, :], (py - y.astype(F))[:, None]
    at = lambda dy, dx: img[np.clip(y + dy, 0, h - 1)[:, None], np.clip(x + dx, 0, w - 1)[None, :]]
    return _lerp(_lerp(at(0, 0), at(0, 1), ws), _lerp(at(1, 0), at(1, 1), ws), wt)


def _axis(p, radius, n):
    """index of offset 0, weight per offset, and where the taps form a block"""
    i = p.astype(np.int32)
    w, inside = {}, (i >= radius) & (i + radius + 1 < n)
    for o in range(-radius, radius + 1):
        f = p + F(o)
        k = f.astype(np.int32)
        w[o] = f - k.astype(F)
        inside &= k == i + o
    return i, w, inside


@pytest.mark.parametrize("radius,offsets", [
    (1, [(i, j) for j in (-1, 0, 1) for i in (-1, 0, 1)]),
    (2, [(i, j) for j in (-2, 0, 2) for i in (-2, 0, 2)] + [(-1, 1), (1, 1), (-1, -1), (1, -1)]),
])
@pytest.mark.parametrize("dst,src", [((640, 455), (1283, 911)), ((1283, 911), (641, 455)), ((960, 540), (1920, 1080)),
                                     ((1920, 1080), (960, 540)), ((316, 320), (632, 640)), ((400, 251), (200, 125))])
def test_block_taps_are_the_taps(radius, offsets, dst, src):
    img = np.random.default_rng(3).random((src[1], src[0]), F) * F(50.0)
    px, py = _position(dst[0], src[0]), _position(dst[1], src[1])
    (xi, xw, xin), (yi, yw, yin) = _axis(px, radius, src[0]), _axis(py, radius, src[1])
    assert xin.mean() > 0.9 and yin.mean() > 0.9          # the block is the rule, edges the exception
    xs, ys = np.flatnonzero(xin), np.flatnonzero(yin)
    for ox, oy in offsets:
        want = _one_by_one(img, px + F(ox), py + F(oy))[np.ix_(ys, xs)]
        row = lambda r: _lerp(img[(yi[ys] + r)[:, None], (xi[xs] + ox)[None, :]],
                              img[(yi[ys] + r)[:, None], (xi[xs] + ox + 1)[None, :]], xw[ox][xs][None, :])
        got = _lerp(row(oy), row(oy + 1), yw[oy][ys][:, None])
        assert got.dtype == F
        np.testing.assert_array_equal(got.view(np.int32), want.view(np.int32))
