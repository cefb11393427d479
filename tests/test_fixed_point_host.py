"""Host-side checks of the fixed-point sample positions of the single-slice
kernels, the ragged batch and the transpose (csrc/fixed.cuh, csrc/ray_weights.cuh), by
emulating their integer arithmetic in numpy (no GPU): how far a position is from FP64, and
grid-aligned angles, where samples sit on cell edges.
"""
import numpy as np
import pytest

from test_geometry_host import exact_coord, f32, split


def tables(v, mid):
    k = 0
    while (1 << k) <= mid:
        k += 1
    return split(v, 23 - k)


def near(v):
    """A position's cell and fraction as the kernels keep them: 23 bits of the fraction after rounding."""
    return np.floor(v * 2.0**23) * 2.0**-23


@pytest.mark.parametrize("N", [3, 725, 2049, 4097])
def test_positions_along_a_ray(N):
    """64-bit coordinates with 32 fraction bits: sine and cosine are off by 2^-33, times at most N / 2 each, and the
    fraction is rounded to 2^-24."""
    mid = (N + 1) // 2
    rng = np.random.default_rng(N)
    for th in np.concatenate([rng.uniform(0, 180, 20), [0.0, 45.0, 90.0, 180.0]]).astype(np.float32):
        a = np.pi * (float(th) - 90.0) / 180.0
        (sa, sr), (ca, cr) = tables(np.sin(a), mid), tables(np.cos(a), mid)
        s = int(np.rint((float(sa) + float(sr)) * 2.0**32))
        c = int(np.rint((float(ca) + float(cr)) * 2.0**32))
        jx, jy = rng.integers(1, N + 1, size=(2, 400))
        x = (mid << 32) - s * (jy - mid) + c * (jx - mid) + (1 << 8)
        y = (mid << 32) + c * (jy - mid) + s * (jx - mid) + (1 << 8)
        xr = np.cos(a) * (jx - mid) - np.sin(a) * (jy - mid) + mid
        yr = np.sin(a) * (jx - mid) + np.cos(a) * (jy - mid) + mid
        for fx, exact in ((x, xr), (y, yr)):
            assert np.abs(near(fx * 2.0**-32) - exact).max() < N * 2.0**-33 + 2.0**-24 + 1e-9
            if th in (0.0, 90.0, 180.0):
                assert np.array_equal(fx >> 32, np.rint(exact).astype(np.int64))   # cells, as on an exact edge


@pytest.mark.parametrize("N, T", [(129, 40), (725, 40), (2049, 40), (4097, 40)])
def test_positions_within_a_tile(N, T):
    """32-bit positions relative to a tile's middle pixel, with 26 fraction bits: the middle's own 1.5e-7, 2^-26 where it is
    cut off, 2^-27 a step for up to 16 pixels in either direction, and the fraction rounded to 2^-24."""
    bound = 1.5e-7 + 2.0**-26 + 32 * 2.0**-27 + 2.0**-24
    assert bound < 5e-7
    mid = (N + 1) // 2
    rng = np.random.default_rng(N)
    one = f32(2.0**26)
    lx, ly = np.meshgrid(np.arange(-16, 16), np.arange(-16, 16))
    for th in rng.uniform(0, 180, T).astype(np.float32):
        a = np.pi * (90.0 - float(th)) / 180.0
        (sa, sr), (ca, cr) = tables(np.sin(a), mid), tables(np.cos(a), mid)
        sx = int(sa * one) + int(np.rint(f32(sr * one)))
        sy = int(ca * one) + int(np.rint(f32(cr * one)))
        x0, y0 = rng.integers(17, N - 15, size=2)
        cell, frac = exact_coord(sa, ca, sr, cr, f32(x0 - mid), f32(y0 - mid), f32(mid))
        p = int(f32(frac) * one) + 4 + lx * sx + ly * sy
        assert np.abs(p).max() < 2**31
        got = near(cell + p * 2.0**-26)
        exact = np.sin(a) * (x0 + lx - mid) + np.cos(a) * (y0 + ly - mid) + mid
        assert np.abs(got - exact).max() < bound
