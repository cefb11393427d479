"""Kernels that carry one slice per thread at exact positions: positions in fixed
point (projector, backprojection of one to three slices, ragged batches).

They read the samples the four-slice gather kernels read and round in another
order; both stay within ~1e-6 of FP64 in relative L2 (tests of the operators), so
they agree to 3e-6.
"""
import numpy as np
import pytest
import torch

from acumen_gb300 import synthetic as syn
from acumen_gb300.batch import RaggedBatch
from acumen_gb300.tomography import Tomography

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def axes(T):
    """Angles on and near the axes, where rays run along the rim of the grid, and evenly spread ones."""
    near = [0.0, 45.0, 90.0, 135.0, 180.0, 89.9999, 90.0001, 1e-5, 179.99999]
    return np.concatenate([near, syn.angles(max(T, 1))])[:max(T, 1)].astype(np.float32)


# grids down to the smallest, around multiples of 32 and at the sides where the rows per thread change; angle counts
# around the 256 held in shared memory
@pytest.mark.parametrize("N, T, S", [(3, 9, 1), (4, 10, 2), (16, 9, 3), (31, 255, 1), (33, 256, 1), (65, 257, 2),
                                     (499, 30, 1), (500, 31, 1), (999, 9, 1), (1000, 20, 1), (2049, 9, 1)])
def test_one_slice_against_the_gather_kernels(N, T, S):
    g = torch.Generator(device="cuda").manual_seed(N)
    t = Tomography(N, axes(T), 2)
    x = torch.randn(S, N, N, device="cuda", generator=g)
    q = torch.randn(S, T, N, device="cuda", generator=g)
    four = lambda f, a: f(a[:1].repeat(4, 1, 1))[:1]   # noqa: E731
    assert rel(t.radon(x)[:1], four(t.radon, x)) < 3e-6
    bp = four(t.backproject, q)
    if bp.isfinite().all() and bp.any():               # on the smallest grids the mask is empty
        assert rel(t.backproject(q)[:1], bp) < 3e-6
        fbp = four(t.iradon, q)
        assert rel(t.iradon(q)[:1], fbp) < 3e-6
    t.close()


def test_ragged_batch_against_single_problems():
    """Sides around the tile heights (16 and 32 rows) and shared angle tables of unequal length."""
    sides, Ts = [17, 33, 63, 129, 200, 5], [257, 20, 256, 90, 31, 12]
    ths = [axes(T) for T in Ts]
    rng = np.random.default_rng(3)
    q = [rng.standard_normal((T, N)).astype(np.float32) for N, T in zip(sides, Ts)]
    x = [rng.standard_normal((N, N)).astype(np.float32) for N in sides]
    b = RaggedBatch(sides, ths, 2)
    for positions in (1, 0, 1):
        b.set_option(8, positions)
        r, i = b.radon(x), b.iradon(q)
        for k, (N, th) in enumerate(zip(sides, ths)):
            t = Tomography(N, th, 2)
            t.set_option(8, positions)
            np.testing.assert_array_equal(r[k], t.radon(x[k]))
            ref = t.iradon(q[k])
            assert np.linalg.norm(i[k] - ref) <= 3e-6 * max(np.linalg.norm(ref), 1e-30)
            t.close()
    b.close()
