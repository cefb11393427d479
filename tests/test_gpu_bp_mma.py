"""The backprojection on the tensor cores (automatic from 37 slices on, more on small
grids, exact positions) against the gather kernel (ACU_OPT_BP_GROUPS = 1) and
the FP64 oracle.

Each sums up to 2 T products in single precision in another order and stays
within 1e-6 of FP64 (the bar of test_exact_positions_backprojection), so they
agree to 2e-6 in relative L2.
"""
import numpy as np
import pytest
import torch

from acumen_gb300 import synthetic as syn
from acumen_gb300.tomography import Tomography

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def both(N, th, q, wpu=None):
    t = Tomography(N, th, wpu or max(4, N // 20))
    got = t.backproject(q)
    t.set_option(10, 1)
    ref = t.backproject(q)
    t.close()
    return got, ref


# sides around multiples of the 16-pixel tile, one and two blocks of 64 slices and more, angle counts around the four
# angles of two stages, angles on and near the axes and the diagonals (the widest windows)
@pytest.mark.parametrize("N, T, S", [(200, 1, 61), (800, 3, 37), (208, 2, 64), (209, 3, 65), (223, 4, 128), (224, 5, 130), (257, 41, 200)])
def test_matches_the_gather_kernel(N, T, S):
    near = [45.0, 0.0, 90.0, 135.0, 180.0, 44.0, 46.5, 89.9999, 90.0001, 1e-5]
    th = np.concatenate([near, syn.angles(T)]).astype(np.float32)[:T]
    q = torch.randn(S, T, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(N))
    got, ref = both(N, th, q)
    assert not torch.equal(got, ref)     # the other path did run
    assert rel(got, ref) < 2e-6
    assert torch.equal((got == 0).all(0), (ref == 0).all(0))   # outside the mask: zero in every slice


def test_against_fp64_and_same_result_twice(oracle, built_lib):
    N, T, S, wpu = 225, 300, 40, 12
    th = (syn.angles(T) + 0.13).astype(np.float32)
    q = np.random.default_rng(7).standard_normal((S, T, N)).astype(np.float32)
    t = Tomography(N, th, wpu)
    qc = torch.from_numpy(q).cuda()
    got = t.backproject(qc)
    assert torch.equal(got, t.backproject(qc))
    o = torch.from_numpy(oracle.backproject(q[:2].astype(np.float64), th, wpu, 64))
    assert rel(got[:2].cpu(), o) < 1e-6
    t.close()


def test_scales_of_slices():
    N, T, S = 209, 30, 64
    q = torch.randn(S, T, N, device="cuda")
    q[0] *= 1e30
    q[1] *= 1e-30
    q[2] = 0
    got, ref = both(N, syn.angles(T), q)
    assert not got[2].any()
    for s in (0, 1, 3):
        top = float(ref[s].abs().max())
        assert torch.isfinite(got[s]).all() and rel(got[s] / top, ref[s] / top) < 2e-6


def test_values_that_are_not_finite_stay_on_their_pixels():
    N, T, S = 209, 30, 64
    q = torch.randn(S, T, N, device="cuda")
    q[1, 3, 60] = float("nan")
    q[2, 7, 150] = float("inf")
    got, ref = both(N, syn.angles(T), q)
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.isinf(got), torch.isinf(ref))
    m = torch.isfinite(ref)
    assert rel(got[m], ref[m]) < 2e-6


def test_no_tile_meets_the_mask():
    """A margin wider than the grid leaves a mask of zeros."""
    q = torch.randn(64, 9, 209, device="cuda")
    got, ref = both(209, syn.angles(9), q, wpu=300)
    assert not got.any() and torch.equal(got, ref)


@pytest.mark.parametrize("S", [64, 130])
def test_a_value_that_is_not_finite_changes_no_other_slice(S):
    N, T = 209, 30
    q = torch.randn(S, T, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(S))
    bad = [5, 44]
    y = q.clone()
    y[5, 3, 60] = float("nan")
    y[44, 7, 150] = float("inf")
    t = Tomography(N, syn.angles(T), 10)
    clean, got = t.backproject(q), t.backproject(y)
    others = [s for s in range(S) if s not in bad]
    assert torch.equal(got[others], clean[others])
    t.set_option(10, 1)
    ref = t.backproject(y)[bad]
    got, m = got[bad], torch.isfinite(ref)
    assert not m.all() and m.any() and torch.equal(torch.isfinite(got), m) and rel(got[m], ref[m]) < 2e-6
    t.close()


def test_more_angles_than_a_grid_has_rows():
    """Sums of 2 T products in single precision in another order differ by sqrt(2 T) 2^-24."""
    N, T, S = 200, 65600, 45
    q = torch.rand(S, T, N, device="cuda")
    t = Tomography(N, syn.angles(T), 10)
    got = t.backproject(q)
    t.set_option(10, 1)
    ref = t.backproject(q)
    t.close()
    assert not torch.equal(got, ref) and rel(got, ref) < 2.2e-5


@pytest.mark.parametrize("S", [64, 130])
def test_a_bright_bin_takes_no_bits_from_the_others(S):
    """Pixels that a slice's one bright bin does not reach are as accurate as without it, however bright."""
    N, T = 209, 30
    th = syn.angles(T)
    q = torch.randn(S, T, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(S))
    y = q.clone()
    bright = {3: 1e4, 17: 1e6, 41: 1e12}
    spot = torch.zeros(4, T, N, device="cuda")
    spot[:, 3, 60] = 1.0
    for s, v in bright.items():
        y[s, 3, 60] = v
    got, ref = both(N, th, y)
    clean, _ = both(N, th, q)
    with Tomography(N, th, max(4, N // 20)) as t:
        away = t.backproject(spot)[0] == 0
    for s in bright:
        assert rel(got[s][away], ref[s][away]) < 2e-6, s
        assert rel(got[s], ref[s]) < 2e-6, s
    others = [s for s in range(S) if s not in bright]
    assert torch.equal(got[others], clean[others])
