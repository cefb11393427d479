"""The projector on the tensor cores (exact positions; automatic from 25 slices on
at sides from 500, from 33 or 45 at smaller ones from 200) against the gather
projector (variant 5) and the FP64 oracle.

Both round each sum to single precision in another order; a sum of up to 3 N
terms of one sign stays within ~1e-6 of FP64 either way (the bar of
test_operators_at_the_2049_grid is 5e-6), so they agree to 3e-6 in relative L2.
"""
import gc

import numpy as np
import pytest
import torch

from acumen_gb300 import synthetic as syn
from acumen_gb300.tomography import Tomography

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


def axes(T):
    """Angles on and near the axes and the diagonals (25-row windows) among evenly spread ones."""
    near = [0.0, 45.0, 90.0, 135.0, 180.0, 44.0, 46.5, 89.9999, 90.0001, 1e-5, 134.2]
    return np.concatenate([syn.angles(max(T - len(near), 1)), near])[:max(T, 1)].astype(np.float32)


def both(N, th, x):
    t = Tomography(N, th, max(4, N // 20))
    got = t.radon(x)
    t.set_option(7, 5)
    ref = t.radon(x)
    t.close()
    return got, ref


# sides at and around multiples of the 16-pixel tile; slices at the rule's lower end and around blocks of 64 and pairs
# of them; angle counts that leave a group of five partly filled
@pytest.mark.parametrize("N, T, S", [(500, 12, 25), (200, 12, 45), (208, 31, 64), (209, 33, 65), (223, 1, 128), (257, 40, 130),
                                     (224, 13, 200)])
def test_matches_the_gather_projector(N, T, S):
    g = torch.Generator(device="cuda").manual_seed(N)
    th = axes(T) if T > 11 else np.array([33.3], np.float32)
    for x in (torch.rand(S, N, N, device="cuda", generator=g), torch.randn(S, N, N, device="cuda", generator=g)):
        got, ref = both(N, th, x)
        assert not torch.equal(got, ref)     # the other path did run
        assert rel(got, ref) < 3e-6


def test_several_chunks_of_angles_and_same_result_twice():
    """Partial sums of 120 angles of two 64-slice blocks exceed what is held at once."""
    N, T, S = 1025, 120, 128
    x = torch.rand(S, N, N, device="cuda")
    t = Tomography(N, syn.angles(T), 50)
    got = t.radon(x)
    assert torch.equal(got, t.radon(x))
    t.set_option(7, 6)
    assert rel(got, t.radon(x)) < 3e-6
    t.close()


def test_against_fp64(oracle, built_lib):
    N, T, S = 225, 40, 48
    th = (syn.angles(T) + 0.21).astype(np.float32)
    x = np.random.default_rng(5).random((S, N, N), dtype=np.float32)
    got, ref = both(N, th, torch.from_numpy(x).cuda())
    o = torch.from_numpy(oracle.radon(x[:2].astype(np.float64), th, 64))
    assert rel(got[:2].cpu(), o) < 1e-6


def test_scales_of_slices_and_tiles():
    """Every tile of a slice has its own power-of-two scale: slices and regions of very different magnitude."""
    N, T, S = 209, 20, 48
    x = torch.rand(S, N, N, device="cuda")
    x[0] *= 1e30
    x[1] *= 1e-30
    x[2, :100] *= 1e6
    x[3] = 0
    x[4] = 0
    x[4, 77, 99] = 1e-20
    got, ref = both(N, axes(T), x)
    for s in range(6):
        assert torch.isfinite(got[s]).all()
        scale = float(ref[s].abs().max())
        assert rel(got[s] / max(scale, 1e-38), ref[s] / max(scale, 1e-38)) < 3e-6 if s != 3 else not got[s].any()


def test_values_that_are_not_finite_stay_on_their_rays():
    """A matrix product would spread a NaN or infinity over its tile: such a call takes plain gathers."""
    N, T, S = 209, 20, 48
    x = torch.rand(S, N, N, device="cuda")
    x[1, 100, 60] = float("nan")
    x[2, 30, 150] = float("inf")
    x[2, 31, 150] = float("-inf")
    got, ref = both(N, axes(T), x)
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.isinf(got), torch.isinf(ref))
    m = torch.isfinite(ref)
    assert rel(got[m], ref[m]) < 3e-6


def test_in_the_solver():
    """TV of a batch with the tensor-core projector against the gather projector, through a captured graph."""
    N, T, S = 209, 60, 48
    th = syn.angles(T)
    f = torch.stack([syn.normalised_sinogram(syn.random_ellipses(s, 0.3 * N), N, th, I0=5e3, seed=s, device="cuda")
                     for s in range(S)])
    t = Tomography(N, th, 10)
    tv, _ = t.tvopt(f, 1, 3, 4, 0.05, 1.0)
    t.set_option(3, 0)
    tv_l, _ = t.tvopt(f, 1, 3, 4, 0.05, 1.0)
    assert torch.equal(tv, tv_l)             # graph and launches
    t.set_option(7, 5)
    ref, _ = t.tvopt(f, 1, 3, 4, 0.05, 1.0)
    mask = t.backproject(torch.ones(1, T, N, device="cuda"))[0] != 0
    assert rel(tv[:, mask], ref[:, mask]) < 2e-5
    t.close()


def test_little_memory():
    """Where the work buffers do not fit, smaller chunks and then the gathers take over."""
    N, T, S = 513, 180, 64
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.rand(S, N, N, device="cuda", generator=g)
    t = Tomography(N, syn.angles(T), 25)
    p, img = t.radon(x), t.iradon(t.radon(x))
    t.close()
    torch.cuda.empty_cache()
    for room in (1500, 550):      # MB: three images of the batch are 200
        t = Tomography(N, syn.angles(T), 25)
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (room << 20), dtype=torch.uint8, device="cuda")
        got = t.radon(x)
        back = t.iradon(p)
        del hold
        torch.cuda.empty_cache()
        assert rel(got, p) < 3e-6 and rel(back, img) < 3e-6
        t.close()


# one to six groups of angles along each axis, one block of 64 slices and pairs of them
@pytest.mark.parametrize("T", [8, 20, 28, 40, 56])
@pytest.mark.parametrize("N, S", [(500, 25), (513, 128)])
def test_rows_that_neighbouring_tiles_share_are_added_in_order(N, T, S):
    """Four warps send the rows of a block and a ray moves among them from tile to tile: a row that was added before the
    first tile's value was stored, or in another order, would differ from call to call."""
    t = Tomography(N, syn.angles(T), 25)
    x = torch.rand(S, N, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(T))
    got = t.radon(x)
    for _ in range(50):
        assert torch.equal(got, t.radon(x))
    t.set_option(7, 5)
    ref = t.radon(x)
    assert not torch.equal(got, ref) and rel(got, ref) < 3e-6
    t.close()


@pytest.mark.parametrize("S", [48, 130])
def test_a_value_that_is_not_finite_changes_no_other_slice(S):
    N, T = 209, 20
    x = torch.rand(S, N, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(S))
    bad = [5, 44]
    y = x.clone()
    y[5, 100, 60] = float("nan")
    y[44, 30, 150] = float("inf")
    t = Tomography(N, axes(T), 10)
    clean, got = t.radon(x), t.radon(y)
    others = [s for s in range(S) if s not in bad]
    assert torch.equal(got[others], clean[others])
    assert got[5].isnan().any() and not got[5].isnan().all() and not got[44].isfinite().all()
    t.set_option(7, 5)
    ref = t.radon(y)[bad]
    got, m = got[bad], torch.isfinite(ref)
    assert torch.equal(torch.isfinite(got), m) and rel(got[m], ref[m]) < 3e-6
    t.close()


def test_less_and_less_memory_and_enough_again():
    """With a little less room than its buffers took the projector does the angles in smaller chunks, with the same bits;
    with what the pixel-line gathers need it is them; either way it is whole again once there is room.  Its buffers
    give way to what another call needs."""
    N, T, S = 513, 180, 64
    th = syn.angles(T)
    gc.collect()
    torch.cuda.empty_cache()         # so that every tensor here takes memory of its own
    x = torch.rand(S, N, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))

    def fresh(variant):
        torch.cuda.empty_cache()
        free = torch.cuda.mem_get_info()[0]
        t = Tomography(N, th, 25)
        t.set_option(7, variant)
        out = t.radon(x)
        torch.cuda.synchronize()
        taken = free - torch.cuda.mem_get_info()[0]
        t.close()
        return out, taken

    whole, most = fresh(7)
    lines, least = fresh(6)          # either counts the result's own memory
    assert not torch.equal(whole, lines) and most - least > 64 << 20
    for room, want in ((most - (16 << 20), whole), (least + (24 << 20), lines)):
        torch.cuda.empty_cache()
        t = Tomography(N, th, 25)
        hold = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
        got = t.radon(x)
        del hold
        torch.cuda.empty_cache()
        assert torch.equal(got, want)
        assert torch.equal(t.radon(x), whole)
        t.close()

    # filtering 256 slices needs 98 MB more than the projection left: 32 are free, its buffers hold the others
    y = torch.rand(256, T, N, device="cuda")
    with Tomography(N, th, 25) as t:
        ref = t.filter(y)
        t.filter(y)                  # leaves torch the memory of another result
    t = Tomography(N, th, 25)
    t.radon(x)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (32 << 20), dtype=torch.uint8, device="cuda")
    got = t.filter(y)
    del hold
    torch.cuda.empty_cache()
    assert torch.equal(got, ref)
    assert torch.equal(t.radon(x), whole)
    t.close()


@pytest.mark.parametrize("bright", [1e4, 1e6])
def test_a_bright_pixel_takes_no_bits_from_other_rays(bright):
    """The scale is a tile's: rays that miss a bright pixel but cross its tile are as accurate as without it."""
    N, T, S = 209, 20, 48
    th = axes(T)
    x = torch.randn(S, N, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(7))
    x[5, 100, 60] = bright
    spot = torch.zeros(4, N, N, device="cuda")
    spot[:, 100, 60] = 1.0
    got, ref = both(N, th, x)
    with Tomography(N, th, 10) as t:
        away = t.radon(spot)[0] == 0
    assert rel(got[5][away], ref[5][away]) < 3e-6 and rel(got[5], ref[5]) < 3e-6


def test_capture_of_a_call_that_found_no_memory_before():
    """The tensor-core projector is not tried again while its stream is captured: it would have to allocate."""
    N, T, S = 513, 180, 64
    gc.collect()
    torch.cuda.empty_cache()
    x = torch.rand(S, N, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    t = Tomography(N, syn.angles(T), 25)
    t.set_option(7, 6)
    lines = t.radon(x)               # with the gathers' buffers
    t.set_option(7, 7)
    out = t.radon(x[:4])             # leaves torch a block; the result below takes one of 24 MB
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (40 << 20), dtype=torch.uint8, device="cuda")
    got = t.radon(x)
    del hold, out
    torch.cuda.empty_cache()
    assert torch.equal(got, lines)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = t.radon(x)
    g.replay()
    assert torch.equal(got, lines)
    assert not torch.equal(t.radon(x), lines)
    t.close()
