"""Kernels that carry one slice per thread at exact positions: positions in fixed
point (projector, backprojection of one to three slices, ragged batches), the
projector's transpose and the projection with detector offsets.

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


@pytest.mark.parametrize("N, T, S", [(3, 9, 1), (16, 9, 4), (33, 40, 1), (64, 37, 3), (129, 30, 5), (257, 12, 1)])
def test_transpose_matches_the_projector(N, T, S):
    """<A x, y> = <x, A' y> per pixel of the rim too: x is one pixel at a time there."""
    g = torch.Generator(device="cuda").manual_seed(N)
    t = Tomography(N, axes(T), 2)
    y = torch.rand(S, T, N, device="cuda", generator=g)
    at = t.radon_adjoint(y)
    x = torch.rand(S, N, N, device="cuda", generator=g)
    lhs, rhs = float((t.radon(x).double() * y).sum()), float((x.double() * at).sum())
    assert abs(lhs - rhs) <= 1e-6 * abs(lhs)
    rim = torch.zeros(N, N, device="cuda")
    rim[:2] = rim[:, :2] = rim[-1] = rim[:, -1] = 1
    z = torch.zeros(4, N, N, device="cuda")
    z[0] = rim
    z[1, N - 1, N // 2] = z[2, 1, N // 2] = z[3, N // 2, N - 1] = 1
    r = t.radon(z)
    for k in range(4):
        lhs, rhs = float((r[k].double() * y[0]).sum()), float((z[k].double() * at[0]).sum())
        assert abs(lhs - rhs) <= 2e-6 * max(abs(lhs), 1e-3)
    t.close()


@pytest.mark.parametrize("N, T", [(33, 20), (129, 90), (200, 61)])
def test_offsets_loss_and_gradients(N, T):
    """Against the double-precision kernels, offsets among them that leave the grid or are not numbers."""
    g = torch.Generator(device="cuda").manual_seed(N)
    t = Tomography(N, (syn.angles(T) + 0.17).astype(np.float32), 4)
    S = 2
    u = torch.rand(S, N, N, device="cuda", generator=g)
    off = 2.0 * torch.randn(S, T, device="cuda", generator=g)
    y = torch.rand(S, T, N, device="cuda", generator=g)
    off[0, 1], off[0, 2] = 3.0 * N, 1e30
    l32, gu, go = t.tv_loss_grad(u, off, y, 0.05, 0.05)
    l64, gd, _ = t.tv_loss_grad(u.double(), off.double(), y.double(), 0.05, 0.05)
    np.testing.assert_allclose(l32, l64, rtol=1e-6)
    assert rel(gu, gd) < 2e-6
    assert not go[0, 1:3].any()
    off[0, 3] = float("nan")
    l32, gu2, go2 = t.tv_loss_grad(u, off, y, 0.05, 0.05)
    assert np.isfinite(l32).all() and torch.isfinite(gu2).all() and float(go2[0, 3]) == 0.0
    only, none, _ = t.tv_loss_grad(u, None, y, 0.05, 0.05, want_grad=False)
    np.testing.assert_allclose(only, t.tv_loss_grad(u, torch.zeros_like(off), y, 0.05, 0.05)[0], rtol=1e-12)
    assert none is None
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


def test_more_slices_than_a_buffer_of_pairs():
    """One slice per thread by option, more slices than the 1 GB of pairs hold at once (64 of 1025^2): those of the
    first and the last share are what they are alone."""
    N, T, S = 1025, 24, 130
    g = torch.Generator(device="cuda").manual_seed(4)
    u = torch.rand(S, N, N, device="cuda", generator=g)
    off = torch.rand(S, T, device="cuda", generator=g) - 0.5
    t = Tomography(N, syn.angles(T), 50)
    y = t.radon(u[:2])
    one = [(t.radon(u[s:s + 1]), t.iradon(y[:1] * (s + 1)), t.backproject(y[:1] * (s + 1)),
            t.tv_loss_grad(u[s:s + 1], off[s:s + 1], y[:1], 0.1, 1e-3)) for s in (0, 63, 64, S - 1)]
    yy = y[:1] * torch.arange(1, S + 1, device="cuda")[:, None, None]
    loss, gu, go = t.tv_loss_grad(u, off, y[:1].expand(S, T, N).contiguous(), 0.1, 1e-3)
    t.set_option(2, 1)
    p, r, b = t.radon(u), t.iradon(yy), t.backproject(yy)
    for k, s in enumerate((0, 63, 64, S - 1)):
        assert torch.equal(p[s], one[k][0][0]) and torch.equal(r[s], one[k][1][0]) and torch.equal(b[s], one[k][2][0])
        assert loss[s] == one[k][3][0][0] and torch.equal(gu[s], one[k][3][1][0]) and torch.equal(go[s], one[k][3][2][0])
    t.close()


# the reference's positions, and a side beyond the fixed-point kernels'
@pytest.mark.parametrize("N, positions", [(2049, 0), (4200, 1)])
def test_pairs_take_memory_only_where_they_are_used(N, positions):
    x = torch.rand(1, N, N, device="cuda")
    with Tomography(33, axes(9), 2) as t:
        t.radon(x[:, :33, :33])              # the library's code is loaded
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    t = Tomography(N, axes(9), 2)
    t.set_option(8, positions)
    y = t.radon(x)
    taken = free - torch.cuda.mem_get_info()[0]
    assert taken < 2 * 4 * N * N + 24e6      # the mask and a transposed image; the sinogram and tables are small
    assert rel(y, t.radon(x.repeat(4, 1, 1))[:1]) < 3e-6
    t.close()


def test_buffers_follow_options_changed_between_the_solvers_steps():
    """Other positions and another filter need other buffers for one slice."""
    N, T = 257, 90
    th = syn.angles(T)
    f = syn.normalised_sinogram(syn.random_ellipses(2, 0.3 * N), N, th, I0=5e3, seed=2, device="cuda")[None]
    for first, then in (((8, 0), (8, 1)), ((1, 1), (1, 0))):
        t = Tomography(N, th, 12)
        t.set_option(*first)
        t.tv_begin(f, 1, 3, 0.05, 1.0)
        t.set_option(*then)
        t.tv_iterate(2)
        u = t.tv_end()
        t.close()
        with Tomography(N, th, 12) as t:
            ref, _ = t.tvopt(f, 1, 2, 3, 0.05, 1.0)
            mask = t.backproject(torch.ones(1, T, N, device="cuda"))[0] != 0
        # TV with either stays within 1e-4 of FP64 inside the mask (test_gpu_tv)
        assert rel(u[:, mask], ref[:, mask]) < 2e-4
