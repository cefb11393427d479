"""Preprocessing kernels at the sizes where they can go wrong: the cross-correlation
at the edges of its stretches (1024 pixels) and lag tiles (64) and on both sides
of its magnitude rules, the median at the edges of its tiles (32 x 16 pixels) and
walks (several projections and two pixels per thread at 400 x 250).  Everything is bit-exact against the oracle."""
import numpy as np
import pytest
import torch

from acumen_gb300.preprocess import Preprocessor

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pp(built_lib):
    return Preprocessor()


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("ndet,nrows,kmax", [(2, 1, 1), (7, 3, 31), (64, 2, 32), (65, 3, 33), (1023, 2, 63), (1024, 3, 64),
                                             (1025, 2, 256), (2049, 5, 512), (130, 700, 8)])
@pytest.mark.parametrize("kind", ["logs", "wide", "large"])
def test_xcorr_tiles(pp, oracle, ndet, nrows, kmax, kind):
    rng = np.random.default_rng(ndet + nrows)
    p0 = rng.normal(0.5, 1.0, (nrows, ndet)).astype(np.float32)
    p180 = (p0[:, ::-1] + rng.normal(0, 0.1, p0.shape)).astype(np.float32)
    if kind == "wide":      # zeros, denormals, products far below and just below the left shift
        p0 *= np.exp2(rng.integers(-140, 7, p0.shape)).astype(np.float32)
        p180 *= np.exp2(rng.integers(-20, 4, p0.shape)).astype(np.float32)
        p0[rng.random(p0.shape) < 0.1] = 0.0
        p180[rng.random(p0.shape) < 0.1] = -0.0
    if kind == "large":     # some stretches take the other route
        p0[rng.random(p0.shape) < 0.5 / (nrows * ndet) ** 0.5] *= np.float32(3e4)
        p180[0, ndet // 2] = 5e3
    kb, ks, corr = pp.xcorr_register(cu(p0), cu(p180), kmax)
    ko, kso, corr_o = oracle.xcorr_register(p0, p180, kmax)
    np.testing.assert_array_equal(corr, corr_o)
    assert kb == ko and ks == pytest.approx(kso, abs=1e-12)


@pytest.mark.parametrize("ndet,nrows,nproj", [(2, 1, 1), (31, 15, 2), (32, 16, 3), (33, 17, 16), (65, 33, 17), (5, 2, 33), (400, 250, 34)])
@pytest.mark.parametrize("special", [False, True])
def test_median_tiles(pp, oracle, ndet, nrows, nproj, special):
    rng = np.random.default_rng(ndet * nproj)
    proj = rng.normal(0, 1, (nproj, nrows, ndet)).astype(np.float32)
    if special:             # ties, both zeros, infinities, a NaN
        proj = np.round(proj * 2).astype(np.float32)
        proj[rng.random(proj.shape) < 0.2] = -0.0
        proj[rng.random(proj.shape) < 0.02] = np.inf
        proj[rng.random(proj.shape) < 0.02] = -np.inf
        proj[nproj // 2, nrows // 2, ndet // 2] = np.nan
    for p in range(nproj if ndet < 100 else 0):
        l, r = proj[max(p - 1, 0)], proj[min(p + 1, nproj - 1)]
        got = pp.median27(cu(l), cu(proj[p]), cu(r)).cpu().numpy()
        np.testing.assert_array_equal(got.view(np.uint32), oracle.median27(l, proj[p], r).view(np.uint32))
    with np.errstate(invalid="ignore"):
        got = pp.proj_to_sino(cu(proj), 0.003, 0.01).cpu().numpy()
        np.testing.assert_array_equal(got, oracle.proj_to_sino(proj, 0.003, 0.01))


@pytest.mark.parametrize("ndet,nrows,shift", [(65, 3, 2), (66, 9, -1), (1025, 4, 5), (300, 120, -3)])
def test_registration_sizes(pp, oracle, ndet, nrows, shift):
    """The search ends where the oracle's does.  Its errors differ by the order of
    FP64 sums, rounded to single precision: steps of 1e-4 times 1.05 and 1/3 end
    within 1e-4 of each other, as in the registration tests."""
    rng = np.random.default_rng(ndet)
    x = np.linspace(0, 1, ndet)[None, :] + 0.02 * np.arange(nrows)[:, None]
    p0 = (np.exp(-((x - 0.45) / 0.2) ** 2) + 0.3 * np.sin(9 * x) ** 2 + 0.01 * rng.normal(size=x.shape)).astype(np.float32)
    p180 = np.ascontiguousarray(np.roll(p0, shift, axis=1)[:, ::-1])
    th_g, sh_g, ne_g = pp.register(cu(p0), cu(p180))
    th_o, sh_o, ne_o = oracle.register(p0, p180, red_mode=1)
    assert abs(th_g - th_o) < 1e-4 and abs(sh_g - sh_o) < 1e-4
    again = pp.register(cu(p0), cu(p180))
    assert again == (th_g, sh_g, ne_g)
