"""The ramp filter at every transform length (16 to 8192) and either layout against
double precision: odd sides at both ends of a length's range, an odd number of
angles, slice counts of both layouts.

Two transforms of length L add up 2 log2(L) roundings of random sign: the error
stays near 2^-24 sqrt(2 log2 L) = 3e-7 at L = 8192 and below 2^-22 = 2.4e-7 of a row's
norm with roundings half that size; 4e-7 leaves a factor of two.
"""
import numpy as np
import pytest
import torch

from acumen_gb300 import synthetic as syn
from acumen_gb300.tomography import Tomography

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [7, 129, 130, 257, 258, 513, 514, 1025, 1026, 2049, 2050])
@pytest.mark.parametrize("T, S", [(1, 1), (5, 2), (6, 3), (3, 5), (4, 9)])
def test_filter_lengths(N, T, S):
    g = torch.Generator(device="cuda").manual_seed(N + T)
    x = torch.randn(S, T, N, device="cuda", generator=g)
    t, d = (Tomography(N, syn.angles(T), max(2, N // 20)) for _ in range(2))
    got, ref = t.filter(x).double(), d.filter(x.double())
    for s in range(S):
        for k in range(T):
            assert float((got[s, k] - ref[s, k]).norm() / ref[s, k].norm()) < 4e-7
    # as pairs, in front of the single-slice backprojection
    a, b = t.iradon(x[:1]).double(), d.iradon(x[:1].double())
    assert float((a - b).norm() / b.norm()) < 2e-6
    t.close()
    d.close()
