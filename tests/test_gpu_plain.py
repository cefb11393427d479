"""The per-slice TV path at exact positions against the FP64 golden result: its
general projector (k_radon) has to use the exact positions too (with the
reference's it ends 1.6e-4 away, past the bar of 1e-4 that all paths share)."""
import pytest
from test_gpu_configs import _solve, rel, tv_case  # noqa: F401

pytestmark = pytest.mark.gpu


def test_plain_path_exact_positions_vs_fp64_golden(tv_case, oracle):  # noqa: F811
    if tv_case["tv64"] is None:
        pytest.skip("golden FP64 result not generated")
    mg = tv_case["mg"]
    mask = oracle.cmask(mg.N, mg.T, mg.WPU, 64) > 0
    assert rel(_solve(tv_case, 1, True), tv_case["tv64"], mask) <= 1e-4
