"""What the plans of a job are rebuilt for, and what they report."""
import re

import numpy as np
import pytest

import hartree_fock_cpp_gb300 as H
from hartree_fock_cpp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _density(K, seed):
    P = np.random.default_rng(seed).uniform(-1.0, 1.0, size=(K, K)) / K
    return P + P.T


@pytest.mark.parametrize("precision", [H.HFX_PREC_FP64, H.HFX_PREC_MIXED])
def test_launch_shape_rebuilds_the_mixed_plan_only(precision, monkeypatch, capfd):
    """The launch shape is the FP32 launches': no FP64 plan is built for it, an
    FP64 job keeps the shape it was given through a tuning, and G stays."""
    monkeypatch.setenv("HFX_TRACE_SETUP", "1")
    plans = lambda: re.findall(r"team plan \((\w+)\)", capfd.readouterr().err)  # noqa: E731
    with H.FockBuilder(config=W.water(), basis_set="6-31G*", precision=precision, fp32_threshold=0.1) as fb:
        mixed = precision == H.HFX_PREC_MIXED
        assert plans() == ["fp64", "mixed"][:1 + mixed]
        P = _density(fb.K, 1)
        G = fb.repulsion_matrix(P)
        fb.set_launch_shape(100, 2000, 4, 10)
        assert plans() == ["mixed"] * mixed
        shape, ms = fb.autotune_launch_shape(P, builds=1)
        assert ms > 0 and shape == fb.launch_shape()
        built = plans()
        assert set(built) == {"mixed"} if mixed else built == []
        if not mixed:
            assert shape == dict(small_chunk=100, warp_chunk=2000, warp_max_warps=4, lane_min_npp=10)
        # 8 K^2 products at most, |D| <= 2 / K, FP32 within 1e-6 of an integral below 0.1
        assert np.abs(fb.repulsion_matrix(P) - G).max() < (1.6e-6 * fb.K if mixed else 1e-12)


def test_plan_rows_report_the_launches_team_sizes():
    """NaCl/cc-pVTZ has tasks for teams of one warp and of 128 threads."""
    with H.FockBuilder(config=W.nacl_scan(8)[3], basis_set="cc-pVTZ") as fb:
        rows = fb.plan()
    assert {r["pck"] for r in rows} == {32, 128}
    assert all(r["kind"] == 2 and r["warps_per_cta"] * 32 == r["pck"] for r in rows)
