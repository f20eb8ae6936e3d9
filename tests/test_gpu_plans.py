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


# Primitive pairs of the super pairs of a first-row atom in cc-pVDZ, whose s
# shells share nine exponents, the p shells four, and the d shell has one: the
# pair of a super shell with itself holds every unordered pair once.
CCPVDZ_ATOM = [45, 36, 10, 9, 4, 1]


@pytest.mark.parametrize("config,basis,pairs", [([("C", (0.1, 0.0, -0.2))], "cc-pVDZ", CCPVDZ_ATOM),
                                                ([("H", (0.0, 0.0, 0.0)), ("H", (0.0, 0.0, 1.4))], "6-31G",
                                                 [6, 1, 6, 1, 3, 3, 9, 3, 3, 1])], ids=["shared", "separate"])
def test_primitive_quartets_are_those_evaluated(config, basis, pairs):
    """Without a screen every unordered pair of super pairs is evaluated, each
    on all its primitive quartets."""
    with H.FockBuilder(config=config, basis_set=basis, screening_threshold=-1.0) as fb:
        fb.repulsion_matrix(_density(fb.K, 2))
        s, rows = fb.stats(), fb.plan()
    n = np.array(pairs)
    assert s["prim_quartets"] == (n.sum() ** 2 + (n * n).sum()) // 2
    assert s["prim_quartets"] == sum(r["prims"] for r in rows)
