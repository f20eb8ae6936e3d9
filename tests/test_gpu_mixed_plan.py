"""Joins of the super-shell kernel with the rest of a build: member quartets
split between FP64 and FP32 launches, f functions of an open shell in mixed
precision, tasks whose bra pairs the density screen drops in part, and plans of
many launches."""
import numpy as np
import pytest

import native_driver
import oracle as O
import hartree_fock_cpp_gb300 as H
from hartree_fock_cpp_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _densities(K, seed):
    rng = np.random.default_rng(seed)
    return [(P + P.T) / K for P in rng.uniform(-1.0, 1.0, size=(2, K, K))]


# A FP32 integral is within 1e-6 of its bound, which is below tau and below the
# largest integral (5 here); an element of J or K sums at most K^2 of them, of
# G 3/2 K^2, with |D| <= 2 / K (|Da + Db| <= 4 / K).
def _tolerance(K, tau):
    return 1e-11 + 4e-6 * min(tau, 5.0) * K


@pytest.mark.parametrize("tau", [1e-7, 1e-3, 0.1, 1e3])
@pytest.mark.parametrize("config,basis", [([("O", (0.0, 0.0, 0.0)), ("H", (0.0, 0.3, 1.8))], "cc-pVDZ"),
                                          (W.water(), "6-31G*"), ([("C", (0.0, 0.0, 0.0)), ("H", (0.0, 0.0, 2.1))], "cc-pVTZ")],
                         ids=["general_contraction", "sp", "f"])
def test_members_split_between_precisions_match_oracle(config, basis, tau):
    """From every quartet in FP64 to every quartet in FP32."""
    orc = O.Oracle(config, basis, stable_boys=True)
    eri = orc.repulsion_tensor_mt(1e-8)
    K = orc.K
    Pa, Pb = _densities(K, 21)
    want = [O.repulsion_matrix(Pa, eri), O.coulomb_matrix(Pa, Pb, eri), O.exchange_matrix(Pa, eri),
            O.exchange_matrix(Pb, eri)]
    with H.FockBuilder(config=config, basis_set=basis, precision=H.HFX_PREC_MIXED, fp32_threshold=tau) as fb:
        for _ in range(2):              # the eager build, then the graph
            got = [fb.repulsion_matrix(Pa)] + list(fb.coulomb_exchange(Pa, Pb))
            for g, w in zip(got, want):
                assert np.abs(g - w).max() < _tolerance(K, tau)
        s = fb.stats()
    assert 0 <= s["quartets_fp32"] <= s["quartets"]
    assert (s["quartets_fp32"] == s["quartets"]) == (tau == 1e3)


SCREENED = r"""
#include <cstdio>
#include <cstdlib>
#include "hfx_engine.hpp"
int main(int argc, char** argv)
{
    const int n = std::atoi(argv[1]);
    const double dthr = std::atof(argv[2]);
    std::vector<const char*> sym(n, "H");
    std::vector<double> xyz(3 * n), P, G;
    for (double& x : xyz) if (std::scanf("%lf", &x) != 1) return 2;
    hfx_molecule m{n, sym.data(), xyz.data(), "6-31G", nullptr};
    hfx_options o{};
    hfx::Job job(hfx::build_basis(m), o);
    const int K = job.K();
    P.resize(K * K);
    G.resize(K * K);
    for (double& x : P) if (std::scanf("%lf", &x) != 1) return 2;
    for (int k = 0; k < 2; ++k) job.fock_rhf_ex(P.data(), G.data(), false, dthr);
    for (double x : G) std::printf("%.17g\n", x);
}
"""


@pytest.mark.parametrize("dthr", [1e-7, 1e-5, 1e-4])
def test_density_screen_drops_single_bra_pairs_of_a_task(tmp_path, dthr):
    """Every super shell of hydrogen in 6-31G is one s function, so a super
    quartet's screen is known exactly: the oracle's integrals without the
    dropped quartets.  The density has elements of all sizes from 1e-8 to 1, so
    that tasks lose bra pairs at their start, in the middle and at their end."""
    rng = np.random.default_rng(4)
    n = 14
    xyz = np.stack([np.arange(n) * 1.7, rng.uniform(-0.5, 0.5, n), rng.uniform(-0.5, 0.5, n)], 1)
    orc = O.Oracle([("H", tuple(p)) for p in xyz], "6-31G", stable_boys=True)
    K = orc.K
    P = rng.choice([-1.0, 1.0], (K, K)) * 10.0 ** rng.uniform(-8.0, 0.0, (K, K)) / K
    P = np.tril(P) + np.tril(P, -1).T
    Q = orc.schwarz_bounds()
    i, j = np.tril_indices(K)
    A = np.abs(P)
    eri = O.full_eri(orc.repulsion_tensor_mt(1e-8), K)[i, j][:, i, j]
    D = np.maximum(A[i, j][:, None], A[i, j][None])
    for r, c in ((i, i), (i, j), (j, i), (j, j)):
        D = np.maximum(D, A[np.ix_(r, c)])
    keep = Q[:, None] * Q[None] * D >= dthr
    assert 0.02 < keep.mean() < 0.98
    kept = np.where(keep, eri, 0.0)
    pair = np.zeros((K, K), dtype=int)
    pair[i, j] = pair[j, i] = np.arange(len(i))
    T = kept[pair][:, :, pair]
    want = np.einsum("kl,ijkl->ij", P, T) - 0.5 * np.einsum("kl,ikjl->ij", P, T)
    c = native_driver.compile_driver(SCREENED, tmp_path / "screened")
    assert c.returncode == 0, c.stderr
    text = " ".join("%.17g" % x for x in np.concatenate([xyz.ravel(), P.ravel()]))
    out = native_driver.run_program(tmp_path / "screened", n, dthr, stdin=text)
    got = np.array([float(x) for x in out.split()]).reshape(K, K)
    assert np.abs(got - want).max() < 1e-11


def test_plan_of_more_than_64_launches():
    """The plan that the allocation-free build is tested with has that many."""
    with H.FockBuilder(config=W.nacl_scan(8)[3], basis_set="cc-pVTZ", precision=H.HFX_PREC_MIXED,
                       fp32_threshold=1e-2) as fb:
        assert 64 < len(fb.plan()) <= 256
