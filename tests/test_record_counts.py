"""Shells of one centre that share exponents, with coefficients that are zero
or cancel: the FP32 tasks of a mixed-precision plan are tiles of the shell-pair
records, so both have to hold the same primitive pairs.

The basis is a general contraction as published tables print it: every column
over all exponents, with zeros where a column does not use one."""
import numpy as np
import pytest

import native_driver
import oracle as O
import hartree_fock_cpp_gb300 as H
from hartree_fock_cpp_gb300 import workloads as W

EXPS = (30.0, 5.5, 1.3, 0.35)
SETS = {
    # two s columns and an s primitive with zeros, two p columns with zeros, d
    "zeros": [("S", EXPS, (0.1, 0.4, 0.5, 0.0)), ("S", EXPS, (-0.02, -0.1, 0.0, 0.9)), ("S", EXPS, (0.0, 0.0, 0.0, 1.0)),
              ("P", EXPS[1:], (0.3, 0.0, 0.8)), ("P", EXPS[1:], (0.0, 0.6, 0.0)), ("D", (0.8,), (1.0,))],
    # products of the two orders that cancel: c_i d_j + c_j d_i = 0
    "cancel": [("S", EXPS[1:], (0.5, 0.5, 0.5)), ("S", EXPS[1:], (0.5, -0.5, 0.5)), ("P", EXPS[1:], (0.4, 0.4, 0.4)),
               ("P", EXPS[1:], (0.4, 0.4, -0.4))],
    # one column with a single coefficient left, one of zeros next to a full one
    "bare": [("S", EXPS, (0.0, 0.0, 1.0, 0.0)), ("S", EXPS, (0.2, 0.3, 0.4, 0.5)), ("P", EXPS[2:], (1.0, 0.0)),
             ("P", EXPS[2:], (0.0, 1.0))],
}
CONFIG = [("C", (0.0, 0.0, 0.0)), ("C", (0.3, -0.2, 2.4)), ("C", (1.9, 1.1, -0.7))]


def _write(tmp_path, name):
    d = tmp_path / name
    d.mkdir()
    rows = ["shell_id,L,primitive_id,exponent,coefficient"]
    for s, (L, ex, co) in enumerate(SETS[name]):
        rows += ["%d,%s,%d,%r,%r" % (s, L, k, e, c) for k, (e, c) in enumerate(zip(ex, co))]
    (d / "C.csv").write_text("\n".join(rows) + "\n")
    return str(tmp_path)


DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include "hfx_engine.hpp"
int main(int argc, char** argv)
{
    std::vector<const char*> sym;
    std::vector<double> xyz;
    for (int a = 3; a + 3 < argc; a += 4) {
        sym.push_back(argv[a]);
        for (int k = 1; k < 4; ++k) xyz.push_back(std::atof(argv[a + k]));
    }
    hfx_molecule m{(int)sym.size(), sym.data(), xyz.data(), argv[2], argv[1][0] ? argv[1] : nullptr};
    const hfx::Basis b = hfx::build_basis(m);
    const hfx::Fragments fr = hfx::single_fragment(b);
    const hfx::SuperData sd = hfx::build_super_data(b, fr);
    const hfx::PairData pd = hfx::build_pair_data(b, fr);
    std::vector<int> plan(pd.hpairs.size(), -1);
    for (size_t p = 0; p < sd.pairs.size(); ++p)
        for (size_t k = 0; k < sd.members[p].size(); ++k) plan[sd.members[p][k]] = sd.member_npp[p][k];
    for (size_t p = 0; p < pd.hpairs.size(); ++p) std::printf("%d %d %d\n", plan[p], pd.hpairs[p].npp, pd.dpairs[p].npp);
}
"""


def _counts(tmp_path, config, basis, path=""):
    args = [path, basis]
    for s, r in config:
        args += [s] + ["%.17g" % x for x in r]
    out = native_driver.run_driver(DRIVER, tmp_path / "counts", *args)
    return np.array([[int(x) for x in line.split()] for line in out.splitlines()])


@pytest.mark.parametrize("name", list(SETS))
def test_plan_counts_equal_record_counts(tmp_path, name):
    c = _counts(tmp_path, CONFIG, name, _write(tmp_path, name))
    assert len(c) == len(SETS[name]) * 3 * (len(SETS[name]) * 3 + 1) // 2
    assert (c[:, 0] == c[:, 1]).all(), c[c[:, 0] != c[:, 1]]
    assert (c[:, 1] == c[:, 2]).all()


@pytest.mark.parametrize("config,basis", [(W.water(), "cc-pVTZ"), (W.benzene(), "cc-pVDZ"), (W.n_decane(), "6-31G*"),
                                          (W.nacl_scan(8)[3], "cc-pVTZ")], ids=["water", "benzene", "decane", "nacl"])
def test_plan_counts_equal_record_counts_of_the_bundled_sets(tmp_path, config, basis):
    c = _counts(tmp_path, config, basis)
    assert (c[:, 0] == c[:, 1]).all()


# Tolerance: the FP32 quartets are those below tau = 0.03, each integral within
# 1e-6 of its bound (24-bit products summed over at most 100 primitive quartets
# of one sign or of mixed signs no larger than the bound's factors); an element
# of G sums at most 8 K^2 of them with |D| <= 2 / K: 0.03 * 1e-6 * 16 K = 1.7e-5
# at K = 36, and 1e-11 in FP64.
@pytest.mark.gpu
@pytest.mark.parametrize("name", list(SETS))
def test_mixed_build_of_a_general_contraction_matches_oracle(tmp_path, name):
    path = _write(tmp_path, name)
    orc = O.Oracle(CONFIG, name, basis_path=path, stable_boys=True)
    eri = orc.repulsion_tensor_mt(1e-8)
    K = orc.K
    rng = np.random.default_rng(11)
    Pa, Pb = [(P + P.T) / K for P in rng.uniform(-1.0, 1.0, size=(2, K, K))]
    b = H.basis_construction(CONFIG, name, path)
    want = [O.repulsion_matrix(Pa, eri), O.coulomb_matrix(Pa, Pb, eri), O.exchange_matrix(Pa, eri),
            O.exchange_matrix(Pb, eri)]
    for precision, tol in ((H.HFX_PREC_FP64, 1e-11), (H.HFX_PREC_MIXED, 0.03 * 1e-6 * 16 * K)):
        with H.FockBuilder(b, precision=precision, fp32_threshold=0.03) as fb:
            for _ in range(2):          # the eager build, then the graph
                got = [fb.repulsion_matrix(Pa)] + list(fb.coulomb_exchange(Pa, Pb))
                for g, w in zip(got, want):
                    assert np.abs(g - w).max() < tol
            s = fb.stats()
        assert (s["quartets_fp32"] > 0) == (precision == H.HFX_PREC_MIXED)
