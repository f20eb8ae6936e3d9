"""The FP64 kernel over super shells at the sizes where it can go wrong: one
function, one primitive quartet per task, batches of several bra pairs, rows
split over tasks, general contractions, SP shells, f functions, the R tables
kept in registers and beyond, and no, usual and coarse screening.  Oracle: the
accurate-Boys restatement of the reference's tensor and contractions.

Tolerance: G, J and K are sums of at most K^2 products |D| |(ij|kl)| with
|D| <= 1 and |(ij|kl)| <= 5 here, each integral within 1e-14 of its size:
1e-11 on a matrix element, 1e-12 on an integral."""
import ctypes

import numpy as np
import pytest

import oracle as O
import hartree_fock_cpp_gb300 as H
from hartree_fock_cpp_gb300 import _lib
from hartree_fock_cpp_gb300 import workloads as W

pytestmark = pytest.mark.gpu

CASES = {
    "one_s": ([("H", (0.1, 0.2, 0.3))], "STO-3G"),
    "two_s": ([("H", (0.0, 0.0, 0.0)), ("H", (0.0, 0.0, 1.4))], "6-31G"),
    "far_pair": ([("He", (0.0, 0.0, 0.0)), ("He", (0.0, 0.0, 18.0))], "cc-pVDZ"),
    "sp": (W.water(), "STO-3G"),
    "sp_d": (W.water(), "6-31G*"),
    "general_contraction": ([("O", (0.0, 0.0, 0.0)), ("H", (0.0, 0.3, 1.8))], "cc-pVDZ"),
    "f": ([("C", (0.0, 0.0, 0.0))], "cc-pVTZ"),
}


def _densities(K, seed):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(2):
        P = rng.uniform(-1.0, 1.0, size=(K, K)) / K
        out.append(P + P.T)
    return out


@pytest.mark.parametrize("thr", [-1.0, 1e-8, 1e-3])
@pytest.mark.parametrize("name", list(CASES))
def test_super_shell_kernel_matches_oracle(name, thr):
    cfg, basis = CASES[name]
    orc = O.Oracle(cfg, basis, stable_boys=True)
    eri = orc.repulsion_tensor_mt(thr if thr >= 0 else 0.0)
    with H.FockBuilder(config=cfg, basis_set=basis, screening_threshold=thr) as fb:
        Pa, Pb = _densities(fb.K, 3)
        for _ in range(2):          # eager build, then the graph
            G = fb.repulsion_matrix(Pa)
            J, Ka, Kb = fb.coulomb_exchange(Pa, Pb)
        got = fb.eri_unique(thr)
    assert np.abs(got - eri).max() < 1e-12
    assert np.abs(G - O.repulsion_matrix(Pa, eri)).max() < 1e-11
    assert np.abs(J - O.coulomb_matrix(Pa, Pb, eri)).max() < 1e-11
    assert np.abs(Ka - O.exchange_matrix(Pa, eri)).max() < 1e-11
    assert np.abs(Kb - O.exchange_matrix(Pb, eri)).max() < 1e-11


def test_allocation_free_build_takes_a_mixed_plan_of_many_launches():
    """NaCl/cc-pVTZ mixed: FP64 launches of every angular momentum beside the
    FP32 classes, more than 64 in all."""
    torch = pytest.importorskip("torch")
    with H.FockBuilder(config=W.nacl_scan(8)[3], basis_set="cc-pVTZ", precision=H.HFX_PREC_MIXED,
                       fp32_threshold=1e-2) as fb:
        P = torch.from_numpy(_densities(fb.K, 7)[0]).cuda()
        want, got = torch.empty_like(P), torch.full_like(P, float("nan"))
        torch.cuda.synchronize()
        fb.repulsion_matrix_device(P.data_ptr(), want.data_ptr())
        _lib.check(_lib.lib.hfx_fock_rhf_device_noalloc(fb._job, ctypes.c_void_p(P.data_ptr()),
                                                        ctypes.c_void_p(got.data_ptr())))
        torch.cuda.synchronize()
    assert float((want - got).abs().max()) < 1e-11


def test_shells_given_as_functions_share_exponents_in_any_order():
    """A centre whose short contraction comes first, two shells with the same
    exponents, a repeated shell, and a second centre at the same point."""
    cfg, basis = CASES["general_contraction"]
    b = H.basis_construction(cfg, basis)
    K = len(b)
    first = [i for i in range(K) if i == 0 or tuple(b.centres[i]) != tuple(b.centres[i - 1]) or
             b.lmn[i].sum() != b.lmn[i - 1].sum() or (b.lmn[i] == [0, 0, b.lmn[i].sum()]).all()]
    shells = [list(range(s, e)) for s, e in zip(first, first[1:] + [K])]
    order = [f for s in reversed(shells) for f in s] + shells[0]
    seg = [slice(b.prim_offset[i], b.prim_offset[i + 1]) for i in order]
    off = np.cumsum([0] + [s.stop - s.start for s in seg])
    mixed = H.Basis(b.centres[order], b.lmn[order], off, *[np.concatenate([v[s] for s in seg])
                                                             for v in (b.alpha, b.coeff, b.norm)])
    Pa, _ = _densities(len(order), 5)
    back = np.zeros((K, K))
    np.add.at(back, (np.array(order)[:, None], np.array(order)[None]), Pa)
    with H.FockBuilder(mixed, screening_threshold=-1.0) as fm, H.FockBuilder(b, screening_threshold=-1.0) as fb:
        J = fm.coulomb_exchange(Pa, Pa)[0]
        want = fb.coulomb_exchange(back, back)[0][np.ix_(order, order)]
    assert np.abs(J - want).max() < 1e-11
