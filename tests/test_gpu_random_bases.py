"""FP64 and mixed builds and the unique integrals over random bases given as
functions: up to three centres, s to f shells that share exponents in any
order, with zero coefficients.  Oracle: the accurate-Boys restatement on the same
functions.

Tolerance: an element sums at most K^2 products |D| |(ij|kl)| with |D| <= 2 / K,
each integral within 1e-14 of the largest; an FP32 integral is within 1e-6 of
its bound, which is below tau and below the largest integral."""
import numpy as np
import pytest

import oracle as O
import hartree_fock_cpp_gb300 as H

pytestmark = pytest.mark.gpu


def _random_basis(seed):
    g = np.random.default_rng(seed)
    centres, lmn, off, alpha, coeff, norm = [], [], [0], [], [], []
    for _ in range(int(g.integers(1, 4))):
        R, pool = g.uniform(-2.5, 2.5, 3), np.exp(g.uniform(-1.5, 6.0, 6))
        for _ in range(int(g.integers(1, 6))):
            L = 0 if g.random() < 0.4 else int(g.integers(0, 4))
            n = int(g.integers(1, 4 if L < 2 else 3))
            if len(lmn) + (L + 1) * (L + 2) // 2 > 14:
                continue
            first = int(g.integers(0, len(pool) - n + 1))
            e = pool[first:first + n].copy()
            if g.random() < 0.3:
                e *= g.uniform(0.9, 1.1, n)
            if g.random() < 0.25:
                g.shuffle(e)
            c = g.uniform(-1.0, 1.0, n)
            c[g.random(n) < 0.2] = 0.0
            for l in O.angmom_partition(L):
                centres.append(R)
                lmn.append(l)
                alpha += list(e)
                coeff += list(c)
                norm += [O.cart_norm(x, *l) for x in e]
                off.append(len(alpha))
    return H.Basis(np.array(centres), np.array(lmn), np.array(off), np.array(alpha), np.array(coeff), np.array(norm))


def _oracle(b):
    orc = O.Oracle([("H", (0.0, 0.0, 0.0))], "STO-3G", stable_boys=True)
    fb = orc.fb
    fb.K = orc.K = b.K
    fb.cx, fb.cy, fb.cz = [np.ascontiguousarray(b.centres[:, k]) for k in range(3)]
    fb.lmn, fb.prim_off = np.ascontiguousarray(b.lmn.reshape(-1)), b.prim_offset
    fb.alpha, fb.coeff, fb.norm = b.alpha, b.coeff, b.norm
    arrays = (fb.cx, fb.cy, fb.cz, fb.lmn, fb.prim_off, fb.alpha, fb.coeff, fb.norm)
    orc._c = O._CBasis(fb.K, *[a.ctypes.data for a in arrays])
    return orc


@pytest.mark.parametrize("seed", range(10))
def test_random_basis_matches_oracle(seed):
    b = _random_basis(seed)
    orc = _oracle(b)
    K = b.K
    g = np.random.default_rng(seed + 100)
    Pa, Pb = [(P + P.T) / K for P in g.uniform(-1.0, 1.0, (2, K, K))]
    tau = 10.0 ** g.uniform(-4.0, 1.0)
    eri = orc.repulsion_tensor_mt(0.0)
    scale = np.abs(eri).max()
    want = [O.repulsion_matrix(Pa, eri), O.coulomb_matrix(Pa, Pb, eri), O.exchange_matrix(Pa, eri),
            O.exchange_matrix(Pb, eri)]
    for precision in (H.HFX_PREC_FP64, H.HFX_PREC_MIXED):
        tol = 4e-14 * scale * K + (4e-6 * min(tau, scale) * K if precision == H.HFX_PREC_MIXED else 0.0)
        with H.FockBuilder(b, screening_threshold=-1.0, precision=precision, fp32_threshold=tau) as fb:
            for _ in range(2):          # the eager build, then the graph
                for got, w in zip([fb.repulsion_matrix(Pa)] + list(fb.coulomb_exchange(Pa, Pb)), want):
                    assert np.abs(got - w).max() < tol
            assert np.abs(fb.eri_unique(-1.0) - eri).max() < 1e-14 * scale
