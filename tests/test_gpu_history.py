"""DIIS histories longer than the default eight on the device: the new row of the
error matrix and the extrapolated Fock matrix over all of them.  The host
driver runs the same loop on the oracle's integrals."""
import ctypes

import numpy as np
import pytest

from hartree_fock_cpp_gb300 import _lib
from hartree_fock_cpp_gb300 import workloads as W
from test_host import _run_rhf_driver

pytestmark = pytest.mark.gpu

KW = dict(epsilon=1e-7, max_iterations=100)


def _options(**kw):
    o = _lib.ScfOptions()
    for k, v in kw.items():
        setattr(o, k, v)
    return o


@pytest.mark.parametrize("history", [4, 8, 9, 16, 17])
def test_rhf_history_matches_the_host_driver(history):
    cfg = W.water()     # 19 to 31 iterations, so that every history fills
    kw = dict(KW, max_history=history)
    st, want, dens = _run_rhf_driver(cfg, "6-31G", **kw)
    m, r = _lib.MoleculeArgs(cfg, "6-31G"), _lib.ScfResult()
    P = np.zeros_like(dens)
    got = _lib.lib.hfx_rhf_diis(m.ref(), ctypes.byref(_options(**kw)), None, ctypes.byref(r), _lib.ptr(P), None, None)
    assert st == got == 0 and r.converged
    assert abs(r.iterations - want.iterations) <= 1 and r.iterations > history
    assert abs(r.E_tot - want.E_tot) < 1e-8
    assert np.abs(P - dens).max() < 1e-6


@pytest.mark.parametrize("history", [9, 16])
def test_uhf_history_reaches_the_default_one_s_energy(history):
    cfg = [("N", (0.0, 0.0, 0.0)), ("H", (0.0, 0.0, 2.3)), ("H", (0.0, 2.2, -0.6))]
    m, E, its = _lib.MoleculeArgs(cfg, "6-31G"), [], []
    for h in (0, history):
        r = _lib.ScfResult()
        st = _lib.lib.hfx_uhf_diis(m.ref(), ctypes.byref(_options(**dict(KW, max_history=h))), 5, 4, None, None,
                                   ctypes.byref(r), None, None, None, None)
        assert st == 0 and r.converged
        E.append(r.E_tot)
        its.append(r.iterations)
    assert its[1] > history and abs(E[1] - E[0]) < 1e-8
