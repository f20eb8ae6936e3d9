"""The library's count of the bytes it copies between host and device, which the
benchmark reports per solve."""
import ctypes

import numpy as np
import pytest

import hartree_fock_cpp_gb300 as H
from hartree_fock_cpp_gb300 import _lib, workloads as W

pytestmark = pytest.mark.gpu


def _copied():
    h, d = ctypes.c_double(), ctypes.c_double()
    _lib.check(_lib.lib.hfx_debug_copied_bytes(ctypes.byref(h), ctypes.byref(d)))
    return np.array([h.value, d.value])


def test_copied_bytes_of_builds_from_host_and_device_memory():
    torch = pytest.importorskip("torch")
    with H.FockBuilder(config=W.water(), basis_set="6-31G*") as fb:
        n = 8 * fb.K ** 2
        P = np.eye(fb.K)
        for _ in range(2):          # the eager build, then the graph
            a = _copied()
            fb.repulsion_matrix(P)
            assert (_copied() - a).tolist() == [n, n]
            a = _copied()
            fb.coulomb_exchange(P, P)
            assert (_copied() - a).tolist() == [2 * n, 3 * n]
        dP = torch.from_numpy(P).cuda()
        G = torch.empty_like(dP)
        torch.cuda.synchronize()
        a = _copied()
        fb.repulsion_matrix_device(dP.data_ptr(), G.data_ptr())
        assert (_copied() - a).tolist() == [0, 0]


def test_a_solve_moves_its_tables_once_and_scalars_per_iteration():
    """Beside the job's tables (the same for any number of iterations) a solve
    reads back a few hundred bytes per iteration."""
    moved = []
    for it in (6, 9):
        a = _copied()
        r = H.rhf_diis(W.water(), "cc-pVDZ", epsilon=1e-12, max_it=it)
        assert r["iterations"] == it
        moved.append(_copied() - a)
    (h0, d0), (h1, d1) = moved
    assert h0 == h1 > 0 and 0 < d1 - d0 < 3 * 2048
