"""The server's admission estimate against the device memory that a job takes:
a job within its reservation cannot push the others past the budget."""
import threading
import time

import numpy as np
import pytest

import hartree_fock_cpp_gb300 as H
from hartree_fock_cpp_gb300 import workloads as W
from hartree_fock_cpp_gb300.server import Server

pytestmark = pytest.mark.gpu


def _tree(n):
    rng, m = np.random.default_rng(1000 + n), None
    while m is None:
        m = W.random_molecule(rng, n)
    return m


@pytest.mark.parametrize("n,basis,pack_max", [(24, "cc-pVDZ", 0), (7, "cc-pVDZ", 4), (24, "STO-3G", 0)])
def test_a_mixed_job_stays_within_its_reservation(n, basis, pack_max):
    torch = pytest.importorskip("torch")
    free = lambda: torch.cuda.mem_get_info()[0]  # noqa: E731
    mol = _tree(n)
    ne = W.n_electrons(mol)
    with Server(max_active=1, pack_max=pack_max, precision=H.HFX_PREC_MIXED, fp32_threshold=0.03) as srv:
        srv.submit(W.water(), "STO-3G")      # the context's and the libraries' own memory
        srv.drain(60)
        before, least, reserved, stop = free(), [free()], [0.0], threading.Event()

        def watch():
            while not stop.is_set():
                reserved[0] = max(reserved[0], srv.stats()["in_use_bytes"])
                least[0] = min(least[0], free())
                time.sleep(0.002)

        t = threading.Thread(target=watch)
        t.start()
        jid = srv.submit(mol, basis, method="UHF", spin=(ne // 2 + 1, ne - ne // 2 - 1), max_it=3)
        info = srv.wait(jid, 300)
        stop.set()
        t.join()
    assert info["state"] in ("done", "failed") and "footprint" not in info["message"], info
    assert info["iterations"] == 3, info
    assert 0 < before - least[0] <= reserved[0]
