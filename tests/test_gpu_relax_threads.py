"""The enthalpy relaxation on grids of different sizes from several host threads at once (one context per thread is
allowed; uc_enthalpy_relax takes its own buffers and stream): each call gives what it gives alone, bit for bit.
The rows decide the shared memory of the kernel (about 100 KB for 127 interior rows, 8 KB for 10), and what one
thread asks for may not take away what another is about to launch with."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_relax_grids_of_different_sizes(oracle):
    from test_gpu_enthalpy import oracle_coefficients
    from unicorn_b200 import unichem
    cases = []
    for lj, li in ((129, 4), (12, 4)):
        g, o = oracle_coefficients(oracle, lj, li, 17)
        call = lambda lj=lj, li=li, g=g, o=o: unichem.enthalpy_relax(lj, li, g["rho"], o["rhsz"], o["z"], g["ht"], isor=2,
                                                                  tol=-1.0)
        cases.append((call, call()))
    wrong, over = [], threading.Event()

    def loop(call, want, times):
        for i in range(times):
            if over.is_set():
                return
            try:
                f, p = call()
            except RuntimeError as e:
                wrong.append((i, str(e)))
                break
            if p != want[1] or not np.array_equal(f, want[0]):
                wrong.append((i, "another result"))
                break
        over.set()
    (large, small) = cases
    threads = [threading.Thread(target=loop, args=(*large, 1500))] + \
              [threading.Thread(target=loop, args=(*small, 10 ** 9)) for _ in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
