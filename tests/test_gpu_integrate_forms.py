"""The two forms of the batched integration, the persistent kernel (16 and 8 warps) and the rounds form, run the same
arithmetic on a cell, in the same order and with every contraction written out: they agree bit for bit, soot and pass
counts included, whatever the tile a cell shares."""
import numpy as np
import pytest

from unicorn_b200.fields import batch_cells, nondimensional

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 1777])
def test_forms_agree_bit_for_bit(oracle, n, monkeypatch):
    from unicorn_b200 import unichem
    f = batch_cells(n, seed=21)
    tk, rho = nondimensional(f, oracle.scales, oracle.wm)
    rng = np.random.default_rng(n)
    stmf, stnd = rng.uniform(0, 1e-4, n), rng.uniform(0, 1e12, n)
    stmf[::3] = stnd[::3] = 0.0
    out = []
    for shape in (16, 8, 3):
        monkeypatch.setenv("UNICHEM_INT_WARPS", str(shape))
        with unichem.UniChem(n) as u:
            assert u.stat("int_warps") == shape
            u.upload(tk, rho, f.y, stmf, stnd)
            u.set_pressure(f.p / oracle.scales["PSTR"])
            u.integrate(1e-3)
            state = u.download()
            out.append((*state, *u.integrate_counts()))
    assert out[0][5].max() > 1
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert np.array_equal(a, b)
