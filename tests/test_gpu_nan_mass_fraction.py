"""A NaN mass fraction shows in the transport properties of its cell and of no other: the reference leaves a
species out of the sub-mixture where Y < 1e-3 (src/unicornd-mild-sd-5.f:842-915), which a NaN is not. Every
species of the cell then depends on it: mu, lambda and all D_k are NaN. Both block sizes of the kernel (8 cells
up to 32 cells per SM, 16 above), a species in each half of the list and a trace species."""
import numpy as np
import pytest

from conftest import random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [257, 32 * 148 + 1])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_nan_mass_fraction_shows_in_its_cell(oracle, n, precision):
    from unicorn_b200 import unichem
    tk, rho, y = random_state(oracle, n, 7)
    bad = {3: 1, 100: 46, 255: 30}                # cell: species (a major, one of the second half, a trace)
    yn = y.copy()
    for c, k in bad.items():
        yn[k, c] = np.nan
    got = []
    for state in (y, yn):
        with unichem.UniChem(n) as u:
            u.upload(tk, rho, state)
            if precision == "fp64":
                got.append(u.props())
            else:
                u.chem_props(unichem.MIXED)
                o = u.download_outputs()
                got.append((o["vmu"], o["vtc"], o["vdf"]))
    clean, nan = got
    cells = np.array(list(bad))
    others = np.setdiff1d(np.arange(n), cells)
    for a, b in zip(clean, nan):
        assert np.isfinite(a).all()
        assert np.isnan(b[..., cells]).all()
        assert np.array_equal(b[..., others], a[..., others])
