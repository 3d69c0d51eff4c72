"""The rate kernel and the tile-resident update at the edges of their tiling: one cell, a tile but one cell, a
tile and one cell, one tile more than the GPU has SMs (the kernels' second round, whose inputs the rate kernel
loads ahead) and one more than three per SM, against the oracle.

Tolerances as in test_gpu_parity.py: RC and d(omega)/dY 1e-11 relative; QDSP 1e-11 of the gross rate; QDOT, a
sum of 52 products QDSP_k h_k, 1e-11 of the sum of the gross rates times |h_k|; Y after the update 1e-9."""
import numpy as np
import pytest

from conftest import random_state
from test_gpu_parity import assert_rel, gross

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("a GPU test ran without a CUDA device")
    from unicorn_b200 import unichem
    return unichem


@pytest.mark.parametrize("n", [1, 31, 33, 148 * 32 + 1, 3 * 148 * 32 + 5])
def test_rates_and_update_at_tile_edges(cuda, oracle, n):
    tk, rho, y = random_state(oracle, n, 40 + n % 7)
    # every 5th cell without hydrogen and oxygen atoms: zero mass fractions in the factored-out sums
    y[2, ::5] = y[3, ::5] = 0.0
    with cuda.UniChem(n) as u:
        u.upload(tk, rho, y)
        om = u.omega()
        rc_g = u.ckrates(return_rc=True)
        passes = u.solvesp(1e-3, isor=2, relx=0.99, tol=0.0)
        yg = u.download()[2]
    q, qd, h, d = oracle.omega(tk, rho, y)
    rc, sour = oracle.rates(tk, rho, y)
    assert_rel(rc_g, rc, 1e-11, 0.0, "RC")
    assert_rel(om.domega_dy, d, 1e-11, 0.0, "d(omega)/dY")
    g = gross(oracle, tk, rho, y)
    assert (np.abs(om.qdsp - q) <= 1e-11 * g).all()
    assert (np.abs(om.qdot - qd) <= 1e-11 * (g * np.abs(h)).sum(0)).all()
    yo, _, po = oracle.species_update(rho, y, rc, sour, 1e-3, isor=2, tol=0.0)
    assert passes == po
    assert_rel(yg, yo, 1e-9, 1e-18, "Y after two passes")
