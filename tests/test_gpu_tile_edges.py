"""The rate kernel and the tile-resident update at the edges of their tiling: one cell, a tile but one cell, a
tile and one cell, one tile more than the GPU has SMs (the kernels' second round, whose inputs the rate kernel
loads ahead) and one more than three per SM, against the oracle.

The properties at the edges of theirs (8 or 16 cells a block, by the field's size) and of the sub-mixture: more
than 32 species in it, one species alone, N2 alone.

The enthalpy relaxation at the edges of its blocks of steps (8, 4, 2 or 1 by the number of rows; a number of steps
that is or is not a multiple), bit for bit.

Tolerances as in test_gpu_parity.py: mu, lambda, D_k, cp 1e-11 relative, h 1e-10; RC and d(omega)/dY 1e-11 relative; QDSP 1e-11 of the gross rate; QDOT, a
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


@pytest.mark.parametrize("n", [1, 7, 9, 32 * 148, 32 * 148 + 1, 512 * 148 + 17])
def test_props_and_cp_h_at_tile_edges(cuda, oracle, n):
    tk, rho, y = random_state(oracle, n, 60 + n % 7)
    y = y.copy()
    m = len(range(0, n, 5))
    y[:, ::5] = np.random.default_rng(1).uniform(0.005, 0.03, (52, m))      # all 52 species in the sub-mixture
    y[:, 1::7] = 1e-12                                                      # one species alone
    y[12, 1::7] = 1.0 - 51e-12
    y[:, 2::7] = 0.0                                                        # N2 alone
    y[51, 2::7] = 1.0
    y /= y.sum(0)
    with cuda.UniChem(n) as u:
        u.upload(tk, rho, y)
        mu, lam, d = u.props()
        cp, h = u.cp_h()
        yc = u.download()[2]
    yo, mu_o, lam_o, d_o, nsub = oracle.props(tk, y)
    assert n < 6 or (nsub.max() > 32 and nsub.min() <= 2)
    assert np.array_equal(yc, yo)
    assert_rel(mu, mu_o, 1e-11, 0, "mu")
    assert_rel(lam, lam_o, 1e-11, 0, "lambda")
    assert_rel(d, d_o, 1e-11, 0, "D_k")
    assert_rel(cp, oracle.cp(tk, yo), 1e-11, 0, "cp")
    hm = oracle.enthalpy(tk, yo)[1]
    assert_rel(h, hm, 1e-10, 1e-12 * np.abs(hm).max(), "h")


@pytest.mark.parametrize("n", [1, 31, 512, 513])
def test_host_copies_on_both_sides_of_the_staged_size(cuda, oracle, n):
    """Fields of up to 512 cells pass through pinned staging rows. The caller's arrays may be overwritten as soon
    as upload returns, uploads may follow one another, and what comes back is what went in."""
    rng = np.random.default_rng(n)
    states = [(rng.uniform(1, 8, n), rng.uniform(0.1, 1, n), rng.uniform(0, 1, (52, n)), rng.uniform(0, 1e-3, n),
               rng.uniform(0, 1e12, n)) for _ in range(3)]
    with cuda.UniChem(n) as u:
        for st in states:
            work = [a.copy() for a in st]
            u.upload(*work)
            for a in work:
                a[...] = -1.0
        for a, b in zip(u.download(), states[-1]):
            assert np.array_equal(a, b)
        u.upload(*states[0][:3])                      # without soot: zeros
        got = u.download()
        assert np.array_equal(got[2], states[0][2]) and not got[3].any() and not got[4].any()
        with pytest.raises(cuda.UniChemError):
            u.download_outputs()                      # nothing computed yet
        tk, rho, y = random_state(oracle, n, 5)
        u.upload(tk, rho, y)
        om, (mu, lam, d) = u.omega(), u.props()
        cp, h = u.cp_h()
        o = u.download_outputs()
    for k, v in dict(qdsp=om.qdsp, qdot=om.qdot, domega_dy=om.domega_dy, vmu=mu, vtc=lam, vdf=d, cp=cp, h=h).items():
        assert np.array_equal(o[k], v), k


# interior rows for blocks of 8 (229 at most), 4 (458), 2 (916) and 1 step
@pytest.mark.parametrize("lj,li", [(3, 10), (3, 11), (10, 3), (231, 5), (232, 6), (460, 4), (461, 4), (918, 4), (919, 3)])
def test_relaxation_at_block_edges(cuda, oracle, lj, li):
    from test_gpu_enthalpy import oracle_coefficients
    g, o = oracle_coefficients(oracle, lj, li, 14)
    fo, po = oracle.enthalpy_relax(lj, li, g["rho"], o["rhsz"], o["z"], g["ht"], isor=5, tol=-1.0)
    fg, pg = cuda.enthalpy_relax(lj, li, g["rho"], o["rhsz"], o["z"], g["ht"], isor=5, tol=-1.0)
    assert pg == po
    assert np.array_equal(fg, fo)


@pytest.mark.parametrize("n", [1, 31, 33, 129, 257])
def test_surrogate_rows_do_not_depend_on_their_tile(cuda, n):
    """The network's rows at the edges of the feature kernel's 32 cells and of the layers' 128-row tiles: the same
    value bit for bit as in a field of 3,001 cells, where they stand in the middle (each row is its own sum)."""
    from unicorn_b200.fields import batch_cells, nondimensional
    from unicorn_b200.surrogate import Surrogate, raw_features
    f = batch_cells(3001, seed=7)

    def run(cells):
        with cuda.UniChem(len(cells)) as u:
            tk, rho = nondimensional(f, u.scales, u.wm)
            u.upload(tk[cells], rho[cells], np.ascontiguousarray(f.y[:, cells]))
            u.set_pressure(f.p[cells] / u.scales["PSTR"])
            if not s.ready:
                q = u.omega().qdsp
                s.net.set_norm(**Surrogate.norm_from_sample(raw_features(f.T, f.p / (u.scales["PBACK"] * u.scales["PSTR"]), f.y), q))
                s.ready = True
            s.net.omega(u, tol=float("inf"))
            out = {"qdsp": np.empty((52, len(cells)))}
            u.download_outputs(out)
        return out["qdsp"]

    class s:
        net, ready = Surrogate(capacity=4096, seed=3), False
    try:
        whole = run(np.arange(3001))
        first = 1000
        assert np.array_equal(run(np.arange(first, first + n)), whole[:, first:first + n])
    finally:
        s.net.close()
