"""The three-warp form of the species-update program (unicorn_b200/csrc/generated/update_program_co.cuh,
what the tile-resident kernels run) on the host, one thread per warp with the device's barriers
(tests/update_co_harness.cpp): it ends, every barrier is used in balance, and Y agrees with the two-array
program, which is the oracle's bit for bit.

Tolerance: only the order of additions and multiplications within a sum differs. A sum has at most 108
terms, all positive, each of at most four factors: both orders are within 112 roundings of the exact sum,
2.5e-14 apart at most; a species' quotient adds a few. The error of one species enters the next ones' sums
once or twice per term and is damped by the quotient (its own loss is in the denominator), so a pass adds
it up over the species at worst: 51 x 2.5e-14 = 1.3e-12 per pass, 4e-12 for three; 1e-11 is asserted."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from conftest import random_state

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("h")
    libs = []
    for src in ("update_program_harness.cpp", "update_co_harness.cpp"):
        so = d / (src + ".so")
        subprocess.run(["g++", "-O1", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared", "-pthread", "-o", str(so),
                        str(ROOT / "tests" / src)], check=True)
        libs.append(ctypes.CDLL(str(so)))
    return libs


@pytest.mark.parametrize("passes", [1, 3])
@pytest.mark.parametrize("soot", [False, True])
def test_three_warp_program_matches_two_array_program(oracle, harness, passes, soot):
    two, co = harness
    tk, rho, y = random_state(oracle, 40, 24)
    stmf, stnd = (np.full(40, 1e-3), np.full(40, 1e12)) if soot else (None, None)
    rc, sour = oracle.rates(tk, rho, y, stmf, stnd)
    assert not soot or (sour[2] > 0).all()
    P = lambda a: np.ascontiguousarray(a).ctypes.data_as(ctypes.POINTER(ctypes.c_double))
    y1, y2 = np.ascontiguousarray(y.copy()), np.ascontiguousarray(y.copy())
    D = ctypes.c_double
    two.harness_update(40, P(rho), P(y), P(y1), P(rc), P(sour), P(oracle.wm), D(1e-3), passes, D(0.99), D(0.0), D(1.0))
    assert co.harness_update_co(40, P(rho), P(y), P(y2), P(rc), P(sour), P(oracle.wm), D(1e-3), passes, D(0.99)) == 0
    assert np.abs(y1 - y).max() > 1e-8            # the update moved Y
    rel = np.abs(y2 - y1)[:51] / np.maximum(np.abs(y1[:51]), 1e-30)
    print(f"\nlargest relative difference {rel.max():.1e}")
    assert rel.max() <= 1e-11
