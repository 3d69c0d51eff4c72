"""The mechanism's data against what the rate kernel's prepared tables hold (unicorn_b200/csrc/rate_limits.h): the
data as it is compiles, and data beyond each limit ends the build (it used to be cut off in silence, or to run
over a table)."""
import copy
import json
import shutil
import subprocess
from pathlib import Path

import pytest

from unicorn_b200.mech import codegen

CSRC = Path(__file__).resolve().parents[1] / "unicorn_b200" / "csrc"


def compiles(tables: str, tmp_path) -> tuple[bool, str]:
    (tmp_path / "generated").mkdir()
    (tmp_path / "generated" / "mech_tables.h").write_text(tables)
    shutil.copy(CSRC / "rate_limits.h", tmp_path)
    (tmp_path / "t.cpp").write_text('#include "rate_limits.h"\n')
    r = subprocess.run(["g++", "-std=c++17", "-fsyntax-only", str(tmp_path / "t.cpp")], capture_output=True, text=True)
    return r.returncode == 0, r.stderr


def first(d, cond):
    return next(k for k, v in d.items() if cond(v))


def more_fall_off(m):
    plain = [r for r in m["reactions"][::2] if r["akf"] > 0]
    for r in plain[:4]:
        r["akf"], r["aklow"] = -r["akf"], 1.0e16


def short_constant(m):
    m["reverse"][first(m["reverse"], lambda v: len(v["q"]) == 3)]["q"].pop()


def long_constant(m):
    q = m["reverse"][first(m["reverse"], lambda v: len(v["q"]) == 5)]["q"]
    q += [q[-1], q[-1]]


def two_mass_fractions(m):
    post = m["rc"][first(m["rc"], lambda v: any(p[1] == "Y" for p in v["post"]))]["post"]
    post.insert(0, list(post[0]))


def many_factors(m):
    post = m["rc"][first(m["rc"], lambda v: len(v["post"]) == 3)]["post"]
    post += [post[-1], post[-1]]


def test_the_data_fits(tmp_path):
    tables = codegen.gen_tables(json.loads(codegen.MECH.read_text()))
    assert tables == (CSRC / "generated" / "mech_tables.h").read_text()
    ok, err = compiles(tables, tmp_path)
    assert ok, err


@pytest.mark.parametrize("change, says", [
    (more_fall_off, "fall-off pairs"), (short_constant, "equilibrium constant"), (long_constant, "equilibrium constant"),
    (two_mass_fractions, "mass fraction"), (many_factors, "factors than its record")])
def test_data_beyond_a_limit_ends_the_build(change, says, tmp_path):
    mech = copy.deepcopy(json.loads(codegen.MECH.read_text()))
    change(mech)
    ok, err = compiles(codegen.gen_tables(mech), tmp_path)
    assert not ok and says in err, err
