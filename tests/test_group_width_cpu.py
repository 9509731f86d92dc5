"""A group of more lanes than a warp has may meet at a barrier, but not sum or
broadcast by shuffles: such a call does not compile."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _compiles(stmt):
    src = f'#include "deb_core.cuh"\nvoid f() {{ deb::Grp<128> g{{0}}; double a = 0, b = 0, c = 0; int i = 0; bool t = false; {stmt}; }}\n'
    r = subprocess.run(["g++", "-std=c++17", "-fsyntax-only", "-I", os.path.join(ROOT, "include"), "-I",
                        os.path.join(ROOT, "disco-eb_gb300", "csrc"), "-x", "c++", "-"], input=src, capture_output=True, text=True)
    return r.returncode == 0, r.stderr


def test_barrier_and_lead_of_a_block():
    ok, err = _compiles("g.sync(); t = g.lead()")
    assert ok, err


@pytest.mark.parametrize("stmt", ["a = g.sum(a)", "g.sum2(a, b)", "g.sum3(a, b, c)", "a = g.bcast(a, 0)", "t = g.any(t)",
                                  "g.argmax(a, i)"])
def test_shuffles_beyond_a_warp_are_refused(stmt):
    ok, err = _compiles(stmt)
    assert not ok and "shuffles reach one warp" in err
