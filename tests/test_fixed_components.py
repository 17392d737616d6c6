"""Small components beside large ones in the integer face solvers: an out-of-plane field, transverse
velocity and field, a transverse velocity alone, the normal field, or both fields of the plane beside a
strong one out of it, 1 to 2^-100 of the others.  Each component is held to 2e-15 of its own scale, against long double: a dozen roundings of
2^-53 each, of the face's states, its fan and the components' products, as binary64 makes them."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
TOL = 2e-15


@pytest.fixture(scope="module")
def checked(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("components") / "check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-o", exe,
                    os.path.join(HERE, "fixed_components_check.cpp")], check=True)
    r = subprocess.run([exe, "10000"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    rows = [ln.split() for ln in r.stdout.splitlines()]
    return [(t[0], t[1], int(t[2]), int(t[4]), int(t[6]), float(t[8])) for t in rows]


@pytest.mark.parametrize("solver,rows", [("hllc", 24), ("hll", 24), ("hlld", 54), ("hllc_mhd", 54)])
def test_small_components_keep_their_digits(checked, solver, rows):
    got = [r for r in checked if r[0] == solver]
    assert len(got) == rows
    for _, name, k, taken, left, worst in got:
        assert taken >= 0.99 * (taken + left), (solver, name, k, taken, left)
        assert worst <= TOL, (solver, name, k, worst)
