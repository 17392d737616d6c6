"""The integer MHD face solvers at a mirror, where the contact stands on the face and the flux may jump
from one side's to the other's: the side below is taken, as where S_M >= 0 is asked of an exact 0, and
every component agrees with long double to 2e-15 of its scale (a dozen roundings of 2^-53)."""
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
    exe = str(tmp_path_factory.mktemp("mirror") / "check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-o", exe,
                    os.path.join(HERE, "fixed_mirror_check.cpp")], check=True)
    r = subprocess.run([exe, "100000"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    rows = [ln.split() for ln in r.stdout.splitlines()]
    return [(t[0], t[1], int(t[3]), int(t[5]), float(t[7])) for t in rows]


@pytest.mark.parametrize("solver", ["hlld", "hllc_mhd"])
def test_mirror_faces(checked, solver):
    got = [r for r in checked if r[0] == solver]
    assert len(got) == 5
    for _, name, taken, left, worst in got:
        assert taken >= 0.99 * (taken + left), (solver, name, taken, left)
        assert worst <= TOL, (solver, name, worst)
