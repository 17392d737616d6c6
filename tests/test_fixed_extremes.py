"""The integer face solvers at the ends of the range they accept (densities and pressures of 2^-127
and 2^126, velocities and fields from the order of the speed of sound down to subnormal numbers),
with the device's own bit arithmetic compiled for the host, against long double.  A face is either
left to the floating-point solver or every flux component is finite and within 1e-12 of its scale
(the face bound of the fast step)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
TOL = 1e-12


@pytest.mark.parametrize("solver", ["hllc", "hll", "hlld", "hllc_mhd"])
def test_faces_at_the_ends_of_the_range(extremes, solver):
    rows = extremes[solver]
    assert len(rows) == 10
    for name, (taken, left, worst) in rows.items():
        assert worst <= TOL, (solver, name, taken, left, worst)
    for name in ("low_end", "high_end", "cold", "hot"):
        taken, left, _ = rows[name]
        assert taken >= 0.9 * (taken + left), (solver, name, taken, left)


@pytest.fixture(scope="module")
def extremes(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("extremes") / "check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-o", exe,
                    os.path.join(HERE, "fixed_extremes_check.cpp")], check=True)
    r = subprocess.run([exe, "20000"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    out = {}
    for ln in r.stdout.splitlines():
        t = ln.split()
        out.setdefault(t[0], {})[t[1]] = (int(t[3]), int(t[5]), float(t[7]))
    return out
