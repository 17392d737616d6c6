"""The face solvers in scaled 64-bit integers (golikov_2d_gb300/csrc/gd_fixed.cuh, gd_fixed_mhd.cuh:
HLLC, HLL, HLLD, HLLC-MHD) that the fast steps run where a tile's states share one binade range,
compiled for the host and checked against the same fluxes in long double: ordinary states, small
and tiny jumps (cancellation), slow and supersonic flow, strong jumps, units over e^+-40, strong
and weak fields, exact zeros and ties.  A flux component differs by at most 1e-12 of its scale,
the face bound of the fast step (the integers keep 2^-50 or less of a tile's unit, and a face's
jumps lose at most the 8 bits that its range may span).  The solver may leave a face to the
floating-point one; it must take nearly all ordinary ones."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
TOL = 1e-12


@pytest.fixture(scope="module")
def checked(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("fixed") / "fixed_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "fixed_check.cpp")],
                   check=True)
    r = subprocess.run([exe, "20000"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    rows = [ln.split() for ln in r.stdout.splitlines()]
    return {(t[0], t[1]): (int(t[3]), int(t[5]), float(t[7])) for t in rows}


@pytest.mark.parametrize("solver", ["hllc", "hll", "hlld", "hllc_mhd"])
def test_integer_faces_match_long_double(checked, solver):
    rows = {c: v for (s, c), v in checked.items() if s == solver}
    assert len(rows) == 9
    for name, (taken, left, worst) in rows.items():
        assert worst <= TOL, (solver, name, taken, left, worst)
        assert taken > 0, (solver, name)
    for name in ("ordinary", "small_jumps", "tiny_jumps", "slow"):
        taken, left, _ = rows[name]
        assert taken >= 0.98 * (taken + left), (solver, name, taken, left)
