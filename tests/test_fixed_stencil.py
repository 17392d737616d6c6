"""The integers a face takes from its four cells (golikov_2d_gb300/csrc/gd_fixed.cuh): reconstructed
states and the fluxes between them against long double, with an outer cell up to 2^40 stronger or
weaker than the two beside the face, weak fields everywhere, and a slow transverse flow beside a
fast one.  A state is off by at most 2^-52 of the larger of its two cells, per component (the cells
are exact within 2^8 of each other, and one of binary64's own roundings is 2^-53); a flux by at most
2e-14 of its scale (the solvers keep 2^-57 of a face's units and lose at most 2^10 of them: three
exponents of room for the outer cells, squared in energies and field stresses)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def checked(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("stencil") / "check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-o", exe,
                    os.path.join(HERE, "fixed_stencil_check.cpp")], check=True)
    r = subprocess.run([exe, "20000"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    rows = [ln.split() for ln in r.stdout.splitlines()]
    return [(t[0], t[1], int(t[3]), int(t[5]), float(t[7]), float(t[9])) for t in rows]


@pytest.mark.parametrize("solver", ["hllc", "hll", "hlld", "hllc_mhd"])
def test_states_and_fluxes_of_a_stencil(checked, solver):
    rows = [r for r in checked if r[0] == solver]
    assert len(rows) == 10
    for _, name, taken, left, state, flux in rows:
        assert taken >= 0.98 * (taken + left), (solver, name, taken, left)
        assert state <= 2.0 ** -52, (solver, name, state)
        assert flux <= 2e-14, (solver, name, flux)
