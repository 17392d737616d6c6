"""Where the fast step changes route.  A tile whose densities and pressures (and squared fields)
each span less than a fixed number of binades runs its faces in scaled 64-bit integers, any
other tile in FP64, and a face whose fan leaves the integers' range is redone in FP64: one step
from states on both sides of those lines, at tile edges and remainders, in ordinary and extreme
units, against the oracle, with the fast step's bound of 1e-12 (relative L1, every conserved
field).  The frozen sphere's test in FP32 with the exact one in the shell its error leaves open:
frozen cells stay bit for bit and all others change, also where a cell lies exactly on the
sphere and where FP32 cannot tell the cells apart.  Batches whose grids all use one Euler solver
take a kernel of their own: they agree bit for bit with mixed batches and single grids."""
import numpy as np
import pytest

import golikov_2d_gb300 as g
from golikov_2d_gb300 import problems
from gpu_util import gpu_run, gpu_step_ref, grid_of, max_rel_l1
from test_gpu_batch import run_batch, small_batch

pytestmark = pytest.mark.gpu

PER_STEP_TOL = 1e-12
METHODS = {"hllc": (g.EULER, g.METHOD_HLLC), "hll": (g.EULER, g.METHOD_HLL),
           "hlld": (g.MHD, g.METHOD_HLLD), "hllc_mhd": (g.MHD, g.METHOD_HLLC_MHD)}
# density unit, pressure unit
UNITS = {"unit": (1.0, 1.0), "tiny": (1e-9, 1e-9), "cold": (1e6, 1e-6), "hot": (1e-20, 1e20)}


def config(physics, method, N, M):
    make = problems.orszag_tang if physics == g.MHD else problems.kelvin_helmholtz
    cfg = make(N, M)[0]
    cfg.method = method
    return cfg


def state(physics, K, span, units, velocity, seed):
    """Densities and pressures 2^(span U[0, 1]), velocities of about the speed of sound."""
    rng = np.random.default_rng(seed)
    r0, p0 = units
    s = np.stack([r0 * 2.0 ** rng.uniform(0, span, K), p0 * 2.0 ** rng.uniform(0, span, K)], 1)
    u = velocity * (p0 / r0) ** 0.5 * rng.uniform(-0.5, 0.5, (K, 2))
    b = (4 * np.pi * p0) ** 0.5 * rng.uniform(-1, 1, (K, 3)) if physics == g.MHD else None
    return s, u, b


@pytest.mark.parametrize("N,M", [(3, 3), (33, 12), (70, 25)])
@pytest.mark.parametrize("units", UNITS)
@pytest.mark.parametrize("solver", METHODS)
def test_step_on_both_sides_of_the_integer_range(cuda, oracle_lib, solver, units, N, M):
    physics, method = METHODS[solver]
    for span in (0.0, 3.0, 7.9, 8.1, 16.0):
        for order, velocity in ((2, 1.0), (2, 0.0), (1, 1.0)):
            cfg = config(physics, method, N, M)
            cfg.order = order
            s, u, b = state(physics, N * M, span, UNITS[units], velocity, 100 * N + int(10 * span))
            # a hundredth of a cell per unit of the fastest signal there can be
            fast = np.sqrt(20 * UNITS[units][1] * 2.0 ** span / UNITS[units][0])
            T = 1e-2 * min(cfg.dx, cfg.dy) / fast
            so, uo, bo, To = oracle_lib.step(grid_of(cfg), s, u, b, T)
            sg, ug, bg, Tg = gpu_step_ref(cfg, s, u, b, T)
            err = max_rel_l1(cfg, (sg, ug, bg), (so, uo, bo))
            assert err <= PER_STEP_TOL, (span, order, velocity, err)
            assert abs(Tg - To) <= 1e-12 * To, (span, order, velocity)


@pytest.mark.parametrize("span", [3.0, 7.9, 8.1, 16.0])
@pytest.mark.parametrize("N,M", [(37, 9), (100, 70)])
def test_hancock_step_on_both_sides_of_the_integer_range(cuda, N, M, span):
    s, u, b = state(g.MHD, N * M, span, (1.0, 1.0), 1.0, 7 * N + int(10 * span))
    b[:, 2] = 0.0
    par, fast = (problems.hancock_config(N, M, 9.0, 5.0, scheme=g.SCHEME_HANCOCK, mode=m)
                 for m in (g.MODE_PARITY, g.MODE_FAST))
    T = 2e-3 / 2.0 ** (span / 2)
    p, f = gpu_step_ref(par, s, u, b, T), gpu_step_ref(fast, s, u, b, T)
    assert max_rel_l1(par, f[:3], p[:3]) <= PER_STEP_TOL
    assert abs(f[3] - p[3]) <= PER_STEP_TOL * p[3]


# x0, y0, radius on a 70 x 53 grid of cells 1 / 64 apart
SPHERES = {"corner": (0.0, 0.0, 0.5), "on_cells": (0.0, 0.0, 25 / 64), "centre": (-0.5, -0.375, 0.25),
           "beyond_fp32": (-2.0 ** 20, 0.0, 2.0 ** 20 - 0.5), "all": (0.0, 0.0, 8.0),
           "none": (4.0, 4.0, 2.0)}


@pytest.mark.parametrize("sphere", SPHERES)
@pytest.mark.parametrize("solver", ["hllc", "hlld"])
def test_frozen_cells_are_exact(cuda, solver, sphere):
    physics, method = METHODS[solver]
    N, M, h = 70, 53, 1 / 64
    cfg = config(physics, method, N, M)
    cfg.dx = cfg.dy = h
    cfg.x0, cfg.y0, cfg.frozen_radius = SPHERES[sphere]
    s, u, b = state(physics, N * M, 3.0, (1.0, 1.0), 1.0, 11)
    s2, u2, b2, _ = gpu_step_ref(cfg, s, u, b, 1e-4)
    X, Y = np.meshgrid(cfg.x0 + np.arange(N) * h, cfg.y0 + np.arange(M) * h)  # exact
    frozen = (np.sqrt(X * X + Y * Y) < cfg.frozen_radius).ravel()
    assert np.array_equal((s2 == s).all(axis=1), frozen)
    assert np.array_equal(u2[frozen], u[frozen])
    assert b is None or np.array_equal(b2[frozen], b[frozen])


def test_one_solver_batches_equal_mixed_ones_and_single_grids(cuda):
    # batch_four_quadrant's grids, each of the two solvers for the same grids
    def grids(methods):
        out = small_batch(8)
        for (c, *_), m in zip(out, methods):
            c.method = m
        return out

    C, H = g.METHOD_HLLC, g.METHOD_HLL
    runs = {k: run_batch(grids(m), 12)[0]
            for k, m in (("hllc", [C] * 8), ("hll", [H] * 8), ("mixed", [C, H] * 4))}
    for k in range(8):
        one = runs["hll" if k % 2 else "hllc"][k]
        mix = runs["mixed"][k]
        assert np.array_equal(one[0], mix[0]) and np.array_equal(one[1], mix[1]), k
        assert one[2].t == mix[2].t and one[2].dt == mix[2].dt, k
    cfg, s, u, _ = grids([C, H] * 4)[1]
    out = gpu_run(cfg, s, u, None, 12)
    assert np.array_equal(out[0], runs["mixed"][1][0])
    assert np.array_equal(out[1], runs["mixed"][1][1])


def test_threads_of_a_tile_change_no_result(cuda):
    """A batch runs its tiles with 192 threads, a single grid with 576 up to 152 tiles and with
    256 beyond: the same bits on both sides of that line."""
    grids = problems.batch_four_quadrant(8, lo=150, hi=250, seed=9)
    tiles = [-(-c.N // 16) * -(-c.M // 16) for c, *_ in grids]
    assert min(tiles) <= 152 < max(tiles)
    batch, _ = run_batch(grids, 5)
    for (cfg, s, u, b), (s2, u2, st) in zip(grids, batch):
        ss, us, _, sst = gpu_run(cfg, s, u, b, 5)
        assert np.array_equal(ss, s2) and np.array_equal(us, u2)
        assert sst.t == st.t and sst.dt == st.dt


@pytest.mark.parametrize("N,M", [(320, 165), (320, 176)])
@pytest.mark.parametrize("solver", ["hlld", "hllc_mhd"])
def test_mhd_step_on_both_sides_of_152_tiles(cuda, oracle_lib, solver, N, M):
    """768 threads per tile up to 152 tiles of 32 x 11, 384 beyond (150 and 160 tiles here)."""
    physics, method = METHODS[solver]
    cfg = config(physics, method, N, M)
    s, u, b = state(physics, N * M, 3.0, (1.0, 1.0), 1.0, 17)
    so, uo, bo, To = oracle_lib.step(grid_of(cfg), s, u, b, 1e-4)
    sg, ug, bg, Tg = gpu_step_ref(cfg, s, u, b, 1e-4)
    assert max_rel_l1(cfg, (sg, ug, bg), (so, uo, bo)) <= PER_STEP_TOL
    assert abs(Tg - To) <= 1e-12 * To
