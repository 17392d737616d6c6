"""A face's arithmetic depends on its own cells alone.  Weak components beside strong ones in the
same tile keep their digits: the quiet side of a jump to 1e-12 of the quiet values themselves against
the oracle, a slow flow across a fast one to rounding.  States with faces out of the integers'
range come out with the same bits whatever tiles, thread counts and bands they are cut into."""
import numpy as np
import pytest

import golikov_2d_gb300 as g
from golikov_2d_gb300 import problems
from gpu_util import gpu_run, gpu_step_ref, grid_of
from test_gpu_batch import run_batch
from test_gpu_hoststep import pinned
from test_gpu_integer_tiles import METHODS, config

pytestmark = pytest.mark.gpu
TOL = 1e-12


@pytest.mark.parametrize("weak", [1e-3, 1e-8, 1e-12])
@pytest.mark.parametrize("solver", ["hlld", "hllc_mhd"])
def test_weak_field_beside_a_strong_one(cuda, oracle_lib, solver, weak):
    """Left half: field of order 1, right half: weak times that; uniform flow through both."""
    N, M = 100, 40
    cfg = config(*METHODS[solver], N, M)
    rng = np.random.default_rng(5)
    K = N * M
    s = np.stack([rng.uniform(1, 1.5, K), rng.uniform(3, 4, K)], 1)
    u = np.tile([0.4, 0.3], (K, 1)) + rng.uniform(-0.05, 0.05, (K, 2))
    b = rng.uniform(-1, 1, (K, 3))
    quiet = np.arange(K) % N >= N // 2 + 3
    b[np.arange(K) % N >= N // 2] *= weak
    T = 0.2 * cfg.dx / 4
    so, uo, bo, _ = oracle_lib.step(grid_of(cfg), s, u, b, T)
    sg, ug, bg, _ = gpu_step_ref(cfg, s, u, b, T)
    quiet &= np.arange(K) % N < N - 3  # the periodic edge is a jump too
    for k in range(3):
        assert np.abs(bg[quiet, k] - bo[quiet, k]).max() <= TOL * weak, k
        assert np.abs(bg[:, k] - bo[:, k]).max() <= TOL, k


@pytest.mark.parametrize("solver", ["hllc", "hll"])
def test_slow_cross_flow(cuda, solver):
    """A flow along x of order 1, uniform in y, that carries a velocity along y; in the right half
    1000 times weaker.  The carried velocity is a passive quantity: scaled by 2^-40 it is the same
    field to rounding (the kinetic energy that it adds at full strength stays in the pressure)."""
    N, M = 100, 40
    cfg = config(*METHODS[solver], N, M)
    rng = np.random.default_rng(6)
    s = np.stack([rng.uniform(1, 1.5, N), rng.uniform(3, 4, N)], 1)
    u = np.stack([rng.uniform(-0.5, 0.5, N), rng.uniform(-1, 1, N)], 1)
    u[N // 2:, 1] *= 1e-3
    s, u = np.tile(s, (M, 1)), np.tile(u, (M, 1))
    T = 0.2 * cfg.dx / 4
    full = gpu_step_ref(cfg, s, u, None, T)[1][:, 1]
    slow = gpu_step_ref(cfg, s, u * [1.0, 2.0 ** -40], None, T)[1][:, 1] * 2.0 ** 40
    col = np.arange(N * M) % N
    for part, unit in ((col < N // 2 - 3, 1.0), ((col >= N // 2 + 3) & (col < N - 3), 1e-3)):
        assert np.abs(slow[part] - full[part]).max() <= 4e-16 * unit


def jumpy(physics, K, seed):
    """Densities over 2^16, pressures over 2^12, velocities and fields over 2^40: a part of the
    faces in integers, a part in floating point."""
    rng = np.random.default_rng(seed)
    s = np.stack([2.0 ** rng.uniform(-4, 12, K), 2.0 ** rng.uniform(0, 12, K)], 1)
    u = rng.uniform(-0.05, 0.05, (K, 2)) * 2.0 ** rng.uniform(-40, 0, (K, 2))
    b = None
    if physics == g.MHD:
        b = rng.uniform(-1, 1, (K, 3)) * 2.0 ** rng.uniform(-40, 0, (K, 3))
    return s, u, b


@pytest.mark.parametrize("N,M", [(200, 140), (321, 177), (640, 400)])
@pytest.mark.parametrize("solver", METHODS)
def test_bands_of_the_host_step_change_no_bit(cuda, solver, N, M):
    """One launch, with the few-tiles kernel or without, and the host step's bands."""
    physics, method = METHODS[solver]
    cfg = config(physics, method, N, M)
    s, u, b = jumpy(physics, N * M, 3)
    T = 1e-3 * cfg.dx / 256
    one = gpu_run(cfg, s, u, b, 1, T_do=T)
    sol = g.Solver(cfg)
    sol.import_state(s, u, b)
    sol.set_time(T, 0.0)
    ins = [pinned(x) for x in (s, u, b)]
    outs = [None if x is None else pinned(np.zeros_like(x)) for x in (s, u, b)]
    sol.step_host(*ins, *outs)
    dt = sol.stats(allow_nonfinite=True).dt
    sol.close()
    for x, y in zip(one[:3], outs):
        assert (x is None and y is None) or np.array_equal(x, np.asarray(y))
    assert one[3].dt == dt


@pytest.mark.parametrize("solver", ["hllc", "hll"])
def test_tile_shapes_and_threads_change_no_bit(cuda, solver):
    """A batch in the tuner's shape, in the default one, and each grid by itself."""
    grids = problems.batch_four_quadrant(8, lo=100, hi=300, seed=12)
    out = []
    for cfg, s, u, _ in grids:
        cfg.method = METHODS[solver][1]
        s, u, _ = jumpy(g.EULER, cfg.N * cfg.M, cfg.N)
        out.append((cfg, s, u, None))
    a, ia = run_batch(out, 3)
    c, ic = run_batch(out, 3, autotune=True)
    for (cfg, s, u, _), x, y in zip(out, a, c):
        one = gpu_run(cfg, s, u, None, 3)
        assert np.array_equal(one[0], x[0]) and np.array_equal(one[1], x[1])
        assert np.array_equal(one[0], y[0]) and np.array_equal(one[1], y[1])
        assert one[3].dt == x[2].dt == y[2].dt


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("solver", ["hlld", "hllc_mhd"])
def test_weak_out_of_plane_field(cuda, solver, order):
    """A field along z too weak to act on the flow is carried by it: scaled by 2^-60 it is the same
    field to rounding."""
    N, M = 70, 45
    cfg = config(*METHODS[solver], N, M)
    cfg.order = order
    rng = np.random.default_rng(8)
    K = N * M
    s = np.stack([rng.uniform(1, 1.5, K), rng.uniform(1, 1.5, K)], 1)
    u = rng.uniform(-0.5, 0.5, (K, 2))
    b = rng.uniform(-2, 2, (K, 3))
    T = 0.2 * cfg.dx / 4
    out = [gpu_step_ref(cfg, s, u, b * [1.0, 1.0, w], T)[2][:, 2] / w for w in (2.0 ** -40, 2.0 ** -100)]
    assert np.abs(out[1] - out[0]).max() <= 2e-15


@pytest.mark.parametrize("solver", ["hlld", "hllc_mhd"])
def test_weak_transverse_wave(cuda, solver):
    """Velocity and field along y, uniform in y, on a strong field along x."""
    N, M = 90, 23
    cfg = config(*METHODS[solver], N, M)
    rng = np.random.default_rng(9)
    s = np.stack([rng.uniform(1, 1.5, N), rng.uniform(3, 4, N)], 1)
    u = np.stack([rng.uniform(-0.5, 0.5, N), rng.uniform(-1, 1, N)], 1)
    b = np.stack([np.full(N, 3.0), rng.uniform(-1, 1, N), rng.uniform(-1, 1, N)], 1)
    s, u, b = (np.tile(x, (M, 1)) for x in (s, u, b))
    T = 0.2 * cfg.dx / 6
    out = []
    for w in (2.0 ** -40, 2.0 ** -90):
        _, u2, b2, _ = gpu_step_ref(cfg, s, u * [1.0, w], b * [1.0, w, w], T)
        out.append((u2[:, 1] / w, b2[:, 1] / w, b2[:, 2] / w))
    for x, y in zip(*out):
        assert np.abs(x - y).max() <= 2e-15


def test_recomputed_mhd_steps_keep_their_bits(cuda):
    """A reverse sweep steps again, with the many-tiles kernel beside its own launches, what the
    recording stepped with the few-tiles one: the same gradient as from the recorded states, with a
    part of the faces in floating point."""
    import torch
    N, M = 100, 70
    cfg = config(*METHODS["hlld"], N, M)
    s, u, b = jumpy(g.MHD, N * M, 4)
    rng = np.random.default_rng(10)
    lam = [torch.from_numpy(rng.standard_normal(x.shape)).cuda() for x in (s, u, b)]
    grads = []
    for every in (1, 6):
        sol = g.Solver(cfg)
        sol.import_state(s, u, b)
        sol.set_time(1e-3 * cfg.dx / 256, 0.0)
        sol.adj_forward(6, every)
        out = [torch.zeros_like(x) for x in lam]
        sol.adj_backward(*lam, *out)
        torch.cuda.synchronize()
        grads.append([x.cpu().numpy() for x in out])
        sol.close()
    for x, y in zip(*grads):
        assert np.isfinite(x).all() and np.array_equal(x, y)


@pytest.mark.parametrize("solver", ["hlld", "hllc_mhd"])
def test_tail_down_to_the_smallest_numbers(cuda, oracle_lib, solver):
    """The front that numerical diffusion sends ahead of a wave: a z field and a transverse velocity
    falling by 1000 per cell, past the smallest normal number.  Every cell to 1e-12 of the larger of
    its neighbours."""
    N, M = 130, 12
    cfg = config(*METHODS[solver], N, M)
    rng = np.random.default_rng(11)
    K = N * M
    tail = 10.0 ** (-3.0 * (np.arange(K) % N))  # 0 from 1e-324 on
    s = np.stack([rng.uniform(1, 1.2, K), rng.uniform(1, 1.2, K)], 1)
    u = np.stack([np.full(K, 0.3), np.zeros(K)], 1)
    b = np.stack([np.zeros(K), np.zeros(K), tail * rng.uniform(0.5, 1, K)], 1)
    T = 0.2 * cfg.dx / 4
    _, _, bo, _ = oracle_lib.step(grid_of(cfg), s, u, b, T)
    _, _, bg, _ = gpu_step_ref(cfg, s, u, b, T)
    scale = np.maximum(np.roll(tail.reshape(M, N), 2, 1), tail.reshape(M, N)).ravel()
    inner = (np.arange(K) % N >= 3) & (np.arange(K) % N < N - 3)
    d = np.abs(bg[:, 2] - bo[:, 2])
    assert (d <= 1e-12 * scale + 1e-307)[inner].all()
    assert np.count_nonzero(bg[inner, 2]) > 0.7 * inner.sum()
