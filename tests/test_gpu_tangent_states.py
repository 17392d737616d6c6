"""gd_tangent runs along the recorded states: it reads those that the recording or a reverse sweep
left in the segment buffers, steps the others again from their checkpoints, leaves the buffers as
they are, and gives the same bits either way."""
import numpy as np
import pytest

import golikov_2d_gb300 as g
from golikov_2d_gb300 import problems
from test_gpu_adjoint import dev, host

pytestmark = pytest.mark.gpu


def call(fn, xs):
    import torch
    xs = [dev(x) for x in xs]
    out = [torch.zeros_like(x) for x in xs]
    pad = [None] * (3 - len(xs))
    fn(*xs, *pad, *out, *pad)
    torch.cuda.synchronize()
    return [host(o) for o in out]


@pytest.mark.parametrize("nsteps,every,stepped", [(8, 4, 0), (7, 7, 0), (5, 1, 0), (11, 4, 3), (13, 3, 6)])
@pytest.mark.parametrize("flow", ["orszag_tang", "kelvin_helmholtz"])
def test_tangent_reads_recorded_states(cuda, flow, nsteps, every, stepped):
    """stepped: states of the segments before the last two that are not at a checkpoint."""
    cfg, s, u, b = getattr(problems, flow)(50, 34)
    sol = g.Solver(cfg)
    sol.import_state(s, u, b)
    sol.set_time(0.0, 0.0)
    sol.init_dt()
    sol.adj_forward(nsteps, every)
    rng = np.random.default_rng(4)
    ins = [x for x in (s, u, b) if x is not None]
    v, lam = ([rng.standard_normal(x.shape) for x in ins] for _ in range(2))
    n0 = sol.launch_count()
    a = call(sol.tangent, v)
    n1 = sol.launch_count()
    assert n1 - n0 == nsteps + stepped
    g1 = call(sol.adj_backward, lam)
    c = call(sol.tangent, v)  # the sweep left other segments in the buffers
    call(sol.adj_replay, ins)  # its work space is one of them
    d = call(sol.tangent, v)
    g2 = call(sol.adj_backward, lam)
    for x, y, z in zip(a, c, d):
        assert np.array_equal(x, y) and np.array_equal(x, z)
    for x, y in zip(g1, g2):
        assert np.array_equal(x, y)
    sol.close()
