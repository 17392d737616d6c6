"""The MHD reverse sweep in the regimes of the HLLD fan that its short form treats apart: upwind
flux only (supersonic along x or y), star and double-star states (subsonic, strong field), no
normal field (the double star falls away), and densities and fields so small that the star
guards |tt| >= 1e-5 fail at every face or at some of them.  In each the dot-product identity
<lam, J v> = <J^T lam, v> with the forward-mode tangent, which differentiates the full chain of
the flux, holds to 1e-10 relative: a face's adjoint carries about 1e-14, a few hundred times
that after six steps and the cancellation of the sums."""
import numpy as np
import pytest

import golikov_2d_gb300 as g
from golikov_2d_gb300 import problems
from test_gpu_adjoint_ragged import dev, host, smooth_state

pytestmark = pytest.mark.gpu

# density and pressure scale, field scale, uniform velocity
REGIMES = {
    "subsonic": (1.0, 1.0, (0.0, 0.0)),
    "strong_field": (1.0, 4.0, (0.0, 0.0)),
    "supersonic_x": (1.0, 1.0, (6.0, 0.0)),
    "supersonic_y": (1.0, 1.0, (0.0, -6.0)),
    "no_field": (1.0, 0.0, (0.0, 0.0)),
    "guards_fail": (1e-7, 3e-4, (0.0, 0.0)),
    "guards_mixed": (5e-6, 2e-3, (0.2, 0.1)),
}


@pytest.mark.parametrize("regime", REGIMES)
def test_dot_product_in_every_region_of_the_fan(cuda, regime):
    import torch
    scale, field, (ux, uy) = REGIMES[regime]
    cfg, s, u, b = smooth_state("mhd", 37, 23)
    s, b = s * scale, b * field
    u = u + np.array([ux, uy])
    sol = g.Solver(cfg)
    sol.import_state(s, u, b)
    sol.set_time(0.0, 0.0)
    sol.init_dt()
    sol.advance(2)
    sol.adj_forward(6, 4)
    rng = np.random.default_rng(5)
    # directions and weights in each field's own scale
    size = (np.array([scale, scale]), np.ones(2), np.full(3, field or scale ** 0.5))
    v = [rng.standard_normal(x.shape) * z for x, z in zip((s, u, b), size)]
    lam = [rng.standard_normal(x.shape) / z for x, z in zip((s, u, b), size)]

    def call(fn, xs):
        out = [torch.zeros_like(dev(x)) for x in xs]
        fn(*[dev(x) for x in xs], *out)
        torch.cuda.synchronize()
        return [host(o) for o in out]

    dot = lambda p, q: sum(float((x * y).sum()) for x, y in zip(p, q))
    lhs, rhs = dot(lam, call(sol.tangent, v)), dot(call(sol.adj_backward, lam), v)
    assert np.isfinite(lhs) and abs(lhs - rhs) <= 1e-10 * max(abs(lhs), abs(rhs)), (lhs, rhs)
    sol.close()


@pytest.mark.parametrize("flow", ["orszag_tang", "kelvin_helmholtz"])
def test_tangent_follows_the_recorded_run(cuda, flow):
    """A long run from an initial state full of exact ties: the tangent takes the branches of the
    recorded states, not of states of its own that drift from them by rounding."""
    import torch
    cfg, s, u, b = getattr(problems, flow)(256, 256)
    sol = g.Solver(cfg)
    sol.import_state(s, u, b)
    sol.set_time(0.0, 0.0)
    sol.init_dt()
    sol.adj_forward(100, 10)
    rng = np.random.default_rng(3)
    ins = [x for x in (s, u, b) if x is not None]
    lam, v = ([rng.standard_normal(x.shape) for x in ins] for _ in range(2))

    def call(fn, xs):
        xs = [dev(x) for x in xs]
        out = [torch.zeros_like(x) for x in xs]
        pad = [None] * (3 - len(xs))
        fn(*xs, *pad, *out, *pad)
        torch.cuda.synchronize()
        return [host(o) for o in out]

    dot = lambda p, q: sum(float((x * y).sum()) for x, y in zip(p, q))
    lhs, rhs = dot(lam, call(sol.tangent, v)), dot(call(sol.adj_backward, lam), v)
    assert np.isfinite(lhs) and abs(lhs - rhs) <= 1e-10 * max(abs(lhs), abs(rhs)), (lhs, rhs)
    sol.close()
