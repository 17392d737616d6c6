"""The workloads this library is timed on, and their results in plain 64-bit torch.

A case is a dict of plain values.  `prepare` makes its inputs on the GPU from a seed and the
solver a program keeps, `run` is one pass through the public entry points, `exact` is what that
pass returns, computed with torch alone.  Kinds of work:

  dropin   the reference's loop protocol on AoS device arrays: step, dt rotation, step, rotation
  run      a run of the resident loop: import, dt pass, n steps, export
  batch    many uneven Euler grids advanced together
  adjoint  a recorded run and its reverse sweep: final state and gradient
  host     one step from pinned host arrays to pinned host arrays
  text     the restart text of a state, written and read back: its length, and the state read

Flow states: `shear` (Kelvin-Helmholtz layer), `quadrants` (four-quadrant Riemann problem),
`vortex` (Orszag-Tang), `wind` (magnetised wind in an ambient medium, axisymmetric, with the
production run's boundaries and frozen sphere), `waves` (a few smooth Fourier modes).
"""
from __future__ import annotations

import math

import numpy as np
import torch

import golikov_2d_gb300 as g
from golikov_2d_gb300 import problems

METHODS = {"hll": g.METHOD_HLL, "hllc": g.METHOD_HLLC, "hllc_mhd": g.METHOD_HLLC_MHD,
           "hlld": g.METHOD_HLLD}
F64 = torch.float64


def _case(name, kind, flow, N, M, method, **kw):
    c = {"kind": kind, "flow": flow, "N": N, "M": M, "method": method, "order": 2, "steps": 1,
         "graph": False}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest calls a coupled driver makes: launches and latency are what count
        _case("small", "dropin", "quadrants", 64, 48, "hllc", steps=2),
        # an ordinary odd-sized grid through the drop-in protocol, HLL faces
        _case("ragged_hll", "dropin", "quadrants", 777, 533, "hll", steps=2),
        # an ordinary resident run replayed as a graph
        _case("shear_512", "run", "shear", 512, 512, "hllc", steps=20, graph=True),
        # the benchmark's largest single grid
        _case("shear_4096", "run", "shear", 4096, 4096, "hllc", steps=2),
        # the MHD benchmark grid
        _case("vortex_1024", "run", "vortex", 1024, 1024, "hlld", steps=4),
        # an odd-sized MHD grid through the drop-in protocol, the other MHD flux
        _case("ragged_mhd", "dropin", "vortex", 333, 211, "hllc_mhd", steps=2),
        # the reference's production problem on its production grid
        _case("wind_3226", "run", "wind", 3226, 1792, "hlld", steps=1),
        # the MUSCL-Hancock scheme on the same grid
        _case("hancock_3226", "run", "wind", 3226, 1792, "hlld", steps=1, hancock=True),
        # a parameter study: uneven four-quadrant problems advanced together
        _case("batch_128", "batch", "quadrants", 64, 512, "hllc", grids=128, steps=4, graph=True),
        # the gradient of an MHD run
        _case("adjoint_mhd", "adjoint", "waves", 512, 512, "hlld", steps=10),
        # a program that keeps its state in host memory
        _case("host_2048", "host", "shear", 2048, 2048, "hllc"),
        # a restart file's text, both directions
        _case("text_512", "text", "vortex", 512, 512, "hlld"),
    ]


def draw(rng):
    def side(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("dropin", "dropin", "run", "run", "wind", "batch", "adjoint", "host", "text"))
    euler = rng.random() < 0.5
    method = rng.choice(("hllc", "hllc", "hll")) if euler else rng.choice(("hlld", "hlld", "hllc_mhd"))
    order = 1 if rng.random() < 0.15 else 2
    if kind == "dropin":
        return _case(None, kind, "quadrants" if euler else "vortex", side(40, 1200), side(40, 1200),
                     method, order=order, steps=2)
    if kind == "run":
        N, M = side(100, 4096 if euler else 1600), side(100, 4096 if euler else 1600)
        steps = max(1, min(20, int((3e7 if euler else 4e6) / (N * M))))
        return _case(None, kind, "shear" if euler else "vortex", N, M, method, order=order, steps=steps,
                     graph=rng.random() < 0.5)
    if kind == "wind":
        N = side(300, 3226)
        hancock = rng.random() < 0.5
        return _case(None, "run", "wind", N, max(40, int(N / 1.8) + rng.randrange(-9, 10)),
                     "hlld" if hancock else rng.choice(("hlld", "hlld", "hllc_mhd")),
                     order=2 if hancock else order, hancock=hancock)
    if kind == "batch":
        return _case(None, kind, "quadrants", 64, side(128, 512), rng.choice(("hllc", "hllc", "hll")),
                     grids=side(8, 128), steps=rng.randrange(1, 5), graph=rng.random() < 0.5)
    if kind == "adjoint":
        return _case(None, kind, "waves", side(64, 512), side(64, 512), "hllc" if euler else "hlld",
                     steps=rng.randrange(4, 11))
    if kind == "host":
        return _case(None, kind, "shear" if euler else "vortex", side(128, 2048 if euler else 1024),
                     side(128, 2048 if euler else 1024), method)
    return _case(None, "text", "shear" if euler else "vortex", side(32, 512), side(32, 512),
                 "hllc" if euler else "hlld")


# ---- inputs ---------------------------------------------------------------------------------

def _mhd(case):
    return case["method"] in ("hlld", "hllc_mhd")


def _sides(case):
    """Grid sides of a batch, log-uniform in [N, M], the same for every seed."""
    return problems.batch_sides(case["grids"], case["N"], case["M"])


def _config(case, N=None, M=None):
    N, M = N or case["N"], M or case["M"]
    if case["flow"] == "wind":
        if case.get("hancock"):
            return problems.hancock_config(N, M)
        return g.Config(N=N, M=M, dx=9.0 / N, dy=5.0 / M, x0=4.5 / N, y0=2.5 / M, gamma=5.0 / 3.0,
                        krit=0.25, physics=g.MHD, geometry=g.AXISYM, order=case["order"],
                        method=METHODS[case["method"]],
                        bc=(g.BC_MIRROR_X, g.BC_OUTFLOW, g.BC_AXIS, g.BC_AMBIENT),
                        frozen_radius=problems.DDIST)
    mhd = _mhd(case)
    bc = g.BC_TRANSMISSIVE if case["flow"] == "quadrants" else g.BC_PERIODIC
    return problems.unit_square(N, M, 5.0 / 3.0 if mhd else 1.4, 0.4,
                                physics=g.MHD if mhd else g.EULER, order=case["order"],
                                method=METHODS[case["method"]], bc=(bc,) * 4)


def _state(case, cfg, gen):
    """Fields (4 or 7, M, N) of the case's flow; every seed is another realisation."""
    dev = gen.device
    n = torch.arange(cfg.N, dtype=F64, device=dev)
    m = torch.arange(cfg.M, dtype=F64, device=dev)
    if case.get("hancock"):
        X, Y = cfg.x0 + n * (cfg.x_max - cfg.x0) / (cfg.N - 1), cfg.y0 + m * cfg.y_max / cfg.M
    else:
        X, Y = cfg.x0 + n * cfg.dx, cfg.y0 + m * cfg.dy
    Y, X = torch.meshgrid(Y, X, indexing="ij")

    def noise(size):
        return size * (2.0 * torch.rand(X.shape, dtype=F64, device=dev, generator=gen) - 1.0)

    tau, zero = 2.0 * math.pi, torch.zeros_like(X)
    if case["flow"] == "shear":
        inner = (Y - 0.5).abs() < 0.25
        return torch.stack([torch.where(inner, 2.0, 1.0).to(F64), zero + 2.5,
                            torch.where(inner, 0.5, -0.5).to(F64), noise(0.01)])
    if case["flow"] == "quadrants":
        part = (X >= 0.5).long() + 2 * (Y >= 0.5).long()
        lo = torch.tensor([0.1, 0.1, -1.0, -1.0], dtype=F64, device=dev)
        hi = torch.tensor([2.0, 2.0, 1.0, 1.0], dtype=F64, device=dev)
        v = lo + (hi - lo) * torch.rand((4, 4), dtype=F64, device=dev, generator=gen)
        return v[part.reshape(-1)].T.reshape(4, cfg.M, cfg.N).contiguous()
    if case["flow"] == "vortex":
        return torch.stack([25.0 / (36.0 * math.pi) * (1.0 + noise(0.01)),
                            5.0 / (12.0 * math.pi) * (1.0 + noise(0.01)),
                            -torch.sin(tau * Y) + noise(0.01), torch.sin(tau * X) + noise(0.01),
                            -torch.sin(tau * Y) + noise(0.01), torch.sin(2.0 * tau * X) + noise(0.01), zero])
    if case["flow"] == "wind":
        gamma, RR, VE = cfg.gamma, problems.RR_0, problems.PHI_0
        rE = 1.0 / (VE * RR) ** 2
        pE = rE * VE ** 2 / (gamma * problems.M_0 ** 2)
        bE = math.sqrt(4.0 * math.pi) / (problems.M_ALF * RR)
        d = torch.sqrt(X * X + Y * Y)
        w = d < cfg.frozen_radius * 1.01
        return torch.stack([torch.where(w, rE * (RR / d) ** 2, 1.0 + noise(0.01)),
                            torch.where(w, pE * (RR / d) ** (2.0 * gamma), (1.0 + noise(0.01)) / gamma),
                            torch.where(w, VE * X / d, noise(0.01)), torch.where(w, VE * Y / d, noise(0.01)),
                            zero, zero, torch.where(w, bE * RR * Y / (d * d), zero)])
    # waves: rho, p about 1, velocities and field below the sound speed
    q = []
    for f in range(7 if _mhd(case) else 4):
        s = zero
        for _ in range(3):
            a, b, c, ph = torch.rand(4, dtype=F64, generator=gen, device=dev).tolist()
            s = s + (0.05 + 0.05 * a) * torch.sin(tau * (int(1 + 3 * b) * X + int(1 + 3 * c) * Y + ph))
        q.append(1.0 + s if f < 2 else 2.0 * s)
    return torch.stack(q)


def _aos(q):
    nf = q.shape[0]
    flat = q.reshape(nf, -1).T
    return flat[:, 0:2].contiguous(), flat[:, 2:4].contiguous(), flat[:, 4:7].contiguous() if nf == 7 else None


def _inputs(case, seed):
    """[(config, fields)] of the case's grids."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    cfgs = [_config(case, k, k) for k in _sides(case)] if case["kind"] == "batch" else [_config(case)]
    return [(c, _state(case, c, gen)) for c in cfgs]


def _seeds_of_adjoint(case, seed, q):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) + 1)
    return torch.rand(q.shape, dtype=F64, device="cuda", generator=gen) - 0.5


# the dt a drop-in or host loop hands to its first step
def _first_dt(cfg):
    return 0.05 * cfg.krit * min(cfg.dx, cfg.dy)


def prepare(case, seed):
    grids = _inputs(case, seed)
    cfg, q = grids[0]
    if case["kind"] == "batch":
        return {"case": case, "batch": g.Batch([c for c, _ in grids]), "in": [_aos(x)[:2] for _, x in grids],
                "out": [tuple(torch.empty_like(t) for t in _aos(x)[:2]) for _, x in grids]}
    U = _aos(q)
    st = {"case": case, "sol": g.Solver(cfg), "U": U, "dt": _first_dt(cfg)}
    blank = lambda: tuple(None if t is None else torch.empty_like(t) for t in U)  # noqa: E731
    if case["kind"] == "dropin":
        st["A"], st["B"] = blank(), blank()
        st["T0"] = torch.tensor([1e7, st["dt"], st["dt"]], dtype=F64, device="cuda")
        st["T"] = st["T0"].clone()
        st["i"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    elif case["kind"] == "host":
        st["U"] = tuple(None if t is None else t.cpu().pin_memory() for t in U)
        st["A"] = tuple(None if t is None else torch.empty_like(t).pin_memory() for t in st["U"])
    elif case["kind"] == "adjoint":
        st["A"], st["B"], st["g"] = blank(), blank(), _aos(_seeds_of_adjoint(case, seed, q))
    else:
        st["A"] = blank()
    return st


def _some(ts):
    return [t for t in ts if t is not None]


def run(st):
    case = st["case"]
    if case["kind"] == "batch":
        b = st["batch"]
        for k, (s, u) in enumerate(st["in"]):
            b.import_grid(k, s, u)
        b.set_time(0.0)
        b.init_dt()
        b.advance(case["steps"], use_graph=case["graph"])
        for k, (s, u) in enumerate(st["out"]):
            b.export_grid(k, s, u)
        return [torch.cat([s for s, _ in st["out"]]), torch.cat([u for _, u in st["out"]])]
    sol = st["sol"]
    if case["kind"] == "dropin":
        T = st["T"]
        T.copy_(st["T0"])
        src, dst = st["U"], (st["A"], st["B"])
        for k in range(case["steps"]):
            sol.kernel_step(*src, *dst[k % 2], T[0:1], T[1:2])
            sol.funk_time(T[0:1], T[1:2], T[2:3], st["i"])
            src = dst[k % 2]
        return _some(src) + [T]
    if case["kind"] == "host":
        sol.set_time(st["dt"])
        sol.step_host(*st["U"], *st["A"])
        return _some(st["A"])
    sol.import_state(*st["U"])
    if case["kind"] == "text":
        text = sol.format_text()
        sol.parse_text(text)
        sol.export_state(*st["A"])
        return [len(text)] + _some(st["A"])
    sol.set_time(0.0)
    sol.init_dt()
    if case["kind"] == "adjoint":
        sol.adj_forward(case["steps"], max(1, case["steps"] // 2))
        sol.export_state(*st["A"])
        sol.adj_backward(*st["g"], *st["B"])
        return _some(st["A"]) + _some(st["B"])
    sol.advance(case["steps"], use_graph=case["graph"])
    sol.export_state(*st["A"])
    return _some(st["A"])


def work(case):
    """Bytes: the state read and written once per pass (a run may keep it on the chip between
    steps).  Operations: those of the scheme's formulas with every face computed once."""
    cells = sum(k * k for k in _sides(case)) if case["kind"] == "batch" else case["N"] * case["M"]
    nf = 7 if _mhd(case) else 4
    if case["kind"] == "text":
        return {"bytes": cells * (8.0 * nf + 75.0) * 2, "flops": 0.0}
    per = (600.0 if _mhd(case) else 200.0) * (1.6 if case.get("hancock") else 1.0)
    steps = case["steps"] * (4.0 if case["kind"] == "adjoint" else 1.0)
    return {"bytes": cells * 8.0 * nf * (4 if case["kind"] == "adjoint" else 2), "flops": cells * per * steps}


# ---- the same in 64-bit torch -----------------------------------------------------------------

def _minmod(a, b):
    return torch.where(a * b > 0, torch.where(a.abs() <= b.abs(), a, b), torch.zeros_like(a))


def _ghost(v, bc, cfg):
    v = v.clone()
    if bc == g.BC_MIRROR_X:
        v[2] = -v[2]
        if len(v) > 4:
            v[4:6] = -v[4:6]
    elif bc == g.BC_AXIS:
        v[3] = -v[3]
        if len(v) > 4:
            v[6] = -v[6]
    elif bc in (g.BC_AMBIENT, g.BC_AMBIENT_KEEPB):
        v[0], v[1], v[2:4] = 1.0, 1.0 / cfg.gamma, 0.0
        if bc == g.BC_AMBIENT and len(v) > 4:
            v[4:] = 0.0
    elif bc == g.BC_OUTFLOW:
        v[2] = torch.where(v[2] < 0, torch.full_like(v[2], 0.01), v[2])
    return v


def _padded(q, axis, bcs, cfg):
    """The fields with two ghost layers on both ends of an axis (1: y, 2: x)."""
    n = q.shape[axis]

    def layer(k, bc):
        return _ghost(q.narrow(axis, k, 1), bc, cfg)

    def src(depth, low, bc):
        if bc == g.BC_PERIODIC:
            return n - depth if low else depth - 1
        if bc in (g.BC_MIRROR_X, g.BC_AXIS):
            return depth - 1 if low else n - depth
        return 0 if low else n - 1

    lo, hi = bcs
    return torch.cat([layer(src(2, True, lo), lo), layer(src(1, True, lo), lo), q,
                      layer(src(1, False, hi), hi), layer(src(2, False, hi), hi)], axis)


def _local(q, axis):
    """Fields in a face's frame: normal component first."""
    if axis == 2:
        return q
    return torch.stack([q[0], q[1], q[3], q[2]] + ([q[5], q[4], q[6]] if len(q) == 7 else []))


def _hllc(L, R, cfg, hll):
    gm = cfg.gamma
    rL, pL, uL, vL = L
    rR, pR, uR, vR = R
    cL, cR = torch.sqrt(gm * pL / rL), torch.sqrt(gm * pR / rR)
    eL = pL / (gm - 1) + 0.5 * rL * (uL * uL + vL * vL)
    eR = pR / (gm - 1) + 0.5 * rR * (uR * uR + vR * vR)
    FL = (rL * uL, (eL + pL) * uL, rL * uL * uL + pL, rL * uL * vL)
    FR = (rR * uR, (eR + pR) * uR, rR * uR * uR + pR, rR * uR * vR)
    UL, UR = (rL, eL, rL * uL, rL * vL), (rR, eR, rR * uR, rR * vR)
    if hll:
        c = torch.maximum(cL, cR)
        SL, SR = torch.minimum(uL, uR) - c, torch.maximum(uL, uR) + c
        F = [torch.where(SL > 0, a, torch.where(SR < 0, b, (SR * a - SL * b + SL * SR * (y - x)) / (SR - SL)))
             for a, b, x, y in zip(FL, FR, UL, UR)]
    else:
        SL, SR = torch.minimum(uL - cL, uR - cR), torch.maximum(uL + cL, uR + cR)
        mL, mR = rL * (SL - uL), rR * (SR - uR)
        SM = (mR * uR - mL * uL + pL - pR) / (mR - mL)

        def star(S, m, r, p, u, v, e, U, F):
            rs = m / (S - SM)
            es = (e * (S - u) + (p + m * (SM - u)) * SM - p * u) / (S - SM)
            return [f + S * (y - x) for f, x, y in zip(F, U, (rs, es, rs * SM, rs * v))]

        sL, sR = star(SL, mL, rL, pL, uL, vL, eL, UL, FL), star(SR, mR, rR, pR, uR, vR, eR, UR, FR)
        F = [torch.where(SL > 0, a, torch.where(SM >= 0, b, torch.where(SR >= 0, c, d)))
             for a, b, c, d in zip(FL, sL, sR, FR)]
    return torch.stack(F), torch.maximum(SL.abs(), SR.abs())


def _mhd_side(q, gm):
    """Total pressure, energy, fast speed, state and flux of a side; field in units of sqrt(4 pi)."""
    r, p, u, v, a, b, c = q
    bb = a * a + b * b + c * c
    pt, e = p + bb / 2, p / (gm - 1) + 0.5 * r * (u * u + v * v) + bb / 2
    s = gm * p + bb
    disc = (s * s - 4 * gm * p * a * a).clamp(min=0.0)
    disc = torch.where(disc > 0, torch.sqrt(torch.where(disc > 0, disc, torch.ones_like(disc))), disc)
    cf = torch.sqrt((s + disc) / (2 * r))
    zero = torch.zeros_like(r)
    F = [r * u, (e + pt) * u - a * (u * a + v * b), r * u * u + pt - a * a, r * u * v - a * b, zero,
         u * b - v * a, u * c, -a * c]
    return pt, e, cf, [r, e, r * u, r * v, a, b, c, zero], F


def _mhd_flux(L, R, cfg, hlld):
    """(mass, energy, normal and tangential momentum, normal, tangential and z field) flux."""
    rL, _, uL, vL, aL, bL, cL = L
    rR, _, uR, vR, aR, bR, cR = R
    ptL, eL, cfL, UL, FL = _mhd_side(L, cfg.gamma)
    ptR, eR, cfR, UR, FR = _mhd_side(R, cfg.gamma)
    c = torch.maximum(cfL, cfR)
    SL, SR = torch.minimum(uL, uR) - c, torch.maximum(uL, uR) + c
    mL, mR = rL * (SL - uL), rR * (SR - uR)
    SM = (mR * uR - mL * uL - ptR + ptL) / (mR - mL)
    pt = (mR * ptL - mL * ptR + mL * mR * (uR - uL)) / (mR - mL)

    def fan(k):
        return (SR * UR[k] - SL * UL[k] + FL[k] - FR[k]) / (SR - SL)

    bn = fan(4)
    UU = torch.maximum(SL.abs(), SR.abs())
    if not hlld:
        bt, bz, r0, m1, m2, m3 = fan(5), fan(6), fan(0), fan(2), fan(3), fan(7)
        vs, sbz = m2 / r0, (bn * m1 + bt * m2 + bz * m3) / r0
        pz = 0.5 * (ptR + mR * (SM - uR) + ptL + mL * (SM - uL))

        def star(S, m, q, p, e, U, F):
            rs = m / (S - SM)
            es = (e * (S - q[2]) + pz * SM - p * q[2] + bn * (q[2] * q[4] + q[3] * q[5] - sbz)) / (S - SM)
            return [f + S * (y - x) for f, x, y in zip(F, U, (rs, es, rs * SM, rs * vs, bn, bt, bz))]

        sL, sR = star(SL, mL, L, ptL, eL, UL, FL), star(SR, mR, R, ptR, eR, UR, FR)
        F = [torch.where(SL >= 0, a, torch.where(SM >= 0, b, torch.where(SR > 0, d, h)))
             for a, b, d, h in zip(FL, sL, sR, FR)]
    else:
        def star(S, m, q, p, e):
            r, _, u, v, a, b, z = q
            tt, rs = m * (S - SM) - bn * bn, m / (S - SM)
            ok = tt.abs() >= 1e-5
            it = 1.0 / torch.where(ok, tt, torch.ones_like(tt))
            k, d = bn * (SM - u) * it, (m * (S - u) - bn * bn) * it
            zero = torch.zeros_like(r)
            vs, ws = torch.where(ok, v - k * b, v), torch.where(ok, -k * z, zero)
            bs, zs = torch.where(ok, b * d, zero), torch.where(ok, z * d, zero)
            sb = SM * bn + vs * bs + ws * zs
            es = (e * (S - u) + pt * SM - p * u + bn * (u * a + v * b - sb)) / (S - SM)
            return rs, vs, ws, bs, zs, sb, es

        r1, v1, w1, b1, z1, s1, e1 = star(SL, mL, L, ptL, eL)
        r2, v2, w2, b2, z2, s2, e2 = star(SR, mR, R, ptR, eR)
        q1, q2 = torch.sqrt(r1), torch.sqrt(r2)
        on = bn.abs() > 1e-6
        sg = torch.where(on, torch.sign(bn), torch.zeros_like(bn))
        S1 = torch.where(on, SM - bn.abs() / q1, SM)
        S2 = torch.where(on, SM + bn.abs() / q2, SM)
        q = q1 + q2
        v3, w3 = (q1 * v1 + q2 * v2 + sg * (b2 - b1)) / q, (q1 * w1 + q2 * w2 + sg * (z2 - z1)) / q
        b3 = (q1 * b2 + q2 * b1 + sg * q1 * q2 * (v2 - v1)) / q
        z3 = (q1 * z2 + q2 * z1 + sg * q1 * q2 * (w2 - w1)) / q
        s3 = SM * bn + v3 * b3 + w3 * z3
        V1, V2 = (r1, e1, r1 * SM, r1 * v1, bn, b1, z1), (r2, e2, r2 * SM, r2 * v2, bn, b2, z2)
        W1 = (r1, e1 - sg * q1 * (s1 - s3), r1 * SM, r1 * v3, bn, b3, z3)
        W2 = (r2, e2 + sg * q2 * (s2 - s3), r2 * SM, r2 * v3, bn, b3, z3)
        F = []
        for k in range(7):
            fl, fr = FL[k] + SL * (V1[k] - UL[k]), FR[k] + SR * (V2[k] - UR[k])
            F.append(torch.where(SL >= 0, FL[k], torch.where(
                (SM >= 0) & (S1 >= 0), fl, torch.where(
                    SM >= 0, fl + S1 * (W1[k] - V1[k]), torch.where(
                        S2 > 0, fr + S2 * (W2[k] - V2[k]), torch.where(SR > 0, fr, FR[k]))))))
    F[4] = -UU * (aR - aL)
    return torch.stack(F[:7]), UU


def _flux(L, R, axis, cfg):
    """The flux in the order (mass, energy, x and y momentum, Bx, By, Bz) and the wave speed."""
    L, R = _local(L, axis), _local(R, axis)
    if len(L) == 4:
        F, UU = _hllc(L, R, cfg, cfg.method == g.METHOD_HLL)
    else:
        F, UU = _mhd_flux(L, R, cfg, cfg.method == g.METHOD_HLLD)
    if axis == 1:
        F = torch.stack([F[0], F[1], F[3], F[2]] + ([F[5], F[4], F[6]] if len(F) == 7 else []))
    return F, UU


def _active(cfg, X, Y):
    return ~(torch.sqrt(X * X + Y * Y) < cfg.frozen_radius) if cfg.frozen_radius > 0 else torch.ones_like(X, dtype=torch.bool)


def _fastest(UU, active, axis):
    """The largest wave speed of the faces that an updated cell uses."""
    off = torch.zeros_like(active.narrow(axis - 1, 0, 1))
    used = torch.cat([off, active], axis - 1) | torch.cat([active, off], axis - 1)
    return torch.where(used, UU.detach(), torch.zeros_like(UU)).max()


def _cfl(cfg, ux, uy):
    hx, hy = (cfg.dy, cfg.dx) if cfg.physics == g.EULER else (cfg.dx, cfg.dy)
    return torch.minimum(torch.minimum(cfg.krit * hx / ux, cfg.krit * hy / uy), torch.full_like(ux, 1000.0))


def _tvd_step(q, cfg, dt):
    """One step of the TVD scheme with time step dt: (fields, the CFL time step of the input).
    The field is in units of sqrt(4 pi)."""
    n = torch.arange(cfg.N, dtype=F64, device=q.device)
    m = torch.arange(cfg.M, dtype=F64, device=q.device)
    Y, X = torch.meshgrid(cfg.y0 + m * cfg.dy, cfg.x0 + n * cfg.dx, indexing="ij")
    act = _active(cfg, X, Y)
    diff, fast, pads = 0.0, {}, {}
    for axis, bcs, h in ((2, cfg.bc[:2], cfg.dx), (1, cfg.bc[2:], cfg.dy)):
        z = _padded(q, axis, bcs, cfg)
        pads[axis] = z
        cnt = q.shape[axis]
        c = z.narrow(axis, 1, cnt + 2)
        lo, hi = c, c
        if cfg.order == 2:
            s = 0.5 * _minmod(c - z.narrow(axis, 0, cnt + 2), z.narrow(axis, 2, cnt + 2) - c)
            lo, hi = c + s, c - s
            pos = torch.tensor([k < 2 for k in range(len(q))], device=q.device).view(-1, 1, 1)
            lo, hi = torch.where(pos & (lo <= 0), c, lo), torch.where(pos & (hi <= 0), c, hi)
        F, UU = _flux(lo.narrow(axis, 0, cnt + 1), hi.narrow(axis, 1, cnt + 1), axis, cfg)
        diff = diff + (dt / h) * (F.narrow(axis, 1, cnt) - F.narrow(axis, 0, cnt))
        fast[axis] = _fastest(UU, act, axis)
    new = _update_euler(q, diff, cfg) if len(q) == 4 else _update_mhd(q, diff, cfg, dt, Y, pads)
    return torch.where(act, new, q), _cfl(cfg, fast[2], fast[1])


def _floor(x, low):
    return torch.where(x <= 0, low if torch.is_tensor(low) else torch.full_like(x, low), x)


def _update_euler(q, d, cfg):
    r, p, u, v = q
    r2 = _floor(r - d[0], 0.0001)
    mx, my = r * u - d[2], r * v - d[3]
    E = p / (cfg.gamma - 1) + 0.5 * r * (u * u + v * v) - d[1]
    p2 = _floor((E - 0.5 * (mx * mx + my * my) / r2) * (cfg.gamma - 1), 0.000001)
    return torch.stack([r2, p2, mx / r2, my / r2])


def _update_mhd(q, d, cfg, dt, Y, pads):
    r, p, u, v, bx, by, bz = q
    px, py = pads[2], pads[1]
    div = dt * ((px[4, :, 3:-1] - px[4, :, 1:-3]) / (2 * cfg.dx) + (py[5, 3:-1] - py[5, 1:-3]) / (2 * cfg.dy))
    ub, bb = u * bx + v * by, bx * bx + by * by + bz * bz
    E = p / (cfg.gamma - 1) + 0.5 * (r * (u * u + v * v) + bb)
    src = [0.0] * 5
    if cfg.geometry == g.AXISYM:
        div = div + dt * by / Y
        k = dt / Y
        src = [k * r * v, k * (r * u * v - bx * by), k * (r * v * v + bz * bz - by * by),
               k * (v * bx - by * u), k * ((E + p + bb / 2) * v - by * ub)]
    r2 = _floor(r - d[0] - src[0], r)
    mx, my = r * u - d[2] - bx * div - src[1], r * v - d[3] - by * div - src[2]
    b1, b2, b3 = bx - d[4] - u * div - src[3], by - d[5] - v * div, bz - d[6]
    E2 = E - d[1] - ub * div - src[4]
    p2 = _floor((E2 - 0.5 * (mx * mx + my * my) / r2 - 0.5 * (b1 * b1 + b2 * b2 + b3 * b3)) * (cfg.gamma - 1), 0.000001)
    return torch.stack([r2, p2, mx / r2, my / r2, b1, b2, b3])


# the points of the Hancock scheme's stencil (offsets in x and y), with its edge substitutes
def _hancock_points(q, cfg):
    N, M = cfg.N, cfg.M
    n = torch.arange(N, device=q.device).view(1, 1, N)
    m = torch.arange(M, device=q.device).view(1, M, 1)

    def at(dx, dy):
        return torch.roll(q, (-dy, -dx), (1, 2))

    def pick(*rules):
        *conds, v = rules
        for c, w in reversed(conds):
            v = torch.where(c, w, v)
        return v

    def mx(c):
        return _ghost(c, g.BC_MIRROR_X, cfg)

    def my(c):
        return _ghost(c, g.BC_AXIS, cfg)

    def out(c):
        return _ghost(c, g.BC_OUTFLOW, cfg)

    def amb(c):
        return _ghost(c, g.BC_AMBIENT_KEEPB, cfg)

    c1 = q
    c2, c3 = pick((n == N - 1, out(c1)), at(1, 0)), pick((m == 0, my(c1)), at(0, -1))
    c4, c5 = pick((n == 0, mx(c1)), at(-1, 0)), pick((m == M - 1, amb(c1)), at(0, 1))
    return [None, c1, c2, c3, c4, c5, pick((n >= N - 2, out(c2)), at(2, 0)),
            pick((m == 1, my(c5)), (m == 0, my(c3)), at(0, -2)), pick((n <= 1, mx(c2)), at(-2, 0)),
            pick((m >= M - 2, c5), at(0, 2)), pick((n == N - 1, c5), (m == M - 1, amb(c2)), at(1, 1)),
            pick((m == 0, my(c2)), (n == N - 1, out(c3)), at(1, -1)),
            pick((m == 0, my(c4)), (n == 0, mx(c3)), at(-1, -1)),
            pick((n == 0, mx(c5)), (m == M - 1, amb(c4)), at(-1, 1))]


def _hancock_move(Q, d, cfg, k, y, low):
    """Q after the flux differences d and the axisymmetric sources of k = time / y."""
    r, p, u, v, bx, by, bz = Q
    bb, ub = bx * bx + by * by + bz * bz, u * bx + v * by
    E = p / (cfg.gamma - 1) + 0.5 * (r * (u * u + v * v) + bb)
    r2 = _floor(r - d[0] - k * r * v, r)
    u2 = (r * u - d[2] - k * (r * u * v - bx * by)) / r2
    v2 = (r * v - d[3] - k * (r * v * v + bz * bz - by * by)) / r2
    b1, b2, b3 = bx - d[4] - k * (v * bx - by * u), by - d[5], bz - d[6]
    E2 = E - d[1] - k * ((E + p + bb / 2) * v - by * ub)
    p2 = _floor((E2 - 0.5 * (r2 * (u2 * u2 + v2 * v2) + b1 * b1 + b2 * b2 + b3 * b3)) * (cfg.gamma - 1), low)
    return torch.stack([r2, p2, u2, v2, b1, b2, b3])


def _hancock_step(q, cfg, dt):
    n = torch.arange(cfg.N, dtype=F64, device=q.device)
    m = torch.arange(cfg.M, dtype=F64, device=q.device)
    Y, X = torch.meshgrid(cfg.y0 + m * cfg.y_max / cfg.M, cfg.x0 + n * (cfg.x_max - cfg.x0) / (cfg.N - 1), indexing="ij")
    act = _active(cfg, X, Y)
    c = _hancock_points(q, cfg)
    pos = torch.tensor([k < 2 for k in range(7)], device=q.device).view(-1, 1, 1)

    def slope(a, b, z, h):
        if cfg.scheme == g.SCHEME_HANCOCK_REF:  # the v_y slope is taken from the pressures
            a, b, z = (torch.stack([t[0], t[1], t[2], t[1], t[4], t[5], t[6]]) for t in (a, b, z))
        return h * _minmod((a - b) / h, (b - z) / h)

    def side(A, D):
        s = A + 0.5 * D
        return torch.where(pos & (s <= 0), A, s)

    def physical(s, axis):
        F = torch.stack(_mhd_side(_local(s, axis), cfg.gamma)[4][:7])
        return F if axis == 2 else torch.stack([F[0], F[1], F[3], F[2], F[5], F[4], F[6]])

    def centred(Q, DX, DY, y):
        d = 0.5 * dt * ((physical(side(Q, DX), 2) - physical(side(Q, -DX), 2)) / cfg.dx +
                        (physical(side(Q, DY), 1) - physical(side(Q, -DY), 1)) / cfg.dy)
        return 0.5 * (Q + _hancock_move(Q, d, cfg, 0.5 * dt / y, y, 0.000001))

    DX, DY = slope(c[2], c[1], c[4], cfg.dx), slope(c[5], c[1], c[3], cfg.dy)
    A = centred(c[1], DX, DY, Y)
    diff, fast = 0.0, {1: [], 2: []}
    # the four neighbours: the neighbour, its x slope, its y slope, its radius
    for k, sx, sy, y, axis, sgn in ((2, (6, 2, 1), (10, 2, 11), Y, 2, 1.0), (4, (1, 4, 8), (13, 4, 12), Y, 2, -1.0),
                                    (5, (10, 5, 13), (9, 5, 1), Y + cfg.dy, 1, 1.0),
                                    (3, (11, 3, 12), (1, 3, 7), Y - cfg.dy, 1, -1.0)):
        dx, dy = slope(*(c[i] for i in sx), cfg.dx), slope(*(c[i] for i in sy), cfg.dy)
        B = centred(c[k], dx, dy, y)
        own, other = side(A, sgn * (DX if axis == 2 else DY)), side(B, -sgn * (dx if axis == 2 else dy))
        F, UU = _flux(*((own, other) if sgn > 0 else (other, own)), axis, cfg)
        diff = diff + sgn * 0.5 * dt / (cfg.dx if axis == 2 else cfg.dy) * F
        fast[axis].append(torch.where(act, UU, torch.zeros_like(UU)).max())
    new = _hancock_move(A, diff, cfg, 0.5 * dt / Y, Y, 0.000001)
    return torch.where(act, new, q), _cfl(cfg, max(fast[2]), max(fast[1]))


SQRT_4PI = math.sqrt(4.0 * math.pi)


def _to_units(q, k):
    return q if len(q) == 4 else torch.cat([q[:4], q[4:] * k])


def _steps(q, cfg, n, dt=None):
    """n steps of the loop protocol (a step uses the CFL time step of the state before): the
    fields, the next time step, and the time steps used.  dt None: that of the input."""
    q = _to_units(q, 1.0 / SQRT_4PI)
    step = _tvd_step if cfg.scheme == g.SCHEME_TVD else _hancock_step
    if dt is None:
        dt = step(q, cfg, torch.zeros((), dtype=F64, device=q.device))[1]
    used = []
    for _ in range(n):
        used.append(dt)
        q, dt = step(q, cfg, dt)
    return _to_units(q, SQRT_4PI), dt, used


def exact(case, seed):
    grids = _inputs(case, seed)
    cfg, q = grids[0]
    n = case["steps"]
    if case["kind"] == "text":
        return _exact_text(cfg, q)
    if case["kind"] == "adjoint":
        q.requires_grad_(True)
        end, _, _ = _steps(q, cfg, n)
        grad, = torch.autograd.grad(end, q, _seeds_of_adjoint(case, seed, q))
        return _some(_aos(end.detach())) + _some(_aos(grad))
    with torch.no_grad():
        if case["kind"] == "batch":
            ends = [_aos(_steps(x, c, n)[0]) for c, x in grids]
            return [torch.cat([e[0] for e in ends]), torch.cat([e[1] for e in ends])]
        if case["kind"] in ("dropin", "host"):
            first = torch.tensor(_first_dt(cfg), dtype=F64, device="cuda")
            end, dt, used = _steps(q, cfg, n, first)
            if case["kind"] == "host":
                return [t.cpu() for t in _some(_aos(end))]
            # T is reset by the rotation; TT adds every new time step to its start
            T = torch.stack([torch.full_like(dt, 1e7), dt, first + sum(used[1:]) + dt])
            return _some(_aos(end)) + [T]
        return _some(_aos(_steps(q, cfg, n)[0]))


def _exact_text(cfg, q):
    k = cfg.N * cfg.M
    cols = np.zeros((k, 9))
    cols[:, 0] = np.tile(cfg.x0 + np.arange(cfg.N) * cfg.dx, cfg.M)
    cols[:, 1] = np.repeat(cfg.y0 + np.arange(cfg.M) * cfg.dy, cfg.N)
    cols[:, 2:2 + len(q)] = q.reshape(len(q), -1).T.cpu().numpy()
    words = [["%.6g" % x for x in row] for row in cols.tolist()]
    text = "".join(" ".join(row) + "\n" for row in words)
    back = torch.tensor([[float(w) for w in row[2:2 + len(q)]] for row in words], dtype=F64).T.contiguous()
    return [len(text)] + _some(_aos(back.reshape(q.shape).cuda()))
