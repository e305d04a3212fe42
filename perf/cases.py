"""The work that users have this framework do, as cases that can be timed and compared.

A case is a dict of plain values.  ``kind`` says which way the framework is used:

  step      a simulation on the device: the state set from device memory, ``steps`` time steps, the
            state read back into device memory
  coupled   a host model that keeps the state itself: the state in from pinned host memory, ``steps``
            steps (one, as a rule), the state out into pinned host memory
  ensemble  many simulations of uneven size stepped in the same launches
  gradient  one Manning calibration pass through torch.autograd: recording forward, backward
  descent   one iteration of a batched calibration on the device: forward, backward, zone
            gradient, projected descent

``gen`` names the generator of cuteflow_gb300.cases that makes the mesh (the mesh of a given size is
always the same one; the state, the weights and the Manning zones come from the seed).
"""
import functools
import math

import numpy as np
import torch

from cuteflow_gb300 import Adjoint, Batch, Solver, cases as gen, gauge_run
from cuteflow_gb300.adjoint import Zones


def listed():
    return [
        # a reach of the size of the reference's own calibration meshes (832 and 1408 triangles), in
        # the scheme that its runs use: thousands of short steps, nothing but latency
        dict(name="canal_1k", kind="step", gen="channel", nx=44, ny=16, iflux=2, inlet=2, steps=200, tuned=False),
        # a river reach settling towards a steady flow: discharge shared over the inlet by depth,
        # the steady-state test on
        dict(name="reach_6k_steady", kind="step", gen="channel", nx=121, ny=25, iflux=1, inlet=3, steps=100,
             tuned=False, steady=True),
        # the 200 m x 200 m circular dam break (80,000 triangles) as a first-time user runs it
        dict(name="dam_80k", kind="step", gen="dam", nx=200, ny=200, iflux=1, steps=100, tuned=False),
        # the same on a mesh of odd size, with the arithmetic setting that autotuning picks
        dict(name="dam_134k_tuned", kind="step", gen="dam", nx=317, ny=211, iflux=1, steps=100, tuned=True),
        # a small flood plain, second order, untuned
        dict(name="flood_25k", kind="step", gen="flood", nx=157, ny=81, iflux=3, ilimiteur=1, wet=0.5, steps=100,
             tuned=False),
        # a deeper flood with another limiter, mostly wet
        dict(name="flood_201k_deep", kind="step", gen="flood", nx=447, ny=225, iflux=3, ilimiteur=3, wet=1.0, steps=50,
             tuned=True),
        # the 1,000,000-triangle wet/dry flood of the benchmark
        dict(name="flood_1m", kind="step", gen="flood", nx=1000, ny=500, iflux=3, ilimiteur=1, wet=0.275, steps=50,
             tuned=True),
        # MUSCL-Hancock on a flood plain of odd size
        dict(name="muscl_201k", kind="step", gen="flood", nx=401, ny=251, iflux=4, ilimiteur=3, wet=0.4, steps=30,
             tuned=True),
        # a coupled model that exchanges the whole state every step
        dict(name="coupled_249k", kind="coupled", gen="flood", nx=501, ny=249, iflux=3, ilimiteur=1, wet=0.4,
             steps=1, tuned=True),
        # an ensemble over uneven flood plains, every member with its own state and time step
        dict(name="ensemble_6", kind="ensemble", members=6, nmin=5000, nmax=60000, iflux=3, wet=0.6,
             steps=40, tuned=True),
        # one gradient of a Manning calibration whose step records fit the memory budget
        dict(name="gradient_51k", kind="gradient", gen="calibration", nx=251, ny=101, zones=12, gauges=40, steps=50,
             budget_mb=4000, tuned=True),
        # one iteration of a batched calibration under sqrt(N) checkpointing, untuned
        dict(name="descent_3x", kind="descent", members=3, nmin=4000, nmax=16000, zones=8, gauges=20, steps=36,
             tuned=False),
    ]


def _size(rng, lo, hi, aspect=4.0):
    """nx, ny of a mesh of lo..hi triangles (spread over the logarithm), of any parity."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a = math.exp(rng.uniform(-0.5, 0.5) * math.log(aspect))
    ny = max(7, round(math.sqrt(n / 2 / a)))
    return max(7, round(n / 2 / ny)), ny


def draw(rng):
    kind = rng.choice(["canal", "reach", "dam", "dam", "flood", "flood", "flood", "muscl", "coupled", "ensemble",
                       "gradient", "descent"])
    tuned = rng.random() < 0.6
    if kind == "canal":
        nx, ny = _size(rng, 800, 20000, 16.0)
        return dict(kind="step", gen="channel", nx=nx, ny=ny, iflux=rng.choice([1, 2, 2]), inlet=2,
                    steps=rng.randint(50, 200), tuned=tuned)
    if kind == "reach":
        nx, ny = _size(rng, 2000, 40000, 16.0)
        return dict(kind="step", gen="channel", nx=nx, ny=ny, iflux=1, inlet=3, steps=rng.randint(30, 100),
                    tuned=tuned, steady=True)
    if kind == "dam":
        nx, ny = _size(rng, 3000, 400000)
        return dict(kind="step", gen="dam", nx=nx, ny=ny, iflux=1, steps=rng.randint(30, 100), tuned=tuned)
    if kind == "flood":
        nx, ny = _size(rng, 5000, 900000)
        return dict(kind="step", gen="flood", nx=nx, ny=ny, iflux=3, ilimiteur=rng.choice([1, 1, 2, 3, 4]),
                    wet=rng.choice([0.2, 0.3, 0.6, 1.0]), steps=rng.randint(20, 50), tuned=tuned)
    if kind == "muscl":
        nx, ny = _size(rng, 5000, 400000)
        return dict(kind="step", gen="flood", nx=nx, ny=ny, iflux=4, ilimiteur=rng.choice([1, 2, 3]),
                    wet=rng.choice([0.2, 0.6, 1.0]), steps=rng.randint(10, 30), tuned=tuned)
    if kind == "coupled":
        nx, ny = _size(rng, 20000, 900000)
        return dict(kind="coupled", gen="flood", nx=nx, ny=ny, iflux=rng.choice([1, 3]), ilimiteur=1, wet=rng.choice([0.3, 0.8]),
                    steps=rng.randint(1, 3), tuned=tuned)
    if kind == "ensemble":
        return dict(kind="ensemble", members=rng.randint(2, 8), nmin=rng.randint(2000, 8000),
                    nmax=rng.randint(20000, 90000), iflux=rng.choice([1, 3]), wet=rng.choice([0.3, 0.6, 1.0]),
                    steps=rng.randint(20, 40), tuned=tuned)
    if kind == "gradient":
        nx, ny = _size(rng, 4000, 60000)
        return dict(kind="gradient", gen="calibration", nx=nx, ny=ny, zones=rng.randint(4, 16),
                    gauges=rng.randint(10, 60), steps=rng.randint(16, 50), budget_mb=4000, tuned=tuned)
    return dict(kind="descent", members=rng.randint(2, 4), nmin=rng.randint(3000, 5000), nmax=rng.randint(8000, 16000),
                zones=rng.randint(4, 12), gauges=rng.randint(10, 30), steps=rng.randint(16, 36), tuned=tuned)


# ---- meshes and states --------------------------------------------------------------------------

_DEV = "cuda"


@functools.lru_cache(maxsize=8)
def _mesh(kind, nx, ny, iflux, ilimiteur, inlet, steady, wet, index):
    """A generator's case (its mesh and parameters), its elements' centroids and beds, and the level of
    its water (for a flood plain the level that leaves a share 1 - wet of it dry)."""
    if kind == "dam":
        c = gen.circular_dam_break(nx, ny, iflux=iflux)
    elif kind == "channel":
        c = gen.channel(nx, ny, lx=10.0 * nx, ly=10.0 * ny, iflux=iflux, inlet=inlet, slope=0.5 / (10.0 * nx))
    elif kind == "calibration":
        c = gen.circular_dam_break(nx, ny, seed=4, lx=2.0 * nx, ly=2.0 * ny)
    else:
        lx, ly = 2.0 * nx, 2.0 * ny
        c = gen.flooding(nx, ny, seed=2 + index, lx=lx, ly=ly, iflux=iflux,
                         nbumps=max(1, round(8.0 * lx * ly / 2.0e6)),
                         bump_scale=min(1.0, math.sqrt(lx * ly / 2.0e6)))
        c.params["ilimiteur"] = ilimiteur
    if steady:
        c.params["tol_reg_perm"] = 1e-7
    xc, yc = gen.cell_centroids(c.x, c.y, c.tri)
    zc, level = gen.cell_bed(c.x, c.y, c.z, c.tri), 1.0
    if kind == "flood":
        level = float(np.quantile(zc, wet)) + (1.0 if wet == 1.0 else 0.0)
        c.params["h_sortie"] = [level]
    return c, xc / c.x.max(), yc / c.y.max(), zc, level


def _mesh_of(case):
    return _mesh(case["gen"], case["nx"], case["ny"], case.get("iflux", 1), case.get("ilimiteur", 1),
                 case.get("inlet", 2), bool(case.get("steady")), case.get("wet", 1.0), 0)


def _waves(x, y, rng):
    """A smooth field of a few waves, values within +-1."""
    f = np.zeros_like(x)
    for _ in range(3):
        a, b = rng.uniform(1.0, 9.0, 2)
        f += np.sin(a * x + rng.uniform(0, 6.28)) * np.cos(b * y + rng.uniform(0, 6.28))
    return f / 3.0


def _state(mesh, kind, seed):
    """(h, hu, hv) per element: a flow under way over the mesh's bed."""
    c, x, y, zc, level = mesh
    rng = np.random.default_rng(seed)
    U = np.zeros((c.nelt, 3))
    if kind in ("dam", "calibration"):
        cx, cy = rng.uniform(0.4, 0.6, 2)
        lx, ly = c.x.max(), c.y.max()
        r = min(lx, ly) * rng.uniform(0.2, 0.3)
        inside = ((x - cx) * lx) ** 2 + ((y - cy) * ly) ** 2 < r * r
        h = np.where(inside, rng.uniform(6.0, 10.0), rng.uniform(1.0, 2.0)) * (1.0 + 0.05 * _waves(x, y, rng))
    else:
        h = level + 0.03 * _waves(x, y, rng) - zc
        h = np.where(h > 2e-3, h, 0.0)
    U[:, 0] = h
    U[:, 1] = h * 0.1 * _waves(x, y, rng)
    U[:, 2] = h * 0.1 * _waves(x, y, rng)
    return U


def _member_sizes(case):
    """The sizes of an ensemble's members, spread unevenly over nmin..nmax."""
    n, out = case["members"], []
    for m in range(n):
        t = case["nmin"] * (case["nmax"] / case["nmin"]) ** (((m + 0.5) / n) ** 1.5)
        ny = max(7, round(math.sqrt(t / 2 / (0.7 + 0.3 * (m % 4)))))
        out.append((max(7, round(t / 2 / ny)), ny))
    return out


def _zone_case(mesh, nzones, ngauges, seed):
    """Manning zones of seeded sites, their values, and gauge elements."""
    c, x, y, _, _ = mesh
    rng = np.random.default_rng(seed + 101)
    s = rng.uniform(0.0, 1.0, (nzones, 2))
    zones = np.argmin((x[:, None] - s[:, 0]) ** 2 + (y[:, None] - s[:, 1]) ** 2, axis=1).astype(np.int32)
    return zones, rng.uniform(0.02, 0.06, nzones), np.sort(rng.choice(c.nelt, ngauges, replace=False)).astype(np.int32)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(_DEV)


# ---- the five uses --------------------------------------------------------------------------------

def _tune(solver, case):
    if case["tuned"]:
        solver.set_tuning(1, 0x1F)   # the setting that autotuning picks on these schemes


def _calibration_meshes(case):
    return [_mesh("calibration", nx, ny, 1, 1, 2, False, 1.0, 0) for nx, ny in _member_sizes(case)]


def prepare(case, seed):
    kind, st = case["kind"], {"case": case}
    if kind in ("step", "coupled"):
        mesh = _mesh_of(case)
        U0 = _state(mesh, case["gen"], seed)
        s = st["solver"] = Solver(mesh[0])
        _tune(s, case)
        if kind == "step":
            st["U0"], st["out"] = _dev(U0), torch.empty(U0.shape, dtype=torch.float64, device=_DEV)
        else:
            st["U0"] = torch.from_numpy(U0).pin_memory().numpy()
            st["out"] = torch.empty(U0.shape, dtype=torch.float64).pin_memory().numpy()
    elif kind == "ensemble":
        meshes = [_mesh("flood", nx, ny, case["iflux"], 1, 2, False, case["wet"], m)
                  for m, (nx, ny) in enumerate(_member_sizes(case))]
        st["solver"] = Batch([m[0] for m in meshes])
        _tune(st["solver"], case)
        st["U0"] = [_state(m, "flood", seed + 31 * i) for i, m in enumerate(meshes)]
    elif kind == "gradient":
        mesh = _mesh_of(case)
        zones, nz, gauges = _zone_case(mesh, case["zones"], case["gauges"], seed)
        s = st["solver"] = Solver(mesh[0])
        _tune(s, case)
        st["adjoint"] = Adjoint(s, case["steps"], gauges, budget_bytes=case["budget_mb"] << 20)
        st["U0"] = _dev(_state(mesh, "calibration", seed)).requires_grad_()
        st["n"] = _dev(nz[zones]).requires_grad_()
        st["w"] = _weights(case["steps"], gauges.size, mesh[0].nelt, seed)
    else:
        meshes = _calibration_meshes(case)
        parts = [_zone_case(m, case["zones"], case["gauges"], seed + 7 * i) for i, m in enumerate(meshes)]
        b = st["solver"] = Batch([m[0] for m in meshes])
        _tune(b, case)
        nz = case["zones"]
        st["zones"] = Zones(b, np.concatenate([z + nz * i for i, (z, _, _) in enumerate(parts)]), nz * len(parts))
        st["values"] = _dev(np.concatenate([v for _, v, _ in parts]))
        member = np.concatenate([np.full(g.size, i, np.int32) for i, (_, _, g) in enumerate(parts)])
        gauges = np.concatenate([g for _, _, g in parts])
        st["adjoint"] = Adjoint(b, case["steps"], gauges, gauge_member=member)
        st["U0"] = [_state(m, "calibration", seed + 31 * i) for i, m in enumerate(meshes)]
        n = sum(b.nelt)
        st["w"] = _weights(case["steps"], gauges.size, n, seed)
        f = dict(dtype=torch.float64, device=_DEV)
        st["buf"] = [torch.empty(case["steps"], gauges.size, **f), torch.empty(n, 3, **f), torch.empty(n, 3, **f),
                     torch.empty(n, **f), torch.empty(nz * len(parts), **f)]
    return st


def _weights(steps, ngauges, nelt, seed):
    """The derivatives of a misfit with respect to the gauge elevations and the final state."""
    rng = np.random.default_rng(seed + 202)
    we = rng.normal(size=(steps, ngauges)) * (np.arange(steps) % 5 == 4)[:, None]
    return _dev(we), _dev(rng.normal(size=(nelt, 3)) * 1e-3)


def run(st):
    case, s = st["case"], st["solver"]
    kind, n = case["kind"], case["steps"]
    if kind == "step":
        s.set_state_device(st["U0"].data_ptr())
        info = s.step(n)
        s.get_state_device(st["out"].data_ptr())
        return st["out"], info.t, info.dt_next
    if kind == "coupled":
        s.set_state(st["U0"])
        info = s.step(n)
        return s.get_state(st["out"]), info.t, info.dt_next
    if kind == "ensemble":
        for m, U in enumerate(st["U0"]):
            s.set_state(m, U)
        infos = s.step(n)
        return [s.get_state(m) for m in range(s.members)], [i.dt_next for i in infos]
    if kind == "gradient":
        eta, UN = gauge_run(st["adjoint"], st["n"], st["U0"])
        gn, gU = torch.autograd.grad((eta, UN), (st["n"], st["U0"]), st["w"])
        return eta.detach(), UN.detach(), gn, gU
    adj, zones = st["adjoint"], st["zones"]
    eta, UN, gU, gn, gz = st["buf"]
    zones.set(st["values"])
    for m, U in enumerate(st["U0"]):
        s.set_state(m, U)
    adj.forward(eta=eta, state=UN)
    adj.backward(st["w"][0], st["w"][1], gU, gn)
    zones.gradient(adj, gz)
    zones.descend(1e-9, 0.005, 0.2)
    return eta, UN, gU, gn, gz, zones.get()[0]


def _triangles(case):
    if case["kind"] in ("ensemble", "descent"):
        return sum(2 * nx * ny for nx, ny in _member_sizes(case))
    return 2 * case["nx"] * case["ny"]


def work(case):
    """Per triangle and step: state in and out, statics, neighbour ids, edge geometry and centroids
    (144 bytes); the scheme's sums, products, quotients and roots, each one operation.  A gradient
    reads the run's record back and differentiates every operation (three for one)."""
    n, steps = _triangles(case), case["steps"]
    flops = {1: 260, 2: 300, 3: 480, 4: 900}[case.get("iflux", 1)]
    grad = case["kind"] in ("gradient", "descent")
    b = 144 + (80 + 80 + 144 if grad else 0)
    io = 48 * n
    return {"bytes": float(n * steps * b + io), "flops": float(n * steps * flops * (4 if grad else 1))}


# ---- the first-order scheme between walls, in plain torch -----------------------------------------
#
# Only the first-order HLLC scheme has a value that any accurate evaluation comes to.  The others
# jump at the last bit (WAF: the sign of a depth difference of zero picks the limiter's branch; the
# star-state HLLC: an exact zero of the contact speed picks the side; MUSCL: limiter branches), so
# for them there is no such value.

def exact(case, seed):
    kind = case["kind"]
    if kind == "step" and case["gen"] == "dam":
        mesh = _mesh_of(case)
        T = _topology(mesh[0])
        U = _dev(_state(mesh, "dam", seed))
        n = _dev(np.asarray(mesh[0].manning, dtype=np.float64))
        t = 0.0
        with torch.no_grad():
            dt = _cfl(U, T)
            for _ in range(case["steps"]):
                U = _step(U, n, dt, T)
                t, dt = t + float(dt), _cfl(U, T)
        return U, t, float(dt)
    if kind == "gradient":
        mesh = _mesh_of(case)
        zones, nz, gauges = _zone_case(mesh, case["zones"], case["gauges"], seed)
        w = _weights(case["steps"], gauges.size, mesh[0].nelt, seed)
        return _gradient(mesh, _dev(nz[zones]), _dev(_state(mesh, "calibration", seed)), gauges, w, case["steps"])
    if kind == "descent":
        meshes = _calibration_meshes(case)
        parts = [_zone_case(m, case["zones"], case["gauges"], seed + 7 * i) for i, m in enumerate(meshes)]
        we, ws = _weights(case["steps"], sum(g.size for _, _, g in parts), sum(m[0].nelt for m in meshes), seed)
        got, gz, g0, e0 = [], [], 0, 0
        for i, (m, (zones, v, gauges)) in enumerate(zip(meshes, parts)):
            g1, e1 = g0 + gauges.size, e0 + m[0].nelt
            r = _gradient(m, _dev(v[zones]), _dev(_state(m, "calibration", seed + 31 * i)), gauges,
                          (we[:, g0:g1], ws[e0:e1]), case["steps"])
            got.append(r)
            gz.append(torch.zeros(case["zones"], dtype=torch.float64, device=r[2].device).index_add_(
                0, _dev(zones.astype(np.int64)), r[2]))
            g0, e0 = g1, e1
        gz = torch.cat(gz)
        vals = torch.clamp(_dev(np.concatenate([v for _, v, _ in parts])) - 1e-9 * gz, 0.005, 0.2)
        return (torch.cat([r[0] for r in got], 1), torch.cat([r[1] for r in got]), torch.cat([r[3] for r in got]),
                torch.cat([r[2] for r in got]), gz, vals)
    return None


_G = 9.81


def _topology(c):
    """Per (element, local edge): the element across (itself at a wall), normal out, length; areas."""
    t = c.tri.astype(np.int64) - 1
    n = t.shape[0]
    a, b = t.ravel(), t[:, [1, 2, 0]].ravel()
    key = np.minimum(a, b) * c.nnt + np.maximum(a, b)
    order = np.argsort(key, kind="stable")
    twin = np.full(3 * n, -1)
    pair = np.nonzero(key[order][1:] == key[order][:-1])[0]
    twin[order[pair]], twin[order[pair + 1]] = order[pair + 1], order[pair]
    wall = twin < 0
    nbr = np.where(wall, np.arange(3 * n), twin) // 3
    dx, dy = c.x[b] - c.x[a], c.y[b] - c.y[a]
    ln = np.hypot(dx, dy)
    L = ln.reshape(n, 3)
    p = L.sum(1) / 2
    area = np.sqrt(p * (p - L[:, 0]) * (p - L[:, 1]) * (p - L[:, 2]))
    return dict(nbr=_dev(nbr), wall=_dev(wall), nx=_dev(dy / ln), ny=_dev(-dx / ln), ln=_dev(ln), area=_dev(area),
                cfl=_dev(c.params["cfl"] * float(np.float32(1.8)) * 0.5 * area / p))


def _cfl(U, T):
    h, u, v = U[:, 0], U[:, 1] / U[:, 0], U[:, 2] / U[:, 0]
    return (T["cfl"] / torch.clamp(torch.sqrt(u * u + v * v) + torch.sqrt(_G * h), min=0.01)).min().detach()


def _step(U, n, dt, T):
    own = torch.arange(3 * U.shape[0], device=U.device) // 3
    nx, ny = T["nx"], T["ny"]

    def frame(q):
        return q[:, 0], (q[:, 1] * nx + q[:, 2] * ny) / q[:, 0], (q[:, 2] * nx - q[:, 1] * ny) / q[:, 0]

    (hl, ul, vl), (hr, ur, vr) = frame(U[own]), frame(U[T["nbr"]])
    al, ar = torch.sqrt(_G * hl), torch.sqrt(_G * hr)
    he = (hl + hr) / 2 - (ur - ul) * (hl + hr) / (al + ar) / 4

    def strength(h):
        low = he < h
        x = torch.where(low, torch.ones_like(h), (he + h) / 2 * he / (h * h))
        return torch.where(low, torch.ones_like(h), torch.sqrt(x))

    sl, sr = ul - al * strength(hl), ur + ar * strength(hr)
    ss = (sl * hr * (ur - sr) - sr * hl * (ul - sl)) / (hr * (ur - sr) - hl * (ul - sl))
    f1, f2 = hl * ul, hl * ul * ul + _G * hl * hl / 2
    g1, g2 = hr * ur, hr * ur * ur + _G * hr * hr / 2
    den = sr - sl + float(np.float32(1e-8))
    m1 = (sr * f1 - sl * g1 + sl * sr * (hr - hl)) / den
    m2 = (sr * f2 - sl * g2 + sl * sr * (hr * ur - hl * ul)) / den
    left, right = sl > 0, sr < 0
    x1 = torch.where(left, f1, torch.where(right, g1, m1))
    x2 = torch.where(left, f2, torch.where(right, g2, m2))
    x3 = x1 * torch.where(left, vl, torch.where(right, vr, torch.where(ss > 0, vl, vr)))
    p = _G * hl * hl / 2
    zero = torch.zeros_like(p)
    w = T["wall"]
    flux = torch.stack([torch.where(w, zero, x1), torch.where(w, nx * p, nx * x2 - ny * x3),
                        torch.where(w, ny * p, ny * x2 + nx * x3)], 1) * T["ln"][:, None]
    R = -flux.reshape(-1, 3, 3).sum(1) / T["area"][:, None]
    # Manning friction with the semi-implicit matrix
    h = U[:, 0]
    u, v = U[:, 1] / h, U[:, 2] / h
    tol = float(np.float32(1e-6))
    s2 = u * u + v * v
    fast = s2 > tol * tol
    s = torch.where(fast, torch.sqrt(torch.where(fast, s2, torch.ones_like(s2))), torch.full_like(s2, tol))
    p13 = h ** (-1.0 / 3.0)
    k = _G * n * n * s * p13
    r2, r3 = R[:, 1] - k * u, R[:, 2] - k * v
    d = torch.where(fast, dt / 2 * _G * n * n * p13 / h, torch.zeros_like(h))
    a21, a31 = -7.0 / 3.0 * d * u * s, -7.0 / 3.0 * d * v * s
    a22, a33 = 1 + d * (2 * u * u + v * v) / s, 1 + d * (u * u + 2 * v * v) / s
    a23 = d * u * v / s
    det = a22 * a33 - a23 * a23
    r1 = R[:, 0]
    q2 = (-(a21 * a33 - a23 * a31) * r1 + a33 * r2 - a23 * r3) / det
    q3 = ((a21 * a23 - a22 * a31) * r1 - a23 * r2 + a22 * r3) / det
    return U + dt * torch.stack([r1, q2, q3], 1)


def _gradient(mesh, n, U0, gauges, w, steps):
    """eta, the final state and the gradients of the weighted sums, every dt held."""
    T = _topology(mesh[0])
    g, z = _dev(gauges.astype(np.int64)), _dev(mesh[3][gauges])
    n, U0 = n.requires_grad_(), U0.requires_grad_()
    U, eta = U0, []
    dt = _cfl(U0.detach(), T)
    for _ in range(steps):
        U = _step(U, n, dt, T)
        dt = _cfl(U.detach(), T)
        eta.append(U[g, 0] + z)
    eta = torch.stack(eta)
    gn, gU = torch.autograd.grad((eta, U), (n, U0), w)
    return eta.detach(), U.detach(), gn, gU
