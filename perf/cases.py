"""Workloads of the explicit shallow-water step, as a program that uses the
package runs them: ``listed()`` names a fixed set, ``draw(rng)`` gives more of
the same ranges, ``prepare`` makes the inputs and the context, ``run`` is one
pass through the public entry points, ``work`` the bytes and operations that
pass cannot do without, ``exact`` the same pass in plain torch at 64 bits.

Ways of using the step (``way``):

* ``device``   the state lives on the GPU: upload_device, rk3_steps,
               download_device (a solver inside a larger GPU program);
* ``host``     rk3_steps_host on numpy arrays (the README's time loop);
* ``percall``  the drop-in operators compute_dij and euler on host arrays, with
               the SSP-RK3 combinations and the boundary data on the host (the
               reference's own time loop, needed wherever boundary data change
               with time).

Flows (``flow``): ``dam`` (dam break over a flat bottom, no friction),
``basin`` (wet/dry basin with Gaussian bumps and Manning friction),
``thacker`` (paraboloid with a moving shoreline and imposed boundary values),
``sgn`` (hyperbolised Serre-Green-Naghdi solitary wave in a channel, five
unknowns), ``ensemble`` (independent dam breaks of many sizes in one batch).

Meshes are jittered lattices whose cells are cut along a random diagonal, so
rows have 2 to 8 neighbours like an unstructured triangulation's; the channel
is a plain lattice.
"""
import math
import os
import sys
from dataclasses import replace

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "shallow-water-eric_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from swe.cases import Params  # noqa: E402
from swe.update import Update  # noqa: E402

FP64, MIXED, SPLIT = 0, 1, 2
VISC = {"viscous": 1, "entropy_visc": 2, "fct": 3}
GRAVITY = 9.81


def _case(name, flow, nx, ny, precision, steps, way="device", visc="fct", instances=1):
    return {"name": name, "flow": flow, "nx": nx, "ny": ny, "precision": precision, "steps": steps, "way": way,
            "visc": visc, "instances": instances}


def listed():
    return [
        # one time step of a small mesh (the size of the reference's shipped ones) through the host-array
        # operators: the smallest calls a program makes
        _case("percall_2k_f64", "basin", 45, 45, FP64, 1, way="percall"),
        # the same operators on a mesh of a regional study, boundary data changed on the host between stages
        _case("percall_50k_f64", "basin", 223, 227, FP64, 1, way="percall"),
        # the unit-square dam break in the default (bit-exact) precision
        _case("dam_10k_f64", "dam", 101, 101, FP64, 16),
        # the same in mixed precision, a stretch of a run between two looks at the state
        _case("dam_10k_mixed", "dam", 101, 101, MIXED, 40),
        # a moving shoreline at a mesh of ordinary size, odd node counts
        _case("thacker_103k_mixed", "thacker", 321, 321, MIXED, 10),
        # mixed precision with the FP64 limiter, steps that leave a remainder of the captured eight
        _case("basin_260k_split", "basin", 511, 509, SPLIT, 9),
        # the bit-exact precision at a large mesh: verification runs
        _case("basin_1m_f64", "basin", 1000, 1000, FP64, 2),
        # the largest single mesh: a production run
        _case("basin_4m_mixed", "basin", 2000, 2000, MIXED, 8),
        # five unknowns, long channel, production precision
        _case("sgn_2m_mixed", "sgn", 10001, 201, MIXED, 8),
        # five unknowns in the bit-exact precision, the reference's own kind of channel run
        _case("sgn_100k_f64", "sgn", 1001, 101, FP64, 4),
        # many independent scenarios at once (2k to 50k nodes each)
        _case("ensemble_48_mixed", "ensemble", 45, 1118, MIXED, 8, instances=48),
        # host arrays in, ten steps, host arrays out
        _case("host_1m_mixed", "basin", 1000, 1000, MIXED, 10, way="host"),
    ]


#: node-stages (nodes x 3 stages x steps) of the largest listed cases, by precision
_MOST = {FP64: 6.0e6, MIXED: 9.6e7, SPLIT: 9.6e7}


def draw(rng):
    flow = rng.choice(["dam", "dam", "basin", "basin", "basin", "thacker", "sgn", "ensemble"])
    precision = rng.choice([FP64, MIXED, MIXED, SPLIT])
    way = rng.choice(["device", "device", "device", "host", "percall"])
    visc = rng.choice(["fct", "fct", "fct", "viscous", "entropy_visc"])
    if flow != "dam":
        visc = "fct"
    if flow == "ensemble" and way == "percall":
        way = "device"
    if way == "percall":
        precision, steps = FP64, 1
        most = 6.0e4                            # host arrays cross at every call
    else:
        steps = rng.choice([1, 2, 3, 4, 5, 7, 8, 9, 10, 16, 25])
        most = _MOST[precision] / (3 * steps) * (0.75 if flow == "sgn" else 1.0)   # five unknowns cost more
    if way == "host":
        most = min(most, 1.0e6)
    if flow == "ensemble":
        instances = rng.randint(3, 48)
        top = max(2.1e3, min(5.0e4, 3.5 * most / instances))
        nx, ny = 45, int(top / 45) + 1           # 45 x 45 nodes the smallest, nx * ny the largest
        return {k: v for k, v in _case("", flow, nx, ny, precision, steps, way, visc, instances).items()
                if k != "name"}
    n = math.exp(rng.uniform(math.log(2.0e3), math.log(max(2.1e3, 0.98 * most))))
    aspect = rng.uniform(20.0, 60.0) if flow == "sgn" else (1.0 if flow == "thacker" else rng.uniform(0.7, 1.5))
    nx = max(5, int(math.sqrt(n * aspect)))
    ny = nx if flow == "thacker" else max(5, int(n / nx))
    return {k: v for k, v in _case("", flow, nx, ny, precision, steps, way, visc).items() if k != "name"}


# ------------------------------------------------------------------ inputs
def _mesh(nx, ny, lx, ly, rng, jitter=0.2, random_diagonals=True):
    """jj (3, me) 1-based counter-clockwise, rr (2, np), and the boundary's
    node lists (x sides, y sides), 0-based."""
    dx, dy = lx / (nx - 1), ly / (ny - 1)
    X = np.broadcast_to(np.linspace(0.0, lx, nx), (ny, nx)).copy()
    Y = np.broadcast_to(np.linspace(0.0, ly, ny)[:, None], (ny, nx)).copy()
    if jitter:
        X[1:-1, 1:-1] += rng.uniform(-jitter, jitter, (ny - 2, nx - 2)) * dx
        Y[1:-1, 1:-1] += rng.uniform(-jitter, jitter, (ny - 2, nx - 2)) * dy
    rr = np.empty((nx * ny, 2))
    rr[:, 0], rr[:, 1] = X.ravel(), Y.ravel()
    sw = (np.arange(ny - 1, dtype=np.int32)[:, None] * nx + np.arange(nx - 1, dtype=np.int32)).ravel() + 1
    se, nw, ne = sw + 1, sw + nx, sw + nx + 1
    up = rng.random(sw.size) < 0.5 if random_diagonals else np.ones(sw.size, bool)
    jj = np.empty((sw.size, 2, 3), np.int32)     # up: cut SW-NE, else SE-NW
    jj[:, 0, 0], jj[:, 0, 1], jj[:, 0, 2] = sw, se, np.where(up, ne, nw)
    jj[:, 1, 0], jj[:, 1, 1], jj[:, 1, 2] = np.where(up, sw, se), ne, nw
    xs = np.concatenate([np.arange(ny) * nx, np.arange(ny) * nx + nx - 1])
    ys = np.concatenate([np.arange(nx), np.arange(nx) + nx * (ny - 1)])
    return jj.reshape(-1, 3).T, rr.T, xs, ys


def _swell(rr, rng, lx, ly, amp):
    """A few long waves: a smooth field of the given amplitude."""
    s = np.zeros(rr.shape[1])
    for _ in range(3):
        kx, ky = rng.uniform(1.0, 6.0, 2) * 2 * math.pi / np.array([lx, ly])
        s += np.sin(kx * rr[0] + ky * rr[1] + rng.uniform(0.0, 2 * math.pi))
    return amp / 3.0 * s


def _scene(case, rng, nx, ny):
    """One mesh with its bathymetry, parameters, initial state (N, S) and the
    imposed boundary values [(component, 0-based nodes, values)]."""
    flow, prec, visc = case["flow"], case["precision"], VISC[case["visc"]]
    if flow in ("dam", "ensemble"):
        lx = 1.0 if flow == "dam" else rng.uniform(1.0, 4.0)
        jj, rr, xs, ys = _mesh(nx, ny, lx, 1.0, rng)
        hu = rng.uniform(0.9, 1.1) if flow == "dam" else rng.uniform(0.5, 2.0)
        hd = rng.uniform(0.08, 0.12) if flow == "dam" else rng.uniform(0.0, 0.2)
        h = np.where(rr[0] < 0.5 * lx, hu, hd) * (1.0 + _swell(rr, rng, lx, 1.0, 0.02))
        qx = 0.1 * h * _swell(rr, rng, lx, 1.0, 1.0)
        qy = 0.1 * h * _swell(rr, rng, lx, 1.0, 1.0)
        z = np.zeros_like(h)
        p = Params(gravity=GRAVITY, cfl=0.25, max_water_h=hu, htiny=1e-4 * hu, viscosity_type=visc, precision=prec,
                   type_test=4 if flow == "dam" else 10, mannings=0.0 if flow == "dam" else rng.uniform(0.01, 0.05))
        u = np.stack([h, qx, qy], 1)
        bc = [(1, xs, np.zeros(xs.size)), (2, ys, np.zeros(ys.size))]
    elif flow == "basin":
        L = 10.0
        jj, rr, xs, ys = _mesh(nx, ny, L, L, rng)
        z = np.zeros(rr.shape[1])
        for _ in range(16):
            a, w, c = rng.uniform(0.1, 0.8), rng.uniform(0.2, 1.5), rng.uniform(0.0, L, 2)
            z += a * np.exp(-((rr[0] - c[0]) ** 2 + (rr[1] - c[1]) ** 2) / w ** 2)
        eta = np.where((rr[0] - 5.0) ** 2 + (rr[1] - 5.0) ** 2 < 1.0, 1.5, 0.5) + _swell(rr, rng, L, L, 0.02)
        h = np.maximum(eta - z, 0.0)
        qx = 0.2 * h * _swell(rr, rng, L, L, 1.0)
        qy = 0.2 * h * _swell(rr, rng, L, L, 1.0)
        mwh = float(h.max())
        p = Params(gravity=GRAVITY, cfl=0.25, max_water_h=mwh, htiny=1e-4 * mwh, mannings=0.03, type_test=10,
                   viscosity_type=visc, precision=prec)
        u = np.stack([h, qx, qy], 1)
        bc = [(1, xs, np.zeros(xs.size)), (2, ys, np.zeros(ys.size))]
    elif flow == "thacker":
        a, h0, hL, ecc = 1.0, 0.1, 4.0, rng.uniform(0.4, 0.5)
        jj, rr, xs, ys = _mesh(nx, ny, hL, hL, rng)
        om = math.sqrt(2 * GRAVITY * h0) / a
        ph = rng.uniform(0.0, 2 * math.pi)
        X, Y = rr[0] - hL / 2, rr[1] - hL / 2
        z = -h0 * (1.0 - (X ** 2 + Y ** 2) / a ** 2)
        wet = np.maximum(ecc * h0 / a ** 2 * (2 * X * math.cos(ph) + 2 * Y * math.sin(ph)) - z, 0.0)
        p = Params(gravity=GRAVITY, cfl=0.2, max_water_h=hL, htiny=1e-4 * hL, type_test=5, viscosity_type=visc,
                   precision=prec)
        u = np.stack([wet + p.htiny, -ecc * om * math.sin(ph) * wet, ecc * om * math.cos(ph) * wet], 1)
        js = np.unique(np.concatenate([xs, ys]))
        bc = [(k, js, u[js, k].copy()) for k in range(3)]
    else:
        h1, h2, Lx, Ly = 1.0, rng.uniform(1.1, 1.2), 0.01 * (nx - 1), 0.01 * (ny - 1)
        jj, rr, xs, ys = _mesh(nx, ny, Lx, Ly, rng, jitter=0.0, random_diagonals=False)
        D = math.sqrt(GRAVITY * h2)
        k = math.sqrt(3.0 * (h2 - h1) / (h2 * h1 ** 2))
        arg = 0.5 * k * (rr[0] - rng.uniform(0.2, 0.5) * Lx)
        sech2 = (1.0 / np.cosh(arg)) ** 2
        h = h1 + (h2 - h1) * sech2
        z = np.zeros_like(h)
        p = Params(gravity=GRAVITY, cfl=5e-4, max_water_h=h2, htiny=1e-4 * h2, lambda_sgn=100.0, type_test=13,
                   syst_size=5, viscosity_type=visc, precision=prec)
        u = np.stack([h, h * D - h1 * D, 0.0 * h, h * h, -D * h1 * ((h1 - h2) * k * sech2 * np.tanh(arg))], 1)
        bc = [(2, ys, np.zeros(ys.size))]
    return {"jj": jj, "rr": rr, "z": z, "p": p, "u": u, "bc": [(k, np.unique(j), v[np.unique(j, return_index=True)[1]])
                                                           for k, j, v in bc]}


def _instances(case):
    """(nx, ny) of an ensemble's instances: node counts spread over their range in the logarithm, aspect ratios
    between 1 and 4, neighbours in the batch of unlike size."""
    lo, hi = 45 * 45, max(45 * 45 + 1, case["nx"] * case["ny"])
    n = case["instances"]
    out = []
    for b in range(n):
        size = lo * (hi / lo) ** (((b * 29) % n + 0.25) / n)
        ny = max(5, int(math.sqrt(size / (1.0 + 3.0 * ((b * 0.618) % 1.0)))))
        out.append((max(5, int(size / ny)), ny))
    return out


def _scenes(case, seed):
    rng = np.random.default_rng(seed)
    if case["flow"] != "ensemble":
        return [_scene(case, rng, case["nx"], case["ny"])]
    return [_scene(case, rng, nx, ny) for nx, ny in _instances(case)]


def prepare(case, seed):
    scenes = _scenes(case, seed)
    upd = Update(batch=[({"jj": s["jj"], "rr": s["rr"]}, s["z"], s["p"]) for s in scenes])
    for b, s in enumerate(scenes):
        for comp, nodes, vals in s["bc"]:
            upd.set_dirichlet(comp, nodes + 1, vals, inst=b)
    u0 = np.concatenate([s["u"] for s in scenes])            # (N, S): the columns of un(S, N)
    state = {"way": case["way"], "steps": case["steps"], "upd": upd, "p": scenes[0]["p"], "bc": scenes[0]["bc"]}
    if case["way"] == "device":
        state["u0"] = torch.from_numpy(u0).cuda()
        state["out"] = torch.empty_like(state["u0"])
    else:
        state["u0"] = u0.T                                   # (S, N), Fortran order
    return state


def _impose(u, bc):
    for comp, nodes, vals in bc:
        u[comp, nodes] = vals


def run(state):
    upd, steps = state["upd"], state["steps"]
    if state["way"] == "device":
        upd.set_time(0.0, 1e30)
        upd.upload_device(state["u0"].data_ptr())
        t, dt, n = upd.rk3_steps(steps)
        upd.download_device(state["out"].data_ptr())
        return {"u": state["out"], "t": t, "dt": dt, "steps": n}
    if state["way"] == "host":
        upd.set_time(0.0, 1e30)
        u = upd.rk3_steps_host(state["u0"], steps)
        t, _, dt = upd.get_time()
        return {"u": u.T, "t": t, "dt": dt}
    # percall: the reference's time loop on the host around the operators
    uo, t = state["u0"], 0.0
    for _ in range(steps):
        dij, dt = upd.compute_dij(uo)
        upd.set_params(replace(state["p"], dt=dt))
        un = upd.euler(uo)
        _impose(un, state["bc"])
        ui = upd.euler(un)
        un = (3 * uo + ui) / 4
        _impose(un, state["bc"])
        ui = upd.euler(un)
        un = (uo + 2 * ui) / 3
        _impose(un, state["bc"])
        uo, t = un, t + dt
    return {"u": np.ascontiguousarray(uo.T), "t": t, "dt": dt, "dij": dij}


# ------------------------------------------------------------------ work
def _sizes(case):
    """Nodes and off-diagonal graph entries of the case."""
    if case["flow"] == "ensemble":
        pairs = _instances(case)
        return (sum(nx * ny for nx, ny in pairs),
                sum(2 * ((nx - 1) * ny + nx * (ny - 1) + (nx - 1) * (ny - 1)) for nx, ny in pairs))
    nx, ny = case["nx"], case["ny"]
    return nx * ny, 2 * ((nx - 1) * ny + nx * (ny - 1) + (nx - 1) * (ny - 1))


def work(case):
    """Compulsory bytes of the stages (per stage: the state and the stage's
    start state in, the new state out, bathymetry, mass and a row pointer per
    node, a column index and c_ij per entry), and a count of the scheme's
    arithmetic (per entry and stage: hydrostatic reconstruction, viscosities,
    low-order and Galerkin rows, antidiffusion, limiter and update, plus the
    wave-speed bound once per stage; per node: flux, residual, limiter,
    update)."""
    n, e = _sizes(case)
    S = 5 if case["flow"] == "sgn" else 3
    word = 8 if case["precision"] == FP64 else 4
    state = 8 + word * (S - 1)                   # the depth is held in 8 bytes in every precision
    stages = 3 * case["steps"]
    per_stage = n * (3 * state + 2 * word + 4) + (n + e) * (4 + 2 * word)
    moved = stages * per_stage
    if case["way"] != "device":                  # host arrays: the state in FP64 in and out of each call
        calls = 1 if case["way"] == "host" else 4 * case["steps"]
        moved += calls * 2 * 8 * S * n
    return {"bytes": moved, "flops": stages * (e * (100 + 25 * S) + n * (40 + 20 * S))}


# ------------------------------------------------------------------ 64-bit reference in plain torch
class _Plain:
    """The scheme over directed edges (i, j), i != j, with the diagonal's own
    terms per node; sums by index_add."""

    def __init__(self, scene, dev):
        p = self.p = scene["p"]
        f = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        rr = f(scene["rr"].T)
        el = f(scene["jj"].T.astype(np.int64)) - 1
        self.n = n = rr.shape[0]
        self.z = f(scene["z"])
        a, b, c = rr[el[:, 0]], rr[el[:, 1]], rr[el[:, 2]]
        two_area = (b[:, 0] - a[:, 0]) * (c[:, 1] - a[:, 1]) - (b[:, 1] - a[:, 1]) * (c[:, 0] - a[:, 0])
        # area * grad(phi_k) = rotated opposite edge / 2
        opp = [c - b, a - c, b - a]
        ag = [torch.stack([-o[:, 1], o[:, 0]], 1) / 2 for o in opp]
        self.m = torch.zeros(n, dtype=torch.float64, device=dev)
        self.cd = torch.zeros(n, 2, dtype=torch.float64, device=dev)
        keys, vals = [], []
        for k in range(3):
            self.m.index_add_(0, el[:, k], two_area / 6)
            self.cd.index_add_(0, el[:, k], ag[k] / 3)
            for q in range(3):
                if q != k:
                    keys.append(el[:, k] * n + el[:, q])
                    vals.append(ag[q] / 3)
        key, inv = torch.unique(torch.cat(keys), return_inverse=True)
        self.c = torch.zeros(key.numel(), 2, dtype=torch.float64, device=dev).index_add_(0, inv, torch.cat(vals))
        self.i, self.j = key // n, key % n
        self.norm = self.c.norm(dim=1)
        self.nrm = self.c / self.norm[:, None]
        self.bc = [(k, f(js.astype(np.int64)), f(v)) for k, js, v in scene["bc"]]

    def rows(self, v):
        return torch.zeros(self.n, dtype=torch.float64, device=v.device).index_add_(0, self.i, v)

    def ovh(self, h):
        return 2 * h / (h * h + torch.clamp(h, min=self.p.htiny) ** 2)

    def raw_d(self, u):
        """|c_ij| times the guaranteed bound of the wave speed."""
        g, i, j = self.p.gravity, self.i, self.j
        o = self.ovh(u[0])
        vn = lambda k: (u[1][k] * self.nrm[:, 0] + u[2][k] * self.nrm[:, 1]) * o[k]  # noqa: E731
        hl, hr, vl, vr, ol, orr = u[0][i], u[0][j], vn(i), vn(j), o[i], o[j]
        sql, sqr = (g * hl.abs()).sqrt(), (g * hr.abs()).sqrt()
        hmin, hmax = torch.minimum(hl, hr), torch.maximum(hl, hr)
        x0 = (2 * math.sqrt(2.0) - 1) ** 2

        def phi(h):
            oh = self.ovh(h)
            side = lambda hk, ok: torch.where(h > hk, (h - hk) * (g / 2 * (oh + ok)).sqrt(),  # noqa: E731
                                              2 * ((g * h).sqrt() - (g * hk).sqrt()))
            return side(hl, ol) + side(hr, orr) + vr - vl

        a = 1 / (2 * math.sqrt(2.0))
        rmin, rmax = hmin.sqrt(), hmax.sqrt()
        h_a = torch.minimum(x0 * hmin, torch.clamp(vl - vr + 2 * sql + 2 * sqr, min=0) ** 2 / (16 * g))
        disc = hmin - 4 * a * (-(hmin * a) - rmin * rmax + rmin * (vr - vl) / (2 * math.sqrt(g)))
        h_b = torch.minimum(x0 * hmax, ((-rmin + torch.clamp(disc, min=0).sqrt()) / (2 * a)) ** 2)
        h_c = rmin * rmax * (1 + math.sqrt(2 / g) * (vl - vr) / (rmin + rmax))
        hs = torch.where(phi(x0 * hmin) >= 0, h_a, torch.where(phi(x0 * hmax) >= 0, h_b, h_c))

        def speed(hk, ok):
            x = torch.clamp((hs - hk) * ok, min=0)
            return ((1 + x / 2) * (1 + x)).sqrt()

        return self.norm * torch.maximum((vl - sql * speed(hl, ol)).abs(), (vr + sqr * speed(hr, orr)).abs())

    def dt(self, u):
        return self.p.cfl / float((self.rows(self.raw_d(u)) / self.m).max())

    def sources(self, u, v, rk, dt):
        p, h = self.p, u[0]
        if p.type_test == 10:
            hs = torch.clamp(h, min=p.htiny) ** (4.0 / 3.0)
            vel = p.gravity * p.mannings ** 2 * (v[0] ** 2 + v[1] ** 2).sqrt()
            fr = self.m * vel * 2 / (hs + torch.maximum(hs, vel * dt))
            return [rk[0], rk[1] - fr * u[1], rk[2] - fr * u[2]]
        if p.type_test == 13:
            pc = p.lambda_sgn * p.gravity / (3 * self.m.sqrt())
            x = u[3] / (h * h)
            press = pc * h ** 3 * (2 + 4 * x ** 3 - 6 * x ** 4)
            s = 3 * pc * (u[3] / h) ** 2 * 12 * (x - 1)
            px = self.rows(press[self.j] * self.c[:, 0]) + press * self.cd[:, 0]
            py = self.rows(press[self.j] * self.c[:, 1]) + press * self.cd[:, 1]
            return [rk[0], rk[1] - px, rk[2] - py, rk[3] + self.m * u[4], rk[4] - self.m * s]
        return rk

    def euler(self, u, dt):
        p, i, j, m, S = self.p, self.i, self.j, self.m, len(u)
        g, h = p.gravity, u[0]
        cx, cy = self.c[:, 0], self.c[:, 1]
        o = self.ovh(h)
        w = [u[1] * o, u[2] * o]                             # velocity of the viscosities
        v = [w[0], torch.zeros_like(h) if p.type_test == 13 else w[1]]
        E = 0.5 * (g * h * h + v[0] * u[1] + v[1] * u[2])
        dh = h[j] - h[i]
        num, den = self.rows(dh).abs(), self.rows(dh.abs())
        al = torch.where(den <= num, torch.ones_like(den), num / den) ** 8
        al = torch.where(h <= p.htiny, torch.ones_like(al), al)
        mu = torch.maximum(torch.clamp(-(cx * w[0][i] + cy * w[1][i]), min=0),
                           torch.clamp(cx * w[0][j] + cy * w[1][j], min=0))
        sc = torch.maximum(al[i], al[j])
        d, mu = torch.maximum(self.raw_d(u), mu) * sc, mu * sc
        zm = torch.maximum(self.z[i], self.z[j])
        Hi, Hj = torch.clamp(h[i] + self.z[i] - zm, min=0), torch.clamp(h[j] + self.z[j] - zm, min=0)
        one = torch.ones_like(Hi)
        ri = torch.where(h[i] <= 0, 0 * Hi, Hi / torch.where(h[i] <= 0, one, h[i]))
        rj = torch.where(h[j] <= 0, 0 * Hj, Hj / torch.where(h[j] <= 0, one, h[j]))
        ti = torch.where(h[i] <= p.htiny, 0 * ri, ri)
        tj = torch.where(h[j] <= p.htiny, 0 * rj, rj)
        cv = cx * v[0][j] + cy * v[1][j]
        cvd = self.cd[:, 0] * v[0] + self.cd[:, 1] * v[1]
        eta = h + self.z
        topo = g * h[i] * (eta[j] - eta[i])

        def rhs(dd, mm, a, b, first):
            rk = [first]
            for q in range(1, S):
                uq = u[q]
                t = (-cv * uq[j] + dd * (uq[j] * b - uq[i] * a) + mm * (uq[j] * (1 - b) - uq[i] * (1 - a)))
                if q < 3:
                    t = t - topo * (cx if q == 1 else cy)
                rk.append(self.rows(t) - cvd * uq)
            return self.sources(u, v, rk, dt)

        def stage(dd, mm):                                    # the roundoff-fixed rows and their update
            fix = -cvd - self.rows(mm + (dd - mm) * ti)
            rk = rhs(dd, mm, ti, tj, self.rows((mm - cv) * h[j] + torch.clamp((dd - mm) * Hj, min=0)))
            return [h * (1 + dt * fix / m) + dt * rk[0] / m] + [u[q] + dt * rk[q] / m for q in range(1, S)]

        uL = stage(d, mu)
        if p.viscosity_type == VISC["viscous"]:
            return uL
        A, B = h[j] * rj - h[i] * ri, h[j] * (1 - rj) - h[i] * (1 - ri)
        rk2 = rhs(d, mu, ri, rj, self.rows(-cv * h[j] + d * A + mu * B) - cvd * h)
        n0, n1, n2 = (u[q] + dt * rk2[q] / m for q in range(3))
        on = self.ovh(n0)
        En = 0.5 * (g * n0 * n0 + n1 * on * n1 + n2 * on * n2)
        rs = m * (En - E) / dt - rk2[0] * (g * h - 0.5 * v[0] ** 2 - 0.5 * v[1] ** 2) - rk2[1] * v[0] - rk2[2] * v[1]
        hi = E.clone().scatter_reduce_(0, i, E[j], "amax")
        lo = E.clone().scatter_reduce_(0, i, E[j], "amin")
        res = rs.abs() / ((hi - lo).abs() / 2 + 1e-10 * g * p.max_water_h ** 2)
        rij = torch.maximum(res[i], res[j])
        dH, mH = torch.minimum(d, rij), torch.minimum(mu, rij)
        if p.viscosity_type == VISC["entropy_visc"]:
            return stage(dH, mH)
        f = (dH - d) * A + (mH - mu) * B
        P = self.rows(torch.clamp(f, max=0)) - 1e-15
        scaled = m / dt * uL[0]
        R = torch.where(scaled <= p.htiny, 0 * scaled, torch.clamp(-scaled / P, max=1))
        lim = torch.where(f >= 0, R[j], R[i])
        dd, dm = (dH - d) * lim, (mH - mu) * lim
        return [uL[q] + dt / m * self.rows(dd * (u[q][j] * rj - u[q][i] * ri)
                                           + dm * (u[q][j] * (1 - rj) - u[q][i] * (1 - ri))) for q in range(S)]

    def impose(self, u):
        for k, js, v in self.bc:
            u[k] = u[k].index_copy(0, js, v)
        return u

    def steps(self, u, steps):
        t = 0.0
        for _ in range(steps):
            dt = self.dt(u)
            a = self.impose(self.euler(u, dt))
            a = self.impose([(3 * x + y) / 4 for x, y in zip(u, self.euler(a, dt))])
            u, t = self.impose([(x + 2 * y) / 3 for x, y in zip(u, self.euler(a, dt))]), t + dt
        return u, t, dt


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    us, ts, dts, dij = [], [], [], None
    for s in _scenes(case, seed):
        plain = _Plain(s, dev)
        u = [torch.from_numpy(np.ascontiguousarray(c)).to(dev) for c in s["u"].T]
        if case["way"] == "percall":                          # d_ij in the order of the rows, diagonal included
            d = plain.raw_d(u)
            row = torch.cat([plain.i, torch.arange(plain.n, device=dev)])
            col = torch.cat([plain.j, torch.arange(plain.n, device=dev)])
            dij = torch.cat([d, -plain.rows(d)])[torch.argsort(row * plain.n + col)].cpu().numpy()
        u, t, dt = plain.steps(u, case["steps"])
        us.append(torch.stack(u, 1))
        ts.append(t)
        dts.append(dt)
    u = torch.cat(us)
    if case["way"] == "device":
        return {"u": u, "t": np.array(ts), "dt": np.array(dts), "steps": None}
    if case["way"] == "host":
        return {"u": u.cpu().numpy(), "t": np.array(ts), "dt": np.array(dts)}
    return {"u": u.cpu().numpy(), "t": ts[0], "dt": dts[0], "dij": dij}
