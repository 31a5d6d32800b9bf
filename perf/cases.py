"""The work that users of gala_gb300 have it do, as cases that can be timed and checked.

Every case goes through the package's public calls with the workloads of its own
benchmark and tests (gala_gb300.workloads): the Milky-Way composite, the Hernquist
sphere, the SCF halo and their orbit populations, in galactic units.

    listed()             the cases, smallest call to largest
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a user's program holds before the call
    run(state)           one pass; returns the call's whole results
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the results in 64 bits from plain torch / numpy

`exact` writes the mathematics out again, independently of the package: potentials
as closed forms, Leapfrog and Ruth4 as their loops, adaptive DOP853 orbits as the
true solution (Gragg-Bulirsch-Stoer extrapolation far below the tolerance).
"""
import math

import numpy as np
import torch

import gala_gb300 as gp
from gala_gb300 import workloads as W
from gala_gb300.batch import integrate_batch
from gala_gb300.mockstream import FardalStreamDF, MockStreamGenerator
from gala_gb300.nbody import integrate_systems, pack_bodies
from gala_gb300.surrogate import NPARAM, SurrogatePotential, init_params

G = 4.498502151469553e-12  # kpc^3 / (Msun Myr^2)
DEV = "cuda"

# Potentials by name: (kind, parameters) per component, in evaluation order.
POTENTIALS = {
    # the benchmark's single sphere
    "hernquist": [("hernquist", 1e11, 1.0)],
    # the benchmark's Milky-Way composite: nucleus, bulge, disk, halo
    "mw": [("hernquist", 1.7e9, 0.07), ("hernquist", 5e9, 1.0), ("mn", 6.8e10, 3.0, 0.28), ("nfw", 5.4e11, 15.6)],
    # a disk and a Plummer bulge in a triaxial halo that rotates with the frame
    "bar": [("plummer", 1e10, 0.5), ("mn", 6.8e10, 3.0, 0.28), ("nfw", 5.4e11, 15.6, 1.0, 0.9, 0.8)],
}
# gradient evaluation, floating-point operations (add, multiply, divide, root, log: one each)
GRAD_FLOPS = {"hernquist": 17, "mw": 81, "bar": 84}


def listed():
    return [
        # an interactive call: the potential and its gradient at a few hundred points, host arrays in and out
        {"name": "points_mw", "kind": "points", "n": 257},
        # one gala-sized call: a few orbits through a bar in its rotating frame, every step kept, host arrays
        {"name": "dop853_rotating_few", "kind": "dop853", "pot": "bar", "n": 37, "n_steps": 400, "dt": 1.0, "stride": 1,
         "precision": "fp64", "host": True},
        # the benchmark's plain Leapfrog: 1,024 orbits, 1,000 steps, all snapshots
        {"name": "leapfrog_hernquist", "kind": "fixed", "pot": "hernquist", "n": 1024, "n_steps": 1000, "dt": 1.0,
         "integrator": "leapfrog", "save_all": True},
        # satellites with massless tracers as direct n-body systems, DOP853
        {"name": "nbody_satellites", "kind": "nbody", "systems": 127, "massive": 2, "tracers": 7, "n_steps": 300},
        # mock streams from many progenitors (Fardal releases, two particles every step)
        {"name": "streams_leapfrog", "kind": "streams", "streams": 64, "n_steps": 400},
        # surrogate training: Adam steps on minibatches (forward, backward, double backward)
        {"name": "surrogate_train", "kind": "train", "steps": 16, "batch": 8192},
        # the trained surrogate's force and potential at many points (tensor-core inference)
        {"name": "surrogate_field", "kind": "surrogate", "n": 100003},
        # SCF expansion: potential and gradient at the points a training set or a map needs
        {"name": "scf_field", "kind": "scf", "n": 131101, "nmax": 12, "lmax": 8},
        # pericentre, apocentre and z_max of a stored population
        {"name": "orbit_extrema", "kind": "extrema", "n": 20011, "n_times": 1001},
        # uneven batch in the plain FP64 form
        {"name": "batch_fp64_uneven", "kind": "batch", "n": 16384, "n_lo": 100, "n_hi": 2000, "precision": "fp64"},
        # the benchmark's headline: uneven batch, FP32 force with compensated state
        {"name": "batch_fp32c_uneven", "kind": "batch", "n": 262144, "n_lo": 100, "n_hi": 20000, "precision": "fp32c"},
        # the benchmark's adaptive population: DOP853 through the composite, every 100th time kept
        {"name": "dop853_mw", "kind": "dop853", "pot": "mw", "n": 20011, "n_steps": 2000, "dt": 0.5, "stride": 100,
         "precision": "fp64", "host": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["points", "dop853", "dop853", "dop853", "fixed", "fixed", "nbody", "streams", "train", "surrogate",
                       "scf", "extrema", "batch", "batch"])
    if kind == "points":
        return {"kind": kind, "n": _log(rng, 1, 20000)}
    if kind == "dop853":
        if rng.random() < 0.3:
            return {"kind": kind, "pot": "bar", "n": _log(rng, 1, 400), "n_steps": _log(rng, 50, 500), "dt": 1.0,
                    "stride": 1, "precision": "fp64", "host": True}
        precision = rng.choice(["fp64", "fp64", "fp32c"])
        return {"kind": kind, "pot": "mw", "n": _log(rng, 50, 20000), "n_steps": _log(rng, 200, 1999), "dt": 0.5,
                "stride": rng.choice([10, 50, 100]), "precision": precision, "host": False}
    if kind == "fixed":
        pot = rng.choice(["hernquist", "mw", "scf"])
        return {"kind": kind, "pot": pot, "n": _log(rng, 1, 1000 if pot == "scf" else 8000),
                "n_steps": _log(rng, 10, 30) if pot == "scf" else _log(rng, 100, 600), "dt": 1.0,
                "integrator": rng.choice(["leapfrog", "ruth4"]), "save_all": rng.random() < 0.5}
    if kind == "nbody":
        return {"kind": kind, "systems": _log(rng, 1, 400), "massive": rng.randint(1, 3), "tracers": rng.randint(0, 13),
                "n_steps": _log(rng, 50, 300)}
    if kind == "streams":
        return {"kind": kind, "streams": _log(rng, 1, 100), "n_steps": _log(rng, 50, 400)}
    if kind == "train":
        return {"kind": kind, "steps": rng.randint(2, 16), "batch": rng.choice([1024, 2048, 4096, 8192])}
    if kind == "surrogate":
        return {"kind": kind, "n": _log(rng, 100, 200000)}
    if kind == "scf":
        return {"kind": kind, "n": _log(rng, 10, 130000), "nmax": rng.randint(2, 14), "lmax": rng.randint(1, 9)}
    if kind == "extrema":
        return {"kind": kind, "n": _log(rng, 1, 30000), "n_times": _log(rng, 100, 1300)}
    if rng.random() < 0.5:
        return {"kind": kind, "n": _log(rng, 100, 20000), "n_lo": 50, "n_hi": _log(rng, 100, 2000), "precision": "fp64"}
    return {"kind": kind, "n": _log(rng, 300, 260000), "n_lo": 100, "n_hi": _log(rng, 200, 20000), "precision": "fp32c"}


# ------------------------------------------------------------------ what a program holds


def _potential(name):
    if name == "scf":
        return W.scf_potential()
    pot = gp.CCompositePotential()
    make = {"hernquist": gp.HernquistPotential, "plummer": gp.PlummerPotential, "mn": gp.MiyamotoNagaiPotential,
            "nfw": gp.NFWPotential}
    for i, (kind, *p) in enumerate(POTENTIALS[name]):
        pot[f"c{i}"] = make[kind](*p)
    return pot if len(pot) > 1 else pot["c0"]


def _orbits(name, n, seed):
    if name == "hernquist":
        return W.hernquist_ics(n, seed=seed)
    if name == "scf":
        return W.scf_ics(n, seed=seed)
    return W.mw_ics(n, seed=seed)


def _points(n, seed, r_lo, r_hi):
    """Positions (3, n), isotropic, radius log-uniform."""
    rng = np.random.default_rng(seed)
    u = rng.normal(size=(3, n))
    r = np.exp(rng.uniform(math.log(r_lo), math.log(r_hi), n))
    return np.ascontiguousarray(u / np.linalg.norm(u, axis=0) * r)


def _uneven(case, seed):
    """Per-orbit n_steps log-uniform, dt of {0.1, 0.5, 1} Myr, Leapfrog for half and Ruth4 for half."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    ns = np.round(np.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"]), n))).astype(np.int64)
    method = (np.arange(n) >= n // 2).astype(np.int32)
    rng.shuffle(method)
    return W.mw_ics(n, seed=seed + 1), ns, rng.choice(np.array([0.1, 0.5, 1.0]), n), method


OMEGA = (0.0, 0.0, 0.04)  # rad / Myr: a bar's pattern speed of about 40 km/s/kpc


def _satellites(case, seed):
    """Systems of satellites on Milky-Way orbits, each of the massive ones a Plummer sphere, and massless tracers around them."""
    rng = np.random.default_rng(seed)
    S, nm, nt = case["systems"], case["massive"], case["tracers"]
    w = W.mw_ics(S * (nm + nt), seed=seed + 1).T.reshape(S, nm + nt, 6) * np.array([3, 3, 3, 1, 1, 1.0])
    m, b = np.exp(rng.uniform(math.log(1e8), math.log(1e10), (S, nm))), rng.uniform(0.5, 2.0, (S, nm))
    return np.ascontiguousarray(w), m, b


def _rosettes(case, seed):
    """Stored orbits (6, n_times, n): epicycles about circular guiding centres with a vertical oscillation."""
    g = torch.Generator().manual_seed(seed)
    u = torch.rand((6, case["n"]), generator=g, dtype=torch.float64).to(DEV)
    t = torch.arange(case["n_times"], dtype=torch.float64, device=DEV)[:, None]
    R, e, h = 2 + 28 * u[0], 0.05 + 0.3 * u[1], 0.1 + 2 * u[2]
    om = 0.22 / R
    ka, nu = 1.4 * om, 2.5 * om
    a, b, c = ka * t + 6.283 * u[3], om * t + 6.283 * u[4], nu * t + 6.283 * u[5]
    r, th = R * (1 - e * torch.cos(a)), b + 2 * om / ka * e * torch.sin(a)
    vr, vt = R * e * ka * torch.sin(a), om + 2 * om * e * torch.cos(a)
    w = torch.empty((6, case["n_times"], case["n"]), dtype=torch.float64, device=DEV)
    co, si = torch.cos(th), torch.sin(th)
    w[0], w[1], w[2] = r * co, r * si, h * torch.cos(c)
    w[3], w[4], w[5] = vr * co - r * vt * si, vr * si + r * vt * co, -h * nu * torch.sin(c)
    return w, np.arange(case["n_times"], dtype=np.float64)


def _scf(nmax, lmax):
    return W.scf_potential(nmax, lmax)


def _training_set(n, seed):
    """A smooth target on the unit ball with its gradient: features, values, gradients, weights."""
    g = torch.Generator().manual_seed(seed)
    x = torch.randn((n, 3), generator=g, dtype=torch.float64)
    x = (x / x.norm(dim=1, keepdim=True) * (0.1 + 0.9 * torch.rand((n, 1), generator=g, dtype=torch.float64))).to(DEV)
    k = torch.tensor([[2.0, 1.0, -1.0], [0.5, -3.0, 1.5], [1.0, 2.0, 4.0]], dtype=torch.float64, device=DEV)
    ph = x @ k.T
    y = 0.3 * torch.sin(ph).sum(dim=1)
    return x.float().contiguous(), y.float(), (0.3 * torch.cos(ph) @ k).float().contiguous(), (0.5 + x.norm(dim=1)).float()


def _streams(case, seed):
    w0, m, b = W.stream_progenitors(case["streams"], seed=seed)
    return w0, m, b, W.stream_progenitor_potentials(m, b)


def prepare(case, seed):
    k, s = case["kind"], {"case": dict(case)}
    if k == "points":
        s["pot"], s["q"] = _potential("mw"), _points(case["n"], seed, 0.1, 100.0)
    elif k == "dop853":
        frame = gp.ConstantRotatingFrame(OMEGA) if case["pot"] == "bar" else None
        s["H"] = gp.Hamiltonian(_potential(case["pot"]), frame)
        w0 = W.mw_ics(case["n"], seed=seed)
        s["w0"] = w0 if case["host"] else torch.from_numpy(w0).to(DEV)
        tol = 1e-8 if case["precision"] == "fp32c" else 1e-10
        s["kw"] = {"rtol": tol, "atol": 0.01 * tol, "out_stride": case["stride"], "precision": case["precision"]}
    elif k == "fixed":
        s["H"] = gp.Hamiltonian(_potential(case["pot"]))
        s["w0"] = torch.from_numpy(_orbits(case["pot"], case["n"], seed)).to(DEV)
    elif k == "nbody":
        w, m, b = _satellites(case, seed)
        s["H"], s["w0"] = gp.Hamiltonian(_potential("mw")), torch.from_numpy(w).to(DEV)
        s["bodies"] = pack_bodies([[gp.PlummerPotential(m=float(mi), b=float(bi)) for mi, bi in zip(ms, bs)] for ms, bs in zip(m, b)])
        s["t"] = np.arange(case["n_steps"] + 1, dtype=np.float64)
    elif k == "streams":
        s["w0"], s["m"], _, s["pots"] = _streams(case, seed)
        s["H"], s["seed"] = gp.Hamiltonian(_potential("mw")), seed
    elif k == "train":
        s["sp"] = SurrogatePotential(_scf(12, 8), seed=seed)
        s["init"] = s["sp"].params.clone()
        s["set"] = _training_set(1 << 17, seed)
    elif k == "surrogate":
        s["sp"] = SurrogatePotential(_scf(12, 8), seed=seed)
        s["sp"].export()
        s["q"] = torch.from_numpy(_points(case["n"], seed, 0.4, 250.0)).to(DEV)
    elif k == "scf":
        s["pot"], s["q"] = _scf(case["nmax"], case["lmax"]), torch.from_numpy(_points(case["n"], seed, 0.5, 200.0)).to(DEV)
    elif k == "extrema":
        s["w"], s["t"] = _rosettes(case, seed)
    elif k == "batch":
        w0, ns, dt, method = _uneven(case, seed)
        s["pot"] = _potential("mw")
        # states, lengths and steps on the device, the integrator codes as the host array a program makes them
        s["args"] = (*(torch.from_numpy(a).to(DEV) for a in (w0, ns, dt)), method)
    return s


# ------------------------------------------------------------------ one pass


def run(s):
    case = s["case"]
    k = case["kind"]
    if k in ("points", "scf"):
        return {"phi": s["pot"].energy(s["q"]), "grad": s["pot"].gradient(s["q"])}
    if k == "dop853":
        o = s["H"].integrate_orbit(s["w0"], Integrator="dop853", Integrator_kwargs=s["kw"], dt=case["dt"],
                                   n_steps=case["n_steps"], return_device=not case["host"])
        return o.w() if case["host"] else o.w_device
    if k == "fixed":
        return s["H"].integrate_orbit(s["w0"], Integrator=case["integrator"], dt=case["dt"], n_steps=case["n_steps"],
                                      save_all=case["save_all"], return_device=True).w_device
    if k == "nbody":
        w, status = integrate_systems(s["H"], s["bodies"], s["w0"], s["t"], save_all=True, out_stride=10)
        return {"w": w, "status": status}
    if k == "streams":
        df = FardalStreamDF(gala_modified=True, random_state=np.random.RandomState(s["seed"] % (1 << 31)))
        r = MockStreamGenerator(df, s["H"]).run_batch(s["w0"], s["m"], s["pots"], dt=1.0, n_steps=case["n_steps"],
                                                      Integrator="leapfrog")
        return {"stream": r.stream_w, "nbody": r.nbody_w, "status": r.status}
    if k == "train":
        sp = s["sp"]
        sp.params = s["init"].clone()
        sp.X, sp.Y, sp.Gt, sp.Wg = s["set"]
        sp.y_scale, sp.history = 1.0, []
        sp.train(steps=case["steps"], batch=case["batch"], seed=2)
        return {"params": sp.params, "loss": [list(h[1:]) for h in sp.history]}
    if k == "surrogate":
        grad, phi = s["sp"].gradient_and_energy(s["q"])
        return {"grad": grad, "phi": phi}
    if k == "extrema":
        o = gp.Orbit.from_w(s["w"], t=s["t"])
        return {"peri": o.pericenter(), "apo": o.apocenter(), "zmax": o.zmax()}
    w, dE = integrate_batch(s["pot"], *s["args"], precision=case["precision"])
    return {"w": w, "dE": dE}


# ------------------------------------------------------------------ what a pass cannot do without


def _scf_flops(nmax, lmax, grad):
    """Per point: the two Gegenbauer recurrences per (n, l), the sums over n for each (l, m), the angular part."""
    N, lm = nmax + 1, (lmax + 1) * (lmax + 2) // 2
    return N * (lmax + 1) * (14 if grad else 5) + lm * N * (8 if grad else 4) + lm * (20 if grad else 8) + 60


def work(case):
    k = case["kind"]
    n = case.get("n", 0)
    if k == "points":
        return {"bytes": n * 56, "flops": n * (81 + 46)}
    if k == "scf":
        return {"bytes": n * 80, "flops": n * (_scf_flops(case["nmax"], case["lmax"], False) + _scf_flops(case["nmax"], case["lmax"], True))}
    if k == "dop853":
        # at these tolerances about 1.4 attempted steps per Myr: 954 operations and 12 right-hand sides each
        steps = n * case["n_steps"] * case["dt"] * 1.4
        out = case["n_steps"] // case["stride"] + 1
        return {"bytes": n * 48 * (1 + out), "flops": steps * (954 + 12 * (GRAD_FLOPS[case["pot"]] + 6))}
    if k == "fixed":
        grad = _scf_flops(12, 8, True) if case["pot"] == "scf" else GRAD_FLOPS[case["pot"]]
        per = 21 + grad if case["integrator"] == "leapfrog" else 63 + 3 * grad
        return {"bytes": n * 48 * (1 + (case["n_steps"] + 1 if case["save_all"] else 1)), "flops": n * case["n_steps"] * per}
    if k == "nbody":
        b = case["massive"] + case["tracers"]
        steps = case["systems"] * case["n_steps"] * 0.2
        return {"bytes": case["systems"] * b * 48 * (2 + case["n_steps"] // 10),
                "flops": steps * b * (954 + 12 * (87 + 23 * (case["massive"])))}
    if k == "streams":
        parts = 2 * (case["n_steps"] + 1) * case["streams"]
        return {"bytes": parts * 48 * 2, "flops": parts * case["n_steps"] / 2 * (21 + 81 + 23)}
    if k == "train":
        # forward, input gradient, double backward and weight gradients of three 256 x 256 layers
        return {"bytes": case["steps"] * (case["batch"] * 32 + NPARAM * 4 * 6),
                "flops": case["steps"] * case["batch"] * 3 * 2 * 256 * 256 * 8}
    if k == "surrogate":
        return {"bytes": n * 56 + 6 * 131072, "flops": n * 6 * 2 * 256 * 256}
    if k == "extrema":
        return {"bytes": n * case["n_times"] * 24 + n * 24, "flops": n * case["n_times"] * 8}
    mean = (case["n_hi"] - case["n_lo"]) / math.log(case["n_hi"] / case["n_lo"])
    return {"bytes": n * (48 * 2 + 8 + 8 + 4 + 8), "flops": n * mean * (102 + 306) / 2}


# ------------------------------------------------------------------ the same results in 64 bits


def _f64(a):
    return torch.as_tensor(np.asarray(a), dtype=torch.float64, device=DEV) if not isinstance(a, torch.Tensor) else a.to(torch.float64)


def _phi(name, q):
    x, y, z = q
    v = 0.0
    for kind, *p in POTENTIALS[name]:
        gm, r2 = G * p[0], x * x + y * y + z * z
        if kind == "hernquist":
            v = v - gm / (torch.sqrt(r2) + p[1])
        elif kind == "plummer":
            v = v - gm / torch.sqrt(r2 + p[1] ** 2)
        elif kind == "mn":
            zd = p[1] + torch.sqrt(z * z + p[2] ** 2)
            v = v - gm / torch.sqrt(x * x + y * y + zd * zd)
        else:
            a, b, c = p[2:] if len(p) > 2 else (1.0, 1.0, 1.0)
            u = torch.sqrt((x / a) ** 2 + (y / b) ** 2 + (z / c) ** 2) / p[1]
            v = v - gm / p[1] * torch.log1p(u) / u
    return v


def _grad(name, q):
    """(3, ...) gradient; plain sphere terms share the radius."""
    x, y, z = q
    fx = 0.0
    gx = gy = gz = 0.0
    r2 = x * x + y * y + z * z
    for kind, *p in POTENTIALS[name]:
        gm = G * p[0]
        if kind == "hernquist":
            r = torch.sqrt(r2)
            fx = fx + gm / (r * (r + p[1]) ** 2)
        elif kind == "plummer":
            fx = fx + gm / (r2 + p[1] ** 2) ** 1.5
        elif kind == "mn":
            s = torch.sqrt(z * z + p[2] ** 2)
            zd = p[1] + s
            f = gm / (x * x + y * y + zd * zd) ** 1.5
            gx, gy, gz = gx + f * x, gy + f * y, gz + f * z * zd / s
        else:
            a, b, c = p[2:] if len(p) > 2 else (1.0, 1.0, 1.0)
            m = torch.sqrt((x / a) ** 2 + (y / b) ** 2 + (z / c) ** 2)
            u = m / p[1]
            f = gm / m ** 3 * (torch.log1p(u) - u / (1 + u))
            gx, gy, gz = gx + f * x / a ** 2, gy + f * y / b ** 2, gz + f * z / c ** 2
    return torch.stack([gx + fx * x, gy + fx * y, gz + fx * z])


TWO13 = 2.0 ** (1.0 / 3.0)
RUTH_C = [1 / (2 * (2 - TWO13)), (1 - TWO13) / (2 * (2 - TWO13)), (1 - TWO13) / (2 * (2 - TWO13)), 1 / (2 * (2 - TWO13))]
RUTH_D = [0.0, 1 / (2 - TWO13), -TWO13 / (2 - TWO13), 1 / (2 - TWO13)]


def _fixed(grad, w0, dt, n_steps, method, save_all):
    """Leapfrog (kick-drift-kick with a half-step velocity) or Ruth4 with one dt for all orbits."""
    x, v = w0[:3].clone(), w0[3:].clone()
    keep = [torch.cat([x, v])]
    if method == "leapfrog":
        vh = v - grad(x) * (dt / 2)
        for _ in range(n_steps):
            x = x + vh * dt
            g = grad(x)
            v, vh = vh - g * (dt / 2), vh - g * dt
            if save_all:
                keep.append(torch.cat([x, v]))
    else:
        for _ in range(n_steps):
            for c, d in zip(RUTH_C, RUTH_D):
                if d:
                    v = v - d * dt * grad(x)
                x = x + c * dt * v
            if save_all:
                keep.append(torch.cat([x, v]))
    return torch.stack(keep, dim=1) if save_all else torch.cat([x, v])[:, None]


def _gbs(rhs, w, t_end, H, out_every, depth):
    """The solution at 0, out_every H, 2 out_every H, ... up to t_end: extrapolated modified midpoint, `depth` even substep numbers."""
    outs = [w]
    ns = [2 * (j + 1) for j in range(depth)]
    for step in range(1, int(round(t_end / H)) + 1):
        f0, table = rhs(w), []
        for j, n in enumerate(ns):
            h = H / n
            a, b = w, w + h * f0
            for _ in range(n - 1):
                a, b = b, a + 2 * h * rhs(b)
            row = [0.5 * (a + b + h * rhs(b))]
            for k in range(1, j + 1):
                row.append(row[-1] + (row[-1] - table[-1][k - 1]) / ((ns[j] / ns[j - k]) ** 2 - 1))
            table.append(row)
        w = table[-1][-1]
        if step % out_every == 0:
            outs.append(w)
    return outs


def _exact_dop853(case, seed):
    if case["precision"] == "fp32c" or case["n"] * case["n_steps"] * case["dt"] > 3e7:
        return None
    w0 = _f64(W.mw_ics(case["n"], seed=seed))
    om = OMEGA[2] if case["pot"] == "bar" else 0.0

    def rhs(w):
        g = _grad(case["pot"], w[:3])
        x, y, _, px, py, pz = w
        return torch.stack([px + om * y, py - om * x, pz, om * py - g[0], -om * px - g[1], -g[2]])

    every = case["dt"] * case["stride"]
    H = 1.0 if every < 2.5 else 2.5
    outs = _gbs(rhs, w0, every * (case["n_steps"] // case["stride"]), H, int(round(every / H)), 5 if H == 1.0 else 8)
    w = torch.stack(outs, dim=1)
    w = w[..., 0] if case["n"] == 1 else w
    return w.cpu().numpy() if case["host"] else w


def _exact_nbody(case, seed):
    w, m, b = _satellites(case, seed)
    if case["n_steps"] < 10:
        return None
    w, gm, b2, nm = _f64(w), G * _f64(m), _f64(b) ** 2, case["massive"]

    def rhs(y):  # y (S, bodies, 6)
        q = y[..., :3]
        a = -_grad("mw", q.permute(2, 0, 1)).permute(1, 2, 0)
        d = q[:, :, None, :] - q[:, None, :nm, :]  # body pulled, body pulling
        a = a - (gm[:, None, :, None] * d / ((d * d).sum(-1, keepdim=True) + b2[:, None, :, None]) ** 1.5).sum(2)
        return torch.cat([y[..., 3:], a], dim=-1)

    outs = _gbs(rhs, w, 10.0 * (case["n_steps"] // 10), 2.5, 4, 7)
    return {"w": torch.stack(outs, dim=1), "status": None}


def _scf_exact(pot, q, want_grad):
    """SCF sum by three-term recurrences, vectorised over the points; gradient by the chain rule in spherical coordinates."""
    S, T = np.asarray(pot.parameters["Snlm"]), np.asarray(pot.parameters["Tnlm"])
    nmax, lmax = S.shape[0] - 1, S.shape[1] - 1
    gm, rs = G * pot.parameters["m"], pot.parameters["r_s"]
    x, y, z = q
    R = torch.sqrt(x * x + y * y)
    r = torch.sqrt(x * x + y * y + z * z)
    s, X, st = r / rs, z / r, R / r
    cp, sp = x / R, y / R
    xi = (s - 1) / (s + 1)
    one, zero = torch.ones_like(s), torch.zeros_like(s)
    cm, sm = [one], [zero]
    for m in range(lmax):
        cm, sm = cm + [cm[m] * cp - sm[m] * sp], sm + [sm[m] * cp + cm[m] * sp]
    P = {}
    for m in range(lmax + 1):  # Legendre functions with the Condon-Shortley phase
        P[m, m] = one if m == 0 else -(2 * m - 1) * st * P[m - 1, m - 1]
        for l in range(m + 1, lmax + 1):
            P[l, m] = (X * (2 * l - 1) * P[l - 1, m] - ((l + m - 1) * P[l - 2, m] if l > m + 1 else 0.0)) / (l - m)
    phi, dr, dth, dph = zero, zero, zero, zero
    for l in range(lmax + 1):
        a, b = 2 * l + 1.5, 2 * l + 2.5
        C, D = [one, 2 * a * xi], [zero, one, 2 * b * xi]
        for n in range(2, nmax + 1):
            C.append((2 * xi * (n + a - 1) * C[n - 1] - (n + 2 * a - 2) * C[n - 2]) / n)
            if n >= 2 and len(D) <= n:
                j = n - 1
                D.append((2 * xi * (j + b - 1) * D[n - 1] - (j + 2 * b - 2) * D[n - 2]) / j)
        u = s ** l * (1 + s) ** (-2 * l - 1)            # radial envelope and its logarithmic derivative
        du = u * (l / s - (2 * l + 1) / (1 + s))
        dxi = 2 / (1 + s) ** 2
        for m in range(l + 1):
            nrm = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m)) * math.sqrt(4 * math.pi)
            fs, ft, gs, gt = zero, zero, zero, zero
            for n in range(nmax + 1):
                fs, ft = fs + float(S[n, l, m]) * C[n], ft + float(T[n, l, m]) * C[n]
                if want_grad:
                    gs, gt = gs + float(S[n, l, m]) * 2 * a * D[n], gt + float(T[n, l, m]) * 2 * a * D[n]
            ang = fs * cm[m] + ft * sm[m]
            Y = nrm * P[l, m]
            phi = phi - u * Y * ang
            if want_grad:
                dang = gs * cm[m] + gt * sm[m]
                dr = dr - Y * (du * ang + u * dxi * dang)
                dY = nrm * (l * X * P[l, m] - ((l + m) * P[l - 1, m] if l > m else 0.0)) / st
                dth = dth - u * dY * ang
                dph = dph - u * m * Y * (ft * cm[m] - fs * sm[m])
    phi = phi * gm / rs
    if not want_grad:
        return phi
    k = gm / rs ** 2
    dr, dth, dph = dr * k, dth / s * k, dph / (s * st) * k
    return phi, torch.stack([st * cp * dr + X * cp * dth - sp * dph, st * sp * dr + X * sp * dth + cp * dph, X * dr - st * dth])


def _exact_batch(case, seed):
    if case["n_hi"] > 2500:
        return None
    w0, ns, dt, method = (_f64(a) if a.dtype == np.float64 else torch.from_numpy(a).to(DEV) for a in _uneven(case, seed))
    out = torch.empty_like(w0)
    for code in (0, 1):
        idx = torch.nonzero(method == code).flatten()
        idx = idx[torch.argsort(ns[idx], descending=True)]
        n_of = ns[idx].cpu().numpy()
        x, v, h = w0[:3, idx].clone(), w0[3:, idx].clone(), dt[idx]
        vh = v - _grad("mw", x) * (h / 2) if code == 0 else None
        live = len(n_of)
        for j in range(int(n_of.max()) if live else 0):
            while live and n_of[live - 1] <= j:
                live -= 1
            X, Hh = x[:, :live], h[:live]
            if code == 0:
                X = X + vh[:, :live] * Hh
                g = _grad("mw", X)
                v[:, :live] = vh[:, :live] - g * (Hh / 2)
                vh[:, :live] -= g * Hh
            else:
                V = v[:, :live]
                for c, d in zip(RUTH_C, RUTH_D):
                    if d:
                        V = V - d * Hh * _grad("mw", X)
                    X = X + c * Hh * V
                v[:, :live] = V
            x[:, :live] = X
        out[:, idx] = torch.cat([x, v])

    def energy(w):
        return 0.5 * (w[3:] ** 2).sum(0) + _phi("mw", w[:3])

    e0 = energy(w0)
    return {"w": out, "dE": ((energy(out) - e0) / e0).abs()}


def _exact_surrogate(case, seed):
    """The network in FP64 with the FP32 weights it was given; the analytic gradient outside the trained radii."""
    q = _f64(_points(case["n"], seed, 0.4, 250.0))
    scf = _scf(12, 8)
    p = _f64(init_params(seed).astype(np.float64))
    r_min, r_max, rho0, rs, gm = 0.5, 200.0, 0.1, 20.0, G * 1e12
    r = q.norm(dim=0)
    n, L = q / r, math.log(r_max / r_min)
    rho, drho = rho0 + (1 - rho0) * torch.log(r / r_min) / L, (1 - rho0) / (r * L)
    a, o, slopes, Ws = (rho * n).T, 0, [], []
    for fan in (3, 256, 256, 256):
        Wm, o = p[o:o + 256 * fan].view(256, fan), o + 256 * fan
        zz = a @ Wm.T + p[o:o + 256]
        o += 256
        sg = torch.sigmoid(zz)
        a = zz * sg
        slopes.append(sg * (1 + zz * (1 - sg)))
        Ws.append(Wm)
    yv, d = a @ p[o:o + 256] + p[o + 256], p[o:o + 256].expand(q.shape[1], 256)
    for Wm, sl in zip(reversed(Ws), reversed(slopes)):
        d = (d * sl) @ Wm
    g = d.T
    l0 = gp.SCFPotential(m=1e12, r_s=rs, Snlm=scf.parameters["Snlm"][:, :1, :1], Tnlm=scf.parameters["Tnlm"][:, :1, :1])
    phi0, g0 = _scf_exact(l0, q, True)
    ph, dph = -gm / (r + rs), gm / (r + rs) ** 2
    ng = (n * g).sum(0)
    grad = g0 + dph * yv * n + ph * (rho / r * (g - n * ng) + drho * n * ng)
    phi = phi0 + ph * yv
    far = (r < r_min) | (r > r_max)
    # the potential is the network's everywhere, the gradient the analytic one outside
    return {"grad": torch.where(far, _scf_exact(scf, q, True)[1], grad), "phi": phi}


def _exact_extrema(case, seed):
    w, t = _rosettes(case, seed)
    out = {}
    r, az = (w[:3] ** 2).sum(0).sqrt(), w[2].abs()
    for name, f in (("peri", -r), ("apo", r), ("zmax", az)):
        a, b, c = f[:-2], f[1:-1], f[2:]
        peak = (b > a) & (b > c)
        val = b - (c - a) ** 2 / (8 * (a - 2 * b + c))  # vertex of the parabola through three even samples
        cnt = peak.sum(0)
        v = torch.where(peak, val, torch.zeros_like(val)).sum(0) / cnt
        v = torch.where(cnt > 0, -v if name == "peri" else v, torch.full_like(v, math.nan)).cpu().numpy()
        out[name] = v if case["n"] > 1 else float(v[0])
    return out


def exact(case, seed):
    k = case["kind"]
    if k == "points":
        q = _f64(_points(case["n"], seed, 0.1, 100.0))
        return {"phi": _phi("mw", q).cpu().numpy(), "grad": _grad("mw", q).cpu().numpy()}
    if k == "scf":
        phi, grad = _scf_exact(_scf(case["nmax"], case["lmax"]), _f64(_points(case["n"], seed, 0.5, 200.0)), True)
        return {"phi": phi.cpu().numpy(), "grad": grad.cpu().numpy()}
    if k == "dop853":
        return _exact_dop853(case, seed)
    if k == "fixed":
        w0 = _f64(_orbits(case["pot"], case["n"], seed))
        scf = _potential("scf") if case["pot"] == "scf" else None
        grad = (lambda q: _scf_exact(scf, q, True)[1]) if scf is not None else (lambda q: _grad(case["pot"], q))
        w = _fixed(grad, w0, case["dt"], case["n_steps"], case["integrator"], case["save_all"])
        # one orbit comes back without its axis, as the call returns it
        return w[..., 0] if case["n"] == 1 and case["save_all"] else w
    if k == "nbody":
        return _exact_nbody(case, seed)
    if k == "surrogate":
        return _exact_surrogate(case, seed)
    if k == "extrema":
        return _exact_extrema(case, seed)
    if k == "batch":
        return _exact_batch(case, seed)
    return None  # streams: the release radii come from a finite difference; training: a chain of optimiser steps
