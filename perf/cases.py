"""The work a user has this library do, as cases that can be timed and compared.

Four kinds, each through the package's public entry points:

* interval -- what the integrator classes do between two outputs of a
  simulation: upload a cloud's state, advance it (DeviceCloud.step, or
  move_particles with the reference's adaptive time step, which is the
  driver's default), download the state;
* monitor  -- the forces and the energy and momentum of a state, FP64;
* batch    -- many uneven clouds stepped together, then downloaded;
* fit      -- a differentiable rollout and the gradients of a trajectory loss.

Clouds are jittered triangular lattices: dust clouds settle into them, and
uniformly random positions hold pairs close enough for the time step to be
unstable.  ``phase`` is the phase [rad] of the harmonic motion a confined
cloud released from rest is in (0: at rest; near pi/2: shooting through the
trap's focus, where a large part of all pairs is inside the cutoff).
Constants are those of the package's workloads.
"""
import math

import numpy as np
import torch

from demon_simulation_code_gb300 import Context, DeviceBatch, DeviceCloud
from demon_simulation_code_gb300 import workloads as W
from demon_simulation_code_gb300.adjoint import AdjointKernels, rollout

Q, M, EPS0 = -1.6e-15, 2.81e-14, 8.8541878e-12
COULOMB = 1.0 / (4.0 * math.pi * EPS0)
# every force of the reference's driver except the three thermal ones
NOT_THERMAL = (W.CONFINEMENT | W.CONFINEMENT_VOID | W.DRAG | W.DRIVING | W.MAGNETIC | W.RECT_CONFINEMENT | W.ROTATIONAL
               | W.SHIELDED_COULOMB | W.TIME_VARYING_DRAG | W.ELECTRIC | W.GRAVITATIONAL | W.VERT_ELECTRIC)


def _interval(name, n, precision, steps, **kw):
    return {"name": name, "kind": "interval", "n": n, "precision": precision, "steps": steps, "dt": 1e-4,
            "adaptive": False, "order": 4, "forces": "basic", "spacing": 3e-4, "phase": 0.0, "kappa": 2e4,
            "confine": 1e8, "pinned": False, **kw}


def listed():
    return [
        # a few dozen grains coupled step by step to a host program: latency
        _interval("grains64", 64, "fp64", 1),
        # the 512-grain disk between two of its outputs, 100 steps apart
        # (weak confinement, long screening: a calm crystal)
        _interval("disk512", 512, "fp64", 100, kappa=5e3, confine=1e4, spacing=6e-4),
        # the driver's default: FP64 with the adaptive time step
        _interval("driver2048", 2048, "fp64", 6, adaptive=True, spacing=4e-4),
        # every deterministic force of the driver, its -I integrator (RK2), an odd size
        _interval("forces4095", 4095, "fp32c", 10, forces="all", order=2, dt=2e-5),
        # the package's headline configuration, with its thermal kicks, from pinned buffers
        _interval("disk16k", 16384, "fp32c", 4, forces="thermal", pinned=True),
        # the same cloud while its confinement pulls it through the focus, at
        # the time step the reference's own test picks for such separations
        _interval("focus16k", 16384, "fp32c", 3, dt=1e-6, phase=1.52, pinned=True),
        # a large cloud in full precision
        _interval("disk16k_fp64", 16384, "fp64", 1),
        # the largest: a rectangular trap, charges spread by 5%, short screening
        _interval("square256k", 262144, "fp32c", 2, forces="rect", kappa=5e4, dt=5e-5, spacing=2e-4, pinned=True),
        # energies and forces of a stored state under the driver's default
        # confinement, an odd size
        {"name": "monitor10007", "kind": "monitor", "n": 10007, "spacing": 2.5e-4, "phase": 0.0, "kappa": 2e4, "confine": 1e2},
        # the parameter sweep: 256 uneven clouds, each with its own constants
        {"name": "batch256", "kind": "batch", "clouds": 256, "nmin": 64, "nmax": 4096, "steps": 16, "dt": 1e-6},
        # a gradient in full precision, screening so long that every pair counts
        {"name": "fit_fp64", "kind": "fit", "clouds": 6, "nmin": 300, "nmax": 2048, "steps": 3, "precision": "fp64",
         "kappa": 400.0, "confine": 4e4, "spacing": 3.5e-4},
        # the trajectory fit's size, short screening: few pairs count
        {"name": "fit64_fp32c", "kind": "fit", "clouds": 64, "nmin": 2048, "nmax": 2048, "steps": 4, "precision": "fp32c",
         "kappa": 2e4, "confine": 1e8, "spacing": 3.5e-4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("interval", "interval", "interval", "monitor", "batch", "fit"))
    if kind == "interval":
        precision = rng.choice(("fp64", "fp32c"))
        n = _log(rng, 64, 16384 if precision == "fp64" else 131072)
        adaptive = rng.random() < 0.35 and n <= 16384
        n = max(4, n // 4 * 4) if adaptive else n
        steps = 1 if n > 8000 and precision == "fp64" else rng.randint(1, 3) if n > 4096 else rng.randint(1, 20)
        c = _interval("", n, precision, steps, adaptive=adaptive, order=rng.choice((4, 4, 2)),
                      forces=rng.choice(("basic", "thermal", "rect") if adaptive else ("basic", "thermal", "rect", "all")),
                      spacing=rng.uniform(2e-4, 5e-4), kappa=rng.uniform(1e4, 4e4), dt=rng.uniform(1e-5, 3e-5),
                      pinned=rng.random() < 0.5)
        if precision == "fp32c" and 4096 <= n <= 20000 and rng.random() < 0.3:
            c.update(phase=rng.uniform(1.3, 1.52), dt=1e-6, steps=min(steps, 3), kappa=2e4, spacing=3e-4, forces="basic")
        del c["name"]
        return c
    if kind == "monitor":
        return {"kind": "monitor", "n": _log(rng, 64, 12000), "spacing": rng.uniform(1.5e-4, 4e-4), "phase": 0.0,
                "kappa": rng.uniform(1e4, 4e4), "confine": rng.uniform(1e2, 1e4)}
    if kind == "batch":
        lo = rng.randint(32, 400)
        return {"kind": "batch", "clouds": _log(rng, 4, 256), "nmin": lo, "nmax": lo + rng.randint(0, 3500),
                "steps": rng.randint(1, 20), "dt": 1e-6}
    precision = rng.choice(("fp64", "fp32c"))
    lo = rng.randint(100, 1000)
    return {"kind": "fit", "clouds": rng.randint(1, 6) if precision == "fp64" else _log(rng, 2, 64), "nmin": lo,
            "nmax": lo + rng.randint(0, 1000), "steps": rng.randint(1, 4), "precision": precision,
            "kappa": rng.choice((400.0, rng.uniform(1e4, 3e4))), "confine": 4e4, "spacing": 3.5e-4}


def _lattice(rng, n, a, square=False):
    """n points of a triangular (square: square) lattice of spacing `a` nearest
    the origin, turned and shifted at random, each moved by up to a/10 per
    axis, in random order."""
    m = int(math.sqrt(n) * 1.1) + 4
    i, j = np.meshgrid(np.arange(-m, m + 1), np.arange(-m, m + 1))
    i, j = i.ravel().astype(float), j.ravel().astype(float)
    x, y = (i, j) if square else (i + 0.5 * (j % 2), j * math.sqrt(0.75))
    if square:
        key = np.maximum(np.abs(x + 0.5 * rng.random()), np.abs(y + 0.5 * rng.random()))
    else:
        x, y = x + rng.random(), y + rng.random()
        t = 2 * math.pi * rng.random()
        x, y = x * math.cos(t) - y * math.sin(t), x * math.sin(t) + y * math.cos(t)
        key = x * x + y * y
    near = rng.permutation(np.argpartition(key, n - 1)[:n])
    return a * (x[near] + rng.uniform(-0.1, 0.1, n)), a * (y[near] + rng.uniform(-0.1, 0.1, n))


def _cloud(c, seed):
    """The case's cloud as the package's own record of one."""
    rng = np.random.default_rng([seed, c["n"]])
    n, forces = c["n"], c.get("forces", "basic")
    x0, y0 = _lattice(rng, n, c["spacing"], square=forces == "rect")
    w = math.sqrt(-Q * c["confine"] / M)  # angular frequency of the confined motion
    cos, sin = math.cos(c["phase"]), math.sin(c["phase"])
    vx, vy = -w * sin * x0 + rng.normal(0, 1e-4, n), -w * sin * y0 + rng.normal(0, 1e-4, n)
    kw = {"flags": W.CONFINEMENT | W.DRAG | W.SHIELDED_COULOMB, "confine": c["confine"]}
    q = np.full(n, Q)
    if forces == "thermal":
        kw.update(flags=kw["flags"] | W.THERMAL, heat=1e-14, seed=seed)
    elif forces == "rect":
        kw = {"flags": W.RECT_CONFINEMENT | W.DRAG | W.SHIELDED_COULOMB, "confine": 0.0, "confine_x": 1e8, "confine_y": 1e8}
        q = rng.normal(Q, 0.05 * abs(Q), n)
    elif forces == "all":
        kw.update(flags=NOT_THERMAL, confine_x=1e7, confine_y=2e7, extra=dict(W.OTHER_FORCES))
    return W.Cloud(x=cos * x0, y=cos * y0, vx=vx, vy=vy, q=q, m=np.full(n, M), shielding=c["kappa"], gamma=3.0, **kw)


def _sizes(c):
    """Cloud sizes from nmin to nmax; whole groups of 32 grains for a 32-bit
    fit, as in the package's own (any size in the others)."""
    unit = 32 if c.get("precision") == "fp32c" else 1
    return [max(1, round(v / unit)) * unit for v in np.linspace(c["nmin"], c["nmax"], c["clouds"]).tolist()]


def _batch_clouds(c, seed):
    rng = np.random.default_rng([seed, c["clouds"]])
    out = []
    for n in rng.permutation(_sizes(c)):
        x, y = _lattice(rng, int(n), 3.8e-4)
        # 2e-3 m/s: a kinetic temperature of about an electron volt
        out.append(W.Cloud(x=x, y=y, vx=rng.normal(0, 2e-3, n), vy=rng.normal(0, 2e-3, n),
                           q=np.full(n, rng.uniform(-2e-15, -1e-15)), m=np.full(n, M),
                           shielding=rng.uniform(1e4, 5e4), confine=rng.uniform(5e3, 2e4), gamma=3.0))
    return out


def _fit_inputs(c, seed):
    """Start state, masses, targets, and the per-cloud (kappa, q, k_c) of a fit."""
    rng = np.random.default_rng([seed, c["clouds"]])
    ns = _sizes(c)
    xy = [_lattice(rng, n, c["spacing"]) for n in ns]
    x, y = np.concatenate([p[0] for p in xy]), np.concatenate([p[1] for p in xy])
    s = [x, y, rng.normal(0, 1e-4, len(x)), rng.normal(0, 1e-4, len(x))]
    target = [0.97 * x + rng.normal(0, 1e-5, len(x)), 0.97 * y + rng.normal(0, 1e-5, len(x))]
    f = 1.0 + rng.uniform(-0.2, 0.2, (3, len(ns)))
    theta = [c["kappa"] * f[0], Q * f[1], c["confine"] * f[2]]
    dev = [torch.tensor(v, dtype=torch.float64, device="cuda") for v in s + target + theta + [np.full(len(x), M)]]
    return ns, dev[:4], dev[4:6], dev[6:9], dev[9]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fit":
        ns, s, target, theta, m = _fit_inputs(case, seed)
        K = AdjointKernels(ns, precision=case["precision"])
        return {"case": case, "K": K, "s": s, "target": target, "theta": theta, "m": m}
    ctx = Context(0)
    if kind == "batch":
        return {"case": case, "ctx": ctx, "batch": DeviceBatch(ctx, _batch_clouds(case, seed))}
    c = _cloud(case, seed)
    cloud = DeviceCloud.from_cloud(ctx, c)
    if kind == "monitor":
        cloud.autotune("fp64")
        return {"case": case, "ctx": ctx, "cloud": cloud}
    cloud.set_integrator(case["order"])
    cloud.autotune(case["precision"])
    start, out = [c.x, c.y, c.vx, c.vy], None
    if case["pinned"]:
        start = [torch.from_numpy(v).pin_memory().numpy() for v in start]
        out = [torch.empty(c.n, dtype=torch.float64, pin_memory=True).numpy() for _ in range(4)]
    return {"case": case, "ctx": ctx, "cloud": cloud, "start": start, "out": out}


def run(state):
    case = state["case"]
    if case["kind"] == "interval":
        cloud = state["cloud"]
        cloud.upload(*state["start"])
        if case["forces"] == "thermal":
            cloud.set_step_counter(0)  # the same kicks in every pass
        if case["adaptive"]:
            t, steps = cloud.move_particles((case["steps"] - 0.5) * case["dt"], case["dt"], 0.0, case["precision"], adaptive=True)
            return {"state": cloud.download(state["out"]), "time": t, "steps": steps}
        t = cloud.step(case["steps"], case["dt"], case["precision"], t=0.0)
        return {"state": cloud.download(state["out"]), "time": t}
    if case["kind"] == "monitor":
        return {"forces": state["cloud"].eval_forces("fp64"), "energies": state["cloud"].diagnostics()}
    if case["kind"] == "batch":
        state["batch"].step(case["steps"], case["dt"])
        return {"state": state["batch"].download()}
    leaves = [v.detach().requires_grad_(True) for v in state["s"] + state["theta"]]
    x, y, vx, vy = rollout(state["K"], *leaves, state["m"], 1e-4, case["steps"])
    loss = ((x - state["target"][0]) ** 2 + (y - state["target"][1]) ** 2).mean()
    return {"loss": loss.detach(), "state": [v.detach() for v in (x, y, vx, vy)], "grads": torch.autograd.grad(loss, leaves)}


def _pairs(n, kappa, a):
    """Ordered pairs inside the cutoff of n grains at spacing `a`."""
    return n * min(n - 1.0, math.pi * (10.0 / kappa) ** 2 / (math.sqrt(0.75) * a * a))


def work(case):
    """Each array across the interface once; 23 operations a pair inside the
    cutoff (93 with its vector-Jacobian product) and 60 a grain, for each
    force evaluation."""
    if case["kind"] in ("interval", "monitor"):
        n = case["n"]
        evals = case["order"] * case["steps"] if case["kind"] == "interval" else 1
        a = case["spacing"] * math.cos(case["phase"])
        return {"bytes": 64.0 * n, "flops": evals * (23.0 * _pairs(n, case["kappa"], a) + 60.0 * n)}
    ns = _sizes(case)
    if case["kind"] == "batch":
        return {"bytes": 64.0 * sum(ns), "flops": 4 * case["steps"] * sum(23.0 * _pairs(n, 2.5e4, 3.8e-4) + 60.0 * n for n in ns)}
    return {"bytes": 96.0 * sum(ns), "flops": 4 * case["steps"] * sum(116.0 * _pairs(n, case["kappa"], case["spacing"]) + 200.0 * n for n in ns)}


# --- the same results in plain 64-bit arithmetic -----------------------------

def _pair_force(x, y, q, kappa):
    """The shielded Coulomb force on every grain of one cloud, all pairs."""
    fx, fy = [], []
    rows = max(1, int(3e7) // len(x))
    for r in range(0, len(x), rows):
        dx, dy = x[r:r + rows, None] - x[None, :], y[r:r + rows, None] - y[None, :]
        r2 = dx * dx + dy * dy
        far = r2 == 0.0
        d = torch.where(far, torch.ones_like(r2), r2).sqrt()
        a = kappa * d
        f = torch.where((a < 10.0) & ~far, COULOMB * q[r:r + rows, None] * q[None, :] * (1.0 + a) * torch.exp(-a) / (d * d * d), 0.0)
        fx.append((f * dx).sum(1))
        fy.append((f * dy).sum(1))
    return torch.cat(fx), torch.cat(fy)


def _kicks(seed, n, step, stage, heat):
    """Gaussian kicks from Philox4x32-10 with counter (grain, step, 0, stage)."""
    mask = np.uint64(0xFFFFFFFF)
    c = [np.arange(n, dtype=np.uint64), np.full(n, step, np.uint64), np.zeros(n, np.uint64), np.full(n, stage, np.uint64)]
    k0, k1 = seed & 0xFFFFFFFF, seed >> 32
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & mask, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = [((v >> np.uint64(8)).astype(float) + 0.5) * 2.0 ** -24 for v in c[:2]]
    amp = heat * np.sqrt(-2.0 * np.log(u[0]))
    return [torch.tensor(amp * f(2 * math.pi * u[1]), device="cuda") for f in (np.cos, np.sin)]


def _total_force(c, x, y, vx, vy, q, m, t, step, stage):
    """Every force of the cloud's flags."""
    fl, e = c.flags, c.extra
    r = (x * x + y * y).sqrt()
    fx, fy = _pair_force(x, y, q, c.shielding)
    k = c.confine * (bool(fl & W.CONFINEMENT) + bool(fl & W.CONFINEMENT_VOID))
    g = c.gamma * bool(fl & W.DRAG) + (e["drag_scale"] * t + e["drag_offset"] if fl & W.TIME_VARYING_DRAG else 0.0)
    rect = bool(fl & W.RECT_CONFINEMENT)
    fx = fx + q * (k + rect * c.confine_x) * x - g * m * vx
    fy = fy + q * (k + rect * c.confine_y) * y - g * m * vy
    if fl & W.CONFINEMENT_VOID:
        s = -q * e["void_decay"] * torch.exp(-e["void_decay"] * r) / r
        fx, fy = fx + s * x, fy + s * y
    if fl & W.DRIVING:
        fx = fx + e["drive_amplitude"] * torch.sin(x * (2 * math.pi / 0.002) - t * 2 * math.pi * 10.0)
    if fl & W.MAGNETIC:
        fx, fy = fx + q * e["magnetic"] * vy, fy - q * e["magnetic"] * vx
    if fl & W.ROTATIONAL:
        s = torch.where((r > e["rot_rmin"]) & (r < e["rot_rmax"]), e["rot_const"] / r, 0.0)
        fx, fy = fx - s * y, fy + s * x
    if fl & W.ELECTRIC:
        s = q * e["electric"] * torch.exp(-r / e["electric_radius"])
        fx, fy = fx + s * x, fy + s * y
    if fl & W.GRAVITATIONAL:
        fy = fy + m * e["gravity"]
    if fl & W.VERT_ELECTRIC:
        fy = fy + q * e["vert_electric"] * torch.exp(y / e["vert_decay"])
    if fl & W.THERMAL:
        kick = _kicks(c.seed, len(x), step, stage, c.heat)
        fx, fy = fx + kick[0], fy + kick[1]
    return fx, fy


def _advance(force, s, m, dt, order, t):
    """One RK4 (order 2: midpoint) step of s = (x, y, vx, vy)."""
    def rate(stage, s, t):
        fx, fy = force(*s, t, stage)
        return (s[2], s[3], fx / m, fy / m)

    def moved(k, f):
        return tuple(a + f * dt * b for a, b in zip(s, k))

    k1 = rate(1, s, t)
    k2 = rate(2, moved(k1, 0.5), t + 0.5 * dt)
    if order == 2:
        return moved(k2, 1.0)
    k3 = rate(3, moved(k2, 0.5), t + 0.5 * dt)
    k4 = rate(4, moved(k3, 1.0), t + dt)
    return tuple(a + dt * (p + 2 * (q + r) + w) / 6.0 for a, p, q, r, w in zip(s, k1, k2, k3, k4))


def _tested_dt(x, y, dt):
    """The reference's adaptive time step: the least separation, in 32 bits,
    of the pairs it looks at (grain k of a block of four against grains k,
    k-1, k-2 mod 4 of every later block, and all pairs inside a block)."""
    x, y, n = x.float(), y.float(), len(x)
    i = torch.arange(n, device=x.device)
    least, rows = math.inf, max(1, int(6e7) // n)
    for r in range(0, n, rows):
        a = i[r:r + rows, None]
        seen = (i[None, :] // 4 > a // 4) & ((a - i[None, :]) % 4 != 3) | (i[None, :] // 4 == a // 4) & (i[None, :] > a)
        d2 = (x[r:r + rows, None] - x[None, :]) ** 2 + (y[r:r + rows, None] - y[None, :]) ** 2
        least = min(least, float(torch.where(seen, d2, math.inf).min().sqrt()))
    dist = np.float32(1e-4)
    while least <= dist:
        dist, dt = np.float32(dist / np.float32(10.0)), dt / 10.0
    return dt


def _exact_interval(case, seed):
    c = _cloud(case, seed)
    s = tuple(torch.tensor(v, device="cuda") for v in (c.x, c.y, c.vx, c.vy))
    q, m = (torch.tensor(v, device="cuda") for v in (c.q, c.m))
    t, step, end = 0.0, 0, (case["steps"] - 0.5) * case["dt"]
    while t < end if case["adaptive"] else step < case["steps"]:
        dt = _tested_dt(s[0], s[1], case["dt"]) if case["adaptive"] else case["dt"]
        s = _advance(lambda x, y, vx, vy, at, k: _total_force(c, x, y, vx, vy, q, m, at, step, k), s, m, dt, case["order"], t)
        t, step = t + dt, step + 1
    return {"state": s, "time": t, "steps": step} if case["adaptive"] else {"state": s, "time": t}


def _exact_monitor(case, seed):
    c = _cloud(case, seed)
    x, y, vx, vy, q, m = (torch.tensor(v, device="cuda") for v in (c.x, c.y, c.vx, c.vy, c.q, c.m))
    potential = torch.zeros((), dtype=torch.float64, device="cuda")
    rows = max(1, int(3e7) // c.n)
    for r in range(0, c.n, rows):
        d = ((x[r:r + rows, None] - x[None, :]) ** 2 + (y[r:r + rows, None] - y[None, :]) ** 2).sqrt()
        keep = (c.shielding * d < 10.0) & (d > 0.0)
        d = torch.where(keep, d, torch.ones_like(d))
        potential += torch.where(keep, COULOMB * q[r:r + rows, None] * q[None, :] * torch.exp(-c.shielding * d) / d, 0.0).sum()
    energies = torch.stack([(0.5 * m * (vx * vx + vy * vy)).sum(), 0.5 * potential,
                            (-0.5 * q * c.confine * (x * x + y * y)).sum(), (m * vx).sum(), (m * vy).sum()])
    return {"forces": _total_force(c, x, y, vx, vy, q, m, 0.0, 0, 1), "energies": energies}


def _exact_fit(case, seed):
    ns, s, target, theta, m = _fit_inputs(case, seed)
    total, loss, states, grads = sum(ns), 0.0, [], []
    at = 0
    for c, n in enumerate(ns):
        part = slice(at, at + n)
        leaves = [v[part].clone().requires_grad_(True) for v in s] + [v[c].clone().requires_grad_(True) for v in theta]
        kappa, qc, kc = leaves[4:]
        mm, at = m[part], at + n

        def force(x, y, vx, vy, t, stage):
            q = qc.expand(len(x))
            fx, fy = _pair_force(x, y, q, kappa)
            return fx + qc * kc * x - 3.0 * mm * vx, fy + qc * kc * y - 3.0 * mm * vy

        now = tuple(leaves[:4])
        for _ in range(case["steps"]):
            now = _advance(force, now, mm, 1e-4, 4, 0.0)
        part_loss = ((now[0] - target[0][part]) ** 2 + (now[1] - target[1][part]) ** 2).sum() / total
        g = torch.autograd.grad(part_loss, leaves)
        loss = loss + part_loss.detach()
        states.append([v.detach() for v in now])
        grads.append(g)
    joined = [torch.cat([g[k] for g in grads]) for k in range(4)] + [torch.stack([g[k] for g in grads]) for k in range(4, 7)]
    return {"loss": loss, "state": [torch.cat([v[k] for v in states]) for k in range(4)], "grads": joined}


def _exact_batch(case, seed):
    out = []
    for c in _batch_clouds(case, seed):
        s = tuple(torch.tensor(v, device="cuda") for v in (c.x, c.y, c.vx, c.vy))
        q, m = (torch.tensor(v, device="cuda") for v in (c.q, c.m))
        for _ in range(case["steps"]):
            s = _advance(lambda x, y, vx, vy, t, k: _total_force(c, x, y, vx, vy, q, m, t, 0, k), s, m, case["dt"], 4, 0.0)
        out.append(s)
    return {"state": [torch.cat([s[k] for s in out]) for k in range(4)]}


def exact(case, seed):
    kind = case["kind"]
    sizes = [case["n"]] if kind in ("interval", "monitor") else _sizes(case)
    evals = 1 if kind == "monitor" else 4 * case["steps"] * (10 if kind == "fit" else 1)
    if sum(n * n for n in sizes) * evals > 1.2e11 or len(sizes) * evals > 20000:
        return None
    return {"interval": _exact_interval, "monitor": _exact_monitor, "batch": _exact_batch, "fit": _exact_fit}[kind](case, seed)
