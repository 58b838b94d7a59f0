"""Performance cases: what programs that use this propagator have it do.

Each case is one call sequence through ``parahpop_b200.api`` on synthetic
environments and populations of the shapes the benchmark and the tests use:

* ``propagate``   host arrays in, final epochs and states out
                  (``Propagator.propagate``; one epoch, duration and step)
* ``resident``    the same with the state kept in device memory
                  (``Propagator.propagate_device``)
* ``trajectory``  states after every k-th step (``Propagator.trajectory``)
* ``uneven``      a device-resident batch with per-object epochs, steps and
                  ends, advanced by a slice of steps
                  (``Propagator.propagate_device_objects``)
* ``serving``     requests of different sizes and durations submitted to a
                  resident server and run to completion (``Server``)

Force models: ``central`` (point mass), ``zonal`` (J2-J6), ``field``
(spherical-harmonic field to ``degree``, nothing else), ``full`` (that field,
Sun, Moon, Jupiter, SRP with shadow, NRLMSISE-00 drag, solid and ocean tides,
relativity), in FP64 or in split precision.
"""
import atexit
import json
import math
import shutil
import tempfile
from pathlib import Path

import numpy as np
import torch

from parahpop_b200 import api
from parahpop_b200 import synthetic as S

EPOCH = 4035.0      # MJD2000 TDB, the common epoch of the benchmark's batches
FIELD_DEGREE = 120  # degree of the synthetic field file; configurations truncate it


def listed():
    return [
        # the smallest call: one object, the point-mass model, ten minutes
        {"name": "central_1", "kind": "propagate", "force": "central", "degree": 0, "split": False,
         "objects": 1, "steps": 10, "step": 60.0},
        # 1,024 objects on the point-mass model for 600 s at 60 s (a first check of a catalogue)
        {"name": "central_1024", "kind": "propagate", "force": "central", "degree": 0, "split": False,
         "objects": 1024, "steps": 10, "step": 60.0},
        # an hour's ephemeris of a small constellation on J2-J6, a state every six minutes
        {"name": "zonal_trajectory_333", "kind": "trajectory", "force": "zonal", "degree": 6, "split": False,
         "objects": 333, "steps": 60, "step": 60.0, "every": 6},
        # a small full-force request: a few objects, ten minutes, where latency counts
        {"name": "full70_33", "kind": "propagate", "force": "full", "degree": 70, "split": False,
         "objects": 33, "steps": 10, "step": 60.0},
        # the gravity field alone on a batch that stays on the device
        {"name": "field70_5000", "kind": "resident", "force": "field", "degree": 70, "split": False,
         "objects": 5000, "steps": 10, "step": 60.0},
        # 10^4 LEO objects, full force at degree 70, twenty minutes of a day's run
        {"name": "full70_10000", "kind": "propagate", "force": "full", "degree": 70, "split": False,
         "objects": 10000, "steps": 20, "step": 60.0},
        {"name": "full70_10000_split", "kind": "propagate", "force": "full", "degree": 70, "split": True,
         "objects": 10000, "steps": 20, "step": 60.0},
        # degree 120: an odd-sized batch in FP64 and 10^5 objects in split precision
        {"name": "full120_20011", "kind": "resident", "force": "full", "degree": 120, "split": False,
         "objects": 20011, "steps": 4, "step": 60.0},
        {"name": "full120_100000_split", "kind": "resident", "force": "full", "degree": 120, "split": True,
         "objects": 100000, "steps": 4, "step": 60.0},
        # slices of the uneven LEO / MEO / GEO population, in both precisions (the benchmark's workload)
        {"name": "uneven70_200000", "kind": "uneven", "force": "full", "degree": 70, "split": False,
         "objects": 200000, "steps": 8, "step": 0.0},
        {"name": "uneven70_1000000_split", "kind": "uneven", "force": "full", "degree": 70, "split": True,
         "objects": 1000000, "steps": 4, "step": 0.0},
        # forty requests of 1 to 3,000 objects and 10 minutes to 2 hours, served together
        {"name": "serving70_40_split", "kind": "serving", "force": "full", "degree": 70, "split": True,
         "objects": 3000, "requests": 40, "step": 60.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    kind = rng.choice(["propagate", "propagate", "resident", "trajectory", "uneven", "uneven", "serving"])
    force = rng.choice(["central", "zonal", "field", "full", "full", "full"])
    if kind == "uneven":
        force = rng.choice(["field", "full", "full"])
    if kind == "serving":
        force = rng.choice(["zonal", "full", "full"])
    degree = {"central": 0, "zonal": 6}.get(force) if force in ("central", "zonal") else rng.choice(
        [20, 36, 55, 70, 70, 90, 120])
    c = {"kind": kind, "force": force, "degree": degree, "split": force in ("field", "full") and rng.random() < 0.5}
    if kind == "uneven":
        c |= {"objects": _log_int(rng, 3000, 500000), "steps": rng.randint(1, 12), "step": 0.0}
    elif kind == "serving":
        c |= {"objects": _log_int(rng, 50, 3000), "requests": rng.randint(5, 40), "step": 60.0}
    else:
        c |= {"objects": _log_int(rng, 1, 100000 if kind != "trajectory" else 3000), "steps": rng.randint(2, 60),
              "step": rng.choice([20.0, 30.0, 60.0])}
        if kind == "trajectory":
            c["every"] = rng.randint(1, 7)
            c["steps"] = max(c["steps"], c["every"])
    while work(c)["flops"] > 0.5 * most and c.get("steps", 0) > max(2, c.get("every", 0)):
        c["steps"] -= 1
    while work(c)["flops"] > 0.5 * most:
        c["objects"] = max(1, c["objects"] // 2)
    return c


# ---- environments and populations ----------------------------------------------------------
_made = {}


def _once(key, make):
    if key not in _made:
        _made[key] = make()
    return _made[key]


def _environment(zonal):
    def make():
        root = Path(tempfile.mkdtemp(prefix="phop_cases_"))
        atexit.register(shutil.rmtree, root, ignore_errors=True)
        return S.write_environment(root, S.EnvSpec(degree=6 if zonal else FIELD_DEGREE, zonal_only=zonal))
    return _once(("environment", zonal), make)


def _config(case):
    """Path of the case's configuration file."""
    env = _environment(case["force"] == "zonal")
    name = "%s_%d.json" % (case["force"], case["degree"])

    def make():
        cfg = S.make_config(env, 3600.0, 60.0, force=case["force"], degree=case["degree"] or 70)
        (env / name).write_text(json.dumps(cfg))
        return env / name
    return _once(("config", env / name), make)


def _propagator(case):
    """The handle a program keeps for a configuration and precision."""
    return _once(("propagator", case["force"], case["degree"], case["split"]),
                 lambda: api.Propagator(_config(case), split=case["split"]))


def _population(case, n, seed):
    """`n` objects of the case's population: orbits, masses and areas of a
    base draw, each turned about the Earth's axis by an angle of its own, so
    that the nodes are uniform and every seed gives other objects."""
    if case["kind"] in ("uneven", "serving"):
        base = _once("mixed", lambda: S.population_mixed(100000, seed=3))
    elif case["force"] == "central":
        base = _once("central", lambda: S.population_central(1024, seed=0))
    else:
        base = _once("leo", lambda: S.population_leo(30000, seed=1))
    rng = np.random.default_rng(seed)
    pop = base.subset(rng.integers(0, len(base), n))
    turn = rng.uniform(0.0, 2.0 * math.pi, n)
    c, s = np.cos(turn), np.sin(turn)
    states = pop.states.copy()
    for k in (0, 3):
        x, y = pop.states[:, k], pop.states[:, k + 1]
        states[:, k], states[:, k + 1] = c * x - s * y, s * x + c * y
    pop.states = states
    return pop


def _arrays(pop):
    return pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr


def prepare(case, seed):
    n = case["objects"]
    if case["kind"] == "serving":
        rng = np.random.default_rng(seed)
        # a server uses its context alone, so it has one of its own
        prop = api.Propagator(_config(case), split=case["split"])
        requests = []
        for u in np.random.default_rng(case["requests"]).uniform(0.0, math.log(n), case["requests"]):
            pop = _population(case, int(math.exp(u)), int(rng.integers(1 << 31)))
            duration = math.exp(rng.uniform(math.log(600.0), math.log(7200.0)))
            requests.append((pop.epochs, pop.states, *_arrays(pop), duration, case["step"]))
        return {"case": case, "server": api.Server(prop, capacity=200000), "requests": requests}
    prop = _propagator(case)
    pop = _population(case, n, seed)
    state = {"case": case, "prop": prop, "pop": pop}
    if case["kind"] == "uneven":
        bc, ams = prop.factors(*_arrays(pop))
        times = prop.object_times(pop.epochs, pop.duration, pop.step)
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        state |= {"begin": (up(pop.states.T).reshape(-1), up(times)), "bc": up(bc), "ams": up(ams)}
        state["work"] = tuple(torch.empty_like(t) for t in state["begin"])
    elif case["kind"] == "resident":
        state["begin"] = torch.from_numpy(np.ascontiguousarray(pop.states.T)).cuda().reshape(-1)
        state["work"] = torch.empty_like(state["begin"])
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "serving":
        server = state["server"]
        ids = [server.submit(*r) for r in state["requests"]]
        server.run_until_idle()
        got = [server.take(i)[:2] for i in ids]
        return np.concatenate([e for e, _ in got]), np.concatenate([s for _, s in got])
    prop, pop = state["prop"], state["pop"]
    duration = case["steps"] * case["step"]
    if case["kind"] == "propagate":
        return prop.propagate(np.full(len(pop), EPOCH), pop.states, *_arrays(pop), duration, case["step"])
    if case["kind"] == "trajectory":
        return prop.trajectory(EPOCH, pop.states, *_arrays(pop), duration, case["step"], every=case["every"])
    if case["kind"] == "resident":
        state["work"].copy_(state["begin"])
        end = prop.propagate_device(state["work"].data_ptr(), len(pop), EPOCH, *_arrays(pop), duration, case["step"])
        return end, state["work"]
    for a, b in zip(state["work"], state["begin"]):
        a.copy_(b)
    soa, times = state["work"]
    left = prop.propagate_device_objects(len(pop), soa.data_ptr(), times.data_ptr(), state["bc"].data_ptr(),
                                         state["ams"].data_ptr(), case["steps"])
    return left, soa, times


def work(case):
    """States, factors and times read and written once, and the tables; per
    step twelve force evaluations (the thirteenth stage only serves the error
    estimate that a fixed step has no use for).  A term of the field: one
    Legendre recurrence (3 fused operations) and six sums; the other forces by
    a count of their formulas."""
    terms = 0 if case["force"] == "central" else (case["degree"] + 1) * (case["degree"] + 2) // 2
    if case["force"] == "zonal":
        terms = 7
    per_eval = 60.0 + 18.0 * terms + (2500.0 if case["force"] == "full" else 0.0)
    n = float(case["objects"])
    if case["kind"] == "serving":
        n *= case["requests"] / max(1.0, math.log(case["objects"]))  # the mean of log-uniform sizes
        object_steps = n * 44.0  # and of the steps of log-uniform durations of 10 min to 2 h at 60 s
    else:
        object_steps = n * case["steps"]
    records = case["steps"] // case["every"] if case["kind"] == "trajectory" else 1
    return {"bytes": n * (48.0 + 16.0 + 48.0 * records + (40.0 if case["kind"] == "uneven" else 0.0))
            + 8.0 * 8.0 * terms,
            "flops": object_steps * (12.0 * per_eval + 600.0)}


# ---- the same results in plain 64-bit torch, for the models without the atmosphere -------------
_A = [[], [2 / 27], [1 / 36, 1 / 12], [1 / 24, 0, 1 / 8], [5 / 12, 0, -25 / 16, 25 / 16], [1 / 20, 0, 0, 1 / 4, 1 / 5],
      [-25 / 108, 0, 0, 125 / 108, -65 / 27, 125 / 54], [31 / 300, 0, 0, 0, 61 / 225, -2 / 9, 13 / 900],
      [2, 0, 0, -53 / 6, 704 / 45, -107 / 9, 67 / 90, 3],
      [-91 / 108, 0, 0, 23 / 108, -976 / 135, 311 / 54, -19 / 60, 17 / 6, -1 / 12],
      [2383 / 4100, 0, 0, -341 / 164, 4496 / 1025, -301 / 82, 2133 / 4100, 45 / 82, 45 / 164, 18 / 41],
      [3 / 205, 0, 0, 0, 0, -6 / 41, -3 / 205, -3 / 41, 3 / 41, 6 / 41, 0],
      [-1777 / 4100, 0, 0, -341 / 164, 4496 / 1025, -289 / 82, 2193 / 4100, 51 / 82, 33 / 164, 12 / 41, 0, 1]]
_C = [0, 2 / 27, 1 / 9, 1 / 6, 5 / 12, 1 / 2, 5 / 6, 1 / 6, 2 / 3, 1 / 3, 1, 0, 1]
_B = [0, 0, 0, 0, 0, 34 / 105, 9 / 35, 9 / 35, 9 / 280, 9 / 280, 0, 41 / 840, 41 / 840]


def _earth_rotation(t):
    """ICRF to the Earth's frame at TDB seconds past J2000, (n, 3, 3): the
    IERS chain for the synthetic series (X, Y, s smooth, no polar motion,
    UT1 - TT constant)."""
    tdb = t / 86400.0 + 0.5
    g = math.radians(357.53) + math.radians(0.9856003) * (tdb - 0.5)
    corr = (0.001658 * torch.sin(g) + 0.000014 * torch.sin(2 * g)) / 86400.0
    tt = tdb - corr
    cy = tt / 36525.0
    X = 1.1e-3 + 9.7e-3 * cy + 4.0e-8 * torch.sin(2 * math.pi * tt / 13.66)
    Y = -3.0e-5 + 1.0e-6 * cy + 3.0e-8 * torch.cos(2 * math.pi * tt / 13.66)
    s = -1.0e-8 - 5.0e-10 * cy
    ut1_tt = (0.3 - 32.184 - 34.0) / 86400.0
    days = tt - 0.5 + ut1_tt
    frac = (t / 86400.0) % 1.0 - corr + ut1_tt
    theta = 2 * math.pi * ((frac + 0.7790572732640 + 0.00273781191135448 * days) % 1.0)
    theta = theta + -6.24e-15 * (tt - 0.5)

    def rz(a):
        c, n, z = torch.cos(a), torch.sin(a), torch.zeros_like(a)
        return torch.stack([c, n, z, -n, c, z, z, z, torch.ones_like(a)], -1).reshape(-1, 3, 3)

    def ry(a):
        c, n, z = torch.cos(a), torch.sin(a), torch.zeros_like(a)
        return torch.stack([c, z, -n, z, torch.ones_like(a), z, n, z, c], -1).reshape(-1, 3, 3)

    e, d = torch.atan2(Y, X), torch.asin(torch.sqrt(X * X + Y * Y))
    return rz(theta - s - e) @ ry(d) @ rz(e)


def _field_table(case, device):
    """Radius, GM and per degree n = 1.. the factors of the gradient's terms
    (normalised solid harmonics one degree up) and of the recurrence."""
    rows = np.loadtxt(_environment(case["force"] == "zonal") / "gravity.tab", delimiter=",", skiprows=1)
    head = (_environment(case["force"] == "zonal") / "gravity.tab").read_text().split("\n", 1)[0].split(",")
    N = case["degree"]
    C, D = np.zeros((2, N + 2, N + 3))
    for n, m, c, s in rows[:, :4]:
        if n <= N:
            C[int(n), int(m)], D[int(n), int(m)] = c, s
    m = np.arange(N + 3, dtype=float)
    steps = []
    for n in range(N + 1):
        k = np.sqrt((2 * n + 1) / (2 * n + 3))
        on = m <= n
        up = np.where(on, k * np.sqrt(np.where(m == 0, 0.5, 1.0) * (n + m + 2) * (n + m + 1)), 0.0)
        down = np.where(on & (m > 0), k * np.sqrt(np.abs(np.where(m == 1, 2.0, 1.0) * (n - m + 2) * (n - m + 1))), 0.0)
        zed = np.where(on, k * np.sqrt(np.abs((n + m + 1) * (n - m + 1))), 0.0)
        with np.errstate(divide="ignore", invalid="ignore"):
            a = np.where(on, np.sqrt((2 * n + 1) * (2 * n + 3) / ((n + 1 - m) * (n + 1 + m))), 0.0)
            b = np.where(m < n, np.sqrt((2 * n + 3) * (n + m) * (n - m) / ((2 * n - 1) * (n + 1 + m) * (n + 1 - m))), 0.0)
        diag = math.sqrt(3.0) if n == 0 else math.sqrt((2 * n + 3) / (2 * n + 2))
        steps.append([torch.tensor(v, dtype=torch.float64, device=device)[:, None]
                      for v in (up * C[n], up * D[n], down * C[n], down * D[n], zed * C[n], zed * D[n], a, b)] + [diag])
    return float(head[0]), float(head[1]), steps


def _field(table, pos):
    """Acceleration of the field (degrees 1 and up) at body-fixed positions (n, 3)."""
    R, gm, steps = table
    r2 = (pos * pos).sum(1)
    x, y, z = (pos[:, k] * R / r2 for k in range(3))
    rho = R * R / r2
    M = len(steps[0][0])
    V, W, V1, W1 = (torch.zeros(M, len(pos), dtype=torch.float64, device=pos.device) for _ in range(4))
    V[0] = R / torch.sqrt(r2)
    acc = torch.zeros_like(pos)
    for n, (cu, du, cd, dd, cz, dz, a, b, diag) in enumerate(steps):
        Vn, Wn = a * z * V - b * rho * V1, a * z * W - b * rho * W1
        Vn[n + 1], Wn[n + 1] = diag * (x * V[n] - y * W[n]), diag * (x * W[n] + y * V[n])
        V1, W1, V, W = V, W, Vn, Wn
        vu, wu, vd, wd = V[1:], W[1:], V[:-1], W[:-1]
        ax = (-cu[:-1] * vu - du[:-1] * wu).sum(0) + (cd[1:] * vd + dd[1:] * wd).sum(0)
        ay = (-cu[:-1] * wu + du[:-1] * vu).sum(0) + (-cd[1:] * wd + dd[1:] * vd).sum(0)
        ax0, ay0 = -cu[0] * V[1], -cu[0] * W[1]  # order 0 has one term, not half of two
        acc[:, 0] += 0.5 * (ax - ax0) + ax0
        acc[:, 1] += 0.5 * (ay - ay0) + ay0
        acc[:, 2] -= (cz * V + dz * W).sum(0)
    return acc * (gm / (R * R))


def exact(case, seed):
    if case["force"] == "full" or case["kind"] == "serving":
        return None
    if float(case["objects"]) * case["steps"] * (case["degree"] + 1) ** 2 > 6e9:
        return None  # minutes in plain torch
    device = "cuda" if torch.cuda.is_available() else "cpu"
    pop = _population(case, case["objects"], seed)
    up = lambda a: torch.tensor(np.asarray(a), dtype=torch.float64, device=device)  # noqa: E731
    n = len(pop)
    gm = {k["NAME"]: k["GM"] for k in S.CONSTANTS if "NAME" in k}["Earth"]
    table = _field_table(case, device) if case["force"] != "central" else None
    y = up(pop.states)
    to_et = lambda mjd: mjd * 86400.0 - 43200.0  # noqa: E731
    if case["kind"] == "uneven":
        cur, step = to_et(up(pop.epochs)), up(pop.step)
        end = to_et(up(pop.epochs) + up(pop.duration) / 86400.0)
    else:
        cur = to_et(torch.full((n,), EPOCH, dtype=torch.float64, device=device))
        step = torch.full_like(cur, case["step"])
        end = to_et(torch.full_like(cur, EPOCH) + case["steps"] * case["step"] / 86400.0)
    dt = torch.minimum(step, end - cur)
    times0 = step.clone()

    def rhs(t, s):
        r = s[:, :3]
        acc = -gm * r / (r * r).sum(1, keepdim=True) ** 1.5
        if table is not None:
            q = _earth_rotation(t)
            out = []
            for i in range(0, n, 20000):
                k = slice(i, i + 20000)
                out.append((q[k].transpose(1, 2) @ _field(table, (q[k] @ r[k, :, None])[..., 0])[..., None])[..., 0])
            acc = acc + torch.cat(out)
        return torch.cat([s[:, 3:], acc], 1)

    records, epochs = [], []
    for j in range(case["steps"]):
        if not bool((dt > 0).any()):
            break
        k = []
        for s in range(13):
            ys = y
            for i, a in enumerate(_A[s]):
                if a:
                    ys = ys + (dt * a)[:, None] * k[i]
            k.append(rhs(cur + dt * _C[s], ys) if s != 10 else None)
        for s in range(13):
            if _B[s]:
                y = y + (dt * _B[s])[:, None] * k[s]
        cur = cur + dt
        rem = end - cur
        dt = torch.where((rem <= 0) | (dt <= 0), torch.zeros_like(dt), torch.minimum(step, rem))
        if case["kind"] == "trajectory" and (j + 1) % case["every"] == 0:
            records.append(y)
            epochs.append(float(cur[0]) / 86400.0 + 0.5)
    if case["kind"] == "trajectory":
        return np.array(epochs), torch.stack(records).cpu().numpy()
    if case["kind"] == "propagate":
        return (cur / 86400.0 + 0.5).cpu().numpy(), y.cpu().numpy()
    if case["kind"] == "resident":
        return float(cur[0]) / 86400.0 + 0.5, y.T.contiguous().reshape(-1)
    return int((dt > 0).sum()), y.T.contiguous().reshape(-1), torch.cat([cur, end, dt, times0])
