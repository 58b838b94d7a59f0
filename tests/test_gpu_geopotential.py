"""The step kernel's geopotential against a plain NumPy evaluation of the same
field in spherical components (Legendre functions and their latitude
derivatives, term by term) inside a plain NumPy RKF78 step.

Degrees around the row pairs and the column blocks of every lane split, an
order below the degree, an unnormalised field and objects on and next to the
polar axis.  Tolerances: positions are near 7,000 km and move for three steps
of 20 s, so double rounding is a few 1e-12 km (bar 1e-9 km).  In split
precision the degrees above 8 are FP32: their acceleration is below 1e-6
km/s^2 here, its relative error below 1e-5 after up to 70 rows, which moves
an object by at most 1e-11 * 60^2 / 2 = 2e-8 km (bar 1e-7 km)."""
import json
import math

import numpy as np
import pytest

from parahpop_b200 import api, synthetic as S

pytestmark = pytest.mark.gpu

A = [[], [2 / 27], [1 / 36, 1 / 12], [1 / 24, 0, 1 / 8], [5 / 12, 0, -25 / 16, 25 / 16], [1 / 20, 0, 0, 1 / 4, 1 / 5],
     [-25 / 108, 0, 0, 125 / 108, -65 / 27, 125 / 54], [31 / 300, 0, 0, 0, 61 / 225, -2 / 9, 13 / 900],
     [2, 0, 0, -53 / 6, 704 / 45, -107 / 9, 67 / 90, 3],
     [-91 / 108, 0, 0, 23 / 108, -976 / 135, 311 / 54, -19 / 60, 17 / 6, -1 / 12],
     [2383 / 4100, 0, 0, -341 / 164, 4496 / 1025, -301 / 82, 2133 / 4100, 45 / 82, 45 / 164, 18 / 41],
     [3 / 205, 0, 0, 0, 0, -6 / 41, -3 / 205, -3 / 41, 3 / 41, 6 / 41, 0],
     [-1777 / 4100, 0, 0, -341 / 164, 4496 / 1025, -289 / 82, 2193 / 4100, 51 / 82, 33 / 164, 12 / 41, 0, 1]]
NODES = [0, 2 / 27, 1 / 9, 1 / 6, 5 / 12, 1 / 2, 5 / 6, 1 / 6, 2 / 3, 1 / 3, 1, 0, 1]
B = [0, 0, 0, 0, 0, 34 / 105, 9 / 35, 9 / 35, 9 / 280, 9 / 280, 0, 41 / 840, 41 / 840]


def norm(n, m):
    return math.sqrt((1 if m == 0 else 2) * (2 * n + 1) * math.exp(math.lgamma(n - m + 1) - math.lgamma(n + m + 1)))


def earth_frame(t):
    """The synthetic IAU body model of the Earth (iau_earth_units)."""
    T, d = t / 3155760000.0, t / 86400.0
    j = np.radians([125.045 - 1935.5364525 * T, 250.089 - 3871.0729 * T])
    ra = math.radians(-0.641 * T - 3.6e-3 * math.sin(j[0]) + 5.0e-4 * math.sin(j[1]))
    dec = math.radians(90.0 - 0.557 * T + 1.3e-3 * math.cos(j[0]) - 2.0e-4 * math.cos(j[1]))
    pm = math.radians((190.147 + 360.9856235 * d + 2.1e-3 * math.sin(j[0]) - 3.0e-4 * math.sin(j[1])) % 360.0)

    def rz(a):
        return np.array([[math.cos(a), math.sin(a), 0], [-math.sin(a), math.cos(a), 0], [0, 0, 1]])

    x = math.pi / 2 - dec
    rx = np.array([[1, 0, 0], [0, math.cos(x), math.sin(x)], [0, -math.sin(x), math.cos(x)]])
    return rz(pm) @ rx @ rz(math.pi / 2 + ra)


def field_accel(C, Sn, N, M, gm, R, p):
    """Body-frame acceleration at p (n, 3) off the polar axis, normalised C, S."""
    x, y, z = p.T
    r, rho = np.sqrt((p * p).sum(1)), np.hypot(x, y)
    s, c, lam = z / r, rho / r, np.arctan2(y, x)
    P = np.zeros((N + 3, N + 3, len(p)))
    P[0, 0] = 1.0
    for n in range(1, N + 2):
        P[n, n] = math.sqrt(3.0 if n == 1 else (2 * n + 1) / (2 * n)) * c * P[n - 1, n - 1]
        for m in range(n):
            a = math.sqrt((2 * n - 1) * (2 * n + 1) / ((n - m) * (n + m)))
            b = math.sqrt((2 * n + 1) * (n + m - 1) * (n - m - 1) / ((2 * n - 3) * (n + m) * (n - m))) if n > m + 1 else 0
            P[n, m] = a * s * P[n - 1, m] - (b * P[n - 2, m] if b else 0)
    ur, up, ul = np.zeros((3, len(p)))
    for n in range(1, N + 1):
        w = gm / (r * r) * (R / r) ** n
        for m in range(min(n, M) + 1):
            k = math.sqrt((0.5 if m == 0 else 1.0) * (n - m) * (n + m + 1))
            dP = k * P[n, m + 1] - m * s / c * P[n, m]
            q = C[n, m] * np.cos(m * lam) + Sn[n, m] * np.sin(m * lam)
            ur -= w * (n + 1) * P[n, m] * q
            up += w * dP * q
            ul += w * m / c * P[n, m] * (Sn[n, m] * np.cos(m * lam) - C[n, m] * np.sin(m * lam))
    cl, sl = np.cos(lam), np.sin(lam)
    return np.stack([c * cl * ur - s * cl * up - sl * ul, c * sl * ur - s * sl * up + cl * ul, s * ur + c * up], 1)


def propagate(C, Sn, N, M, gm, R, gm0, epoch, states, steps, step):
    y, t = states.copy(), (epoch - 0.5) * 86400.0

    def rhs(t, s):
        q = earth_frame(t)
        r = s[:, :3]
        acc = -gm0 * r / ((r * r).sum(1) ** 1.5)[:, None] + field_accel(C, Sn, N, M, gm, R, r @ q.T) @ q
        return np.concatenate([s[:, 3:], acc], 1)

    for _ in range(steps):
        k = []
        for j in range(13):
            k.append(rhs(t + NODES[j] * step, y + step * sum((a * k[i] for i, a in enumerate(A[j])), 0 * y)))
        y = y + step * sum(b * k[i] for i, b in enumerate(B))
        t += step
    return y


def case(tmp_path, degree, order, normalised):
    held = max(degree, 2)  # the generator's fields hold at least degree 2
    d = S.write_environment(tmp_path, S.EnvSpec(degree=held, earth_frame="iau"))
    C, Sn = S.kaula_field(held, 7)
    if degree == 1:
        C[1, 0], C[1, 1], Sn[1, 1] = 2e-7, -3e-7, 5e-7
    C[:, order + 1:] = 0.0
    Sn[:, order + 1:] = 0.0
    with open(d / "gravity.tab", "w") as f:
        f.write(f"6378.1363, 398600.4415, 0.0, {degree}, {degree}, {int(normalised)}, 0, 0\n")
        for n in range(1, degree + 1):
            for m in range(n + 1):
                w = 1.0 if normalised else norm(n, m)
                f.write(f"{n}, {m}, {w * C[n, m]:.17e}, {w * Sn[n, m]:.17e}, 0.0, 0.0\n")
    cfg = S.make_config(d, 60.0, 20.0, force="field", degree=degree)
    cfg["model"]["environment"]["bodies"]["Earth"]["gravity"]["shape"]["order"] = order
    (d / "config.json").write_text(json.dumps(cfg))
    pop = S.population_leo(35, seed=5)
    # next to the polar axis, where the longitude turns fast
    q = earth_frame((float(pop.epochs[0]) - 0.5) * 86400.0)
    for i, off in enumerate((1e-3, 1.0, 30.0)):
        pop.states[i, :3] = q.T @ np.array([off, -0.5 * off, (-1) ** i * 7000.0])
        pop.states[i, 3:] = q.T @ np.array([7.5, 0.3, 0.0])
    return d / "config.json", C, Sn, pop


@pytest.mark.parametrize("degree,order,normalised",
                         [(1, 1, True), (2, 2, True), (3, 3, True), (7, 5, True), (9, 9, False), (30, 30, True),
                          (31, 31, True), (32, 4, True), (33, 33, True), (62, 62, True)])
def test_field_matches_numpy(tmp_path, degree, order, normalised):
    cfg, C, Sn, pop = case(tmp_path, degree, order, normalised)
    ref = propagate(C, Sn, degree, order, 398600.4415, 6378.1363, 398600.4415, float(pop.epochs[0]), pop.states, 3, 20.0)
    for split in (False, True):
        for lanes, pair in ((1, 0), (1, 1), (2, 0), (2, 1), (4, 0), (4, 1), (8, 0), (16, 0)):
            p = api.Propagator(cfg, lanes=lanes, split=split)
            p.set_option("pair_sh", pair)
            if split:
                p.set_option("split_fp64_degree", 8)
            _, st = p.propagate(pop.epochs, pop.states, pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr, 60.0,
                                20.0)
            off = np.abs(st[:, :3] - ref[:, :3]).max()
            assert off <= (1e-7 if split else 1e-9), (split, lanes, pair, off)
            p.close()


def test_field_on_the_polar_axis(tmp_path):
    """On the axis itself (cos phi = 0 to rounding) the result continues the
    one a micrometre beside it: the field's gradient is below 1e-5 per km, so
    1e-9 km apart the accelerations agree to 1e-14 km/s^2."""
    cfg, _, _, pop = case(tmp_path, 33, 33, True)
    epoch = float(pop.epochs[0])
    q = earth_frame((epoch - 0.5) * 86400.0)
    st = np.zeros((2, 6))
    st[0, :3] = q.T @ np.array([0.0, 0.0, 7000.0])
    st[1, :3] = q.T @ np.array([1e-9, 0.0, 7000.0])
    one = np.ones(2)
    p = api.Propagator(cfg, lanes=1)
    _, out = p.propagate(np.full(2, epoch), st, 100 * one, one, one, one, one, 2.0, 2.0)
    assert np.isfinite(out).all()
    assert np.abs(out[0] - out[1]).max() <= 2e-9
    p.close()


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("degree", [92, 120])
def test_streamed_tile_matches_global_reads(tmp_path, degree, split):
    """A tile that does not fit shared memory is streamed through rings (at
    degree 92 in split precision it fits and is staged); with "tile_smem" 0
    the same rows are read from global memory.  The same sums, so the same
    bits, on a shared time grid and on per-object epochs."""
    d = S.write_environment(tmp_path, S.EnvSpec(degree=degree))
    (d / "config.json").write_text(json.dumps(S.make_config(d, 240.0, 60.0, degree=degree)))
    pop = S.population_leo(99, seed=11)
    args = (pop.states, pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr)
    for lanes, pair, deep in ((1, 0, 0), (1, 1, 0), (2, 0, 1), (2, 1, 1), (4, 0, 1), (4, 1, 1)):
        p = api.Propagator(d / "config.json", lanes=lanes, split=split)
        p.set_option("pair_sh", pair)
        p.set_option("deep_registers", deep)
        for epochs in (pop.epochs, pop.epochs + np.linspace(0.0, 0.01, len(pop))):
            got = []
            for staged in (1, 0):
                p.set_option("tile_smem", staged)
                got.append(p.propagate(epochs, *args)[1])
                assert p.stats()["tile_in_smem"] == (1 if staged and split and degree == 92 else 0)
            assert np.isfinite(got[0]).all()
            np.testing.assert_array_equal(got[0], got[1])
        p.close()
