"""The Earth's tides beside fields below degree 6, of an order below the degree
and unnormalised: deltas beyond the field's degree or order do not act, those
of an unnormalised field join its coefficients as they are.

The states in golden/tides_small_fields.json were recorded with the step
kernel's former field sums, which added each delta to its coefficient.  The
tides move the objects by some 1e-5 km here; both forms round at a few 1e-12
km (bar 1e-9)."""
import json
import math
from pathlib import Path

import numpy as np
import pytest

from parahpop_b200 import api, synthetic as S

pytestmark = pytest.mark.gpu

GOLD = Path(__file__).resolve().parent / "golden" / "tides_small_fields.json"
CASES = [(n, m, norm) for n, m in ((2, 2), (3, 1), (4, 0), (4, 4), (5, 3), (6, 6), (9, 4)) for norm in (True, False)]


def norm_factor(n, m):
    return math.sqrt((1 if m == 0 else 2) * (2 * n + 1) * math.exp(math.lgamma(n - m + 1) - math.lgamma(n + m + 1)))


def small_field(directory, degree, order, normalised):
    d = S.write_environment(directory, S.EnvSpec(degree=degree))
    C, Sn = S.kaula_field(degree, 7)
    with open(d / "gravity.tab", "w") as f:
        f.write(f"6378.1363, 398600.4415, 0.0, {degree}, {degree}, {int(normalised)}, 0, 0\n")
        for n in range(1, degree + 1):
            for m in range(n + 1):
                w = 1.0 if normalised else norm_factor(n, m)
                f.write(f"{n}, {m}, {w * C[n, m]:.17e}, {w * Sn[n, m]:.17e}, 0.0, 0.0\n")
    cfg = S.make_config(d, 600.0, 60.0, degree=degree, drag=False, relativity=False)
    cfg["model"]["environment"]["bodies"]["Earth"]["gravity"]["shape"]["order"] = order
    (d / "config.json").write_text(json.dumps(cfg))
    return d / "config.json"


def states(config, lanes, split=False):
    pop = S.population_leo(7, seed=8, screen_duration=600.0)
    p = api.Propagator(config, lanes=lanes, split=split)
    out = p.propagate(pop.epochs, pop.states, pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr)[1]
    p.close()
    return out


@pytest.mark.parametrize("degree,order,normalised", CASES)
def test_tides_beside_small_fields(tmp_path, degree, order, normalised):
    ref = np.array(json.loads(GOLD.read_text())["%d_%d_%d" % (degree, order, normalised)])
    config = small_field(tmp_path, degree, order, normalised)
    for lanes in (1, 4, 16):
        for split in (False, True):
            assert np.abs(states(config, lanes, split)[:, :3] - ref[:, :3]).max() <= 1e-9, (lanes, split)
