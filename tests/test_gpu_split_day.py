"""Split precision against FP64 over whole days: an FP32 rounding that repeats
from row to row or from evaluation to evaluation does not average out along an
orbit, so the errors of short runs do not show it.

Bars, in mm (p99, max): what the same runs gave with the spherical-component
sums that the solid harmonics replaced; and for objects of up to a day against
the reference's recorded outputs, likewise."""
import json

import numpy as np
import pytest

from parahpop_b200 import api, synthetic as S

pytestmark = pytest.mark.gpu

DAY = 86400.0


def day_errors(config, pop, lanes, deep):
    out = []
    for split in (False, True):
        p = api.Propagator(config, lanes=lanes, split=split)
        p.set_option("pair_sh", 1)
        p.set_option("deep_registers", deep)
        out.append(p.propagate(pop.epochs, pop.states, pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr,
                               pop.duration, pop.step)[1][:, :3])
        p.close()
    return np.linalg.norm(out[1] - out[0], axis=1) * 1e6


@pytest.mark.parametrize("population,degree,lanes,deep,p99,worst",
                         [("leo", 70, 4, 1, 1.94, 6.41), ("mixed", 70, 1, 0, 0.75, 6.33), ("leo", 120, 2, 1, 1.65, 8.30)])
def test_day_errors_stay_at_their_former_values(tmp_path, population, degree, lanes, deep, p99, worst):
    d = S.write_environment(tmp_path, S.EnvSpec(degree=degree))
    (d / "config.json").write_text(json.dumps(S.make_config(d, DAY, 60.0, max_steps=10 ** 8, degree=degree)))
    if population == "mixed":
        pop = S.population_mixed(100000, seed=5)
        pop.duration = np.minimum(pop.duration, DAY)
    else:
        pop = S.population_leo(10000 if degree == 70 else 100000, 1, screen_duration=DAY)
        pop.duration, pop.step = np.full(len(pop), DAY), np.full(len(pop), 60.0)
    err = day_errors(d / "config.json", pop, lanes, deep)
    assert np.percentile(err, 99) <= p99 and err.max() <= worst, (np.percentile(err, 99), err.max())


@pytest.mark.parametrize("name", ["c1_full_24h", "c3_leo_19h"])
def test_day_against_the_reference(golden, name):
    case = golden(name)
    p = api.Propagator(case.config_path, lanes=4, split=True)
    _, st = p.propagate_targets(case.targets)
    err = np.linalg.norm(st[:, :3] - case.ref_states[:, :3], axis=1) * 1e6
    assert err.max() <= 2.24, err.max()
    p.close()
