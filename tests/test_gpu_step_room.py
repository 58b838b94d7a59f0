"""Autotuned full-force batches at degrees whose staged tile leaves least of
the shared memory beside a one-lane pair kernel's own (FP64 79 to 82, split
precision 101 to 106), up to the one wave of that shape: every probe launches,
and the result is that of a pinned lane count (FP64 sums in another order: a
few 1e-12 km in four steps, bar 1e-9; in split precision the FP32 rows, whose
acceleration of 1e-6 km/s^2 is good to 1e-5, move an object by less than
1e-11 * 240^2 / 2 = 3e-7 km)."""
import json

import numpy as np
import pytest

from parahpop_b200 import api, synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree,split", [(79, False), (80, False), (81, False), (82, False), (101, True), (103, True),
                                          (104, True), (106, True)])
def test_batches_of_up_to_one_wave_launch(tmp_path, degree, split):
    d = S.write_environment(tmp_path, S.EnvSpec(degree=degree))
    (d / "config.json").write_text(json.dumps(S.make_config(d, 240.0, 60.0, degree=degree)))
    tuned, pinned = api.Propagator(d / "config.json", split=split), api.Propagator(d / "config.json", lanes=8, split=split)
    for n in (33, 9500, 15000):
        pop = S.population_leo(n, seed=n, screen_duration=240.0)
        args = (pop.epochs, pop.states, pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr)
        a, b = tuned.propagate(*args)[1], pinned.propagate(*args)[1]
        assert np.isfinite(a).all()
        assert np.abs(a[:, :3] - b[:, :3]).max() <= (3e-7 if split else 1e-9)
    tuned.close()
    pinned.close()
