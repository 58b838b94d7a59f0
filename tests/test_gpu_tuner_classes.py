"""The drag model on a second warp is right up to one wave of warp pairs, a
limit inside the autotuner's size classes (powers of two): batches on both
sides of it are timed apart, in either order, and each keeps its choice."""
import json

import numpy as np
import pytest

from parahpop_b200 import api, synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(4200, 8000), (8000, 4200), (1100, 1250)])
def test_sizes_on_both_sides_of_a_wave_are_timed_apart(tmp_path, sizes):
    d = S.write_environment(tmp_path, S.EnvSpec(degree=20))
    (d / "config.json").write_text(json.dumps(S.make_config(d, 120.0, 60.0, degree=20)))
    p = api.Propagator(d / "config.json")
    pop = S.population_leo(max(sizes), seed=3, screen_duration=120.0)

    def launches(n):
        k = pop.subset(np.arange(n))
        p.propagate(k.epochs, k.states, k.mass, k.drag_area, k.srp_area, k.cd, k.cr)
        return p.stats()["launches"]

    probed = [launches(n) for n in sizes]
    kept = [launches(n) for n in sizes]
    assert all(a >= b + 3 for a, b in zip(probed, kept)), (probed, kept)  # three launches a probed shape
    assert kept[0] == kept[1]
    p.close()
