"""Small batches run the drag model on a second warp where the autotuner finds
it faster (and the server for slices of one wave): the same results bit for
bit as one warp alone, whichever shape it chose, at one object, at part-filled
warps and at the largest single wave, on both time grids and precisions."""
import json

import numpy as np
import pytest

from parahpop_b200 import api, synthetic as S

pytestmark = pytest.mark.gpu


def config(tmp_path, degree=70):
    d = S.write_environment(tmp_path, S.EnvSpec(degree=degree))
    (d / "config.json").write_text(json.dumps(S.make_config(d, 240.0, 60.0, degree=degree)))
    return d / "config.json"


@pytest.mark.parametrize("degree", [20, 100])
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("uniform", [False, True])
def test_tuned_shape_matches_the_same_shape_pinned(tmp_path, degree, split, uniform):
    cfg = config(tmp_path, degree)
    for n in (1, 7, 33, 600, 4737):
        pop = S.population_leo(n, seed=n)
        epochs = pop.epochs if uniform else pop.epochs + np.linspace(0.0, 0.3, n) + 0.01 * (n == 1)
        step = 60.0 if uniform else np.where(np.arange(n) % 2, 60.0, 45.0)
        args = (epochs, pop.states, pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr, 240.0, step)
        p = api.Propagator(cfg, split=split)
        _, tuned = p.propagate(*args)
        s = p.stats()
        for key, value in (("lanes", s["lanes"]), ("pair_sh", s["pair_sh"]), ("deep_registers", s["deep_registers"])):
            p.set_option(key, value)
        _, pinned = p.propagate(*args)
        assert p.stats()["lanes"] == s["lanes"] and np.isfinite(tuned).all()
        np.testing.assert_array_equal(tuned, pinned)
        p.close()


@pytest.mark.parametrize("split", [False, True])
def test_served_alone_and_beside_a_large_request(tmp_path, split):
    """40 objects beside 12,000: their slices are of more than one wave (one
    warp each) until the large request ends, of one wave after it, and of one
    wave throughout when served alone."""
    prop = api.Propagator(config(tmp_path), split=split)
    small, large = S.population_leo(40, seed=5), S.population_leo(12000, seed=6)

    def serve(both):
        srv = api.Server(prop, 20000, slice_ms=5.0)
        of = lambda pop, duration: srv.submit(pop.epochs, pop.states, pop.mass, pop.drag_area, pop.srp_area, pop.cd,  # noqa: E731
                                              pop.cr, duration, 60.0)
        if both:
            of(large, 300.0)
        rid = of(small, 1800.0)
        srv.run_until_idle()
        out = srv.take(rid)[:2]
        srv.close()
        return out

    alone, mixed = serve(False), serve(True)
    np.testing.assert_array_equal(alone[0], mixed[0])
    np.testing.assert_array_equal(alone[1], mixed[1])
    prop.close()
