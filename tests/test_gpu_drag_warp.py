"""The kernels with the drag model on a second warp against those of one warp:
the same results bit for bit, at every lane count that has them, the tile
staged, streamed and read from global memory, on both time grids, with and
without an order of objects, for one wave and more, and in the server whatever
shares a slice.  The terms outside the field are plain expressions that the
compiler contracts in each kernel by itself, so this holds for the kernels as
built, not by construction.  Both sides' statistics name the kernel that ran."""
import json

import numpy as np
import pytest

from parahpop_b200 import api, synthetic as S

pytestmark = pytest.mark.gpu


def config(tmp_path, degree):
    d = S.write_environment(tmp_path, S.EnvSpec(degree=degree))
    (d / "config.json").write_text(json.dumps(S.make_config(d, 240.0, 60.0, degree=degree)))
    return d / "config.json"


def both(prop, run, streamed=None):
    out = []
    for duo in (0, 1):
        prop.set_option("drag_warp", duo)
        out.append(run(prop))
        form = prop.stats()["kernel_form"]
        assert form & 1 == duo, form
        if streamed is not None:
            assert (form >> 1) & 1 == int(streamed), form
    assert np.isfinite(out[0]).all()
    np.testing.assert_array_equal(out[0], out[1])


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("degree", [20, 120])
@pytest.mark.parametrize("lanes", [1, 2, 4, 8, 16])
def test_every_lane_count(tmp_path, lanes, degree, split):
    cfg = config(tmp_path, degree)
    leo, uneven = S.population_leo(131, seed=lanes), S.population_mixed(131, seed=lanes)
    uneven.duration = np.minimum(uneven.duration, 1800.0)
    p = api.Propagator(cfg, lanes=lanes, split=split)
    p.set_option("deep_registers", 1 if lanes in (2, 4) else 0)
    for pop in (leo, uneven):
        both(p, lambda p: p.propagate(pop.epochs, pop.states, pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr,
                                      pop.duration if pop is uneven else None, pop.step if pop is uneven else None)[1],
             streamed=degree == 120 and lanes <= 4)
    p.close()


@pytest.mark.parametrize("name", ["full_1h", "lunar_shadow_30m", "iau_earth_1h", "moon_j2_2h", "zonal_2h", "tide_free_2h",
                                  "c3_leo_19h", "c3_geo_3d"])
@pytest.mark.parametrize("split", [False, True])
def test_every_force_model(golden, name, split):
    case = golden(name)
    for lanes in (2, 16):
        p = api.Propagator(case.config_path, lanes=lanes, split=split)
        p.set_option("deep_registers", 1 if lanes == 2 else 0)
        both(p, lambda p: p.propagate_targets(case.targets)[1])
        p.close()


def test_more_than_one_wave(tmp_path):
    """2.5 waves of pairs at two lanes: work from the queue, partners kept."""
    p = api.Propagator(config(tmp_path, 20), lanes=2)
    p.set_option("deep_registers", 1)
    pop = S.population_leo(24001, seed=9, screen_duration=240.0)
    both(p, lambda p: p.propagate(pop.epochs, pop.states, pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr)[1])
    p.close()


@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("degree", [20, 70, 120])
def test_served_alone_and_in_a_mix(tmp_path, degree, split):
    """An uneven request served alone, with the drag model on second warps
    throughout and with none, and beside a LEO request of more than one wave
    and another uneven one."""
    prop = api.Propagator(config(tmp_path, degree), split=split)
    asked = S.population_mixed(60, seed=41)
    asked.duration = np.minimum(asked.duration, 7200.0)
    other = S.population_mixed(500, seed=42)
    other.duration = np.minimum(other.duration, 3600.0)
    large = S.population_leo(12000, seed=6, screen_duration=240.0)
    large.duration = np.full(len(large), 240.0)

    def serve(duo, beside):
        prop.set_option("drag_warp", duo)
        srv = api.Server(prop, 20000, slice_ms=5.0)
        of = lambda pop: srv.submit(pop.epochs, pop.states, pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr,  # noqa: E731
                                    pop.duration, pop.step)
        for pop in beside:
            of(pop)
        rid = of(asked)
        srv.run_until_idle()
        out = srv.take(rid)[:2]
        srv.close()
        return out

    alone = serve(-1, [])
    assert np.isfinite(alone[1]).all()
    for duo, beside in ((0, []), (1, []), (-1, [large]), (-1, [other, large]), (0, [other])):
        got = serve(duo, beside)
        np.testing.assert_array_equal(alone[0], got[0])
        np.testing.assert_array_equal(alone[1], got[1])
    prop.close()
