"""The density cut-off over a figure that is not oblate (a negative flattening
is accepted): its poles lie above the sphere of its equatorial radius, so an
object there can be above the cut-off from that sphere and below it from the
figure.  With the cut-off at 300 km, objects 305 to 318 km above the sphere
and 286 to 299 km above the pole meet the same air as with the cut-off at
1,000 km (one step of 10 s near the pole: the same density in both runs, so
the same states; without drag they differ by some 1e-7 km, bar 1e-11)."""
import json

import numpy as np
import pytest

from parahpop_b200 import api, synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes", [1, 8])
def test_cutoff_over_a_prolate_figure(tmp_path, lanes):
    d = S.write_environment(tmp_path, S.EnvSpec(degree=4, earth_frame="iau"))
    cfg = S.make_config(d, 10.0, 10.0, degree=4)
    earth = cfg["model"]["environment"]["bodies"]["Earth"]
    earth["flattening"] = -0.003  # poles 19.1 km above the equatorial radius
    pop = S.population_leo(6, seed=5)
    pole = np.array([0.0, 0.0, 1.0])  # the frame's pole is the z axis to 0.01 degrees
    for i, h in enumerate((305.0, 308.0, 311.0, 314.0, 316.0, 318.0)):
        pop.states[i, :3] = (6378.137 + h) * pole
        pop.states[i, 3:] = np.array([7.7, 0.0, 0.0])
    pop.mass[:], pop.drag_area[:], pop.cd[:] = 10.0, 50.0, 2.2
    out = {}
    for cutoff, drag in ((300.0, True), (1000.0, True), (1000.0, False)):
        earth["atmosphere"]["nrlmsise00"]["hCutoff"] = cutoff
        config = d / f"config_{cutoff:g}_{drag}.json"
        config.write_text(json.dumps(cfg))
        p = api.Propagator(config, lanes=lanes)
        area = pop.drag_area if drag else 1e-9 * pop.drag_area
        out[cutoff, drag] = p.propagate(pop.epochs, pop.states, pop.mass, area, pop.srp_area, pop.cd, pop.cr, 10.0, 10.0)[1]
        p.close()
    assert (np.abs(out[1000.0, True] - out[1000.0, False])[:, 0] > 1e-8).all()
    assert np.abs(out[300.0, True] - out[1000.0, True])[:, :3].max() <= 1e-11
