"""Pinned lane counts and the allocation-free entry point at a degree whose
tile does not fit shared memory: the kernel that streams it runs unless the
wide bound is asked for, with the pinned deep kernel's bits; below, the wide
kernel as before."""
import ctypes as C
import json

import numpy as np
import pytest

from parahpop_b200 import api, synthetic as S

pytestmark = pytest.mark.gpu


def config(tmp_path, degree):
    d = S.write_environment(tmp_path, S.EnvSpec(degree=degree))
    (d / "config.json").write_text(json.dumps(S.make_config(d, 240.0, 60.0, max_steps=1000, degree=degree)))
    return d / "config.json"


@pytest.mark.parametrize("degree", [70, 120])
@pytest.mark.parametrize("split", [False, True])
def test_pinned_lanes(tmp_path, degree, split):
    cfg = config(tmp_path, degree)
    pop = S.population_leo(101, seed=2, screen_duration=240.0)
    for lanes in (1, 2, 4):
        out = {}
        for deep in (-1, 0, 1):
            p = api.Propagator(cfg, lanes=lanes, split=split)
            p.set_option("deep_registers", deep)
            out[deep] = p.propagate(pop.epochs, pop.states, pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr)[1]
            s = p.stats()
            p.close()
            if deep < 0:
                assert s["deep_registers"] == (lanes > 1 and degree == 120)
                assert s["kernel_form"] == (2 if degree == 120 else 0)
            if deep == 0 and lanes > 1:
                assert s["kernel_form"] == (4 if degree == 120 else 0) and s["deep_registers"] == 0
        assert np.isfinite(out[-1]).all()
        np.testing.assert_array_equal(out[-1], out[1 if degree == 120 else 0])


@pytest.mark.parametrize("split,degree", [(False, 88), (False, 120), (True, 120)])
@pytest.mark.parametrize("lanes,duo", [(2, 0), (4, 0), (8, 0), (16, 0), (8, 1), (16, 1)])
def test_first_blocks_staged(tmp_path, lanes, duo, split, degree):
    """The staged blocks are those of global memory: the same bits, on both
    time grids, with part-filled warps and several items a warp."""
    cfg = config(tmp_path, degree)
    for n in (1, 37, 20000 // lanes):
        pop = S.population_leo(n, seed=n, screen_duration=240.0)
        for epochs in (pop.epochs, pop.epochs + np.linspace(0.001, 0.01, n)):
            got = []
            for smem in (1, 0):
                p = api.Propagator(cfg, lanes=lanes, split=split)
                for key, value in (("tile_smem", smem), ("deep_registers", 0), ("drag_warp", duo)):
                    p.set_option(key, value)
                got.append(p.propagate(epochs, pop.states, pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr)[1])
                s = p.stats()
                assert s["kernel_form"] == duo + (4 if smem else 0) and s["tile_in_smem"] == 0
                p.close()
            assert np.isfinite(got[0]).all()
            np.testing.assert_array_equal(got[0], got[1])


@pytest.mark.parametrize("lanes", [1, 2, 4, 8, 16])
def test_noalloc(tmp_path, lanes):
    """To the entry points' parity tolerance, 1 mm and 1e-6 m/s; a refused
    call's limits are as before."""
    import torch
    p = api.Propagator(config(tmp_path, 120), lanes=lanes)
    pop = S.population_leo(333, seed=4, screen_duration=240.0)
    soa = torch.from_numpy(np.ascontiguousarray(pop.states.T).reshape(-1))
    bc, ams = (torch.from_numpy(a).cuda() for a in p.factors(pop.mass, pop.drag_area, pop.srp_area, pop.cd, pop.cr))
    ref, got = soa.clone().cuda(), soa.clone().cuda()
    p.propagate_device(ref.data_ptr(), len(pop), float(pop.epochs[0]), pop.mass, pop.drag_area, pop.srp_area, pop.cd,
                       pop.cr, 240.0, 60.0)
    f = api.library().phop_propagate_device_noalloc
    f.argtypes = [C.c_void_p, C.c_int64] + [C.c_void_p] * 3 + [C.c_double] * 3 + [C.POINTER(C.c_double)]
    end = C.c_double()
    torch.cuda.synchronize()
    assert f(p._h, len(pop), got.data_ptr(), bc.data_ptr(), ams.data_ptr(), float(pop.epochs[0]), 240.0, 60.0,
             C.byref(end)) == 0
    d = (got - ref).cpu().numpy().reshape(6, -1)
    assert np.abs(d[:3]).max() * 1e3 <= 1e-3 and np.abs(d[3:]).max() * 1e3 <= 1e-6
    p.close()
