"""Fields of many degrees and few orders in the allocation-free entry point.

Its 512-KiB rule counts one entry per term; the coefficient tile holds whole
row pairs of seven words and columns one order further, so such fields need
more room (659,456 bytes at degree 221, order 55 and four lanes) and must
still be taken.  Compared with the regular device-resident entry point, to
that entry point's parity tolerance."""
import ctypes as C
import json

import numpy as np
import pytest

from parahpop_b200 import api, synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree,order,lanes", [(221, 55, 4), (221, 20, 8)])
def test_noalloc_takes_fields_of_many_degrees(tmp_path, degree, order, lanes):
    import torch
    d = S.write_environment(tmp_path, S.EnvSpec(degree=degree))
    cfg = S.make_config(d, 600.0, 60.0, max_steps=1000, force="field", degree=degree)
    text = json.dumps(cfg).replace('"order": %d' % degree, '"order": %d' % order)
    assert '"order": %d' % order in text
    (d / "config.json").write_text(text)
    pop = S.population_leo(33, seed=5)
    n = len(pop)
    soa = np.ascontiguousarray(pop.states.T).reshape(-1)
    bc = torch.from_numpy(pop.cd * pop.drag_area * 1e-6 / pop.mass).cuda()
    ams = torch.from_numpy(pop.cr * pop.srp_area * 1e-6 / pop.mass).cuda()
    prop = api.Propagator(d / "config.json", lanes=lanes)
    ref = torch.from_numpy(soa.copy()).cuda()
    prop.propagate_device(ref.data_ptr(), n, float(pop.epochs[0]), pop.mass, pop.drag_area, pop.srp_area, pop.cd,
                          pop.cr, prop.duration, prop.step)
    got = torch.from_numpy(soa.copy()).cuda()
    f = api.library().phop_propagate_device_noalloc
    f.argtypes = [C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p, C.c_void_p, C.c_double, C.c_double, C.c_double,
                  C.POINTER(C.c_double)]
    f.restype = C.c_int
    epoch = C.c_double()
    rc = f(prop._h, n, C.c_void_p(got.data_ptr()), C.c_void_p(bc.data_ptr()), C.c_void_p(ams.data_ptr()),
           float(pop.epochs[0]), prop.duration, prop.step, C.byref(epoch))
    assert rc == 0, api.library().phop_last_error(prop._h).decode()
    diff = (got - ref).cpu().numpy().reshape(6, n)
    assert np.abs(diff[:3]).max() * 1e3 <= 1e-3  # m
    assert np.abs(diff[3:]).max() * 1e3 <= 1e-6  # m/s
    prop.close()
