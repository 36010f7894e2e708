"""Which form a step takes (SalsaStep.last_lane_cells): one cell per lane or per warp."""
import ctypes as C

import pytest
import torch

from uclales_salsa_gb300 import api, capi
from uclales_salsa_gb300.inputs import make_inputs, make_outputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,lane", [(dict(X=1, Y=1, Z=1), False), (dict(X=8, Y=8, Z=8), False),
                                       (dict(X=64, Y=48, Z=32), True)])
def test_last_lane_cells(size, lane):
    inp = make_inputs("grid384x384x160", "cuda", **size)
    step = api.SalsaStep(inp.cfg)
    assert step.last_lane_cells() == 0
    f = {k: v.clone() for k, v in inp.fields.items()}
    rc, st = step.run(inp, f, make_outputs(inp), time=1.0)
    assert rc == 0 and st.n_cells == inp.ncells
    assert step.last_lane_cells() == (inp.ncells if lane else 0)
    if lane:   # the entry point without allocations always takes the warp form
        L = api.library()
        L.salsa_gb300_run_noalloc.argtypes = L.salsa_gb300_run_async.argtypes
        f = {k: v.clone() for k, v in inp.fields.items()}
        cf = capi.make_fields(f, make_outputs(inp))
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        assert L.salsa_gb300_run_noalloc(step.h, inp.nzp, inp.nxp, inp.nyp, inp.ns, inp.dt, 1.0, 1, inp.level, 0, 0,
                                         C.byref(cf), C.c_void_p(s.cuda_stream), 1, C.byref(st)) == 0
        assert st.n_cells == inp.ncells and step.last_lane_cells() == 0
    step.close()
