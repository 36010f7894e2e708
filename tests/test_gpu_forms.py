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


def _scattered(cells, cloudy, precision, sip):
    """`cells` of grid384x384x160, a share of them in cloud with ice."""
    inp = make_inputs("grid384x384x160", "cuda", X=16, Y=cells // 512, Z=32, precision=precision, gases=sip,
                      overrides=dict(cloudy=cloudy, pattern="random"))
    if sip:
        for sw in (inp.cfg.lssecice, inp.cfg.lssiprimespln, inp.cfg.lssipdropfrac, inp.cfg.lssipicecollbreak):
            sw.sw, sw.mode = 1, 1
        for name in ("sipdrfr", "siprmspl", "sipiibr"):
            inp.fields[name] = inp.fields["nice"] * 0.02
    return inp


@pytest.mark.parametrize("cells,cloudy,precision,sip,lane", [
    (24576, 0.0, 0, False, True), (24576, 0.02, 0, False, False), (24576, 0.1, 0, False, False),
    (24576, 1.0, 0, False, True), (61440, 0.02, 0, False, True), (24064, 1.0, 0, False, False),
    (40960, 0.02, 1, False, False), (40960, 1.0, 1, False, True), (81920, 0.02, 1, False, True),
    (8192, 0.0, 0, True, True), (8192, 0.02, 0, True, False), (8192, 1.0, 0, True, True), (24576, 0.02, 0, True, True),
    (8192, 0.1, 1, True, False), (8192, 1.0, 1, True, True)])
def test_few_cloudy_cells_take_the_warp_form(cells, cloudy, precision, sip, lane):
    """The form follows the kinds of cells; a large call that takes the warp form gives every
    cell what smaller calls give it, bit for bit."""
    inp = _scattered(cells, cloudy, precision, sip)
    outs = {k: v for k, v in make_outputs(inp).items()}
    step = api.SalsaStep(inp.cfg)
    f = {k: v.clone() for k, v in inp.fields.items()}
    rc, st = step.run(inp, f, outs, time=1.0)
    assert rc == 0 and st.n_cells == cells
    assert step.last_lane_cells() == (cells if lane else 0)
    if not lane:
        n = inp.nyp // 3
        sub = type(inp)(**{**inp.__dict__, "nyp": n})
        sub.fields = {k: v[..., :n, :, :].contiguous() for k, v in inp.fields.items()}
        part = make_outputs(sub)
        rc, st = step.run(sub, {k: v.clone() for k, v in sub.fields.items()}, part, time=1.0)
        assert rc == 0 and step.last_lane_cells() == 0
        for k, v in part.items():
            assert torch.equal(v[..., 2:-2, 2:-2, 1:-1], outs[k][..., 2:n - 2, 2:-2, 1:-1]), k
    step.close()
