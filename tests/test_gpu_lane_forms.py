"""The lane form against the warp form where they are one call each: SalsaStep.run on enough
cells, and salsa_gb300_run_noalloc, which always takes the warp form.  Secondary ice in every
scheme and mode, both precisions; the bound is that of test_gpu_lane.py (rounding, 1e-10 of the
new state, and for the ill-conditioned share of the values 1e-6 of the field's largest change),
for the tracers and the rate diagnostics 1e-6 of the field's largest value.
"""
import ctypes as C

import pytest
import torch

from uclales_salsa_gb300 import api, capi
from uclales_salsa_gb300.inputs import make_inputs, make_outputs
from parity import STATE_OF, floor_of, interior
from sip_cases import sip_state
from test_gpu_sip import SCHEMES, _parity

pytestmark = pytest.mark.gpu
# ragged sizes above the least call of the lane form, whose kinds of cells choose it
SIP_SIZE = {0: dict(X=20, Y=22, Z=21), 1: dict(X=21, Y=26, Z=23)}


def _outputs(inp, fields, noalloc, initialize=0):
    out = {k: v.cuda() for k, v in make_outputs(inp).items()}
    f = {k: v.clone().cuda() for k, v in fields.items()}
    step = api.SalsaStep(inp.cfg)
    if noalloc:
        L = api.library()
        L.salsa_gb300_run_noalloc.argtypes = L.salsa_gb300_run_async.argtypes
        cf, st, s = capi.make_fields(f, out), capi.Status(), torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        rc = L.salsa_gb300_run_noalloc(step.h, inp.nzp, inp.nxp, inp.nyp, inp.ns, inp.dt, 1.0, 1, inp.level, 0, initialize,
                                       C.byref(cf), C.c_void_p(s.cuda_stream), 1, C.byref(st))
        torch.cuda.synchronize()
    else:
        rc, st = step.run(inp, f, out, time=1.0, initialize=initialize)
    assert rc == 0 and st.n_cells == inp.ncells, (rc, st.as_dict())
    assert step.last_lane_cells() == (0 if noalloc else inp.ncells)
    step.close()
    for k in ("indef", "sipdrfr", "siprmspl", "sipiibr"):
        if k in f:
            out[k] = f[k]
    return out


def _compare(inp, a, b, sip):
    dims = (inp.nzp, inp.nxp, inp.nyp)
    for k in a:
        x, y = interior(a[k], *dims), interior(b[k], *dims)
        if k in ("sipdrfr", "siprmspl", "sipiibr"):
            assert float((x - y).abs().max()) <= 1e-6 * float(y.abs().max()), k
            continue
        if k == "diag" and sip:
            for i in (17, 18, 19):
                assert float((x[i] - y[i]).abs().max()) <= 1e-6 * float(y[i].abs().max()), i
        if k in STATE_OF:
            old = interior(inp.fields[STATE_OF[k]].cuda(), *dims)
            scale = torch.maximum((old + y * inp.dt).abs(), old.abs()).clamp(min=floor_of(k))
            rel = (x - y).abs() * inp.dt / scale
        else:
            rel = (x - y).abs() / y.abs().amax().clamp(min=1e-300)
        assert bool(torch.isfinite(rel).all()), k
        assert float((rel <= 1e-10).double().mean()) >= 0.99, (k, float((rel <= 1e-10).double().mean()))
        assert float((x - y).abs().max()) <= 1e-6 * float(y.abs().max()), k


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("scheme,mode", SCHEMES + [("all", 1)])
def test_secondary_ice_lane_form_equals_warp_form(scheme, mode, precision):
    if scheme == "all":
        inp = sip_state(mode, coag_only=False, **SIP_SIZE[precision])
        for sw in (inp.cfg.lssipdropfrac, inp.cfg.lssipicecollbreak):
            sw.sw, sw.mode = 1, 1
    else:
        inp = sip_state(mode, scheme=scheme, **SIP_SIZE[precision])
    inp.cfg.precision = precision
    a, b = _outputs(inp, inp.fields, False), _outputs(inp, inp.fields, True)
    _compare(inp, a, b, True)
    # the scheme acts: its rate is not zero everywhere
    rate = {"lssipdropfrac": 17, "lssiprimespln": 18, "lssipicecollbreak": 19}.get(scheme, 18)
    assert float(b["diag"][rate].abs().max()) > 0.0


def test_secondary_ice_lane_form_against_the_oracle():
    """All processes and the three schemes on a block that takes the lane form."""
    inp = sip_state(1, coag_only=False, **SIP_SIZE[0])
    for sw in (inp.cfg.lssipdropfrac, inp.cfg.lssipicecollbreak):
        sw.sw, sw.mode = 1, 1
    _parity(inp, 1e-10, 2.2e-16)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kind", ["plain", "dt", "initialize", "kappa"])
def test_noalloc_differs_from_a_large_run_by_rounding(kind, precision):
    """The configured call; a step length without an exact reciprocal; the initial equilibration
    of the aerosol water; kappa and supersaturation per cell."""
    if kind == "kappa":
        inp = make_inputs("batch65536", "cuda", X=1, Y=1, Z=41001, precision=precision)
    else:
        inp = make_inputs("grid384x384x160", "cuda", X=32, Y=43, Z=31, precision=precision)
    if kind == "dt":
        inp.dt = 0.7
    init = int(kind == "initialize")
    _compare(inp, _outputs(inp, inp.fields, False, init), _outputs(inp, inp.fields, True, init), False)


@pytest.mark.parametrize("precision", [0, 1])
def test_stored_kernels_of_bins_that_are_empty_now(precision):
    """Low-frequency kernels (lscoag mode 2): a fetching step after the cloud droplets fell
    below their number limit, with their water left, still collects it by the stored kernels;
    the lane form (one call) as the warp form (calls on parts of the grid)."""
    size = dict(X=32, Y=31, Z=27) if precision == 0 else dict(X=32, Y=43, Z=31)
    inp = make_inputs("grid384x384x160", "cuda", precision=precision, **size)
    inp.cfg.lscoag.mode, inp.cfg.cgintvl = 2, 10.0
    later = {k: v.clone() for k, v in inp.fields.items()}
    later["ncloud"] = torch.where(later["ncloud"] > 0, 0.9 / later["dn"].clamp(min=1e-3), later["ncloud"])

    def two_steps(grid, first, second, fetch=True):
        step = api.SalsaStep(grid.cfg)
        for fields, t, istp in ((first, 10.0, 1), (second, 13.0 if fetch else 20.0, 4)):
            out = make_outputs(grid)
            rc, st = step.run(grid, {k: v.clone() for k, v in fields.items()}, out, time=t, istp=istp)
            assert rc == 0 and st.n_cells == grid.ncells
        lanes = step.last_lane_cells()
        step.close()
        return out, lanes

    whole, lanes = two_steps(inp, inp.fields, later)
    assert lanes == inp.ncells
    new = {k: torch.zeros_like(v) for k, v in whole.items()}
    cut = 2 + (inp.nyp - 4) // 2
    for j0, j1 in ((2, cut), (cut, inp.nyp - 2)):
        sub = type(inp)(**{**inp.__dict__, "nyp": j1 - j0 + 4})
        sl = slice(j0 - 2, j1 + 2)
        part = [{k: v[..., sl, :, :].contiguous() for k, v in f.items()} for f in (inp.fields, later)]
        o, lanes = two_steps(sub, *part)
        assert lanes == 0
        for k, v in o.items():
            new[k][..., j0:j1, :, :] = v[..., 2:-2, :, :]
    base = dict(inp.fields)
    inp.fields = later
    _compare(inp, whole, new, False)
    # it shows: a step that computes its kernels finds these pairs empty
    computed, _ = two_steps(inp, base, later, fetch=False)
    d = (computed["mprecpt"] - whole["mprecpt"]).abs().max()
    assert float(d) > 1e-3 * float(whole["mprecpt"].abs().max())
