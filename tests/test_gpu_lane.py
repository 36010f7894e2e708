"""The step's lane form (one cell per lane, calls of 24,576 cells and more) against the warp
form (one warp per cell, smaller calls): the same cells, once in one call and once in parts.

Cells are independent, so both must give the same tendencies up to rounding.  The bound is
the parity tests': 1e-10 of the new state or, where the scheme is ill-conditioned (Aitken
water in supersaturation, new ice), a small share of the values, each within 1e-6 of the
field's largest change.  Ragged sizes leave a tile and a block partly filled.
"""
import pytest
import torch

from uclales_salsa_gb300.api import SalsaStep
from uclales_salsa_gb300.inputs import make_inputs, make_outputs
from parity import STATE_OF, floor_of, interior

pytestmark = pytest.mark.gpu

CASES = {
    "columns": ("grid384x384x160", dict(X=32, Y=31, Z=27), {}, None),          # 26,784 cells
    "moist": ("grid256x256x128", dict(X=29, Y=31, Z=28), {}, None),             # 25,172
    "warm": ("grid16x16x40", dict(X=25, Y=25, Z=40), {}, None),                 # 25,000
    "gases": ("grid384x384x160", dict(X=32, Y=32, Z=24), dict(gases=True), None),   # 24,576, the least
    "ice_modes": ("grid256x256x128", dict(X=32, Y=32, Z=25), {}, "ice"),
    "classic_ice_melting": ("grid384x384x160", dict(X=32, Y=32, Z=25), {}, "classic"),
    "cloudbase_charge": ("grid384x384x160", dict(X=32, Y=32, Z=25), {}, "cloudbase"),
    "autoconv2_nocoag": ("grid384x384x160", dict(X=32, Y=32, Z=25), {}, "nocoag"),
}


def _modify(inp, kind):
    c = inp.cfg
    if kind == "ice":
        c.lsicehom = c.lsiceimm = c.lsicedep = 1
    if kind == "classic":
        c.ice_theta_dist = 0
        c.lsicehom = c.lsiceimm = c.lsicedep = 1
        inp.fields["temp"] += 12.0
        inp.fields.pop("indef")
    if kind == "cloudbase":
        c.lsactiv.mode = 2
        c.chargeCollEnh = 0.5
        g = torch.Generator(device="cuda").manual_seed(3)
        shp = (inp.layout.nliquid,) + tuple(inp.fields["press"].shape)
        inp.fields["chargeTime"] = torch.rand(shp, generator=g, device="cuda", dtype=torch.float64) * 500
    if kind == "nocoag":
        c.lscoag.sw = 0
        c.lsauto.mode = 2


def _run(inp, fields, lcharge):
    outs = make_outputs(inp)
    step = SalsaStep(inp.cfg)
    f = {k: v.clone() for k, v in fields.items()}
    rc, st = step.run(inp, f, outs, time=1.0, lcharge=lcharge)
    torch.cuda.synchronize()
    n = step.last_launches()
    step.close()
    assert rc == 0 and st.n_cells == inp.ncells, (rc, st.as_dict(), n)
    for k in ("indef", "chargeTime"):
        if k in f:
            outs[k] = f[k]
    return outs


@pytest.mark.parametrize("name", list(CASES))
def test_lane_form_equals_warp_form(name):
    wl, size, kw, kind = CASES[name]
    inp = make_inputs(wl, "cuda", **size, **kw)
    _modify(inp, kind)
    lcharge = int("chargeTime" in inp.fields)
    whole = _run(inp, inp.fields, lcharge)
    # the same cells in two calls: y rows with their halo
    nyp, parts = inp.nyp, {k: torch.zeros_like(v) for k, v in whole.items()}
    cut = 2 + (nyp - 4) // 2
    for j0, j1 in ((2, cut), (cut, nyp - 2)):
        sub = type(inp)(**{**inp.__dict__, "nyp": j1 - j0 + 4})
        sl = slice(j0 - 2, j1 + 2)
        f = {k: v[..., sl, :, :].contiguous() for k, v in inp.fields.items()}
        sub.fields = f
        o = _run(sub, f, lcharge)
        for k, v in o.items():
            parts[k][..., j0:j1, :, :] = v[..., 2:-2, :, :]
    dims = (inp.nzp, inp.nxp, inp.nyp)
    for k, a in whole.items():
        a, b = interior(a, *dims), interior(parts[k], *dims)
        if k in STATE_OF:
            old = interior(inp.fields[STATE_OF[k]], *dims)
            scale = torch.maximum((old + b * inp.dt).abs(), old.abs()).clamp(min=floor_of(k))
            rel = (a - b).abs() * inp.dt / scale
        else:
            rel = (a - b).abs() / b.abs().amax().clamp(min=1e-300)
        assert bool(torch.isfinite(rel).all())
        assert float((rel <= 1e-10).double().mean()) >= 0.99, (k, float((rel <= 1e-10).double().mean()))
        top = float(b.abs().max())
        assert float((a - b).abs().max()) <= 1e-6 * top, (k, float((a - b).abs().max()), top)
