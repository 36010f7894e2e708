"""The step's lane form (one cell per lane, calls of 24,576 cells and more, 40,960 in
the mixed form) against the warp
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
    "mixed_columns": ("grid384x384x160", dict(X=32, Y=43, Z=31), dict(precision=1), None),
    "mixed_moist": ("grid256x256x128", dict(X=37, Y=38, Z=30), dict(precision=1, diagnostics=0), None),
    "mixed_warm": ("grid16x16x40", dict(X=32, Y=32, Z=40), dict(precision=1), None),
    "no_diagnostics": ("grid384x384x160", dict(X=32, Y=31, Z=27), dict(diagnostics=0), None),
    "large_layout": ("grid384x384x160", dict(X=32, Y=31, Z=27), {}, "bins"),
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
    if kind == "bins":
        _large_layout(inp)
    if kind == "nocoag":
        c.lscoag.sw = 0
        c.lsauto.mode = 2


def _large_layout(inp):
    """The default layouts of 20 drop and 20 crystal bins (equal sizes in both: pairs of a
    drop and a crystal bin take the self-coagulation offset), populated where the workload's
    seven bins are."""
    from uclales_salsa_gb300.layout import build_layout
    c, old = inp.cfg, inp.layout
    c.prc_nbins, c.prc_dlo, c.prc_vol_ratio = 20, 20.e-6, 2.0
    c.ice_nbins, c.ice_dlo, c.ice_vol_ratio = 20, 20.e-6, 2.0
    lay = build_layout(c)
    f = inp.fields
    for n, m, nb0, nsp, o in (("nprecp", "mprecp", old.nprc, old.nwet, lay.nbins + lay.ncld),
                              ("nice", "mice", old.nice, old.nwet + 1, lay.nliquid)):
        num, mas = f[n], f[m].view(nsp, nb0, *f[m].shape[1:])
        frac = mas / mas.sum(0, keepdim=True).clamp(min=1e-300)
        g = torch.Generator(device="cuda").manual_seed(11)
        new_n = torch.zeros((20,) + tuple(num.shape[1:]), dtype=torch.float64, device="cuda")
        new_m = torch.zeros((nsp, 20) + tuple(num.shape[1:]), dtype=torch.float64, device="cuda")
        for b in range(20):
            q = num[b % nb0] * (0.2 + 0.3 * torch.rand(num.shape[1:], generator=g, device="cuda", dtype=torch.float64))
            new_n[b] = q
            new_m[:, b] = frac[:, b % nb0] * q * 0.5236 * lay.dmid[o + b] ** 3 * 900.0
        f[n], f[m] = new_n, new_m.reshape(nsp * 20, *num.shape[1:]).contiguous()
    g = torch.Generator(device="cuda").manual_seed(12)
    f["indef"] = torch.rand((lay.nliquid,) + tuple(f["press"].shape), generator=g, device="cuda", dtype=torch.float64) * 0.05
    inp.layout = lay


def _run(inp, fields, lcharge):
    outs = make_outputs(inp, with_diag=bool(inp.cfg.diagnostics))
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


@pytest.mark.parametrize("precision", [0, 1])
def test_stored_kernels_in_the_lane_form(precision):
    """Low-frequency kernels (lscoag mode 2): the step that stores them equals the step that
    computes them; a later step that fetches them equals it too while the state is the same."""
    inp = make_inputs("grid384x384x160", "cuda", X=32, Y=32, Z=24 if precision == 0 else 40, precision=precision)
    ref = _run(inp, inp.fields, 0)
    inp.cfg.lscoag.mode, inp.cfg.cgintvl = 2, 10.0
    step = SalsaStep(inp.cfg)
    for t, istp in ((10.0, 1), (13.0, 4)):      # update step, then a fetching one
        f = {k: v.clone() for k, v in inp.fields.items()}
        out = make_outputs(inp)
        rc, st = step.run(inp, f, out, time=t, istp=istp)
        assert rc == 0
        for k in out:
            assert float((out[k] - ref[k]).abs().max()) <= 1e-9 * float(ref[k].abs().max()), (k, t)
    step.close()
