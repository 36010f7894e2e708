"""States at the limits of the step, lane form (one call) against warp form (the same cells in
two calls below the lane form's size)."""
import pytest
import torch

from uclales_salsa_gb300.api import SalsaStep
from uclales_salsa_gb300.inputs import make_inputs, make_outputs
from parity import interior

pytestmark = pytest.mark.gpu
BINS = ("naerot", "ncloudt", "nprecpt", "nicet", "maerot", "mcloudt", "mprecpt", "micet")
CELLS = ((2, 2, 1), (5, 9, 14), (20, 33, 27), (32, 17, 3))   # y, x, z


def _run(inp, fields):
    outs = make_outputs(inp)
    step = SalsaStep(inp.cfg)
    f = {k: v.clone() for k, v in fields.items()}
    rc, st = step.run(inp, f, outs, time=1.0)
    torch.cuda.synchronize()
    step.close()
    assert rc in (0, 4) and st.n_cells == inp.ncells, (rc, st.as_dict())
    return outs, st


def _both(inp):
    """Outputs of one call, of the same cells in two calls (y rows with their halo), and the
    counts of cells with non-finite numbers."""
    whole, st = _run(inp, inp.fields)
    nyp, parts, bad = inp.nyp, {k: torch.zeros_like(v) for k, v in whole.items()}, 0
    cut = 2 + (nyp - 4) // 2
    for j0, j1 in ((2, cut), (cut, nyp - 2)):
        sub = type(inp)(**{**inp.__dict__, "nyp": j1 - j0 + 4})
        f = {k: v[..., j0 - 2:j1 + 2, :, :].contiguous() for k, v in inp.fields.items()}
        sub.fields = f
        o, s = _run(sub, f)
        bad += s.n_nonfinite
        for k, v in o.items():
            parts[k][..., j0:j1, :, :] = v[..., 2:-2, :, :]
    dims = (inp.nzp, inp.nxp, inp.nyp)
    return {k: interior(v, *dims) for k, v in whole.items()}, {k: interior(v, *dims) for k, v in parts.items()}, \
        st.n_nonfinite, bad


@pytest.mark.parametrize("precision", [0, 1])
def test_negative_ice_without_coagulation(precision):
    """Advection can leave slightly negative ice.  Coagulation sets it to zero; without it the
    freezing of a liquid bin does so in the crystal bin that it freezes to, and nowhere else.
    (A populated crystal bin of negative volume has no diameter: NaN in both forms.)"""
    inp = make_inputs("grid384x384x160", "cuda", X=32, Y=43, Z=31, precision=precision,
                      overrides=dict(cloudy=0.3, pattern="random"))   # 42,656 cells
    inp.cfg.lscoag.sw = 0
    f = inp.fields
    g = torch.Generator(device="cuda").manual_seed(4)
    for name in ("nice", "mice"):
        r = torch.rand(f[name].shape, generator=g, device="cuda", dtype=torch.float64)
        f[name] = torch.where(r < 0.3, -1e-3 * f[name].abs().amax() * r, f[name])
    a, b, _, _ = _both(inp)
    for key in ("nicet", "micet"):
        old = interior(f[key[:-1]], inp.nzp, inp.nxp, inp.nyp)
        assert torch.equal(torch.isnan(a[key]), torch.isnan(b[key])), key
        # which of the negative values stay, and which are set to zero
        stay = [(old < 0) & (old + o[key] * inp.dt <= 0.5 * old) for o in (a, b)]
        assert torch.equal(stay[0], stay[1]), (key, int((stay[0] != stay[1]).sum()))
        assert bool(stay[1].any()) and bool(((old < 0) & ~stay[1]).any())


@pytest.mark.parametrize("coag", [0, 1])
@pytest.mark.parametrize("value", [float("nan"), float("inf"), 0.0])
def test_density_that_is_not_a_positive_number(value, coag):
    """0 dn and 0 / dn are NaN then: the empty bins of such a cell show it too, and no other
    cell does."""
    inp = make_inputs("grid384x384x160", "cuda", X=32, Y=31, Z=27, overrides=dict(cloudy=0.0))   # 26,784 cells
    inp.cfg.lscoag.sw = coag
    for j, i, k in CELLS:
        inp.fields["dn"][j, i, k] = value
    a, b, na, nb = _both(inp)
    assert na == nb
    for key in BINS:
        assert torch.equal(torch.isnan(a[key]), torch.isnan(b[key])), key
    # (coagulation sets infinite numbers to zero, and 1/dn is zero: nothing is left to see)
    ok = torch.ones(b["naerot"].shape[1:], dtype=torch.bool, device="cuda")
    for j, i, k in CELLS:
        assert bool(torch.isnan(a["naerot"][:, j - 2, i - 2, k - 1]).any()) == (not (coag and value > 0.0))
        ok[j - 2, i - 2, k - 1] = False
    for key in BINS:
        d = (a[key] - b[key])[:, ok].abs()
        assert float(d.max()) <= 1e-6 * float(b[key][:, ok].abs().max()), key
