"""The calls of this framework whose time is tracked, over the sizes and options it is used with.

A case is one call (or the pair of calls of `after_step`) of the public Python interface:
SalsaStep.run, SalsaStep.tend_constrain + diagnostics, SalsaStep.sedimentation,
SalsaChain.forward and the gradient through chain_apply.  Inputs are the seeded synthetic
fields of uclales_salsa_gb300.inputs, on blocks of the repository's workloads; `prepare`
makes them, the arrays a model keeps (tendencies, diagnostics) and the handle.

listed() names the cases, draw(rng) gives more of the same ranges, prepare / run / work
measure one, and exact gives reference values in plain torch where the arithmetic is a
formula per element (the tendency clamp).  The step, the sedimentation and the chain have no
closed form: a 64-bit restatement of them takes far longer than the calls.
"""
import math

import torch

from uclales_salsa_gb300.api import SalsaStep
from uclales_salsa_gb300.chain import SalsaChain, chain_apply, chain_config, pack_state
from uclales_salsa_gb300.inputs import make_inputs, make_outputs
from uclales_salsa_gb300.post_case import TRACERS, post_arrays, sedim_arrays


def listed():
    return [
        # the smallest calls: a ragged block of 105 cells (a column model, a unit test, the
        # corner of a decomposed grid), where the launch and the call itself count
        dict(name="step_105_cells", kind="step", workload="grid384x384x160", X=5, Y=3, Z=7, precision=0),
        # the warm box case of the tests: level 4, no ice, the whole 16 x 16 x 40 grid
        dict(name="step_warm_16x16x40", kind="step", workload="grid16x16x40", X=16, Y=16, Z=40, precision=0),
        # one rank's share of the convective grid (10 % cloudy columns with ice, the rest clear)
        dict(name="step_384_rank", kind="step", workload="grid384x384x160", X=48, Y=40, Z=160, precision=0),
        # a large block of it: the benchmark's mix at full height
        dict(name="step_384_large", kind="step", workload="grid384x384x160", X=96, Y=72, Z=160, precision=0),
        # the same block in the FP32-mixed form
        dict(name="step_384_mixed", kind="step", workload="grid384x384x160", X=96, Y=72, Z=160, precision=1),
        # stratiform mix near saturation: 30 % cloudy cells scattered among moist clear ones,
        # which activate (odd sizes)
        dict(name="step_256_moist", kind="step", workload="grid256x256x128", X=61, Y=53, Z=47, precision=0),
        # a batch of independent cells with kappa and supersaturation per cell (parcel studies)
        dict(name="step_batch_kappa", kind="step", workload="batch65536", X=1, Y=1, Z=65536, precision=0),
        # all cells in cloud with ice, the three secondary-ice schemes and gas condensation on
        dict(name="step_secondary_ice", kind="step_sip", workload="grid384x384x160", X=24, Y=24, Z=24, precision=0),
        # a model whose arrays stay in host memory: the slab pipeline around the step
        dict(name="step_host_arrays", kind="step_host", workload="grid384x384x160", X=24, Y=32, Z=40, precision=0),
        # what the time step runs after the SALSA step: the tendency clamp and SALSA_diagnostics
        dict(name="after_step_256", kind="after", workload="grid256x256x128", X=128, Y=128, Z=64, precision=0),
        # bin sedimentation of all four categories
        dict(name="sedimentation_256", kind="sedim", workload="grid256x256x128", X=96, Y=96, Z=128, precision=0),
        # gradients of the final cloud state through a chain of coagulation + condensation
        # steps: forward with checkpoints, then the adjoint
        dict(name="chain_gradient", kind="grad", workload="chain65536", X=1, Y=1, Z=8192, nsub=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _block(rng, cells, zmax):
    """An interior of about `cells` cells with any height up to zmax, odd sizes included."""
    z = min(zmax, max(3, _log(rng, 5, zmax)))
    xy = max(1.0, cells / z)
    x = max(1, int(round(math.sqrt(xy) * rng.uniform(0.6, 1.6))))
    return dict(X=max(2, x), Y=max(2, int(round(xy / max(2, x)))), Z=z)


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "step_sip", "step_host", "after", "sedim", "grad"])
    if kind == "grad":
        return dict(kind=kind, workload="chain65536", X=1, Y=1, Z=_log(rng, 64, 12000), nsub=rng.randint(1, 8))
    if kind == "after":
        return dict(kind=kind, workload=rng.choice(["grid256x256x128", "grid384x384x160", "grid16x16x40"]), precision=0,
                    **_block(rng, _log(rng, 2000, 1500000), 160))
    if kind == "sedim":
        return dict(kind=kind, workload=rng.choice(["grid256x256x128", "grid384x384x160", "grid16x16x40"]), precision=0,
                    **_block(rng, _log(rng, 2000, 1200000), 160))
    if kind == "step_sip":
        return dict(kind=kind, workload="grid384x384x160", precision=rng.choice([0, 0, 1]),
                    **_block(rng, _log(rng, 100, 14000), 60))
    if kind == "step_host":
        return dict(kind=kind, workload=rng.choice(["grid256x256x128", "grid384x384x160", "grid16x16x40"]),
                    precision=rng.choice([0, 1]), **_block(rng, _log(rng, 100, 30000), 60))
    wl = rng.choice(["grid384x384x160", "grid384x384x160", "grid256x256x128", "grid16x16x40", "batch65536"])
    top = {"grid384x384x160": 900000, "grid256x256x128": 250000, "grid16x16x40": 400000, "batch65536": 65536}[wl]
    n = _log(rng, 40, top)
    size = dict(X=1, Y=1, Z=n) if wl == "batch65536" else _block(rng, n, 160)
    return dict(kind=kind, workload=wl, precision=rng.choice([0, 0, 1]), **size)


def _inputs(case, seed, **kw):
    device = "cpu" if case["kind"] == "step_host" else "cuda"
    return make_inputs(case["workload"], device, X=case["X"], Y=case["Y"], Z=case["Z"],
                       precision=case.get("precision", 0), seed=seed, **kw)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "grad":
        inp = _inputs(case, seed)
        inp.cfg = chain_config()
        x, thermo, kappa, ssat = pack_state(inp)
        lay = inp.layout
        nl = lay.nbins + lay.ncld + lay.nprc
        # the scalar whose gradient is taken: the final cloud numbers and masses, each bin
        # relative to its initial value
        y = torch.zeros_like(x)
        for b in range(lay.nbins, lay.nbins + lay.ncld):
            for c in [b] + [nl + s * nl + b for s in range(lay.nwet)]:
                y[:, c] = 1.0 / x[:, c].abs().clamp(min=1e-30)
        return dict(kind=kind, chain=SalsaChain(inp.cfg), thermo=thermo, y=y, nsub=case["nsub"], dt=inp.dt,
                    x=x.requires_grad_(), kappa=kappa.requires_grad_(), ssat=ssat.requires_grad_())
    if kind == "step_sip":
        inp = _inputs(case, seed, gases=True, overrides=dict(cloudy=1.0, pattern="random"))
        for sw in (inp.cfg.lssecice, inp.cfg.lssiprimespln, inp.cfg.lssipdropfrac, inp.cfg.lssipicecollbreak):
            sw.sw, sw.mode = 1, 1
        for k, name in enumerate(("sipdrfr", "siprmspl", "sipiibr")):   # fragments of earlier steps
            inp.fields[name] = inp.fields["nice"] * (0.02 * (k + 1))
    else:
        inp = _inputs(case, seed)
    outs = make_outputs(inp)
    st = dict(kind=kind, inp=inp, step=SalsaStep(inp.cfg), fields=inp.fields, outs=outs)
    if kind == "step_host":     # page-locked, as a coupled model registers its arrays
        st["fields"] = {k: v.pin_memory() for k, v in inp.fields.items()}
        st["outs"] = {k: v.pin_memory() for k, v in outs.items()}
    if kind in ("after", "sedim"):
        # the state as it stands after one step's tendencies
        gen = torch.Generator(device="cuda").manual_seed(seed * 31 + 7)
        for v, t in TRACERS:
            if v not in inp.fields or t not in outs:
                continue
            r = torch.rand(outs[t].shape, generator=gen, device="cuda", dtype=torch.float64)
            # changes of a few per cent of a bin in a step, some of which would empty it
            outs[t].copy_(inp.fields[v] / inp.dt * torch.where(r < 0.02, -1.5 - r, (r - 0.5) * 0.1))
        if kind == "after":
            st["arrays"] = post_arrays(inp, inp.fields, outs)
        else:
            st["arrays"] = sedim_arrays(inp, inp.fields, outs)
    return st


def run(state):
    kind = state["kind"]
    if kind == "grad":
        x, kappa, ssat = state["x"], state["kappa"], state["ssat"]
        xN = chain_apply(state["chain"], x, kappa, ssat, state["thermo"], state["nsub"], state["dt"])
        gx, gk, gs = torch.autograd.grad(xN, [x, kappa, ssat], grad_outputs=state["y"])
        return dict(xN=xN, grad_x=gx, grad_kappa=gk, grad_ssat=gs)
    inp, step = state["inp"], state["step"]
    if kind == "after":
        a = state["arrays"]
        step.tend_constrain(inp.nzp, inp.nxp, inp.nyp, inp.dt, a)
        step.diagnostics(inp.nzp, inp.nxp, inp.nyp, a)
        return a
    if kind == "sedim":
        a = state["arrays"]
        step.sedimentation(inp.nzp, inp.nxp, inp.nyp, inp.dt, (1, 1, 1, 1), a)
        return {k: a[k] for k in a if k not in ("tk", "adn", "th", "ustar", "dzt", "naero", "maero", "ncloud", "mcloud",
                                                "nprecp", "mprecp", "nice", "mice")}
    step.run(inp, state["fields"], state["outs"], time=1.0)
    out = dict(state["outs"])
    for k in ("indef", "sipdrfr", "siprmspl", "sipiibr"):
        if k in state["fields"]:
            out[k] = state["fields"][k]
    return out


# floating-point operations of one cell and step (a library function counted as 20): the
# mean collision kernels, equilibration passes, condensation substeps and freezing rates per
# cell that the workloads need
_STEP_FLOPS = {"grid384x384x160": 5.0e4, "grid256x256x128": 7.0e4, "grid16x16x40": 4.0e4, "batch65536": 4.0e4}


def work(case):
    kind = case["kind"]
    cells = case["X"] * case["Y"] * case["Z"]
    if kind == "grad":
        # a state in and out of every step of the forward and of the adjoint
        nstate = 38 * 7
        return dict(bytes=8.0 * nstate * cells * (2 + 2 * case["nsub"]), flops=3 * 1.0e5 * cells * case["nsub"])
    plane = (case["X"] + 4) * (case["Y"] + 4) * (case["Z"] + 2)
    lvl5 = case["workload"] not in ("grid16x16x40", "batch65536")
    if kind in ("after", "sedim"):
        values = (17 + 14 + 7) * 7 + (7 * 8 if lvl5 else 0)
        if kind == "after":     # values and tendencies, the IN deficit, the diagnostics
            return dict(bytes=8.0 * plane * (2 * values + values + (38 if lvl5 else 0) + 10), flops=float(plane * values))
        fall = 14 if lvl5 else 7
        return dict(bytes=8.0 * plane * (3 * values + fall + 7), flops=150.0 * plane * 30)
    bytes_cell = 9368.0 if lvl5 else 7368.0
    flops = _STEP_FLOPS[case["workload"]] * (6 if kind == "step_sip" else 1)
    return dict(bytes=bytes_cell * cells, flops=flops * cells)


def exact(case, seed):
    """The clamped tendencies and IN deficit of `after_step`: max((-1 + 1e-8) p / dt, t) and
    [0, 1].  The other outputs and cases have no value here (see the head of the file)."""
    if case["kind"] != "after":
        return None
    st = prepare(case, seed)
    a, inp = st["arrays"], st["inp"]
    out = {k: None for k in a}
    for v, t in TRACERS:
        if v in a and t in a:
            out[t] = torch.maximum((-1.0 + 1.0e-8) * a[v] / inp.dt, a[t])
    if "indef" in a:
        out["indef"] = a["indef"].clamp(0.0, 1.0)
    return out
