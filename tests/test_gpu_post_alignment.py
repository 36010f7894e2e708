"""tend_constrain2 on arrays that are not 16-byte aligned (an LES slice) and of odd lengths:
bit for bit the result on aligned copies."""
import pytest
import torch

from uclales_salsa_gb300.api import SalsaStep
from post_cases import post_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [(0, 1), (1, 0), (1, 1)])   # values, tendencies: doubles off alignment
def test_tend_constrain_any_alignment(shift):
    inp, a = post_state("grid384x384x160", X=3, Y=3, Z=5)     # 7 x 7 x 7 points: odd counts

    def put(v, off):
        buf = torch.empty(v.numel() + 2, dtype=torch.float64, device="cuda")
        out = buf[off:off + v.numel()].view(v.shape)
        out.copy_(v)
        return out

    step = SalsaStep(inp.cfg)
    res = []
    for vs, ts in ((0, 0), shift):
        d = {k: put(v, ts if k.endswith("t") else vs) for k, v in a.items()}
        step.tend_constrain(inp.nzp, inp.nxp, inp.nyp, inp.dt, d)
        torch.cuda.synchronize()
        res.append({k: v.cpu() for k, v in d.items()})
    step.close()
    for k in a:
        assert torch.equal(res[0][k], res[1][k]), k
    assert any(not torch.equal(res[0][k], a[k]) for k in a)
