"""The skinny register path's scalar form (one wave of jobs) and its pair form
(more jobs, and grouped runs): the FP64 loop nest within FP32's tolerance, and
each other's bits, at K tails, boxes with positions outside the tensor and k
slices."""
import numpy as np
import pytest

from helpers import seeded_normal
from oracle import LoopNest, error_metrics
from tccg_b200 import make_contraction
from tccg_b200.plan import Tuning

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ksplit", [1, 2])
@pytest.mark.parametrize("m,n,k", [(300, 3, 1), (5001, 8, 23), (5001, 9, 32), (5001, 16, 33), (39000, 7, 17),
                                   (40000, 12, 33), (155000, 4, 30)])
@pytest.mark.parametrize("la", ["mk", "km"])
def test_forms_agree(cuda, la, m, n, k, ksplit):
    import torch
    from tccg_b200.grouped import Group
    sizes = dict(m=m, n=n, k=k)
    con = make_contraction("mn", la, "kn", sizes, 1.25, -0.5)
    ln = LoopNest("mn", la, "kn", sizes)
    A, B, C = (seeded_normal(s, 71 + i).astype(np.float32)
               for i, s in enumerate((ln.size_a, ln.size_b, ln.size_c)))
    dA, dB, dC = (torch.from_numpy(x).cuda() for x in (A, B, C))
    grp = Group([con], "fp32", tunings=[Tuning(skinny=1, ksplit=ksplit)])
    assert "path=registers" in grp.plans[0].describe()
    grp.bind([dA], [dB], [dC])
    grp.run()
    torch.cuda.synchronize()
    grouped = dC.clone()
    dC.copy_(torch.from_numpy(C))
    grp.run_per_item()
    torch.cuda.synchronize()
    assert grp.plans[0].status() == 0
    assert torch.equal(grouped, dC)
    ref = ln.run(A.astype(np.float64), B.astype(np.float64), C.astype(np.float64), 1.25, -0.5)
    assert error_metrics(dC.cpu().numpy(), ref)["normwise"] <= 1e-6
