"""Split-BF16x3 plans with a narrow side of at most 16 and a short K (under 8
chunks of 32) whose wide operand is contracted along its stride-one index run
FP32 multiply-adds (the register path), not split products: their results keep
FP32's error, which a split product's (4e-6) would exceed forty times over."""
import numpy as np
import pytest

from helpers import seeded_normal
from oracle import LoopNest, error_metrics
from tccg_b200 import make_contraction
from tccg_b200.plan import Plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(12400, 3, 40), (14726, 6, 70), (16384, 16, 33), (20001, 9, 168), (13000, 12, 224)])
def test_short_k_keeps_fp32(cuda, m, n, k):
    import torch
    sizes = dict(m=m, n=n, k=k)
    con = make_contraction("mn", "km", "kn", sizes, 1.0, 0.5)
    ln = LoopNest("mn", "km", "kn", sizes)
    A, B, C = (seeded_normal(s, 51 + i).astype(np.float32)
               for i, s in enumerate((ln.size_a, ln.size_b, ln.size_c)))
    p = Plan(con, "bf16x3")
    assert "path=registers" in p.describe()
    dA, dB, dC = (torch.from_numpy(x).cuda() for x in (A, B, C))
    p.run(dA, dB, dC)
    torch.cuda.synchronize()
    assert p.status() == 0
    ref = ln.run(A.astype(np.float64), B.astype(np.float64), C.astype(np.float64), 1.0, 0.5)
    # K + 2 roundings of at most 2^-24 of the partial sums: below 1e-6 of the
    # result's norm for N(0, 1) values (K <= 224)
    assert error_metrics(dC.cpu().numpy(), ref)["normwise"] <= 1e-6
