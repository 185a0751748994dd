"""Skinny kernels on a wide operand whose stride-one index is contracted (loads
along k): quads of k as 16-byte loads where rows are aligned, single elements
otherwise (odd K, rows off a 16-byte boundary, the operand itself off one),
boxes with positions outside the tensor, K tails, k slices. Oracle: the FP64
loop nest, with the tolerances of the other skinny tests."""
import numpy as np
import pytest

from helpers import seeded_normal
from oracle import LoopNest, error_metrics
from tccg_b200 import make_contraction
from tccg_b200.plan import Plan, Tuning

pytestmark = pytest.mark.gpu

# name: (C, A, B, extents): the wide operand is A[k.., x, y..]
CASES = {
    "aligned": ("xyn", "kxy", "kn", dict(x=37, y=29, n=7, k=64)),
    "quad_tail": ("xyn", "kxy", "kn", dict(x=152, y=5, n=16, k=36)),
    "long": ("xyn", "kxy", "kn", dict(x=23, y=40, n=13, k=292)),  # 10 chunks: quads on the register path
    "odd_k": ("xyn", "kxy", "kn", dict(x=50, y=21, n=9, k=283)),
    "few_k": ("xyn", "kxy", "kn", dict(x=90, y=11, n=5, k=3)),
    "two_modes": ("xyn", "kxly", "kln", dict(x=31, y=17, n=18, k=20, l=15)),
    "c_along_n": ("nxy", "kxy", "kn", dict(x=19, y=60, n=20, k=96)),
}


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("precision,skinny", [("bf16x3", 2), ("fp32", 1)])
@pytest.mark.parametrize("name", sorted(CASES))
def test_load_along_k(cuda, name, precision, skinny, offset):
    import torch
    lc, la, lb, sizes = CASES[name]
    con = make_contraction(lc, la, lb, sizes, 0.75, 0.5)
    ln = LoopNest(lc, la, lb, sizes)
    A, B, C = (seeded_normal(n, 31 + i).astype(np.float32)
               for i, n in enumerate((ln.size_a, ln.size_b, ln.size_c)))
    buf = torch.empty(A.size + 4, device="cuda")
    dA = buf[offset:offset + A.size]  # offset 1: off a 16-byte boundary
    dA.copy_(torch.from_numpy(A))
    ref = ln.run(A.astype(np.float64), B.astype(np.float64), C.astype(np.float64), 0.75, 0.5)
    for ksplit in (1, 2):
        p = Plan(con, precision, tuning=Tuning(skinny=skinny, ksplit=ksplit))
        assert "load=k" in p.describe() and "skinny" in p.describe()
        dC = torch.from_numpy(C).cuda()
        p.run(dA, torch.from_numpy(B).cuda(), dC)
        torch.cuda.synchronize()
        assert p.status() == 0
        out = dC.cpu().numpy()
        assert error_metrics(out, ref)["normwise"] <= (1e-5 if precision == "bf16x3" else 1e-6)
