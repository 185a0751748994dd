"""CUDA-core epilogue: C moves by quads of m wherever every quad of rows is
consecutive and aligned in C, also where the first M mode's extent is not a
multiple of 4 but the rows run on densely into the next mode; element by
element where one quad is not. Both against the FP64 loop nest."""
import numpy as np
import pytest

from helpers import seeded_normal
from oracle import LoopNest, error_metrics
from tccg_b200 import make_contraction
from tccg_b200.plan import Plan, Tuning

pytestmark = pytest.mark.gpu

# name: (C, A, B, extents, quads)
CASES = {
    "modes_run_on": ("abcd", "aeb", "edc", dict(a=37, b=28, c=13, d=11, e=23), 1),
    "even_first_mode": ("abcd", "aeb", "edc", dict(a=26, b=54, c=9, d=17, e=18), 1),
    "one_mode": ("mn", "mk", "kn", dict(m=132, n=70, k=30), 1),
    "odd_columns": ("mn", "mk", "kn", dict(m=131, n=70, k=30), 0),
    "split_modes": ("acbd", "aeb", "edc", dict(a=37, b=28, c=13, d=11, e=23), 0),
}


@pytest.mark.parametrize("precision,tol", [("fp32", 1e-6), ("fp64", 1e-13)])
@pytest.mark.parametrize("beta", [0.0, -0.5])
@pytest.mark.parametrize("name", sorted(CASES))
def test_quads(cuda, name, beta, precision, tol):
    import torch
    lc, la, lb, sizes, quads = CASES[name]
    con = make_contraction(lc, la, lb, sizes, 1.25, beta)
    ln = LoopNest(lc, la, lb, sizes)
    dt = np.float64 if precision == "fp64" else np.float32
    A, B, C = (seeded_normal(s, 61 + i).astype(dt) for i, s in enumerate((ln.size_a, ln.size_b, ln.size_c)))
    tuning = Tuning(shortk=-1, skinny=-1) if precision == "fp32" else Tuning(shortk=-1)
    p = Plan(con, precision, tuning=tuning)
    assert "simt_gett" in p.describe() and "cquads=%d" % quads in p.describe()
    ref = ln.run(A.astype(np.float64), B.astype(np.float64), C.astype(np.float64), 1.25, beta)
    for offset in (0, 1):  # C itself on and off a vector's boundary
        buf = torch.zeros(C.size + 4, dtype=torch.from_numpy(C).dtype, device="cuda")
        dC = buf[offset:offset + C.size]
        dC.copy_(torch.from_numpy(C))
        p.run(torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda(), dC)
        torch.cuda.synchronize()
        assert p.status() == 0
        assert error_metrics(dC.cpu().numpy(), ref)["normwise"] <= tol


@pytest.mark.parametrize("beta", [0.0, 0.75])
def test_fp64_many_tiles(cuda, beta):
    """FP64 with 10 and more tiles per SM: quads where C is read and aligned,
    elements on a C off the alignment; the same bits."""
    import torch
    m, n, k = 2052, 6000, 30
    con = make_contraction("mn", "mk", "kn", dict(m=m, n=n, k=k), 1.25, beta)
    p = Plan(con, "fp64", tuning=Tuning(shortk=-1))
    assert "simt_gett" in p.describe() and "cquads=1" in p.describe()
    g = torch.Generator(device="cuda").manual_seed(1)
    draw = lambda s: torch.randn(s, generator=g, device="cuda", dtype=torch.float64)
    A, B, C = draw(m * k), draw(k * n), draw(m * n)
    outs = []
    for offset in (0, 1):
        buf = torch.empty(m * n + 4, dtype=torch.float64, device="cuda")
        out = buf[offset:offset + m * n]
        out.copy_(C)
        p.run(A, B, out)
        outs.append(out)
    torch.cuda.synchronize()
    assert p.status() == 0 and torch.equal(outs[0], outs[1])
    ref = 1.25 * (B.view(n, k) @ A.view(k, m)) + beta * C.view(n, m)
    assert ((outs[0].view(n, m) - ref).norm() / ref.norm()).item() <= 1e-13
