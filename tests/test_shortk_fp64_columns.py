"""FP64 short-K calls on a 2-D C whose columns start off 16-byte boundaries take
the short-K kernel's element form by themselves: the FP64 product, every column
offset, beta read or not, nothing outside C written."""
import pytest

from tccg_b200 import make_contraction
from tccg_b200.plan import Plan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [0.0, -0.5])
@pytest.mark.parametrize("m,n,k", [(2305, 2307, 16), (4097, 1025, 1), (129, 20001, 9)])
def test_odd_columns(cuda, m, n, k, beta):
    import torch
    con = make_contraction("mn", "mk", "kn", dict(m=m, n=n, k=k), 1.25, beta)
    p = Plan(con, "fp64")
    assert "simt_shortk<f64>" in p.describe() and "cblock=cp.async(" in p.describe()
    g = torch.Generator(device="cuda").manual_seed(m)
    draw = lambda s: torch.randn(s, generator=g, device="cuda", dtype=torch.float64)
    A, B, whole = draw(m * k), draw(k * n), draw(m * n + 8)
    ref = 1.25 * (B.view(n, k) @ A.view(k, m))
    for offset in (0, 1):
        buf = whole.clone()
        out = buf[4 + offset:4 + offset + m * n]
        want = ref + beta * out.view(n, m)
        p.run(A, B, out)
        torch.cuda.synchronize()
        assert p.status() == 0
        assert ((out.view(n, m) - want).norm() / want.norm()).item() <= 1e-13
        assert torch.equal(buf[:4 + offset], whole[:4 + offset])
        assert torch.equal(buf[4 + offset + m * n:], whole[4 + offset + m * n:])
