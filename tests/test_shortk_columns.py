"""The short-K kernel on a 2-D C whose columns start off 16-byte boundaries
(FP32: one bulk copy per column and its edge elements): every column offset
modulo 16 bytes, columns shorter and longer than a tile, C itself off a
boundary, beta read or not. Same k order and epilogue arithmetic as the tile
kernel, so bit for bit its result; and nothing outside C is written."""
import pytest

from tccg_b200 import make_contraction
from tccg_b200.plan import Plan, Tuning

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beta", [0.0, -0.5])
@pytest.mark.parametrize("offset", [0, 1, 2, 3])
@pytest.mark.parametrize("m,n,k", [(1, 5, 7), (3, 130, 1), (5, 128, 16), (127, 129, 32), (129, 64, 19),
                                   (130, 257, 4), (259, 300, 17), (384, 131, 31), (513, 40, 25)])
def test_bitwise_and_in_bounds(cuda, m, n, k, offset, beta):
    import torch
    con = make_contraction("mn", "mk", "kn", dict(m=m, n=n, k=k), 1.25, beta)
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    A = torch.randn(m * k, generator=g, device="cuda")
    B = torch.randn(k * n, generator=g, device="cuda")
    whole = torch.randn(m * n + 16, generator=g, device="cuda")
    outs = []
    for tuning in (Tuning(shortk=1, ksplit=1), Tuning(shortk=-1, direct=-1, ksplit=1, simt_tile=1)):
        p = Plan(con, "fp32", tuning=tuning)
        buf = whole.clone()
        p.run(A, B, buf[4 + offset:4 + offset + m * n])
        torch.cuda.synchronize()
        assert p.status() == 0
        outs.append((p.describe(), buf))
    assert "simt_shortk" in outs[0][0] and "simt_gett" in outs[1][0]
    assert torch.equal(outs[0][1], outs[1][1])
    out = outs[0][1]
    assert torch.equal(out[:4 + offset], whole[:4 + offset])
    assert torch.equal(out[4 + offset + m * n:], whole[4 + offset + m * n:])
