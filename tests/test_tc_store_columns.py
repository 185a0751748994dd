"""Column stores of the tensor-core epilogue: whole and ragged tiles, k slices
(lanes past M take part in no column store there), beta read or not, and a C
whose column offsets pass 32 bits (the 64-bit path).

Tolerances: products of bf16 operands (and of the parts of a split) are exact;
K <= 500 terms with truncating sums stay below K * 2^-23 / sqrt(K) = 2.7e-6 of
the result's norm plus, for split-BF16x3, the dropped low product's 2^-16
(rms 2^-17.6): 1e-5 for both, 1e-6 for the six-product split."""
import pytest

from tccg_b200 import make_contraction
from tccg_b200.plan import Plan, Tuning

pytestmark = pytest.mark.gpu

TOL = {"bf16": 1e-5, "bf16x3": 1e-5, "fp32": 1e-6}


def _check(prec, m, n, k, beta, ksplit, ldc=None):
    import torch
    con = make_contraction("mn", "mk", "kn", dict(m=m, n=n, k=k), 1.25, beta)
    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    A = torch.randn(k, m, generator=g, device="cuda")
    B = torch.randn(n, k, generator=g, device="cuda")
    if prec == "bf16":
        A, B = A.bfloat16().float(), B.bfloat16().float()
    far = ldc is not None
    ldc = ldc or m + 3
    buf = torch.empty(ldc * (n - 1) + m, device="cuda")
    C = torch.as_strided(buf, (n, m), (ldc, 1))
    if not far:
        buf.fill_(7.0)
    C.copy_(torch.randn(n, m, generator=g, device="cuda"))
    want = 1.25 * (B.double() @ A.double()) + beta * C.double()
    p = Plan(con, prec, tuning=Tuning(variant=1 if prec == "bf16" else 4, ksplit=ksplit, skinny=-1),
             strides={"C": {"n": ldc}})
    assert "gett_tc<" in p.describe()
    assert ("ksplit=1 " in p.describe()) == (ksplit == 1)
    ws = torch.empty(max(p.workspace_bytes, 1), dtype=torch.uint8, device="cuda")
    p.run_ptr(A.data_ptr(), B.data_ptr(), buf.data_ptr(), 1.25, beta, ws.data_ptr(), ws.numel(),
              torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert p.status() == 0
    err = ((C.double() - want).norm() / want.norm()).item()
    assert err <= TOL[prec], err
    if not far:
        assert torch.all(torch.as_strided(buf, (n - 1, 3), (ldc, 1), m) == 7.0)


@pytest.mark.parametrize("beta", [0.0, -0.5])
@pytest.mark.parametrize("m,n,k", [(128, 192, 200), (129, 161, 180), (31, 97, 500), (256, 320, 130),
                                   (160, 33, 260), (300, 1, 200), (1, 200, 333), (2000, 3001, 150)])
@pytest.mark.parametrize("prec,ksplit", [("bf16", 1), ("bf16", 3), ("bf16x3", 1), ("bf16x3", 3),
                                         ("fp32", 1)])  # FP32: a split asked for stays off them
def test_tiles(cuda, prec, m, n, k, ksplit, beta):
    _check(prec, m, n, k, beta, ksplit)


@pytest.mark.parametrize("beta", [0.0, 0.5])
@pytest.mark.parametrize("prec", ["bf16", "bf16x3", "fp32"])
def test_far_columns(cuda, prec, beta):
    _check(prec, 150, 4, 140, beta, 1, ldc=1 << 30)
