"""The FP32 split with several tiles per CTA (every barrier's phase carried from
one tile to the next), its tail split and its k slices, against FP64. 1e-6 is
the FP32 tests' tolerance; on N(0, 1) operands the split's error is below 2e-7
at any K."""
import pytest

from tccg_b200 import make_contraction
from tccg_b200.plan import Plan, Tuning

pytestmark = pytest.mark.gpu

# (m, n, k, tuning, what the plan must be)
CASES = {
    "tail": (3000, 2000, 2048, dict(), "tail=16x"),
    "tail_chunk_1": (3000, 2000, 1100, dict(variant=1), "tail=16x"),
    "three_tiles": (2600, 2700, 300, dict(variant=4), "tail=0x1"),
    "two_fills": (2600, 2700, 4096 + 65, dict(variant=4, ksplit=1), "ksplit=1"),
    "odd_chunk": (2600, 2700, 1000, dict(variant=3, ksplit=1), "chunk=3"),
    "slices": (500, 300, 12000, dict(variant=2), "chunk=2"),
}


@pytest.mark.parametrize("beta", [0.0, 0.5])
@pytest.mark.parametrize("name", sorted(CASES))
def test_against_fp64(cuda, name, beta):
    import torch
    m, n, k, tuning, what = CASES[name]
    con = make_contraction("mn", "mk", "kn", dict(m=m, n=n, k=k), 1.25, beta)
    g = torch.Generator(device="cuda").manual_seed(k)
    A, B, C = (torch.randn(s, generator=g, device="cuda") for s in (m * k, k * n, m * n))
    ref = 1.25 * (B.double().view(n, k) @ A.double().view(k, m)) + beta * C.double().view(n, m)
    p = Plan(con, "fp32", tuning=Tuning(**tuning))
    d = p.describe()
    assert "gett_tc<F32X6>" in d and what in d and "tail=16x1 " not in d
    tiles = -(-m // 128) * -(-n // 160)
    assert name == "slices" or tiles > 2 * 148
    for _ in range(2):  # the second run finds the first one's workspace
        out = C.clone()
        p.run(A, B, out)
    torch.cuda.synchronize()
    assert p.status() == 0
    assert ((out.double().view(n, m) - ref).norm() / ref.norm()).item() <= 1e-6
