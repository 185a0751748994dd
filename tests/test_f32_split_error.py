"""FP32 calls that the library sends to the tensor cores by itself are no less
accurate than the same calls on the CUDA cores, also where the split's
truncations all go one way: operands of one sign, exponentials, wide ranges.
RMS error relative to |A| |B|, which every element counts in, against FP64."""
import pytest

from tccg_b200 import make_contraction
from tccg_b200.plan import Plan, Tuning

pytestmark = pytest.mark.gpu

DRAW = {
    "normal": lambda n, u: n,
    "uniform": lambda n, u: u,
    "exponential": lambda n, u: -(u + 1e-12).log(),
    "half_normal": lambda n, u: n.abs(),
    "lognormal1": lambda n, u: n.exp(),
    "lognormal2": lambda n, u: (2 * n).exp(),
    "log_uniform": lambda n, u: (-20 * u).exp(),
    "many_magnitudes": lambda n, u: (-55 * u).exp(),
}


def _errors(m, n, k, draw, **tuned):
    import torch
    g = torch.Generator(device="cuda").manual_seed(m + k)
    both = lambda s: (torch.randn(s, generator=g, device="cuda", dtype=torch.float64),
                      torch.rand(s, generator=g, device="cuda", dtype=torch.float64))
    A, B = DRAW[draw](*both(m * k)).float(), DRAW[draw](*both(k * n)).float()
    a, b = A.double().view(k, m), B.double().view(n, k)
    ref, scale = b @ a, b.abs() @ a.abs()  # C is [n][m]
    con = make_contraction("mn", "mk", "kn", dict(m=m, n=n, k=k))
    out = []
    for tuning in (Tuning(**tuned), Tuning(variant=-1, **tuned)):
        p = Plan(con, "fp32", tuning=tuning)
        C = torch.empty(m * n, device="cuda")
        p.run(A, B, C)
        torch.cuda.synchronize()
        assert p.status() == 0
        e = (C.double().view(n, m) - ref) / scale
        out.append((p.describe(), (e * e).mean().sqrt().item()))
    return out


# K at the edges of the chunk rule; few tiles (k slices on both sides)
@pytest.mark.parametrize("m,n,k,chunk", [(2048, 2080, 256, 1), (2048, 2080, 511, 1), (2048, 2080, 512, 2),
                                         (2048, 2080, 767, 2), (2048, 2080, 768, 3), (2048, 2080, 1535, 3),
                                         (2048, 2080, 1536, 4), (12648, 85, 4418, 3)])
@pytest.mark.parametrize("draw", sorted(DRAW))
def test_no_larger_error(cuda, m, n, k, chunk, draw):
    (d0, split), (d1, ffma) = _errors(m, n, k, draw)
    assert "gett_tc<F32X6>" in d0 and "chunk=%d " % chunk in d0 and "simt_gett" in d1
    assert split <= ffma


# many k slices: FFMA's errors of independent slices partly cancel
@pytest.mark.parametrize("m,n,k", [(1215, 72, 11200), (525, 320, 3600), (2856, 540, 352)])
@pytest.mark.parametrize("draw", ["normal", "uniform", "exponential", "half_normal", "lognormal1"])
def test_no_larger_error_in_slices(cuda, m, n, k, draw):
    (d0, split), (d1, ffma) = _errors(m, n, k, draw, tail_split=-1)
    assert "gett_tc<F32X6>" in d0 and "chunk=1 " in d0 and "simt_gett" in d1
    assert split <= ffma


def test_short_chains_stay(cuda):
    plan = lambda m, n, k: Plan(make_contraction("mn", "mk", "kn", dict(m=m, n=n, k=k)), "fp32").describe()
    for m, n, k in ((2048, 2080, 128), (4096, 4096, 255)):
        assert "simt_gett" in plan(m, n, k)
