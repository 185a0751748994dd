"""The range of values that automatic FP32 plans run on the tensor cores:
everything finite up to |a| |b| K of about 2^78, down to subnormal operands and
results (operands are split times 2^23, their sums divided by 2^46)."""
import numpy as np
import pytest

from tccg_b200 import make_contraction
from tccg_b200.plan import Plan, Tuning

M, N, K = 2000, 2030, 600  # chunks of 2 k-blocks


def _bf16(x):
    """Round to nearest even bf16, as float32."""
    u = x.view(np.uint32)
    return ((u + (0x7FFF + ((u >> 16) & 1))) & np.uint32(0xFFFF0000)).view(np.float32)


def test_scaled_split_is_exact():
    """hi + mid + lo == 2^23 x, every part a bf16 number that is normal or zero,
    for every exponent of x from the subnormals to the largest that scales."""
    rng = np.random.default_rng(0)
    for e in range(0, 254 - 23):
        m = rng.integers(0, 1 << 23, 2000, dtype=np.uint32)
        m[:5] = 0, 1, (1 << 23) - 1, 0x7FFF, 0x8000
        x = (np.uint32(e << 23) | m).view(np.float32)
        y = x * np.float32(2.0 ** 23)
        assert np.array_equal(y.astype(np.float64), x.astype(np.float64) * 2.0 ** 23)
        hi = _bf16(y)
        mid = _bf16(y - hi)
        lo = y - hi - mid
        assert np.array_equal((hi.astype(np.float64) + mid) + lo, y.astype(np.float64))
        for part in (hi, mid, lo):
            assert np.array_equal(_bf16(part), part)
            assert ((part == 0) | (np.abs(part) >= 2.0 ** -126)).all()


def _operands(seed):
    """Magnitudes in [0.5, 2) of either sign: scaled by powers of two exactly."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    draw = lambda n: ((0.5 + 1.5 * torch.rand(n, generator=g, device="cuda")) *
                      (torch.randint(0, 2, (n,), generator=g, device="cuda") * 2.0 - 1.0))
    return draw(M * K), draw(K * N)


def _run(A, B, variant=0):
    import torch
    p = Plan(make_contraction("mn", "mk", "kn", dict(m=M, n=N, k=K)), "fp32", tuning=Tuning(variant=variant))
    assert ("gett_tc<F32X6>" in p.describe()) == (variant >= 0)
    C = torch.empty(M * N, device="cuda")
    p.run(A, B, C)
    torch.cuda.synchronize()
    assert p.status() == 0
    return C


def _rms(C, A, B):
    ref = B.double().view(N, K) @ A.double().view(K, M)
    scale = B.double().abs().view(N, K) @ A.double().abs().view(K, M)
    return (((C.double().view(N, M) - ref) / scale) ** 2).mean().sqrt().item()


@pytest.mark.gpu
@pytest.mark.parametrize("sa,sb", [(0, 0), (-60, -30), (-125, 60), (20, -100), (10, 15), (-53, -53)])
def test_powers_of_two(cuda, sa, sb):
    """The same arithmetic at any magnitude: bits scaled by the same power; at
    0 also the bits of a tuning that asks for the split."""
    import torch
    A, B = _operands(1)
    base = _run(A, B, variant=2)
    out = _run(A * 2.0 ** sa, B * 2.0 ** sb)
    assert torch.equal(out, base * 2.0 ** (sa + sb))
    assert not torch.equal(out, _run(A * 2.0 ** sa, B * 2.0 ** sb, variant=-1))


@pytest.mark.gpu
@pytest.mark.parametrize("name,sa,sb", [("subnormal_operand", -140, 60), ("subnormal_result", -70, -72),
                                        ("both", -130, -5)])
def test_subnormals(cuda, name, sa, sb):
    A, B = _operands(2)
    A, B = A * 2.0 ** sa, B * 2.0 ** sb
    assert (A != 0).all()
    assert _rms(_run(A, B), A, B) <= _rms(_run(A, B, variant=-1), A, B)


@pytest.mark.gpu
@pytest.mark.parametrize("decades", [30, 80])
def test_exponentials(cuda, decades):
    """Values down to 1e-30 in both operands, down to subnormals in one."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)
    draw = lambda n, d: torch.exp(-2.302585 * d * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)).float()
    A, B = draw(M * K, min(decades, 42)), draw(K * N, 30 if decades == 30 else 2)
    assert _rms(_run(A, B), A, B) <= _rms(_run(A, B, variant=-1), A, B)


@pytest.mark.gpu
@pytest.mark.parametrize("exponent,split", [(31, True), (36, False), (60, False), (120, False)])
def test_large_values(cuda, exponent, split):
    """Past the window's upper end the call gives the CUDA cores' bits, infinite
    sums among them."""
    import torch
    A, B = _operands(4)
    A, B = A * 2.0 ** exponent, B * 2.0 ** exponent
    out, ffma = _run(A, B), _run(A, B, variant=-1)
    if split:
        assert torch.equal(out, _run(A, B, variant=2)) and not torch.equal(out, ffma)
    else:
        assert torch.equal(torch.nan_to_num(out), torch.nan_to_num(ffma))
        assert torch.equal(torch.isnan(out), torch.isnan(ffma))
