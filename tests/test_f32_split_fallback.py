"""FP32 calls on the tensor cores whose values the split does not represent
(infinity, NaN, magnitudes near the largest): they give, bit for bit, what the
same call gives on the CUDA cores -- for operands of several modes read along
rows and along k, C read with beta, behind a tail split, with k slices, alone
and grouped."""
import pytest

from tccg_b200 import make_contraction
from tccg_b200.plan import Plan, Tuning

pytestmark = pytest.mark.gpu

# name: (C, A, B, extents, grouped tuning)
CASES = {
    "modes": ("ixyj", "kilj", "lykx", dict(i=40, j=50, x=44, y=36, k=20, l=28), False),
    "rows_fast": ("mn", "mk", "nk", dict(m=2001, n=1777, k=515), False),
    "k_fast": ("mn", "km", "kn", dict(m=1999, n=2050, k=700), False),
    "tail": ("mn", "mk", "kn", dict(m=3000, n=2000, k=2048), False),
    "runs": ("lykx", "kilj", "ixyj", dict(l=8, k=128, y=64, x=32, i=16, j=96), False),
    "slices": ("mn", "mk", "kn", dict(m=1215, n=72, k=11200), True),
    "slices_modes": ("xyn", "kxly", "kln", dict(x=25, y=21, n=320, k=60, l=60), True),
    "narrow": ("mn", "km", "nk", dict(m=12648, n=85, k=4418), True),
}
VALUES = {"inf": float("inf"), "nan": float("nan"), "near_max": 3.3e38}


def _data(con, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(t.num_elements(), generator=g, device="cuda") for t in (con.A0, con.B0, con.C0)]


def _tuning(name, **kw):
    return Tuning(tail_split=-1, **kw) if CASES[name][4] else Tuning(**kw)


def _equal(a, b):
    import torch
    return torch.equal(a.view(torch.int32), b.view(torch.int32)) or (
        torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.nan_to_num(a), torch.nan_to_num(b)))


@pytest.mark.parametrize("where", ["A", "B"])
@pytest.mark.parametrize("value", sorted(VALUES))
@pytest.mark.parametrize("name", sorted(CASES))
def test_bits_of_the_cuda_cores(cuda, name, value, where):
    import torch
    con = make_contraction(*CASES[name][:4], 1.5, 0.5)
    A, B, C = _data(con, 5)
    t = A if where == "A" else B
    t[t.numel() // 3] = VALUES[value]
    outs = []
    for tuning in (_tuning(name), _tuning(name, variant=-1)):
        p = Plan(con, "fp32", tuning=tuning)
        out = C.clone()
        p.run(A, B, out)
        torch.cuda.synchronize()
        assert p.status() == 0
        outs.append((p.describe(), out))
    assert "gett_tc<F32X6>" in outs[0][0] and "simt_gett" in outs[1][0]
    if name == "tail":
        assert "tail=16x" in outs[0][0] and "tail=16x1 " not in outs[0][0]
    if name.startswith("slices"):
        assert "ksplit=1 " not in outs[0][0] and "ksplit=1 " not in outs[1][0]
    assert _equal(outs[0][1], outs[1][1])


def test_group(cuda):
    """Items with and without such values in one captured launch: the per-item
    bits, and for the items with them the CUDA cores' bits."""
    import torch
    from tccg_b200.grouped import Group
    names = sorted(CASES) * 2
    items = [make_contraction(*CASES[n][:4], 1.25, -0.5) for n in names]
    data = [_data(c, 11 + i) for i, c in enumerate(items)]
    bad = range(0, len(names), 2)
    for i in bad:
        t = data[i][(i // 2) % 2]
        t[t.numel() // 5] = VALUES[sorted(VALUES)[i % 3]]
    outs = []
    for tunings in (None, [Tuning(variant=-1)] * len(items)):
        grp = Group(items, "fp32", tunings=tunings)
        Cs = [d[2].clone() for d in data]
        grp.bind([d[0] for d in data], [d[1] for d in data], Cs)
        grp.capture()
        for c, d in zip(Cs, data):
            c.copy_(d[2])
        grp.replay()
        torch.cuda.synchronize()
        outs.append([c.clone() for c in Cs])
        if tunings is None:
            assert sum("F32X6" in p.describe() for p in grp.plans) >= len(items) // 2
            for c, d in zip(Cs, data):
                c.copy_(d[2])
            grp.run_per_item()
            torch.cuda.synchronize()
            assert all(_equal(a, b) for a, b in zip(outs[0], Cs))
    for i in bad:
        assert _equal(outs[0][i], outs[1][i])
