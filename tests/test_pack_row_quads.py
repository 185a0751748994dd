"""BF16 packs that read the operands by quads of rows: the packed values are
those of the element-wise reads (taken when a buffer is off the quads'
alignment), so results are equal bit for bit -- tiles and K ragged, padding of
K, rows visited along another mode than the first, operands in FP32 and BF16,
packed for a call and for a group."""
import pytest

from tccg_b200 import make_contraction
from tccg_b200.plan import Plan, Tuning

pytestmark = pytest.mark.gpu

CASES = {
    "one_tile": ("mn", "mk", "nk", dict(m=128, n=128, k=64)),
    "ragged_rows": ("mn", "mk", "nk", dict(m=132, n=64, k=200)),
    "k_one": ("mn", "mk", "nk", dict(m=260, n=100, k=1)),
    "k_ragged": ("mn", "mk", "nk", dict(m=124, n=384, k=133)),
    "k_modes": ("abn", "akbl", "nlk", dict(a=20, b=9, n=68, k=7, l=11)),
    "visit": ("abn", "bak", "nk", dict(a=37, b=44, n=72, k=150)),
    "one_side": ("mn", "mk", "kn", dict(m=256, n=96, k=96)),   # B streams along k
}


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_bitwise(cuda, name, dtype):
    import torch
    lc, la, lb, sizes = CASES[name]
    con = make_contraction(lc, la, lb, sizes, 1.0, 0.0)
    tdt = torch.float32 if dtype == "f32" else torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(len(name))
    A = torch.randn(con.A0.num_elements(), generator=g, device="cuda").to(tdt)
    B = torch.randn(con.B0.num_elements(), generator=g, device="cuda").to(tdt)
    p = Plan(con, "bf16", dtype=dtype, tuning=Tuning(variant=16, skinny=-1))
    assert "rquad a=1" in p.describe() or "rquad a=0 b=1" in p.describe(), p.describe()
    outs = []
    for off in (0, 1):
        bufs = [torch.empty(x.numel() + 8, dtype=tdt, device="cuda")[off:off + x.numel()] for x in (A, B)]
        for b, x in zip(bufs, (A, B)):
            b.copy_(x)
        C = torch.full((con.C0.num_elements(),), float("nan"), device="cuda")
        p.run(bufs[0], bufs[1], C)
        torch.cuda.synchronize()
        assert p.status() == 0
        outs.append(C)
    assert torch.equal(outs[0], outs[1])


def test_in_a_group(cuda):
    import torch
    from tccg_b200.grouped import Group
    items = [make_contraction(*CASES[n], 1.0, 0.0) for n in ("ragged_rows", "k_ragged", "one_side")]
    g = torch.Generator(device="cuda").manual_seed(3)
    new = lambda c: [torch.randn(t.num_elements(), generator=g, device="cuda") for t in (c.A0, c.B0)]
    ops = [new(c) for c in items]
    grp = Group(items, "bf16", tunings=[Tuning(variant=16, skinny=-1)] * len(items))
    Cs = [torch.zeros(c.C0.num_elements(), device="cuda") for c in items]
    grp.bind([o[0] for o in ops], [o[1] for o in ops], Cs)
    grp.run()
    torch.cuda.synchronize()
    for c, (A, B), C in zip(items, ops, Cs):
        off = [torch.empty(x.numel() + 8, device="cuda")[1:1 + x.numel()].copy_(x) for x in (A, B)]
        want = torch.zeros_like(C)
        Plan(c, "bf16", tuning=Tuning(variant=16, skinny=-1)).run(off[0], off[1], want)
        torch.cuda.synchronize()
        assert torch.equal(C, want)


@pytest.mark.parametrize("k,l,n", [(8, 32, 100), (12, 20, 33), (4, 64, 257), (36, 28, 64)])
def test_bf16_k_blocks(cuda, k, l, n):
    """BF16 operands whose unit-stride mode is a later K mode (8-byte quads)."""
    import torch
    con = make_contraction("mn", "kml", "lnk", dict(m=400, n=n, k=k, l=l), 1.0, 0.0)
    g = torch.Generator(device="cuda").manual_seed(k + l)
    A = torch.randn(con.A0.num_elements(), generator=g, device="cuda").bfloat16()
    B = torch.randn(con.B0.num_elements(), generator=g, device="cuda").bfloat16()
    p = Plan(con, "bf16", dtype="bf16", tuning=Tuning(variant=16, skinny=-1))
    assert "b=%dx%dx" % (k, l) in p.describe(), p.describe()
    outs = []
    for off in (0, 1):
        b = torch.empty(B.numel() + 8, dtype=B.dtype, device="cuda")[off:off + B.numel()].copy_(B)
        C = torch.full((con.C0.num_elements(),), float("nan"), device="cuda")
        p.run(A, b, C)
        torch.cuda.synchronize()
        assert p.status() == 0
        outs.append(C)
    assert torch.equal(outs[0], outs[1])
