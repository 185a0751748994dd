"""BF16 packs whose operands are read in different ways, in one launch: row
quads beside a streamed, a k-block and a 32-row operand, each as the larger
and as the smaller one (where the quads are dropped), both operand types, alone
and grouped. Packing only moves and rounds values, so every form of a
contraction gives the same bits as the same operands read from buffers off the
vectors' alignment, which drop to the element forms."""
import pytest

from tccg_b200 import make_contraction
from tccg_b200.plan import Plan, Tuning

pytestmark = pytest.mark.gpu

# name: (C, A, B, extents); A along its rows by quads
CASES = {
    "larger_beside_stream": ("mn", "mk", "kn", dict(m=512, n=68, k=260)),
    "smaller_beside_stream": ("mn", "mk", "kn", dict(m=68, n=700, k=260)),
    "larger_beside_rows": ("mn", "mk", "nk", dict(m=512, n=67, k=130)),
    "smaller_beside_rows": ("mn", "mk", "nk", dict(m=68, n=601, k=130)),
    "larger_beside_kblock": ("mn", "mkl", "lnk", dict(m=512, n=66, k=24, l=16)),
    "smaller_beside_kblock": ("mn", "mkl", "lnk", dict(m=68, n=600, k=24, l=16)),
    "both": ("mn", "mk", "nk", dict(m=260, n=132, k=70)),
    "neither": ("mn", "mkl", "lnk", dict(m=67, n=66, k=24, l=16)),
}


def _data(con, dtype, offset, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    out = []
    for t in (con.A0, con.B0):
        n = t.num_elements()
        buf = torch.empty(n + 8, dtype=dtype, device="cuda")
        x = buf[offset:offset + n]
        x.copy_(torch.randn(n, generator=g, device="cuda"))
        out.append(x)
    return out


@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_same_bits_as_element_reads(cuda, name, dtype):
    import torch
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    con = make_contraction(*CASES[name])
    p = Plan(con, "bf16", dtype=dtype, tuning=Tuning(variant=16))
    assert ("rquad a=1" in p.describe()) == (name != "neither")
    outs = []
    for offset in (0, 1):
        A, B = _data(con, dt, offset, 7)
        C = torch.empty(con.C0.num_elements(), device="cuda")
        p.run(A, B, C)
        outs.append(C)
    torch.cuda.synchronize()
    assert p.status() == 0
    assert torch.equal(outs[0], outs[1])
    lc, la, lb, _ = CASES[name]
    A, B = _data(con, dt, 0, 7)
    view = lambda t, x: x.double().view([i.size for i in reversed(t.indices)])
    ref = torch.einsum("%s,%s->%s" % (la[::-1], lb[::-1], lc[::-1]),
                       view(con.A0, A.to(torch.bfloat16)), view(con.B0, B.to(torch.bfloat16))).reshape(-1)
    # FP32 accumulation of exact products, at most 4 truncations per 64 k: 2e-6
    assert ((outs[0].double() - ref).norm() / ref.norm()).item() <= 4e-6


@pytest.mark.parametrize("names", [sorted(CASES), ["neither", "neither"]])
@pytest.mark.parametrize("dtype", ["bf16", "f32"])
def test_group(cuda, dtype, names):
    import torch
    from tccg_b200.grouped import Group
    dt = torch.bfloat16 if dtype == "bf16" else torch.float32
    items = [make_contraction(*CASES[n]) for n in names]
    data = [_data(c, dt, 0, i) for i, c in enumerate(items)]
    Cs = [torch.zeros(c.C0.num_elements(), device="cuda") for c in items]
    grp = Group(items, "bf16", dtype=dtype, tunings=[Tuning(variant=16)] * len(items))
    grp.bind([d[0] for d in data], [d[1] for d in data], Cs)
    grp.run()
    torch.cuda.synchronize()
    grouped = [c.clone() for c in Cs]
    grp.run_per_item()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(grouped, Cs))
