"""FP32 contractions on the tensor cores (kernel gett_tc<F32X6>): operands as
exact three-way bf16 splits, six products per term.

Error bound used below: products of the split are exact, the dropped ones are
below 2^-24 of a term, and each of the 8 MMAs of a 128-k chunk truncates its
sum by less than 2^-23 of it: 8 * 2^-23 < 1e-6 of the chunk's sum at worst,
and the chunk sums are added with round to nearest. So 1e-6 normwise at any
K, the tolerance of the FP32 tests."""
import numpy as np
import pytest

from helpers import seeded_normal
from oracle import LoopNest, error_metrics
from tccg_b200 import make_contraction
from tccg_b200.plan import Plan, Tuning

# name: (C, A, B, extents, alpha, beta, accumulation chunk in k-blocks of 32)
CASES = {
    "one_tile": ("mn", "mk", "kn", dict(m=128, n=160, k=32), 1.0, 0.0, 4),
    "rows_cols_ragged": ("mn", "mk", "kn", dict(m=129, n=161, k=47), 1.0, 0.0, 4),
    "k_one": ("mn", "mk", "kn", dict(m=70, n=90, k=1), 2.0, 0.5, 4),
    "k_16": ("mn", "km", "kn", dict(m=200, n=333, k=16), 1.0, 0.0, 4),
    "k_tail_17": ("mn", "km", "nk", dict(m=300, n=500, k=8 * 32 + 17), 1.0, -0.5, 2),
    "chunk_edge": ("mn", "mk", "nk", dict(m=140, n=100, k=256), 1.0, 0.0, 4),
    # the small products' accumulator is added up every 4096 k
    "fills_edge": ("mn", "mk", "kn", dict(m=130, n=170, k=4096), 1.0, 0.0, 4),
    "fills_past": ("mn", "mk", "kn", dict(m=130, n=170, k=4096 + 33), 1.0, 1.0, 4),
    # asks for one chunk of 6400 k: the plan keeps to 128
    "chunk_past_fill": ("mn", "mk", "kn", dict(m=64, n=64, k=8192 + 5), 1.0, 0.0, 200),
    # more tiles than CTAs, C's runs shorter than a warp (staged stores)
    "runs": ("anbm", "mak", "bkn", dict(a=11, n=40, b=61, m=97, k=70), 1.0, 0.0, 4),
    "swap": ("pqr", "qs", "spr", dict(p=37, q=129, r=31, s=253), 0.75, -0.5, 1),
    # few tiles: k slices added by the reduction
    "split": ("mn", "mk", "kn", dict(m=96, n=70, k=3 * 4096 + 65), 1.25, 0.5, 4),
    "k_modes": ("abij", "iman", "mnjb", dict(a=9, b=33, i=21, j=17, m=12, n=20), 1.0, 0.0, 4),
}


def _data(name, con_case):
    lc, la, lb, sizes = con_case[:4]
    ln = LoopNest(lc, la, lb, sizes)
    draw = lambda n, s: seeded_normal(n, s).astype(np.float32)
    return ln, draw(ln.size_a, 11), draw(ln.size_b, 12), draw(ln.size_c, 13)


def _run(con, tuning, A, B, C):
    import torch
    p = Plan(con, "fp32", tuning=tuning)
    dA, dB, dC = (torch.from_numpy(x).cuda() for x in (A, B, C))
    p.run(dA, dB, dC)
    torch.cuda.synchronize()
    assert p.status() == 0
    return dC.cpu().numpy(), p


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
def test_against_oracle(cuda, name):
    lc, la, lb, sizes, alpha, beta, chunk = CASES[name]
    con = make_contraction(lc, la, lb, sizes, alpha, beta)
    ln, A, B, C = _data(name, CASES[name])
    out, p = _run(con, Tuning(variant=chunk), A, B, C)
    assert "gett_tc<F32X6>" in p.describe()
    ref = ln.run(A.astype(np.float64), B.astype(np.float64), C.astype(np.float64), alpha, beta)
    assert error_metrics(out, ref)["normwise"] <= 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("k", [128, 513, 2048])
def test_no_larger_error_than_ffma(cuda, k):
    con = make_contraction("mn", "mk", "kn", dict(m=300, n=350, k=k))
    ln, A, B, C = _data("", ("mn", "mk", "kn", dict(m=300, n=350, k=k)))
    ref = ln.run(A.astype(np.float64), B.astype(np.float64), C.astype(np.float64), 1.0, 0.0)
    split, _ = _run(con, Tuning(variant=4), A, B, C)
    ffma, p = _run(con, Tuning(variant=-1, ksplit=1), A, B, C)
    assert "simt_gett" in p.describe()
    assert error_metrics(split, ref)["normwise"] <= error_metrics(ffma, ref)["normwise"]


SPECIAL = {"inf": np.inf, "nan": np.nan, "near_max": 3.3e38, "min_normal": 1.2e-38,
           "subnormal": 1e-42, "below_2^-100": 2.0 ** -101}


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["A", "B"])
@pytest.mark.parametrize("value", sorted(SPECIAL))
@pytest.mark.parametrize("shape", [dict(m=300, n=170, k=97), dict(m=3000, n=2000, k=300),
                                   dict(m=100, n=60, k=3000)])
def test_values_the_split_does_not_represent(cuda, value, where, shape):
    """Such operands run on the CUDA cores, bit for bit as with variant = -1,
    C read with beta as it was (also behind a tail split and a k-split); infinities and NaN
    come out where FFMA puts them."""
    con = make_contraction("mn", "mk", "kn", shape, 1.5, 0.5)
    _, A, B, C = _data("", ("mn", "mk", "kn", shape))
    (A if where == "A" else B)[len(A) // 3] = SPECIAL[value]
    split, _ = _run(con, Tuning(variant=4), A, B, C)
    ffma, _ = _run(con, Tuning(variant=-1, ksplit=1), A, B, C)
    assert np.array_equal(split, ffma, equal_nan=True)


@pytest.mark.gpu
def test_range_is_per_run(cuda):
    """The ranges belong to one run's operands: the same plan and workspace
    take ordinary values again after a run that could not."""
    import torch
    con = make_contraction("mn", "mk", "kn", dict(m=256, n=320, k=130))
    _, A, B, C = _data("", ("mn", "mk", "kn", dict(m=256, n=320, k=130)))
    p = Plan(con, "fp32", tuning=Tuning(variant=4))
    ws = torch.empty(p.workspace_bytes, dtype=torch.uint8, device="cuda")
    dA, dB = torch.from_numpy(A).cuda(), torch.from_numpy(B).cuda()
    bad = dA.clone()
    bad[5] = float("inf")
    outs = []
    for a in (dA, bad, dA):
        dC = torch.empty(C.size, device="cuda")
        p.run(a, dB, dC, workspace=ws)
        outs.append(dC)
    torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[2]) and not torch.isfinite(outs[1]).all()


@pytest.mark.gpu
def test_group(cuda):
    """A grouped run mixing split items (one with values they cannot take)
    with CUDA-core items, under a graph: bit for bit the per-item runs."""
    import torch
    from tccg_b200.grouped import Group
    names = ["runs", "fills_past", "swap", "k_modes", "split"]
    items = [make_contraction(*CASES[n][:4], CASES[n][4], CASES[n][5]) for n in names]
    items += [make_contraction("mn", "mk", "kn", dict(m=300, n=260, k=200), 1.0, 0.5)] * 2
    tunings = [Tuning(variant=CASES[n][6]) for n in names] + [Tuning(variant=4), Tuning(variant=-1)]
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda t: torch.randn(t.num_elements(), generator=g, device="cuda")
    As, Bs, C0 = ([rnd(getattr(c, t)) for c in items] for t in ("A0", "B0", "C0"))
    As[2][7] = float("inf")
    Cs = [c.clone() for c in C0]
    grp = Group(items, "fp32", tunings=tunings)
    assert sum("F32X6" in p.describe() for p in grp.plans) == 6
    grp.bind(As, Bs, Cs)
    grp.capture()
    for c, c0 in zip(Cs, C0):
        c.copy_(c0)
    grp.replay()
    torch.cuda.synchronize()
    grouped = [c.clone() for c in Cs]
    for c, c0 in zip(Cs, C0):
        c.copy_(c0)
    grp.run_per_item()
    torch.cuda.synchronize()
    for a, b in zip(grouped, Cs):
        assert torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))


@pytest.mark.gpu
def test_choice(cuda):
    kernel = lambda m, n, k, **t: Plan(make_contraction("mn", "mk", "kn", dict(m=m, n=n, k=k)), "fp32",
                                       tuning=Tuning(**t)).describe()
    assert "F32X6" in kernel(4096, 4096, 1024) and "launch=dependent" in kernel(4096, 4096, 1024)
    for t in (dict(variant=-1), dict(ksplit=3), dict(simt_tile=1), dict(direct=1)):
        assert "simt_gett" in kernel(4096, 4096, 1024, **t)
    # short K, or too few tiles for the persistent grid
    assert "simt_gett" in kernel(4096, 4096, 100) and "simt_gett" in kernel(512, 512, 4096)


def _bf16(x):
    """Round to nearest even bf16, as float32."""
    u = x.view(np.uint32)
    return ((u + (0x7FFF + ((u >> 16) & 1))) & np.uint32(0xFFFF0000)).view(np.float32)


def test_split_is_exact():
    """hi + mid + lo == x with bf16 parts for random significands over every
    exponent the range rule admits (2^-100 to below 2^127), in numpy."""
    rng = np.random.default_rng(0)
    for e in range(27, 254):
        m = rng.integers(0, 1 << 23, 2000, dtype=np.uint32)
        m[:4] = 0, 1, (1 << 23) - 1, 0x7FFF
        x = (np.uint32(e << 23) | m).view(np.float32)
        hi = _bf16(x)
        mid = _bf16(x - hi)
        lo = x - hi - mid
        assert np.isfinite(hi).all() and np.array_equal(_bf16(lo), lo)
        assert np.array_equal((hi.astype(np.float64) + mid) + lo, x.astype(np.float64))
