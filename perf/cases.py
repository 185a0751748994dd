"""The work that programs give this framework, as cases that can be timed.

``listed()`` names twelve cases, ``draw(rng)`` gives further ones of the same
ranges; ``prepare`` makes what a program holds before the call (compiled
contraction, tensors, bound group), ``run`` is one call through the public
entry points, ``exact`` the same result from torch in 64 bits.

Kinds:

* ``call``  -- ``tccg_b200.compile(...)`` once, then ``c(A, B, C)`` per pass.
* ``train`` -- ``GettFunction.apply`` and the gradients of A and B.
* ``batch`` -- a ``Group`` of mixed contractions, bound and captured once,
  replayed per pass.

Tensors are column-major (the first index has stride one): the buffer of
``A[i,m,a]`` is a contiguous tensor of shape (a, m, i).
"""
import torch

import tccg_b200
from tccg_b200.grouped import Group
from tccg_b200.workloads import batched_workload

# The five families of contractions: C, A and B indices. "small" is a
# three-index call of a few microseconds; the others are the repository's
# benchmark configurations 1 (plain), 2 (bandwidth bound), 3 (compute bound)
# and 4 (differentiation).
FAMILIES = {
    "small": ("a,b,i", "i,m,a", "m,b"),
    "plain": ("a,b,i,j", "i,m,a", "m,j,b"),
    "bandwidth": ("a,b,c,d", "a,e,b", "e,d,c"),
    "compute": ("a,b,c,i,j,k", "a,m,b,n,c", "m,i,n,j,k"),
    "gradient": ("i,x,y,j", "k,i,l,j", "l,y,k,x"),
}


def _case(name, kind, family, precision, dtype="f32", beta=0.0, **sizes):
    case = {"name": name, "kind": kind, "family": family, "precision": precision, "dtype": dtype,
            "beta": beta}
    case.update({"n_" + label: size for label, size in sizes.items()})
    return case


def listed():
    return [
        # the smallest call of an application loop: only latency and launches count
        _case("small_fp32", "call", "small", "fp32", a=7, b=9, i=5, m=11),
        # configuration 1: the plain contraction, all extents 48
        _case("plain48_fp32", "call", "plain", "fp32", a=48, b=48, i=48, j=48, m=48),
        # the same with uneven, odd extents on the tensor cores
        _case("plain_odd_bf16x3", "call", "plain", "bf16x3", a=47, b=53, i=61, j=37, m=51),
        # configuration 2: short K, C read and written (beta = 1), FP32
        _case("bandwidth96_fp32", "call", "bandwidth", "fp32", beta=1.0, a=96, b=96, c=96, d=96, e=16),
        # configuration 2 with BF16 operands; uneven extents, so that C's rows are ragged
        _case("bandwidth_odd_bf16", "call", "bandwidth", "bf16", dtype="bf16", beta=1.0, a=90, b=77,
              c=85, d=101, e=19),
        # configuration 3, the headline: M = N = 32768, K = 4096, split-BF16x3
        _case("compute32_bf16x3", "call", "compute", "bf16x3", a=32, b=32, c=32, i=32, j=32, k=32, m=64,
              n=64),
        # the same contraction in plain FP32 (M = N = 13824)
        _case("compute24_fp32", "call", "compute", "fp32", a=24, b=24, c=24, i=24, j=24, k=24, m=64, n=64),
        # and in FP64, with uneven extents (M = 3825, N = 4056, K = 3080)
        _case("compute_odd_fp64", "call", "compute", "fp64", dtype="f64", a=17, b=15, c=15, i=24, j=13,
              k=13, m=56, n=55),
        # configuration 4: forward, dA and dB of a training step, FP32 and BF16 operands
        _case("train64_fp32", "train", "gradient", "fp32", i=64, j=64, x=64, y=64, k=32, l=32),
        _case("train64_bf16", "train", "gradient", "bf16", dtype="bf16", i=64, j=64, x=64, y=64, k=32, l=32),
        # configuration 5: many mixed contractions (2 to 6 indices, extents
        # 8-128, 1e6-1e10 FLOP each) as one captured grouped launch
        {"name": "batch64_bf16x3", "kind": "batch", "precision": "bf16x3", "count": 64, "workload": 0},
        {"name": "batch48_fp32", "kind": "batch", "precision": "fp32", "count": 48, "workload": 5},
    ]


def _between(rng, lo, hi):
    """An extent of [lo, hi], spread over its logarithm."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["small", "plain", "bandwidth", "compute", "compute", "gradient", "batch", "batch"])
    if kind == "batch":
        return {"kind": "batch", "precision": rng.choice(["bf16x3", "fp32"]),
                "count": rng.randint(16, 64), "workload": rng.randrange(1, 1 << 20)}
    if kind == "small":
        ranges, precision = {l: (3, 16) for l in "abim"}, "fp32"
    elif kind == "plain":
        ranges, precision = {l: (24, 64) for l in "abijm"}, rng.choice(["fp32", "bf16x3"])
    elif kind == "bandwidth":
        ranges, precision = {l: (64, 104) for l in "abcd"}, rng.choice(["fp32", "bf16"])
        ranges["e"] = (10, 24)
    elif kind == "compute":
        precision = rng.choice(["bf16x3", "fp32", "fp64"])
        top = {"bf16x3": 30, "fp32": 22, "fp64": 16}[precision]
        ranges = {l: (top // 2, top) for l in "abcijk"}
        ranges.update(m=(32, 64), n=(32, 64))
    else:
        ranges, precision = {l: (32, 64) for l in "ijxy"}, rng.choice(["fp32", "bf16"])
        ranges.update(k=(16, 32), l=(16, 32))
    dtype = {"fp64": "f64", "bf16": "bf16"}.get(precision, "f32")
    case = _case("", "train" if kind == "gradient" else "call", kind, precision, dtype,
                 1.0 if kind == "bandwidth" else 0.0,
                 **{l: _between(rng, *ranges[l]) for l in sorted(ranges)})
    del case["name"]
    return case


def _contractions(case):
    if case["kind"] == "batch":
        return batched_workload(case["count"], seed=case["workload"])
    c, a, b = (t.split(",") for t in FAMILIES[case["family"]])
    sizes = {k[2:]: v for k, v in case.items() if k.startswith("n_")}
    return [tccg_b200.make_contraction(c, a, b, sizes, 1.0, case["beta"])]


_DTYPES = {"f32": torch.float32, "f64": torch.float64, "bf16": torch.bfloat16}


def _inputs(case, cons, seed):
    """(A, B, C) of each contraction, N(0, 1); C is the preloaded result where
    beta is not 0 (or the upstream gradient of a training step) and else None."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = _DTYPES[case.get("dtype", "f32")]
    out = torch.float64 if dtype == torch.float64 else torch.float32
    made = []
    for con in cons:
        def normal(t, dt):
            shape = tuple(reversed([i.size for i in t.indices]))
            wide = torch.randn(shape, generator=gen, device="cuda",
                               dtype=torch.float64 if dt == torch.float64 else torch.float32)
            return wide.to(dt)
        a, b = normal(con.A0, dtype), normal(con.B0, dtype)
        c = normal(con.C0, out) if case["kind"] == "train" or case.get("beta") else None
        made.append((a, b, c))
    return made


def prepare(case, seed):
    cons = _contractions(case)
    made = _inputs(case, cons, seed)
    if case["kind"] == "batch":
        a, b = [m[0] for m in made], [m[1] for m in made]
        c = [torch.empty(con.C0.num_elements(), device="cuda") for con in cons]
        group = Group(cons, precision=case["precision"])
        group.bind(a, b, c)
        group.capture()
        return {"case": case, "group": group, "c": c}
    a, b, c = made[0]
    if case["kind"] == "train":
        return {"case": case, "con": cons[0], "a": a.requires_grad_(), "b": b.requires_grad_(), "dc": c}
    call = tccg_b200.compile(cons[0], float_type="d" if case["precision"] == "fp64" else "s",
                             precision=case["precision"], dtype=case["dtype"])
    if c is None:
        c = torch.empty(tuple(reversed([i.size for i in cons[0].C0.indices])), device="cuda",
                        dtype=torch.float64 if case["precision"] == "fp64" else torch.float32)
    return {"case": case, "call": call, "a": a, "b": b, "c": c}


def run(state):
    kind = state["case"]["kind"]
    if kind == "call":
        return state["call"](state["a"], state["b"], state["c"])
    if kind == "train":
        c = tccg_b200.GettFunction.apply(state["a"], state["b"], state["con"], state["case"]["precision"])
        da, db = torch.autograd.grad(c, (state["a"], state["b"]), state["dc"])
        return c, da, db
    state["group"].replay()
    return state["c"]


def work(case):
    """Operands read and results written once; two operations per multiply-add
    of the contraction (three contractions in a training step)."""
    wide = {"f32": 4, "f64": 8, "bf16": 2}[case.get("dtype", "f32")]
    out = 8 if wide == 8 else 4
    moved = flops = 0.0
    for con in _contractions(case):
        a, b, c = (t.num_elements() for t in (con.A0, con.B0, con.C0))
        moved += wide * (a + b) + out * c * (2 if case.get("beta") else 1)
        flops += con.flop_count(0.0)
        if case["kind"] == "train":  # dC read, the gradients written in the operands' type
            moved += out * c + wide * (a + b)
            flops += 2 * con.flop_count(0.0)
    return {"bytes": moved, "flops": flops}


def _product(into, left, right, tensors):
    def labels(t):
        return "".join(reversed([i.label for i in t.indices]))
    return torch.einsum("%s,%s->%s" % (labels(left), labels(right), labels(into)), *tensors)


def exact(case, seed):
    cons = _contractions(case)
    results = []
    for con, (a, b, c) in zip(cons, _inputs(case, cons, seed)):
        a, b = a.double(), b.double()
        product = _product(con.C0, con.A0, con.B0, (a, b))
        if case["kind"] == "train":
            return (product, _product(con.A0, con.C0, con.B0, (c.double(), b)),
                    _product(con.B0, con.A0, con.C0, (a, c.double())))
        if case["kind"] == "call":
            return product if c is None else product + c.double()
        results.append(product.reshape(-1))
    return results
