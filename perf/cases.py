"""What users have the contraction engine do, as measurable cases.

A case is one expression with its extents, executed once per pass through the public entry a program would use:
`Plan` on device tensors, `ExternalShard` for one GPU's share of a sharded contraction, `FusedPlan` for several terms
into one output, `sd_t_d2_fusion` for host arrays.  A program keeps its plan and its tensors from pass to pass, so both
are made in `prepare`.
"""
import importlib
import math
import re

import numpy as np
import torch

tc = importlib.import_module("cgo2019-ae_b200")
shard = importlib.import_module("cgo2019-ae_b200.shard")

# The terms of the CCSD(T) doubles contribution: operator, indices of the left and of the right input.
DOUBLES_TERMS = [("-=", "p7,p4,h1,h2", "p7,h3,p6,p5"), ("-=", "p7,p4,h2,h3", "p7,h1,p6,p5"), ("+=", "p7,p4,h1,h3", "p7,h2,p6,p5"),
                 ("+=", "p7,p5,h1,h2", "p7,h3,p6,p4"), ("+=", "p7,p5,h2,h3", "p7,h1,p6,p4"), ("-=", "p7,p5,h1,h3", "p7,h2,p6,p4"),
                 ("-=", "p7,p6,h1,h2", "p7,h3,p5,p4"), ("-=", "p7,p6,h2,h3", "p7,h1,p5,p4"), ("+=", "p7,p6,h1,h3", "p7,h2,p5,p4")]

# The families of expressions: "output | contraction | left | right".
SMALL = ["i,j,k|l|l,k,i|j,l", "a,b,c|d|d,c,a|b,d"]
TRANSFORM_3D = ["a,b,c|d|d,c,a|b,d", "a,c,b|d|c,d,a|d,b"]  # b is the short new index
TRANSFORM_4D = ["a,c,b,d|e|d,c,e,a|e,b", "a,b,c,d|e|d,e,c,a|b,e", "a,c,b,d|e|e,c,a,d|b,e"]
TRANSFORM_5D = ["a,d,b,c,e|f|e,f,d,a,c|b,f", "a,c,d,b,e|f|e,c,d,f,a|f,b", "a,b,c,d,e|f|e,f,c,a,d|b,f"]
ONE_INDEX_4D = ["a,b,c,d|e|a,e,b,d|e,c", "a,b,c,d|e|e,a|e,b,c,d", "a,b,c,d|e|e,b|a,e,c,d", "a,b,c,d|e|e,c|a,b,e,d"]
TWO_INDEX_4D = ["a,b,c,d|e,f|e,c,a,f|b,f,d,e", "a,b,c,d|e,f|a,e,b,f|d,f,c,e", "a,b,c,d|e,f|a,e,b,f|f,d,e,c", "a,b,c,d|e,f|a,e,c,f|b,f,d,e",
                "a,b,c,d|e,f|a,e,c,f|f,b,e,d", "a,b,c,d|e,f|a,e,d,f|b,f,c,e", "a,b,c,d|e,f|a,e,f,b|f,d,c,e", "a,b,c,d|e,f|e,a,f,b|f,d,e,c",
                "a,b,c,d|e,f|e,a,f,c|b,f,d,e", "a,b,c,d|e,f|e,a,f,d|f,b,e,c"]
LONG_SUM = ["a,b|c,d|c,a,d|d,c,b", "a,b|c,d|a,c,d|d,b,c"]
MATRIX = ["a,b|c|c,a|c,b", "a,b|c|a,c|c,b", "a,b|c|a,c|b,c"]
SINGLES_6D = ["a,b,c,i,j,k|l|l,a,i,j|b,c,k,l"]
TRIPLES_6D = ["a,b,c,d,e,f|g|d,e,g,a|g,f,b,c", "a,b,c,d,e,f|g|d,e,g,b|g,f,a,c", "a,b,c,d,e,f|g|d,e,g,c|g,f,a,b", "a,b,c,d,e,f|g|d,f,g,a|g,e,b,c",
              "a,b,c,d,e,f|g|d,f,g,b|g,e,a,c", "a,b,c,d,e,f|g|d,f,g,c|g,e,a,b", "a,b,c,d,e,f|g|e,f,g,a|g,d,b,c", "a,b,c,d,e,f|g|e,f,g,b|g,d,a,c",
              "a,b,c,d,e,f|g|e,f,g,c|g,d,a,b"]
SLAB_6D = "a,b,c,d,e,f|g|g,a,b,c|d,e,f,g"


def expression(form, op, extents):
    """The expression line of a form and the extents of its indices."""
    out, summed, left, right = form.split("|")
    sized = lambda idx: ",".join("%s,%d" % (i, extents[i]) for i in idx.split(","))
    return "C [%s] %s sum(%s) * A [%s] * B [%s];" % (sized(out), op, sized(summed), left, right)


def listed():
    every = lambda form, n: {i: n for part in form.split("|") for i in part.split(",")}
    return [
        # a small three-index contraction, as called inside an iteration over blocks: latency and launches count
        {"name": "small_3d_f64", "call": "plan", "dtype": "f64", "expr": expression(SMALL[0], "+=", {"i": 64, "j": 48, "k": 32, "l": 40})},
        # one step of an integral transformation: a large tensor read across its layout, one index replaced by a short one
        {"name": "transform_3d_f64", "call": "plan", "dtype": "f64",
         "expr": expression(TRANSFORM_3D[0], "+=", {"a": 312, "b": 24, "c": 296, "d": 312})},
        # the same on a four-index tensor with equal extents: ordinary size
        {"name": "one_index_4d_f64", "call": "plan", "dtype": "f64", "expr": expression(ONE_INDEX_4D[0], "+=", every(ONE_INDEX_4D[0], 96))},
        # orbital spaces of no round size, result overwritten
        {"name": "ragged_4d_f64", "call": "plan", "dtype": "f64",
         "expr": expression(ONE_INDEX_4D[0], "=", {"a": 61, "b": 59, "c": 67, "d": 53, "e": 71})},
        # ring and ladder terms of coupled cluster: two indices contracted, both inputs permuted
        {"name": "two_index_4d_f64", "call": "plan", "dtype": "f64", "expr": expression(TWO_INDEX_4D[0], "+=", every(TWO_INDEX_4D[0], 64))},
        # a small output from a long sum (density and Fock matrices from four-index quantities)
        {"name": "long_sum_f64", "call": "plan", "dtype": "f64",
         "expr": expression(LONG_SUM[0], "+=", {"a": 312, "b": 296, "c": 312, "d": 312})},
        # a triples term of coupled cluster on a tile of the orbital space, subtracted
        {"name": "triples_6d_f64", "call": "plan", "dtype": "f64",
         "expr": expression(TRIPLES_6D[0], "-=", {"a": 24, "b": 16, "c": 16, "d": 24, "e": 16, "f": 16, "g": 24})},
        # a triples-style term in single precision
        {"name": "triples_6d_f32", "call": "plan", "dtype": "f32", "expr": expression(SINGLES_6D[0], "+=", every(SINGLES_6D[0], 24))},
        # one GPU's share of a large output that is sharded over eight: 4 GB of output per pass, the largest
        {"name": "slab_6d_f64", "call": "shard", "dtype": "f64", "rank": 3, "world": 8, "expr": expression(SLAB_6D, "+=", every(SLAB_6D, 40))},
        # a matrix-shaped contraction in single precision, bound by arithmetic
        {"name": "matrix_f32", "call": "plan", "dtype": "f32", "expr": expression(MATRIX[0], "+=", {"a": 4096, "b": 4096, "c": 2048})},
        # all nine doubles terms of CCSD(T) accumulated into one tile of the triples
        {"name": "fused_doubles_f64", "call": "fused", "dtype": "f64", "h": "24,24,24", "p": "24,24,24", "p7": 24},
        # the drop-in entry on host arrays, as existing drivers call it (plain pageable memory)
        {"name": "host_4d_f64", "call": "host", "dtype": "f64", "expr": expression(ONE_INDEX_4D[0], "+=", every(ONE_INDEX_4D[0], 48))},
    ]


def _size(rng, lo, hi):
    """An extent, even over the logarithm; two in five are multiples of 8, as blocked codes choose them."""
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.4:
        n = (n + 4) // 8 * 8
    return min(max(n, lo), hi)


def draw(rng):
    family = rng.choice(["small", "transform", "transform", "one_index", "ragged", "two_index", "long_sum", "triples", "triples_f32",
                         "slab", "matrix", "fused", "host"])
    op = rng.choice(["+=", "+=", "-=", "="])
    dtype = "f64"

    def sized(form, lo, hi, short=None, odd=False):
        names = []
        for part in form.split("|"):
            names += [i for i in part.split(",") if i not in names]
        ext = {}
        for i in names:
            ext[i] = _size(rng, 8, 48) if i == short else _size(rng, lo, hi)
            if odd and ext[i] % 2 == 0:
                ext[i] -= 1
        return expression(form, op, ext)

    if family == "fused":
        h, p = [_size(rng, 10, 24) for _ in range(3)], [_size(rng, 10, 24) for _ in range(3)]
        return {"call": "fused", "dtype": "f64", "h": ",".join(map(str, h)), "p": ",".join(map(str, p)), "p7": _size(rng, 10, 24)}
    if family == "slab":
        rank = rng.randrange(8)
        return {"call": "shard", "dtype": "f64", "rank": rank, "world": 8, "expr": sized(SLAB_6D, 16, 40)}
    if family == "host":
        return {"call": "host", "dtype": "f64", "expr": sized(rng.choice(ONE_INDEX_4D), 16, 56)}
    if family == "small":
        dtype = rng.choice(["f64", "f64", "f32"])
        expr = sized(rng.choice(SMALL), 12, 96)
    elif family == "transform":
        forms, lo, hi = rng.choice([(TRANSFORM_3D, 64, 400), (TRANSFORM_4D, 24, 80), (TRANSFORM_5D, 16, 48)])
        expr = sized(rng.choice(forms), lo, hi, short="b")
    elif family == "one_index":
        expr = sized(rng.choice(ONE_INDEX_4D), 32, 96)
    elif family == "ragged":
        dtype = rng.choice(["f64", "f32"])
        expr = sized(rng.choice(ONE_INDEX_4D + TWO_INDEX_4D[:2]), 25, 73, odd=True)
    elif family == "two_index":
        expr = sized(rng.choice(TWO_INDEX_4D), 24, 64)
    elif family == "long_sum":
        expr = sized(rng.choice(LONG_SUM), 64, 312)
    elif family == "triples":
        expr = sized(rng.choice(TRIPLES_6D), 10, 26)
    elif family == "triples_f32":
        dtype = "f32"
        expr = sized(rng.choice(SINGLES_6D + TRIPLES_6D[6:]), 10, 26)
    else:
        dtype = rng.choice(["f32", "f64"])
        expr = sized(rng.choice(MATRIX), 256, 4096 if dtype == "f32" else 2048)
    return {"call": "plan", "dtype": dtype, "expr": expr}


def _fused_lines(case):
    h3, h2, h1 = (int(x) for x in case["h"].split(","))
    p6, p5, p4 = (int(x) for x in case["p"].split(","))
    out = "t3 [h3,%d,h2,%d,h1,%d,p6,%d,p5,%d,p4,%d]" % (h3, h2, h1, p6, p5, p4)
    return ["%s %s sum(p7,%d) * t2_%d [%s] * v2_%d [%s];" % (out, op, case["p7"], k, left, k, right)
            for k, (op, left, right) in enumerate(DOUBLES_TERMS)]


def _counts(expr):
    """Elements of the output, the left and the right input; number of multiply-adds; the operator."""
    p = tc.parse(expr)
    ext = dict(zip(p["out_idx"] + p["sum_idx"], p["out_ext"] + p["sum_ext"]))
    counts = [math.prod(ext[i] for i in p[key]) for key in ("out_idx", "left_idx", "right_idx")]
    return counts, math.prod(ext.values()), p["op"]


def _slowest(expr):
    """The output's slowest index: cut along it, a rank's share of the output is one contiguous block."""
    return tc.parse(expr)["out_idx"][-1]


def _maker(case, seed):
    """A function that makes the next input of so many elements, on the GPU."""
    dtype = torch.float64 if case["dtype"] == "f64" else torch.float32
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return lambda n: torch.empty(n, dtype=dtype, device="cuda").uniform_(-1.0, 1.0, generator=gen)


def prepare(case, seed):
    code = tc.F64 if case["dtype"] == "f64" else tc.F32
    make = _maker(case, seed)
    if case["call"] == "fused":
        lines = _fused_lines(case)
        counts = [_counts(line)[0] for line in lines]
        return {"call": "fused", "plan": tc.FusedPlan(lines).commit(), "C": make(counts[0][0]),
                "A": [make(c[1]) for c in counts], "B": [make(c[2]) for c in counts]}
    if case["call"] == "shard":
        part = shard.ExternalShard(case["expr"], code, rank=case["rank"], world=case["world"], index=_slowest(case["expr"]))
        if part.plan is not None:
            part.plan.commit()
        counts, _, _ = _counts(case["expr"])
        return {"call": "shard", "plan": part, "C": make(part.geom.c_slab_elems), "A": make(counts[1]), "B": make(counts[2])}
    counts, _, _ = _counts(case["expr"])
    state = {"call": case["call"], "C": make(counts[0]), "A": make(counts[1]), "B": make(counts[2])}
    if case["call"] == "host":
        p = tc.parse(case["expr"])
        state.update({k: state[k].cpu().numpy().copy() for k in "CAB"}, expr=case["expr"], sizes=p["out_ext"] + p["sum_ext"], code=code)
    else:
        state["plan"] = tc.Plan(case["expr"], code).commit()
    return state


def run(state):
    if state["call"] == "host":
        tc.sd_t_d2_fusion(state["expr"], state["sizes"], state["C"], state["A"], state["B"], state["code"])
    elif state["call"] == "shard":
        state["plan"].execute(state["C"], state["A"], state["B"], c_is_slab=True)
    else:
        state["plan"].execute(state["C"], state["A"], state["B"])
    return state["C"]


def work(case):
    es = 8 if case["dtype"] == "f64" else 4
    if case["call"] == "fused":
        each = [_counts(line) for line in _fused_lines(case)]
        return {"bytes": es * (2 * each[0][0][0] + sum(c[1] + c[2] for c, _, _ in each)), "flops": 2 * sum(n for _, n, _ in each)}
    if case["call"] == "shard":
        geom = shard.ShardGeometry(case["expr"], _slowest(case["expr"]), case["rank"], case["world"])
        share = geom.count / geom.full_extents[geom.index]
        (c, a, b), n, op = _counts(case["expr"])
        cut = [share if geom.index in geom.parsed[key] else 1.0 for key in ("left_idx", "right_idx")]
        return {"bytes": es * ((1 if op == "=" else 2) * c * share + a * cut[0] + b * cut[1]), "flops": 2 * n * share}
    (c, a, b), n, op = _counts(case["expr"])
    return {"bytes": es * ((1 if op == "=" else 2) * c + a + b), "flops": 2 * n}


def tolerance(case):
    """Four times what was measured between this path and the same sums in another order and in 64 bits.

    fp64: up to 2.7e-15 (2-norm) and 2.2e-14 (largest) for sums of 97 000 products.  fp32: 1.7e-7 and 1.5e-6 for 24
    products, 3.6e-6 and 1.3e-5 from 512 on, where accumulation chains end."""
    if case["dtype"] == "f64":
        return {"rel": 1e-14, "max": 1e-13}
    p = tc.parse(case["expr"])
    chain = min(math.prod(p["sum_ext"]), 512)
    return {"rel": 7e-7 + 2.8e-8 * chain, "max": 6e-6 + 9e-8 * chain}


def _taken_apart(expr):
    """(indices of the output, of the left and of the right input; extents; operator) of an expression line."""
    found = re.fullmatch(r"\s*\w+ \[(.*?)\] (\S+) sum\((.*?)\) \* \w+ \[(.*?)\] \* \w+ \[(.*?)\];", expr)
    sized = lambda text: list(zip(text.split(",")[0::2], map(int, text.split(",")[1::2])))
    out, summed = sized(found[1]), sized(found[3])
    return [[i for i, _ in out], found[4].split(","), found[5].split(",")], dict(out + summed), found[2]


def _added(expr, flat_c, flat_a, flat_b, only=None):
    """C op A * B in 64 bits on flat tensors whose first index is the fastest; `only` = (index, first, last) keeps those values of an index."""
    names, ext, op = _taken_apart(expr)
    letter = {n: chr(97 + k) for k, n in enumerate(ext)}
    a, b = (t.double().view([ext[i] for i in reversed(idx)]) for t, idx in ((flat_a, names[1]), (flat_b, names[2])))
    if only:
        index, first, last = only
        a, b = (t.narrow(len(idx) - 1 - idx.index(index), first, last - first) if index in idx else t for t, idx in ((a, names[1]), (b, names[2])))
    text = ["".join(letter[i] for i in reversed(idx)) for idx in names]
    product = torch.einsum("%s,%s->%s" % (text[1], text[2], text[0]), a, b).reshape(-1)
    if op == "=":
        return product
    return product.neg_().add_(flat_c) if op == "-=" else product.add_(flat_c)


def exact(case, seed):
    make = _maker(case, seed)
    if case["call"] == "fused":
        lines = _fused_lines(case)
        taken = [_taken_apart(line) for line in lines]
        counts = [[math.prod(ext[i] for i in idx) for idx in names] for names, ext, _ in taken]
        c = make(counts[0][0])
        lefts, rights = [make(n[1]) for n in counts], [make(n[2]) for n in counts]
        for line, a, b in zip(lines, lefts, rights):
            c = _added(line, c, a, b)
        return c
    names, ext, _ = _taken_apart(case["expr"])
    counts, only = [math.prod(ext[i] for i in idx) for idx in names], None
    if case["call"] == "shard":
        # the first ranks get one value more where the extent does not divide
        cut, (each, more) = names[0][-1], divmod(ext[names[0][-1]], case["world"])
        first = case["rank"] * each + min(case["rank"], more)
        only = (cut, first, first + each + (case["rank"] < more))
        if only[1] == only[2]:
            return None
        counts[0] = counts[0] // ext[cut] * (only[2] - only[1])
    result = _added(case["expr"], *(make(n) for n in counts), only=only)
    return result.cpu().numpy() if case["call"] == "host" else result
