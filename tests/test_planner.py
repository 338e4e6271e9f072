"""Host-side planner (no GPU): index classes, fusion, loaders, tiles, costs, errors."""
import pytest

from conftest import CONFIGS


def _plan(pkg, expr, dtype="float64", **kw):
    return pkg.Plan(expr, pkg.F64 if dtype == "float64" else pkg.F32, **kw)


def test_algorithmic_costs_of_the_benchmark_configurations(pkg):
    # flops = 2 * prod(extents); bytes = elemsize * (2|C| + |A| + |B|)
    want = [(7864320, 2243584), (16307453952, 2038505472), (137438953472, 536870912),
            (9172942848, 1531478016), (327680000000, 65576960000)]
    for (expr, dt, _), (fl, by) in zip(CONFIGS, want):
        f, b = _plan(pkg, expr, dt).cost()
        assert (f, b) == (fl, by)


def test_index_classes_and_fusion(pkg):
    d = [_plan(pkg, e, dt).describe() for e, dt, _ in CONFIGS]
    # cfg1: M = {i,k} (left operand), N = {j}, K = {l}
    assert [x["extent"] for x in d[0]["M"]] == [64, 32] and [x["extent"] for x in d[0]["N"]] == [48]
    assert d[0]["Kflat"] == 40 and not d[0]["swapped"]
    # cfg2: nothing fuses (b,d adjacent in A but not in C)
    assert [x["extent"] for x in d[1]["M"]] == [96, 96, 96] and d[1]["Nflat"] == 96
    # cfg3: two contraction indices flatten to 4096
    assert d[2]["Mflat"] == d[2]["Nflat"] == d[2]["Kflat"] == 4096
    # cfg4: (i,j) and (b,c) fuse: adjacent in the output and in their operand
    assert [x["extent"] for x in d[3]["M"]] == [24, 576] and [x["extent"] for x in d[3]["N"]] == [576, 24]
    # cfg5: becomes a plain 64000 x 64000 x 40 product
    assert [x["extent"] for x in d[4]["M"]] == [64000] and [x["extent"] for x in d[4]["N"]] == [64000]
    assert d[4]["M"][0]["s_in"] == 40 and d[4]["M"][0]["s_out"] == 1


def test_operands_swap_when_output_fastest_index_is_in_the_right_operand(pkg):
    d = _plan(pkg, "C [a,8,b,8] += sum(c,8) * A [c,b] * B [a,c];").describe()
    assert d["swapped"] and d["M"][0]["s_out"] == 1 and d["vec_c"] == 4


def test_loader_and_vector_choices(pkg):
    d2 = _plan(pkg, CONFIGS[1][0]).describe()
    assert d2["vec_x"] and not d2["vec_y"] and d2["lanes_k_y"] == 4 and d2["vec_c"] == 4
    d4 = _plan(pkg, CONFIGS[3][0], "float32").describe()
    assert not d4["vec_x"] and d4["lanes_k_x"] == 8 and d4["vec_y"] and d4["vec_c"] == 4
    odd = _plan(pkg, "C [a,7,b,5] += sum(c,3) * A [a,c] * B [c,b];").describe()
    assert not odd["vec_x"] and odd["vec_c"] == 1
    even = _plan(pkg, "C [a,6,b,5] += sum(c,3) * A [a,c] * B [c,b];").describe()
    assert even["vec_x"] and even["vec_c"] == 2


def test_tile_choices(pkg):
    d = [_plan(pkg, e, dt).describe() for e, dt, _ in CONFIGS]
    # fp64 with enough tiles: the persistent warp-specialised kernel (variant 2)
    assert d[1]["kernel"] == "dmma_ws_64x96" and d[1]["tiles"] == [13824, 1]   # N = 96 is exactly one tile wide
    assert d[2]["kernel"] == "dmma_ws_128x64" and d[2]["tiles"] == [32, 64]
    # output-bound fp64 (K = 40): the kernel that keeps the output tile resident in shared memory
    assert d[4]["kernel"] == "dmma_wc_128x64" and d[4]["tiles"] == [500, 1000] and d[4]["tma_ct"] and d[4]["mblock_w"] == 32
    longer = _plan(pkg, CONFIGS[4][0].replace("g,40", "g,96")).describe()
    assert longer["kernel"].startswith("dmma_w") and longer["estimate_us"] > 2 * d[4]["estimate_us"]   # pipe-bound: time follows K
    # a skinny right operand (one external index of 24): the 32-wide tile wastes a quarter of its columns, not five eighths
    skinny = _plan(pkg, "t3 [a,312,b,24,c,296] += sum(d,312) * t2 [d,c,a] * v2 [b,d];").describe()
    assert skinny["kernel"] == "dmma_ws_128x32" and skinny["tiles"] == [722, 1] and skinny["estimate_us"] > 0
    # fp32: 96 rows = 4 whole runs of the 24-long fastest output index; (a, bc) blocks leave as bulk chunks
    # (default: the tcgen05 form of the three-TF32 product as the persistent kernel; one CTA per tile or the mma.sync
    # form on request or for small problems)
    assert d[3]["math"] == "tf32x3_tcgen05" and d[3]["kernel"] == "tf32wt_96x128" and d[3]["ksplit"] == 1
    per_tile = _plan(pkg, CONFIGS[3][0], "float32", path=pkg.PATH_TCGEN05, tile=(96, 128), variant=1).describe()
    assert per_tile["kernel"] == "tf32tc_96x128"
    sync = _plan(pkg, CONFIGS[3][0], "float32", path=pkg.PATH_3XTF32).describe()
    assert sync["math"] == "tf32x3" and sync["kernel"] == "tf32_96x128"
    # a 96-wide N leaves a quarter of a 128-wide tcgen05 tile empty and every tile ragged: mma.sync form
    n96 = _plan(pkg, CONFIGS[1][0], "float32").describe()
    assert n96["math"] == "tf32x3" and n96["kernel"] == "tf32_96x128"
    ffma = _plan(pkg, CONFIGS[3][0], "float32", path=pkg.PATH_FFMA).describe()
    assert ffma["math"] == "ffma" and ffma["kernel"] == "ffma_96x128"
    assert d[3]["epi_run"] == 24 and d[3]["epi_n_span"] == 576
    assert d[0]["kernel"] == "dmma_64x64_w4"                                    # tiny problem: one CTA per tile
    # operands whose fastest index is contracted are staged contraction-major with 16-byte copies
    assert d[4]["kvec_x"] and d[4]["vec_y"] and not d[4]["vec_x"]
    assert d[2]["kvec_x"] and d[2]["vec_y"]
    # forcing a persistent kernel disables the K split
    forced = _plan(pkg, "C [a,33,b,17] += sum(c,1000,d,9) * A [a,c,d] * B [d,b,c];", tile=(128, 64), variant=3).describe()
    assert forced["ksplit"] == 1 and forced["kernel"] == "dmma_ws_128x64"


def test_output_tensor_boxes(pkg):
    """Which outputs the persistent fp64 kernel may write as tiled TMA boxes (per warp batch / per tile)."""
    d = [_plan(pkg, e, dt).describe() for e, dt, _ in CONFIGS]
    # cfg2: (a, b) are contiguous in C although not in A: runs of 9216 hold the 64-row tiles; N = c alone
    assert d[1]["tma_c"] and d[1]["tma_ct"]
    # cfg5: M and N both fuse into one dimension
    assert d[4]["tma_c"] and d[4]["tma_ct"]
    # cfg3: the fastest M dimension (64) is shorter than the 128-row tile
    assert not d[2]["tma_c"] and not d[2]["tma_ct"]
    kw = dict(tile=(64, 96), variant=3)
    # N = (b: 32, d: 2): a batch of 16 rows stays inside b, a 96-row tile does not
    e = _plan(pkg, "C [a,128,b,32,c,3,d,2] += sum(e,24) * A [e,a,c] * B [b,d,e];", **kw).describe()
    assert e["tma_c"] and not e["tma_ct"]
    # N's fastest dimension 24 is not a multiple of 16 and N has a second dimension
    e = _plan(pkg, "C [a,128,b,24,c,3,d,4] += sum(e,16) * A [e,a,c] * B [b,d,e];", **kw).describe()
    assert not e["tma_c"]
    # ... but (b, c) contiguous in C count as one dimension of 96 whatever their order in B
    e = _plan(pkg, "C [a,128,b,24,c,4] += sum(e,16) * A [e,a] * B [b,e,c];", **kw).describe()
    assert e["tma_c"] and e["tma_ct"]
    # odd extent of the only N dimension: n cannot split into (parity, n / 2)
    e = _plan(pkg, "C [a,128,b,33] += sum(e,16) * A [e,a] * B [e,b];", **kw).describe()
    assert not e["tma_c"]
    # fp32 and the one-CTA-per-tile kernels never use them
    assert not d[3]["tma_c"] and not d[0]["tma_c"]


def test_k_split_plans(pkg):
    p = _plan(pkg, "C [a,33,b,17] += sum(c,1000,d,9) * A [a,c,d] * B [d,b,c];")
    d = p.describe()
    assert d["ksplit"] > 1 and d["launches"] == 2 and d["workspace_bytes"] == d["ksplit"] * 64 * 64 * 8
    assert d["k_chunk"] % 16 == 0 and d["k_chunk"] * d["ksplit"] >= 9000
    assert _plan(pkg, "C [a,33,b,17] += sum(c,1000,d,9) * A [a,c,d] * B [d,b,c];", split_k=1).describe()["ksplit"] == 1
    assert _plan(pkg, CONFIGS[1][0]).describe()["ksplit"] == 1


def test_extent_override_and_errors(pkg):
    p = _plan(pkg, "t3 [a,16,b,16,c,16] += sum(d,16) * t2 [d,c,a] * v2 [b,d];")
    p.set_extents({"a": 312, "b": 24, "c": 296, "d": 312})
    assert p.cost()[0] == 2.0 * 312 * 24 * 296 * 312
    with pytest.raises(pkg.TcError) as e:
        p.set_extents({"z": 3})
    assert e.value.status == 2
    with pytest.raises(pkg.TcError) as e:
        p.set_extents({"a": 0})
    assert e.value.status == 4
    with pytest.raises(pkg.TcError) as e:
        _plan(pkg, CONFIGS[0][0], tile=(48, 48)).describe()
    assert e.value.status == 3
    with pytest.raises(pkg.TcError) as e:
        _plan(pkg, CONFIGS[0][0], path=pkg.PATH_FFMA).describe()
    assert e.value.status == 2
    with pytest.raises(pkg.TcError) as e:
        _plan(pkg, CONFIGS[3][0], "float32", path=pkg.PATH_DMMA).describe()
    assert e.value.status == 2


def test_strided_views(pkg):
    p = _plan(pkg, "C [a,4,b,3] += sum(c,5) * A [c,a] * B [b,c];")
    p.set_strides(pkg.TENSOR_OUT, [1, 4]).set_strides(pkg.TENSOR_RIGHT, [1, 7])
    d = p.describe()
    assert d["N"][0]["s_in"] == 1 and d["N"][0]["s_out"] == 4
    with pytest.raises(pkg.TcError) as e:
        _plan(pkg, "C [a,4,b,3] += sum(c,5) * A [c,a] * B [b,c];").set_strides(pkg.TENSOR_OUT, [1, 2]).describe()
    assert e.value.status == 4  # output elements would alias
    with pytest.raises(pkg.TcError) as e:
        p.set_strides(pkg.TENSOR_OUT, [1])
    assert e.value.status == 2


def test_sizes_beyond_32_bit(pkg):
    # 4.096e9 output elements: offsets are 64-bit (the reference's int arithmetic cannot address this)
    d = _plan(pkg, CONFIGS[4][0]).describe()
    assert d["tiles"][0] * d["tiles"][1] == 500 * 1000
    assert d["N"][0]["s_out"] == 64000


def test_index_classes_reproduce_the_contraction(pkg, orc):
    """What the kernels are told -- the digits of M, N and K with their strides, the operand swap -- evaluated in numpy
    gives the checker's result for random expressions: the classes cover every element once, fusion, splitting and
    re-ordering of digits included."""
    import random

    import numpy as np

    from test_parser import _random_expr

    def flat(dims, key):
        # flattened index f = sum digit_i * prod(extent_j, j < i)  ->  offset
        off = np.zeros(1, dtype=np.int64)
        for d in dims:
            off = (np.arange(d["extent"], dtype=np.int64)[:, None] * d[key] + off[None, :]).reshape(-1)
        return off

    rng = random.Random(99)
    seen_split = 0
    for n in range(250):
        expr = _random_expr(rng, max_out=6, max_sum=3)
        p = orc.parse(expr)
        # extents from a set that triggers vector, fusion and digit-splitting rules
        ext = {i: rng.choice([1, 2, 3, 4, 4, 5, 8, 8, 12, 16]) for i in p["out_idx"] + p["sum_idx"]}
        expr = orc.with_extents(expr, ext)
        if np.prod([float(v) for v in ext.values()]) > 3e6:
            continue
        c0, a, b = orc.make_inputs(expr, n, "float64")
        want = orc.contract(expr, c0.copy(), a, b)
        d = _plan(pkg, expr).describe()
        x, y = (b, a) if d["swapped"] else (a, b)
        om_x, om_c = flat(d["M"], "s_in"), flat(d["M"], "s_out")
        on_y, on_c = flat(d["N"], "s_in"), flat(d["N"], "s_out")
        ok_x, ok_y = flat(d["K"], "s_in"), flat(d["K"], "s_out")
        assert len(om_x) == d["Mflat"] and len(on_y) == d["Nflat"] and len(ok_x) == d["Kflat"]
        prod = x[om_x[:, None] + ok_x[None, :]] @ y[on_y[:, None] + ok_y[None, :]].T
        where = (om_c[:, None] + on_c[None, :]).reshape(-1)
        assert len(np.unique(where)) == c0.size == where.size, expr      # every output element exactly once
        got = c0.copy()
        op = p["op"]
        got[where] = prod.reshape(-1) if op == "=" else got[where] + (prod.reshape(-1) if op == "+=" else -prod.reshape(-1))
        assert orc.rel_error(got, want) <= 1e-12, (expr, d["M"], d["N"], d["K"])
        seen_split += any(dd["extent"] == 4 and dd["s_out"] != 1 for dd in d["M"][1:2])
    assert seen_split > 0  # the digit re-ordering was exercised


def test_few_tiles_and_a_long_contraction(pkg):
    """fp64 problems that cannot fill the GPU with tiles: the persistent kernel with K slices where its tiles do not
    pad much more than small ones (or the small kernel would gather both operands by element), else one CTA per tile."""
    both_gathered = _plan(pkg, "t3 [a,312,b,296] += sum(c,312,d,312) * t2 [c,a,d] * v2 [d,c,b];").describe()
    assert both_gathered["kernel"] == "dmma_ws_128x64" and both_gathered["ksplit"] > 1 and both_gathered["tiles"] == [3, 5]
    assert both_gathered["workspace_bytes"] == both_gathered["ksplit"] * 15 * 128 * 64 * 8
    assert both_gathered["k_chunk"] % 16 == 0 and both_gathered["k_chunk"] >= 256
    one_vector = _plan(pkg, "t3 [a,312,b,296] += sum(c,296,d,312) * t2 [a,c,d] * v2 [d,b,c];").describe()
    assert one_vector["kernel"] == "dmma_64x64_w4" and one_vector["ksplit"] > 1
    narrow = _plan(pkg, "t3 [a,72,b,72,c,72] += sum(d,72,e,72) * t2 [a,d,e,c] * v2 [e,b,d];").describe()
    assert narrow["kernel"] == "dmma_ws_128x64" and narrow["ksplit"] > 1 and narrow["tiles"] == [41, 2]
    short = _plan(pkg, "C [a,312,b,296] += sum(c,40) * A [c,a] * B [c,b];").describe()
    assert short["kernel"] == "dmma_64x64_w4" and short["ksplit"] == 1
    # on request the persistent kernel slices K whatever the shape
    forced = _plan(pkg, "C [a,200,b,70] -= sum(c,1003) * A [c,a] * B [b,c];", tile=(128, 64), variant=3, split_k=5).describe()
    assert forced["kernel"] == "dmma_ws_128x64" and forced["ksplit"] == 5


def test_no_default_fp32_plan_runs_a_tensor_core_chain_longer_than_512(pkg):
    """fp32 on the tensor cores accumulates with truncation, so the planner bounds every accumulation chain:
    K slices where their scratch fits 1 GiB, sequential passes into C beyond that."""
    import random
    rng = random.Random(9)
    seen = set()
    for n in range(300):
        m = rng.choice([64, 96, 500, 4096, 20000, 60000])
        nn = rng.choice([64, 128, 1000, 4096, 30000])
        k = rng.choice([16, 500, 512, 513, 1024, 4100, 8192, 50000])
        expr = "C [a,%d,b,%d] %s sum(c,%d) * A [c,a] * B [c,b];" % (m, nn, rng.choice(["+=", "-=", "="]), k)
        for path in (pkg.PATH_AUTO, pkg.PATH_TCGEN05, pkg.PATH_3XTF32):
            d = _plan(pkg, expr, "float32", path=path).describe()
            assert d["math"].startswith("tf32x3")
            assert d["chain"] <= 512, (expr, d)
            assert d["passes"] == 1 or d["ksplit"] == 1
            assert d["workspace_bytes"] <= (1 << 30) + 128 * 128 * 4 * d["ksplit"] * 148, (expr, d)
            seen.add("passes" if d["passes"] > 1 else "slices" if d["ksplit"] > 1 else "single")
    assert seen == {"passes", "slices", "single"}
    # the caller may override the rule explicitly, and FFMA never needs it
    assert _plan(pkg, "C [a,4096,b,8192] += sum(c,8192) * A [c,a] * B [c,b];", "float32", split_k=1).describe()["chain"] == 8192
    assert _plan(pkg, "C [a,4096,b,8192] += sum(c,8192) * A [c,a] * B [c,b];", "float32", path=pkg.PATH_FFMA).describe()["passes"] == 1


def test_operands_that_are_matrices_are_marked_as_boxes(pkg):
    """An operand is a TMA box tensor when it is a plain matrix: contraction index fastest with the externals
    contiguous among themselves (tma_x / tma_y, fp64 and fp32), or the external class one contiguous run with the
    contraction index at a constant pitch (tma_xe / tma_ye, fp32).  Rows must be 16 bytes apart or more."""
    def flags(expr, dt):
        d = pkg.Plan(expr, dt).describe()
        return tuple(bool(d[k]) for k in ("tma_x", "tma_y", "tma_xe", "tma_ye"))
    assert flags("C [a,512,b,512] += sum(c,256) * A [c,a] * B [c,b];", pkg.F32) == (True, True, False, False)
    assert flags("C [a,512,b,512] += sum(c,256) * A [a,c] * B [b,c];", pkg.F32) == (False, False, True, True)
    assert flags("C [a,512,b,512] += sum(c,256) * A [c,a] * B [b,c];", pkg.F32) == (True, False, False, True)
    assert flags("C [a,512,b,512] += sum(c,256) * A [c,a] * B [b,c];", pkg.F64) == (True, False, False, False)
    # rows of 250 floats are not 16 bytes apart; 250 doubles are
    assert flags("C [a,512,b,512] += sum(c,250) * A [c,a] * B [c,b];", pkg.F32) == (False, False, False, False)
    assert flags("C [a,512,b,512] += sum(c,250) * A [c,a] * B [c,b];", pkg.F64) == (True, True, False, False)
    # fused externals stay a box while they are contiguous among themselves; a permuted pair is not
    assert flags("C [a,64,b,8,c,512] += sum(d,64) * A [d,a,b] * B [d,c];", pkg.F32)[0]
    assert not flags("C [a,64,b,8,c,512] += sum(d,64) * A [d,b,a] * B [d,c];", pkg.F32)[0]
    assert flags("C [a,64,b,8,c,512] += sum(d,64) * A [a,b,d] * B [d,c];", pkg.F32)[2]


def _wc_layouts():
    """(expression, what it is for): outputs whose cut tiles take every form."""
    yield "C [a,24,b,16,c,16,d,24,e,16,f,16] -= sum(g,24) * A [d,e,g,a] * B [g,f,b,c];"
    yield "C [a,24,b,16,c,16,d,24,e,16,f,16] -= sum(g,24) * A [d,e,g,b] * B [g,f,a,c];"
    yield "C [a,20,b,11,c,13,d,17,e,10,f,9] += sum(g,15) * A [d,e,g,c] * B [g,f,a,b];"
    yield "C [a,10,b,26,c,7,d,5,e,12,f,31] = sum(g,22) * A [d,f,g,a] * B [g,e,b,c];"
    yield "C [a,24,b,16,c,16,d,24,e,16,f,6] -= sum(g,24) * A [d,f,g,b] * B [g,e,a,c];"
    yield "C [a,2,b,40,c,30,d,50] += sum(e,8) * A [a,e,b,d] * B [e,c];"
    yield "C [a,400,b,300] += sum(c,16) * A [c,a] * B [c,b];"
    yield "C [a,50,b,64,c,70,d,3] += sum(e,20) * A [d,a,e] * B [c,e,b];"


@pytest.mark.parametrize("expr", list(_wc_layouts()))
def test_cut_tiles_cover_the_output_once_and_are_boxes_of_it(pkg, expr):
    """Output-resident kernel: the rows and columns of a cut tile, decoded through the index classes as the loaders do,
    lie at the places of C that the tile's box in the rank-5 view has at the same place of the buffer."""
    import numpy as np
    d = _plan(pkg, expr, tile=(128, 64), variant=4).describe()
    if "cbox" not in d:
        d = _plan(pkg, expr).describe()
    assert "cbox" in d, d["kernel"]
    box = d["cbox"]

    def class_out(dims, cut, tiles):
        """Per tile: offsets in C of its rows (-1: none), as cut_flat and decode compute them."""
        off = np.zeros(1, dtype=np.int64)
        for q in dims:
            off = (np.arange(q["extent"], dtype=np.int64)[:, None] * q["s_out"] + off[None, :]).reshape(-1)
        b0, b1, e0, e1, t0, t1 = cut
        out = []
        for t in range(tiles):
            v0, v1, rest = t % t0 * b0, t // t0 % t1 * b1, t // t0 // t1
            rows = [v0 + r % b0 + e0 * (v1 + r // b0 + e1 * rest) if v0 + r % b0 < e0 and v1 + r // b0 < e1 else -1
                    for r in range(b0 * b1)]
            assert all(r < off.size for r in rows)
            out.append((np.array([off[r] if r >= 0 else -1 for r in rows]), (v0, v1, rest)))
        return out

    assert box["m"][0] % 2 == 0 and box["m"][0] * box["m"][1] <= 128 and box["n"][0] * box["n"][1] <= 64
    ms, ns = class_out(d["M"], box["m"], d["tiles"][0]), class_out(d["N"], box["n"], d["tiles"][1])
    n0, n1, m1, mr0, mr1, nr0, nr1 = box["slots"]
    seen = np.zeros(int(np.prod([e for e in d["expr"]["out_ext"]])), dtype=np.int32)
    b0, nb = box["m"][0], box["n"][0] * box["n"][1]
    for om, (mv0, mv1, mrest) in ms:
        for on, (nv0, nv1, nrest) in ns:
            corner = [mv0, 0, 0, 0, 0]
            for slot, v in ((n0, nv0), (n1, nv1), (m1, mv1), (mr0, mrest % box["rest"][0]), (mr1, mrest // box["rest"][0]),
                            (nr0, nrest % box["rest"][1]), (nr1, nrest // box["rest"][1])):
                if slot:
                    corner[slot] = v
            if mr0 and mr0 == nr0:
                corner[mr0] = mrest * box["steps"][0] + nrest * box["steps"][1]
            # the box as the copy engine lays it out: first dimension fastest, -1 outside the tensor
            place = np.zeros(1, dtype=np.int64)
            for k, (ext, size, stride) in enumerate(box["dims"]):
                at = corner[k] + np.arange(size, dtype=np.int64)
                step = np.where(at < ext, at * stride, np.int64(-1) << 50)
                place = (step[:, None] + place[None, :]).reshape(-1)
            m, n = np.arange(om.size), np.arange(on.size)
            pos = (m % b0 + m // b0 * (b0 * nb))[:, None] + (n * b0)[None, :]
            want = np.where((om[:, None] >= 0) & (on[None, :] >= 0), om[:, None] + on[None, :], -1)
            got = place[pos]
            assert pos.max() < place.size
            assert np.array_equal(np.where(got < 0, -1, got), want)
            np.add.at(seen, want[want >= 0], 1)
    assert (seen == 1).all()


def test_cut_tiles_keep_pairs_of_an_input_together(pkg):
    """An input read 16 bytes at a time along N's first index: a tile starts at an even value of it and holds an even
    number (21 of 42 would save a third of the tiles)."""
    d = _plan(pkg, "C [a,24,b,42,c,200,d,9] += sum(e,24) * A [e,a,c] * B [b,e,d];", tile=(128, 64), variant=4).describe()
    assert d["vec_y"] and d["cbox"]["n"][0] % 2 == 0 and d["cbox"]["n"][2] == 42
    odd = _plan(pkg, "C [a,24,b,43,c,200,d,9] += sum(e,24) * A [e,a,c] * B [b,e,d];", tile=(128, 64), variant=4).describe()
    assert not odd["vec_y"] and "cbox" in odd


def test_blocked_contractions_name_every_value_once(pkg):
    """Two inputs that start with different contraction indices: 4 x 4 blocks of K, rounded up, with holes."""
    for c, d in ((64, 64), (61, 66), (4, 130), (63, 50), (7, 41), (62, 62)):
        p = _plan(pkg, "t3 [a,2048,b,2048] += sum(c,%d,d,%d) * t2 [c,a,d] * v2 [d,b,c];" % (c, d)).describe()
        assert p["kernel"].startswith("dmma_w") and [k["extent"] for k in p["K"][:2]] == [4, 4]
        assert p["Kflat"] == (c + 3) // 4 * 4 * ((d + 3) // 4 * 4)
    small = _plan(pkg, "t3 [a,20,b,20] += sum(c,6,d,7) * t2 [c,a,d] * v2 [d,b,c];").describe()
    assert small["Kflat"] == 42   # kernels that know no holes keep the plain order


def _short_run_cuts():
    """Output-resident plans whose cuts hold runs that are not whole fours (14 of 28, 18 of 36, ...)."""
    yield "C [a,28,b,60,c,20,d,60] += sum(g,200) * A [d,a,g,b] * B [g,c];"
    yield "C [a,36,b,40,c,7,d,12] += sum(e,16) * A [e,a,c] * B [e,b,d];"
    yield "C [a,52,b,44,c,9,d,52] -= sum(e,24) * A [d,a,e,b] * B [e,c];"


@pytest.mark.parametrize("expr", list(_short_run_cuts()) + list(_wc_layouts()))
def test_rows_the_stand_in_takes_together_are_neighbours_in_the_output(pkg, expr):
    """Where an output cannot be addressed as boxes, the cut tiles run on a kernel that moves standin_vec_c consecutive
    rows of a tile as neighbours in C."""
    import numpy as np
    d = _plan(pkg, expr, tile=(128, 64), variant=4).describe()
    b0, b1, e0, e1, t0, t1 = d["cbox"]["m"] if "cbox" in d else (128, 1, d["Mflat"], 1, d["tiles"][0], 1)
    off = np.zeros(1, dtype=np.int64)
    for q in d["M"]:
        off = (np.arange(q["extent"], dtype=np.int64)[:, None] * q["s_out"] + off[None, :]).reshape(-1)
    for t in range(d["tiles"][0]):
        v0, v1, rest = t % t0 * b0, t // t0 % t1 * b1, t // t0 // t1
        rows = [v0 + r % b0 + e0 * (v1 + r // b0 + e1 * rest) if r < b0 * b1 and v0 + r % b0 < e0 and v1 + r // b0 < e1 else -1
                for r in range(128)]
        for r in range(0, 128, 4) if d["standin_vec_c"] == 4 else ():
            four = [off[q] if q >= 0 else -1 for q in rows[r:r + 4]]
            assert four == [-1] * 4 or four == [four[0] + i for i in range(4)], (d["cbox"]["m"], t, r)


@pytest.mark.parametrize("tma", [1, 2])
@pytest.mark.parametrize("expr", list(_short_run_cuts()))
def test_outputs_kept_from_the_copy_engine_have_plain_tiles(pkg, expr, tma):
    boxes = _plan(pkg, expr, tile=(128, 64), variant=4).describe()
    assert boxes["cbox"]["m"][0] % 4 == 2 and boxes["vec_c"] == 4 and boxes["standin_vec_c"] == 2
    plain = _plan(pkg, expr, tile=(128, 64), variant=4, tma=tma).describe()
    assert "cbox" not in plain and plain["tiles"] == [(plain["Mflat"] + 127) // 128, (plain["Nflat"] + 63) // 64]


@pytest.mark.parametrize("expr,options,kernel", [
    ("C [a,18,b,76,c,8,d,221,e,2,f,2] = sum(k,8) * A [k,d] * B [k,e,f,b,c,a];", dict(variant=4, tma=1), "dmma_wc_128x64"),
    ("C [a,16,b,268,c,4,d,48,e,9] -= sum(k,215) * A [b,c,k] * B [e,d,k,a];", dict(variant=4, tma=2), "dmma_wc_128x64"),
    ("C [a,4,b,16,c,32,d,16,e,140,f,8] = sum(k,4) * A [e,a,d,c,k] * B [k,f,b];", dict(variant=4, tma=3, c_path=1), "dmma_wc_128x64"),
    ("C [a,70,b,13,c,20,d,270] += sum(k,4,l,26,m,19) * A [k,m,a,d,l] * B [c,m,l,b,k];", dict(variant=4, tma=4, c_path=3), "dmma_wc_128x64"),
    ("C [a,8,b,64,c,275,d,22] -= sum(k,8,l,39,m,1) * A [m,d,l,k,c] * B [m,l,k,a,b];", dict(variant=4, c_path=1), "dmma_wc_128x64"),
    ("C [a,48,b,48,c,18,d,9,e,25] += sum(k,9) * A [c,b,k,a] * B [d,k,e];", dict(variant=2), "dmma_128x64_w8"),
    ("C [a,8,b,96,c,236,d,48] = sum(k,4,l,7) * A [l,k,b] * B [k,l,d,c,a];", dict(variant=1, tma=3), "dmma_64x96_w4"),
])
def test_a_named_variant_gets_a_tile_it_has(pkg, expr, options, kernel):
    """Variant named, tile left to the planner: the choice does not follow the rules for cut tiles to one that the
    variant is not compiled for."""
    assert _plan(pkg, expr, **options).describe()["kernel"] == kernel


@pytest.mark.parametrize("expr", [
    "t3 [a,1200,b,512] += sum(c,30,d,30) * t2 [c,a,d] * v2 [d,b,c];",                         # 900 values, 1024 positions
    "C [a,24,b,64,c,33,d,8] = sum(k,5,l,1,m,292) * A [m,b,l,d,k] * B [k,l,a,m,c];",           # 1460 and 2336
    "C [a,16,b,8,c,6,d,5,e,31] += sum(k,12,l,34,m,2) * A [l,e,b,d,k,m,c] * B [m,k,l,a];",     # 816 and 1728
    "C [a,67,b,14,c,6,d,48] += sum(k,344,l,2) * A [l,k,a] * B [k,d,b,l,c];",                  # 688 and 1376
])
def test_rounding_a_contraction_up_asks_for_no_scratch(pkg, expr):
    """... so that such a plan runs without a workspace, through the entry that never allocates and on several streams."""
    assert _plan(pkg, expr).describe()["workspace_bytes"] == 0


def test_rounding_a_contraction_up_makes_no_further_slices(pkg):
    """split_k is bounded by the steps of the true length: 2 x 7 values are one step, not the two of 4 x 8 positions."""
    d = _plan(pkg, "C [a,38,b,282,c,8,d,163] += sum(k,2,l,7) * A [k,d,a,l,c] * B [l,b,k];", split_k=2, tile=(128, 64), variant=3).describe()
    assert d["ksplit"] == 1 and d["workspace_bytes"] == 0


@pytest.mark.parametrize("c,d", [(30, 30), (22, 22), (2, 200), (200, 2), (100, 3), (6, 50), (5, 5), (17, 17), (63, 5), (5, 8000), (33, 16)])
def test_contractions_that_blocks_would_pad_keep_the_plain_order(pkg, c, d):
    """More added products than the larger operand's traffic saves."""
    p = _plan(pkg, "t3 [a,2048,b,2048] += sum(c,%d,d,%d) * t2 [c,a,d] * v2 [d,b,c];" % (c, d)).describe()
    assert p["Kflat"] == c * d


def test_blocks_may_add_more_where_the_operand_streams_from_memory(pkg):
    """26 x 50 x 50 values, 12 % more in blocks: taken for 248 columns (129 MB), not for 24 (12 MB)."""
    expr = "C [a,8,b,%d,c,1] -= sum(k,26,l,50,m,50) * A [k,m,a,l] * B [l,k,c,b,m];"
    assert _plan(pkg, expr % 248).describe()["Kflat"] == 28 * 52 * 50
    assert _plan(pkg, expr % 24).describe()["Kflat"] == 26 * 50 * 50


@pytest.mark.parametrize("tiles_m", [1, 3, 7, 11, 16, 37, 73])
@pytest.mark.parametrize("k", [1100, 2048, 9000, 97344])
def test_few_slices_do_not_lengthen_the_chains_of_additions(pkg, tiles_m, k):
    """A slice is added up in segments no longer than four work items for each of the 148 multiprocessors, or sixteen
    steps, would make slices."""
    d = _plan(pkg, "C [a,%d,b,128] += sum(c,%d) * A [c,a] * B [b,c];" % (128 * tiles_m, k)).describe()
    if d["kernel"] != "dmma_ws_128x64" or d["ksplit"] == 1:
        return
    tiles, steps = d["tiles"][0] * d["tiles"][1], (k + 15) // 16
    most = max(1, min((4 * 148 + tiles - 1) // tiles, steps // 16))
    assert 0 < d["k_seg"] <= (steps + most - 1) // most and 16 * d["k_seg"] <= d["k_chunk"]


@pytest.mark.parametrize("expr", [
    "C [a,34,b,24,c,28,d,35] = sum(k,35,l,33) * A [k,l,b] * B [l,k,a,d,c];",     # 261 tiles: a round holds one slice of each
    "C [a,123,b,15,c,299,d,4,e,1] = sum(k,12,l,152) * A [k,a,l,d,e] * B [l,k,c,b];",
    "C [a,32,b,215,c,84] += sum(k,39,l,30) * A [k,c,b,l] * B [l,a,k];",
    "C [a,96,b,96,c,96,d,96] += sum(e,96) * A [a,e,b,d] * B [e,c];",             # not sliced at all
])
def test_only_slices_are_added_up_in_segments(pkg, expr):
    """A sum that is not sliced goes into C in one piece."""
    d = _plan(pkg, expr).describe()
    assert d["ksplit"] > 1 or d["k_seg"] * 16 >= d["Kflat"]


@pytest.mark.parametrize("expr", [
    "C [a,20,b,6,c,6,d,95,e,2,f,23] = sum(k,2) * A [k,e,d,c,a,f] * B [k,b];",      # boxes of 20 x 6
    "C [a,26,b,4,c,6,d,36,e,8,f,4] = sum(k,6) * A [k,b] * B [k,f,a,e,d,c];",
    "C [a,2,b,24,c,10,d,2,e,21,f,172] = sum(k,10) * A [k,a] * B [d,c,b,e,f,k];",   # runs of two
    "C [a,32,b,8,c,9,d,2,e,216,f,3] += sum(k,3) * A [e,d,a,f,k,c] * B [k,b];",
    "C [a,4,b,35,c,220,d,96] -= sum(k,34) * A [k,a] * B [k,c,b,d];",
])
def test_outputs_of_thin_boxes_stay_off_the_resident_tile(pkg, expr):
    """A resident tile takes some 4000 cycles however little of the output is in its box."""
    assert not _plan(pkg, expr).describe()["kernel"].startswith("dmma_wc")


@pytest.mark.parametrize("expr", [
    "C [a,24,b,16,c,16,d,24,e,16,f,16] -= sum(g,24) * A [d,e,g,a] * B [g,f,b,c];",
    "C [a,40,b,40,c,40,d,40,e,40,f,5] += sum(g,40) * A [g,a,b,c] * B [d,e,f,g];",
])
def test_outputs_of_full_boxes_stay_on_the_resident_tile(pkg, expr):
    assert _plan(pkg, expr).describe()["kernel"].startswith("dmma_wc")


@pytest.mark.parametrize("expr", [
    "C [a,96,b,8,c,31,d,40] += sum(k,282,l,15,m,8) * A [l,b,a,m,c,k] * B [l,k,m,d];",
    "C [a,64,b,32,c,121,d,6] = sum(k,260,l,240) * A [k,c,l] * B [l,b,a,k,d];",
])
def test_the_choice_of_a_tile_brings_no_slices(pkg, expr):
    """Whether there are too few tiles to fill the GPU is the plain model's question: these sums need no scratch."""
    assert _plan(pkg, expr).describe()["workspace_bytes"] == 0


def test_pairs_of_ctas_need_no_scratch(pkg):
    # few tiles (64 of 128 x 128) and one or four chains: the pairs cut the chains themselves, what stands in for them where a
    # tensor is not aligned runs in passes
    for k, passes in ((512, 1), (2000, 4)):
        d = _plan(pkg, "C [a,900,b,900] += sum(c,%d) * A [c,a] * B [c,b];" % k, "float32").describe()
        assert d["pair"] and d["workspace_bytes"] == 0 and d["ksplit"] == 1 and d["launches"] == 1, d
        assert d["passes"] == passes and d["chain"] <= 512, d


# Panels: where they measured slower than the ring kernel it runs, and where faster, they do (K = 8 to 48).
@pytest.mark.parametrize("extents,k,left,right,op,panel", [
    ((22, 16, 19, 16, 24, 16), 38, "e,f,g,b", "g,d,a,c", "+=", False),   # the tiles cut M's first digit: 199 against 387 us
    ((26, 20, 18, 22, 20, 16), 40, "d,e,g,a", "g,f,b,c", "=", False),    # ... X gathered, C only written: 264, 447
    ((24, 16, 16, 24, 16, 16), 40, "d,f,g,b", "g,e,a,c", "+=", False),   # ... 187, 207
    ((16, 17, 16, 24, 17, 15), 38, "e,f,g,b", "g,d,a,c", "=", True),     # whole digit, whole sectors: 114, 99
    ((24, 16, 16, 24, 16, 16), 24, "d,e,g,a", "g,f,b,c", "-=", True),    # X gathered: 156, 129
    ((16, 22, 11, 17, 24, 26), 10, "d,e,g,a", "g,f,b,c", "+=", False),   # ... short contraction: 110, 124
    ((16, 16, 24, 24, 16, 11), 10, "d,e,g,a", "g,f,b,c", "=", True),     # ... C only written
    ((10, 16, 20, 21, 14, 16), 20, "e,f,g,a", "g,d,b,c", "+=", False),   # ... runs of 80 bytes: 57, 59
    ((24, 24, 10, 26, 16, 22), 38, "g,a,d,e", "b,c,g,f", "=", False),    # X in tiled boxes: 193, 201
    ((25, 19, 30, 31, 32, 18), 36, "g,a,b,c", "d,e,f,g", "+=", False),   # fewer panels than CTAs: 759, 937
    ((40, 40, 40, 40, 40, 5), 40, "g,a,b,c", "d,e,f,g", "+=", True),     # a slab of the 40^6 output: 1 736, 1 633
])
def test_panels_where_they_pay(pkg, extents, k, left, right, op, panel):
    out = ",".join("%s,%d" % x for x in zip("abcdef", extents))
    expr = "C [%s] %s sum(g,%d) * A [%s] * B [%s];" % (out, op, k, left, right)
    d = _plan(pkg, expr).describe()
    assert d["kernel"] == "dmma_wc_128x64" and d["panel"] == panel and d["tiles"][0] * d["tiles"][1] >= 8 * 148, d


def test_a_named_kernel_is_the_one_that_runs(pkg):
    expr = "C [a,384,b,256] = sum(c,1028) * A [c,a] * B [c,b];"
    for kw in (dict(path=pkg.PATH_TCGEN05, tile=(128, 128), variant=2), dict(tile=(128, 128), variant=1), dict(path=pkg.PATH_TCGEN05, tile=(96, 128), variant=2)):
        d = _plan(pkg, expr, "float32", **kw).describe()
        assert not d["pair"] and d["runs"] == d["kernel"] and d["runs_tile"] == d["tile"][:2] == list(kw["tile"]) and d["ran"] is None, d
    # left to the planner: what runs is named beside what the plan was made for
    d = _plan(pkg, "C [a,1024,b,768] = sum(c,1028) * A [c,a] * B [c,b];", "float32").describe()
    assert d["pair"] and d["kernel"] == "tf32wt_128x128" and d["runs"] == "tf32wd_256x256" and d["runs_tile"] == [256, 256], d
    d = _plan(pkg, "C [a,4096,b,4096] = sum(c,1028) * A [c,a] * B [c,b];", "float32", variant=2).describe()
    assert not d["pair"] and d["runs"] == d["kernel"], d
    six = "C [a,24,b,16,c,16,d,24,e,16,f,16] -= sum(g,24) * A [d,e,g,a] * B [g,f,b,c];"
    d = _plan(pkg, six).describe()
    assert d["panel"] and d["runs"] == "dmma_wp_128x64", d
    d = _plan(pkg, six, tile=(128, 64), variant=4, tma=1).describe()   # no boxes of the output: the reduce-add kernel
    assert d["runs"] == "dmma_ws_128x64" and d["kernel"] == "dmma_wc_128x64", d


# fp64 sums of few tiles that are not sliced: on the persistent 128 x 32 kernels, but for short waits (times in us on those and
# on the one-tile kernel).
@pytest.mark.parametrize("form,op,runs", [
    (((1088, 688), 436, "a,c", "c,b"), "+=", "dmma_w"),                # 40, 62
    (((786, 160), 67, "a,c", "c,b"), "+=", "dmma_w"),                  # 8.2, 13.7: C in pairs
    (((529, 496), 70, "a,c", "c,b"), "+=", "dmma_w"),                  # 12.3, 23.2: odd, added to C
    (((1121, 219), 68, "a,c", "b,c"), "=", "dmma_64x64"),              # 16.4, 12.7: odd, only written
    (((115, 1008), 105, "a,c", "b,c"), "=", "dmma_64x64"),             # 16.4, 13.9
    (((392, 240), 92, "a,c", "b,c"), "=", "dmma_64x64"),               # 10.3, 9.1: 16-byte loads and stores
    (((392, 240), 120, "a,c", "b,c"), "=", "dmma_w"),                  # ... two steps more
    (((1088, 688), 60, "a,c", "c,b"), "+=", "dmma_64x64"),             # four steps
])
def test_few_tiles_on_the_narrow_persistent_kernels(pkg, form, op, runs):
    (m, n), k, left, right = form
    d = _plan(pkg, "C [a,%d,b,%d] %s sum(c,%d) * A [%s] * B [%s];" % (m, n, op, k, left, right)).describe()
    assert d["runs"].startswith(runs) and d["ksplit"] == 1 and d["workspace_bytes"] == 0, d
    if runs == "dmma_w":
        assert d["runs_tile"] == [128, 32], d


# fp32 without any alignment: tcgen05, one tile per CTA, but for few columns or few rows.
@pytest.mark.parametrize("extents,k,runs", [((55, 31, 39, 39), 61, "tf32tc_128x128"), ((1641, 11, 23, 9), 61, "tf32tc_128x128"),
                                            ((57, 31, 39, 29), 63, "tf32_64x64"), ((333, 333, 7, 9), 41, "tf32_64x64")])
def test_fp32_without_alignment(pkg, extents, k, runs):
    out = ",".join("%s,%d" % x for x in zip("abcd", extents))
    left, right = ("e,a", "e,b,c,d") if extents[0] < 64 and extents[0] != 55 else ("a,b,e", "e,c,d")
    d = _plan(pkg, "C [%s] += sum(e,%d) * A [%s] * B [%s];" % (out, k, left, right), "float32").describe()
    assert d["vec_c"] == 1 and not (d["vec_x"] or d["kvec_x"] or d["vec_y"] or d["kvec_y"]) and d["runs"] == runs, d
