"""Kernels and dispatch rules at the sizes where they can go wrong, against the CPU loop nest: cut tiles of the
output-resident fp64 kernels, blocked contractions with holes, element epilogues, K slices combined in parts, kernels
chained in a stream, the fused kernel's boxes.  fp64 tolerance as everywhere: 1e-12 of the largest value."""
import pytest

pytestmark = pytest.mark.gpu


def _run(pkg, orc, expr, seed=3, dtype="float64", **kw):
    import torch
    torch.cuda.set_device(0)
    c0, a, b = orc.make_inputs(expr, seed, dtype)
    ref = orc.contract(expr, c0.copy(), a, b)
    plan = pkg.Plan(expr, pkg.F64 if dtype == "float64" else pkg.F32, **kw)
    d = plan.describe()
    dc, da, db = (torch.from_numpy(x).cuda() for x in (c0, a, b))
    plan.execute(dc, da, db)
    torch.cuda.synchronize()
    err = orc.rel_error(dc.cpu().numpy(), ref)
    assert plan.status() == 0
    plan.close()
    return d, err


CUT = [
    "C [a,24,b,8,c,7,d,10,e,6,f,5] -= sum(g,24) * A [d,e,g,a] * B [g,f,b,c];",     # runs of 24, five per tile, gathered across
    "C [a,22,b,9,c,11,d,6,e,4,f,5] += sum(g,15) * A [d,e,g,b] * B [g,f,a,c];",     # 22-element runs: pairs straddle no quad
    "C [a,10,b,26,c,7,d,5,e,4,f,3] = sum(g,22) * A [d,f,g,a] * B [g,e,b,c];",
    "C [a,24,b,6,c,10,d,8,e,6,f,5] -= sum(g,24) * A [d,f,g,b] * B [g,e,a,c];",     # six dimensions, two sharing one of the map
    "C [a,2,b,40,c,30,d,9] += sum(e,8) * A [a,e,b,d] * B [e,c];",                  # shortest runs
    "C [a,24,b,42,c,20,d,9] += sum(e,24) * A [e,a,c] * B [b,e,d];",                # an input read in pairs along N's first index
    "C [a,30,b,7,c,26,d,10] += sum(e,33) * A [d,c,e,a] * B [e,b];",                # narrow tile's shape, ragged both ways
]


@pytest.mark.parametrize("tile", [(128, 64), (128, 32)])
@pytest.mark.parametrize("expr", CUT)
def test_cut_tiles_against_the_loop_nest(pkg, orc, expr, tile):
    d, err = _run(pkg, orc, expr, tile=tile, variant=4)
    assert d["kernel"] == "dmma_wc_%dx%d" % tile and "cbox" in d
    assert err <= 1e-12, (d["cbox"], err)


def test_cut_tiles_of_a_misaligned_output_run_without_boxes(pkg, orc):
    import torch
    expr = CUT[0]
    c0, a, b = orc.make_inputs(expr, 5, "float64")
    ref = orc.contract(expr, c0.copy(), a, b)
    plan = pkg.Plan(expr, tile=(128, 64), variant=4)
    buf = torch.zeros(c0.size + 1, dtype=torch.float64, device="cuda")
    buf[1:].copy_(torch.from_numpy(c0))                                            # 8 bytes past an aligned address
    plan.execute(buf[1:], torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda())
    torch.cuda.synchronize()
    assert plan.status() == 0 and orc.rel_error(buf[1:].cpu().numpy(), ref) <= 1e-12
    plan.close()


@pytest.mark.parametrize("c_path", [0, 2])
@pytest.mark.parametrize("tma", [1, 2])
@pytest.mark.parametrize("expr", [
    "C [a,28,b,60,c,20,d,60] += sum(g,200) * A [d,a,g,b] * B [g,c];",               # the boxes would hold runs of 14
    "C [a,36,b,40,c,7,d,12] += sum(e,16) * A [e,a,c] * B [e,b,d];",                 # ... of 18
])
def test_output_resident_plans_kept_from_the_copy_engine(pkg, orc, expr, tma, c_path):
    d, err = _run(pkg, orc, expr, tile=(128, 64), variant=4, tma=tma, c_path=c_path)
    assert "cbox" not in d and err <= 1e-12


@pytest.mark.parametrize("c,d,b", [(61, 66, 1100), (64, 64, 70), (4, 150, 70), (7, 41, 70), (63, 50, 1300), (9, 10, 5000),
                                   (5, 10, 70), (3, 3, 70)])
@pytest.mark.parametrize("split", [0, 3])
def test_blocked_contractions_against_the_loop_nest(pkg, orc, c, d, b, split):
    expr = "t3 [a,70,b,%d] += sum(c,%d,d,%d) * t2 [c,a,d] * v2 [d,b,c];" % (b, c, d)
    desc, err = _run(pkg, orc, expr, tile=(128, 64), variant=3, split_k=split)
    rounded = (c + 3) // 4 * 4 * ((d + 3) // 4 * 4)
    assert desc["Kflat"] == (c * d if c * d < 91 else rounded) and err <= 1e-12  # the last three add 60 to 90 %: plain order


def test_contractions_that_were_rounded_up_run_without_scratch(pkg, orc):
    import torch
    expr = "t3 [a,1200,b,512] += sum(c,30,d,30) * t2 [c,a,d] * v2 [d,b,c];"
    c0, a, b = orc.make_inputs(expr, 8, "float64")
    ref = orc.contract(expr, c0.copy(), a, b)
    plan = pkg.Plan(expr).commit()
    dc, da, db = (torch.from_numpy(x).cuda() for x in (c0, a, b))
    plan.execute_noalloc(dc, da, db)
    torch.cuda.synchronize()
    assert plan.workspace_bytes() == 0 and plan.status() == 0 and orc.rel_error(dc.cpu().numpy(), ref) <= 1e-12
    plan.close()


@pytest.mark.parametrize("tile,variant", [((128, 64), 3), ((64, 96), 3), ((128, 32), 3)])
@pytest.mark.parametrize("op", ["+=", "=", "-="])
def test_odd_outputs_and_ragged_edges(pkg, orc, tile, variant, op):
    # 67 columns: groups of columns outside the tensor; 61 x 13 rows: a warp's rows outside it; every row at odd offsets
    _, err = _run(pkg, orc, "C [a,61,b,13,c,67,d,3] %s sum(e,21) * A [a,e,b,d] * B [e,c];" % op, tile=tile, variant=variant)
    assert err <= 1e-12


@pytest.mark.parametrize("dtype,tol", [("float64", 1e-12), ("float32", 1e-5)])
@pytest.mark.parametrize("split", [2, 7, 19])
def test_slices_combined_in_parts(pkg, orc, dtype, tol, split):
    _, err = _run(pkg, orc, "C [a,70,b,45] -= sum(c,700) * A [c,a] * B [c,b];", dtype=dtype, split_k=split)
    assert err <= tol


@pytest.mark.parametrize("expr", [
    "C [a,510,b,316] += sum(c,64,d,64) * A [c,a,d] * B [d,b,c];",       # 14 slices of 19 steps, in segments of ten
    "C [a,310,b,200] -= sum(c,9000) * A [c,a] * B [c,b];",              # a last segment that is shorter, a last step of eight
    "C [a,270,b,66,c,21] = sum(k,4,l,352) * A [l,c,k] * B [a,k,l,b];",
    "C [a,34,b,24,c,28,d,35] = sum(k,35,l,33) * A [k,l,b] * B [l,k,a,d,c];",    # 261 tiles: more than a slice of each to a round
])
def test_slices_added_up_in_segments(pkg, orc, expr):
    d, err = _run(pkg, orc, expr)
    assert d["kernel"] == "dmma_ws_128x64" and d["ksplit"] > 1 and 16 * d["k_seg"] < d["k_chunk"] and err <= 1e-12


@pytest.mark.parametrize("expr,kw", [
    ("C [i,64,j,48,k,32] += sum(l,40) * A [l,k,i] * B [j,l];", {}),
    ("C [a,70,b,45] += sum(c,700) * A [c,a] * B [c,b];", {"split_k": 5}),
])
def test_kernels_chained_in_a_stream_see_their_predecessors(pkg, orc, expr, kw):
    """Each pass adds to what the pass before wrote, and reads an input that a kernel just before it wrote."""
    import torch
    c0, a, b = orc.make_inputs(expr, 6, "float64")
    ref = c0.copy()
    plan = pkg.Plan(expr, **kw)
    dc, da, db = (torch.from_numpy(x).cuda() for x in (c0, a, b))
    scaled = torch.empty_like(da)
    for n in range(40):
        torch.mul(da, float(n % 5 + 1), out=scaled)
        plan.execute(dc, scaled, db)
    for n in range(5):  # the loop nest once per factor: 40 passes are 8 of each
        one = orc.contract(expr, c0 * 0, a * (n + 1), b)
        ref = ref + 8 * one
    torch.cuda.synchronize()
    assert orc.rel_error(dc.cpu().numpy(), ref) <= 1e-12
    plan.close()


@pytest.mark.parametrize("k", [2, 8, 10, 16, 22, 34])
@pytest.mark.parametrize("ext", [(4, 4, 4, 4, 4, 4), (5, 3, 9, 1, 6, 7), (10, 11, 4, 8, 2, 13)])
def test_fused_boxes_against_the_loop_nest(pkg, orc, k, ext):
    import torch
    torch.cuda.set_device(0)
    out = "t3 [h3,%d,h2,%d,h1,%d,p6,%d,p5,%d,p4,%d]" % ext
    lines = ["%s %s sum(p7,%d) * x%d [%s] * y%d [%s];" % (out, op, k, n, l, n, r) for n, (op, l, r) in enumerate([
        ("-=", "p7,p4,h1,h2", "p7,h3,p6,p5"), ("+=", "p7,p5,h2,h3", "p7,h1,p6,p4")])]
    if ext[0] == 5:  # four indices in one input: two values each in a box
        lines.append("%s -= sum(p7,%d) * x2 [p7,h3,p6] * y2 [p7,h1,h2,p5,p4];" % (out, k))
    plan = pkg.FusedPlan(lines)
    assert plan.describe()["kernel"] == "tc_fused_box_kernel"
    c0 = orc.uniform(60, 0, orc.sizes(lines[0])[0])
    ref, ins = c0.copy(), []
    for n, line in enumerate(lines):
        _, na, nb = orc.sizes(line)
        a, b = orc.uniform(61 + n, 1, na), orc.uniform(61 + n, 2, nb)
        ins.append((a, b))
        orc.contract(line, ref, a, b)
    dc = torch.from_numpy(c0).cuda()
    plan.execute(dc, [torch.from_numpy(a).cuda() for a, _ in ins], [torch.from_numpy(b).cuda() for _, b in ins])
    torch.cuda.synchronize()
    assert orc.rel_error(dc.cpu().numpy(), ref) <= 1e-12
    plan.close()


@pytest.mark.parametrize("k", [160, 264, 520, 1032])
def test_split_groups_of_the_persistent_fp32_kernel(pkg, orc, k):
    """Odd and even numbers of K steps, a last step of eight, more than one tile per CTA, three launches in a row."""
    expr = "C [a,3072,b,2048] += sum(c,%d) * A [c,a] * B [c,b];" % k
    import numpy as np
    import torch
    torch.cuda.set_device(0)
    a = torch.rand(3072, k, device="cuda") - 0.5
    b = torch.rand(2048, k, device="cuda") - 0.5
    c = torch.rand(2048, 3072, device="cuda")
    want = (c.double() + b.double() @ a.double().T).cpu().numpy()
    plan = pkg.Plan(expr, pkg.F32)
    assert plan.describe()["kernel"].startswith("tf32wt")
    for n in range(3):
        got = c.clone()
        plan.execute(got, a, b)
        torch.cuda.synchronize()
        assert plan.status() == 0
        assert np.abs(got.cpu().numpy() - want).max() / np.abs(want).max() <= 1e-5
    plan.close()


REFUSED_LAUNCH = """
import ctypes, sys
sys.path.insert(0, {root!r})
import __graft_entry__ as entry
import torch
pkg = entry.load_package()
torch.cuda.set_device(0)
small = pkg.Plan("C [i,64,j,48,k,32] += sum(l,40) * A [l,k,i] * B [j,l];").commit()        # one-tile kernel
sliced = pkg.Plan("C [a,70,b,45] += sum(c,700) * A [c,a] * B [c,b];", split_k=5).commit()  # ... and a combine step
large = pkg.Plan("C [a,48,b,48,c,48,d,48] += sum(e,48) * A [a,e,b,d] * B [e,c];").commit()  # persistent kernel
bufs = [torch.zeros(n, dtype=torch.float64, device="cuda") for n in (48 ** 4, 48 ** 4, 48 ** 3)]
for plan in (small, sliced, large):
    plan.execute(*bufs)
torch.cuda.synchronize()
rt = ctypes.CDLL("libcudart.so.12")
for refused in (small, sliced):
    stream, graph = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(stream)) == 0
    assert rt.cudaStreamBeginCapture(stream, 0) == 0
    try:
        refused.execute(*bufs, stream=1)       # the legacy stream: the runtime refuses it while a blocking stream captures
        raise SystemExit("accepted")
    except pkg.TcError as e:
        assert e.status == 5, e
    assert rt.cudaStreamEndCapture(stream, ctypes.byref(graph)) != 0
    rt.cudaGetLastError()
    large.execute(*bufs)                       # not this call's failure
    torch.cuda.synchronize()
    assert large.status() == 0
print("held")
"""


def test_a_refused_launch_is_not_reported_again():
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", REFUSED_LAUNCH.format(root=root)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "held", r.stdout + r.stderr


# Panels: every loader of both operands, one to three K steps with remainders, fewer panels than CTAs and more (whole
# panels first, then runs of the rest), an odd number of tiles in a row, cut tiles.  Up to two K steps are panels only where
# X is gathered across its sectors.
PANEL_SIZES = [(38, 90, 283, 10, "+="), (130, 150, 64, 8, "-="), (128, 149, 65, 8, "=")]
PANELS = [(x, y, (33, 40, 48)[(i + j) % 3], PANEL_SIZES[(i + 2 * j) % 3]) for i, x in enumerate(("e,a,b", "a,e,b", "e,b,a", "b,e,a"))
          for j, y in enumerate(("e,c,d", "c,d,e", "e,d,c", "d,e,c"))]
PANELS += [("b,e,a", y, k, PANEL_SIZES[(i + k) % 3]) for i, k in enumerate((1, 16, 17, 24)) for y in ("e,c,d", "d,e,c")]


@pytest.mark.parametrize("left,right,k,size", PANELS)
def test_panels_against_the_loop_nest(pkg, orc, left, right, k, size):
    expr = "C [a,%d,b,%d,c,%d,d,%d] %s sum(e,%d) * A [%s] * B [%s];" % (*size, k, left, right)
    desc, err = _run(pkg, orc, expr, tile=(128, 64), variant=4)
    assert desc["kernel"] == "dmma_wc_128x64" and desc["panel"] and err <= 1e-12, (desc["cbox"], err)


# fp32 on pairs of CTAs: both orientations of either operand, rows and columns off the 256-wide tile, contractions whose
# last unit of 32 has one to four groups of eight, chains of one and several segments, more tiles than pairs, rows in runs of
# 32 and 64 of a three-index output; against 64 bits.
PAIRS = [("C [a,%d,b,%d] += sum(c,%d) * A [c,a] * B [c,b];", (2048, 2048, 256)), ("C [a,%d,b,%d] -= sum(c,%d) * A [a,c] * B [c,b];", (1796, 1300, 260)),
         ("C [a,%d,b,%d] = sum(c,%d) * A [c,a] * B [b,c];", (720, 2064, 1104)), ("C [a,%d,b,%d] += sum(c,%d) * A [a,c] * B [b,c];", (3328, 3332, 520)),
         ("C [a,%d,b,%d] = sum(c,%d) * A [a,c] * B [c,b];", (2052, 1028, 2076)), ("C [a,32,b,%d,d,%d] += sum(c,%d) * A [c,a,d] * B [b,c];", (2400, 104, 548)),
         ("C [a,64,b,%d,d,%d] -= sum(c,%d) * A [c,a,d] * B [c,b];", (2200, 54, 308))]


@pytest.mark.parametrize("form,size", PAIRS)
@pytest.mark.parametrize("shift", [0, 1])
def test_pairs_of_ctas(pkg, form, size, shift):
    import torch
    torch.cuda.set_device(0)
    expr = form % size
    p = pkg.parse(expr)
    ext = dict(zip(p["out_idx"] + p["sum_idx"], p["out_ext"] + p["sum_ext"]))
    numel = lambda key: int(torch.tensor([ext[i] for i in p[key]]).prod())
    gen = torch.Generator(device="cuda").manual_seed(7)
    # shift 1: no tensor is 16-byte aligned, and the plan runs on single CTAs
    c, a, b = (torch.rand(numel(key) + 4, device="cuda", generator=gen)[shift:][:numel(key)] - 0.5 for key in ("out_idx", "left_idx", "right_idx"))
    if shift:
        c, a, b = (torch.cat([torch.zeros(1, device="cuda"), t])[1:] for t in (c, a, b))
    view = lambda t, key: t.double().view([ext[i] for i in reversed(p[key])])
    text = ["".join(reversed(p[key])) for key in ("out_idx", "left_idx", "right_idx")]
    want = torch.einsum("%s,%s->%s" % (text[1], text[2], text[0]), view(a, "left_idx"), view(b, "right_idx")).reshape(-1)
    want = want if p["op"] == "=" else c.double() - want if p["op"] == "-=" else c.double() + want
    plan = pkg.Plan(expr, pkg.F32)
    d = plan.describe()
    assert d["pair"] and d["chain"] <= 512 and d["workspace_bytes"] == 0, d
    for _ in range(2):
        got = torch.cat([torch.zeros(4, device="cuda"), c])[4:] if not shift else torch.cat([torch.zeros(1, device="cuda"), c])[1:]
        plan.execute(got, a, b)
        torch.cuda.synchronize()
        assert plan.status() == 0
        assert float((got.double() - want).abs().max() / want.abs().max()) <= 1e-5
    plan.close()


# The pairs run without scratch, whatever the number of tiles, and so does what stands in for them where one tensor is not
# 16-byte aligned: the entry that allocates nothing takes both.
@pytest.mark.parametrize("shift", [(0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 1)])
@pytest.mark.parametrize("k", [512, 2000])
def test_pairs_of_ctas_on_few_tiles_need_no_scratch(pkg, k, shift):
    import torch
    torch.cuda.set_device(0)
    n = 900
    gen = torch.Generator(device="cuda").manual_seed(9)
    c, a, b = (torch.rand(size + 4, device="cuda", generator=gen)[s:s + size] - 0.5 for size, s in zip((n * n, n * k, n * k), (0, 0, 0)))
    place = lambda t, s: torch.cat([torch.zeros(s, device="cuda"), t])[s:]
    c, a, b = (place(t, s) for t, s in zip((c, a, b), shift))
    want = c.double() + (b.double().view(n, k) @ a.double().view(n, k).T).reshape(-1)
    plan = pkg.Plan("C [a,%d,b,%d] += sum(c,%d) * A [c,a] * B [c,b];" % (n, n, k), pkg.F32).commit()
    d = plan.describe()
    assert d["pair"] and d["workspace_bytes"] == 0 and plan.workspace_bytes() == 0 and d["ksplit"] == 1, d
    plan.execute_noalloc(c, a, b)
    torch.cuda.synchronize()
    assert plan.status() == 0
    assert float((c.double() - want).abs().max() / want.abs().max()) <= 1e-5
    plan.close()


def _matrices(m, n, k, shift=(0, 0, 0), seed=11):
    """C [b,a], A [a,c], B [b,c] as flat fp32 tensors, each `shift` elements past an aligned address, and C + A * B in 64 bits."""
    import torch
    torch.cuda.set_device(0)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    place = lambda size, s: torch.cat([torch.zeros(s, device="cuda"), torch.rand(size, device="cuda", generator=gen) - 0.5])[s:]
    c, a, b = (place(size, s) for size, s in zip((m * n, m * k, n * k), shift))
    return c, a, b, c.double() + (b.double().view(n, k) @ a.double().view(m, k).T).reshape(-1)


def _off(got, want):
    return float((got.double() - want).abs().max() / want.abs().max())


# Which kernel a plan for pairs takes where one tensor is not 16-byte aligned: without the output the one-tile kernel in
# passes, without an operand the single CTAs' kernel with that operand fetched element by element.
@pytest.mark.parametrize("shift,ran", [((0, 0, 0), "tf32wd_256x256"), ((1, 0, 0), "tf32tc_128x128"), ((0, 1, 0), "tf32wt_128x128"),
                                       ((0, 0, 1), "tf32wt_128x128"), ((1, 1, 1), "tf32tc_128x128")])
def test_pairs_of_ctas_and_what_stands_in_for_them(pkg, shift, ran):
    import torch
    c, a, b, want = _matrices(1024, 768, 1028, shift)
    plan = pkg.Plan("C [a,1024,b,768] += sum(c,1028) * A [c,a] * B [c,b];", pkg.F32)
    plan.execute(c, a, b)
    torch.cuda.synchronize()
    assert plan.status() == 0 and plan.describe()["ran"] == ran and _off(c, want) <= 1e-5, (plan.describe(), _off(c, want))
    plan.close()


# The single CTAs' kernel by name, at the lengths at which the planner now takes pairs.
@pytest.mark.parametrize("k", [160, 264, 520, 1032])
def test_split_groups_of_the_named_single_cta_kernel(pkg, k):
    import torch
    c, a, b, want = _matrices(3072, 2048, k)
    plan = pkg.Plan("C [a,3072,b,2048] += sum(c,%d) * A [c,a] * B [c,b];" % k, pkg.F32, path=pkg.PATH_TCGEN05, tile=(128, 128), variant=2)
    for _ in range(3):
        got = c.clone()
        plan.execute(got, a, b)
        torch.cuda.synchronize()
        assert plan.status() == 0 and plan.describe()["ran"] == "tf32wt_128x128" and _off(got, want) <= 1e-5
    plan.close()


# The pairs' kernel, repeatedly: several segments per tile, every stage and slot used again, each pass checked.
@pytest.mark.parametrize("m,n,k", [(1024, 768, 1028), (1024, 768, 2112), (5120, 4096, 520)])
def test_pairs_of_ctas_repeatedly(pkg, m, n, k):
    import torch
    c, a, b, want = _matrices(m, n, k)
    plan = pkg.Plan("C [a,%d,b,%d] += sum(c,%d) * A [c,a] * B [c,b];" % (m, n, k), pkg.F32)
    for _ in range(20):
        got = c.clone()
        plan.execute(got, a, b)
        torch.cuda.synchronize()
        assert plan.status() == 0 and _off(got, want) <= 1e-5
    assert plan.describe()["ran"] == "tf32wd_256x256"
    plan.close()


def test_pairs_of_ctas_on_blocks_of_larger_matrices(pkg):
    import torch
    m, n, k = 1024, 768, 260
    c, a, b, _ = _matrices(m, 896, 300, seed=12)             # B as [c,b]: b in [64, 832), c in [32, 292)
    b = b.view(300, 896)
    plan = pkg.Plan("C [a,%d,b,%d] += sum(c,%d) * A [c,a] * B [b,c];" % (m, n, k), pkg.F32)
    plan.set_strides(pkg.TENSOR_LEFT, [1, 300]).set_strides(pkg.TENSOR_RIGHT, [1, 896])
    want = c.double().view(896, m).clone()
    want[64:832] += b.double()[32:292, 64:832].T @ a.double().view(m, 300)[:, 32:292].T
    got = c.clone()
    plan.execute(got[64 * m:], a[32:], b.reshape(-1)[32 * 896 + 64:])
    torch.cuda.synchronize()
    got = got.view(896, m)
    assert plan.status() == 0 and plan.describe()["ran"] == "tf32wd_256x256" and _off(got, want) <= 1e-5
    assert torch.equal(got[:64], c.view(896, m)[:64]) and torch.equal(got[832:], c.view(896, m)[832:])
    plan.close()


def test_a_wait_of_the_pairs_that_gives_up(pkg):
    import torch
    expr = "C [a,1024,b,768] += sum(c,300) * A [c,a] * B [c,b];"
    c, a, b, want = _matrices(1024, 768, 300)
    bad = pkg.Plan(expr, pkg.F32, test_fault=1)
    bad.execute(c.clone(), a, b)
    torch.cuda.synchronize()
    assert bad.status() in range(10, 18) and bad.describe()["ran"] == "tf32wd_256x256"
    bad.close()
    for _ in range(2):  # tensor memory was released
        good, got = pkg.Plan(expr, pkg.F32), c.clone()
        good.execute(got, a, b)
        torch.cuda.synchronize()
        assert good.status() == 0 and _off(got, want) <= 1e-5
        good.close()


# Output-resident kernels, panels and ring, whose waits run out (one stage is left unannounced): Y by copies of the threads,
# by boxes, X by boxes; they end by themselves with the tiles of C that were on their way landed, and the next plan is right.
GIVE_UP = [("C [a,24,b,16,c,16,d,24,e,16,f,16] -= sum(g,24) * A [d,e,g,a] * B [g,f,b,c];", {}, "dmma_wp_128x64", (False, False)),
           ("C [a,48,b,64,c,40,d,80] += sum(e,40) * A [a,b,e] * B [e,c,d];", dict(tile=(128, 64), variant=4), "dmma_wp_128x64", (False, True)),
           ("C [a,48,b,64,c,40,d,80] = sum(e,40) * A [e,a,b] * B [c,d,e];", dict(tile=(128, 64), variant=4), "dmma_wp_128x64", (True, False)),
           ("C [a,48,b,64,c,40,d,20] += sum(e,40) * A [e,a,b] * B [e,c,d];", dict(tile=(128, 64), variant=4), "dmma_wc_128x64", (True, True)),
           ("C [a,48,b,64,c,40,d,20] += sum(e,40) * A [a,e,b] * B [c,e,d];", dict(tile=(128, 32), variant=4), "dmma_wc_128x32", (False, False))]


@pytest.mark.parametrize("expr,kw,runs,boxes", GIVE_UP)
def test_resident_tiles_and_waits_that_give_up(pkg, orc, expr, kw, runs, boxes):
    import torch
    torch.cuda.set_device(0)
    c0, a, b = (torch.from_numpy(x).cuda() for x in orc.make_inputs(expr, 14, "float64"))
    bad = pkg.Plan(expr, test_fault=1, **kw)
    d = bad.describe()
    assert d["runs"] == runs and (d["tma_x"], d["tma_y"]) == boxes, d
    bad.execute(c0.clone(), a, b)
    torch.cuda.synchronize()          # returns: every wait is bounded
    assert bad.status() in (1, 2, 3, 4, 5, 6) and bad.describe()["ran"] == runs
    bad.close()
    d, err = _run(pkg, orc, expr, seed=14, **kw)
    assert d["runs"] == runs and err <= 1e-12, err


def test_helper_threads_are_one_set_for_all_plans(pkg, orc):
    """Pageable host arrays: the helpers that share the copies belong to the process, not to each plan, and go with the last
    plan that used them.  Two plans at once, from two threads, each checked."""
    import threading
    import numpy as np
    import torch
    torch.cuda.set_device(0)
    tasks = lambda: len(__import__("os").listdir("/proc/self/task"))
    exprs = ["C [a,128,b,96,c,40,d,10] %s sum(e,6) * A [a,e,b,d] * B [e,c];" % op for op in ("+=", "-=")]  # 39 MB of output: slabs
    data = [orc.make_inputs(e, 15 + n, "float64") for n, e in enumerate(exprs)]
    refs = [orc.contract(e, c.copy(), a, b) for e, (c, a, b) in zip(exprs, data)]
    with_threads = pkg.Plan(exprs[0])                      # whatever the driver starts for itself is there after this
    with_threads.execute_host(data[0][0].copy(), *data[0][1:])
    with_threads.close()
    start = tasks()
    plans = [pkg.Plan(e) for e in exprs]
    got = [[c.copy() for _ in range(3)] for c, _, _ in data]

    def work(n):
        for c in got[n]:
            plans[n].execute_host(c, *data[n][1:])

    callers = [threading.Thread(target=work, args=(n,)) for n in range(2)]
    for t in callers:
        t.start()
    for t in callers:
        t.join()
    assert tasks() - start <= 12, (start, tasks())
    plans[0].close()
    plans[1].close()
    assert tasks() <= start, (start, tasks())
    for ref, results in zip(refs, got):
        for c in results:
            assert np.abs(c - ref).max() <= 1e-12 * np.abs(ref).max()


# Epilogues of the one-tile kernels: few columns of a tile (groups of eight and sixteen outside the tensor), even rows whose
# pairs leave by 16 bytes, odd ones that do not, on tiles that are full and ragged.
@pytest.mark.parametrize("op", ["=", "+=", "-="])
@pytest.mark.parametrize("dtype,tile,kernel", [("float64", (64, 64), "dmma_64x64_w4"), ("float64", (64, 96), "dmma_64x96_w4"), ("float32", (64, 64), "tf32_64x64")])
@pytest.mark.parametrize("m,n", [(58, 8), (58, 9), (59, 16), (130, 17), (131, 49), (22, 73), (66, 111)])
def test_one_tile_epilogues_on_few_columns(pkg, orc, op, dtype, tile, kernel, m, n):
    expr = "C [a,%d,b,%d,c,3] %s sum(d,23) * A [d,a,c] * B [b,d];" % (m, n, op)
    d, err = _run(pkg, orc, expr, seed=16, dtype=dtype, tile=tile, variant=1)
    assert d["runs"] == kernel and d["vec_c"] == 2 - m % 2, d
    assert err <= (1e-12 if dtype == "float64" else 1e-5), err
