"""Several contractions accumulated into one output in one pass (tc_plan_create_fused / tc_execute_fused).

The term lists are the reference's CCSD(T) doubles terms: sd_t_d2 and sd_t_d1
(cogent/input_strings/ccsd_t/original-expressions/sd_t_d2.in:4-30, sd_t_d1.in), written in the expression grammar
with one pair of inputs per term, as the reference's drivers hold them (cogent/drivers/ccsd_t/code_main_sd2_1.c:12-14:
host_t2_1..9, host_v2_1..9).  The checker applies the nine loop nests one after another."""
import numpy as np
import pytest

OUT = "t3 [h3,{h3},h2,{h2},h1,{h1},p6,{p6},p5,{p5},p4,{p4}]"
# (operator, left indices, right indices): which of the output's indices each input of the term carries
SD2 = [("-=", "p7,p4,h1,h2", "p7,h3,p6,p5"), ("-=", "p7,p4,h2,h3", "p7,h1,p6,p5"), ("+=", "p7,p4,h1,h3", "p7,h2,p6,p5"),
       ("+=", "p7,p5,h1,h2", "p7,h3,p6,p4"), ("+=", "p7,p5,h2,h3", "p7,h1,p6,p4"), ("-=", "p7,p5,h1,h3", "p7,h2,p6,p4"),
       ("-=", "p7,p6,h1,h2", "p7,h3,p5,p4"), ("-=", "p7,p6,h2,h3", "p7,h1,p5,p4"), ("+=", "p7,p6,h1,h3", "p7,h2,p5,p4")]
SD1 = [("-=", "h7,p4,p5,h1", "h3,h2,p6,h7"), ("+=", "h7,p4,p5,h2", "h3,h1,p6,h7"), ("-=", "h7,p4,p5,h3", "h2,h1,p6,h7"),
       ("-=", "h7,p5,p6,h1", "h3,h2,p4,h7"), ("+=", "h7,p5,p6,h2", "h3,h1,p4,h7"), ("-=", "h7,p5,p6,h3", "h2,h1,p4,h7"),
       ("+=", "h7,p4,p6,h1", "h3,h2,p5,h7"), ("-=", "h7,p4,p6,h2", "h3,h1,p5,h7"), ("+=", "h7,p4,p6,h3", "h2,h1,p5,h7")]


def _lines(terms, ext, sum_name):
    out = OUT.format(**ext)
    return ["%s %s sum(%s,%d) * t2_%d [%s] * v2_%d [%s];" % (out, op, sum_name, ext[sum_name], k + 1, l, k + 1, r)
            for k, (op, l, r) in enumerate(terms)]


def test_fused_plan_shape_without_a_gpu(pkg):
    ext = dict(h3=16, h2=16, h1=16, p6=24, p5=16, p4=20, p7=24)
    d = pkg.FusedPlan(_lines(SD2, ext, "p7")).describe()
    assert d["terms"] == 9 and d["rank"] == 6 and d["box"] == [4] * 6 and d["box_elems"] == 4096
    assert d["rows_cols"] == [[64, 64]] * 9
    assert d["boxes"] == 4 * 4 * 4 * 6 * 4 * 5
    out = 16 * 16 * 16 * 24 * 16 * 20
    assert d["flops"] == 9 * 2.0 * out * 24
    # the output travels once instead of nine times
    assert d["bytes_term_by_term"] - d["bytes"] == 8 * 2.0 * 8 * out
    # terms must share the output; '=' cannot be fused; more than 64 rows per box is refused
    with pytest.raises(pkg.TcError) as e:
        pkg.FusedPlan(["t3 [a,4,b,4] += sum(c,4) * x [c,a] * y [c,b];", "t3 [b,4,a,4] += sum(c,4) * x [c,a] * y [c,b];"])
    assert e.value.status == 2
    with pytest.raises(pkg.TcError) as e:
        pkg.FusedPlan(["t3 [a,4,b,4] = sum(c,4) * x [c,a] * y [c,b];"])
    assert e.value.status == 3
    one = pkg.FusedPlan(["t3 [a,40,b,40] += sum(c,4) * x [c,a] * y [c,b];"]).describe()
    assert one["box"] == [40, 40] and one["rows_cols"] == [[40, 40]]


def _retried(pkg, lines):
    """A plan whose first commit met a limit in its last term, given extents that fit."""
    plan = pkg.FusedPlan(lines, extents={"q7": 1 << 31})
    with pytest.raises(pkg.TcError) as e:
        plan.commit()
    assert e.value.status == 3
    names = (pkg.ctypes.c_char_p * 1)(b"q7")
    assert pkg.lib().tc_fused_set_extents(plan._h, 1, names, (pkg.ctypes.c_int64 * 1)(16)) == 0
    return plan


RETRIED = [
    ["t3 [a,33,b,20] += sum(p7,16) * x1 [p7,a] * y1 [p7,b];", "t3 [a,33,b,20] -= sum(q7,16) * x2 [q7,a] * y2 [q7,b];"],
    ["t3 [a,8,b,9,c,5,d,7] += sum(p7,16) * x1 [p7,c,a] * y1 [p7,b,d];", "t3 [a,8,b,9,c,5,d,7] -= sum(q7,16) * x2 [q7,b,a] * y2 [q7,d,c];"],
    ["t3 [h3,8,h2,8,h1,4,p6,5,p5,4,p4,9] += sum(p7,10) * x1 [p7,p4,h1,h2] * y1 [p7,h3,p6,p5];",
     "t3 [h3,8,h2,8,h1,4,p6,5,p5,4,p4,9] += sum(q7,10) * x2 [q7,p5,h1,h2] * y2 [q7,h3,p6,p4];"],
]


@pytest.mark.parametrize("lines", RETRIED)
def test_a_commit_after_one_that_failed_builds_the_plan_anew(pkg, lines):
    got = _retried(pkg, lines).describe()
    fresh = pkg.FusedPlan(lines, extents={"q7": 16}).describe()
    assert got == fresh and got["kernel"] == "tc_fused_box_kernel"
    for left, right in got["maps"]:
        assert sorted(left + right) == list(range(got["rank"]))


@pytest.mark.gpu
@pytest.mark.parametrize("lines", RETRIED)
def test_a_plan_committed_on_a_second_try_against_the_loop_nests(pkg, orc, lines):
    import torch
    torch.cuda.set_device(0)
    sized = [lines[0], lines[1].replace("q7,10)", "q7,16)")]
    plan = _retried(pkg, lines)
    c0 = orc.uniform(62, 0, orc.sizes(lines[0])[0])
    ref, ins = c0.copy(), []
    for n, line in enumerate(sized):
        _, na, nb = orc.sizes(line)
        a, b = orc.uniform(63 + n, 1, na), orc.uniform(63 + n, 2, nb)
        orc.contract(line, ref, a, b)
        ins.append((torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()))
    dc = torch.from_numpy(c0).cuda()
    plan.execute(dc, [a for a, _ in ins], [b for _, b in ins])
    torch.cuda.synchronize()
    assert orc.rel_error(dc.cpu().numpy(), ref) <= 1e-12
    plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name,terms,sum_name,ext", [
    ("sd2", SD2, "p7", dict(h3=16, h2=16, h1=16, p6=16, p5=16, p4=16, p7=16)),
    ("sd1", SD1, "h7", dict(h3=16, h2=16, h1=16, p6=16, p5=16, p4=16, h7=16)),
    ("sd2 mixed", SD2, "p7", dict(h3=20, h2=16, h1=24, p6=16, p5=20, p4=16, p7=24)),
    ("sd1 ragged", SD1, "h7", dict(h3=10, h2=7, h1=9, p6=6, p5=11, p4=5, h7=13)),
])
def test_fused_terms_against_the_loop_nests(pkg, orc, name, terms, sum_name, ext):
    import torch
    torch.cuda.set_device(0)
    lines = _lines(terms, ext, sum_name)
    n_out = orc.sizes(lines[0])[0]
    c0 = orc.uniform(60, 0, n_out)
    ins = []
    ref = c0.copy()
    for k, line in enumerate(lines):
        _, na, nb = orc.sizes(line)
        a, b = orc.uniform(61 + k, 1, na), orc.uniform(61 + k, 2, nb)
        ins.append((a, b))
        orc.contract(line, ref, a, b, threads=orc.max_threads())   # the nine nests, one after another
    plan = pkg.FusedPlan(lines)
    dc = torch.from_numpy(c0).cuda()
    das = [torch.from_numpy(a).cuda() for a, _ in ins]
    dbs = [torch.from_numpy(b).cuda() for _, b in ins]
    plan.execute(dc, das, dbs)
    torch.cuda.synchronize()
    assert orc.rel_error(dc.cpu().numpy(), ref) <= 1e-12, name
    # the same terms one by one through ordinary plans give the same tensor (up to the order of the additions)
    dc2 = torch.from_numpy(c0).cuda()
    for line, da, db in zip(lines, das, dbs):
        q = pkg.Plan(line)
        q.execute(dc2, da, db)
        q.close()
    torch.cuda.synchronize()
    assert orc.rel_error(dc2.cpu().numpy(), ref) <= 1e-12
    assert orc.rel_error(dc.cpu().numpy(), dc2.cpu().numpy()) <= 1e-12
    plan.close()


@pytest.mark.gpu
def test_fused_terms_with_other_shapes(pkg, orc):
    """Two contraction indices (fastest in different inputs), a 4-D and a 2-D output, odd contraction extents."""
    import torch
    torch.cuda.set_device(0)
    cases = [
        ["C [a,12,b,9,c,10,d,7] += sum(e,5,f,6) * X1 [e,a,f,c] * Y1 [f,b,e,d];",
         "C [a,12,b,9,c,10,d,7] -= sum(e,5,f,6) * X2 [b,e,d,f] * Y2 [e,f,c,a];",
         "C [a,12,b,9,c,10,d,7] += sum(e,5,f,6) * X3 [f,e,a,b] * Y3 [c,d,f,e];"],
        ["C [a,70,b,45] += sum(k,33) * X1 [k,a] * Y1 [k,b];", "C [a,70,b,45] -= sum(k,33) * X2 [a,k] * Y2 [b,k];"],
    ]
    for lines in cases:
        n_out = orc.sizes(lines[0])[0]
        c0 = orc.uniform(70, 0, n_out)
        ref = c0.copy()
        ins = []
        for k, line in enumerate(lines):
            _, na, nb = orc.sizes(line)
            a, b = orc.uniform(71 + k, 1, na), orc.uniform(71 + k, 2, nb)
            ins.append((a, b))
            orc.contract(line, ref, a, b)
        plan = pkg.FusedPlan(lines)
        dc = torch.from_numpy(c0).cuda()
        plan.execute(dc, [torch.from_numpy(a).cuda() for a, _ in ins], [torch.from_numpy(b).cuda() for _, b in ins])
        torch.cuda.synchronize()
        assert orc.rel_error(dc.cpu().numpy(), ref) <= 1e-12, lines[0]
        plan.close()


@pytest.mark.gpu
@pytest.mark.parametrize("p7,kernel", [(16, "tc_fused_box_kernel"), (15, "tc_fused_kernel")])
def test_terms_are_summed_before_they_meet_the_output(pkg, orc, p7, kernel):
    """One rounding against C's magnitude however many terms there are: with values of C around 1e6 and terms around 1,
    the result is within half a unit in the last place of C plus the exact sum of the terms (whose own error, 1e-12 of
    their largest value as everywhere, is a thousandth of that unit)."""
    import torch
    torch.cuda.set_device(0)
    lines = _lines(SD2, dict(h3=5, h2=8, h1=6, p6=4, p5=9, p4=7, p7=p7), "p7")
    plan = pkg.FusedPlan(lines)
    assert plan.describe()["kernel"] == kernel
    c0 = orc.uniform(70, 0, orc.sizes(lines[0])[0]) * 1e6
    total, ins = np.zeros_like(c0), []
    for n, line in enumerate(lines):
        _, na, nb = orc.sizes(line)
        a, b = orc.uniform(71 + n, 1, na), orc.uniform(71 + n, 2, nb)
        orc.contract(line, total, a, b)
        ins.append((torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()))
    dc = torch.from_numpy(c0).cuda()
    plan.execute(dc, [a for a, _ in ins], [b for _, b in ins])
    torch.cuda.synchronize()
    got = dc.cpu().numpy()
    off = np.abs(got.astype(np.longdouble) - (c0.astype(np.longdouble) + total.astype(np.longdouble)))
    assert (off <= 0.5 * np.spacing(np.abs(got)) + 1e-12 * np.abs(total).max()).all()
    plan.close()


def test_fused_status_calls_check_their_arguments(pkg):
    plan = pkg.FusedPlan(RETRIED[0], extents={"q7": 16})
    lib = pkg.lib()
    word = pkg.ctypes.c_int()
    assert lib.tc_fused_status(plan._h, pkg.ctypes.byref(word)) == 7 and lib.tc_fused_status_reset(plan._h) == 7
    assert lib.tc_fused_status(None, pkg.ctypes.byref(word)) == 2 and lib.tc_fused_status(plan._h, None) == 2
    assert lib.tc_fused_status_reset(None) == 2
    assert lib.tc_fused_set_test_fault(plan._h, 2) == 2 and lib.tc_fused_set_test_fault(None, 1) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("p7", [10, 40])  # the stage left out is the second term's, or the first term's second
def test_a_fused_wait_that_gives_up_reports_and_leaves_the_output(pkg, orc, p7):
    """One CTA never gets one stage: its waits run out, the kernel ends, the status word says so, that CTA's boxes of C
    are as they were, and the context goes on working."""
    import torch
    torch.cuda.set_device(0)
    lines = _lines(SD2, dict(h3=4, h2=4, h1=4, p6=4, p5=4, p4=4, p7=p7), "p7")  # one box
    c0, total, ins = orc.uniform(80, 0, orc.sizes(lines[0])[0]), None, []
    total = c0.copy()
    for n, line in enumerate(lines):
        _, na, nb = orc.sizes(line)
        a, b = orc.uniform(81 + n, 1, na), orc.uniform(81 + n, 2, nb)
        orc.contract(line, total, a, b)
        ins.append((torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()))
    lefts, rights = [a for a, _ in ins], [b for _, b in ins]
    bad = pkg.FusedPlan(lines, test_fault=1)
    assert bad.describe()["kernel"] == "tc_fused_box_kernel"
    dc = torch.from_numpy(c0).cuda()
    bad.execute(dc, lefts, rights)
    assert bad.status() != 0
    assert np.array_equal(dc.cpu().numpy(), c0)
    with pytest.raises(pkg.TcError) as e:
        bad.execute(dc, lefts, rights)
    assert e.value.status == 9
    bad.status_reset()
    assert bad.status() == 0
    bad.execute(dc, lefts, rights)
    assert bad.status() != 0
    bad.close()
    good = pkg.FusedPlan(lines)
    good.execute(dc, lefts, rights)
    assert good.status() == 0 and orc.rel_error(dc.cpu().numpy(), total) <= 1e-12
    good.close()
