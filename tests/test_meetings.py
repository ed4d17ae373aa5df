"""The 32-item kernel's meetings between ops (gen_fp2ops.py: meeting_kinds,
check_meetings): the reduced ones are proved from what the programs read and write, the
proof refuses the ones that would race, and the kernel takes them from the generator."""
import os
import re

import pytest

import gen_fp2ops as G

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "icp-gpu_b200", "csrc")
NAMES = [n for n, _, _ in G.PROGRAMS]
SEQS = [G.kernel_ops(G.driver_sequence(norm)) for norm in (False, True)]


@pytest.fixture(params=[0, 1], ids=["raw", "normalised"])
def ops(request):
    return SEQS[request.param]


def test_reduced_meetings_hold(ops):
    kinds, sets = G.meeting_kinds(ops), G.cyc_sets()
    assert sets == [{0, 4}, {1, 2, 3, 5}]
    assert kinds.count(G.MEET_SETS) > 250 and kinds.count(G.MEET_NONE) > 50
    G.check_meetings(ops, kinds, sets)


def name(op):
    code = op[0] & ~G.COND_ML
    return "LOAD" if code == G.OP_LOAD_LINES else NAMES[code] if code < len(NAMES) else "other"


@pytest.mark.parametrize("pair", [("LOAD", "LINE"), ("LINE", "SQR"), ("CYCSQR", "CYCSQR"), ("CYCSQR", "MUL")],
                         ids="-".join)
def test_a_meeting_left_out_is_refused(ops, pair):
    kinds = G.meeting_kinds(ops)
    at = next(i for i in range(len(ops) - 1) if name(ops[i]).startswith(pair[0]) and name(ops[i + 1]).startswith(pair[1]))
    kinds[at] = G.MEET_NONE
    with pytest.raises(AssertionError):
        G.check_meetings(ops, kinds, G.cyc_sets())


@pytest.mark.parametrize("sets", [[{0}, {4}, {1, 2, 3, 5}], [{0, 4}, {1, 2}, {3, 5}], [{0, 1}, {4, 2, 3, 5}]], ids=str)
def test_sets_that_read_each_other_are_refused(ops, sets):
    with pytest.raises(AssertionError):
        G.check_meetings(ops, G.meeting_kinds(ops), sets)


@pytest.mark.parametrize("change", ["stores a partial sum", "writes the point"])
def test_a_line_load_in_the_way_is_refused(ops, monkeypatch, change):
    real = G.line_pair

    def line_pair(k):
        c = real(k)
        if c is not None and change == "stores a partial sum":
            c.prods[0] = [c.prods[0][0][:4] + (("sum", 0),)]
        if c is not None and change == "writes the point":
            c.dst = G.ref(G.B_A, 0) if k == 0 else c.dst
        return c
    monkeypatch.setattr(G, "line_pair", line_pair)
    loads = [(op[0], *ops[i - 1][1:4], op[4]) if op[0] == G.OP_LOAD_LINES else op for i, op in enumerate(ops)]
    with pytest.raises(AssertionError):
        G.check_meetings(loads, G.meeting_kinds(loads), G.cyc_sets())


def test_kernel_takes_them_from_the_generator():
    inc = open(os.path.join(CSRC, "fp2ops.inc")).read()
    rows = re.search(r"kSeq\[2\]\[\d+\] = \{(.*?)\n\};", inc, re.S).group(1).split("},")
    for norm in range(2):
        words = [int(w, 16) for w in re.findall(r"0x([0-9a-f]+)u", rows[norm])]
        ops, seq = SEQS[norm], G.driver_sequence(bool(norm))
        kinds = G.meeting_kinds(ops)
        got = [w >> G.MEET_SHIFT for w, op in zip(words, seq) if op[0] != NAMES.index("LSCALE")]
        assert got == kinds
    src = open(os.path.join(CSRC, "verify_w.cu")).read()
    assert "f2::kMeetSet >> k" in src and "f2::kMeetShift" in src and not re.search(r"k == 4", src)
