"""The paired-warp form of the tower programs (gen_fp2ops.py; verify_w.cu) on the CPU:
every program against the oracle on redundant inputs, the whole verify through its
op sequence, and the line load against LSCALE."""
import pytest

import gen_fp2ops as G
import test_fp2_programs as T


@pytest.fixture(autouse=True)
def paired_warp_form(monkeypatch):
    monkeypatch.setattr(G, "Emulator", G.PairEmulator)


def test_programs_against_oracle():
    T.test_programs_against_oracle()
    T.test_lines_against_oracle()
    T.test_inverse_of_zero_is_zero()


@pytest.mark.parametrize("normalised", [False, True], ids=["raw-lines", "normalised-lines"])
def test_full_verify_through_programs(golden, normalised):
    T.test_full_verify_through_programs(golden, normalised)


def test_line_load_is_lscale():
    """the line load's descriptors name LSCALE's outputs and operands"""
    outs = dict((n, o) for n, o, _ in G.build())["LSCALE"]
    want = {(t.dst, h): t.prods[h] for t in (G.Pair(o) for o in outs if o is not None) for h in range(2)}
    got = {}
    for k in range(6):
        c = G.line_pair(k)
        for h in range(2 if c is not None else 0):
            (uf, _, vf, vr, store), = c.prods[h]
            assert uf == G.X_LINE and not c.adds[h]
            got[(c.dst, h)] = [((G.X_0, G.X_1)[h], G.ref(G.B_C, 6 * (k // 3) + k % 3), vf, vr, store)]
    assert got == want
