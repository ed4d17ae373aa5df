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


@pytest.mark.parametrize("lanes", [2, 4])
def test_split_lists_hold_the_same_products(lanes):
    """every product once, each stored sum the work of one lane from its start, and no
    lane with more than its share by two"""
    for name, outs, _ in G.build():
        for c in G.pairs(outs):
            for h in range(2 if c else 0):
                lists = G.split_products(c, h, lanes)
                assert sorted(p[:4] for q in lists for p in q) == sorted(p[:4] for p in c.prods[h]), name
                want, cur = {}, []
                for p in c.prods[h]:
                    cur.append(p[:4])
                    if p[4]:
                        want[p[4][1]] = sorted(cur if p[4][0] == "sum" else cur[-1:])
                        cur = []
                got = {}
                for q in lists:
                    stores = [i for i, p in enumerate(q) if p[4]]
                    assert len(stores) <= 1
                    for i in stores:
                        assert q[i][4][0] == "sum"
                        got[q[i][4][1]] = sorted(p[:4] for p in q[:i + 1])
                assert got == want, name
                assert max(map(len, lists)) <= -(-len(c.prods[h]) // lanes) + 2


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
