"""The bench's product and reduction counts of the 32-item kernel are those of its own
programs and sequence (the five-item kernel's: test_fp2_programs.py)."""
import bench
import gen_fp2ops as G


def test_counts_of_the_paired_warp_sequence():
    progs = [G.pairs(outs) for _, outs, _ in G.build()]
    products = reductions = 0
    for op in G.kernel_ops(G.driver_sequence(True)):
        if op[0] & G.COND_ML:
            continue
        row = [G.line_pair(k) for k in range(6)] if op[0] == G.OP_LOAD_LINES else progs[op[0]] if op[0] < len(progs) else []
        for c in row:
            for h in range(2 if c is not None else 0):
                products += len(c.prods[h])
                reductions += bool(c.prods[h]) and not c.invfp
    assert (products, reductions) == bench.OWN_WORK["k_verify_w"]
    assert bench.OWN_WORK["k_verify_fp2"] == (bench.OWN_PRODUCTS_PER_VERIFY, bench.OWN_REDC_PER_VERIFY)
