"""Searches without the distance and context-vector terms: sizes at the ends
of the kernel's 128 columns and 32 rows, frequencies and backgrounds outside
the ranges in which it multiplies by reciprocals (zeros, tiny and subnormal
products, small divisors: those blocks divide), with and without the SS term.
Scores and modular scores equal the oracle's bit for bit; the tensor-core
forms, which take their sums from another kernel, agree within 3e-5 (twice
their stated error in a cell's score)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _search(ss, q, db, ssswgt, form=0):
    import cother_b200 as cb
    o = cb.Options.defaults()
    o.ddmswgt = 0.0
    o.ssswgt = ssswgt
    o.tc_form = form
    o.autotune = 0
    with cb.BatchProcessing(ss, o) as bp:
        bp.transfer_cpm_data(db)
        bp.process_score_matrix(q)
        return bp.read_score_matrix(q.npositions, db.npositions)[:2]


@pytest.mark.parametrize("Lq,lens", [(1, [1]), (31, [127]), (32, [100, 28]), (33, [129, 3]), (70, [300, 1, 84])])
@pytest.mark.parametrize("values", ["usual", "zeros", "tiny", "divisors"])
def test_cells(ss_table, oracle_lib, Lq, lens, values):
    from cother_b200 import synth
    rng = np.random.default_rng(Lq)
    q = synth.make_profiles([Lq], 1300 + Lq, True)
    db = synth.make_profiles(lens, 1400 + Lq, False)
    if values == "zeros":
        q.tf[:10] *= rng.random((10, Lq)) < 0.5
        db.tf[:10] *= rng.random((10, db.npositions)) < 0.5
    elif values == "tiny":
        q.tf[::2] *= np.float32(1e-22)
        db.tf[1::3] *= np.float32(1e-21)
    elif values == "divisors":
        q.bkg[3] = 1e-6
        db.bkg[3] = 1e-7
        db.bkg[4] = 0.9999999
    for ssswgt in (0.12, 0.0):
        sc, ms = _search(ss_table, q, db, ssswgt)
        want = oracle_lib.score_matrix(q, db, ss_table, ssswgt=ssswgt, ddmswgt=0.0, nthreads=4)
        assert np.array_equal(sc, want[0])
        assert np.array_equal(ms, want[1])
        if values == "usual":
            for form in (1, 2):
                tsc, tms = _search(ss_table, q, db, ssswgt, form)
                assert np.abs(tsc - want[0]).max() < 3e-5
                assert np.array_equal(tms, want[1])
