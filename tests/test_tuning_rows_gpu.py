"""The tuner's choice of the score kernel's rows per block: the variant that
is the fastest on whole searches (8 rows with the distance term, 32 without),
unless the sample shows another to be faster by more than its noise."""
import pytest

pytestmark = pytest.mark.gpu

ROWS = (16, 8, 32, 16, 16)              # of the candidates, in the order of their times
WINDOWS = (1024, 1024, 1024, 256, 4096)
MARGIN = 0.015


@pytest.mark.parametrize("ddmswgt,preferred", [(0.2, 1), (0.0, 2)])
def test_preferred_rows(ss_table, ddmswgt, preferred):
    import cother_b200 as cb
    from cother_b200 import synth
    db = synth.make_profiles([200] * 40, 2101, False)
    o = cb.Options.defaults()
    o.ddmswgt = ddmswgt
    for Lq in (70, 130, 200, 260, 330, 400):
        # two queries, whose kernel without the distance term has the variants too
        qs = [synth.make_profiles([n], 2110 + n, True) for n in (Lq - 40, 40)]
        with cb.BatchProcessing(ss_table, o) as bp:
            bp.transfer_cpm_data(db)
            bp.process_batch(qs)
            t = bp.tuning(Lq)
        ms = t["score_candidates_ms"]
        best = min(range(5), key=lambda k: ms[k])
        want = best if ms[best] <= (1.0 - MARGIN) * ms[preferred] else preferred
        assert (t["score_rows"], t["order_window"]) == (ROWS[want], WINDOWS[want]), (Lq, t)
